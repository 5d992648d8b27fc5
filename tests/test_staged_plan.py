"""How products of staged rows are dealt to blocks (fk_qplan.h), compiled and run on the host."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DRIVER = r"""
#include "fk_qplan.h"
#include <stdio.h>
#include <stdlib.h>
#include <vector>
#define CHECK(x) do { if (!(x)) { printf("line %d: m %d ntiles %d nsb %d sm %d: %s\n", __LINE__, m, nt, nsb, sm, #x); return 1; } } while (0)

// every storing warp of every block, each giving up at a piece of its own or never: the ticket words end at zero, and a tile that no warp
// gave up on is finished once
static int tickets(int m, int nt, int nsb, int sm, int share) {
    const QPlan p = fkq_plan(m, nt, nsb, sm);
    if (p.whole) return 0;
    std::vector<int> word((size_t)p.tiles * FKQ_EPI, 0), finished(word.size(), 0), lost(word.size(), 0);
    for (int b = 0; b < p.grid; ++b)
        for (int ew = 0; ew < FKQ_EPI; ++ew) {
            const int stop = rand() % 100 < share ? rand() % 3 : 1 << 30;
            auto count = [&](int tile) {
                int &c = word[(size_t)tile * FKQ_EPI + ew];
                if (++c == fkq_parts(p.tiles, nsb, p.grid, tile)) { c = 0; return true; }
                return false;
            };
            fkq_pieces(p.whole, p.tiles, nsb, b, p.grid, [&](int v, const QWork &w) {
                if (v >= stop) return false;
                if (!fkq_part(w, nsb)) ++finished[(size_t)w.tile * FKQ_EPI + ew];
                else if (count(w.tile)) ++finished[(size_t)w.tile * FKQ_EPI + ew];
                return true;
            }, [&](const QWork &w) { count(w.tile); });
            QWork w;
            for (int v = stop; v < 1 << 29 && fkq_work(p.whole, p.tiles, nsb, b, p.grid, v, w); ++v) ++lost[(size_t)w.tile * FKQ_EPI + ew];
        }
    for (size_t i = 0; i < word.size(); ++i) { CHECK(word[i] == 0); CHECK(finished[i] == 1 || lost[i]); }
    return 0;
}

// every step of every tile is dealt once; only tiles of up to FKQ_SPLIT_ROWS rows in parts, two of them a block at most, each in a slot of its own
static int cover(int m, int nt, int nsb, int sm) {
    const QPlan p = fkq_plan(m, nt, nsb, sm);
    CHECK(p.bn >= 16 && p.bn <= 128 && p.grid >= 1 && p.grid <= sm && (p.whole || p.bn <= FKQ_SPLIT_ROWS));
    CHECK(p.whole || p.tiles <= FKQ_COUNTERS / FKQ_EPI);
    std::vector<int> next(p.tiles, 0), slot(2 * p.grid, 0), parts(p.tiles, 0);
    for (int b = 0; b < p.grid; ++b) {
        QWork w;
        for (int v = 0; fkq_work(p.whole, p.tiles, nsb, b, p.grid, v, w); ++v) {
            CHECK(w.tile >= 0 && w.tile < p.tiles && w.k0 < w.k1 && next[w.tile] == w.k0);
            next[w.tile] = w.k1;
            if (!fkq_part(w, nsb)) continue;
            const int s = fkq_slot(p.tiles, nsb, p.grid, b, w.tile);
            CHECK(!p.whole && s >= 0 && s < 2 * p.grid && slot[s]++ == 0 && fkq_owner(p.tiles, nsb, p.grid, w.tile * nsb) + parts[w.tile]++ == b);
        }
    }
    for (int t = 0; t < p.tiles; ++t) CHECK(next[t] == nsb && (parts[t] == 0 || parts[t] == fkq_parts(p.tiles, nsb, p.grid, t)));
    return 0;
}

int main(int argc, char **argv) {
    srand(7);
    const int sms[] = {132, 148, 160}, ms[] = {1, 5, 16, 17, 32, 33, 100, 1000};
    if (argc > 1) {
        for (int sm : sms) for (int m : ms) for (int i = 0; i < 400; ++i) if (cover(m, 1 + rand() % (i % 2 ? 2600 : 160), 1 + rand() % 64, sm)) return 1;
        printf("ok\n");
        return 0;
    }
    for (int sm : sms) for (int m : ms) for (int i = 0; i < 150; ++i) {
        const int nt = 1 + rand() % 2600, nsb = 1 + rand() % 64;
        for (int share : {0, 3, 100}) if (tickets(m, nt, nsb, sm, share)) return 1;
    }
    printf("ok\n");
    return 0;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(DRIVER)
    exe = str(d / "plan")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "fusekit_b200", "csrc"), "-o", exe, str(d / "plan.cpp")])
    return exe


def test_ticket_words_are_zero_after_every_launch(driver):
    """Also after one in which storing warps gave up: the next product would otherwise take old parts for its own."""
    p = subprocess.run([driver], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and p.stdout == "ok\n", p.stdout


def test_every_step_is_dealt_once_and_parts_are_narrow(driver):
    p = subprocess.run([driver, "cover"], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and p.stdout == "ok\n", p.stdout
