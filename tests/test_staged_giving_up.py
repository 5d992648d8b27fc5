"""Storing warps of a staged product that give up: none of them is waited for at a barrier afterwards (fk_qplan.h, compiled and run on the host)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DRIVER = r"""
#include "fk_qplan.h"
#include <stdio.h>
#include <stdlib.h>
// The four storing warps of an accumulator over the pieces of a block, warp `who` giving up at piece `at`.  At a whole tile of FKQ_MOST_ROWS rows they vote at a
// barrier of all four and leave together; at a part each leaves by itself.  False: a barrier waits for a warp that left.
static bool walk(const QPlan &p, int nsb, int b, int who, int at) {
    bool left[4] = {false, false, false, false};
    QWork w;
    for (int v = 0; fkq_work(p.whole, p.tiles, nsb, b, p.grid, v, w); ++v) {
        if (fkq_part(w, nsb)) { if (v == at) left[who] = true; continue; }
        if (left[0] && left[1] && left[2] && left[3]) return true;
        for (bool l : left) if (l) return false;
        if (v == at) for (bool &l : left) l = true;
    }
    return true;
}
int main() {
    srand(11);
    const int most[3][3] = {{74, 33, 15}, {74, 36, 18}, {74, 0, 0}};
    int wide = 0;
    for (int i = 0; i < 20000; ++i) {
        // among them a run of a part, a whole tile and a part when tiles of 128 rows are dealt in equal runs: 1018 x 10752 -> 5888
        const int m = i ? 1 + rand() % 1100 : 1018, nt = i ? 1 + rand() % (i % 2 ? 2600 : 400) : 368, nsb = i ? 1 + rand() % 64 : 21;
        const QPlan p = fkq_choose(m, nt, nsb, i % 3 ? 148 : 132, most[i % 3]);
        if (p.whole < 0 || p.bn != FKQ_MOST_ROWS) continue;      // a cluster's blocks have one piece; narrower tiles meet at no barrier
        ++wide;
        for (int b = 0; b < p.grid; b += 1 + rand() % 7) for (int who = 0; who < 4; ++who) for (int at = 0; at < 5; ++at)
            if (!walk(p, nsb, b, who, at)) { printf("m %d ntiles %d nsb %d block %d: warp %d gone at piece %d\n", m, nt, nsb, b, who, at); return 1; }
    }
    printf("%s\n", wide > 1000 ? "ok" : "few");
    return 0;
}
"""


def test_no_barrier_waits_for_a_warp_that_gave_up(tmp_path):
    (tmp_path / "walk.cpp").write_text(DRIVER)
    exe = str(tmp_path / "walk")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "fusekit_b200", "csrc"), "-o", exe, str(tmp_path / "walk.cpp")])
    p = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and p.stdout == "ok\n", p.stdout
