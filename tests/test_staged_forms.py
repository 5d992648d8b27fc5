"""Shapes that make the staged product take each of its forms (fk_qplan.h, compiled and run on the host), so that a change of its dispatch drops none of them from the GPU
tests that run these shapes."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# (m, k, n) -> the form: "cluster", "parts" (sums that meet in memory, with ticket words), "lines" (tiles of 128 rows, whole), "tiles" (narrower ones, whole); long:
# sums in stretches
FORMS = {(40, 1024, 512): "cluster", (16, 4096, 304): "cluster", (200, 4096, 4096): "cluster", (16, 4096, 40000): "parts", (32, 5632, 40000): "parts long", (300, 512, 20000): "lines",
         (200, 5632, 12800): "lines long", (64, 512, 40000): "tiles", (64, 5632, 37000): "tiles long"}

DRIVER = r"""
#include "fk_qplan.h"
#include <stdio.h>
#include <stdlib.h>
int main(int argc, char **argv) {
    const int most[4][3] = {{74, 33, 15}, {74, 36, 18}, {72, 32, 14}, {74, 37, 16}};        // clusters of 2, 4 and 8 blocks that a device holds
    for (int i = 1; i + 2 < argc; i += 3) {
        const int m = atoi(argv[i]), nsb = (atoi(argv[i + 1]) + 511) / 512, ntiles = (atoi(argv[i + 2]) + 15) / 16;
        for (auto &c : most) {
            const QPlan p = fkq_choose(m, ntiles, nsb, 148, c);
            bool parts = false;
            QWork w;
            if (!p.whole) for (int b = 0; b < p.grid; ++b) for (int v = 0; fkq_work(0, p.tiles, nsb, b, p.grid, v, w); ++v) parts = parts || fkq_part(w, nsb);
            printf("%s%s%s", p.whole < 0 ? "cluster" : parts ? "parts" : p.bn == FKQ_MOST_ROWS ? "lines" : "tiles", p.whole >= 0 && nsb > FKQ_SUM_STEPS ? " long" : "", &c == &most[3] ? "\n" : "|");
        }
    }
    return 0;
}
"""


def test_every_form_has_a_shape(tmp_path):
    (tmp_path / "forms.cpp").write_text(DRIVER)
    exe = str(tmp_path / "forms")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "fusekit_b200", "csrc"), "-o", exe, str(tmp_path / "forms.cpp")])
    out = subprocess.check_output([exe] + [str(v) for shape in FORMS for v in shape], text=True).splitlines()
    assert [set(line.split("|")) for line in out] == [{form} for form in FORMS.values()]
    assert len(set(FORMS.values())) == 7
