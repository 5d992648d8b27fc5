"""What the CTAs of a cluster store into each other's shared memory (fk_sdpa_layout.h), compiled and run on the host: nothing that a CTA keeps for itself lies there."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DRIVER = r"""
#include "fk_sdpa_layout.h"
#include <initializer_list>
#include <stdio.h>
struct Range { const char *name; int a, b; };
template <int HD, int CW> static int look(int G, int CL) {
    using L = SdpaMmaLayout<HD, CW>;
    const int per = (G * HD + CL - 1) / CL;
    const Range got[] = {{"outputs", L::cpart(), L::cpart() + CL * per * 4}, {"maxima and sums", L::wexp(G), L::wexp(G) + CL * G * 8}};
    const Range own[] = {{"queries", L::q(), L::q() + 8 * L::QSTRIDE}, {"tiles", L::tiles(), L::tiles() + CW * L::WTILE}, {"partials", L::tiles(), L::tiles() + (CW - 1) * L::WTILE + G * (HD + 2) * 4},
                         {"factors", L::fexp(G), L::fexp(G) + 18 * G * 4}, {"sums of q", L::qsum(G), L::qsum(G) + (8 * (HD / 64) + 8) * 4}};
    if (got[0].b > got[1].a || L::qsum(G) % 4 || L::fexp(G) % 4) { printf("hd %d G %d: received ranges\n", HD, G); return 1; }
    if (own[3].b > own[4].a) { printf("hd %d G %d: factors and sums\n", HD, G); return 1; }
    for (const Range &o : own) {
        if (o.b > (int)sdpa_mma_smem_bytes<CW>(G, HD)) { printf("hd %d G %d: %s past the end\n", HD, G, o.name); return 1; }
        for (const Range &r : got) if (o.a < r.b && r.a < o.b) { printf("hd %d CW %d G %d CL %d: %s in received %s\n", HD, CW, G, CL, o.name, r.name); return 1; }
    }
    return 0;
}
int main() {
    for (int CL : {1, 2, 4, 8, 16}) for (int G = 1; G <= 8; ++G) {
        if (look<64, 8>(G, CL) || look<64, 16>(G, CL) || look<128, 8>(G, CL) || look<128, 16>(G, CL)) return 1;
        if (G <= 2 && (look<256, 8>(G, CL) || look<256, 16>(G, CL))) return 1;
    }
    printf("ok\n");
    return 0;
}
"""


def test_received_ranges_hold_nothing_else(tmp_path):
    (tmp_path / "layout.cpp").write_text(DRIVER)
    exe = str(tmp_path / "layout")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "fusekit_b200", "csrc"), "-o", exe, str(tmp_path / "layout.cpp")])
    p = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert p.returncode == 0 and p.stdout == "ok\n", p.stdout
