"""The split of the symmetric products under scratch limits (csrc/product_plan.h), built for the host."""
import os
import subprocess

from conftest import ROOT

MAIN = r"""
#include <cstdio>
#include "product_plan.h"
int main()
{
    using namespace rmw;
    long long bad = 0, finer = 0;
    for (int n = 256; n < 60000; n += n < 3000 ? 17 : 331)
        for (int comps : {3, 6})
            for (int form = 0; form < 3; ++form) {  // df64, FP64, periodic FP64
                const double slot = sym_slot_bytes(n, comps), packed = (comps == 6 ? 96.0 : 64.0) * n, big = 1e11;
                const int s = sym_split(form > 0, form == 2, n, comps, packed, big, 0.0);
                bad += s < 1 || s > kSplitMax || (s > 1 && slot * s > kSplitBytes * comps / 3);
                for (int c = 1; c <= s; ++c)
                    for (double cap : {packed + slot * c, packed * 0.5 + slot * c, packed + slot * (c + 0.9)}) {
                        if (cap < packed + slot) continue;  // even whole tile pairs are refused
                        const int t = sym_split(form > 0, form == 2, n, comps, packed, cap, cap);
                        // fits, and no finer split of the rule's would
                        bad += packed + slot * t > cap || (t < s && packed + slot * (t + 1) <= cap);
                        finer += t > 1;
                    }
                bad += sym_split(form > 0, form == 2, n, comps, packed, 0.5 * slot, 0.0) != 1;
            }
    std::printf("%lld %lld\n", bad, finer);
    return 0;
}
"""


def test_split_fits_the_scratch_cap(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "plan"
    csrc = os.path.join(ROOT, "rigidmultiblobswall_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", csrc, str(tmp_path / "main.cpp"), "-o", str(exe)], check=True)
    bad, finer = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert bad == 0 and finer > 1000
