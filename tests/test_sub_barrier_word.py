"""The word of the substeps' barrier over very long calls, on the CPU: its bit 63 turns
at the last arrival of every barrier and at no other, whatever escapes are counted."""
import subprocess

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "dem_kernels.cuh"
// every CTA reports an escape at every barrier, all of them of one parity
static int run(unsigned n, int parity, bool counted, unsigned long long flagged) {
    unsigned long long word = 0;
    for (unsigned long long done = 0; done < flagged; done += n) {
        const unsigned long long before = word;
        for (unsigned i = 0; i < n; ++i) {
            word += dem::sub_arrival(i == (unsigned)(done % n), n, parity, true, counted);
            if ((((word ^ before) >> 63) != 0) != (i == n - 1)) return 1;
        }
        if ((word << 1) >> 53) return 2;  // bits 52..62 are back at zero
    }
    return 0;
}
int main() {
    const unsigned ns[] = {2, 95, 296, 1184};
    for (unsigned n : ns)
        for (int parity = 0; parity < 2; ++parity) {
            // up to the host's limit of 3e7 substeps x CTAs, three barriers each, half of each parity
            if (run(n, parity, true, 45000000ull)) return printf("counted, %u CTAs, parity %d\n", n, parity), 1;
            // beyond 2^26 of one parity no count is added
            if (run(n, parity, false, (1ull << 26) + 4 * n)) return printf("not counted, %u CTAs, parity %d\n", n, parity), 1;
        }
    return 0;
}
"""


def test_arrivals_alone_turn_the_barrier_word(tmp_path):
    from mbd_icenav_b200 import build
    src, exe = tmp_path / "word.cu", tmp_path / "word"
    src.write_text(PROGRAM)
    subprocess.run([build.nvcc_path(), "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17",
                    "--expt-relaxed-constexpr", "-I", f"{ROOT}/include", "-I", build.CSRC, "-o", str(exe), str(src)],
                   check=True, capture_output=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout
