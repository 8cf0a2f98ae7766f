"""The EMT kernels' shared-memory layout holds what a batch of mixed sizes runs in it: for every
trajectory no larger than the batch's largest, the beads evaluated together fit the staged places
and, more than one, their energies' array; no array reaches into the next.  Compiled for the host."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "md_tian2_gb300" / "csrc"

SOURCE = r"""
#include <algorithm>
#include <cstdio>
#include "mdt_emt.cuh"
using namespace mdt;
static long bad = 0, seen = 0;
template <typename R> static void layout(const EmtLayout &L, bool kernel) {
    unsigned char *const base = reinterpret_cast<unsigned char *>(uintptr_t(4096));
    const SmemEmt<R> s = carve_smem<R>(base, L);
    auto at = [&](const void *p) { return (const unsigned char *)p - base; };
    if (s.bytes != smem_bytes<R>(L)) ++bad;
    const size_t p = L.places;
    // the accumulators of all places, then the energies (if any), the cell and its groups, the places' atoms
    const R *const acc[5] = {s.sig, s.A, s.fx, s.fy, s.fz};
    for (int k = 0; k < 4; ++k)
        if (at(acc[k] + p) > at(acc[k + 1])) ++bad;
    if (at(s.fz + p) > at(s.en ? (void *)s.en : (void *)s.cell)) ++bad;
    if (at(s.seg + 6) > at(s.perm) || at(s.perm + L.max_atoms) > (long)s.bytes) ++bad;
    if (sizeof(R) == 8 && at(s.pz + p) > at(s.red)) ++bad;
    if (sizeof(R) == 4 && at(s.pl + p) > at(s.red)) ++bad;
    if (!kernel) return;
    for (int N : {1, 2, 3, 5, 36, 37, 65, 101, 128, 145, 162, 163, 256, 257, 288, 289, 325, 511, 512, 513, L.max_atoms / 2,
                  (L.max_atoms + 1) / 2, L.max_atoms - 1, L.max_atoms}) {
        if (N < 1 || N > L.max_atoms) continue;
        for (int nb = 1; nb <= L.max_beads; ++nb)
            for (int team = 1; team <= 8; team *= 2) {
                const int per = (nb + team - 1) / team, G = emt_group(s.places, s.en != nullptr, N, per);
                ++seen;
                if (G < 1 || G > per || (size_t)G * N > p) ++bad;
                if (G > 1 && (!s.en || at(s.en + (size_t)G * N) > at(s.cell))) ++bad;
            }
    }
}
int main() {
    for (int n : {1, 2, 7, 16, 37, 85, 127, 128, 145, 170, 171, 255, 256, 257, 300, 325, 341, 511, 512, 513, 577, 1000, 3000, 4096})
        for (int nb = 1; nb <= 32; ++nb) {
            layout<double>(emt_layout(n, nb), true);
            layout<float>(emt_layout(n, nb), true);
            layout<double>(emt_layout_one(n, nb), false);
        }
    std::printf("%ld %ld\n", bad, seen);
    return 0;
}
"""


def test_emt_layout(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    (tmp_path / "layout.cu").write_text(SOURCE)
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O1", "-std=c++17", "-I", str(CSRC),
                    str(tmp_path / "layout.cu"), "-o", str(tmp_path / "layout")], check=True, capture_output=True)
    bad, seen = map(int, subprocess.run([str(tmp_path / "layout")], check=True, capture_output=True,
                                        text=True).stdout.split())
    assert seen > 1000 and bad == 0


# what the network kernels laid out beside their own buffers before the image table
SIZES = r"""
#include <cstdio>
#include "mdt_emt.cuh"
using namespace mdt;
int main() {
    auto r16 = [](size_t b) { return (b + 15) & ~size_t(15); };
    long larger = 0;
    for (int n = 1; n <= 4096; ++n)
        for (int nb : {1, 2, 8, 32}) {
            const size_t was = 8 * r16(8 * n) + 2 * r16(8 * 64) + r16(8 * rp_cells(nb)) + 256 + 2 * r16(n);
            larger += smem_bytes<double>(emt_layout_one(n, nb)) > was;
        }
    std::printf("%ld\n", larger);
    return 0;
}
"""


def test_fallback_layout_no_larger(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    (tmp_path / "sizes.cu").write_text(SIZES)
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O1", "-std=c++17", "-I", str(CSRC),
                    str(tmp_path / "sizes.cu"), "-o", str(tmp_path / "sizes")], check=True, capture_output=True)
    assert int(subprocess.run([str(tmp_path / "sizes")], check=True, capture_output=True, text=True).stdout) == 0
