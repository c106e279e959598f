"""The lane grids' shared memory (CPU): a host program over the kernels' own
header prints what a warp reserves and what each size lays out. A plan's small
pass reserves by its largest n and lays out by each matrix's n, so the
reservation has to cover every size up to it."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r"""
#include <cstdio>
#include "mixed_grid.cuh"
using namespace lufqhe::mixed;
template <int NP>
size_t end_of() {  // matrices, then F, then 2 NP ints of each, as the kernels place them
  using Gd = SmallGrid<NP>;
  return Gd::G * Gd::kHL * sizeof(float4) + Gd::G * Gd::kF * sizeof(float2) +
         Gd::G * 2 * NP * sizeof(int);
}
int main() {
  for (int n = 1; n <= kSmallMaxN; ++n) {
    const int np = small_np(n);
    printf("%d %d %zu %zu\n", n, np, np == 8 ? end_of<8>() : np == 12 ? end_of<12>() : end_of<16>(),
           small_warp_bytes(n));
  }
}
"""


def test_small_pass_reservation_covers_every_size(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    src, exe = tmp_path / "layout.cu", tmp_path / "layout"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-gencode",
                    "arch=compute_103a,code=sm_103a", "-I", str(ROOT / "include"), "-I",
                    str(ROOT / "lion-codes_gb300" / "csrc"), str(src), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    rows = [tuple(map(int, line.split())) for line in
            subprocess.run([str(exe)], check=True, capture_output=True, text=True)
            .stdout.splitlines()]
    assert [r[0] for r in rows] == list(range(1, 17))
    for nm, _, _, reserved in rows:
        for n, np_, end, _ in rows[:nm]:
            assert np_ >= n
            assert end <= reserved, f"n={n} ends at {end} of {reserved} bytes for nm={nm}"
