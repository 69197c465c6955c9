"""Launch shapes of the tensor-core convolution kernels, computed by the
library's own host code (compiled here with nvcc; no GPU)."""

import shutil
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parent.parent
SM_SHARED = 228 * 1024  # bytes of shared memory an SM gives its CTAs
CTA_RESERVED = 1024     # of which the system keeps this much per CTA
TMEM_COLUMNS = 512

PROBE = r"""
#include <cmath>
#include <cstdio>
#include "efsi_conv3d.cuh"
int main() {
  using namespace efsi::conv;
  const int ch[][2] = {{16, 16}, {16, 32}, {32, 32}, {32, 48}, {48, 48}, {48, 64}, {64, 64}, {112, 48}, {80, 32},
                       {48, 16}, {64, 256}, {176, 16}, {128, 48}};
  const int dim[][3] = {{1, 1, 1}, {5, 6, 7}, {8, 8, 8}, {32, 32, 32}, {16, 18, 32}, {64, 72, 128}, {130, 33, 61}};
  for (auto& c : ch)
    for (auto& d : dim) {
      ConvTile f, b;
      WgradTile w;
      if (conv_tile(d[0], d[1], d[2], c[0], c[1], f)) std::printf("%u %d\n", f.cols, f.smem);
      if (conv_tile(d[0], d[1], d[2], c[1], c[0], b)) std::printf("%u %d\n", b.cols, b.smem);
      if (c[0] * c[1] <= 256 * 28 && wgrad_tile(d[0], d[1], d[2], c[0], c[1], w)) std::printf("%u %d\n", w.cols, w.smem);
    }
}
"""


@pytest.fixture(scope="module")
def launches(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("boxes")
    (d / "probe.cu").write_text(PROBE)
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                    str(REPO / "easyfsi_b200" / "csrc"), str(d / "probe.cu"), "-o", str(d / "probe")], check=True)
    out = subprocess.run([str(d / "probe")], check=True, capture_output=True, text=True).stdout
    return {tuple(map(int, line.split())) for line in out.splitlines()}


def test_resident_ctas_of_any_launches_leave_each_its_tensor_memory(launches):
    """Convolutions and weight gradients run beside each other, so the CTAs that
    fit an SM's shared memory together, of whatever launches, may not ask for
    more than its tensor memory: the least shared memory of any set of CTAs
    with more than 512 columns is more than an SM has."""
    least = {}
    for cols, smem in launches:
        least[cols] = min(least.get(cols, 1 << 30), smem + CTA_RESERVED)
    assert len(least) >= 3
    best = {0: 0}  # columns -> least bytes
    for cols in range(32, 2 * TMEM_COLUMNS + 1, 32):
        best[cols] = min((best[cols - c] + b for c, b in least.items() if cols - c in best), default=1 << 30)
    assert min(b for c, b in best.items() if c > TMEM_COLUMNS) > SM_SHARED


def test_every_launch_fits_an_sm(launches):
    for cols, smem in launches:
        assert 32 <= cols <= TMEM_COLUMNS and cols & (cols - 1) == 0
        assert smem <= 222 * 1024
