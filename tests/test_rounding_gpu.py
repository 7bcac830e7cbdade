"""The straight-line reciprocal, square root and quotient of the projections
(csrc/project_dev.cuh) against the IEEE operators, and frames whose constraints leave their
operand range against the CPU oracle.  Everything is bit for bit: no tolerance."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from tests.helpers import bits, make_pair
from xrtailor_gb300 import build as xb
from xrtailor_gb300 import scenes

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "project_dev.cuh"
using namespace xrt;
// bad[0] recip, bad[1] sqrt_rn: every significand in the binades 2^e and 2^(e + 1)
__global__ void k_unary(int e, unsigned long long* bad) {
  const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;  // 2^24 threads
  const float x = __uint_as_float(((uint32_t)(127 + e) << 23) + m);
  if (!in_range(x)) return;
  if (__float_as_uint(recip(x)) != __float_as_uint(1.0f / x)) atomicAdd(bad, 1ull);
  if (__float_as_uint(sqrt_rn(x)) != __float_as_uint(sqrtf(x))) atomicAdd(bad + 1, 1ull);
}
// bad[2] div_rn: mixed pairs; significands drawn at random, next to 1 or next to 2, exponents over
// the whole range, either sign of the numerator
__global__ void k_quotient(unsigned long long* bad) {
  uint64_t s = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) * 0x9E3779B97F4A7C15ull + 1;
  for (int i = 0; i < 1000; ++i) {
    float v[2];
    for (int k = 0; k < 2; ++k) {
      s = s * 6364136223846793005ull + 1442695040888963407ull;
      const uint32_t r = (uint32_t)(s >> 33), kind = r & 3u;
      uint32_t m = (uint32_t)(s >> 20) & 0x7FFFFFu;
      if (kind == 1) m &= 31u;
      if (kind == 2) m |= 0x7FFFE0u;
      const uint32_t e = 67 + (r >> 2) % 120;  // 2^-60 .. 2^59
      v[k] = __uint_as_float((e << 23) | m);
    }
    const float a = (s >> 40) & 1u ? -v[0] : v[0];
    if (__float_as_uint(div_rn(a, v[1])) != __float_as_uint(a / v[1])) atomicAdd(bad + 2, 1ull);
  }
}
extern "C" int rounding_mismatches(unsigned long long* out) {
  unsigned long long* d;
  if (cudaMalloc(&d, 24) != cudaSuccess) return 1;
  cudaMemset(d, 0, 24);
  const int exps[] = {-60, -31, -1, 0, 30, 58};
  for (int e : exps) k_unary<<<1 << 16, 256>>>(e, d);
  k_quotient<<<1 << 12, 256>>>(d);
  const cudaError_t e = cudaMemcpy(out, d, 24, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e != cudaSuccess;
}
"""


def test_straight_line_operations_round_as_the_operators(xrt, tmp_path):
    src, lib = tmp_path / "rounding.cu", tmp_path / "rounding.so"
    src.write_text(SOURCE)
    subprocess.run([xb._nvcc()] + xb.COMMON + xb.ARCH + ["-I", xb.CSRC, "-shared", str(src), "-o",
                                                         str(lib)], check=True)
    out = (C.c_ulonglong * 3)()
    assert C.CDLL(str(lib)).rounding_mismatches(out) == 0
    assert list(out) == [0, 0, 0]


def _mesh(shape):
    nx, ny = 23, 14
    m = scenes.rect_cloth(nx, ny, 1.0, 0.6, jitter=1e-3, seed=5)
    x = m.positions.astype(np.float64)
    if shape == "tiny":        # squared areas below the range
        x *= 1e-9
    elif shape == "huge":      # squared areas above it
        x *= 1e8
    elif shape == "welded":    # edges of length 0, triangles of area 0
        x[1::5] = x[0::5][:len(x[1::5])]
    elif shape == "folded":    # every other column back on the first: angles of 0
        j = np.arange(len(x)) % nx
        x[:, 0] = (j % 2) * 0.05
        x[:, 1] = 0.0
        x[:, 2] = (np.arange(len(x)) // nx) * 0.05
    m.positions = x.astype(np.float32)
    return m


def _same(a, b):
    """Bit for bit; a NaN equals a NaN (processors encode them differently)."""
    nan = np.isnan(a)
    np.testing.assert_array_equal(nan, np.isnan(b))
    np.testing.assert_array_equal(bits(a)[~nan], bits(b)[~nan])


@pytest.mark.parametrize("compliance", [0.0, 1e-6])
@pytest.mark.parametrize("tile", [32, 256])
@pytest.mark.parametrize("shape", ["plain", "tiny", "huge", "welded", "folded"])
def test_frames_with_operands_out_of_range(xrt, shape, tile, compliance):
    p = scenes._params(num_substeps=2, num_iterations=4, stretch_compliance=compliance,
                       bend_compliance=compliance, num_collision_passes=1,
                       enable_self_collision=0)
    m = _mesh(shape)
    m.fixed_indices = np.array([0, 22], np.uint32)
    g, o = make_pair(p, [m], tile_vertices=tile)
    for _ in range(2):
        g.step()
        o.step()
        _same(g.host_positions(), o.host_positions())
        _same(g.host_velocities(), o.host_velocities())
