"""The resident kernel's division (quotients() in vs_resident.cuh) against the IEEE float division, value for value:
normal numerators, the switches at 2^-80 and 2^100, subnormal numerators and quotients, ties, zeros, infinities and
NaN, and denominators outside the range of the reciprocal form."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "vocalsim-2p5d-fdtd_b200" / "csrc"
SOURCE = """
#include "vs_resident.cuh"
namespace vsb { namespace {
// eight quotients a thread, as a block of four rows of two cells; a partial last warp is none
__global__ void quotients_kernel(const float* a, const float* b, float* out, float top) {
    const size_t at = 8 * ((size_t)blockIdx.x * blockDim.x + threadIdx.x);
    u64 n[4], nb[4], y[4];
    for (int k = 0; k < 4; ++k) {
        const float* p = a + at + 2 * k;
        const float* d = b + at + 2 * k;
        n[k] = pk(p[0], p[1]);
        nb[k] = pk(-d[0], -d[1]);
        y[k] = pk(fdiv(1.0f, d[0]), fdiv(1.0f, d[1]));
    }
    quotients<4>(n, nb, y, top);
    for (int k = 0; k < 4; ++k) {
        out[at + 2 * k] = plo(n[k]);
        out[at + 2 * k + 1] = phi(n[k]);
    }
}
} }
extern "C" int run_quotients(const float* a, const float* b, float* out, int blocks, float top) {
    vsb::quotients_kernel<<<blocks, 128>>>(a, b, out, top);
    return (int)cudaDeviceSynchronize();
}
"""
BLOCK = 8 * 128              # quotients of one block of threads
WARP = 8 * 32


@pytest.fixture(scope="module")
def divide(tmp_path_factory, cuda_ok):
    import torch
    d = tmp_path_factory.mktemp("quotients")
    (d / "q.cu").write_text(SOURCE)
    subprocess.run(["nvcc", "-O3", "-std=c++17", "--fmad=false", "-gencode", "arch=compute_100a,code=sm_100a",
                    f"-I{CSRC}", f"-I{ROOT / 'include'}", "-Xcompiler", "-fPIC", "-shared", str(d / "q.cu"),
                    "-o", str(d / "q.so")], check=True, capture_output=True)
    lib = C.CDLL(str(d / "q.so"))
    lib.run_quotients.argtypes = [C.c_void_p] * 3 + [C.c_int, C.c_float]

    def call(a, b, top=0.0):
        n = len(a) // BLOCK * BLOCK
        assert n > 0
        x, y = (torch.from_numpy(np.ascontiguousarray(v[:n])).cuda() for v in (a, b))
        out = torch.empty_like(x)
        assert lib.run_quotients(x.data_ptr(), y.data_ptr(), out.data_ptr(), n // BLOCK, top) == 0
        with np.errstate(all="ignore"):
            return out.cpu().numpy(), a[:n] / b[:n]
    return call


def floats(rng, n, lo, hi):
    """Random mantissas (one in four near all zeros or ones), signs, and exponents lo .. hi."""
    m = rng.integers(0, 1 << 23, n)
    edge = rng.random(n) < 0.25
    m[edge] = (m[edge] % 4) - 2 & 0x7fffff
    v = (1.0 + m / 2.0 ** 23) * 2.0 ** rng.integers(lo, hi + 1, n)
    return (v * rng.choice([-1.0, 1.0], n)).astype(np.float32)


# numerator exponents, denominator exponents: all of a warp's, so every path is taken by itself
RANGES = {"normal": ((-80, 99), (-26, 45)), "depths": ((-60, 30), (-10, -3)), "tiny": ((-149, -81), (-26, 45)),
          "subnormal_numerator": ((-149, -127), (-22, 20)), "subnormal_quotient": ((-126, -81), (0, 45)),
          "large": ((101, 127), (-22, 20))}


@pytest.mark.parametrize("name", RANGES)
def test_ranges(name, divide):
    rng = np.random.default_rng(len(name))
    (alo, ahi), (blo, bhi) = RANGES[name]
    n = BLOCK * 2000
    a, b = floats(rng, n, alo, ahi), np.abs(floats(rng, n, blo, bhi))
    got, want = divide(a, b)
    np.testing.assert_array_equal(got, want)


def test_warps_that_mix_the_ranges(divide):
    """One lane's tiny, large, infinite or undefined numerator sends its whole warp to the other forms."""
    rng = np.random.default_rng(7)
    n = BLOCK * 1000
    a, b = floats(rng, n, -80, 99), np.abs(floats(rng, n, -22, 20))
    special = np.array([0.0, -0.0, 1e-45, -1e-45, 1e-38, 2.0 ** -80, np.nextafter(np.float32(2.0 ** -80), np.float32(0)),
                        2.0 ** 100, np.nextafter(np.float32(2.0 ** 100), np.float32(np.inf)), 3e38, np.inf, -np.inf, np.nan],
                       np.float32)
    at = np.arange(0, n, WARP) + rng.integers(0, WARP, n // WARP)
    a[at] = rng.choice(special, len(at))
    got, want = divide(a, b)
    np.testing.assert_array_equal(got, want)


def test_ties_of_subnormal_quotients(divide):
    """Numerators (k + 1/2) 2^-149 b exactly: the quotient lies half-way between two subnormals."""
    rng = np.random.default_rng(11)
    n = BLOCK * 500
    k = rng.integers(1, 1 << 10, n)
    b = (rng.integers(1, 1 << 12, n) * 2.0 ** rng.integers(0, 20, n)).astype(np.float32)
    a = ((2 * k + 1) * 2.0 ** -150 * b.astype(np.float64)).astype(np.float32)
    got, want = divide(a, b)
    np.testing.assert_array_equal(got, want)


def test_other_denominators_divide(divide):
    rng = np.random.default_rng(13)
    n = BLOCK * 500
    a, b = floats(rng, n, -126, 127), np.abs(floats(rng, n, -126, 127))
    got, want = divide(a, b, top=np.inf)
    np.testing.assert_array_equal(got, want)


def test_maps_with_other_denominators(cuda_ok):
    """A caller's depths of 2^40 to 2^127 and, where no wave arrives, below 2^-128 (an infinite reciprocal): the
    step kernel's values, subnormal pressures among them."""
    import vocalsim_b200 as V
    from vocalsim_b200 import synthetic as S
    rng = np.random.default_rng(17)
    tubes, res, depths = [S.vowel_tube(2), S.batch_tube(6)[:2]], [], None
    for shape in (len(V.tile_shapes()) - 1, 7):
        b = V.Batch([V.params(cross_sectional_shape=2) for _ in tubes], [V.Geometry(*t) for t in tubes])
        if depths is None:
            depths = [(2.0 ** rng.uniform(40, 127, (d["frame_h"], d["frame_w"]))).astype(np.float32) for d in b.dims]
            for dp in depths:
                dp[1:4, 1:9] = dp[-4:-1, 1:9] = 1e-40
        b.set_tile(shape)
        for i, dp in enumerate(depths):
            b.set_maps(i, depth_p=dp, z_inv=0.0)
        res.append([b.run(80)] + [f for i in range(2) for f in b.fields(i)])
        b.close()
    for f in res[1]:
        assert np.all(np.isfinite(f))
    assert any(0 < np.abs(f[f != 0]).min() < 2.0 ** -126 for f in res[1][1:])
    for x, y in zip(*res):
        np.testing.assert_array_equal(x, y)
