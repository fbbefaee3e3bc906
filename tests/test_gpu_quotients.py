"""The branch-free quotients and roots of the FP64 form (csrc/ns3d_device.cuh)
against the device's own division and square root, bit for bit: over their
range, at its edges, outside it, at zeros of both signs, infinities and NaN."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT, ref_cfg, scheme_id
from test_gpu_parity import params_from_cfg
from test_gpu_routes import _solver

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "ns3d_device.cuh"
using namespace ns3d;
// which: 0 quot_mid, 1 quot_wide by a constant, 2 div_wide by a variable, 3 sqrt_mid; out[0] the form's value, out[n] IEEE
__global__ void k(int which, long long n, const double* a, const double* b, double* out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double x = a[i], d = b[i];
    double v;
    if (which == 0) v = quot_mid(x, d);
    else if (which == 1) { const double y = 1.0 / d; v = quot_wide(x, d * 0x1p54, y, y * 0x1p-54); }
    else if (which == 2) { const double y = rcp_cubic(d); v = div_wide(x, d * 0x1p54, y, y * 0x1p-54); }
    else v = sqrt_mid(x);
    out[i] = v;
    out[n + i] = which == 3 ? sqrt(x) : x / d;
}
extern "C" int run(int which, long long n, const double* a, const double* b, double* out) {
    k<<<(unsigned)((n + 255) / 256), 256>>>(which, n, a, b, out);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("quotients")
    (d / "q.cu").write_text(SOURCE)
    so = str(d / "q.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--fmad=false",
                    "-Xcompiler", "-fPIC", "-shared", "-I", os.path.join(ROOT, "ns3d_cpp_b200", "csrc"),
                    str(d / "q.cu"), "-o", so], check=True, capture_output=True, text=True)
    lib = ctypes.CDLL(so)
    lib.run.argtypes = [ctypes.c_int, ctypes.c_longlong] + [ctypes.c_void_p] * 3
    return lib


def _both(lib, which, a, b):
    import torch
    a, b = np.broadcast_arrays(np.asarray(a, float), np.asarray(b, float))
    ta, tb = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (a, b))
    out = torch.empty((2, a.size), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert lib.run(which, a.size, ta.data_ptr(), tb.data_ptr(), out.data_ptr()) == 0
    got, want = out.cpu().numpy()
    return got, want


def _same(got, want):
    nan = np.isnan(want)
    return np.array_equal(np.isnan(got), nan) and np.array_equal(got[~nan].view(np.uint64), want[~nan].view(np.uint64))


def _random(lo, hi, n, seed, signed=False):
    """Values with exponents uniform in [lo, hi), some mantissas all zeros or all ones."""
    r = np.random.default_rng(seed)
    m = 1.0 + r.random(n)
    m[r.random(n) < 0.05] = 1.0
    m[r.random(n) < 0.05] = 2.0 - 2.0 ** -52
    x = np.ldexp(m, r.integers(lo, hi, n))
    return np.where(r.random(n) < 0.5, x, -x) if signed else x


SPECIAL = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.0 ** -1022, 1e-310, 1e-300, 2.0 ** -481,
                    2.0 ** -480, 2.0 ** 480, 2.0 ** 479, -1.0, 1.0, 3.0, 1e300, 1.7e308])


def test_quot_mid(lib):
    n = 1 << 20
    assert _same(*_both(lib, 0, _random(-480, 480, n, 1), _random(-480, 480, n, 2)))
    assert _same(*_both(lib, 0, _random(-1074, 1023, n, 3, True), _random(-1074, 1023, n, 4, True)))
    a, b = np.meshgrid(SPECIAL, SPECIAL)
    assert _same(*_both(lib, 0, a.ravel(), b.ravel()))


def test_sqrt_mid(lib):
    n = 1 << 20
    assert _same(*_both(lib, 3, _random(-480, 480, n, 5), 1.0))
    assert _same(*_both(lib, 3, np.concatenate([SPECIAL, _random(-1074, 1023, n, 6)]), 1.0))


@pytest.mark.parametrize("b", [2 * np.pi / 256, 12 * 2 * np.pi / 100, 60 * 2 * np.pi / 33, 0.72, 6.0, 1e-3])
def test_quot_wide_by_a_constant(lib, b):
    """The IEEE quotient where that is normal; a subnormal one to its last place
    (its residual is exact, so only a tie can go the other way), a dividend above
    2^969 to an ulp."""
    a = np.concatenate([_random(-1074, 969, 1 << 19, 7, True), np.arange(-2000, 2000) * 5e-324])
    got, want = _both(lib, 1, a, b)
    normal = (np.abs(want) >= 2.0 ** -1022) | (a == 0.0)
    assert _same(got[normal], want[normal])
    assert np.all(np.abs(got - want)[~normal] <= 5e-324)
    assert _same(*_both(lib, 1, np.array([0.0, -0.0, np.inf, -np.inf, np.nan]), b))
    got, want = _both(lib, 1, _random(969, 1010, 1 << 19, 8, True), b)
    assert np.all(np.abs(got - want) <= np.abs(np.spacing(want)))


def test_div_wide(lib):
    """The velocities of a stage: momenta of any size by a density that is a
    divisor_ok(); zeros keep their sign."""
    n = 1 << 20
    a, b = _random(-900, 900, n, 9, True), _random(-40, 40, n, 10)
    b[(b.view(np.uint64) & np.uint64(0xffffffff)) == np.uint64(0xffffffff)] = 1.25
    a[:64:2], a[1:64:2] = 0.0, -0.0
    assert _same(*_both(lib, 2, a, b))


def test_density_one_rounding_below_one(oracle_mod):
    """Powers of two over 1 - 2^-53, whose quotients lie 2^-106 from a midpoint:
    c^2 = gamma p / rho with gamma p = 2, momenta of 2^-k, Roe averages over
    sqrt(rho) + sqrt(rho)."""
    n = 16
    for kw in (dict(recon="LINEAR", fvs_type="LaxFriedrichs"), dict(recon="LINEAR", char_recon="true"), dict()):
        cfg = ref_cfg(n, **kw)
        cfg["gamma"] = 1.5
        r = np.random.default_rng(2)
        W = np.empty((5, n, n, n))
        W[0] = np.where(r.random((n, n, n)) < 0.5, 1.0 - 2.0 ** -53, 1.0)
        W[1:4] = np.ldexp(1.0, -r.integers(1, 4, (3, n, n, n)))
        W[4] = 4.0 / 3.0
        W[4, ::2] = 8.0
        want = oracle_mod.Oracle(cfg).rhs(W)
        for small in ("0", "10000000"):
            with _solver(params_from_cfg(cfg), {"NS3D_SMALL": small}) as s:
                s.upload_primitive(W)
                got = s.compute_rhs()
            # mass: no viscous term (whose T^1.5 may differ by an ulp)
            assert np.array_equal(got[0], want[0]), (kw, small)


@pytest.mark.parametrize("small", ["0", "10000000"], ids=["marching", "small"])
@pytest.mark.parametrize("scale", [1e-300, 1e-280, 1.0])
def test_velocities_of_any_size_match_oracle(oracle_mod, scale, small):
    """A step of a box whose velocities are tiny (the far tail of a disturbance):
    the linear scheme's state equals the oracle's bit for bit, zeros and signs too."""
    n = 16
    cfg = ref_cfg(n, fvs_type="LaxFriedrichs", recon="LINEAR")
    W = np.empty((5, n, n, n))
    W[0], W[4], W[3], W[2] = 1.3, 8.0 * 1.3, 0.0, -0.0
    W[1] = scale * np.random.default_rng(1).standard_normal((n, n, n))
    want, dt, st = oracle_mod.Oracle(cfg).cfl_step(W)
    assert st == 0
    with _solver(params_from_cfg(cfg), {"NS3D_SMALL": small}) as s:
        s.upload_primitive(W)
        s.step(1)
        got = s.download_primitive()
    for q in range(5):
        assert np.array_equal(got[q].view(np.uint64), np.ascontiguousarray(want[q]).view(np.uint64)), q


@pytest.mark.parametrize("small", ["0", "10000000"], ids=["marching", "small"])
@pytest.mark.parametrize("kw", [dict(), dict(fvs_type="LaxFriedrichs"), dict(char_recon="true")], ids=scheme_id)
def test_windows_that_vary_hugely_match_oracle(oracle_mod, kw, small):
    """WENO5 windows that vary by 2^240 and more, whose weights' terms are too small
    for the branch-free quotients: the mass equation (no T^1.5) has the oracle's bits."""
    n = 16
    cfg = ref_cfg(n, **kw)
    r = np.random.default_rng(3)
    W = np.empty((5, n, n, n))
    W[0] = 1.0 + 0.1 * r.random((n, n, n))
    W[1:4] = r.standard_normal((3, n, n, n))
    W[4] = 10.0 ** r.uniform(140, 156, (n, n, n))  # split mass fluxes of rho c
    want = oracle_mod.Oracle(cfg).rhs(W)
    with _solver(params_from_cfg(cfg), {"NS3D_SMALL": small}) as s:
        s.upload_primitive(W)
        got = s.compute_rhs()
    assert np.array_equal(got[0], want[0], equal_nan=True)
