"""Kernels chosen by size, and the branch-free FP64 arithmetic's fall-backs.

k_flux_small (FP64, small boxes) performs the operations of the marching
sweeps and the viscous kernels in the same order, so states and right-hand
sides agree bit for bit; NS3D_SMALL=0 (read when a context is created) selects
the marching kernels. The branch-free quotients and roots hand extreme values
to the IEEE operations, so infinities and NaN appear where the oracle has them.
"""
import os

import numpy as np
import pytest

import ns3d_cpp_b200 as ns
from ns3d_cpp_b200 import initial
from conftest import ref_cfg, relerr, scheme_id
from test_gpu_parity import params_from_cfg

pytestmark = pytest.mark.gpu


def _solver(params, env):
    old = {k: os.environ.get(k) for k in env}
    os.environ.update(env)
    try:
        return ns.Solver(params)
    finally:
        for k, v in old.items():
            os.environ.pop(k) if v is None else os.environ.__setitem__(k, v)


def _box_params(box, **kw):
    p = params_from_cfg(ref_cfg(16, Ma=0.3, Re=400, **kw))
    p.global_nx, p.global_ny, p.global_nz = box
    return p.derive()


def _field(box, seed=5):
    """A smooth periodic state with noise, all five variables varying along x, y and z."""
    nx, ny, nz = box
    Z, Y, X = np.meshgrid(*[np.arange(m) * (2 * np.pi / m) for m in (nz, ny, nx)], indexing="ij")
    W = np.stack([1 + 0.1 * np.sin(X + 0.3) * np.cos(Y + Z), np.sin(X) * np.cos(Y) * np.cos(Z),
                  -np.cos(X) * np.sin(Y) * np.cos(Z) + 0.1, 0.3 * np.sin(Z + X),
                  7.9 + 0.5 * np.cos(2 * X) * np.cos(Y + Z)])
    return W * (1 + 1e-3 * np.random.default_rng(seed).standard_normal(W.shape))


# one line a block and a partial last group of lines, the shortest and the
# longest lines a block holds, extents on both sides of a warp and a tile
BOXES = [(8, 8, 8), (33, 17, 9), (400, 8, 9), (8, 400, 10), (9, 8, 397), (32, 32, 16), (64, 24, 31)]
KW = [dict(), dict(sw_entropy_eps=1e-3, vis_scheme="C6th"), dict(fvs_type="LaxFriedrichs", recon="MDCD"),
      dict(recon="UD7L", vis_scheme="C4th"), dict(recon="LINEAR"), dict(recon="MDCD_HYBRID")]


CHAR_KW = [dict(char_recon="true"), dict(char_recon="true", fvs_type="LaxFriedrichs", recon="MDCD", vis_scheme="C4th"),
           dict(char_recon="true", recon="UPWIND_7TH"), dict(char_recon="true", recon="MDCD_HYBRID"),
           dict(char_recon="true", recon="LINEAR")]
CHAR_BOXES = [(8, 8, 8), (33, 17, 9), (300, 8, 9), (8, 300, 9), (9, 8, 298), (32, 24, 16)]


@pytest.mark.parametrize("box,kw", [(b, k) for k in KW for b in BOXES] + [(b, k) for k in CHAR_KW for b in CHAR_BOXES],
                         ids=lambda v: scheme_id(v) if isinstance(v, dict) else "x".join(map(str, v)))
def test_small_box_kernel_bits(box, kw):
    p, W = _box_params(box, **kw), _field(box)
    out = []
    for env in ({"NS3D_SMALL": "0"}, {"NS3D_SMALL": "10000000"}):
        with _solver(p, env) as s:
            s.upload_primitive(W)
            rhs = s.compute_rhs()
            s.step(3)
            out.append((rhs, s.download_primitive(), s.last_dt(), s.device_bytes()))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
    assert out[0][2] == out[1][2]
    assert out[1][3] > out[0][3]  # the second context took the kernel (its terms are kept apart)


# k_sweep_x_rows (FP32 form, Lax-Friedrichs, nx no multiple of 32, more than
# 140000 cells): one segment and several, a last block of rows that is not
# full, columns that are no multiple of eight, against the oracle with the FP32
# form's bound on the right-hand side (5e-5 of each variable's largest value)
@pytest.mark.parametrize("kw", [dict(), dict(recon="MDCD"), dict(recon="UD7L"), dict(recon="LINEAR")], ids=scheme_id)
@pytest.mark.parametrize("box", [(70, 51, 41), (9, 130, 121), (500, 17, 18)], ids=lambda b: "x".join(map(str, b)))
def test_fp32_x_rows_matches_oracle(oracle_mod, box, kw):
    cfg = ref_cfg(16, Ma=0.3, Re=400, fvs_type="LaxFriedrichs", **kw)
    cfg.update(global_nx=box[0], global_ny=box[1], global_nz=box[2])
    nx, ny, nz = box
    Z, Y, X = np.meshgrid(*[np.arange(m) * (2 * np.pi / m) for m in (nz, ny, nx)], indexing="ij")
    W = np.stack([1 + 0.1 * np.sin(X + 0.3) * np.cos(Y + Z), np.sin(X) * np.cos(Y) * np.cos(Z),
                  -np.cos(X) * np.sin(Y) * np.cos(Z) + 0.1, 0.3 * np.sin(Z + X),
                  7.9 + 0.5 * np.cos(2 * X) * np.cos(Y + Z)])
    with ns.Solver(params_from_cfg(cfg).replace(precision="fp32acc64")) as s:
        s.upload_primitive(W)
        got = s.compute_rhs()
    assert np.all(relerr(got, oracle_mod.Oracle(cfg).rhs(W)) <= 5e-5)


def test_small_box_stop_leaves_state():
    """Kernels after a device-side stop return at entry on the small-box path too."""
    p = _box_params((16, 12, 10))
    p.dt_fixed, p.TotalTime, p.output_Timefreq = 1e-3, 2.5e-3, 1.0
    W = _field((16, 12, 10))
    out = []
    for env in ({"NS3D_SMALL": "0"}, {"NS3D_SMALL": "10000000"}):
        with _solver(p, env) as s:
            s.upload_primitive(W)
            t, k = s.time_advance(8)
            assert k == 3 and t == pytest.approx(2.5e-3, abs=1e-12)
            out.append(s.download_primitive())
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("n", [(33, 33, 36), (34, 34, 35)], ids=["39204_cells", "40460_cells"])
def test_noalloc_either_side_of_the_separate_terms(n):
    """39321 cells is the most whose separate terms fit the fixed scratch."""
    import ctypes
    import torch
    from ns3d_cpp_b200 import _lib
    p, W = _box_params(n), _field(n)
    with ns.Solver(p) as s:
        s.upload_primitive(W)
        want = s.compute_rhs()
    d = torch.from_numpy(W).cuda()
    rhs = torch.empty_like(d)
    st = _lib.load().ns3d_compute_rhs_noalloc(ctypes.byref(p), *[d[q].data_ptr() for q in range(5)],
                                              rhs.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert st == 0
    torch.cuda.synchronize()
    assert np.array_equal(rhs.cpu().numpy(), want)


def test_noalloc_captured_in_a_graph():
    """The entry point enqueues on the caller's stream only, so it can be
    captured (after a first call); a replay on new inputs gives their result."""
    import ctypes
    import torch
    from ns3d_cpp_b200 import _lib
    box = (20, 18, 16)
    p = _box_params(box)
    d = torch.from_numpy(_field(box)).cuda()
    rhs = torch.empty_like(d)

    def call(out):
        st = _lib.load().ns3d_compute_rhs_noalloc(ctypes.byref(p), *[d[q].data_ptr() for q in range(5)],
                                                  out.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert st == 0

    call(rhs)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call(rhs)
    d.copy_(torch.from_numpy(_field(box, seed=9)))
    g.replay()
    want = torch.empty_like(d)
    torch.cuda.synchronize()
    call(want)
    torch.cuda.synchronize()
    assert torch.equal(rhs, want) and bool(torch.isfinite(rhs).all())


# k_adj_flux (every extent at most 300) and the marching adjoint kernels, with
# a partial last group of lines and the last extent each side of the limit
@pytest.mark.parametrize("kw", [dict(sw_entropy_eps=1e-3), dict(fvs_type="LaxFriedrichs", recon="MDCD"),
                                dict(recon="UD7L", vis_scheme="C6th"), dict(recon="LINEAR", vis_scheme="C4th")],
                         ids=scheme_id)
@pytest.mark.parametrize("box", [(10, 9, 8), (33, 12, 8), (300, 8, 8), (8, 301, 8), (9, 8, 304)],
                         ids=lambda b: "x".join(map(str, b)))
def test_rhs_vjp_routes_dot_product(box, kw):
    """<lam, dR[v]> by 4-point central differences equals <R^T lam, v> (the
    1e-7 of the cubic box's test, of the product's largest possible value)."""
    p = _box_params(box, **kw)
    nx, ny, nz = box
    Z, Y, X = np.meshgrid(*[np.arange(m) * (2 * np.pi / m) for m in (nz, ny, nx)], indexing="ij")
    W = np.stack([1 + 0.1 * np.sin(X + 0.3) * np.cos(Y + Z), 0.5 + 0.2 * np.sin(X) * np.cos(Y) * np.cos(Z),
                  0.4 - 0.2 * np.cos(X) * np.sin(Y) * np.cos(Z), 0.6 + 0.1 * np.sin(Z + X),
                  7.9 + 0.5 * np.cos(2 * X) * np.cos(Y + Z)])
    rng = np.random.default_rng(4)
    lam, v = rng.standard_normal(W.shape), np.stack([0.01 * np.sin(X + 2 * Y), np.cos(Y - Z), np.sin(Z + X),
                                                     np.cos(X + Y + Z), 0.3 * np.sin(2 * Z - X)])
    h, r = 1e-5, {}
    with ns.Solver(p) as s:
        for k in (-2, -1, 1, 2):
            s.upload_primitive(W + k * h * v)
            r[k] = s.compute_rhs()
        s.upload_primitive(W)
        g = s.rhs_vjp(lam)
    fd = float(np.sum(lam * (-r[2] + 8 * r[1] - 8 * r[-1] + r[-2])) / (12 * h))
    ad = float(np.sum(g * v))
    assert abs(fd - ad) <= 1e-7 * np.linalg.norm(g) * np.linalg.norm(v), (fd, ad)


def test_adjoint_leaves_end_state_and_recorded_state():
    """After ns3d_adjoint the context holds the end state and the last step's
    start as U0, whether the last segment is whole, partial or the only one."""
    box, W = (16, 12, 10), _field((16, 12, 10))
    p = _box_params(box, sw_entropy_eps=1e-3)
    with ns.Solver(p) as s:
        s.upload_primitive(W)
        _, _, dts = s.adjoint(4, 2)
        grads = []
        for K in (1, 2, 3, 4, 9):
            s.upload_primitive(W)
            g, J, d = s.adjoint(4, K, dts=dts)
            end, res = s.download_primitive(), s.residuals()
            s.upload_primitive(W)
            s.step_dts(dts)
            assert np.array_equal(end, s.download_primitive())
            assert np.array_equal(res, s.residuals())
            grads.append(g)
    for g in grads[1:]:
        assert np.array_equal(g, grads[0])


EXTREME = [("p", 1e160), ("p", np.inf), ("u", np.nan), ("u", 1e200), ("rho", 1e305),
           ("w", -np.inf), ("p", -1.0), ("p", 0.0)]


@pytest.mark.parametrize("small", ["0", "10000000"], ids=["marching", "small"])
@pytest.mark.parametrize("kw", [dict(), dict(sw_entropy_eps=1e-3), dict(fvs_type="LaxFriedrichs"),
                                dict(char_recon="true")], ids=scheme_id)
@pytest.mark.parametrize("what", EXTREME, ids=lambda w: f"{w[0]}={w[1]:g}")
def test_extreme_cell_matches_oracle(oracle_mod, what, kw, small):
    """One extreme cell: the right-hand side is NaN and infinite where the
    oracle's is, and equal elsewhere to rounding: 1e-12 of the value (the same
    operations but for T^1.5, an ulp) or of the undisturbed field's largest."""
    n = 16
    cfg = ref_cfg(n, **kw)
    W = initial.taylor_green(n, Ma=0.1, perturb=0.05, seed=2)
    o = oracle_mod.Oracle(cfg)
    clean = np.abs(o.rhs(W)).max()
    W["rho u v w p".split().index(what[0]), 5, 9, 3] = what[1]
    ref = o.rhs(W)
    with _solver(params_from_cfg(cfg), {"NS3D_SMALL": small}) as s:
        s.upload_primitive(W)
        got = s.compute_rhs()
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    inf = np.isinf(ref)
    assert np.array_equal(np.isinf(got), inf) and np.array_equal(got[inf], ref[inf])
    ok = np.isfinite(ref)
    assert np.all(np.abs(got[ok] - ref[ok]) <= 1e-12 * np.maximum(np.abs(ref[ok]), clean))
