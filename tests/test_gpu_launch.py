"""Launch routes that must not change a bit: launches overlapped by programmatic
dependent launch (NS3D_PDL=0 serialises them), and the FP32 form's staged x
sweep k_sweep_x_rows (NS3D_XROWS=1 always, 0 never). Both are read when a
context is created."""
import numpy as np
import pytest

from conftest import scheme_id
from test_gpu_routes import _box_params, _field, _solver

pytestmark = pytest.mark.gpu


# boxes of every rule under which launches overlap: FP64 through k_flux_small
# (component- and characteristic-wise) and through the marching kernels, FP32
# below and above 30000 cells, eight-point schemes on warp rows
@pytest.mark.parametrize("precision,box,kw,env", [
    ("fp64", (16, 12, 10), dict(sw_entropy_eps=1e-3), {}),
    ("fp64", (64, 24, 31), dict(fvs_type="LaxFriedrichs", recon="MDCD"), {}),
    ("fp64", (33, 17, 9), dict(char_recon="true"), {}),
    ("fp64", (20, 18, 16), dict(), {"NS3D_SMALL": "0"}),
    ("fp64", (64, 48, 32), dict(recon="UD7L", vis_scheme="C4th"), {"NS3D_SMALL": "0"}),
    ("fp64", (410, 8, 9), dict(), {}),
    ("fp32acc64", (8, 8, 8), dict(), {}),
    ("fp32acc64", (24, 20, 16), dict(fvs_type="LaxFriedrichs", recon="MDCD_HYBRID"), {}),
    ("fp32acc64", (70, 40, 30), dict(sw_entropy_eps=1e-3, vis_scheme="C6th"), {}),
    ("fp32acc64", (32, 200, 16), dict(recon="LINEAR"), {}),
    ("fp32acc64", (128, 32, 40), dict(recon="UPWIND_7TH"), {}),
    ("fp32acc64", (100, 75, 70), dict(fvs_type="LaxFriedrichs"), {"NS3D_XROWS": "1"}),
], ids=lambda v: scheme_id(v) if isinstance(v, dict) else ("x".join(map(str, v)) if isinstance(v, tuple) else v))
def test_overlapped_launches_bits(precision, box, kw, env):
    p, W, out = _box_params(box, **kw).replace(precision=precision), _field(box), []
    for pdl in ("0", "1"):
        with _solver(p, {"NS3D_PDL": pdl, **env}) as s:
            s.upload_primitive(W)
            rhs = s.compute_rhs()
            s.step(12)
            a = s.download_primitive()
            s.upload_primitive(W)
            s.step(5)
            out.append((rhs, a, s.download_primitive(), s.last_dt()))
    for q in range(3):
        assert np.array_equal(out[0][q], out[1][q])
    assert out[0][3] == out[1][3]


@pytest.mark.parametrize("box", [(16, 12, 10), (9, 8, 301)], ids=["flux_kernel", "long_lines"])
def test_overlapped_adjoint_bits(box):
    p, W, out = _box_params(box, sw_entropy_eps=1e-3), _field(box), []
    for pdl in ("0", "1"):
        with _solver(p, {"NS3D_PDL": pdl}) as s:
            s.upload_primitive(W)
            g, J, dts = s.adjoint(5, 2)
            out.append((g, J, dts, s.rhs_vjp(W), s.download_primitive()))
    for a, b in zip(*out):
        assert np.array_equal(a, b)


# a single block of rows, a partial last one, several segments, rows shorter
# than the window and a chunk, columns that are no multiple of eight
@pytest.mark.parametrize("recon", ["WENO5", "MDCD", "UD7L", "LINEAR", "MDCD_HYBRID"])
@pytest.mark.parametrize("box", [(33, 17, 9), (9, 130, 41), (500, 17, 18), (70, 75, 80)], ids=lambda b: "x".join(map(str, b)))
def test_fp32_x_rows_bits(box, recon):
    p = _box_params(box, fvs_type="LaxFriedrichs", recon=recon).replace(precision="fp32acc64")
    W, out = _field(box), []
    for rows in ("0", "1"):
        with _solver(p, {"NS3D_XROWS": rows}) as s:
            s.upload_primitive(W)
            rhs = s.compute_rhs()
            s.step(2)
            out.append((rhs, s.download_primitive()))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])


def test_small_box_context_without_room_for_the_separate_terms():
    """A context of a box of k_flux_small takes 15 T_acc values a cell; where
    the device has room for the 5 of the marching kernels only, it is created
    with those and gives the same bits."""
    import torch
    box = (200, 150, 130)
    n = box[0] * box[1] * box[2]
    p, W, out, size = _box_params(box, fvs_type="LaxFriedrichs", recon="MDCD"), _field(box), [], []
    hog = None
    for room in (None, 8 * (18 + 9 + 10) * n):  # state, viscous fluxes, T_acc between the two
        if room is not None:
            torch.cuda.empty_cache()
            hog = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
        with _solver(p, {}) as s:
            s.upload_primitive(W)
            s.step(2)
            out.append(s.download_primitive())
            size.append(s.device_bytes())
    del hog
    torch.cuda.empty_cache()
    assert np.array_equal(*out)
    assert size[0] - size[1] == 8 * 10 * n


@pytest.mark.parametrize("kw,S", [(dict(), 6), (dict(recon="UD7L"), 8)], ids=["WENO5", "UD7L"])
def test_adjoint_scratch_of_long_lines(kw, S):
    """A right-hand side's VJP with a line above 300 cells keeps, per cell, the
    cotangents in and out (5 each), the windows' (2 S 5) and the viscous ones (16)."""
    box = (304, 10, 9)
    p, W = _box_params(box, **kw), _field(box)
    with _solver(p, {}) as s:
        s.upload_primitive(W)
        before = s.device_bytes()
        s.rhs_vjp(W)
        assert s.device_bytes() - before == 8 * (5 + 5 + 10 * S + 16) * 304 * 10 * 9


def test_workload_reports_the_one_launch_fluxes():
    """The library books them under "other"; the workload runner lists them with
    their bandwidth, as it does the sweeps of larger boxes."""
    from ns3d_cpp_b200 import workloads
    w = workloads.WORKLOADS["tgv32"]
    k = workloads.run_one(w, workloads.initial_for(w), "weno5", "fp64", 4, 0)["kernels"]
    assert k["fluxes"]["launches"] == k["update"]["launches"] == 12 and k["fluxes"]["hbm_frac"] > 0
    assert "sweep_x" not in k and "other" not in k


@pytest.mark.parametrize("box", [(9, 11, 13), (15, 15, 15), (9, 11, 14)], ids=lambda b: "x".join(map(str, b)))
def test_spectrum_of_an_odd_number_of_cells(oracle_mod, box):
    """u and w of such a box start on an 8-byte boundary, which cuFFT refuses; the
    spectrum and the state after it are as for any other box."""
    W = _field(box)
    with _solver(_box_params(box), {}) as s:
        s.upload_primitive(W)
        s.step(1)
        res, state = s.residuals(), s.download_primitive()
        E = s.compute_energy_spectrum()
        assert np.array_equal(s.residuals(), res) and np.array_equal(s.download_primitive(), state)
    want = oracle_mod.spectrum(*state[1:4])
    assert E.shape == want.shape and np.all(np.abs(E - want) <= 1e-12 * want.max())
