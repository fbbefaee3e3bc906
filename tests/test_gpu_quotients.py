"""The branch-free quotients and roots of the FP64 form (csrc/ns3d_device.cuh):
the IEEE values."""
import numpy as np
import pytest

from conftest import ref_cfg
from test_gpu_parity import params_from_cfg
from test_gpu_routes import _solver

pytestmark = pytest.mark.gpu


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
