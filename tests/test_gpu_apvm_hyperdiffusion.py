"""APVM with hyperdiffusion in FP32 (its first application formed by APVM's
kernels, the divergence and vorticity of it by the cell kernel) against the
FP64 handle, alone and with the Laplacian term, in both cell-centred variants.
Four steps are sixteen evaluations of a few hundred FP32 roundings (6e-8 each),
so 1e-5 of each field's norm bounds them."""
import numpy as np
import pytest

from imodel_gb300 import swm
from imodel_gb300.swm import SWM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k2", [0.0, 1.0e5])
@pytest.mark.parametrize("level", [1, 4, 6])
def test_fp32_follows_fp64(grid_at, level, k2):
    g = grid_at(level)
    rng = np.random.default_rng(level)
    h, u = swm.initialize_fields_tc2(g)
    h = h + rng.normal(0, 5.0, g.nv)
    u = u + rng.normal(0, 0.5, g.ne)
    dt = 400.0 * 2.0 ** min(0, 5 - level)
    out = {}
    for name, prec, variant in (("fp64", "fp64", 0), ("v1", "fp32", 1), ("v2", "fp32", 2)):
        m = SWM(g, prec)
        if prec == "fp32":
            m.set_tuning(variant=variant)
        m.set_diffusion(k2=k2, k4=5.12e14 if level < 6 else 6.4e13)
        m.set_apvm(0.5, dt)
        if prec == "fp32":
            assert m.launch_count(1) == 20
        out[name] = m.ode_rk4(h, u, dt, 4)
        # and off again: hyperdiffusion alone
        m.set_apvm(0.0, dt)
        out[name] += m.ode_rk4(h, u, dt, 4)
        m.close()
    for a, b, c in zip(out["fp64"], out["v1"], out["v2"]):
        assert np.linalg.norm(b - a) <= 1e-5 * np.linalg.norm(a)
        assert np.linalg.norm(c - a) <= 1e-5 * np.linalg.norm(a)
