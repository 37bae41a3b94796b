"""The FP32 kernels have an instance that waits for its predecessor and one that
does not, chosen by the number of blocks: block sizes on both sides of the line
give the same tendencies and step."""
import numpy as np
import pytest

from imodel_gb300 import swm
from imodel_gb300.swm import SWM

pytestmark = pytest.mark.gpu

# blocks of triangles, edges, cells (thousands) with 128, 256 and 512 threads:
# level 7 2.6 3.8 1.3, 1.3 1.9 0.6, 0.6 1.0 0.3; level 8 10 15 5, 5 7.7 2.6;
# level 9 31 and 10 (edges, cells) with 256, 15 and 5 with 512.  The lines are
# at 8,192 blocks and, for variant 0's edges, at 1,024.
CASES = [(7, 512, 256), (8, 128, 256), (9, 256, 512)]


@pytest.mark.parametrize("scheme,variant,apvm", [
    ("trsk10", 0, False), ("pxt16", 0, False), ("gass18", 0, True), ("dtred", 0, False),
    ("dtred", 1, False), ("gass18", 1, False), ("trsk10", 2, True)])
@pytest.mark.parametrize("level,a,b", CASES)
def test_both_sides_of_the_line(grid_at, level, a, b, scheme, variant, apvm):
    g = grid_at(level)
    rng = np.random.default_rng(level)
    h, u = swm.initialize_fields_tc2(g)
    h = h + rng.normal(0, 5.0, g.nv)
    u = u + rng.normal(0, 0.5, g.ne)
    dt = 110.0 * 2.0 ** (8 - level)
    out = []
    for bs in (a, b):
        m = SWM(g, "fp32", h_ref=2900.0, scheme=scheme)
        m.set_tuning(variant=variant, bs_tri=bs, bs_pre=bs, bs_cell=bs, bs_edge=bs)
        if apvm:
            m.set_apvm(0.5, dt)
        out.append(m.tendency(h, u) + m.ode_rk4(h, u, dt, 1))
        m.close()
    # The instances may fuse products differently, a rounding of each term: of
    # the potential across an edge and of the six to ten fluxes of a sum.  A
    # stage that read what the one before it had left would be off by a
    # noticeable part of the tendency.
    ulp = 2.0 ** -23
    um, hm = np.abs(u).max(), h.max()
    d = g.edhx_leng.min() * swm.ERAD
    bern = swm.GRAV * np.abs(h - 2900.0).max() + um * um
    tol_h = 16 * ulp * 6 * um * hm / d
    tol_u = 8 * ulp * (bern / d + 10 * um * 2 * swm.OMEGA)
    # a step amplifies the stages' differences by less than the CFL number's
    # few units
    for x, y, tol in zip(out[0], out[1], (tol_h, tol_u, 16 * dt * tol_h, 16 * dt * tol_u)):
        assert np.all(np.isfinite(x)) and np.max(np.abs(x - y)) <= tol
    assert np.max(np.abs(out[0][1])) > 300 * tol_u
