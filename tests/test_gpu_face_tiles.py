"""The face pass at the edges of its tiles against the oracle: boxes one cell
below, at and above multiples of the 16-cell tile, thin ones and single
cells, on a rough seeded flow whose faces are subsonic, supersonic either
way and above the velocity cap.  Tolerance: 1e-12 of max|RHS| per component,
the reference's own for one right-hand side (GRHDFixedBGTest.cpp:419-421)."""
import numpy as np
import pytest

import cases
import oracle_lib as O

pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def rough_flow(background, n):
    dx = 0.4
    kw = (dict(background=O.BG_KERR_SCHILD, ks_mass=1.0, ks_spin=0.7,
               use_metric_volume_time_sources=0)
          if background == "ks" else
          dict(background=O.BG_BINARY_PN, pn_mass_1=0.6, pn_mass_2=0.4,
               pn_separation=8.0, pn_softening_radius=1.0,
               use_metric_volume_time_sources=0))
    p = O.default_params(gamma=5 / 3, dx=dx, center=(-5.0, 3.0, 2.0),
                         atmo_rho_floor=1e-3, atmo_pressure_floor=1e-4,
                         atmo_max_velocity_squared=0.8,
                         rec_max_iterations=80,
                         rec_max_velocity_squared=0.97, limiter_theta=1.5,
                         **kw)
    box = O.make_box(n)
    s = O.new_state(box)
    V = O.state_view(box, s)
    rng = np.random.default_rng(int(np.prod(n)) + len(background))
    V[O.RHO] = 10.0 ** rng.uniform(-3.0, 0.0, V[O.RHO].shape)
    V[O.PRESS] = V[O.RHO] * 10.0 ** rng.uniform(-2.0, 0.0, V[O.RHO].shape)
    V[O.EPS] = V[O.PRESS] / ((p.gamma - 1.0) * V[O.RHO])
    u = rng.normal(size=(3,) + V[O.RHO].shape)
    u *= rng.uniform(0.0, 0.75, V[O.RHO].shape) / np.linalg.norm(u, axis=0)
    V[O.V1], V[O.V2], V[O.V3] = u
    O.fill_conserved_from_primitives(p, box, s)
    return p, box, s


@pytest.mark.parametrize("background", ["ks", "pn"])
@pytest.mark.parametrize("n", [(1, 1, 1), (15, 16, 17), (16, 32, 16),
                               (17, 33, 1), (31, 2, 50), (48, 47, 3)])
def test_rhs_matches_oracle(background, n):
    p, box, s = rough_flow(background, n)
    op = cases.gpu_operator(p)
    lv = cases.gpu_level(box, s)
    rhs = lv.new_rhs()
    op.compute_rhs(rhs, lv, time=0.3)
    ref = O.compute_rhs(p, box, s.copy(), 0.3).reshape(5, -1)
    err = cases.rel_err(rhs.cpu().numpy().reshape(5, -1), ref)
    assert np.all(err <= 1e-12), f"per-component rel err {err}"
