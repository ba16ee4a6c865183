"""Frozen primitives of excised cells that are not numbers (a user may mark
the region so), in the right-hand side of every other cell, bit for bit.

The box lies deep inside the horizon of a very heavy hole on the +x axis, so
that the excision sphere cuts it in one plane and every wave on the plane's
faces runs towards the hole: the face flux is the fluid side's.  A limited
slope beside a neighbour that is not a number is theta times the other side's
difference, which is also its value beside a finite neighbour a thousand
times as far on the other side; without reconstruction the neighbour is not
looked at.  So the NaN state and that finite state must agree everywhere
outside the excised cells, and two planes further in also with the
unmodified state."""
import numpy as np
import pytest

import cases
import oracle_lib as O

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

NX, NY, NZ, CUT = 20, 17, 9, 8
R = 500.0


def _case(use_recon):
    # cell (CUT - 1, *, *) has its centre within R of the hole, CUT has not
    p = O.default_params(background=O.BG_KERR_SCHILD, ks_mass=1e4,
                         ks_spin=0.0, gamma=5 / 3, dx=1.0,
                         center=(CUT - R, 0.5 * NY, 0.5 * NZ),
                         atmo_rho_floor=1e-10, atmo_pressure_floor=1e-12,
                         atmo_max_velocity_squared=0.8,
                         rec_max_velocity_squared=0.9,
                         use_reconstruction=use_recon, excision_radius=R)
    box = O.make_box((NX, NY, NZ))
    s = O.new_state(box)
    V = O.state_view(box, s)
    rng = np.random.default_rng(20261206)
    shape = V[O.RHO].shape
    V[O.RHO] = 1e-3 * (1.0 + 0.3 * rng.uniform(-1, 1, shape))
    V[O.PRESS] = 1e-5 * (1.0 + 0.3 * rng.uniform(-1, 1, shape))
    V[O.EPS] = V[O.PRESS] / ((p.gamma - 1.0) * V[O.RHO])
    for d in range(3):
        V[O.V1 + d] = 0.05 * rng.uniform(-1, 1, shape)
    O.fill_conserved_from_primitives(p, box, s)
    return p, box, s


def _rhs(p, box, s, precision):
    op = cases.gpu_operator(p, precision=precision)
    lv = cases.gpu_level(box, s.copy())
    rhs = lv.new_rhs()
    op.compute_rhs(rhs, lv, time=0.0)
    return rhs.cpu().numpy()[..., CUT:]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("use_recon", [0, 1])
def test_rhs_beside_excised_nans(precision, use_recon):
    p, box, s = _case(use_recon)
    g = box.lo[0] - box.glo[0]
    nan, far = s.copy(), s.copy()
    Vn, Vf = O.state_view(box, nan), O.state_view(box, far)
    for c in range(O.RHO, 11):
        Vn[c][..., :g + CUT] = np.nan
        a, b = Vf[c][..., g + CUT], Vf[c][..., g + CUT + 1]
        Vf[c][..., g + CUT - 1] = a - 1e3 * (b - a)
    want_clean = _rhs(p, box, s, precision)
    want = _rhs(p, box, far, precision)
    got = _rhs(p, box, nan, precision)
    assert np.isfinite(want_clean).all() and np.abs(want_clean).max() > 0.0
    assert np.array_equal(got, want)
    assert np.array_equal(got[..., 2:], want_clean[..., 2:])
    if not use_recon:
        assert np.array_equal(got, want_clean)
