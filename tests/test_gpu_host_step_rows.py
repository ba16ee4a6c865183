"""The copies of grhd_advance_rk4_cfl_host (a chunk's components go as one
pitched copy) with long rows: a 132 x 128 x 20 box, whose chunks of 8 planes
have rows of 1.15 MB and a last one of 6 ghosted planes shorter ones, with an
excised region eight planes and more across, so that all components, the
conserved ones and those around the pressure are copied.  The results equal the device step's bit for bit, and every
primitive that the step does not read is NaN beforehand.  The same state with
a component stride above the largest pitch a pitched copy may have (2^31 - 1
bytes) gives the same."""
import ctypes as C

import numpy as np
import pytest

import cases
import oracle_lib as O
from test_gpu_host_step import _excised_planes

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

N = (132, 128, 20)
LONG = (1 << 28) + 8   # doubles: 64 bytes above 2^31


def _case():
    dx = 0.3
    p = O.default_params(background=O.BG_KERR_SCHILD, ks_mass=1.0,
                         ks_spin=0.0, gamma=4 / 3, dx=dx,
                         center=tuple(0.5 * n * dx for n in N),
                         atmo_rho_floor=1e-12, atmo_pressure_floor=1e-16,
                         atmo_max_velocity_squared=0.8,
                         rec_max_iterations=100, rec_pressure_floor=1e-16,
                         rec_max_velocity_squared=0.8, limiter_theta=2.0,
                         excision_radius=1.6)
    box = O.make_box(N)
    s = O.new_state(box)
    V = O.state_view(box, s)
    rng = np.random.default_rng(20261206)
    V[O.RHO] = 1e-3 * (1.0 + 0.3 * rng.uniform(-1, 1, V[O.RHO].shape))
    V[O.PRESS] = 1e-5 * (1.0 + 0.3 * rng.uniform(-1, 1, V[O.RHO].shape))
    V[O.EPS] = V[O.PRESS] / ((p.gamma - 1.0) * V[O.RHO])
    for d in range(3):
        V[O.V1 + d] = 0.02 * rng.uniform(-1, 1, V[O.RHO].shape)
    O.fill_conserved_from_primitives(p, box, s)
    O.recover_primitives(p, box, s)
    return p, box, s


def _poison(V, keep, precision):
    for c in range(5, 11):
        if precision == "mixed" and c == O.PRESS:
            continue
        poisoned = np.full_like(V[c], np.nan)
        poisoned[keep] = V[c][keep]
        V[c] = poisoned


def _device_step(op, box, s):
    lv = cases.gpu_level(box, s)
    mi = op.compute_max_inverse_dt(lv, time=0.0)
    dt, nxt, d = op.advance_rk4_cfl(lv, 0.25, time=0.0, max_inverse_dt=mi)
    return lv, mi, dt, nxt, lv.state.cpu()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_long_rows(precision):
    p, box, s = _case()
    keep = _excised_planes(p, box)
    assert keep.stop - keep.start >= 8
    op = cases.gpu_operator(p, precision=precision)
    lv, mi, dt, nxt, want = _device_step(op, box, s)
    host = torch.from_numpy(s.copy()).reshape(want.shape).pin_memory()
    _poison(host.numpy(), keep, precision)
    dt_h, nxt_h, _, _, _ = op.advance_rk4_cfl_host(host, lv, 0.25, time=0.0,
                                                   max_inverse_dt=mi)
    assert (dt_h, nxt_h) == (dt, nxt)
    assert torch.equal(host, want), (host - want).abs().max()


def test_stride_above_the_largest_pitch():
    p, box, s = _case()
    op = cases.gpu_operator(p)
    lv, mi, dt, nxt, want = _device_step(op, box, s)
    n = want[0].numel()
    V = s.reshape(want.shape).copy()
    _poison(V, _excised_planes(p, box), "fp64")
    # (the gaps between the components are never touched)
    host = torch.empty(11 * LONG, dtype=torch.float64)
    for c in range(11):
        host[c * LONG:c * LONG + n] = torch.from_numpy(V[c].reshape(-1))
    mi_h, dt_h = C.c_double(mi), C.c_double()
    cb = lv.c_box()
    op._check(op._lib.grhd_advance_rk4_cfl_host(
        op._ctx, C.c_void_p(host.data_ptr()), LONG, C.byref(cb),
        op._inv(None), 0.0, 0.25, 0.0, C.byref(mi_h), C.byref(dt_h), None,
        None, None, None))
    assert (dt_h.value, mi_h.value) == (dt, nxt)
    for c in range(11):
        assert torch.equal(host[c * LONG:c * LONG + n],
                           want[c].reshape(-1)), c
