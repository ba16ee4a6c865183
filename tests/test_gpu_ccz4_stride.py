"""grhd_ccz4_compute_rhs into a right-hand side whose component stride is not
the interior volume (the kernels write with that stride, the entry point then
copies): the same values bit for bit as with it, and nothing written between
the components."""
import ctypes as C

import pytest

import oracle_lib as O
from test_gpu_ccz4 import _case, _gpu_level, _gpu_op, _inv

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gap", [1, 1000])
def test_rhs_stride(gap):
    p, box, s = _case("ksdisk")
    s36 = O.ccz4_state(p, box, s)
    op = _gpu_op(p)
    lv = _gpu_level(box, s36)
    want = lv.new_rhs()
    op.compute_rhs(want, lv, inverse_dx_U=_inv(p))
    n = want[0].numel()
    out = torch.full((5, n + gap), 7.0, dtype=torch.float64, device="cuda")
    lv = _gpu_level(box, s36)
    cb = lv.c_box()
    op._check(op._lib.grhd_ccz4_compute_rhs(
        op._ctx, C.c_void_p(out.data_ptr()), n + gap,
        C.c_void_p(lv.state.data_ptr()), lv.state[0].numel(), C.byref(cb),
        op._inv(_inv(p)), None))
    assert torch.equal(out[:, :n], want.reshape(5, n))
    assert (out[:, n:] == 7.0).all()
