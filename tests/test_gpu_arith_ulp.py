"""The one-step FP64 reciprocal and reciprocal square root of the face fluxes,
the root solve and the Kerr-Schild cell (rcp_ulp, rsqrt_ulp in
grhd_device.cuh) through grhd_eval_arith_ulp, against extended precision.

Bounds: the hardware's approximate values are good to 2^-20, so the
third-order step leaves 2^-60, a 128th of an ulp, beside roundings: half an
ulp for the reciprocal's last operation; for the square root's that half and
as much again from the rounding of a y (2^-53 of it, halved)."""
import numpy as np
import pytest

import cases

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if np.finfo(np.longdouble).nmant < 63:
    pytest.skip("no extended precision", allow_module_level=True)


@pytest.fixture(scope="module")
def op():
    p, _, _, _ = cases.CASES["fixedbg"]()
    return cases.gpu_operator(p)


def _ulps(got, exact):
    want = exact.astype(np.float64)
    return np.abs((got.astype(np.longdouble) - exact)
                  / np.spacing(np.abs(want)).astype(np.longdouble))


@pytest.mark.parametrize("lo,hi", [(-12.0, 3.0), (-0.5, 0.5), (-150.0, 150.0),
                                   (-300.0, 300.0)])
def test_reciprocals(op, lo, hi):
    rng = np.random.default_rng(20261206)
    n = 1 << 22
    a = 10.0 ** rng.uniform(lo, hi, n)
    # both ends of a binade
    a[:1000] = 1.0 + np.arange(1000) * 2.0 ** -52
    a[1000:2000] = 2.0 - np.arange(1, 1001) * 2.0 ** -52
    da = torch.from_numpy(a).cuda()
    out = torch.empty(2 * n, dtype=torch.float64, device="cuda")
    assert op._lib.grhd_eval_arith_ulp(op._ctx, n, da.data_ptr(),
                                       out.data_ptr(), None) == 0
    out = out.cpu().numpy().reshape(-1, 2)
    x = a.astype(np.longdouble)
    r = _ulps(out[:, 0], 1 / x).max()
    s = _ulps(out[:, 1], 1 / np.sqrt(x)).max()
    print("max ulp (1/a, 1/sqrt a):", float(r), float(s))
    assert r <= 0.51 and s <= 1.02
