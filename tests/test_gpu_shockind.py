"""shockind.f on states where about half of the vertices exceed the indicator's
limit, next to each other: a vertex's indicator uses its neighbours' gradients
as they were before any was set to zero, and the result is the same every
time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fvm2d_gb300 import _lib as L  # noqa: E402
from fvm2d_gb300.ogrid import naca_ogrid  # noqa: E402


@pytest.mark.parametrize("ni,nr", [(40, 30), (200, 120), (300, 200)])   # blocks of 64, 128, 256
@pytest.mark.parametrize("prec", [L.FP64, L.FP32])
def test_many_shocks(oracle_lib, fvm_lib, prec, ni, nr):
    kw = dict(mach=0.5, cfl=0.5)
    g = naca_ogrid(ni, nr, radius=20.0, first_spacing=1e-2)
    o = oracle_lib.Oracle(g.coord, g.elem, g.ptype, **kw)
    s = fvm_lib.Solver(fvm_lib.make_params(precision=prec, **kw), o.mesh_arrays())
    o.d("prim")[:, 0] *= 1 + 0.5 * np.random.default_rng(3).uniform(-1, 1, g.np)
    s.set_state(o.d("prim"))
    o.gradient()
    ind = o.shockind()
    assert 0.1 < (ind > 1).mean() < 0.9
    zero = np.all(o.d("qx") == 0, axis=1)
    clear = np.abs(ind - 1) > 1e-2   # FP32: away from the limit by more than its rounding
    first = None
    for _ in range(20):
        s.gradient()
        s.shockind()
        st = s.get_state()
        if prec == L.FP64:
            np.testing.assert_array_equal(st["qx"], o.d("qx"))
            np.testing.assert_array_equal(st["qy"], o.d("qy"))
        else:
            np.testing.assert_array_equal(np.all(st["qx"] == 0, axis=1)[clear], zero[clear])
        first = first or st
        for k in ("qx", "qy"):
            np.testing.assert_array_equal(st[k], first[k])
