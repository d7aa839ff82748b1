"""The largest density change (conres.f:17-21) of FP32 states whose density
overflows in an iteration: |gra| > fresi holds for an infinite change, so fresi
is infinite and iresi the first such point, in a batch and in a handle (whose
blocks are smaller).  States found by search: the density of a few points (a
handful, beside NaN and finite ones) becomes infinite in the last stage."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fvm2d_gb300 import _lib as L  # noqa: E402
from fvm2d_gb300.ogrid import naca_ogrid  # noqa: E402


@pytest.mark.parametrize("ni,nr,seed", [(20, 6, 206), (20, 6, 682), (20, 6, 2697), (40, 24, 771),
                                        (40, 24, 2241), (40, 24, 3344)])
def test_overflowing_change_is_the_largest(fvm_lib, ni, nr, seed):
    from fvm2d_gb300.batch import Batch
    g = naca_ogrid(ni, nr, radius=20.0, first_spacing=1e-2)
    m = fvm_lib.build_geometry(g.coord, g.elem, g.ptype)
    rng = np.random.default_rng(seed)
    cfl = 10 ** rng.uniform(-1, 2)
    top = 10 ** rng.uniform(35.5, 37.9)
    spread = 10 ** rng.uniform(0.01, 1.5)
    p = 10 ** rng.uniform(-1, 2)
    prim = np.zeros((m.np, 4))
    prim[:, 0] = top / spread ** rng.random(m.np)
    prim[:, 3] = p * (1 + 0.5 * rng.random(m.np) * rng.integers(0, 2))
    par = fvm_lib.make_params(precision=L.FP32, mach=0.5, cfl=cfl, iflux=L.HLLC, ilimit=0,
                              bugcompat=0)
    b = Batch(L.FP32, vertices=m.np, meshes=1)
    slot = b.add(par, m)
    b.set_state(slot, prim)
    b.start(slot, 1)
    b.step(1)
    h = b.history(slot, 0, 1)
    rho = b.get_state(slot)["prim"][:, 0]
    b.close()
    assert np.isinf(rho).any()   # or the state no longer tests anything
    s = fvm_lib.Solver(par, m)
    s.set_state(prim)
    _, hs = s.iterate(1)
    np.testing.assert_array_equal(s.get_state()["prim"][:, 0], rho)
    for x in (h, hs):
        assert x["fresi"][0] == np.inf
        assert x["iresi"][0] == np.flatnonzero(np.isinf(rho))[0] + 1
