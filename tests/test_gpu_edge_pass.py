"""The FP64 flux pass in two kernels (edges, then gather): residuals and whole
iterations against the oracle at the sizes where its work items can go wrong:
fewer edges than one item, one block exactly full, one vertex row more, several
blocks with ragged items, and boundary edges cut between blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fvm2d_gb300 import _lib as L  # noqa: E402
from fvm2d_gb300.ogrid import naca_ogrid  # noqa: E402

SIZES = [(8, 3), (16, 16), (16, 17), (34, 23), (130, 31)]


def pair(oracle_lib, fvm_lib, ni, nr, **kw):
    g = naca_ogrid(ni, nr, radius=20.0, first_spacing=2e-2)
    o = oracle_lib.Oracle(g.coord, g.elem, g.ptype, **kw)
    st, _ = o.iterate(2)
    assert st == 0
    s = fvm_lib.Solver(fvm_lib.make_params(**kw), o.mesh_arrays())
    s.set_state(o.d("prim"), o.d("nut"), o.d("mul"), o.d("mu"), iterlast=o.scalars()["iter"])
    return o, s


@pytest.mark.parametrize("ni,nr", SIZES)
@pytest.mark.parametrize("ilimit", [0, 1])
def test_residual_and_iterations_bitwise(oracle_lib, fvm_lib, ni, nr, ilimit):
    o, s = pair(oracle_lib, fvm_lib, ni, nr, ilimit=ilimit, mach=0.5, cfl=0.5)
    o.residu()
    s.residu()
    np.testing.assert_array_equal(s.residual(), o.d("res"))
    st, h = s.iterate(5)
    ost, oh = o.iterate(5)
    assert st == ost == 0
    np.testing.assert_array_equal(s.get_state()["prim"], o.d("prim"))
    np.testing.assert_array_equal(h["iresi"], oh["iresi"])


@pytest.mark.parametrize("ni,nr", SIZES)
@pytest.mark.parametrize("iflux", [L.KFVS, L.HLLC])
def test_other_fluxes(oracle_lib, fvm_lib, ni, nr, iflux):
    """erf, exp and pow differ from libm by a few ulp: 1e-12 of the largest
    residual, as in the parity tests."""
    o, s = pair(oracle_lib, fvm_lib, ni, nr, iflux=iflux, mach=0.5, cfl=0.5, bugcompat=0)
    o.residu()
    s.residu()
    r, ro = s.residual(), o.d("res")
    assert np.abs(r - ro).max() <= 1e-12 * np.abs(ro).max()


def test_mixed_batch_equals_single(fvm_lib):
    """Meshes of several sizes and solvers share the pass and its buffers."""
    from fvm2d_gb300.batch import Batch
    flows = [dict(iflux=L.ROE), dict(iflux=L.KFVS), dict(iflux=L.HLLC, bugcompat=0)]
    ms = []
    for ni, nr in ((16, 17), (34, 23), (130, 31)):
        g = naca_ogrid(ni, nr, radius=20.0, first_spacing=2e-2)
        ms.append(fvm_lib.build_geometry(g.coord, g.elem, g.ptype))
    b = Batch(L.FP64, vertices=sum(m.np for m in ms) + 64, meshes=3, overlap=2)
    slots = [b.add(fvm_lib.make_params(mach=0.5, cfl=0.5, **f), m) for f, m in zip(flows, ms)]
    for s in slots:
        b.start(s, 12)
    b.step(12)
    for s, f, m in zip(slots, flows, ms):
        one = fvm_lib.Solver(fvm_lib.make_params(mach=0.5, cfl=0.5, **f), m)
        one.iterate(12)
        np.testing.assert_array_equal(b.get_state(s)["prim"], one.get_state()["prim"])
    b.close()
