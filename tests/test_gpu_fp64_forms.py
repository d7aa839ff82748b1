"""FP64 kernels that exist in more than one form: the gradient of inviscid
meshes alone or beside viscous ones, and the edge pass by its number of edges.
Every form does the same operations, so all equal the oracle and one another
bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fvm2d_gb300 import _lib as L  # noqa: E402
from fvm2d_gb300.ogrid import naca_ogrid  # noqa: E402

EULER = dict(mach=0.5, cfl=0.5)
LAMINAR = dict(iflow=L.LAMINAR, mach=0.5, aoa_deg=1.0, rey=5000.0, cfl=0.5)


@pytest.mark.parametrize("ni,nr", [(8, 3), (34, 23), (130, 31)])
def test_inviscid_beside_viscous_equals_alone(fvm_lib, ni, nr):
    from fvm2d_gb300.batch import Batch
    g = naca_ogrid(ni, nr, radius=20.0, first_spacing=2e-2)
    m = fvm_lib.build_geometry(g.coord, g.elem, g.ptype)
    b = Batch(L.FP64, vertices=2 * m.np + 64, meshes=2, viscous=True)
    slots = [b.add(fvm_lib.make_params(**f), m) for f in (EULER, LAMINAR)]
    for s in slots:
        b.start(s, 6)
    b.step(6)
    for s, f in zip(slots, (EULER, LAMINAR)):
        one = fvm_lib.Solver(fvm_lib.make_params(**f), m)
        one.iterate(6)
        np.testing.assert_array_equal(b.get_state(s)["prim"], one.get_state()["prim"])
    b.close()


# the forms' limits are 29k and 78k edges on 152 SMs
@pytest.mark.parametrize("ni,nr", [(160, 58), (160, 66), (250, 96), (250, 110)])
def test_edge_forms_bitwise(oracle_lib, fvm_lib, ni, nr):
    g = naca_ogrid(ni, nr, radius=20.0, first_spacing=1e-2)
    o = oracle_lib.Oracle(g.coord, g.elem, g.ptype, **EULER)
    st, _ = o.iterate(1)
    assert st == 0
    s = fvm_lib.Solver(fvm_lib.make_params(**EULER), o.mesh_arrays())
    s.set_state(o.d("prim"), o.d("nut"), o.d("mul"), o.d("mu"), iterlast=o.scalars()["iter"])
    st, _ = s.iterate(2)
    ost, _ = o.iterate(2)
    assert st == ost == 0
    np.testing.assert_array_equal(s.get_state()["prim"], o.d("prim"))


@pytest.mark.parametrize("iflux", [L.KFVS, L.HLLC, L.ROE])
def test_few_edges_alone_equal_many_in_batch(fvm_lib, iflux):
    from fvm2d_gb300.batch import Batch
    kw = dict(EULER, iflux=iflux, bugcompat=0 if iflux == L.HLLC else 1)
    g = naca_ogrid(160, 40, radius=20.0, first_spacing=1e-2)
    m = fvm_lib.build_geometry(g.coord, g.elem, g.ptype)
    one = fvm_lib.Solver(fvm_lib.make_params(**kw), m)
    one.iterate(6)
    want = one.get_state()["prim"]
    for n in (3, 5):
        b = Batch(L.FP64, vertices=n * m.np + 64 * n, meshes=n)
        slots = [b.add(fvm_lib.make_params(**kw), m) for _ in range(n)]
        for s in slots:
            b.start(s, 6)
        b.step(6)
        for s in slots:
            np.testing.assert_array_equal(b.get_state(s)["prim"], want)
        b.close()
