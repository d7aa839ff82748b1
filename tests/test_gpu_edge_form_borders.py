"""The FP64 edge pass on either side of its rule's two borders (items of four
warps in one wave; edge entries in one wave of threads), where the form really
changes: a handle of each size against the oracle, and batches that grow over
both borders against one mesh alone, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fvm2d_gb300 import _lib as L  # noqa: E402
from fvm2d_gb300.ogrid import naca_ogrid  # noqa: E402


def params(iflux):
    return dict(mach=0.5, cfl=0.5, iflux=iflux, bugcompat=0 if iflux == L.HLLC else 1)


# sizes next to the borders on 152 SMs, each in
# blocks of 64 (to 10000 vertices) or 128
@pytest.mark.parametrize("iflux", [L.ROE, L.KFVS, L.HLLC])
@pytest.mark.parametrize("below,above,forms", [((160, 50), (160, 54), (2, 0)),
                                               ((250, 88), (250, 94), (0, 1))])
def test_handles_beside_each_border(oracle_lib, fvm_lib, below, above, forms, iflux):
    got = []
    for ni, nr in (below, above):
        g = naca_ogrid(ni, nr, radius=20.0, first_spacing=1e-2)
        o = oracle_lib.Oracle(g.coord, g.elem, g.ptype, **params(iflux))
        st, _ = o.iterate(5)
        assert st == 0
        s = fvm_lib.Solver(fvm_lib.make_params(**params(iflux)), o.mesh_arrays())
        got.append(s.edge_form())
        s.set_state(o.d("prim"), o.d("nut"), o.d("mul"), o.d("mu"), iterlast=o.scalars()["iter"])
        o.residu()
        s.residu()
        if iflux == L.ROE:
            np.testing.assert_array_equal(s.residual(), o.d("res"))
        else:   # pow, erf and exp differ from the C library's by a few ulp
            assert np.abs(s.residual() - o.d("res")).max() < 1e-12 * np.abs(o.d("res")).max()
    assert tuple(got) == forms


@pytest.mark.parametrize("iflux", [L.ROE, L.KFVS, L.HLLC])
def test_batch_growing_over_both_borders(fvm_lib, iflux):
    from fvm2d_gb300.batch import Batch
    g = naca_ogrid(160, 40, radius=20.0, first_spacing=1e-2)
    m = fvm_lib.build_geometry(g.coord, g.elem, g.ptype)
    par = fvm_lib.make_params(**params(iflux))
    one = fvm_lib.Solver(par, m)
    one.iterate(6)
    want = one.get_state()["prim"]
    b = Batch(L.FP64, vertices=4 * m.np + 256, meshes=4)
    forms = []
    for _ in range(4):
        slots = [b.add(par, m)]
        forms.append(b.edge_form())
        b.start(slots[0], 6)
        b.step(6)
        np.testing.assert_array_equal(b.get_state(slots[0])["prim"], want)
    b.close()
    assert forms == [2, 0, 0, 1]
