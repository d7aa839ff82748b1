"""A single mesh's handle splits its leaves of 256 vertices into blocks of 64 or
128 when the mesh is small; a batch keeps whole leaves.  Both number the
vertices alike and add in the same pairs, so states, residual norms and forces
must be equal bit for bit on either side of each border of the rule (10000 and
50000 vertices) and between, with a last leaf that is ragged."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fvm2d_gb300 import _lib as L  # noqa: E402
from fvm2d_gb300.ogrid import naca_ogrid  # noqa: E402


@pytest.mark.parametrize("ni,nr", [(20, 5), (100, 99), (100, 101), (200, 161), (200, 249), (200, 251)])
@pytest.mark.parametrize("prec", [L.FP64, L.FP32])
@pytest.mark.parametrize("flow", [dict(mach=0.6, aoa_deg=1.25, cfl=0.8),
                                  dict(iflow=L.LAMINAR, mach=0.5, rey=5000.0, cfl=0.5)])
def test_handle_equals_batch(fvm_lib, ni, nr, prec, flow):
    from fvm2d_gb300.batch import Batch
    g = naca_ogrid(ni, nr, radius=20.0, first_spacing=2e-3)
    m = fvm_lib.build_geometry(g.coord, g.elem, g.ptype)
    par = fvm_lib.make_params(precision=prec, **flow)
    s = fvm_lib.Solver(par, m)
    _, h = s.iterate(12)
    b = Batch(prec, vertices=m.np, meshes=1, viscous=True)
    slot = b.add(par, m)
    b.start(slot, 12)
    b.step(12)
    hb = b.history(slot, 0, 12)
    for k in ("fres", "iresi", "fresi", "cl", "cd"):
        np.testing.assert_array_equal(h[k], hb[k])
    st, sb = s.get_state(), b.get_state(slot)
    for k in ("prim", "qx", "qy", "mul"):
        np.testing.assert_array_equal(st[k], sb[k])
    b.close()
