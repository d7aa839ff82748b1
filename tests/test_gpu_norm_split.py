"""The residual norm (conres.f) of a handle, whose blocks of 256 vertices are
split when the mesh is small, equals a batch's bit for bit also where the sums
of FP32 states' squares are not exact: densities over three decades."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fvm2d_gb300 import _lib as L  # noqa: E402
from fvm2d_gb300.ogrid import naca_ogrid  # noqa: E402


@pytest.mark.parametrize("ni,nr", [(100, 60), (200, 150)])   # blocks of 64, of 128
@pytest.mark.parametrize("prec", [L.FP32, L.FP64])
def test_norm_does_not_depend_on_the_split(fvm_lib, prec, ni, nr):
    from fvm2d_gb300.batch import Batch
    g = naca_ogrid(ni, nr, radius=20.0, first_spacing=2e-2)
    m = fvm_lib.build_geometry(g.coord, g.elem, g.ptype)
    par = fvm_lib.make_params(precision=prec, mach=0.5, cfl=0.1)
    s = fvm_lib.Solver(par, m)
    prim = s.get_state()["prim"]
    i, j = np.arange(m.np) % ni, np.arange(m.np) // ni
    scale = 10.0 ** (1.5 * np.sin(6 * np.pi * i / ni) * np.cos(4 * np.pi * j / nr))
    prim[:, 0] *= scale
    prim[:, 3] *= scale
    s.set_state(prim)
    _, h = s.iterate(8)
    b = Batch(prec, vertices=m.np, meshes=1)
    slot = b.add(par, m)
    b.set_state(slot, prim)
    b.start(slot, 8)
    b.step(8)
    hb = b.history(slot, 0, 8)
    for k in ("fresi", "iresi", "fres"):
        np.testing.assert_array_equal(h[k], hb[k])
    b.close()
