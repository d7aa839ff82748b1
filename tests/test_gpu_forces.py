"""clcd.f's force sums of the FP64 path: the terms of a tile of wall edges are
formed by all threads, the additions are one chain in edge order.  Checked bit
for bit against the same chain in Python on the handle's own state, with fewer
wall edges than a tile (256), exactly one, one edge more and several tiles, and
with the viscous terms zero (Euler) and not (laminar)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fvm2d_gb300 import _lib as L  # noqa: E402
from fvm2d_gb300.ogrid import naca_ogrid  # noqa: E402


def chain(m, st, par):
    """clcd.f:20-46 in its own order of operations."""
    xf = yf = 0.0
    n2b3 = 2.0 / 3.0
    for e in m.beindx[m.nswe1 - 1:m.nswe2]:
        n = m.edge[e - 1] - 1
        d = m.coord[n[1]] - m.coord[n[0]]
        sx, sy = float(d[1]), -float(d[0])
        t = []
        for v in n:
            mu, qx, qy = float(st["mu"][v]), st["qx"][v], st["qy"][v]
            t.append((n2b3 * mu * (2.0 * float(qx[1]) - float(qy[2])),
                      mu * (float(qy[1]) + float(qx[2])),
                      n2b3 * mu * (2.0 * float(qy[2]) - float(qx[1]))))
        txx, txy, tyy = (0.5 * (a + b) for a, b in zip(*t))
        pp = 0.5 * (float(st["prim"][n[0], 3]) + float(st["prim"][n[1], 3]))
        xf = xf + pp * sx - txx * sx - txy * sy
        yf = yf + pp * sy - txy * sx - tyy * sy
    q = 0.5 * par.r_inf * (par.q_inf * par.q_inf)
    s, c = math.sin(par.aoa), math.cos(par.aoa)
    return (-s * xf + c * yf) / q, (c * xf + s * yf) / q


@pytest.mark.parametrize("ni", [32, 256, 258, 770])
@pytest.mark.parametrize("flow", [dict(mach=0.8, aoa_deg=1.25),
                                  dict(iflow=L.LAMINAR, mach=0.5, aoa_deg=2.0, rey=5000.0, cfl=0.8)])
def test_force_chain_bitwise(fvm_lib, ni, flow):
    g = naca_ogrid(ni, 10, radius=20.0, first_spacing=2e-3)
    m = fvm_lib.build_geometry(g.coord, g.elem, g.ptype)
    par = fvm_lib.make_params(**flow)
    s = fvm_lib.Solver(par, m)
    _, h = s.iterate(3)
    st = s.get_state()
    # the iteration's own forces use the state after its last stage and the
    # gradients and viscosity that stage started from: what get_state returns
    cl, cd = chain(m, st, par)
    assert (h["cl"][-1], h["cd"][-1]) == (cl, cd)
    assert s.clcd() == (cl, cd)
    s.close()
