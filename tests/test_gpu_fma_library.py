"""The library with contracted FP64 kernels (FVM_LIB_VARIANT=fp64fma): a mesh's
result does not depend on the meshes that are resident with it (their number of
edges chooses the form of the edge pass, viscous ones the form of the
gradient)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
import sys
import numpy as np
import fvm2d_gb300 as f
from fvm2d_gb300 import _lib as L
from fvm2d_gb300.batch import Batch
from fvm2d_gb300.ogrid import naca_ogrid
assert L.LIB.endswith("_fp64fma.so")

def mesh(ni, nr):
    g = naca_ogrid(ni, nr, radius=20.0, first_spacing=1e-2)
    return g, f.build_geometry(g.coord, g.elem, g.ptype)

iflux, flow = int(sys.argv[1]), sys.argv[2]
kw = dict(mach=0.5, aoa_deg=1.0, cfl=0.5, iflux=iflux, bugcompat=0 if iflux == L.HLLC else 1)
if flow == "laminar":
    kw.update(iflow=L.LAMINAR, rey=5000.0)
g, m = mesh(60, 20)
other = dict(kw, iflow=L.LAMINAR, rey=5000.0)
got = []
for beside in ((), ((300, 40, kw),), ((300, 40, kw), (300, 90, kw)), ((40, 12, other),),
               ((300, 120, other),)):
    ms = [mesh(a, b)[1] for a, b, _ in beside]
    b = Batch(L.FP64, vertices=m.np + sum(x.np for x in ms) + 64 * (1 + len(ms)),
              meshes=1 + len(ms), viscous=True)
    s = b.add(f.make_params(**kw), m)
    for x, (_, _, k) in zip(ms, beside):
        b.start(b.add(f.make_params(**k), x), 6)
    b.start(s, 6)
    b.step(6)
    got.append(b.get_state(s)["prim"])
    b.close()
off = [float(np.abs(x - got[0]).max()) for x in got]
print(off)
assert not any(off)
"""


@pytest.mark.parametrize("iflux", [1, 2, 3])
@pytest.mark.parametrize("flow", ["euler", "laminar"])
def test_company_changes_no_bit(fvm_lib, iflux, flow):
    env = dict(os.environ, FVM_LIB_VARIANT="fp64fma", PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", PROGRAM, str(iflux), flow], cwd=ROOT, env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
