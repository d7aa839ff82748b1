"""Handles and batches of different block sizes side by side: what a kernel may
take of shared memory is set per function for the whole process, so a small one
created later must not take it from a larger one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fvm2d_gb300 import _lib as L  # noqa: E402
from fvm2d_gb300.ogrid import naca_ogrid  # noqa: E402

EULER = dict(mach=0.5, cfl=0.5)
LAMINAR = dict(iflow=L.LAMINAR, mach=0.5, aoa_deg=1.0, rey=5000.0, cfl=0.5)
RANS = dict(iflow=L.TURBULENT, mach=0.5, rey=1e5, cfl=0.5)


def mesh(fvm_lib, ni, nr):
    g = naca_ogrid(ni, nr, radius=20.0, first_spacing=1e-2)
    return fvm_lib.build_geometry(g.coord, g.elem, g.ptype, wall_distance=True)


@pytest.mark.parametrize("prec", [L.FP64, L.FP32])
@pytest.mark.parametrize("flow", [EULER, LAMINAR, RANS])
def test_small_handle_after_a_large_one(fvm_lib, prec, flow):
    big, small = mesh(fvm_lib, 300, 180), mesh(fvm_lib, 20, 5)   # blocks of 256, of 64

    def work(other):
        s = fvm_lib.Solver(fvm_lib.make_params(precision=prec, **flow), big)
        o = fvm_lib.Solver(fvm_lib.make_params(precision=prec, **EULER), small) if other else None
        s.iterate(3)
        s.residu()
        out = s.get_state()
        s.gradient()
        out["edge_qx"] = s.get_state()["qx"]
        s.close()
        if o:
            o.close()
        return out

    want, got = work(False), work(True)
    for k in want:
        np.testing.assert_array_equal(got[k], want[k])


@pytest.mark.parametrize("prec,form", [(L.FP64, "fused"), (L.FP64, "loads"), (L.FP32, "loads"),
                                       (L.FP32, "bulk"), (L.FP32, "pipe")])
def test_small_handle_beside_a_batch(fvm_lib, prec, form):
    from fvm2d_gb300.batch import Batch
    big, small = mesh(fvm_lib, 200, 60), mesh(fvm_lib, 20, 5)

    def work(other):
        b = Batch(prec, vertices=big.np, meshes=1, viscous=True)
        slot = b.add(fvm_lib.make_params(precision=prec, **LAMINAR), big)
        b.set_form(form)
        s = fvm_lib.Solver(fvm_lib.make_params(precision=prec, **EULER), small) if other else None
        b.start(slot, 3)
        b.step(3)
        out = b.get_state(slot)
        b.close()
        if s:
            s.close()
        return out

    want, got = work(False), work(True)
    for k in want:
        np.testing.assert_array_equal(got[k], want[k])
