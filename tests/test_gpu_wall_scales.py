"""wall_dist.f on the GPU bit for bit against the oracle where FP32, in which
far edges are dropped, ends: coordinates so small or so large that their squares
leave its range, edges of 1e20 beside short ones, and walls so far from the
origin that the FP64 foot points themselves are rounded coarsely."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fvm2d_gb300.ogrid import naca_ogrid  # noqa: E402


def check(fvm_lib, oracle_lib, coord, edge, ptype):
    for bc in (0, 1):
        a = fvm_lib.wall_dist(coord, edge, ptype, bc)
        b = oracle_lib.wall_dist(coord, edge, ptype, bc)
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("scale", [1e-300, 1e-160, 1e-40, 1e-25, 1e-23, 1e-22, 1e-21, 1e-18, 1e-14,
                                   1e-9, 1e9, 1e14, 1e19, 1e30, 1e160])
def test_scaled_airfoils(fvm_lib, oracle_lib, scale):
    g = naca_ogrid(130, 24, radius=50.0, first_spacing=1e-6, camber=0.03)
    m = fvm_lib.build_geometry(g.coord, g.elem, g.ptype, setup_on_gpu=False)
    check(fvm_lib, oracle_lib, m.coord * scale, m.edge, m.ptype)


@pytest.mark.parametrize("shift", [1e7, 1e9, 1e11, 1e12, 1e13])
def test_far_from_the_origin(fvm_lib, oracle_lib, shift):
    g = naca_ogrid(130, 24, radius=50.0, first_spacing=1e-2, camber=0.03)
    m = fvm_lib.build_geometry(g.coord, g.elem, g.ptype, setup_on_gpu=False)
    check(fvm_lib, oracle_lib, m.coord + np.array([shift, -0.7 * shift]), m.edge, m.ptype)


def test_very_long_edges(fvm_lib, oracle_lib):
    rng = np.random.default_rng(5)
    n = 400
    t = rng.uniform(0.1, 0.9, n)
    long_wall = np.array([[-1e20, -1e20], [1e20, 1e20]])       # through the origin at 45 degrees
    short_wall = np.array([[2e5, -2e5], [2.1e5, -2e5]])
    pts = np.stack([t, t], 1) * 2e6 + rng.uniform(1.0, 1e3, (n, 1)) * np.array([[-1.0, 1.0]])
    coord = np.concatenate([long_wall, short_wall, pts])
    edge = np.array([[1, 2], [3, 4]], np.int32)
    ptype = np.zeros(len(coord), np.int32)
    ptype[:4] = 3
    check(fvm_lib, oracle_lib, coord, edge, ptype)


def test_all_scales_at_once(fvm_lib, oracle_lib):
    rng = np.random.default_rng(11)
    n = 2500
    coord = rng.normal(size=(n, 2)) * 10.0 ** rng.uniform(-30, 22, size=(n, 1))
    ptype = np.zeros(n, np.int32)
    ptype[:600] = 3
    edge = np.stack([rng.integers(1, 601, 700), rng.integers(1, 601, 700)], 1).astype(np.int32)
    edge = edge[edge[:, 0] != edge[:, 1]]
    check(fvm_lib, oracle_lib, coord, edge, ptype)
