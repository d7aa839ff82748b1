"""wall_dist.f on the GPU bit for bit against the oracle, where dropping far
edges could go wrong: airfoils with fewer wall edges than a tile (256), exactly
one tile and several; walls far from the origin (FP32 differences cancel);
points on, very near and very far from the wall; long and short edges side by
side; no wall at all; both forms of line 46."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fvm2d_gb300.ogrid import naca_ogrid  # noqa: E402


def check(fvm_lib, oracle_lib, coord, edge, ptype):
    for bc in (0, 1):
        a = fvm_lib.wall_dist(coord, edge, ptype, bc)
        b = oracle_lib.wall_dist(coord, edge, ptype, bc)
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("ni,nr,first", [(16, 5, 1e-2), (256, 24, 1e-6), (258, 24, 1e-3), (700, 9, 1e-4)])
@pytest.mark.parametrize("shift", [0.0, 1.0e4])
def test_airfoils(fvm_lib, oracle_lib, ni, nr, first, shift):
    g = naca_ogrid(ni, nr, radius=50.0, first_spacing=first, camber=0.03)
    m = fvm_lib.build_geometry(g.coord, g.elem, g.ptype, setup_on_gpu=False)
    check(fvm_lib, oracle_lib, m.coord + shift, m.edge, m.ptype)


def test_scattered_edges(fvm_lib, oracle_lib):
    rng = np.random.default_rng(7)
    n = 3000
    coord = rng.normal(size=(n, 2)) * 10.0 ** rng.uniform(-6, 3, size=(n, 1))
    ptype = np.zeros(n, np.int32)
    ptype[:700] = 3
    edge = np.stack([rng.integers(1, 701, 900), rng.integers(1, 701, 900)], 1).astype(np.int32)
    edge = edge[edge[:, 0] != edge[:, 1]]
    coord[2000:2100] = coord[:100]                    # points on wall points
    coord[2100:2200] = coord[:100] * (1 + 1e-15)
    check(fvm_lib, oracle_lib, coord, edge, ptype)


def test_no_wall(fvm_lib, oracle_lib):
    rng = np.random.default_rng(3)
    coord = rng.normal(size=(50, 2))
    edge = np.array([[1, 2], [2, 3]], np.int32)
    check(fvm_lib, oracle_lib, coord, edge, np.zeros(50, np.int32))
