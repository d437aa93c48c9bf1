"""Searches of the track compiler where their shortcuts end: routes with many waypoints at one distance from a cell
(32-bit comparisons leave the order open and 64 bits decide), and feature transforms of rows around the sizes where the
row pass changes its staging (12288 cells) and the type of its squared distances (32767 cells), with sparse and dense
features and their ties. Packed tracks equal the oracle's bit for bit."""
import numpy as np
import pytest

import oracle
from warporacer3d_gb300.tracks import compile as C

pytestmark = pytest.mark.gpu


def assert_bits(ours, ref):
    assert ours.shape == ref.shape
    assert np.array_equal(ours.view(np.uint32), ref.view(np.uint32))


def circle(n, radius):
    t = np.linspace(0, 2 * np.pi, n, endpoint=False)
    return np.column_stack([radius * np.cos(t), radius * np.sin(t), 0 * t])


@pytest.mark.parametrize("radius,half_width,cell,shift", [
    (2.0, 2.2, 0.05, 0.0),    # every ball holds the centre, where all waypoints are equally far
    (2.0, 0.5, 0.031, 1e6),   # places far from the origin
    (40.0, 0.3, 0.4, 0.0),    # most cells far from the road, blocks wider than its bend
])
def test_equidistant_waypoints_equal_oracle(radius, half_width, cell, shift):
    route = circle(300, radius) + [shift, -shift, 0.0]
    assert_bits(C.ribbon(route, half_width, 0.1, cell), oracle.track_ribbon(route, half_width, 0.1, cell))


@pytest.mark.parametrize("nx,ny", [(31, 40), (32, 33), (33, 7), (65, 200), (721, 100), (12288, 3), (12289, 4), (32767, 3),
                                   (32768, 3), (3, 32768)])
@pytest.mark.parametrize("density", [0.002, 0.5])
def test_feature_transform_sizes_equal_oracle(nx, ny, density):
    rng = np.random.default_rng(nx + ny)
    free = rng.random((ny, nx)) < density
    free[ny // 2, nx // 2], free[0, 0] = True, False
    t = np.linspace(0, 2 * np.pi, 120, endpoint=False)
    loop = np.column_stack([ny / 2 + ny / 3 * np.sin(t), nx / 2 + nx / 3 * np.cos(t)])
    cell = 4.0 / max(nx, ny)
    assert_bits(C.compile_image(free, loop, 0.0, 0.0, cell), oracle.track_image(free, loop, 0.0, 0.0, cell))
