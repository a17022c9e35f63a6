"""The staged light and camera passes and the photons' spatial order at the sizes where their
work division can go wrong.

The staged shapes (4-6) must store exactly the records of the persistent shape 0: path
counts around a warp's 32, a block's 128 and the refill of ended lanes, images of odd
sizes.  The spatial order must answer radius queries exactly whatever its cut into chunks
(around 31/32 photons), its sort tiles (4096 keys) and its key width (32-bit up to 2048
radii across, 64-bit beyond), clamped and coincident points included.
"""
import numpy as np
import pytest

from realcausticsengine_gb300 import scenes
from realcausticsengine_gb300.session import Renderer, kd_query

pytestmark = pytest.mark.gpu


def _canonical(a):
    w = np.ascontiguousarray(a).view(np.uint32)
    return w[np.lexsort(w.T[::-1])]


@pytest.mark.parametrize("paths", [1, 31, 33, 127, 4097, 60001])
def test_staged_light_pass_stores_the_same_photons(paths):
    r = Renderer(scenes.test_scene(32, 24, subdiv=2, rough_glass=True, dispersion=0.03), max_path_length=8,
                 photons_per_iter=paths, seed=9)
    r.prepare()
    want = _canonical(r.light_photons_shape(0, 1))
    for shape in (4, 5, 6):
        got = _canonical(r.light_photons_shape(shape, 1))
        assert got.shape == want.shape and (got == want).all(), f"shape {shape}"
    r.release()


@pytest.mark.parametrize("size", [(1, 1), (7, 5), (33, 31), (161, 97)])
def test_staged_camera_pass_writes_the_same_queries(size):
    r = Renderer(scenes.test_scene(*size, subdiv=2, dispersion=0.03), max_path_length=8, photons_per_iter=64, seed=3)
    r.prepare()
    want = _canonical(r.camera_queries(2))
    for shape in (4, 5, 6):
        got = _canonical(r.camera_queries(2, shape))
        assert got.shape == want.shape and (got == want).all(), f"shape {shape}"
    r.release()


@pytest.mark.parametrize("lanes,paths", [(1, 2735), (2, 2737), (31, 57455), (32, 57457)])
def test_small_passes_spread_over_warps_store_the_same(lanes, paths):
    """On 152 SMs a warp of the persistent shapes holds `lanes` paths at these sizes."""
    r = Renderer(scenes.test_scene(paths // 97, 97, subdiv=2, rough_glass=True, dispersion=0.03), max_path_length=6,
                 photons_per_iter=paths, seed=5)
    r.prepare()
    photons, queries = _canonical(r.light_photons_shape(4, 1)), _canonical(r.camera_queries(1, 4))
    for shape in range(4):
        for got, want in ((r.light_photons_shape(shape, 1), photons), (r.camera_queries(1, shape), queries)):
            got = _canonical(got)
            assert got.shape == want.shape and (got == want).all(), f"shape {shape}"
    r.release()


@pytest.mark.parametrize("radius", [0.4, 2e-3, 1e-5])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 4095, 4097, 20011])
def test_spatial_order_finds_every_photon(n, radius):
    """Against every pair, with the reference's FP32 predicate."""
    rng = np.random.default_rng(n)
    p = rng.uniform(-3, 3, (n, 3)).astype(np.float32)
    spot = rng.integers(0, n, n // 2)
    p[spot] = p[0] + rng.normal(scale=radius, size=(len(spot), 3)).astype(np.float32)   # a dense spot
    p[rng.integers(0, n, n // 8)] = p[0]                                                # coincident
    q = np.concatenate([p[rng.integers(0, n, 300)], rng.uniform(-9, 9, (100, 3)).astype(np.float32)])
    r2 = np.float32(radius) * np.float32(radius)
    counts, sets = kd_query(p, q, float(r2))
    for j in range(0, len(q), 7):
        d = q[j] - p
        inside = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2] < r2
        assert counts[j] == inside.sum()
        assert (np.sort(sets[j]) == np.nonzero(inside)[0]).all()


@pytest.mark.parametrize("n,q", [(1, 40), (33, 400), (2011, 333), (3001, 4001)])
def test_parking_gather_finds_every_photon(n, q):
    """Every query's sphere holds most photons, so every warp parks (no subtrees with one
    chunk, chunks only, whole subtrees, and more items than the list holds)."""
    rng = np.random.default_rng(q)
    p = rng.normal(scale=0.5, size=(n, 3)).astype(np.float32)
    at = rng.normal(scale=0.1, size=(q, 3)).astype(np.float32)
    want, sets = kd_query(p, at, 1.0, variant=0)
    for j in range(0, q, 97):
        d = at[j] - p
        inside = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2] < np.float32(1.0)
        assert (np.sort(sets[j]) == np.nonzero(inside)[0]).all()
    for variant in (8, 9):
        counts, got = kd_query(p, at, 1.0, variant=variant)
        assert (counts == want).all()
        assert all((np.sort(a) == np.sort(b)).all() for a, b in zip(got, sets))
