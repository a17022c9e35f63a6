"""The staged passes over several scenes, and in several chunks: every launch shape must store,
for each scene, the records of the scene's own persistent pass.

Lanes of one warp work for different scenes there (a parked path carries its scene's index),
and a pass of more than 2^24 paths takes them in chunks that reuse the scratch; here the
chunks are small."""
import numpy as np
import pytest

from realcausticsengine_gb300 import _native, scenes
from realcausticsengine_gb300.session import Context, Renderer, pass_records


def _canonical(a):
    w = np.ascontiguousarray(a).view(np.uint32)
    return w[np.lexsort(w.T[::-1])]


def _same(got, want, what):
    assert len(got) == len(want)
    for i, (g, w) in enumerate(zip(got, want)):
        g = _canonical(g)
        assert g.shape == w.shape and (g == w).all(), (what, i)


# (scene, light paths): sizes far apart, so that some warps hold one scene and some five
def _specs():
    displaced, _ = scenes.batch_scene(3, 96, 96)
    return [
        (scenes.test_scene(64, 48, rough_glass=True, dispersion=0.03), 30000),
        (scenes.glass_sphere_point(1, 1, subdiv=1), 1),
        (displaced, 70001),
        (scenes.test_scene(3, 5, subdiv=1), 7),
        (scenes.water_pool(31, 17, grid=20), 333),
        (scenes.gem_cluster(33, 31, n_gems=5), 4097),
    ]


@pytest.fixture(scope="module")
def held():
    ctxs = []
    for k, (sc, paths) in enumerate(_specs()):
        c = Context()
        with c:
            Renderer(sc, max_path_length=8, photons_per_iter=paths, seed=30 + k).prepare()
        ctxs.append(c)
    want = [[_canonical(pass_records([c], which, 0, 2)[0]) for c in ctxs] for which in (0, 1)]
    assert all(len(w) > 0 for w in (want[0][0], want[0][2], want[0][5], want[1][0], want[1][2], want[1][5]))
    yield ctxs, want
    for c in ctxs:
        with c:
            _native.lib().rc_release()
        c.destroy()


@pytest.mark.gpu
@pytest.mark.parametrize("which", [0, 1], ids=["light", "camera"])
@pytest.mark.parametrize("shape", range(7))
def test_batch_shapes_store_each_scenes_records(held, which, shape):
    ctxs, want = held
    _same(pass_records(ctxs, which, shape, 2), want[which], shape)
    _same(pass_records(ctxs[::-1], which, shape, 2), want[which][::-1], shape)


@pytest.mark.gpu
@pytest.mark.parametrize("which", [0, 1], ids=["light", "camera"])
@pytest.mark.parametrize("shape", [4, 5, 6])
@pytest.mark.parametrize("chunk", [1000, 4096, 30011])
def test_staged_chunks_store_the_same_records(held, which, shape, chunk):
    """A ragged last chunk, chunks that start inside a scene, and one that ends with the
    first scene's 30,000 paths nearly."""
    ctxs, want = held
    _same(pass_records(ctxs, which, shape, 2, chunk), want[which], (shape, chunk))
    for k in (0, 2):
        _same(pass_records([ctxs[k]], which, shape, 2, chunk), [want[which][k]], (shape, chunk, k))


def test_pass_records_refuses_bad_arguments():
    import ctypes as C
    L = _native.lib()
    n = (C.c_longlong * 2)()
    c = Context()
    h = (C.c_void_p * 2)(c.handle, c.handle)
    try:
        for args in ((None, 1, 0, 0, 0, 0), (h, 0, 0, 0, 0, 0), (h, 1, 2, 0, 0, 0), (h, 1, 0, 7, 0, 0), (h, 1, 0, 0, -1, 0),
                     (h, 1, 0, 0, 0, -1), (h, 2, 0, 0, 0, 0)):
            assert L.rc_pass_records(*args, None, 0, n) == -2, args
        assert L.rc_pass_records(h, 1, 0, 0, 0, 0, None, 5, n) == -2
        assert L.rc_pass_records(h, 1, 0, 0, 0, 0, None, 0, None) == -2
        assert L.rc_pass_records(h, 1, 0, 0, 0, 0, None, 0, n) == -1      # no scene
    finally:
        c.destroy()
