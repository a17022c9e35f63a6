"""Limits of the render passes' scratch: the gather's list of parked work, and the staged
passes' parked paths."""
import json
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from realcausticsengine_gb300 import _native, scenes
from realcausticsengine_gb300.session import Context, Renderer, kd_query

ROOT = Path(__file__).resolve().parents[1]

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant,group", [(8, 16), (9, 32)])
def test_a_full_parked_list_is_not_asked_again(variant, group):
    """990 photons are 32 chunks under one node, all inside every query's sphere, so every
    group wants to park at most 32 items.  The list's 65,535 run out after some 2,200 of
    40,000 groups; past that only warps in flight (64 on each of at most 160 SMs) may still
    have asked, or the 32-bit count would grow with the launch and wrap in a larger one."""
    rng = np.random.default_rng(5)
    p = rng.normal(scale=0.05, size=(990, 3)).astype(np.float32)
    q = rng.normal(scale=0.05, size=(40000 * group, 3)).astype(np.float32)
    counts, _ = kd_query(p, q, 9.0, with_indices=False, variant=variant)
    assert (counts == 990).all()
    asked = _native.lib().rc_gather_parked_items()
    assert 65535 <= asked <= 65535 + 160 * 64 * 32


def _canonical(a):
    w = np.ascontiguousarray(a).view(np.uint32)
    return w[np.lexsort(w.T[::-1])]


def test_staged_shapes_without_scratch_run_persistent():
    """Over the limit every staged shape gives the persistent shapes' photons and queries;
    with the limit lifted too."""
    r = Renderer(scenes.test_scene(65, 33, subdiv=2, rough_glass=True), max_path_length=8, photons_per_iter=5000, seed=2)
    r.prepare()
    want = _canonical(r.light_photons_shape(0, 1)), _canonical(r.camera_queries(1, 0))
    try:
        for limit in (0, 48 * 2000, -1):
            _native.check(r.L.rc_pass_scratch_limit(limit), "rc_pass_scratch_limit")
            for shape in (4, 5, 6):
                for got, w in zip((r.light_photons_shape(shape, 1), r.camera_queries(1, shape)), want):
                    got = _canonical(got)
                    assert got.shape == w.shape and (got == w).all()
    finally:
        r.L.rc_pass_scratch_limit(-1)
        r.release()


# 2.6M paths on the pool: the staged light pass wins there (1.01 against 1.28 ms), so a
# process that has timed the shapes replays it
RENDER = """
import ctypes, sys, numpy as np
sys.path.insert(0, {root!r})
from realcausticsengine_gb300 import scenes, _native
from realcausticsengine_gb300.session import Context, Renderer, batch_render
images = []
for limit in (0, -1, 0):
    ctypes.CDLL(None).fflush(None)   # (the library prints through C's stdout)
    print("limit", limit, flush=True)
    c = Context()
    with c:
        _native.check(c.L.rc_pass_scratch_limit(limit), "limit")
        r = Renderer(scenes.water_pool(160, 90, grid=24), photons_per_iter=2600000, max_path_length=8, seed=4, verbose=True)
        r.render(4)
        images.append(r.image())
        batch_render([c], 2)
        images.append(r.image())
        r.release()
    c.destroy()
for k in (2, 3, 4, 5):
    np.testing.assert_allclose(images[k], images[k % 2], rtol=1e-5, atol=1e-7)
assert images[0].sum() > 0
"""


def test_no_shape_is_kept_from_a_context_without_scratch():
    """Rendered and batched without scratch, nothing is timed (a shape that could not run
    would look the fastest, for every context of the process); a context with scratch then
    times the shapes, and one without renders the same image beside it."""
    out = subprocess.run([sys.executable, "-c", RENDER.format(root=str(ROOT))], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    parts = out.stdout.split("limit ")[1:]
    tuned = [[json.loads(line)["autotune"] for line in p.splitlines() if line.startswith('{"autotune":')] for p in parts]
    passes = [[t for t in p if t != "gather"] for p in tuned]
    assert passes[0] == [] and passes[2] == []
    assert sorted(passes[1]) == ["batch passes", "camera pass", "light pass"]


BATCH_FIRST = """
import ctypes, sys, numpy as np
sys.path.insert(0, {root!r})
from realcausticsengine_gb300 import scenes
from realcausticsengine_gb300.session import Context, Renderer, batch_render
c = Context()
with c:
    r = Renderer(scenes.water_pool(160, 90, grid=24), photons_per_iter=300000, max_path_length=8, seed=4, verbose=True)
    batch_render([c], 3)
    ctypes.CDLL(None).fflush(None)
    print("alone", flush=True)
    r.render(2)
    r.render(2)
    assert r.stats()["iterations"] == 7
    image = r.image()
    r.release()
    r = Renderer(scenes.water_pool(160, 90, grid=24), photons_per_iter=300000, max_path_length=8, seed=4)
    r.render(7)
    np.testing.assert_allclose(image, r.image(), rtol=1e-5, atol=1e-7)
    r.release()
c.destroy()
"""


def test_a_scene_first_rendered_in_a_batch_times_its_own_passes():
    """The batch renders a scene's first iteration without timing the scene's own passes; the
    first render of the scene alone does it, once, and goes on to replay."""
    out = subprocess.run([sys.executable, "-c", BATCH_FIRST.format(root=str(ROOT))], capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0, out.stderr
    batch, alone = out.stdout.split("alone\n")
    assert '{"autotune": "light pass"' not in batch and '{"autotune": "camera pass"' not in batch
    for name in ("light pass", "camera pass"):
        assert alone.count('{"autotune": "%s"' % name) == 1
    assert '{"replayed_iterations": 2' in alone
