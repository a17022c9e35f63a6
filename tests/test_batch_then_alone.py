"""Scenes that a batch rendered first, rendered alone afterwards."""
import json
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

pytestmark = pytest.mark.gpu

# 2.6M paths on the pool: the staged light pass wins there, and an untimed one is persistent
TWO = """
import ctypes, sys, numpy as np
sys.path.insert(0, {root!r})
from realcausticsengine_gb300 import scenes
from realcausticsengine_gb300.session import Context, Renderer, batch_render
def out(s):
    ctypes.CDLL(None).fflush(None)
    print(s, flush=True)
cs, rs = [Context(), Context()], []
for k, c in enumerate(cs):
    with c:
        rs.append(Renderer(scenes.water_pool(160, 90, grid=24), photons_per_iter=(2600000, {second})[k], max_path_length=8,
                           seed=4 + k, verbose=True))
batch_render(cs, 2)
for c, r in zip(cs, rs):
    out("alone")
    with c:
        r.render(3)
        image = r.image()
with cs[1]:
    r = Renderer(scenes.water_pool(160, 90, grid=24), photons_per_iter={second}, max_path_length=8, seed=5)
    r.render(5)
    np.testing.assert_allclose(image, r.image(), rtol=1e-5, atol=1e-7)
"""


@pytest.mark.parametrize("second", [2600000, 4500000, 1500000], ids=["the same class", "the next", "the one before"])
def test_the_second_scene_of_a_class_replays_the_shapes_timed_for_the_first(second):
    """Both scenes get their capacities from the batch, in which nothing of their own was
    timed.  The first one rendered alone times its class; the second one, of that class of
    paths or a neighbouring one, has nothing left to time and must not stay with the shapes
    that it was given in the batch."""
    out = subprocess.run([sys.executable, "-c", TWO.format(root=str(ROOT), second=second)], capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0, out.stderr
    first, second = [[json.loads(line) for line in part.splitlines() if line.startswith('{"autotune":') or
                      line.startswith('{"replayed_iterations":')] for part in out.stdout.split("alone\n")[1:3]]
    timed = {t["autotune"]: t["variant"] for t in first if "autotune" in t}
    replay = [t for t in second if "replayed_iterations" in t]
    assert not [t for t in second if t.get("autotune") in ("light pass", "camera pass")]
    assert len(replay) == 1 and replay[0]["replayed_iterations"] == 3
    assert (replay[0]["light_shape"], replay[0]["camera_shape"]) == (timed["light pass"], timed["camera pass"])
