"""What the autotuner times: launches that a render pays for in its first iteration of a size
class, so their number is bounded and a scene of the same class adds none."""
import json
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

STILLS = """
import ctypes, sys
sys.path.insert(0, {root!r})
from realcausticsengine_gb300 import scenes
from realcausticsengine_gb300.session import Renderer
for grid in (50, 90, 47, 50, 300):       # 4.8k, 15.8k, 4.2k, 4.8k, 179k triangles with the floor's
    ctypes.CDLL(None).fflush(None)       # (the library prints through C's stdout)
    print("still", flush=True)
    r = Renderer(scenes.water_pool(160, 90, grid=grid), photons_per_iter=100000, max_path_length=6, seed=4, verbose=True)
    r.render(3)
    r.release()
"""


def test_stills_of_other_meshes_time_no_shapes_again():
    """Meshes between 2^12 and 2^14 triangles are one class: only the first still times the
    light and camera passes' shapes, and the first beyond times them again, each shape at
    most once and not the family that its first timing shows to be slower."""
    out = subprocess.run([sys.executable, "-c", STILLS.format(root=str(ROOT))], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    timed = []
    for part in out.stdout.split("still\n")[1:]:
        rows = [json.loads(line) for line in part.splitlines() if line.startswith('{"autotune_shape"')]
        timed.append({name: [(r["variant"], r["ms"]) for r in rows if r["autotune_shape"] == name]
                      for name in ("light pass", "camera pass")})
    assert [len(t["light pass"]) > 0 for t in timed] == [True, False, False, False, True]
    assert [len(t["camera pass"]) > 0 for t in timed] == [True, False, False, False, True]
    for t in (timed[0], timed[4]):
        for name, rows in t.items():
            shapes, ms = [v for v, _ in rows], dict(rows)
            assert len(shapes) == len(set(shapes)) and set(shapes) <= set(range(7)), name
            assert {0, 6} <= set(shapes)
            if ms[6] > 1.16 * ms[0]:
                assert not {4, 5} & set(shapes), name
            if ms[0] > 1.16 * ms[6]:
                assert not {1, 2, 3} & set(shapes), name


BATCHES = """
import ctypes, sys
sys.path.insert(0, {root!r})
from realcausticsengine_gb300 import scenes
from realcausticsengine_gb300.session import Context, Renderer, batch_render
for grid, paths in ((24, 20000), (28, 25000), (24, 200000), (300, 20000), (24, 20000)):
    held = []
    for k in range(2):
        c = Context()
        with c:
            Renderer(scenes.water_pool(80, 45, grid=grid), photons_per_iter=paths, max_path_length=6, seed=4 + k)
        held.append(c)
    c = Context()
    with c:
        Renderer(scenes.water_pool(80, 45, grid=grid), photons_per_iter=1000, max_path_length=6, seed=2, verbose=True)
        batch_render(held + [c], 2)
        ctypes.CDLL(None).fflush(None)
    for c in held + [c]:
        c.destroy()
    print("end of batch", flush=True)
"""


def test_batches_of_another_size_class_time_their_own_shapes():
    """A batch's light and camera passes take the shapes timed on a batch of their size: the
    second batch (the same classes of paths and triangles) times nothing, the third (more
    paths) its light pass, the fourth (larger meshes) both, and the first again nothing."""
    out = subprocess.run([sys.executable, "-c", BATCHES.format(root=str(ROOT))], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    timed = []
    for part in out.stdout.split("end of batch\n")[:5]:
        rows = [json.loads(line) for line in part.splitlines() if line.startswith('{"autotune_shape"')]
        timed.append({r["autotune_shape"] for r in rows if r["autotune_shape"].startswith("batch")})
    both = {"batch light pass", "batch camera pass"}
    assert timed == [both, set(), {"batch light pass"}, both, set()]
