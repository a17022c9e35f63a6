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
for grid in (50, 160, 50, 181, 300):     # 4.8k, 51k, 4.8k, 65k (up to 2^16), 179k triangles with the floor's
    ctypes.CDLL(None).fflush(None)       # (the library prints through C's stdout)
    print("still", flush=True)
    r = Renderer(scenes.water_pool(160, 90, grid=grid), photons_per_iter=100000, max_path_length=6, seed=4, verbose=True)
    r.render(3)
    r.release()
"""


def test_stills_of_other_meshes_time_no_shapes_again():
    """Meshes between 2^12 and 2^16 triangles are one class: only the first still times the
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
