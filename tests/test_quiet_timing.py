"""Launch shapes are timed while no other thread renders."""
import re
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

pytestmark = pytest.mark.gpu

# four threads, each with scenes of size classes of its own to time and further updates
THREADS = """
import sys, threading, numpy as np
sys.path.insert(0, {root!r})
from realcausticsengine_gb300 import scenes
from realcausticsengine_gb300.session import Context, Renderer
images = {{}}
def work(t):
    for k in range(4):
        c = Context()
        with c:
            r = Renderer(scenes.glass_sphere_point(64 + 32 * t, 48, subdiv=3), photons_per_iter=3000 << (2 * k + t % 2), max_path_length=6,
                         seed=t, verbose=True)
            for _ in range(5):
                r.render(2)
            images[t, k] = r.image()
            r.release()
        c.destroy()
ts = [threading.Thread(target=work, args=(t,)) for t in range(4)]
[t.start() for t in ts]
[t.join() for t in ts]
for (t, k), image in images.items():
    r = Renderer(scenes.glass_sphere_point(64 + 32 * t, 48, subdiv=3), photons_per_iter=3000 << (2 * k + t % 2), max_path_length=6, seed=t)
    r.render(10)
    np.testing.assert_allclose(image, r.image(), rtol=1e-5, atol=1e-7)
    r.release()
assert len(images) == 16
"""


def test_no_other_thread_renders_while_shapes_are_timed():
    """The lines that a timing prints follow one another: another thread's iteration or timing
    in between would have run beside it.  Nothing is timed twice, and the images are those of
    a thread alone."""
    out = subprocess.run([sys.executable, "-c", THREADS.format(root=str(ROOT))], capture_output=True, text=True, timeout=240)
    assert out.returncode == 0, out.stderr
    lines = [line for line in out.stdout.splitlines() if line.startswith("{")]
    timing, timed = None, 0
    for line in lines:
        shape = re.match(r'\{"autotune_shape": "([^"]*)"', line)
        done = re.match(r'\{"autotune": "([^"]*)"', line)
        if shape:
            assert timing in (None, shape.group(1)), line
            timing = shape.group(1)
        elif done:
            assert timing == done.group(1)
            timing, timed = None, timed + 1
        else:
            assert timing is None, line
    assert timed >= 8
