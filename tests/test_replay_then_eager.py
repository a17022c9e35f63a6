"""Iterations with host round trips after replayed ones, with the camera pass on the main
stream: the events that a replayed iteration (or a batch) records belong to its graph, and a
stream cannot wait for them."""
import ctypes as C

import numpy as np
import pytest

from realcausticsengine_gb300 import _native, abi, scenes
from realcausticsengine_gb300.session import Context, Renderer, batch_render

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("replayed_by", ["render", "batch"])
def test_metropolis_after_replayed_iterations(replayed_by):
    """A scene's settings change from uniform paths, whose iterations were replayed, to short
    Metropolis chains (their camera pass runs after them): the image is that of a context
    that replays nothing."""
    sc = scenes.test_scene(64, 48, subdiv=2, rough_glass=True)
    images = []
    for replay in (True, False):
        c = Context()
        with c:
            r = Renderer(sc, photons_per_iter=20000, seed=3, graph_replay=replay)
            if replay and replayed_by == "batch":
                batch_render([c], 3)
            else:
                r.render(3)
            cfg = abi.RcConfig()
            _native.check(r.L.rc_default_config(C.byref(cfg)), "rc_default_config")
            cfg.photons_per_iter, cfg.seed, cfg.write_exr, cfg.sampler = 20000, 5, 0, abi.SAMPLER_HYBRID
            _native.check(r.L.rc_set_config(C.byref(cfg)), "rc_set_config")
            r.render(2)
            images.append(r.image())
            r.release()
        c.destroy()
    assert images[1].sum() > 0
    np.testing.assert_allclose(images[0], images[1], rtol=1e-5, atol=1e-7)
