"""The Metropolis chains of the render (a warp's searches in phases, sample vectors drawn as
far as a path needs them, finished steps settled together) against the same chains one step
at a time with whole sample vectors: the same photons bit for bit and the same step counts,
in another order."""
import ctypes as C

import numpy as np
import pytest

from realcausticsengine_gb300 import _native, abi, scenes
from realcausticsengine_gb300.session import Renderer

pytestmark = pytest.mark.gpu


def _canonical(a):
    w = np.ascontiguousarray(a).view(np.uint32)
    return w[np.lexsort(w.T[::-1])]


def _both(sc, sampler, paths, chains, depth, seed, iteration):
    r = Renderer(sc, max_path_length=depth, photons_per_iter=paths, seed=seed)
    cfg = abi.RcConfig()
    _native.check(r.L.rc_default_config(C.byref(cfg)), "rc_default_config")
    cfg.max_path_length, cfg.photons_per_iter, cfg.seed, cfg.write_exr = depth, paths, seed, 0
    cfg.sampler, cfg.mlt_chains = sampler, chains
    _native.check(r.L.rc_set_config(C.byref(cfg)), "rc_set_config")
    try:
        return r.mlt_photons(0, iteration), r.mlt_photons(1, iteration)
    finally:
        r.release()


SAMPLERS = [pytest.param(abi.SAMPLER_HYBRID, id="hybrid"), pytest.param(abi.SAMPLER_PSSMLT, id="pssmlt")]


@pytest.mark.parametrize("sampler", SAMPLERS)
@pytest.mark.parametrize("paths,chains,depth", [
    (1, 1, 6), (5, 64, 6), (1000, 1, 8),          # one lane of a warp; more chains than paths
    (4099, 31, 8), (4099, 33, 12), (70001, 1000, 8),    # ragged warps, blocks and last chains
    (20000, 512, 0), (20000, 512, 1),             # paths of a segment or two
])
def test_chains_store_the_step_chains_photons(sampler, paths, chains, depth):
    sc = scenes.test_scene(32, 24, subdiv=2, rough_glass=True, dispersion=0.03)
    (a, a_steps), (b, b_steps) = _both(sc, sampler, paths, chains, depth, 9, 3)
    assert a_steps == b_steps and b_steps[1] > 0
    a, b = _canonical(a), _canonical(b)
    assert a.shape == b.shape and (a == b).all()
    assert len(b) > 0 or paths < 100 or depth < 2


@pytest.mark.parametrize("sampler", SAMPLERS)
@pytest.mark.parametrize("scene", ["gems", "water"])
def test_chains_of_other_scenes_store_the_step_chains_photons(sampler, scene):
    """Overlapping dispersive gems (long paths, many world leaves) and smooth water."""
    sc = scenes.gem_cluster(64, 36) if scene == "gems" else scenes.water_pool(64, 36, grid=40, roughness=0.0)
    (a, a_steps), (b, b_steps) = _both(sc, sampler, 1 << 17, 4096, 8, 5, 0)
    assert a_steps == b_steps
    a, b = _canonical(a), _canonical(b)
    assert len(b) > 1000 and a.shape == b.shape and (a == b).all()
