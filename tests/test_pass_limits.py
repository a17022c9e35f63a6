"""Limits of the render passes' scratch: the gather's list of parked work."""
import numpy as np
import pytest

from realcausticsengine_gb300 import _native
from realcausticsengine_gb300.session import kd_query

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
