"""The gather's list of parked work at any length: what does not fit is done where it was
found, and a render's list holds what a dense focus parks."""
import numpy as np
import pytest

from realcausticsengine_gb300 import _native
from realcausticsengine_gb300.session import kd_query

pytestmark = pytest.mark.gpu

RENDER_LIST = (1 << 20) - 1


@pytest.fixture
def limit():
    L = _native.lib()
    yield lambda n: L.rc_gather_parked_limit(n)
    L.rc_gather_parked_limit(65535)


@pytest.mark.parametrize("variant", [8, 9])
@pytest.mark.parametrize("items", [1, 17, 4096, 65535, RENDER_LIST])
def test_photon_sets_do_not_depend_on_the_list(variant, items, limit):
    """A focus of 4,000 photons over a floor of 4,000, ragged groups: the sets of a shape
    that does not park."""
    rng = np.random.default_rng(7)
    p = np.concatenate([rng.normal(scale=0.03, size=(4000, 3)), rng.uniform(-1, 1, size=(4000, 3))]).astype(np.float32)
    q = np.concatenate([rng.normal(scale=0.03, size=(1003, 3)), rng.uniform(-1, 1, size=(2002, 3))]).astype(np.float32)
    want, want_ids = kd_query(p, q, 0.01, variant=5)
    assert limit(items) == 0
    got, ids = kd_query(p, q, 0.01, variant=variant)
    assert (got == want).all()
    assert all((np.sort(a) == np.sort(b)).all() for a, b in zip(ids, want_ids))


def test_a_renders_list_holds_a_dense_focus(limit):
    """53,600 queries that all accept all of 20,000 photons (1,024 chunks): a group of 32
    parks its last two levels of the tree, 526 items, where a list of 65,535 was full after
    125 of the 1,675 groups and left the others' photons to a warp each."""
    rng = np.random.default_rng(9)
    p = rng.normal(scale=0.05, size=(20000, 3)).astype(np.float32)
    q = rng.normal(scale=0.05, size=(53600, 3)).astype(np.float32)
    asked = {}
    for items in (65535, RENDER_LIST):
        assert limit(items) == 0
        counts, _ = kd_query(p, q, 4.0, with_indices=False, variant=9)
        assert (counts == len(p)).all()
        asked[items] = _native.lib().rc_gather_parked_items()
    assert asked[65535] >= 65535
    assert 1675 * 32 <= asked[RENDER_LIST] <= RENDER_LIST


def test_list_lengths_out_of_range_are_refused(limit):
    for items in (-1, 0, RENDER_LIST + 1):
        assert limit(items) != 0
