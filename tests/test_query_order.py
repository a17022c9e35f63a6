"""The gather's query orders: Morton for the shapes that keep a group's work in its warp,
Hilbert (as the photons) for the shapes that park."""
import numpy as np
import pytest

from realcausticsengine_gb300.session import gather_variants, query_order

pytestmark = pytest.mark.gpu

PARKING = (8, 9)


def _spread(v):
    v = v.astype(np.uint64)
    return sum(((v >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b) for b in range(10))


def _morton_order(q, r):
    """Stable order of the 30-bit Morton codes of the queries' cells in a 1024^3 grid over
    their box, in the kernel's FP32 operations."""
    f = np.float32
    lo, hi = q.min(0), q.max(0)
    bits = 10
    while bits < 20 and (hi - lo).max() > f(2) * f(r) * f(1 << bits):
        bits += 1
    cells = f(f(1 << bits) - f(0.01))
    ext = hi - lo
    scale = np.array([cells / e if e > 0 else f(0) for e in ext], f) * (f(1023.99) / cells)
    c = np.clip((q - lo) * scale, f(0), f(1023)).astype(np.uint32)
    return np.argsort(_spread(c[:, 0]) | (_spread(c[:, 1]) << np.uint64(1)) | (_spread(c[:, 2]) << np.uint64(2)), kind="stable")


@pytest.mark.parametrize("n", [1, 2, 33, 4096, 4097, 50001])
@pytest.mark.parametrize("radius", [0.5, 1e-5])
def test_shapes_without_parking_take_the_morton_order(n, radius):
    """Across a tile of the sort and its remainder, in a frame of 10 bits per axis and in a
    finer one; with duplicates and a flat axis too."""
    rng = np.random.default_rng(n)
    q = rng.normal(size=(n, 3)).astype(np.float32) * np.float32([3.0, 0.2, 1.0])
    q[::7] = q[0]
    for flat in (False, True):
        if flat:
            q[:, 2] = 1.25
        want = _morton_order(q, np.sqrt(np.float32(radius * radius)))
        for v in range(-1, gather_variants()):
            if v not in PARKING:
                assert (query_order(q, radius * radius, v) == want).all(), (v, flat)


@pytest.mark.parametrize("variant", PARKING)
@pytest.mark.parametrize("radius", [0.5, 1e-5])
def test_parking_shapes_take_the_hilbert_order(variant, radius):
    """Over a whole 16^3 grid, consecutive queries of the Hilbert order are neighbours."""
    g = np.stack(np.meshgrid(*[np.arange(16)] * 3, indexing="ij"), -1).reshape(-1, 3)
    # (cell centres, with the box's corners at the grid's ends)
    q = np.random.default_rng(1).permutation(g)
    p = (q + 0.5).astype(np.float32)
    p = np.concatenate([p, np.float32([[0, 0, 0], [16, 16, 16]])])
    order = query_order(p, radius * radius, variant)
    assert (np.sort(order) == np.arange(len(p))).all()
    cells = q[order[order < len(q)]]
    assert (np.abs(np.diff(cells, axis=0)).sum(1) == 1).all()
