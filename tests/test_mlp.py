"""The learned emission proposal's MLP on the tensor cores (tcgen05, BF16 operands,
FP32 accumulation) against a NumPy model.

* forward: the NumPy model rounds the encoded input, the weights and every hidden
  activation to BF16 exactly where the kernel does and accumulates in FP64; outputs
  agree within 2% of their scale (a hidden value that rounds to the other BF16
  neighbour moves the result by about one BF16 ulp, 0.4%).
* gradients: analytic FP64 backward of the weighted mixture negative log-likelihood
  on the same BF16-rounded weights and inputs; the kernel's gradient vector agrees to
  cosine similarity > 0.999 and relative error < 3% per layer (its activation
  gradients are BF16).
* training: Adam on a fixed batch lowers the loss.
"""
import ctypes as C

import numpy as np
import pytest

from realcausticsengine_gb300 import _native

pytestmark = pytest.mark.gpu

IN, IN_REAL, HID, OUT, LOBES, FREQS, ALPHA = 80, 75, 64, 80, 16, 12, 0.2
DIMS = [(IN, HID), (HID, HID), (HID, HID), (HID, OUT)]


def bf16(x):
    u = np.ascontiguousarray(x, np.float32).view(np.uint32)
    r = ((u + 0x7FFF + ((u >> 16) & 1)) >> 16) << 16
    return r.astype(np.uint32).view(np.float32).astype(np.float64)


def encode(pos):
    cols = []
    for i in range(3):
        c = pos[:, i].astype(np.float32)
        cols.append(c.astype(np.float64))
        f = 1.0
        for _ in range(FREQS):
            cols.append(np.sin(np.pi * f * c.astype(np.float64)))
            cols.append(np.cos(np.pi * f * c.astype(np.float64)))
            f *= 2.0
    x = np.stack(cols, 1)
    return np.concatenate([x, np.zeros((len(pos), IN - IN_REAL))], 1)


def init_params(rng):
    ps = []
    for l, (i, o) in enumerate(DIMS):
        real = IN_REAL if l == 0 else i
        W = np.zeros((o, i), np.float32)
        W[:, :real] = rng.uniform(-1, 1, (o, real)) * np.sqrt(6.0 / (real + o))
        b = (rng.normal(size=o) * 0.1).astype(np.float32)
        ps.append((W, b))
    return ps


def pack(ps):
    return np.concatenate([np.concatenate([W.reshape(-1), b]) for W, b in ps]).astype(np.float32)


def unpack(flat):
    out, o = [], 0
    for i, n in DIMS:
        W = flat[o:o + i * n].reshape(n, i); o += i * n
        b = flat[o:o + n]; o += n
        out.append((W, b))
    return out


def forward_np(ps, pos):
    x = bf16(encode(pos))
    acts = [x]
    for l, (W, b) in enumerate(ps):
        z = x @ bf16(W).T + b.astype(np.float64)
        if l < 3:
            x = bf16(np.maximum(z, 0.0))
            acts.append(x)
        else:
            return z, acts


def softplus(v):
    return np.where(v > 20, v, np.log1p(np.exp(np.minimum(v, 20))))


def loss_and_dout(out, d, w, pl):
    n = len(out)
    o = out.reshape(n, LOBES, 5)
    lg = o[:, :, 0]
    pi = np.exp(lg - lg.max(1, keepdims=True)); pi /= pi.sum(1, keepdims=True)
    r = o[:, :, 1:4]
    rl = np.maximum(np.linalg.norm(r, axis=2), 1e-6)
    mu = r / rl[..., None]
    raw = o[:, :, 4]
    kap = np.minimum(0.1 + softplus(raw), 2000.0)
    ca = (mu * d[:, None, :]).sum(2)
    vmf = kap / (2 * np.pi * (1 - np.exp(-2 * kap))) * np.exp(kap * (ca - 1))
    s = pi * vmf
    S = s.sum(1)
    q = np.maximum(ALPHA * pl + (1 - ALPHA) * S, 1e-20)
    loss = np.sum(-w * np.log(q)) / n
    c = -(1 - ALPHA) * w / (q * n)
    g = np.zeros_like(o)
    g[:, :, 0] = c[:, None] * (s - pi * S[:, None])
    gm = c[:, None] * s * kap / rl
    g[:, :, 1:4] = gm[..., None] * (d[:, None, :] - ca[..., None] * mu)
    e2 = np.exp(-2 * kap)
    dlog = 1 / kap - 2 * e2 / (1 - e2) + (ca - 1)
    dk = np.where(kap >= 2000.0, 0.0, 1 / (1 + np.exp(-raw)))
    g[:, :, 4] = c[:, None] * s * dlog * dk
    return loss, g.reshape(n, OUT)


def backward_np(ps, acts, dout):
    grads = [None] * 4
    dy = dout
    for l in range(3, -1, -1):
        W, b = ps[l]
        grads[l] = (dy.T @ acts[l], dy.sum(0))
        if l > 0:
            dx = dy @ bf16(W)
            dy = dx * (acts[l] > 0)
    return grads


def batch(rng, n):
    pos = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    # target directions: a lobe around -z tilted with position, plus noise
    d = np.stack([0.6 * (pos[:, 0] - 0.5), 0.6 * (pos[:, 1] - 0.5), -np.ones(n)], 1)
    d += 0.15 * rng.normal(size=d.shape)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    w = rng.uniform(0.5, 1.5, n)
    pl = np.maximum(-d[:, 2], 0) / np.pi            # cosine density about -z
    pos4 = np.concatenate([pos, pl[:, None]], 1).astype(np.float32)
    dir4 = np.concatenate([d, w[:, None]], 1).astype(np.float32)
    return pos4, dir4


def lib():
    L = _native.lib()
    L.rc_mlp_param_count.restype = C.c_int
    L.rc_mlp_forward_test.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_void_p]
    L.rc_mlp_grad_test.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p]
    L.rc_mlp_train_test.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_float, C.c_void_p,
                                    C.c_void_p]
    return L


def test_mlp_forward_matches_numpy():
    L = lib()
    rng = np.random.default_rng(0)
    ps = init_params(rng)
    flat = pack(ps)
    assert L.rc_mlp_param_count() == len(flat)
    n = 1000
    pos4, _ = batch(rng, n)
    out = np.zeros((n, OUT), np.float32)
    assert L.rc_mlp_forward_test(n, flat.ctypes.data, pos4.ctypes.data, out.ctypes.data) == 0
    want, _ = forward_np(ps, pos4[:, :3])
    scale = np.abs(want).max()
    assert np.abs(out - want).max() < 0.02 * scale


def test_mlp_gradients_match_fp64():
    L = lib()
    rng = np.random.default_rng(1)
    ps = init_params(rng)
    flat = pack(ps)
    n = 4096
    pos4, dir4 = batch(rng, n)
    grads = np.zeros_like(flat)
    loss = np.zeros(1, np.float32)
    assert L.rc_mlp_grad_test(n, flat.ctypes.data, pos4.ctypes.data, dir4.ctypes.data, grads.ctypes.data,
                              loss.ctypes.data) == 0
    out, acts = forward_np(ps, pos4[:, :3])
    want_loss, dout = loss_and_dout(out, dir4[:, :3].astype(np.float64), dir4[:, 3].astype(np.float64),
                                    pos4[:, 3].astype(np.float64))
    assert abs(loss[0] - want_loss) < 1e-3 * abs(want_loss) + 1e-4
    gw = unpack(grads)
    want = backward_np(ps, acts, dout)
    for l in range(4):
        for a, b in ((gw[l][0], want[l][0]), (gw[l][1], want[l][1])):
            a = a.astype(np.float64).reshape(-1)
            b = b.reshape(-1)
            cos = a @ b / (np.linalg.norm(a) * np.linalg.norm(b) + 1e-30)
            rel = np.linalg.norm(a - b) / (np.linalg.norm(b) + 1e-30)
            assert cos > 0.999 and rel < 0.03, (l, cos, rel)


@pytest.mark.parametrize("n", [1, 64, 127, 128, 129, 152 * 128, 152 * 128 + 1])
def test_mlp_gradients_at_tile_edges(n):
    """Rows of weight zero change nothing: twice the gradients of a batch of 2 n rows whose
    second half weighs nothing are those of its first half.  1 / n against 1 / (2 n) is an
    exact power of two and every row's products are the same, so only the order of FP32 sums
    differs: at most 128 partial sums of 19,457 rows, 1e-5 of each layer's norm.  The first
    half agrees with the FP64 model where rows enough average its BF16 roundings."""
    L = lib()
    rng = np.random.default_rng(3)
    ps = init_params(rng)
    flat = pack(ps)
    pos4, dir4 = batch(rng, 2 * n)
    dir4[n:, 3] = 0.0
    grads, losses = [], []
    for m in (n, 2 * n):
        g, loss = np.zeros_like(flat), np.zeros(1, np.float32)
        assert L.rc_mlp_grad_test(m, flat.ctypes.data, pos4.ctypes.data, dir4.ctypes.data, g.ctypes.data,
                                  loss.ctypes.data) == 0
        grads.append(g)
        losses.append(float(loss[0]))
    assert abs(losses[0] - 2 * losses[1]) <= 1e-5 * abs(losses[0])
    for a, b in zip(unpack(grads[0]), unpack(grads[1])):
        for x, y in zip(a, b):
            assert np.linalg.norm(x) > 0
            assert np.linalg.norm(x - 2 * y) <= 1e-5 * np.linalg.norm(x)
    if n >= 4096:
        out, acts = forward_np(ps, pos4[:n, :3])
        _, dout = loss_and_dout(out, *(dir4[:n, :3].astype(np.float64), dir4[:n, 3].astype(np.float64),
                                       pos4[:n, 3].astype(np.float64)))
        for a, b in zip(unpack(grads[0]), backward_np(ps, acts, dout)):
            for x, y in zip(a, b):
                assert np.linalg.norm(x - y) < 0.03 * np.linalg.norm(y)


def test_mlp_training_lowers_loss():
    L = lib()
    rng = np.random.default_rng(2)
    flat = pack(init_params(rng))
    n, steps = 8192, 150
    pos4, dir4 = batch(rng, n)
    losses = np.zeros(steps, np.float32)
    out = np.zeros_like(flat)
    assert L.rc_mlp_train_test(n, flat.ctypes.data, pos4.ctypes.data, dir4.ctypes.data, steps, C.c_float(3e-3),
                               losses.ctypes.data, out.ctypes.data) == 0
    assert np.isfinite(losses).all()
    assert losses[-10:].mean() < losses[0] - 0.5, (losses[0], losses[-10:].mean())
