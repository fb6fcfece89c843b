"""Child of tests/test_gpu_large.py: a library set up for 16,384 tokens (one process has one set-up).  Prints one JSON line: check -> "ok" or what is wrong."""
import ctypes as C
import json
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
sys.path.insert(0, os.path.join(ROOT, "tests"))
from maple_runtime_b200 import lib as ml  # noqa: E402
from oracle import oracle as orc  # noqa: E402
from conftest import SEED, same_bits  # noqa: E402

MAXTOK, PART = 16384, 2048          # parts of 2048 tokens and fewer are what the other tests compare with the oracle
g = ml.Gpre(MAXTOK)
for layer in range(2):
    g.synth_layer(SEED, layer)
X = ml.synth_hidden(g.lib, SEED, 9000, MAXTOK)
ZIPF = ml.synth_zipf_bias(g.lib, 7)


def group(nb, kind):
    rng = np.random.default_rng(nb)
    p = None
    if kind == "skew":
        p = 1.0 / np.arange(1, 257) ** 1.2
    scores = rng.random((nb, 256)) ** (1.0 if p is None else (p.min() / p))
    top = np.argsort(-scores, axis=1)[:, :8].astype(np.int32)
    if kind == "same":
        top[:] = top[0]
    tw = rng.random((nb, 8)).astype(np.float32)
    nu, ue, ustart, utok, uw, tp = orc.Oracle().group(top, tw)
    g.poke("top", top.reshape(-1)); g.poke("topw", tw.reshape(-1))
    g.stage("group", 0, nb)
    assert int(g.peek("nu", nb)[0]) == nu
    assert np.array_equal(g.peek("ue", nb)[:nu], ue[:nu]) and np.array_equal(g.peek("ustart", nb)[:nu + 1], ustart[:nu + 1])
    assert np.array_equal(g.peek("utok", nb), utok) and np.array_equal(g.peek("tp", nb), tp) and same_bits(g.peek("uw", nb), uw)


def parts(x, bias):
    out = x.copy()
    for at in range(0, len(x), PART):
        piece = out[at:at + PART].copy()
        g.forward(piece, 0, 2, bias)
        out[at:at + PART] = piece
    return out


def router_of(nb):
    """A last part below 512 tokens takes the exact-order router by itself: the comparison then pins that one."""
    return 1 if 0 < nb % PART < 512 else 0


def stack(nb, router, bias):
    x = X[:nb]
    g.set_router(router)
    want = parts(x, bias)
    for call in range(3):           # plainly, while captured, as a replay
        got = x.copy()
        g.forward(got, 0, 2, bias)
        assert same_bits(got, want), "call %d: %d rows differ" % (call, (got != want).any(1).sum())


def layer_call(nb):
    g.set_router(1)
    x = X[:nb]
    want = np.concatenate([g.moe(1, x[at:at + PART], ZIPF)[0] for at in range(0, nb, PART)])
    assert same_bits(g.moe(1, x, ZIPF)[0], want)


def streamed(sizes):
    g.set_router(0)
    n = max(sizes) * 2048
    bufs = [g.lib.gmoe_pinned_alloc(n * 4) for _ in range(4)]
    arr = [np.frombuffer((C.c_float * n).from_address(b), np.float32) for b in bufs]
    at, out, want = 0, [], parts(X[:sum(sizes)], None)
    for i, nb in enumerate(sizes):
        if i >= 2:
            assert g.lib.gmoe_forward_wait() >= 0
            out.append(arr[2 + i % 2][:sizes[i - 2] * 2048].copy())
        arr[i % 2][:nb * 2048] = X[at:at + nb].reshape(-1)
        assert g.lib.gmoe_forward_submit(arr[i % 2].ctypes.data, arr[2 + i % 2].ctypes.data, nb, 0, 2, None) == 0
        at += nb
    for i in range(max(0, len(sizes) - 2), len(sizes)):
        assert g.lib.gmoe_forward_wait() >= 0
        out.append(arr[2 + i % 2][:sizes[i] * 2048].copy())
    del arr
    for b in bufs:
        g.lib.gmoe_pinned_free(b)
    assert same_bits(np.concatenate(out).reshape(-1, 2048), want)


def plugin(nb):
    rng = np.random.default_rng(nb)
    top = np.argsort(rng.random((nb, 256)), axis=1)[:, :8].astype(np.int32)
    tw = rng.random((nb, 8)).astype(np.float32)

    def call(a, b):
        nu, ue, ustart, utok, uw, tp = orc.Oracle().group(top[a:b], tw[a:b])
        loc = np.ascontiguousarray(ml.gloc_for_contiguous()[ue[:nu]])
        return g.gpre_moe(np.ascontiguousarray(X[a:b]), nu, loc, np.array([g.layer_region[0], -1, -1, -1], np.int32), ustart[:nu + 1].copy(), utok, uw, tp)[0]
    assert same_bits(call(0, nb), np.concatenate([call(at, min(at + PART, nb)) for at in range(0, nb, PART)]))


def attention(nb):
    rng = np.random.default_rng(nb)
    if not getattr(attention, "ready", False):
        for rows in (2048, 512, 512):
            g.dense_add(0, (rng.integers(0, 3, (rows, 512)) * 0x55).astype(np.uint8), rng.uniform(0.01, 0.05, rows).astype(np.float32), rows, 2048)
        g.dense_done(MAXTOK)
        angle = np.arange(MAXTOK)[:, None] * (10000.0 ** (-np.arange(32) / 32))[None, :]
        g.rope_table(np.stack([np.cos(angle), np.sin(angle)], -1))
        attention.ready = True
    pos, one = np.arange(nb, dtype=np.int32), np.ones(128, np.float32)
    qkv = g.dense(0, X[:nb], 3072)[0]
    got = g.qk_rope(qkv, pos, 0, one, one)
    for at in range(0, nb, PART):
        e = min(at + PART, nb)
        assert same_bits(g.dense(0, X[at:e], 3072)[0], qkv[at:e])
        for a, b in zip(got[:3], g.qk_rope(qkv[at:e], pos[at:e], 0, one, one)[:3]):
            assert same_bits(np.ascontiguousarray(a[at:e]), b)


CHECKS = {}
for nb in (2049, 3000, 4096, 4097, 8191, 16384):
    for kind in ("even", "skew", "same"):
        CHECKS["grouping of %d tokens, %s" % (nb, kind)] = (group, nb, kind)
for nb in (2049, 4096, 4097, 10000, 16384):
    CHECKS["stack of %d tokens" % nb] = (stack, nb, router_of(nb), None)
CHECKS["stack of 4096 tokens, exact-order router"] = (stack, 4096, 1, None)
CHECKS["stack of 16384 tokens, skewed"] = (stack, 16384, 0, ZIPF)
CHECKS["layer call of 5000 tokens"] = (layer_call, 5000)
CHECKS["streamed chunks of 4096 tokens"] = (streamed, (4096, 4096, 4096, 2048))
CHECKS["streamed chunks of 8192 tokens"] = (streamed, (8192, 8192))
CHECKS["plug-in call of 4096 tokens"] = (plugin, 4096)
CHECKS["plug-in call of 4999 tokens"] = (plugin, 4999)
CHECKS["attention sides of 4097 tokens"] = (attention, 4097)
CHECKS["attention sides of 16384 tokens"] = (attention, 16384)

if __name__ == "__main__":
    said = {}
    for name, (f, *args) in CHECKS.items():
        try:
            f(*args)
            said[name] = "ok"
        except (AssertionError, RuntimeError) as e:
            said[name] = "%s: %s" % (type(e).__name__, e)
    print(json.dumps(said))
