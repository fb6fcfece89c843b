"""Decode batches whose rows the kernels read and write in page-locked host memory (gmoe_moe's own buffer, the caller's in gmoe_forward_submit),
and the fused kernels between their layers, against the per-stage path that the oracle tests cover: the same bits, on the first call (plain
launches) and the following ones (graph replay)."""
import ctypes as C
import numpy as np
import pytest

from conftest import SEED, same_bits

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def synth(gpu):
    for L in (3, 4, 5, 6):
        gpu.synth_layer(SEED, L)


@pytest.fixture()
def g(gpu, synth):
    yield gpu
    gpu.keep_stages(True)


# 3/4: all weights in flight at once or not; 8/9, 64/65: top-8 inside the grouping, one CTA or eight; 32/33: its bit table; 128/129: four warps per CTA or eight; 208: the last on mma.sync; 96/97: rows in place or copied
@pytest.mark.parametrize("nb", [1, 2, 3, 4, 8, 9, 17, 32, 33, 64, 65, 96, 97, 128, 129, 208, 256])
def test_fused_decode_layers_equal_stages(nb, g, weights, clib):
    from maple_runtime_b200 import lib as ml
    x = weights.hidden(2100 + nb, nb)
    for bias in (None, ml.synth_zipf_bias(clib, 7)):
        g.keep_stages(True)
        want = x.copy(); g.forward(want, 3, 2, bias)
        want_y, _ = g.moe(3, x, bias)
        g.keep_stages(False)
        for call in range(3):
            y = x.copy(); g.forward(y, 3, 2, bias)
            assert same_bits(y, want), f"stack, call {call}"
            y, _ = g.moe(3, x, bias)
            assert same_bits(y, want_y), f"layer, call {call}"


@pytest.mark.parametrize("nl", [2, 3, 4])
@pytest.mark.parametrize("step", [0, 1])
def test_one_token_through_several_layers(nl, step, g, weights, clib):
    """The joint of two layers inside the next router's kernel: the hidden row alternates between two buffers."""
    from maple_runtime_b200 import lib as ml
    x = weights.hidden(2300, 1)
    clib.gmoe_set_step_order(step)
    try:
        for bias in (None, ml.synth_zipf_bias(clib, 7)):
            g.keep_stages(True)
            want = x.copy(); g.forward(want, 3, nl, bias)
            g.keep_stages(False)
            for call in range(3):
                y = x.copy(); g.forward(y, 3, nl, bias)
                assert same_bits(y, want), f"call {call}"
    finally:
        clib.gmoe_set_step_order(0)


@pytest.mark.parametrize("shift", [0, 1])
def test_streamed_decode_batches(shift, g, weights, clib):
    """Two batches outstanding, each from and to its own page-locked rows; shift: rows that are not 16-byte aligned take the copies."""
    nb = 40
    n = nb * 2048
    xs = [weights.hidden(2500 + k, nb) for k in range(4)]
    g.keep_stages(True)
    want = [x.copy() for x in xs]
    for w in want:
        g.forward(w, 3, 2)
    g.keep_stages(False)
    bufs = [clib.gmoe_pinned_alloc(n * 4 + 16) for _ in range(4)]
    arr = [np.frombuffer((C.c_float * (n + 4)).from_address(b), np.float32)[shift:shift + n].reshape(nb, 2048) for b in bufs]
    for r in range(2):
        for k in range(2):
            arr[k][:] = xs[2 * r + k]
            assert clib.gmoe_forward_submit(arr[k].ctypes.data, arr[2 + k].ctypes.data, nb, 3, 2, None) == 0
        for k in range(2):
            assert clib.gmoe_forward_wait() >= 0
            assert same_bits(arr[2 + k].copy(), want[2 * r + k])
    del arr
    for b in bufs:
        clib.gmoe_pinned_free(b)
