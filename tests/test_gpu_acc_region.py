"""The tcgen05 expert kernels keep the accumulators of two items in one region of tensor memory, even items at its low end and odd ones at its high end
(csrc/k_expert_umma.cu: acc_place).  Tile sizes around the MMA's steps of 16 and pairs of neighbours that do (and do not) fit the region together, against
the mma.sync kernels, which have no such region: the same bits."""
import numpy as np
import pytest

from conftest import SEED, same_bits

pytestmark = pytest.mark.gpu


def routing(nb, counts):
    """Eight distinct experts per token so that expert e gets counts[e] pairs: the tokens in turn take the experts with the most places left."""
    left = np.array(counts)
    assert left.sum() == nb * 8 and left.max() <= nb
    top = np.empty((nb, 8), np.int32)
    for t in range(nb):
        top[t] = np.argsort(-left, kind="stable")[:8]
        left[top[t]] -= 1
    assert (left == 0).all()
    return top


def spread(nb, cycle):
    """256 counts that repeat the given ones, the remainder shared out by ones."""
    c = np.minimum(np.resize(np.array(cycle), 256), nb)
    while c.sum() > nb * 8:
        c[np.flatnonzero(c > 1)[-1]] -= 1
    i = 0
    while c.sum() < nb * 8:
        c[i % 256] += c[i % 256] < nb
        i += 1
    return c


CASES = {
    "every step": (512, [1, 15, 16, 17, 31, 32, 33, 47, 48, 49, 2, 3]),                    # 1 row to 48 and over
    "64 and 80": (2048, [64, 65, 79, 80, 81, 63, 72]),                                    # neighbours fill the region exactly, or just do not fit it
    "96 and its neighbours": (1500, [96, 95, 97, 1, 96, 192, 193, 96, 16]),               # a full tile beside a full one, a full one beside one row
    "one popular expert": (700, [700] + [21] * 250),                                      # eight tiles of one expert in a row
}


@pytest.mark.parametrize("name", CASES)
def test_neighbouring_tiles(name, gpu):
    from maple_runtime_b200 import lib as ml
    g = gpu
    nb, cycle = CASES[name]
    g.synth_layer(SEED, 0)
    rng = np.random.default_rng(nb)
    top = routing(nb, spread(nb, cycle))
    flat = top.reshape(-1)
    order = np.argsort(flat, kind="stable")
    used, counts = np.unique(flat, return_counts=True)
    ustart = np.zeros(len(used) + 1, np.int32)
    ustart[1:] = np.cumsum(counts)
    place = np.empty(nb * 8, np.int32)
    place[order] = np.arange(nb * 8, dtype=np.int32)
    x = rng.standard_normal((nb, 2048)).astype(np.float32)
    args = (x, len(used), np.ascontiguousarray(ml.gloc_for_contiguous()[used]), np.array([g.layer_region[0], -1, -1, -1], np.int32), ustart,
            (order // 8).astype(np.int32), rng.random(nb * 8).astype(np.float32), np.sort(place.reshape(nb, 8), axis=1))
    def run(path, keep):                                     # keep: the kernels that also store their integer sums
        g.set_path(path)
        g.keep_stages(keep)
        try:
            return g.gpre_moe(*args)[0]
        finally:
            g.set_path(0)
            g.keep_stages(True)

    want = run(1, False)
    for keep in (False, True):
        assert same_bits(run(2, keep), want)
