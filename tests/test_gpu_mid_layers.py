"""Several layers at 161 to 511 tokens, where the combine of a layer and the norm of the next are one kernel on the compact down rows
(csrc/k_route.cu: edge_kernel<true>), against the same layers one call each, which the other tests compare with the oracle."""
import numpy as np
import pytest

from conftest import SEED, same_bits

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def stacks(gpu, weights):
    """Layers 0..2 as generated; layers 3 and 4 whose gate and up rows have one sign and one scale, which makes every SiLU output of a pair equal, so that
    down rows of all +1 (all -1) give dots of +-65024, past the compact rows' 16 bits."""
    from maple_runtime_b200 import lib as ml
    c = ml.CONST
    for L in range(3):
        gpu.synth_layer(SEED, L)
    router, post_ln, experts = weights.layer(2)
    ex = experts.copy().reshape(256, c.EXPERT_BYTES)
    for m in range(2):
        ex[:, m * c.GU_BYTES:m * c.GU_BYTES + c.GU_CODES] = 0xAA
        ex[:, m * c.GU_BYTES + c.GU_CODES:(m + 1) * c.GU_BYTES].view(np.float32)[:] = 0.02
    dn = ex[:, 2 * c.GU_BYTES:2 * c.GU_BYTES + c.GU_CODES].reshape(256, 2048, 128)
    dn[:, 0:300, :] = 0xAA
    dn[:, 300:640, :] = 0x00
    span = ml.page_aligned(ex.nbytes)
    span[:ex.nbytes] = ex.reshape(-1)
    rid = gpu.region(span)
    for L in (3, 4):
        gpu.set_layer(L, router, post_ln, ml.gloc_for_contiguous(0, slot=0), np.array([rid, -1, -1, -1], np.int32))


@pytest.mark.parametrize("nb", [161, 209, 301, 511])
@pytest.mark.parametrize("l0", [0, 2])
def test_layers_in_one_call_equal_layers_one_by_one(nb, l0, stacks, gpu, weights):
    g = gpu
    x = weights.hidden(900 + nb, nb)
    want = x.copy()
    for L in range(l0, l0 + 3):
        g.forward(want, L, 1)
    if l0 == 2:
        assert np.abs(g.peek("dn_dots", nb)).max() == 65024
    g.keep_stages(False)
    try:
        for _ in range(3):                      # plainly, while captured, as a replay
            got = x.copy()
            g.forward(got, l0, 3)
            assert same_bits(got, want)
    finally:
        g.keep_stages(True)


@pytest.mark.parametrize("nb", [48, 49, 104, 105, 160, 161, 208, 256, 257, 511, 512, 1152, 1153, 1307, 1308, 1536, 1537])
def test_where_the_expert_kernels_change(nb, stacks, gpu, weights):
    """Up to 48, 104 and 160 tokens the mma.sync down kernel takes one, two and four blocks of rows per CTA; from 161 the tcgen05 kernels run.  From 257 the pairs are placed by the
    kernel that moves their rows, from 512 two layers have no joint; up to 1152, 1307 and 1536 combine starts early, the tcgen05 kernels hand over blocks of 256 columns, SiLU starts
    early.  Either path alone and the one that the size chooses: the same bits."""
    g = gpu
    x = weights.hidden(950 + nb, nb)
    out = {}
    g.keep_stages(False)
    try:
        for path in (1, 2, 0):
            g.set_path(path)
            out[path] = x.copy()
            g.forward(out[path], 0, 3)
    finally:
        g.set_path(0)
        g.keep_stages(True)
    assert same_bits(out[0], out[1]) and same_bits(out[0], out[2])
