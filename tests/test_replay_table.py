"""Which captured layer loops are kept (csrc/replay.c), driven as csrc/gpre_api.c drives it: a new key runs plainly and asks for a slot, the second sight
captures, later ones replay."""
import ctypes as C
import random

import pytest

LAYERS, STACKS, IDLE = 2304, 256, 4 * 2560


class Key(C.Structure):
    _fields_ = [(n, C.c_int) for n in ("nb", "l0", "nl", "bias", "path", "prof", "ep")]


class Slot(C.Structure):
    _fields_ = [("key", Key), ("next", C.c_int), ("tried", C.c_int), ("launches", C.c_long), ("used", C.c_uint64), ("exec", C.c_void_p)]


DESTROY = C.CFUNCTYPE(None, C.c_void_p)


class Host:
    def __init__(self, clib):
        self.lib, self.live, self.destroyed, self.made = clib, {}, [], 0
        clib.replay_find.restype = clib.replay_admit.restype = C.POINTER(Slot)
        clib.replay_find.argtypes = [C.POINTER(Key)]
        clib.replay_admit.argtypes = [C.POINTER(Key), C.POINTER(C.c_void_p)]
        clib.replay_clear.argtypes = [DESTROY]
        self.clear()

    def clear(self):
        self.lib.replay_clear(DESTROY(self.destroyed.append))

    def call(self, nb, l0=0, nl=0, bias=0):
        """'plain', 'capture' or 'replay'"""
        k = Key(nb, l0, nl, bias, 0, 0, 0)
        s = self.lib.replay_find(k)
        if not s:
            gone = C.c_void_p(7)
            got = self.lib.replay_admit(k, gone)
            if gone.value:
                self.destroyed.append(gone.value)
            assert got or not gone.value
            return "plain"
        s = s.contents
        assert (s.key.nb, s.key.l0, s.key.nl, s.key.bias) == (nb, l0, nl, bias)
        if not s.exec:
            self.made += 1
            s.exec = self.made
            self.live[(nb, l0, nl, bias)] = self.made
            return "capture"
        assert s.exec == self.live[(nb, l0, nl, bias)]
        return "replay"


@pytest.fixture()
def host(clib):
    h = Host(clib)
    yield h
    h.clear()


def test_every_batch_size_of_a_decoding_server_is_replayed(host):
    keys = [(nb, layer) for nb in range(1, 97) for layer in range(24)]
    assert len(keys) == LAYERS
    assert {host.call(*k) for k in keys} == {"plain"} and {host.call(*k) for k in keys} == {"capture"}
    for _ in range(3):
        assert {host.call(*k) for k in keys} == {"replay"}
    assert not host.destroyed


def test_more_keys_than_slots(host):
    """In the same order every time: nothing that was captured leaves, most slots are in use, the other keys run plainly."""
    keys = [(nb, layer) for nb in range(1, 151) for layer in range(24)]
    for _ in range(15):
        got = [host.call(*k) for k in keys]
    assert not host.destroyed and got.count("replay") > 0.85 * LAYERS and got.count("capture") < 50


def test_keys_that_come_once_do_not_push_out_those_in_use(host):
    rng = random.Random(3)
    for i in range(30000):
        host.call(1000 + i, 0, 24)
        kind = host.call(rng.randrange(1, 25), 0, 24)
        if i > 2000:
            assert kind == "replay"
    assert not host.destroyed


def test_loops_that_nobody_asks_for_make_room(host):
    old, new = [(n, 0, 24) for n in range(1, STACKS + 1)], [(n, 1, 23) for n in range(1, 101)]
    for _ in range(2):
        for k in old:
            host.call(*k)
    for _ in range(IDLE // 100 + 12):
        got = [host.call(*k) for k in new]
    assert got.count("replay") > 95
    gone = set(host.destroyed)
    assert len(gone) == len(host.destroyed) >= 95 and gone <= {host.live[k + (0,)] for k in old}
    left = {v for v in host.live.values()} - gone
    host.destroyed.clear(); host.clear()
    assert set(host.destroyed) == left and not host.lib.replay_find(Key(1, 1, 23, 0, 0, 0, 0))
