"""The host side of the calls that take pageable buffers (csrc/hostio.c): the rows' int8 form against the reference statement of
tests/dense_ref.py, and the pool of helper threads."""
import ctypes as C
import numpy as np
import pytest

import dense_ref


def quant(clib, x):
    x = np.ascontiguousarray(x, np.float32)
    q = np.empty(x.shape, np.int8); qs = np.empty(len(x), np.float32); qsum = np.empty(len(x), np.int32)
    clib.hio_quant_rows.argtypes = [C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p]; clib.hio_quant_rows.restype = None
    clib.hio_quant_rows(x.ctypes.data, len(x), q.ctypes.data, qs.ctypes.data, qsum.ctypes.data)
    return q, qs, qsum


@pytest.mark.parametrize("scale", [1.0, 1e-30, 1e30, 3e-36])
def test_quant_rows_equal_reference_statement(clib, scale):
    rng = np.random.default_rng(3)
    x = (rng.standard_normal((33, 2048)) * scale).astype(np.float32)
    x[4] = 0.0; x[5] = x[6]; x[7, 100] = 50 * scale; x[8] = np.round(x[8] / scale) * np.float32(scale)
    x[9] = np.linspace(-127, 127, 2048) * scale                     # values on and next to rounding boundaries
    q, qs, qsum = quant(clib, x)
    want, want_s = dense_ref.prep(x)
    assert np.array_equal(q, want) and np.array_equal(qs.view(np.uint32), want_s.view(np.uint32)) and np.array_equal(qsum, want.sum(1))


def test_quant_rows_without_a_finite_scale(clib):
    """Rows whose maximum has no finite reciprocal scale, or that hold a NaN or an infinity: the device's conversion rules (saturate, NaN -> 0)."""
    x = np.zeros((3, 2048), np.float32)
    x[0, :2] = (1e-44, -1e-44)                                       # scale rounds to zero, 1 / 0 = inf
    x[1, :3] = (np.nan, 2.0, -1.0)
    x[2, :3] = (np.inf, 5.0, -np.inf)
    q, qs, qsum = quant(clib, x)
    assert qs[0] == 0 and q[0, 0] == -1 and q[0, 1] == 0 and not q[0, 2:].any()
    assert q[1, 0] == 0 and q[1, 1] == 127 and q[1, 2] == -64 and qsum[1] == 63
    assert np.isinf(qs[2]) and not q[2].any() and qsum[2] == 0


def test_pool_runs_every_piece_once(clib):
    fn_t = C.CFUNCTYPE(None, C.c_void_p, C.c_int)
    clib.hio_submit.argtypes = [fn_t, C.c_void_p, C.c_int]; clib.hio_submit.restype = C.c_uint
    clib.hio_wait.argtypes = [C.c_uint]; clib.hio_wait.restype = None
    clib.hio_done.argtypes = [C.c_uint]
    seen = np.zeros((200, 40), np.int64)
    keep, tickets = [], []
    for job in range(200):                                            # more jobs than the pool has slots
        def piece(arg, i, job=job):
            seen[job, i] += 1
        keep.append(fn_t(piece))
        tickets.append(clib.hio_submit(keep[-1], None, 1 + job % 40))
        if job % 7 == 0:
            clib.hio_wait(tickets[-1])
            assert clib.hio_done(tickets[-1]) == 1
    for t in tickets:
        clib.hio_wait(t)
    for job in range(200):
        assert (seen[job, :1 + job % 40] == 1).all() and not seen[job, 1 + job % 40:].any()


def test_helpers_sleep_when_the_work_is_done(clib):
    """Cores are the host's again after a call: what the process uses while its caller sleeps.  Three helpers that spun for 0.4 ms would use 1.2 ms."""
    import time
    a, b = np.zeros(1 << 22, np.uint8), np.zeros(1 << 22, np.uint8)
    clib.hio_copy_shared.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t]; clib.hio_copy_shared.restype = None
    used = []
    for _ in range(20):
        clib.hio_copy_shared(b.ctypes.data, a.ctypes.data, a.nbytes)
        t0 = time.process_time()
        time.sleep(0.005)
        used.append(time.process_time() - t0)
    assert sorted(used)[10] < 3e-4
