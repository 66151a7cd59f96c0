"""Copies between host arrays and the device: pageable ones go through page-locked rings (csrc/host_copy.cuh)."""
import ctypes as C
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture()
def dev():
    from grilly_next import cabi
    with cabi.Device(0) as d:
        yield d


def host(dev, n, pinned, fill=0):
    """n bytes of host memory and what gives them back."""
    if not pinned:
        return np.full(n, fill, np.uint8), lambda: None
    p = C.c_void_p()
    assert dev.L.grl_host_alloc(C.c_size_t(n), C.byref(p)) == 0
    a = np.frombuffer((C.c_uint8 * n).from_address(p.value), np.uint8)
    a[:] = fill
    return a, lambda: dev.L.grl_host_free(p)


def slow_kernels(dev, buf, n):
    """n products of 2048^3 (a quarter of a millisecond or more each) on the handle's stream; buf holds 3 * 16 MiB."""
    from grilly_next import cabi
    x, y, z = (C.c_void_p(buf.value + i * (16 << 20)) for i in range(3))
    for _ in range(n):
        cabi.check(dev.L.grl_gemm_f32(dev.h, x, y, z, 2048, 2048, 2048))


def test_upload_does_not_wait_for_a_download_of_another_thread(dev):
    from grilly_next import cabi
    rng = np.random.default_rng(1)
    want_up, want_down = (rng.integers(0, 256, n, dtype=np.uint8) for n in (1 << 20, 4 << 20))
    scratch = dev.malloc(48 << 20)
    cabi.check(dev.L.grl_memset(dev.h, scratch, 0, 48 << 20))
    up, down = dev.upload(want_up * 0), dev.upload(want_down)
    got = np.zeros_like(want_down)
    dev.download(down, got.shape, np.uint8)              # both rings exist now
    slow_kernels(dev, scratch, 2)
    dev.sync()
    slow_kernels(dev, scratch, 600)                      # 150 ms at least
    done = {}

    def download():
        done["rc"] = dev.L.grl_memcpy_d2h(dev.h, got.ctypes.data, down, got.nbytes)
        done["down"] = time.perf_counter()

    t = threading.Thread(target=download)
    t.start()
    time.sleep(0.02)
    cabi.check(dev.L.grl_memcpy_h2d(dev.h, up, want_up.ctypes.data, want_up.nbytes))
    done["up"] = time.perf_counter()
    t.join()
    cabi.check(done["rc"])
    dev.sync()
    assert np.array_equal(got, want_down)
    assert np.array_equal(dev.download(up, want_up.shape, np.uint8), want_up)
    assert done["up"] < done["down"] - 0.05, done


def test_threads_copy_through_one_handle(dev):
    from grilly_next import cabi
    rng = np.random.default_rng(2)
    sizes = (9 * (1 << 20) + 13, 3 * (1 << 20) + 4097, (1 << 20) + 1, 700001)
    bufs = [dev.malloc(n) for n in sizes]
    wrong = []

    def work(i, seed):
        r = np.random.default_rng(seed)
        for _ in range(6):
            a, b = r.integers(0, 256, sizes[i], dtype=np.uint8), np.zeros(sizes[i], np.uint8)
            cabi.check(dev.L.grl_memcpy_h2d(dev.h, bufs[i], a.ctypes.data, a.nbytes))
            cabi.check(dev.L.grl_memcpy_d2h(dev.h, b.ctypes.data, bufs[i], b.nbytes))
            if not np.array_equal(a, b):
                wrong.append(i)

    ts = [threading.Thread(target=work, args=(i, int(rng.integers(1 << 30)))) for i in range(len(sizes))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    dev.sync()
    assert not wrong


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("part,parts,short", [
    (3 << 20, 4, 1 << 20),       # parts longer than a staging piece, the last one short
    (300_000, 5, 17),            # shorter than a piece, not aligned
    (1000, 3, 0),                # too small for the ring
    (1 << 20, 3, 1 << 20)])      # a part with nothing left to copy
def test_download_in_parts_waits_for_each_part(dev, pinned, part, parts, short):
    from grilly_next import cabi
    n = part * parts - short
    want = np.random.default_rng(part).integers(1, 256, n, dtype=np.uint8)
    made, src, scratch = dev.upload(want), dev.malloc(n), dev.malloc(48 << 20)
    cabi.check(dev.L.grl_memset(dev.h, src, 0, n))
    cabi.check(dev.L.grl_memset(dev.h, scratch, 0, 48 << 20))
    dev.sync()
    got, free = host(dev, n, pinned)
    events = []
    with cabi.Device(0) as down:
        for i in range(parts):       # a part is made behind a few slow kernels: one that is copied too early reads zeros
            off, m = i * part, min(part, max(0, n - i * part))
            slow_kernels(dev, scratch, 8)
            if m:
                cabi.check(dev.L.grl_memcpy_d2d(dev.h, C.c_void_p(src.value + off), C.c_void_p(made.value + off), m))
            events.append(dev.event())
            dev.record(events[-1])
        ev = (C.c_void_p * parts)(*[e.value for e in events])
        cabi.check(dev.L.grl_memcpy_d2h_parts(down.h, got.ctypes.data, src, n, ev, parts, part))
        if pinned:
            down.sync()
        assert np.array_equal(got, want)
        dev.sync()
        bad = (C.c_void_p * 65)(*[events[0].value] * 65)
        for args in ((ev, 0, part), (bad, 65, part), (ev, parts, part - short // parts - 1), ((C.c_void_p * parts)(), parts, part), (ev, parts, 0)):
            with pytest.raises(cabi.GrlError):
                cabi.check(dev.L.grl_memcpy_d2h_parts(down.h, got.ctypes.data, src, n, *args))
        down.sync()
    for e in events:
        dev.L.grl_event_destroy(e)
    free()
