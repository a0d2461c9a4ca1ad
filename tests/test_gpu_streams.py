"""Explicit device-pointer calls are asynchronous: calls on several streams and
captured calls prepare their weights into memory that no other call touches."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

SHAPE = (2048, 16, 512, 2, 96)


def _set(bf, torch, shape, seed):
    """(dims, E, A, G, J of the exact kernel)."""
    d = bf.Dims(*shape)
    E = torch.empty(d.esize, dtype=torch.uint8, device="cuda")
    A = torch.empty(d.asize, dtype=torch.uint8, device="cuda")
    bf.fill_random_device(E, seed, 0)
    bf.fill_random_device(A, seed, 1)
    G = torch.from_numpy(bf.gains(d)).cuda() * (1.0 + seed % 3)
    return d, E, A, G, _exact(bf, torch, d, E, A, G)


def _exact(bf, torch, d, E, A, G):
    J = torch.empty(d.jsize, dtype=torch.uint8, device="cuda")
    bf.set_kernel("simt")
    try:
        bf.form_beams_ex(d, J, E, A, G)
        bf.stream_status()
    finally:
        bf.set_kernel("auto")
    return J


@pytest.mark.parametrize("shape", [SHAPE, (4096, 1, 512, 2, 128), (8192, 2, 256, 2, 16)])
def test_calls_on_streams_do_not_share_weights(bflib, cuda, shape):
    sets = [_set(bflib, cuda, shape, k) for k in range(3)]
    streams = [cuda.cuda.Stream() for _ in sets]
    cuda.cuda.synchronize()
    out = []
    for _ in range(20):
        for (d, E, A, G, want), s in zip(sets, streams):
            with cuda.cuda.stream(s):
                J = cuda.empty(d.jsize, dtype=cuda.uint8, device="cuda")
                bflib.form_beams_ex(d, J, E, A, G, stream=s)
            assert bflib.last_kernel() == "tensor"
            out.append((J, want))
    cuda.cuda.synchronize()
    bflib.stream_status()
    for J, want in out:
        assert cuda.equal(J, want)


def _capture(bf, torch, d, E, A, G):
    J = torch.zeros(d.jsize, dtype=torch.uint8, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        bf.form_beams_ex(d, J, E, A, G)
        assert bf.last_kernel() == "tensor"
    return g, J


def test_captured_calls_keep_their_scratch(bflib, cuda):
    """Replays beside larger and other calls, with the graph's inputs changed, and
    after other graphs are gone."""
    d, E, A, G, want = _set(bflib, cuda, SHAPE, 1)
    big = _set(bflib, cuda, (1024, 32, 1024, 2, 256), 2)
    gone, _ = _capture(bflib, cuda, d, E, A, G)
    g, J = _capture(bflib, cuda, d, E, A, G)
    other = _set(bflib, cuda, SHAPE, 3)
    g2, J2 = _capture(bflib, cuda, *other[:4])
    del gone
    s1, s2 = cuda.cuda.Stream(), cuda.cuda.Stream()
    cuda.cuda.synchronize()
    Jb = cuda.empty(big[0].jsize, dtype=cuda.uint8, device="cuda")
    for rep in range(6):
        if rep == 3:  # new voltages and weights in the captured buffers
            bflib.fill_random_device(E, 9, 0)
            bflib.fill_random_device(A, 9, 1)
            want = _exact(bflib, cuda, d, E, A, G)
        J.zero_(), J2.zero_(), Jb.zero_()
        cuda.cuda.synchronize()
        with cuda.cuda.stream(s1):
            g.replay()
        with cuda.cuda.stream(s2):
            g2.replay()
        bflib.form_beams_ex(big[0], Jb, *big[1:4])
        cuda.cuda.synchronize()
        bflib.stream_status()
        assert cuda.equal(J, want) and cuda.equal(J2, other[4]) and cuda.equal(Jb, big[4])


def test_capture_while_other_threads_call(bflib, cuda):
    """Calls on other threads go on, and their scratch grows, while this one captures
    in global mode; the capture survives them."""
    import threading

    d, E, A, G, want = _set(bflib, cuda, (512, 4, 512, 2, 96), 4)
    big = [_set(bflib, cuda, (256, 40 + 20 * k, 1024, 2, 200), 5 + k) for k in range(2)]
    s = cuda.cuda.Stream()
    Jb = [cuda.empty(x[0].jsize, dtype=cuda.uint8, device="cuda") for x in big]
    failed = []

    def call():
        try:
            for x, j in zip(big, Jb):
                bflib.form_beams_ex(x[0], j, *x[1:4], stream=s)
        except Exception as e:  # noqa: BLE001 - reported below
            failed.append(e)

    cuda.cuda.synchronize()
    J = cuda.zeros(d.jsize, dtype=cuda.uint8, device="cuda")
    g = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(g):
        bflib.form_beams_ex(d, J, E, A, G)
        th = threading.Thread(target=call)
        th.start()
        th.join()
        bflib.form_beams_ex(d, J, E, A, G)
    assert not failed
    g.replay()
    cuda.cuda.synchronize()
    assert cuda.equal(J, want)
    for x, j in zip(big, Jb):
        assert cuda.equal(j, x[4])


def test_odd_resident_calls_while_another_thread_captures(bflib, cuda):
    """A call on a shape that takes the padded copy needs new scratch: neither it nor
    the other thread's capture, in global mode, is lost."""
    import threading

    T, F, D, B = 3001, 12, 253, 45
    d, E, A, G, want = _set(bflib, cuda, (T, F, D, 2, B), 11)
    W = bflib.ResidentWeights(F, B, D, A, G)
    s = cuda.cuda.Stream()
    J = cuda.empty(d.jsize, dtype=cuda.uint8, device="cuda")
    x = cuda.ones(64, device="cuda")
    failed = []

    def call():
        try:
            W.form_beams(J, E, T, stream=s)
            if bflib.last_kernel() != "tensor":
                failed.append(bflib.last_kernel())
        except Exception as e:  # noqa: BLE001 - reported below
            failed.append(e)

    cuda.cuda.synchronize()
    g = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(g):
        y = x + 1
        th = threading.Thread(target=call)
        th.start()
        th.join()
        y = y + 1
    assert not failed
    g.replay()
    cuda.cuda.synchronize()
    assert cuda.equal(J, want) and bool((y == 3).all())


def test_odd_resident_calls_wait_for_no_other_thread(bflib, cuda):
    """A checked call holds the device's lock until its stream is through (here for as
    long as a stalled launch takes to give up, 1.5 s); a call on resident weights has
    no use for the lock, whichever kernel takes its shape."""
    import threading
    import time

    T, F, D, B = 201, 2, 61, 9
    d, E, A, G, want = _set(bflib, cuda, (T, F, D, 2, B), 12)
    W = bflib.ResidentWeights(F, B, D, A, G)
    J = cuda.empty(d.jsize, dtype=cuda.uint8, device="cuda")
    d2, E2, A2, G2, _ = _set(bflib, cuda, (64, 1, 64, 2, 40), 13)
    J2 = cuda.empty(d2.jsize, dtype=cuda.uint8, device="cuda")
    s1, s2 = cuda.cuda.Stream(), cuda.cuda.Stream()
    W.form_beams(J, E, T, stream=s2)
    cuda.cuda.synchronize()
    status = []

    def stalled():
        try:
            bflib.form_beams_adler(d2, J2, E2, A2, G2, stream=s1)
            status.append(bflib.OK)
        except bflib.BeamformError as e:
            status.append(e.status)

    bflib.lib().bf_set_test_stall(1)
    th = threading.Thread(target=stalled)
    try:
        th.start()
        time.sleep(0.3)  # the stalled launch is queued, its call waits
    finally:
        bflib.lib().bf_set_test_stall(0)
    t0 = time.monotonic()
    W.form_beams(J, E, T, stream=s2)
    took = time.monotonic() - t0
    assert th.is_alive()
    th.join()
    assert status == [bflib.ERR_DEVICE_TIMEOUT]
    assert bflib.last_kernel() == "simt" and took < 0.3, took
    cuda.cuda.synchronize()
    assert cuda.equal(J, want)


def test_threads_that_end_wait_for_no_other_stream(bflib, cuda):
    """A thread whose only call reads the status of an idle stream is not held up by
    another stream's work (a stalled launch, which gives up after 1.5 s), neither in
    the call nor at its end."""
    import ctypes
    import time

    d, E, A, G, _ = _set(bflib, cuda, (64, 1, 64, 2, 40), 14)
    J = cuda.empty(d.jsize, dtype=cuda.uint8, device="cuda")
    s1, s2 = cuda.cuda.Stream(), cuda.cuda.Stream()
    libc = ctypes.CDLL(None)
    libc.pthread_create.argtypes = [ctypes.POINTER(ctypes.c_void_p)] + 3 * [ctypes.c_void_p]
    libc.pthread_join.argtypes = [ctypes.c_void_p, ctypes.POINTER(ctypes.c_void_p)]
    status = ctypes.cast(bflib.lib().bf_stream_status, ctypes.c_void_p)  # int (void *), as a thread's function
    bflib.stream_status(s2)
    bflib.lib().bf_set_test_stall(1)
    try:
        bflib.form_beams_ex(d, J, E, A, G, stream=s1)
    finally:
        bflib.lib().bf_set_test_stall(0)
    t0 = time.monotonic()
    tid, out = ctypes.c_void_p(), ctypes.c_void_p()
    assert libc.pthread_create(ctypes.byref(tid), None, status, s2.cuda_stream) == 0
    assert libc.pthread_join(tid, ctypes.byref(out)) == 0
    took = time.monotonic() - t0
    with pytest.raises(bflib.BeamformError):
        bflib.stream_status(s1)
    assert (out.value or 0) & 0xFFFFFFFF == bflib.OK and took < 0.3, took


def test_more_streams_than_keep_memory_and_calls_of_other_sizes(bflib, cuda):
    """Seven streams (the first four that call keep their memory), each with calls that
    need more, less and more again than the one before; in place and through the
    padded copy."""
    shapes = [(512, 4, 512, 2, 40), (1024, 8, 1024, 2, 130), (1001, 9, 250, 2, 45), (2048, 16, 512, 2, 96)]
    sets = [_set(bflib, cuda, shape, 20 + k) for k, shape in enumerate(shapes)]
    streams = [cuda.cuda.Stream() for _ in range(7)]
    cuda.cuda.synchronize()
    out = []
    for rep in range(8):
        for k, s in enumerate(streams):
            d, E, A, G, want = sets[(rep * 3 + k) % len(sets)]
            with cuda.cuda.stream(s):
                J = cuda.empty(d.jsize, dtype=cuda.uint8, device="cuda")
                bflib.form_beams_ex(d, J, E, A, G, stream=s)
            assert bflib.last_kernel() == "tensor"
            out.append((J, want))
    cuda.cuda.synchronize()
    bflib.stream_status()
    for J, want in out:
        assert cuda.equal(J, want)


def test_threads_on_one_stream(bflib, cuda):
    """Threads whose calls (resident weights on an odd shape, and weights with the call)
    meet on one stream: each has its scratch to itself until its launches are queued."""
    import threading

    T, F, D, B = 1001, 9, 250, 45
    sets = [_set(bflib, cuda, (T, F, D, 2, B), 30 + k) for k in range(4)]
    W = [bflib.ResidentWeights(F, B, D, x[2], x[3]) for x in sets]
    s = cuda.cuda.Stream()
    J = [[cuda.empty(x[0].jsize, dtype=cuda.uint8, device="cuda") for _ in range(30)] for x in sets]
    cuda.cuda.synchronize()
    failed = []

    def call(k):
        d, E, A, G, _ = sets[k]
        try:
            for i, j in enumerate(J[k]):
                if (i + k) % 3:
                    W[k].form_beams(j, E, T, stream=s)
                else:
                    bflib.form_beams_ex(d, j, E, A, G, stream=s)
        except Exception as e:  # noqa: BLE001 - reported below
            failed.append(e)

    threads = [threading.Thread(target=call, args=(k,)) for k in range(len(sets))]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    cuda.cuda.synchronize()
    bflib.stream_status()
    assert not failed
    for x, js in zip(sets, J):
        for j in js:
            assert cuda.equal(j, x[4])
