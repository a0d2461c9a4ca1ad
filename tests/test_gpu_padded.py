"""Shapes the tensor-core kernel does not take in place (times, dishes or
addresses that do not suit TMA, one polarization) run on it through the padded
copy when they are large enough: the bytes equal the exact dp4a kernel's (itself
checked against the oracle) and, where that is quick, the oracle's."""
from __future__ import annotations

import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(bf, torch, d, seed, e_off=0):
    E = torch.empty(d.esize + 16, dtype=torch.uint8, device="cuda")
    A = torch.empty(d.asize, dtype=torch.uint8, device="cuda")
    bf.fill_random_device(E, seed, 0)
    bf.fill_random_device(A, seed, 1)
    return E[e_off:e_off + d.esize], A, torch.from_numpy(bf.gains(d)).cuda()


def _run(bf, torch, d, E, A, G, kernel, want, j_off=0, j_layout="linear"):
    """J of one call, with guard bytes on both sides checked."""
    buf = torch.full((d.jsize + 64,), 0x5A, dtype=torch.uint8, device="cuda")
    J = buf[16 + j_off:16 + j_off + d.jsize]
    bf.set_kernel(kernel)
    try:
        bf.form_beams_layout(d, J, E, A, G, j_layout=j_layout)
        assert bf.last_kernel() == want
        bf.stream_status()
    finally:
        bf.set_kernel("auto")
    assert bool((buf[:16 + j_off] == 0x5A).all()) and bool((buf[16 + j_off + d.jsize:] == 0x5A).all())
    return J.clone()


# (t, f, d, p, b): times around multiples of 4, 64 and 128, dishes around
# multiples of 8 and 128 up to the largest, odd beams, several passes, widths of
# every layout, one polarization with even and odd times
SHAPES = [
    (1001, 9, 510, 2, 96), (1002, 9, 250, 2, 45), (1004, 9, 512, 2, 33), (1023, 5, 513, 2, 7), (257, 1, 2041, 2, 60),
    (2001, 3, 1017, 2, 200), (8000, 3, 505, 2, 16), (2049, 4, 385, 2, 97), (1001, 9, 510, 1, 96), (1000, 9, 512, 1, 40),
    (4003, 5, 391, 1, 12), (256, 1, 2047, 2, 1),
]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("j_layout", ["linear", "j2"])
def test_padded_equals_exact_kernel(bflib, cuda, shape, j_layout):
    d = bflib.Dims(*shape)
    E, A, G = _inputs(bflib, cuda, d, sum(shape))
    want = _run(bflib, cuda, d, E, A, G, "simt", "simt", j_layout=j_layout)
    got = _run(bflib, cuda, d, E, A, G, "auto", "tensor", j_layout=j_layout)
    assert cuda.equal(got, want)


@pytest.mark.parametrize("e_off,j_off", [(1, 0), (3, 2), (0, 1), (8, 4)])
@pytest.mark.parametrize("shape", [(1040, 9, 512, 2, 96), (1041, 9, 509, 2, 40), (1001, 9, 510, 1, 33)])
def test_padded_takes_any_alignment(bflib, cuda, shape, e_off, j_off):
    d = bflib.Dims(*shape)
    E, A, G = _inputs(bflib, cuda, d, 5 + e_off, e_off)
    want = _run(bflib, cuda, d, E, A, G, "simt", "simt", j_off)
    assert cuda.equal(_run(bflib, cuda, d, E, A, G, "auto", "tensor", j_off), want)


def test_padded_matches_oracle_with_checksum_and_huge_gains(bflib, cuda, oracle):
    d = bflib.Dims(515, 7, 389, 2, 37)
    E, A, G = _inputs(bflib, cuda, d, 3)
    G[:37] *= 1e30  # the narrowing requantisation of the first frequency
    J = cuda.empty(d.jsize, dtype=cuda.uint8, device="cuda")
    got = bflib.form_beams_adler(d, J, E, A, G)
    assert bflib.last_kernel() == "tensor"
    want = oracle.form_beams(oracle.Dims(515, 7, 389, 2, 37), E.cpu().numpy(), A.cpu().numpy(), G.cpu().numpy())
    np.testing.assert_array_equal(J.cpu().numpy(), want)
    assert got == zlib.adler32(want.tobytes())


@pytest.mark.parametrize("p,t", [(2, 2101), (1, 4303)])
def test_padded_chunks_of_times(bflib, cuda, p, t):
    """A copy of more than 256 MiB goes in chunks of times."""
    d = bflib.Dims(t, 64, 2041, p, 5)
    E, A, G = _inputs(bflib, cuda, d, 9)
    want = _run(bflib, cuda, d, E, A, G, "simt", "simt")
    assert cuda.equal(_run(bflib, cuda, d, E, A, G, "auto", "tensor"), want)


def test_padded_resident_weights_on_two_streams(bflib, cuda):
    """Calls on two streams share the scratch: each waits for the one before."""
    d = bflib.Dims(2001, 9, 509, 2, 64)
    s1, s2 = cuda.cuda.Stream(), cuda.cuda.Stream()
    sets = []
    for k, s in ((0, s1), (1, s2)):
        E, A, G = _inputs(bflib, cuda, d, 50 + k)
        W = bflib.ResidentWeights(9, 64, 509, A, G)
        sets.append((E, A, G, W, s, _run(bflib, cuda, d, E, A, G, "simt", "simt")))
    cuda.cuda.synchronize()
    out = []
    for rep in range(4):
        for E, A, G, W, s, want in sets:
            J = cuda.empty(d.jsize, dtype=cuda.uint8, device="cuda")
            with cuda.cuda.stream(s):
                if rep % 2:
                    W.form_beams(J, E, 2001, stream=s)
                else:
                    bflib.form_beams_ex(d, J, E, A, G, stream=s)
            assert bflib.last_kernel() == "tensor"
            out.append((J, want))
    cuda.cuda.synchronize()
    for J, want in out:
        assert cuda.equal(J, want)


def test_padded_shape_under_capture_runs_the_exact_kernel(bflib, cuda):
    """A graph cannot wait for the shared scratch, so a captured call keeps the dp4a kernel."""
    d = bflib.Dims(1001, 9, 250, 2, 45)
    E, A, G = _inputs(bflib, cuda, d, 77)
    want = _run(bflib, cuda, d, E, A, G, "simt", "simt")
    _run(bflib, cuda, d, E, A, G, "auto", "tensor")
    J = cuda.zeros(d.jsize, dtype=cuda.uint8, device="cuda")
    g = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(g):
        bflib.form_beams_ex(d, J, E, A, G)
        assert bflib.last_kernel() == "simt"
    g.replay()
    cuda.cuda.synchronize()
    assert cuda.equal(J, want)


# a few times, from 16; dishes just over the one chunk of 128 that the dp4a kernel keeps
SMALL = [(16, 1, 130, 2, 7), (16, 2, 200, 1, 33), (17, 3, 129, 1, 16), (18, 1, 2047, 1, 9), (19, 4, 433, 2, 42),
         (26, 3, 539, 1, 63), (63, 2, 131, 2, 97), (65, 1, 255, 1, 17), (80, 7, 192, 1, 20), (79, 14, 439, 2, 11),
         (127, 1, 260, 2, 128)]


@pytest.mark.parametrize("shape", SMALL)
@pytest.mark.parametrize("j_layout", ["linear", "j2"])
def test_padded_small_shapes_match_oracle(bflib, cuda, oracle, shape, j_layout):
    d = bflib.Dims(*shape)
    E, A, G = _inputs(bflib, cuda, d, 7 * sum(shape))
    got = _run(bflib, cuda, d, E, A, G, "auto", "tensor", j_off=1, j_layout=j_layout)
    od = oracle.Dims(*shape)
    want = oracle.form_beams(od, E.cpu().numpy(), A.cpu().numpy(), G.cpu().numpy())
    if j_layout == "j2":
        want = oracle.J_to_J2(od, want)
    np.testing.assert_array_equal(got.cpu().numpy(), want)
