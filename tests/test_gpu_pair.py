"""The kernel on pairs of SMs at the edges of its tiles and rings: tile counts that
leave the second half of a pair empty, fewer K stages than unpack groups, W
resident and streamed, beam passes of every padding, and the sums of the extreme
operands.  Every byte of J equals the oracle's."""
from __future__ import annotations

import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# fill bytes: random, the extreme values of E and A and all-zero nibbles
FILLS = [(None, None), (0xFF, 0x00), (0x00, 0x0F), (0xFF, 0xF0), (0x00, 0xFF)]

# (t, f, d, b).  Times: less than, exactly and just over one or two tiles of 64.
# Dishes: 1, 2, 3, 4, 8 and 16 K stages of 128, whole and partial.  Beams: N of
# 64 .. 192 with and without padding, signed codes (<= 64) and W + 8, several
# passes with a partial last one.
SHAPES = [
    (16, 1, 64, 96), (64, 3, 8, 72), (80, 3, 128, 96), (128, 2, 128, 17), (144, 2, 256, 88), (192, 9, 376, 65),
    (272, 1, 384, 64), (208, 2, 512, 41), (1040, 3, 512, 96), (528, 2, 1024, 200), (336, 2, 1024, 96), (272, 1, 2048, 96),
    (144, 1, 2048, 130), (80, 160, 128, 80),
    # two passes that share the unpacked operand and keep both W (and neighbours
    # that only keep W, or neither): ranges that start and end between the passes
    (16, 1, 512, 97), (528, 2, 512, 128), (8208, 3, 512, 128), (80, 160, 256, 112), (272, 50, 8, 104), (400, 77, 384, 120),
    (528, 20, 256, 192), (528, 20, 520, 128),
]


def _host_inputs(bf, d, seed, e_fill=None, a_fill=None):
    E, A, G = bf.seeded_host_inputs(d, seed)
    if e_fill is not None:
        E[:] = e_fill
        A[:] = a_fill
    return E, A, G


def _oracle_J(oracle, d, E, A, G, j_layout="linear"):
    od = oracle.Dims(d.ntimes, d.nfrequencies, d.ndishes, d.npolarizations, d.nbeams)
    J = oracle.form_beams(od, E, A, G)
    return oracle.J_to_J2(od, J) if j_layout == "j2" else J


@pytest.mark.parametrize("shape", SHAPES)
def test_pair_edges(bflib, cuda, oracle, shape):
    t, f, dd, b = shape
    d = bflib.Dims(t, f, dd, 2, b)
    E, A, G = _host_inputs(bflib, d, sum(shape))
    Ed, Ad, Gd = (cuda.from_numpy(x).cuda() for x in (E, A, G))
    J = cuda.full((d.jsize + 32,), 0x5A, dtype=cuda.uint8, device="cuda")
    for j_layout in ("linear", "j2"):
        want = _oracle_J(oracle, d, E, A, G, j_layout)
        J.fill_(0x5A)
        got = bflib.form_beams_adler(d, J[16:-16], Ed, Ad, Gd, j_layout=j_layout)
        assert bflib.last_kernel() == "tensor"
        np.testing.assert_array_equal(J[16:-16].cpu().numpy(), want)
        assert bool((J[:16] == 0x5A).all()) and bool((J[-16:] == 0x5A).all())
        assert got == zlib.adler32(want.tobytes())


@pytest.mark.parametrize("fill", FILLS[1:])
@pytest.mark.parametrize("shape", [(64, 1, 2048, 96), (64, 1, 2048, 33), (144, 1, 1000, 72)])
def test_pair_extreme_sums(bflib, cuda, oracle, shape, fill):
    """Gains of the order of 1 / raw keep the largest sums off the clamp."""
    t, f, dd, b = shape
    d = bflib.Dims(t, f, dd, 2, b)
    E, A, _ = _host_inputs(bflib, d, 0, *fill)
    E[::7] ^= 0x01
    G = (np.arange(1, f * b + 1, dtype=np.float32) / np.float32(f * b * 128 * dd / 7)).astype(np.float32)
    G[:b:5] *= np.float32(1e30)  # the narrowing requantisation
    Ed, Ad, Gd = (cuda.from_numpy(x).cuda() for x in (E, A, G))
    J = cuda.empty(d.jsize, dtype=cuda.uint8, device="cuda")
    bflib.form_beams_ex(d, J, Ed, Ad, Gd)
    assert bflib.last_kernel() == "tensor"
    bflib.stream_status()
    np.testing.assert_array_equal(J.cpu().numpy(), _oracle_J(oracle, d, E, A, G))


@pytest.mark.parametrize("wide", [True, False])
@pytest.mark.parametrize("dd", [64, 128, 384, 512, 2048])
def test_pair_batch_mixes_widths_and_weights(bflib, cuda, oracle, dd, wide):
    """One launch over problems of one and two passes, without and (wide) with
    weights of both forms."""
    probs = []
    for i, (t, b) in enumerate([(272, 96), (64, 16), (528, 64), (80, 128), (16, 72), (144, 41)]):
        if not wide and b in (96, 72):
            continue
        d = bflib.Dims(t, 1, dd, 2, b)
        E, A, G = _host_inputs(bflib, d, 50 + i)
        W = bflib.ResidentWeights(1, b, dd, A, G)
        J = cuda.full((d.jsize,), 0x5A, dtype=cuda.uint8, device="cuda")
        probs.append((d, (E, A, G), W, cuda.from_numpy(E).cuda(), J))
        if b == 128:  # more tiles than clusters: ranges start anywhere
            for k in range(40):
                probs.append((d, (E, A, G), W, probs[-1][3], cuda.full((d.jsize,), 0x5A, dtype=cuda.uint8, device="cuda")))
    batch = bflib.Batch([(W, d.ntimes, Ed, J) for d, _, W, Ed, J in probs])
    for _ in range(2):
        batch.run()
        bflib.stream_status()
        for d, host, _, _, J in probs:
            np.testing.assert_array_equal(J.cpu().numpy(), _oracle_J(oracle, d, *host), err_msg=str(d))
            J.fill_(0x5A)
