"""The one-CTA kernel's wider layouts, which run where a device has no room for a
cluster of two SMs: eight and twelve epilogue warps, one unpack group, two with the
W forwarder, row sums in each.  Every byte of J equals the oracle's."""
from __future__ import annotations

import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def one_cta(bflib, cuda):
    bflib.set_test_one_cta(True)
    yield bflib
    bflib.set_test_one_cta(False)


def _J(oracle, d, E, A, G, j_layout="linear"):
    od = oracle.Dims(d.ntimes, d.nfrequencies, d.ndishes, d.npolarizations, d.nbeams)
    J = oracle.form_beams(od, E, A, G)
    return oracle.J_to_J2(od, J) if j_layout == "j2" else J


# (t, f, d, b): signed codes in two unpack groups (17 to 64 beams), W + 8 in one (65 to
# 96) and in several passes; 1, 2, 4, 5 and 16 K stages; empty halves, ragged dishes
SHAPES = [(64, 3, 8, 72), (80, 3, 128, 96), (208, 2, 512, 41), (272, 1, 384, 64), (1040, 3, 512, 96), (144, 2, 256, 24),
          (528, 2, 1024, 200), (336, 2, 1024, 96), (144, 1, 2048, 130), (8208, 3, 512, 128), (80, 160, 128, 80),
          (272, 50, 520, 104), (4096, 5, 512, 33)]


@pytest.mark.parametrize("shape", SHAPES)
def test_layouts_match_oracle(one_cta, cuda, oracle, shape):
    bf, (t, f, dd, b) = one_cta, shape
    d = bf.Dims(t, f, dd, 2, b)
    E, A, G = bf.seeded_host_inputs(d, sum(shape))
    Ed, Ad, Gd = (cuda.from_numpy(x).cuda() for x in (E, A, G))
    J = cuda.full((d.jsize + 32,), 0x5A, dtype=cuda.uint8, device="cuda")
    for j_layout in ("linear", "j2"):
        want = _J(oracle, d, E, A, G, j_layout)
        J.fill_(0x5A)
        assert bf.form_beams_adler(d, J[16:-16], Ed, Ad, Gd, j_layout=j_layout) == zlib.adler32(want.tobytes())
        assert bf.last_kernel() == "tensor"
        np.testing.assert_array_equal(J[16:-16].cpu().numpy(), want)
        assert bool((J[:16] == 0x5A).all()) and bool((J[-16:] == 0x5A).all())
    W = bf.ResidentWeights(f, b, dd, Ad, Gd)
    J.fill_(0x5A)
    W.form_beams(J[16:-16], Ed, t)
    bf.stream_status()
    np.testing.assert_array_equal(J[16:-16].cpu().numpy(), _J(oracle, d, E, A, G))


@pytest.mark.parametrize("fill", [(0xFF, 0x00), (0x00, 0x0F), (0xFF, 0xF0), (0x00, 0xFF)])
@pytest.mark.parametrize("b", [96, 33])
def test_extreme_sums(one_cta, cuda, oracle, b, fill):
    bf = one_cta
    d = bf.Dims(64, 1, 2048, 2, b)
    E, A, _ = bf.seeded_host_inputs(d, 0)
    E[:], A[:] = fill
    E[::7] ^= 0x01
    G = (np.arange(1, b + 1, dtype=np.float32) / np.float32(b * 128 * 2048 / 7)).astype(np.float32)
    J = cuda.empty(d.jsize, dtype=cuda.uint8, device="cuda")
    bf.form_beams_ex(d, J, *(cuda.from_numpy(x).cuda() for x in (E, A, G)))
    bf.stream_status()
    np.testing.assert_array_equal(J.cpu().numpy(), _J(oracle, d, E, A, G))


@pytest.mark.parametrize("dd", [128, 512, 2048])
def test_batch_and_odd_shapes(one_cta, cuda, oracle, dd):
    """Grouped launches over problems of both forms of the codes, one and two passes
    (with the ring plans that only these launches take), and the padded route."""
    bf = one_cta
    probs = []
    for i, (t, b) in enumerate([(272, 96), (64, 16), (528, 64), (8192, 128), (16, 72), (144, 41)]):
        d = bf.Dims(t, 1, dd, 2, b)
        host = bf.seeded_host_inputs(d, 50 + i)
        W = bf.ResidentWeights(1, b, dd, *host[1:])
        probs.append((d, host, W, cuda.from_numpy(host[0]).cuda(), cuda.full((d.jsize,), 0x5A, dtype=cuda.uint8,
                                                                               device="cuda")))
    batch = bf.Batch([(W, d.ntimes, E, J) for d, _, W, E, J in probs])
    batch.run()
    bf.stream_status()
    for d, host, _, _, J in probs:
        np.testing.assert_array_equal(J.cpu().numpy(), _J(oracle, d, *host), err_msg=str(d))
    d = bf.Dims(1001, 3, dd - 3, 2, 96)
    host = bf.seeded_host_inputs(d, 3)
    J = cuda.empty(d.jsize, dtype=cuda.uint8, device="cuda")
    bf.form_beams_ex(d, J, *(cuda.from_numpy(x).cuda() for x in host))
    bf.stream_status()
    np.testing.assert_array_equal(J.cpu().numpy(), _J(oracle, d, *host))


@pytest.mark.parametrize("b", [96, 32])
def test_stalled_launch_gives_up(one_cta, cuda, b):
    """The failure path of these layouts: the waits end and the next call is right."""
    bf = one_cta
    d = bf.Dims(256, 2, 128, 2, b)
    E, A = (cuda.empty(n, dtype=cuda.uint8, device="cuda") for n in (d.esize, d.asize))
    bf.fill_random_device(E, 1, 0)
    bf.fill_random_device(A, 1, 1)
    G = cuda.from_numpy(bf.gains(d)).cuda()
    J = [cuda.empty(d.jsize, dtype=cuda.uint8, device="cuda") for _ in range(2)]
    bf.set_test_stall(True)
    try:
        bf.form_beams_ex(d, J[0], E, A, G)
        with pytest.raises(bf.BeamformError) as e:
            bf.stream_status()
        assert e.value.status == bf.ERR_DEVICE_TIMEOUT
    finally:
        bf.set_test_stall(False)
    bf.form_beams_ex(d, J[0], E, A, G)
    bf.set_kernel("simt")
    bf.form_beams_ex(d, J[1], E, A, G)
    bf.set_kernel("auto")
    bf.stream_status()
    assert cuda.equal(J[0], J[1])
