"""The failure path of launches on pairs of SMs: a launch whose copies never come
gives up within its time limit, in every form of resident weights, and the next call
is right."""
from __future__ import annotations

import time

import pytest

pytestmark = pytest.mark.gpu


# W of one pass resident, of two (shared operand; row sums), a ring
@pytest.mark.parametrize("d,b", [(512, 48), (512, 128), (256, 192), (1024, 96)])
def test_stalled_pair_launch_gives_up(bflib, cuda, d, b):
    dims = bflib.Dims(2048, 9, d, 2, b)
    E, A = (cuda.empty(n, dtype=cuda.uint8, device="cuda") for n in (dims.esize, dims.asize))
    bflib.fill_random_device(E, d, 0)
    bflib.fill_random_device(A, b, 1)
    G = cuda.from_numpy(bflib.gains(dims)).cuda()
    W = bflib.ResidentWeights(9, b, d, A, G)
    J = [cuda.empty(dims.jsize, dtype=cuda.uint8, device="cuda") for _ in range(2)]
    batch = bflib.Batch([(W, 2048, E, J[0])])
    bflib.set_kernel("simt")
    bflib.form_beams_ex(dims, J[1], E, A, G)
    bflib.set_kernel("auto")
    bflib.stream_status()
    t0 = time.monotonic()
    bflib.set_test_stall(True)
    try:
        W.form_beams(J[0], E, 2048)
        with pytest.raises(bflib.BeamformError) as e:
            bflib.stream_status()
        assert e.value.status == bflib.ERR_DEVICE_TIMEOUT
    finally:
        bflib.set_test_stall(False)
    assert time.monotonic() - t0 < 4.0  # one limit of 1.5 s; no exit wait runs into it again
    for run in (lambda: W.form_beams(J[0], E, 2048), batch.run):
        J[0].zero_()
        run()
        bflib.stream_status()
        assert cuda.equal(J[0], J[1])
