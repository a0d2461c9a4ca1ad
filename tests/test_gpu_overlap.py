"""Calls that overlap on the device: a pass, new weights (with other gains) and the
next pass on one stream without a wait in between.  The second pass may be resident
while the first still runs, and must read what the update between them wrote."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def _pass_exact(bf, torch, d, E, A, G):
    J = torch.empty(d.jsize, dtype=torch.uint8, device="cuda")
    bf.set_kernel("simt")
    try:
        bf.form_beams_ex(d, J, E, A, G)
        bf.stream_status()
    finally:
        bf.set_kernel("auto")
    return J


def _sets(bf, torch, d, n=3):
    """n sets of E, A and G, their gains 1, -3 and (needing the narrowing requantisation) 1e30 times the usual ones."""
    out = []
    for k in range(n):
        E = torch.empty(d.esize, dtype=torch.uint8, device="cuda")
        A = torch.empty(d.asize, dtype=torch.uint8, device="cuda")
        bf.fill_random_device(E, k, 0)
        bf.fill_random_device(A, k, 1)
        G = torch.from_numpy(bf.gains(d)).cuda() * (1.0, -3.0, 1e30)[k % 3]
        out.append((E, A, G, _pass_exact(bf, torch, d, E, A, G)))
    return out


# narrow passes (two CTAs to an SM, several launches resident) of few and many
# tiles, and pairs of SMs with both forms of the codes
@pytest.mark.parametrize("shape", [(64, 1, 64, 2, 8), (256, 3, 64, 2, 16), (2048, 7, 128, 2, 16), (128, 2, 512, 2, 64),
                                   (2048, 4, 512, 2, 96)])
def test_updates_between_passes(bflib, cuda, shape):
    d = bflib.Dims(*shape)
    sets = _sets(bflib, cuda, d)
    W = bflib.ResidentWeights(d.nfrequencies, d.nbeams, d.ndishes, sets[0][1], sets[0][2])
    reps = 60
    J = cuda.empty((reps, d.jsize), dtype=cuda.uint8, device="cuda")
    cuda.cuda.synchronize()
    for i in range(reps):
        E, A, G, _ = sets[i % len(sets)]
        W.update(A, G)
        W.form_beams(J[i], E, d.ntimes)
    bflib.stream_status()
    for i in range(reps):
        assert cuda.equal(J[i], sets[i % len(sets)][3]), i


@pytest.mark.parametrize("shape", [(64, 1, 64, 2, 8), (2048, 4, 512, 2, 96), (1001, 9, 250, 2, 45)])
def test_explicit_calls_follow_each_other(bflib, cuda, shape):
    """The same with the weights given to each call, and a checked call's sums."""
    d = bflib.Dims(*shape)
    sets = _sets(bflib, cuda, d)
    sums = [bflib.adler32_device(s[3]) for s in sets]
    reps = 60
    J = cuda.empty((reps, d.jsize), dtype=cuda.uint8, device="cuda")
    for i in range(reps):
        E, A, G, _ = sets[i % len(sets)]
        if i % 4 == 3:
            assert bflib.form_beams_adler(d, J[i], E, A, G) == sums[i % len(sets)]
        else:
            bflib.form_beams_ex(d, J[i], E, A, G)
    bflib.stream_status()
    for i in range(reps):
        assert cuda.equal(J[i], sets[i % len(sets)][3]), i
