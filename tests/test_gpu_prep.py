"""The weight preparation's ways of reading A (16-byte rows, rows that are not
multiples of 16, A off a 16-byte boundary, A2) give the exact kernel's bytes."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dishes,beams,a_off,a_layout", [
    (512, 96, 0, "linear"), (512, 96, 8, "linear"), (512, 33, 1, "linear"), (1032, 40, 0, "linear"),
    (8, 1, 0, "linear"), (2048, 17, 0, "linear"), (256, 70, 0, "a2"), (512, 9, 3, "a2")])
def test_prep_reads_any_weights(bflib, cuda, dishes, beams, a_off, a_layout):
    d = bflib.Dims(64, 3, dishes, 2, beams)
    E = cuda.empty(d.esize, dtype=cuda.uint8, device="cuda")
    A = cuda.empty(d.asize + 16, dtype=cuda.uint8, device="cuda")
    bflib.fill_random_device(E, dishes, 0)
    bflib.fill_random_device(A, beams, 1)
    A = A[a_off:a_off + d.asize]
    G = cuda.from_numpy(bflib.gains(d)).cuda()
    out = {}
    for kernel in ("tensor", "simt"):
        J = cuda.zeros(d.jsize, dtype=cuda.uint8, device="cuda")
        bflib.set_kernel(kernel)
        try:
            bflib.form_beams_layout(d, J, E, A, G, a_layout=a_layout)
            bflib.stream_status()
        finally:
            bflib.set_kernel("auto")
        out[kernel] = J
    assert cuda.equal(out["tensor"], out["simt"])


@pytest.mark.parametrize("dishes,beams,a_off", [(512, 96, 0), (512, 33, 1), (1032, 40, 0), (129, 7, 0), (130, 100, 3),
                                                (2050, 5, 0)])
def test_update_keeps_the_weights_it_read(bflib, cuda, dishes, beams, a_off):
    """The prepared operand and the kept copies of A and G (which the exact kernel
    reads) are those of the update, also after the caller's buffers change."""
    F, T = 3, 64
    d = bflib.Dims(T, F, dishes, 2, beams)
    E = cuda.empty(d.esize, dtype=cuda.uint8, device="cuda")
    bflib.fill_random_device(E, dishes, 0)
    buf = cuda.empty(d.asize + 16, dtype=cuda.uint8, device="cuda")
    A = buf[a_off:a_off + d.asize]
    G = cuda.from_numpy(bflib.gains(d)).cuda()
    bflib.fill_random_device(A, 1, 1)
    W = bflib.ResidentWeights(F, beams, dishes, A, G)
    bflib.fill_random_device(A, 2, 1)
    G *= 0.5
    W.update(A, G)
    want = cuda.empty(d.jsize, dtype=cuda.uint8, device="cuda")
    bflib.set_kernel("simt")
    try:
        bflib.form_beams_ex(d, want, E, A, G)
        bflib.stream_status()
        A.fill_(0)
        G.fill_(0)
        J = cuda.empty_like(want)
        W.form_beams(J, E, T)
        bflib.stream_status()
        assert cuda.equal(J, want)
    finally:
        bflib.set_kernel("auto")
    J2 = cuda.empty_like(want)
    W.form_beams(J2, E, T)
    bflib.stream_status()
    assert cuda.equal(J2, want)
