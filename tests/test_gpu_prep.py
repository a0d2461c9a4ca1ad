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
