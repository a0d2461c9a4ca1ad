"""The workloads whose speed matters to a user of this library, each as one pass
through the public entry points.

A case is a dict of plain values.  ``kind`` says which call it stands for:

  resident  a chunk of voltages beamformed with weights that stay on the device
  call      the explicit call with device arrays, weights prepared each time
  checked   the explicit call that also returns the checksum of J, with the
            A2 / J2 wire formats
  exact     the explicit call on shapes the tensor-core kernel does not take
  host      the drop-in form_beams(J, E, A, G) on ordinary host arrays
  refresh   new weights for a resident handle, then a chunk with them
  batch     many uneven problems behind one replayed launch
  served    a burst of chunks submitted to the server from pinned host memory,
            waited for one by one
"""
import math
import random

import numpy as np
import torch

import beamforming_gb300 as bf

BATCH_BEAMS = (16, 32, 64, 96, 128)
SERVED_TIMES = (1024, 2048, 4096, 8192, 16384)


def _case(name, kind, t, f, d, b, p=2, **more):
    c = {"kind": kind, "t": t, "f": f, "d": d, "p": p, "b": b, **more}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: one channel, few dishes and beams; launch and host cost
        _case("smallest", "resident", 64, 1, 64, 8),
        # one channel's chunk as the server's clients send it, beamformed on its own
        _case("channel", "resident", 4096, 1, 512, 96),
        # an ordinary call with everything on the device (the CPU-runnable shape)
        _case("ordinary", "call", 2048, 16, 512, 96),
        # sizes that fill no tile: times, dishes and beams all ragged
        _case("ragged", "resident", 8208, 21, 328, 41),
        # the full single-GPU chunk
        _case("full_chunk", "resident", 32768, 84, 512, 96),
        # the wide array: six beam passes, compute-bound
        _case("wide", "resident", 16384, 16, 1024, 512),
        # the wire formats of the downstream stages, with the checksum of J
        _case("checked", "checked", 8192, 16, 256, 64),
        # odd times and dishes: the exact integer kernel
        _case("exact", "exact", 2001, 9, 250, 45),
        # weights regenerated for a wide array, then a chunk with them
        _case("refresh", "refresh", 1024, 16, 1024, 512),
        # 128 uneven problems behind one replayed launch
        _case("batch", "batch", 32768, 1, 512, 128, n=128, shapes=2),
        # the drop-in call on host memory
        _case("host", "host", 2048, 16, 512, 96),
        # a burst of chunks through the server, from and to pinned host memory
        _case("served", "served", 16384, 64, 512, 96, n=32, shapes=3),
    ]


def _log(rng, lo, hi, multiple=1):
    """A multiple of `multiple` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, max(1, round(v / multiple)) * multiple))


def draw(rng):
    kind = rng.choice(("resident", "resident", "resident", "call", "checked", "exact", "refresh", "batch", "host", "served"))
    if kind in ("resident", "call"):
        while True:
            c = _case(None, kind, _log(rng, 16, 32768, 16), _log(rng, 1, 84), _log(rng, 64, 2048, 8), _log(rng, 5, 512))
            if _cmacs(c) <= 2.7e11 and c["t"] * c["f"] * c["d"] * 2 <= 2.8e9 and c["t"] * c["f"] * c["b"] * 2 <= 5.4e8:
                return c
    if kind == "checked":
        return _case(None, kind, _log(rng, 64, 32768, 16), _log(rng, 1, 32), rng.choice((256, 512)), _log(rng, 8, 128))
    if kind == "exact":
        return _case(None, kind, _log(rng, 15, 8192), _log(rng, 1, 16), _log(rng, 31, 600), _log(rng, 7, 128), p=rng.choice((1, 2)))
    if kind == "refresh":
        return _case(None, kind, _log(rng, 64, 4096, 16), _log(rng, 1, 84), _log(rng, 64, 1024, 8), _log(rng, 16, 512))
    if kind == "host":
        return _case(None, kind, _log(rng, 64, 8192, 16), _log(rng, 1, 32), _log(rng, 64, 512, 8), _log(rng, 8, 128))
    if kind == "batch":
        return _case(None, kind, _log(rng, 1024, 32768, 256), 1, rng.choice((256, 512, 1024)), 128, n=_log(rng, 8, 128), shapes=rng.randrange(1 << 20))
    return _case(None, kind, rng.choice(SERVED_TIMES), rng.choice((16, 64)), 512, rng.choice((32, 64, 96)), n=_log(rng, 4, 48), shapes=rng.randrange(1 << 20))


def _problems(c):
    """(times, beams) of each problem of a batch: times log-uniform, multiples of 256."""
    r = random.Random(c["shapes"])
    return [(_log(r, min(512, c["t"]), c["t"], 256), r.choice(BATCH_BEAMS)) for _ in range(c["n"])]


def _chunks(c):
    """(channel, times) of each chunk of a served burst."""
    r = random.Random(c["shapes"])
    return [(r.randrange(c["f"]), r.choice([t for t in SERVED_TIMES if t <= c["t"]])) for _ in range(c["n"])]


def _parts(c):
    """(times, frequencies, beams) of each beamforming problem of a case."""
    if c["kind"] == "batch":
        return [(t, 1, b) for t, b in _problems(c)]
    if c["kind"] == "served":
        return [(t, 1, c["b"]) for _, t in _chunks(c)]
    return [(c["t"], c["f"], c["b"])]


def _cmacs(c):
    return sum(t * f * b for t, f, b in _parts(c)) * c["p"] * c["d"]


def work(c):
    d, p, parts = c["d"], c["p"], _parts(c)
    e = sum(t * f for t, f, _ in parts) * d * p
    j = sum(t * f * b for t, f, b in parts) * p
    if c["kind"] == "served":  # a burst reads the weights of the channels it has
        rows = len({ch for ch, _ in _chunks(c)}) * c["b"]
    else:
        rows = sum(f * b for _, f, b in parts)
    return {"bytes": e + j + rows * (d + 4), "flops": 8 * _cmacs(c)}


def _bytes(n, gen):
    """n uniform bytes on the device: every nibble uniform on [-8, 7]."""
    return torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda", generator=gen)


def _gains(f, d, b):
    return bf.gains(bf.Dims(1, f, d, 2, b))


def _weights(c, gen, f, b):
    A = _bytes(f * b * c["d"], gen)
    G = torch.from_numpy(_gains(f, c["d"], b)).cuda()
    return A, G


def _inputs(c, seed):
    """The voltages and weights of a case, from the seed alone: (E, A, G) of each problem."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    d, p = c["d"], c["p"]
    if c["kind"] == "batch":
        return [(_bytes(t * d * p, gen), *_weights(c, gen, 1, b)) for t, b in _problems(c)]
    if c["kind"] == "served":
        A, G = _weights(c, gen, c["f"], c["b"])
        return [(_bytes(t * d * p, gen), A, G) for _, t in _chunks(c)]
    E = _bytes(c["t"] * c["f"] * d * p, gen)
    return [(E, *_weights(c, gen, c["f"], c["b"]))]


def _pinned(n):
    return torch.empty(n, dtype=torch.uint8, pin_memory=True).numpy()


def prepare(case, seed):
    c, kind = case, case["kind"]
    t, f, d, p, b = (c[k] for k in ("t", "f", "d", "p", "b"))
    inputs = _inputs(c, seed)
    E, A, G = inputs[0]
    s = {"kind": kind, "dims": bf.Dims(t, f, d, p, b)}
    if kind == "batch":
        sizes = [(n, nb) for n, nb in _problems(c)]
        ends = np.cumsum([n * nb * p for n, nb in sizes]).tolist()
        s["J"] = torch.empty(ends[-1], dtype=torch.uint8, device="cuda")
        views = [s["J"][e - n * nb * p:e] for e, (n, nb) in zip(ends, sizes)]
        s["weights"] = [bf.ResidentWeights(1, nb, d, a, g) for (n, nb), (_, a, g) in zip(sizes, inputs)]
        s["batch"] = bf.Batch([(w, n, e, j) for w, (n, _), (e, _, _), j in zip(s["weights"], sizes, inputs, views)])
        return s
    if kind == "served":
        chunks = _chunks(c)
        s["weights"] = bf.ResidentWeights(f, b, d, A, G)
        s["server"] = bf.Server(s["weights"], hbm_budget_bytes=4 << 30, spin_wait=True)
        ends = np.cumsum([n * b * p for _, n in chunks]).tolist()
        s["J"] = _pinned(ends[-1])
        s["chunks"] = []
        for (ch, n), (e, _, _), end in zip(chunks, inputs, ends):
            host = _pinned(e.numel())
            host[:] = e.cpu().numpy()
            s["chunks"].append((ch, n, host, s["J"][end - n * b * p:end]))
        return s
    if kind == "host":
        s.update(E=E.cpu().numpy(), A=A.cpu().numpy(), G=G.cpu().numpy(), J=np.zeros(s["dims"].jsize, np.uint8))
        return s
    s.update(E=E, A=A, G=G, J=torch.empty(s["dims"].jsize, dtype=torch.uint8, device="cuda"))
    if kind == "resident":
        s["weights"] = bf.ResidentWeights(f, b, d, A, G)
    if kind == "refresh":  # the handle holds other weights until the first refresh
        s["weights"] = bf.ResidentWeights(f, b, d, A.flip(0), G)
    return s


def run(s):
    kind = s["kind"]
    if kind == "resident":
        s["weights"].form_beams(s["J"], s["E"], s["dims"].ntimes)
    elif kind in ("call", "exact"):
        bf.form_beams_ex(s["dims"], s["J"], s["E"], s["A"], s["G"])
    elif kind == "checked":
        return s["J"], bf.form_beams_adler(s["dims"], s["J"], s["E"], s["A"], s["G"], a_layout="a2", j_layout="j2")
    elif kind == "refresh":
        s["weights"].update(s["A"], s["G"])
        s["weights"].form_beams(s["J"], s["E"], s["dims"].ntimes)
    elif kind == "batch":
        s["batch"].run()
    elif kind == "served":
        tickets = [s["server"].submit(ch, n, e, j) for ch, n, e, j in s["chunks"]]
        for ticket in tickets:
            s["server"].wait(ticket)
    else:
        bf.set_dims(s["dims"])
        bf.form_beams(s["J"], s["E"], s["A"], s["G"])
    return s["J"]


# ------------------------------------------------------------ the same in 64 bits


def _parts_of(x):
    """Real and imaginary parts of stored bytes (value + 8 in each nibble), as 64-bit floats."""
    return (x >> 4).double() - 8, (x & 15).double() - 8


def _a2_parts(A, f, b, d):
    """The weights of A2 bytes: per (f, b) the real then the imaginary nibbles of all
    dishes, two to a byte (even positions low), dish bits in the order 8 | 5..0 | 7..6."""
    nib = torch.stack((A & 15, A >> 4), dim=-1).reshape(f, b, 2, d).double() - 8
    i = torch.arange(d, device=A.device)
    at = (i & 0x100) | ((i & 0x3F) << 2) | ((i >> 6) & 3)
    return nib[:, :, 0, at], nib[:, :, 1, at]


def _beams(c, E, A, G, t, f, b):
    """J[b][f][p][t] (J2[b][f][t][p] for checked) of one problem."""
    d, p, wire = c["d"], c["p"], c["kind"] == "checked"
    ar, ai = _a2_parts(A, f, b, d) if wire else _parts_of(A.reshape(f, b, d))
    E, G = E.reshape(t, f, d, p), G.reshape(f, b)
    J = torch.empty((b, f, t, p) if wire else (b, f, p, t), dtype=torch.uint8, device=E.device)
    for k in range(f):
        for t0 in range(0, t, 4096):
            x = E[t0:t0 + 4096, k].permute(2, 0, 1).contiguous()  # p, t, d
            er, ei = _parts_of(x)
            re = er @ ar[k].T - ei @ ai[k].T  # p, t, b
            im = ei @ ar[k].T + er @ ai[k].T
            q = []
            for raw in (re, im):
                # the gain multiplies in single precision; ties round to even
                v = torch.round((G[k] * raw.float()).double()).clamp(-7, 7)
                q.append((v + 8).to(torch.uint8))
            out = (q[0] << 4) | q[1]
            if wire:
                J[:, k, t0:t0 + 4096, :] = out.permute(2, 1, 0)
            else:
                J[:, k, :, t0:t0 + 4096] = out.permute(2, 0, 1)
    return J.reshape(-1)


def _adler32(x):
    """The adler32 of a device tensor of bytes."""
    n, m = x.numel(), 65521
    a, s = 0, 0
    for i in range(0, n, 1 << 22):
        v = x[i:i + (1 << 22)].to(torch.int64)
        a += int(v.sum())
        s += int((v * ((n - torch.arange(i, i + v.numel(), device=x.device)) % m)).sum())
    return (((n + s) % m) << 16) | ((1 + a) % m)


def exact(case, seed):
    c, kind = case, case["kind"]
    out = []
    channels = [ch for ch, _ in _chunks(c)] if kind == "served" else [0] * len(_parts(c))
    for (t, f, b), (E, A, G), ch in zip(_parts(c), _inputs(c, seed), channels):
        if kind == "served":
            n = b * c["d"]
            A, G = A[ch * n:(ch + 1) * n], G[ch * b:(ch + 1) * b]
        out.append(_beams(c, E, A, G, t, f, b))
    J = torch.cat(out)
    if kind == "checked":
        return J, _adler32(J)
    return J.cpu().numpy() if kind in ("host", "served") else J
