"""A CPU model of the barrier protocol of the kernel on pairs of SMs
(bf_form_beams_pair), explored under random schedules like the one-CTA kernel's
(test_pipeline_protocol.py, whose barriers it uses), and the row sums of the one-CTA
kernel's wider layouts, which that model does not have.

Modelled: two CTAs, each with its E producer, W producer, unpack warps (a unit is the
warps that work on the same boxes of a stage) and epilogue; the leader's MMA issuer,
whose commits arrive in both CTAs, each at its own time; the peer's relay, which tells
the leader that its W and digit rows have landed; W resident for one or two passes of
a frequency and given back in rounds, or an ordinary ring; the operand that the
passes of a tile share; the row sums of E in the tile of the offset MMA; and the exit:
producers drain their copies, the leader its commits, and the peer, after the
cluster's last meeting, the commits that the leader counted for it.  A cluster's range
of tiles may start and end anywhere in a table of problems of one to three passes.
"""
from __future__ import annotations

import random

import pytest

from test_pipeline_protocol import Barrier, Hazard, Model, _seed


def drive(m, roles, rng, inorder=True, fail=None, last_roles=None):
    """Runs the roles under random schedules to their end, then `last_roles()` (those
    behind the cluster's last meeting).  `fail` as in Model.run."""
    err = [False]

    def rounds(roles):
        blocked, done, nwaits = {}, set(), dict.fromkeys(roles, 0)

        def resume(name, value):
            while True:
                try:
                    op = roles[name].send(value)
                except StopIteration:
                    done.add(name)
                    return
                blocked[name] = op
                kind, bar, phase = op
                if kind == "step":
                    return
                if kind == "wait":
                    nwaits[name] += 1
                    if fail == (name, nwaits[name]):
                        err[0] = True
                        value = False
                        continue
                if not m.check_wait(bar, phase):
                    return
                value = True

        for name in list(roles):
            resume(name, None)
        while len(done) < len(roles):
            choices = []
            for n in roles:
                if n in done:
                    continue
                kind, bar, phase = blocked[n]
                if kind == "step" or m.check_wait(bar, phase):
                    choices.append(("role", n, True))
                elif kind == "wait" and err[0]:
                    choices.append(("role", n, False))
            choices += [("event", i, None) for i in range(len(m.events))]
            if m.mma_queue:
                choices.append(("mma", 0, None))
            dc = m.deliverable_commits()
            # the two arrivals of a commit are independent; in order: per CTA
            heads = []
            for c in dc:
                if not inorder or all(h[2] != c[2] for h in heads):
                    heads.append(c)
            choices += [("commit", c, None) for c in heads]
            if not choices:
                raise Hazard("deadlock: " + str([(n, getattr(blocked[n][1], "name", None), blocked[n][2])
                                                 for n in roles if n not in done]))
            kind, i, val = rng.choice(choices)
            if kind == "role":
                resume(i, val)
            elif kind == "event":
                m.events.pop(i)()
            elif kind == "mma":
                m.complete_next_mma()
            else:
                m.commits.remove(i)
                i[0].arrive()

    rounds(roles)
    if last_roles:
        rounds(last_roles())
    assert not m.events, f"copies still to land at exit: {[e.barrier for e in m.events]}"
    assert not m.mma_queue, f"{len(m.mma_queue)} MMAs still running at exit"
    assert not m.commits, f"commits still to land at exit: {[c[0].name for c in m.commits]}"
    return err[0]


class Tile:
    """One tile of a launch: its problem, frequency, time pair and pass."""

    def __init__(self, prob, f, tp, ps, npass, ntp):
        self.prob, self.f, self.tp, self.ps, self.npass, self.ntp = prob, f, tp, ps, npass, ntp
        self.w, self.a = (prob, f, ps), (prob, f, tp)

    # PairCursor's rules
    def first_of_w(self, n, sets):
        return self.npass > sets or n < self.npass or self.tp == 0

    def last_of_w(self, n, sets):
        return self.npass > sets or (self.tp + 1 == self.ntp and n > self.npass - self.ps)

    def first_of_a(self, share, range_first):
        return not share or self.ps == 0 or range_first

    def last_of_a(self, share, range_last):
        return not share or self.ps + 1 == self.npass or range_last


def tiles_of(table):
    """The tiles of a table of (passes, time pairs, frequencies): pass fastest."""
    return [Tile(i, f, tp, ps, npass, ntp) for i, (npass, ntp, F) in enumerate(table)
            for f in range(F) for tp in range(ntp) for ps in range(npass)]


class Pair(Model):
    """The two CTAs of a cluster over `tiles`.  CTA 0 leads."""

    def __init__(self, tiles, S, SW, R, sets, share, nk, groups, sums, rng):
        self.tiles, self.S, self.SW, self.R, self.sets, self.share = tiles, S, SW, R, sets, bool(share) and not sums
        self.nk, self.G, self.sums, self.rng = nk, groups, sums, rng
        self.stream = SW < nk
        self.parts = 2 // groups  # units that work on one stage
        per_cta = lambda n, name, count: [[Barrier(f"{name}{i}@{c}", count) for i in range(n)] for c in (0, 1)]
        leader = lambda n, name, count: [Barrier(f"{name}{i}", count) for i in range(n)]
        self.raw_full, self.raw_empty = per_cta(R, "raw_full", 1), per_cta(R, "raw_empty", self.parts)
        self.w_full, self.w_empty = per_cta(SW, "w_full", 1), per_cta(SW, "w_empty", 1)
        self.d_full, self.d_empty = per_cta(2, "d_full", 1), per_cta(2, "d_empty", 1)
        self.empty, self.accfull = per_cta(S, "empty", 1), per_cta(2, "accfull", 1)
        self.w_peer, self.d_peer = leader(SW, "w_peer", 1), leader(2, "d_peer", 1)
        self.a_full, self.accempty = leader(S, "a_full", 2 * self.parts), leader(2, "accempty", 2)
        self.rs_full = leader(2, "rs_full", 4)
        # slot contents per CTA
        self.raw, self.wslot, self.dslot = ([[None] * n, [None] * n] for n in (R, SW, 2))
        self.stage = [[[None] * self.parts for _ in range(S)] for _ in (0, 1)]
        self.rs = [[[None, None], [None, None]] for _ in (0, 1)]  # [cta][tile & 1][unit]
        self.raw_left = [[0] * R, [0] * R]
        self.acc = [None, None]
        self.acc_reading, self.acc_read = [set(), set()], [set(), set()]
        self.readers, self.events, self.mma_queue, self.commits = {}, [], [], []
        self.mma_issued = self.mma_done = 0
        self.acc_tile_done = {}
        self.cut_done = [Barrier(f"cut_done@{c}", 1) for c in (0, 1)]
        self.counts = (0, [0, 0], [0, 0], 0, 0)
        self.planted = None

    # ------------------------------------------------------------- slots
    def load(self, slot, c, i, what, bar):
        kind = "wslot" if slot is self.wslot else "dslot" if slot is self.dslot else "raw"
        if self.busy((kind, c), i):
            raise Hazard(f"a copy overwrites {kind}[{i}] of CTA {c} while the tensor core reads it")
        if kind == "raw" and self.raw_left[c][i]:
            raise Hazard(f"a copy overwrites raw[{i}] of CTA {c} before the unpack has read {slot[c][i]}")
        slot[c][i] = (what, False)
        if kind == "raw":
            self.raw_left[c][i] = self.parts

        def land():
            slot[c][i] = (what, True)
        bar.arrive(expect_tx=1)
        self.tma(bar, 1, land)

    def issue(self, reads, tile_no):
        """One MMA of the pair: reads (kind, slot, expected) in both CTAs."""
        mid = self.mma_issued
        self.mma_issued += 1
        keys = []
        for kind, i, want in reads:
            for c in (0, 1):
                have = getattr(self, kind)[c][i]
                have = have if isinstance(have, list) else [have]
                if any(h != (want, True) for h in have):
                    raise Hazard(f"an MMA reads {kind}[{i}] of CTA {c} holding {have}, wants {want}")
                keys.append(((kind, c), i))
                self.readers.setdefault(keys[-1], set()).add(mid)
        self.mma_queue.append((keys, tile_no, mid))

    def complete_next_mma(self):
        keys, t, mid = self.mma_queue.pop(0)
        for k in keys:
            self.readers[k].discard(mid)
        self.mma_done += 1
        self.acc_tile_done[t] = self.acc_tile_done.get(t, 0) + 1

    def commit(self, bars):
        for c in (0, 1):
            self.commits.append((bars[c], self.mma_issued, c))

    # ------------------------------------------------------------- roles
    def e_producer(self, c):
        it = 0
        ok = True
        for n, t in enumerate(self.tiles):
            if not t.first_of_a(self.share, n == 0):
                continue
            for ks in range(self.nk):
                r = it % self.R
                if it >= self.R:
                    ok = yield self.wait(self.raw_empty[c][r], it // self.R - 1)
                if not ok:
                    break
                self.load(self.raw, c, r, (t.a, ks), self.raw_full[c][r])
                it += 1
            if not ok:
                break
        for q in range(max(0, it - self.R), it):
            yield ("drain", self.raw_full[c][q % self.R], q // self.R)

    def w_producer(self, c):
        it = dit = 0
        ok = True
        for n, t in enumerate(self.tiles):
            fresh = t.first_of_w(n, self.sets)
            if not (fresh or self.stream):
                continue
            if fresh:
                d = dit % 2
                if dit >= 2:
                    ok = yield self.wait(self.d_empty[c][d], dit // 2 - 1)
                if not ok:
                    break
                self.load(self.dslot, c, d, t.w, self.d_full[c][d])
                dit += 1
            for ks in range(self.nk):
                s = it % self.SW
                if it >= self.SW:
                    ok = yield self.wait(self.w_empty[c][s], it // self.SW - 1)
                if not ok:
                    break
                self.load(self.wslot, c, s, (t.w, ks), self.w_full[c][s])
                it += 1
            if not ok:
                break
        for q in range(max(0, it - self.SW), it):
            yield ("drain", self.w_full[c][q % self.SW], q // self.SW)
        for q in range(max(0, dit - 2), dit):
            yield ("drain", self.d_full[c][q % 2], q // 2)

    def relay(self):
        it = dit = 0
        for n, t in enumerate(self.tiles):
            fresh = t.first_of_w(n, self.sets)
            if fresh:
                if self.planted != "relay" and not (yield self.wait(self.d_full[1][dit % 2], dit // 2)):
                    return
                self.d_peer[dit % 2].arrive()
                dit += 1
            if fresh or self.stream:
                for _ in range(self.nk):
                    if self.planted != "relay" and not (yield self.wait(self.w_full[1][it % self.SW], it // self.SW)):
                        return
                    self.w_peer[it % self.SW].arrive()
                    it += 1

    def unpack(self, c, unit):
        group, part = (unit, 0) if self.G == 2 else (0, unit)
        ntiles, nk = len(self.tiles), self.nk
        operands = [t.a for n, t in enumerate(self.tiles) if t.first_of_a(self.share, n == 0)]
        tile, kpos = 0, group

        def settle():
            nonlocal tile, kpos
            while self.sums and kpos >= nk and tile < ntiles:
                if tile >= 2 and self.planted != "rs" and not (yield self.wait(self.accfull[c][tile & 1], tile // 2 - 1)):
                    return False
                if self.busy(("rs", c), tile & 1):
                    raise Hazard(f"row sums of tile {tile} overwrite a tile that the tensor core reads")
                self.rs[c][tile & 1][unit] = (tile, True)
                self.rs_full[tile & 1].arrive()
                tile += 1
                kpos -= nk
            return True

        if not (yield from settle()):
            return
        for k in range(group, len(operands) * nk, self.G):
            r, s, want = k % self.R, k % self.S, (operands[k // nk], k % nk)
            if not (yield self.wait(self.raw_full[c][r], k // self.R)):
                return
            if self.raw[c][r] != (want, True):
                raise Hazard(f"unpack of {want} reads raw[{r}] of CTA {c} holding {self.raw[c][r]}")
            if k >= self.S and not (yield self.wait(self.empty[c][s], k // self.S - 1)):
                return
            if self.busy(("stage", c), s):
                raise Hazard(f"unpack of {want} writes stage {s} of CTA {c} while the tensor core reads it")
            self.stage[c][s][part] = (want, False)
            self.raw_left[c][r] -= 1
            self.raw_empty[c][r].arrive()
            yield ("step", None, None)  # the stores into tensor memory take time
            if self.busy(("stage", c), s):
                raise Hazard(f"the tensor core reads stage {s} of CTA {c} while the unpack of {want} writes it")
            self.stage[c][s][part] = (want, True)
            self.a_full[s].arrive()
            if self.sums:
                kpos += self.G
                if not (yield from settle()):
                    return

    def issuer(self):
        nk, S, SW = self.nk, self.S, self.SW
        ar = a0 = it = dit = 0
        nstage = nacc = finished = 0
        nw, nd = [0, 0], [0, 0]  # of each resident W (or ring: the first), of each digit slot
        w_at, d_at = [0, 0], [0, 0]
        for n, t in enumerate(self.tiles):
            fresh, last = t.first_of_w(n, self.sets), t.last_of_w(len(self.tiles) - n, self.sets)
            if self.planted == "release":
                last = self.sets < t.npass or t.tp + 2 == t.ntp
            new_a = t.first_of_a(self.share, n == 0)
            last_a = t.last_of_a(self.share, n + 1 == len(self.tiles))
            odd, ab = t.ps & 1, n & 1
            if new_a:
                a0 = ar
            else:
                ar = a0
            if fresh:
                w_at[odd], d_at[odd] = (0 if self.stream else it % SW), dit % 2
            w0, ds = w_at[odd], d_at[odd]
            if n >= 2 and not (yield self.wait(self.accempty[ab], n // 2 - 1)):
                break
            if fresh:
                if not (yield self.wait(self.d_full[0][ds], dit // 2)):
                    break
                if not (yield self.wait(self.d_peer[ds], dit // 2)):
                    break
                dit += 1
            if n >= 2 and any(n - 2 not in self.acc_read[c] for c in (0, 1)):
                raise Hazard(f"tile {n} overwrites an accumulator that was not read")

            def offset():
                self.issue([("dslot", ds, t.w)] + ([("rs", ab, n)] if self.sums else []), n)
                if last:
                    self.commit([self.d_empty[0][ds], self.d_empty[1][ds]])
                return int(last)

            if not self.sums:
                late = offset()
                nd[ds] += 0 if self.planted == "count" else late
            ok = True
            for ks in range(nk):
                reload, release = fresh or self.stream, last or self.stream
                sw = it % SW if self.stream else w0 + ks
                if reload:
                    ok = (yield self.wait(self.w_full[0][sw], it // SW)) and (yield self.wait(self.w_peer[sw], it // SW))
                    if not ok:
                        break
                s = ar % S
                if new_a:
                    ok = yield self.wait(self.a_full[s], ar // S)
                    if not ok:
                        break
                self.issue([("stage", s, (t.a, ks)), ("wslot", sw, (t.w, ks))], n)
                if last_a:
                    self.commit([self.empty[0][s], self.empty[1][s]])
                    nstage += 1
                if release:
                    self.commit([self.w_empty[0][sw], self.w_empty[1][sw]])
                    nw[int(w0 > 0)] += 1
                it += int(reload)
                ar += 1
            if not ok:
                break
            if self.sums:
                if not (yield self.wait(self.rs_full[ab], n // 2)):
                    break
                nd[ds] += offset()
            elif self.planted == "count":
                nd[ds] += late
            self.commit([self.accfull[0][ab], self.accfull[1][ab]])
            nacc += 1
            finished += 1
        cut = int(finished < len(self.tiles) and self.planted != "cut")
        if cut:
            self.commit(self.cut_done)
            assert self.cut_commits(finished, sum(nw), sum(nd)) == (nw[1], nd[1])
        self.counts = (nstage, nw, nd, nacc, cut)
        yield from self.drain(0)

    def cut_commits(self, cut, nw, nd):
        """The kernel's walk over the tiles: from the totals, the commits on the second
        resident W and on the second digit slot."""
        it = dit = w = d = w1 = d1 = 0
        w_at, d_at = [0, 0], [0, 0]
        for n, t in enumerate(self.tiles[:cut + 1]):
            odd = t.ps & 1
            if t.first_of_w(n, self.sets):
                w_at[odd], d_at[odd] = it % self.SW, dit % 2
                it, dit = it + self.nk, dit + 1
            last = t.last_of_w(len(self.tiles) - n, self.sets)
            tw, td = (nw - w, nd - d) if n == cut else (self.nk * last, int(last))
            w, d = w + tw, d + td
            w1 += tw if self.SW >= self.nk and w_at[odd] else 0
            d1 += td if d_at[odd] else 0
        return w1, d1

    def drain(self, c):
        nstage, nw, nd, nacc, cut = self.counts
        if cut:
            yield ("drain", self.cut_done[c], 0)
        for q in range(max(0, nstage - self.S), nstage):
            yield ("drain", self.empty[c][q % self.S], q // self.S)
        if not cut or self.planted == "rounds":  # the releases run through the rings in rounds
            for bars, n, ring in ((self.w_empty[c], sum(nw), self.SW), (self.d_empty[c], sum(nd), 2)):
                for q in range(max(0, n - ring), n):
                    yield ("drain", bars[q % ring], q // ring)
        else:
            ring = min(self.SW, self.nk)
            for w in (0, 1):
                for q in range(max(0, nw[w] - ring), nw[w]):
                    yield ("drain", self.w_empty[c][w * ring + q % ring], q // ring)
                if nd[w]:
                    yield ("drain", self.d_empty[c][w], nd[w] - 1)
        for q in range(max(0, nacc - 2), nacc):
            yield ("drain", self.accfull[c][q % 2], q // 2)

    def epilogue(self, c):
        for n in range(len(self.tiles)):
            if not (yield self.wait(self.accfull[c][n & 1], n // 2)):
                return
            if self.acc_tile_done.get(n, 0) != 1 + self.nk:
                raise Hazard(f"CTA {c} reads tile {n} with {self.acc_tile_done.get(n, 0)} of {1 + self.nk} MMAs done")
            yield ("step", None, None)
            self.acc_read[c].add(n)
            self.accempty[n & 1].arrive()

    def explore(self, inorder=True, fail=None):
        roles = {"MMA": self.issuer(), "relay": self.relay()}
        for c in (0, 1):
            roles.update({f"E{c}": self.e_producer(c), f"W{c}": self.w_producer(c), f"epi{c}": self.epilogue(c),
                          f"unpack{c}0": self.unpack(c, 0), f"unpack{c}1": self.unpack(c, 1)})
        peer = None if self.planted == "peer" else lambda: {"exit": self.drain(1)}
        return drive(self, roles, self.rng, inorder, fail, peer)


ROLES = ["MMA", "relay"] + [r + str(c) for c in (0, 1) for r in ("E", "W", "epi")] + \
    [f"unpack{c}{u}" for c in (0, 1) for u in (0, 1)]


def _range(rng, table, limit):
    """A cluster's share of a launch: up to `limit` tiles from anywhere."""
    tiles = tiles_of(table)
    n = rng.randint(1, min(limit, len(tiles)))
    first = rng.randint(0, len(tiles) - n)
    return tiles[first:first + n]


def _table(rng, two_pass):
    return [(rng.choice((1, 2, 3) if two_pass else (1, 3, 1)), rng.randint(1, 4), rng.randint(1, 3))
            for _ in range(rng.randint(1, 4))]


def _planned(bflib):
    """Every distinct layout the planner gives: its sizes (K stages per tile up to 5,
    rings kept) and whether the launch has row sums."""
    out = set()
    for D in (8, 128, 256, 384, 512, 640, 1024, 2048):
        for nb in range(24, 97, 8):
            for two_pass in (False, True):
                for groups in (1, 2) if nb > 64 else (2,):
                    p = bflib.plan_pair(D, nb, two_pass, groups)
                    assert p is not None, (D, nb, two_pass, groups)
                    out.add((p["stages"], p["wslots"], p["raw"], p["sets"], p["share"], p["nk"], groups, nb > 64, two_pass))
    return sorted(out)


def test_every_planned_layout_passes_the_model(bflib):
    """Random ranges of random tables under random schedules, commits in and out of
    order, and with one role's wait giving up."""
    layouts = _planned(bflib)
    assert len(layouts) >= 40
    failed = 0
    for S, SW, R, sets, share, nk, groups, sums, two_pass in layouts:
        key = (S, SW, R, sets, share, nk, groups, sums, two_pass)
        for seed in range(10 if nk <= 4 else 4):
            for fail in (False, True):
                rng = random.Random(_seed(*key, seed, fail))
                m = Pair(_range(rng, _table(rng, two_pass), 14 if nk <= 4 else 6), S, SW, R, sets, share, nk, groups, sums,
                         rng)
                failed += m.explore(inorder=bool(seed % 2),
                                    fail=(rng.choice(ROLES), rng.randint(1, 10)) if fail else None)
    assert failed > 200


# sizes that make the rings and the rounds short: S, SW, R, sets, share, nk, groups, sums
SMALL = {
    "one stage a tile, W of two passes": (2, 2, 2, 2, 0, 1, 2, True),
    "shared operand": (4, 4, 2, 2, 1, 2, 2, False),
    "shared operand, no spare stage": (4, 8, 4, 2, 1, 4, 2, False),
    "W of one pass": (2, 3, 4, 1, 0, 3, 2, True),
    "W a ring": (2, 2, 4, 2, 0, 3, 2, True),
    "one group": (2, 2, 3, 1, 0, 2, 1, True),
    "one group, W of two passes": (2, 4, 3, 2, 0, 2, 1, True),
    "narrow, no sums": (6, 1, 2, 1, 0, 1, 2, False),
}


@pytest.mark.parametrize("name", sorted(SMALL))
@pytest.mark.parametrize("inorder", [True, False])
def test_small_rings(name, inorder):
    for seed in range(120):
        rng = random.Random(_seed(name, inorder, seed))
        Pair(_range(rng, _table(rng, True), 16), *SMALL[name], rng).explore(inorder)


@pytest.mark.parametrize("name", sorted(SMALL))
@pytest.mark.parametrize("inorder", [True, False])
def test_one_role_gives_up(name, inorder):
    """One role's wait gives up, the others at later polls: nothing is left to land,
    and no MMA to run, when the CTAs have gone."""
    failed = 0
    for seed in range(150):
        rng = random.Random(_seed("fail", name, inorder, seed))
        m = Pair(_range(rng, _table(rng, True), 10), *SMALL[name], rng)
        failed += m.explore(inorder, (rng.choice(ROLES), rng.randint(1, 12)))
    assert failed > 50


@pytest.mark.parametrize("planted,name,fails", [
    ("relay", "W of one pass", False),         # the peer tells the leader before its W has landed
    ("rs", "one stage a tile, W of two passes", False),  # row sums written over a tile still in use
    ("release", "shared operand", False),      # W given back a tile too early
    ("peer", "W of one pass", False),          # the peer leaves without waiting for its commits
    ("count", "narrow, no sums", True),        # the offset MMA's commit counted at the end of the tile
    ("cut", "shared operand", True),           # no commit behind the MMAs of a tile that ends early
    ("rounds", "shared operand", True),        # W's commits waited for in ring order, odd pass first or not
])
def test_the_model_finds(planted, name, fails):
    for seed in range(400):
        rng = random.Random(_seed(planted, seed))
        tiles = _range(rng, _table(rng, True), 16) if planted != "rounds" else tiles_of([(2, 3, 2)])[1:]
        m = Pair(tiles, *SMALL[name], rng)
        m.planted = planted
        fail = ("MMA" if rng.random() < 0.5 else rng.choice(ROLES), rng.randint(1, 12)) if fails else None
        try:
            m.explore(inorder=False, fail=fail)
        except AssertionError:
            return
    raise AssertionError("the planted mistake was not found")


@pytest.mark.parametrize("S,R", [(2, 3), (3, 4)])
def test_the_model_finds_rings_that_change_groups(S, R):
    """A raw slot or a stage that passes from one group to the other."""
    for seed in range(400):
        rng = random.Random(seed)
        try:
            Pair(_range(rng, _table(rng, False), 16), S, 2, R, 1, 0, 2, 2, True, rng).explore(inorder=False)
        except Hazard:
            return
    raise AssertionError("the odd ring was not found")


SMEM_PER_CTA = 232448  # 227 KiB opt-in per block


def test_every_planned_layout_fits_the_hardware(bflib):
    """Shared memory, tensor-memory columns that do not overlap, rings that keep a slot
    with one unpack group, and resident passes that the slots hold."""
    for D in (8, 64, 128, 192, 384, 512, 1000, 1024, 2048):
        for nb in range(24, 97, 8):
            for two_pass in (False, True):
                for groups in (1, 2) if nb > 64 else (2,):
                    p = bflib.plan_pair(D, nb, two_pass, groups)
                    what = (D, nb, two_pass, groups, p)
                    assert p["smem_bytes"] <= SMEM_PER_CTA, what
                    assert p["stages"] >= 2 and p["stages"] % groups == 0 and p["raw"] >= 2 and p["raw"] % groups == 0, what
                    assert p["raw"] <= 16 and p["stages"] <= 8, what
                    n, acc2, per = p["acc_cols"], p["acc2_col"], p["stages_per_acc"]
                    assert n >= 2 * nb and n % 32 == 0 and n <= acc2 and acc2 + n <= p["tmem_cols"] == 512, what
                    starts = [(n if i < per else acc2 + n) + 64 * (i % per) for i in range(p["stages"])]
                    used = sorted([(0, n), (acc2, acc2 + n)] + [(a, a + 64) for a in starts])
                    assert all(a[1] <= b[0] for a, b in zip(used, used[1:])) and used[-1][1] <= 512, what
                    assert p["stages"] <= 2 * per and p["stage_end_col"] == max(starts) + 64, what
                    if p["wslots"] >= p["nk"]:
                        assert p["wslots"] in (p["nk"], 2 * p["nk"]) and p["sets"] == p["wslots"] // p["nk"], what
                    else:
                        assert p["wslots"] >= 2 and p["sets"] == 2, what
                    if p["share"]:
                        assert two_pass and nb <= 64 and p["nk"] <= p["stages"], what


def test_planner_refuses_what_no_pair_launch_runs(bflib):
    assert bflib.plan_pair(512, 16) is None  # two CTAs on each SM instead
    assert bflib.plan_pair(512, 104) is None  # no tensor memory for two stages
    assert bflib.plan_pair(512, 64, groups=1) is None  # row sums only beside passes wider than 64 beams
    assert bflib.plan_pair(4096, 96) is None


# ------------------------------------------------- the one-CTA kernel's row sums


class OneCtaSums(Model):
    """The one-CTA model where the unpack groups leave row sums for the offset MMA,
    which then comes last (passes of more than 16 beams)."""

    def __init__(self, *a, **k):
        super().__init__(*a, **k)
        self.rs_full = [Barrier(f"rs_full{i}", self.G) for i in range(2)]
        self.rs = [None, None]
        self.rs_parts = [set(), set()]

    def unpack(self, g):
        tile, kpos = 0, g

        def settle():
            nonlocal tile, kpos
            while kpos >= self.nk and tile < self.nt:
                if tile >= 2 and not (yield self.wait(self.accfull[tile & 1], tile // 2 - 1)):
                    return False
                if self.busy("rs", tile & 1):
                    raise Hazard(f"row sums of tile {tile} overwrite a tile that the tensor core reads")
                if self.rs[tile & 1] != (tile, False):
                    self.rs[tile & 1], self.rs_parts[tile & 1] = (tile, False), set()
                self.rs_parts[tile & 1].add(g)
                if len(self.rs_parts[tile & 1]) == self.G:
                    self.rs[tile & 1] = (tile, True)
                self.rs_full[tile & 1].arrive()
                tile += 1
                kpos -= self.nk
            return True

        if not (yield from settle()):
            return
        for k in range(g, self.total, self.G):
            r, s = k % self.R, k % self.S
            if not (yield self.wait(self.raw_full[r], k // self.R)):
                return
            if self.raw[r] != (k, True):
                raise Hazard(f"unpack of sequence {k} reads raw[{r}] holding {self.raw[r]}")
            self.raw[r] = (("consumed", k), True)
            self.raw_empty[r].arrive()
            if k >= self.S and not (yield self.wait(self.empty[s], k // self.S - 1)):
                return
            if self.busy("stage", s):
                raise Hazard(f"unpack of sequence {k} writes TMEM stage {s} while the tensor core reads it")
            self.stage[s] = (k, False)
            yield ("step", None, None)
            self.stage[s] = (k, True)
            if not self.fwd:
                if k >= self.S:
                    self.w_empty[(k - self.S) % self.SW].arrive()
                if not (yield self.wait(self.w_full[k % self.SW], k // self.SW)):
                    return
            self.a_full[s].arrive()
            kpos += self.G
            if not (yield from settle()):
                return

    def mma_thread(self):
        k = nstage = ndig = nacc = 0
        for t in range(self.nt):
            ab = t % 2
            if t >= 2 and not (yield self.wait(self.accempty[ab], t // 2 - 1)):
                break
            if not (yield self.wait(self.d_full[ab], t // 2)):
                break
            if t >= 2 and (self.acc_reading[ab] is not None or t - 2 not in self.acc_read):
                raise Hazard(f"tile {t} overwrites accumulator {ab} before the epilogue has read tile {t - 2}")
            ok = True
            for _ in range(self.nk):
                s, sw = k % self.S, k % self.SW
                ok = yield self.wait(self.a_full[s], k // self.S)
                if not ok:
                    break
                self.mma([("stage", s, k), ("wslot", sw, k)], t)
                self.commit(self.empty[s])
                nstage += 1
                k += 1
            if not ok:
                break
            if not (yield self.wait(self.rs_full[ab], t // 2)):
                break
            self.mma([("dslot", ab, t), ("rs", ab, t)], t)
            self.commit(self.d_empty[ab])
            ndig += 1
            self.commit(self.accfull[ab])
            nacc += 1
        for bars, n, ring in ((self.empty, nstage, self.S), (self.d_empty, ndig, 2), (self.accfull, nacc, 2)):
            for q in range(max(0, n - ring), n):
                yield ("drain", bars[q % ring], q // ring)


def test_one_cta_layouts_with_row_sums(bflib):
    """Every layout of the one-CTA planner wider than 16 beams, with the row sums."""
    layouts = {}
    for D in (8, 128, 256, 512, 1024, 2048):
        for nb in range(24, 97, 8):
            for wslots, raw in ((0, 0), (4, 8), (2, 12)):
                p = bflib.plan_rings(D, nb, wslots, raw)
                layouts.setdefault((p["stages"], p["wslots"], p["raw"], p["groups"]), set()).add(min(p["nk"], 8))
    assert len(layouts) >= 8
    for (S, SW, R, groups), nks in sorted(layouts.items()):
        roles = ["E", "W", "MMA", "epi", "unpack0"] + (["unpack1", "fwd"] if groups > 1 else [])
        for nk in sorted(nks):
            for seed in range(12):
                rng = random.Random(_seed("sums", S, SW, R, groups, nk, seed))
                cfg = dict(S=S, SW=SW, R=R, groups=groups, nk=nk, ntiles=6, rng=rng)
                OneCtaSums(**cfg).run(inorder_commits=bool(seed % 2))
                OneCtaSums(**cfg).run(inorder_commits=bool(seed % 2), fail=(rng.choice(roles), rng.randint(1, 12)))
