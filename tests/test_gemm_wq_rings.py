"""The rings and barriers of the weight-only GEMM (csrc/gemm_wq_tc.cu) as a model on the host: every role is a generator, a scheduler
picks who goes on, copies land and matrix products retire when the scheduler says so.  A barrier answers as the hardware's does, by
the parity of its phase, so a wait that may look for a phase too early takes the one before for it, and the role then meets the wrong unit.

What is modelled: the rings of weights, activations and tensor-memory operands, the two sets of dequant warps (two warps each), one or
two issuing warps, one CTA or a pair, the accumulators and the epilogue, both forms (DEFER: the epilogue reads every unit), and the last tile that
stays in its accumulators until all warps finish it (EARLY: each CTA of a pair decides for itself).  What each slot holds is followed, and every read and overwrite is checked.  The ring sizes are those that the
library names for every row count and group, with activations staged and read in place."""
import ctypes
import os
import random

import pytest

from torchao_fork_b200 import _lib

if not os.path.exists(_lib.LIB_PATH):
    pytest.skip("libao_b200.so not built (python -m torchao_fork_b200.build)", allow_module_level=True)

A_SLOTS = 4   # of 128 k in tensor memory


def cut(m, np_, kp, group):
    """How the library cuts up a call (ao_b200_mm_plan; group 0: int8)"""
    c = _lib.MmCut()
    _lib.check(_lib.lib().ao_b200_mm_plan(m, np_, kp, group, ctypes.byref(c)), "mm_plan")
    return c


def plan(m, group, np_=16384):
    """The rings of a call of m rows"""
    c = cut(m, np_, 8192, group)
    return dict(w=c.weight_slots, x=c.activation_slots, a=c.operand_slots, n_mma=c.issuers, d=2 if c.rows_per_tile <= 128 else 1, defer=bool(c.defer),
                pair=bool(c.pair))


class Wrong(Exception):
    pass


class Barrier:
    def __init__(self, count):
        self.count = self.left = count
        self.phase = 0

    def arrive(self):
        self.left -= 1
        if self.left == 0:
            self.left, self.phase = self.count, self.phase + 1

    def over(self, parity):
        return self.phase % 2 != parity


class Ring:
    def __init__(self, n, start=0, use=0):
        self.n, self.slot, self.use = n, start, use
        while self.slot >= n:
            self.slot -= n
            self.use ^= 1

    def step(self, by):
        self.slot += by
        if self.slot >= self.n:
            self.slot -= self.n
            self.use ^= 1


WARPS = 2   # dequant warps per set (the kernel has 8: they do the same)
EPI = 2     # epilogue warps (the kernel has 4)


class Model:
    def __init__(self, rng, cfg, units, ku, first=0, a_first=None, early=False, early_before_products=False):
        self.rng, self.c, self.u0, self.u1, self.ku = rng, cfg, first, first + units, ku
        ranks = range(2 if cfg["pair"] else 1)
        self.ranks, self.lead = ranks, 0
        bars = lambda n, c: [[Barrier(c) for _ in range(n)] for _ in ranks]  # noqa: E731
        w, x, a, d = cfg["w"], cfg["x"], cfg["a"], cfg["d"]
        self.wfull, self.wempty = bars(w, 1), bars(w, WARPS + (EPI if cfg["defer"] else 0))
        self.xfull, self.xpeer, self.xdone, self.dread = bars(x, 1), bars(x, 1), bars(x, 1), bars(x, EPI)
        self.afull, self.adone = bars(a, WARPS * len(ranks)), bars(a, 1)
        self.dfull, self.dempty = bars(d, cfg["n_mma"]), bars(d, EPI * len(ranks))
        # contents: unit, and who may still read it
        self.wslot = [[None] * w for _ in ranks]
        self.wread = [[0] * w for _ in ranks]
        self.xslot = [[None] * x for _ in ranks]
        self.aslot = [[[None] * WARPS for _ in range(a)] for _ in ranks]
        self.abusy = [0] * a                    # products in flight on it
        self.xbusy = [0] * x
        self.dbuf = [[set() for _ in range(cfg["n_mma"])] for _ in range(d)]
        self.dslot = [None] * x                 # DEFER: accumulator per slot of x
        self.flying = []                        # copies in flight: any may land next
        self.queue = [[] for _ in range(cfg["n_mma"])]  # products and commits, in order per issuing warp
        # (wq_gemm_kernel: a_first)
        self.a_first = (w % 2 == 1 and w < a + 2) if a_first is None else a_first
        self.done_tiles = [[] for _ in ranks]
        # EARLY: the last tile is shared with the next CTA, whose share this rank finds there (by time, so at random), or does not
        self.stays = [early and not cfg["defer"] and self.u1 % ku != 0 and first <= self.u1 // ku * ku and rng.random() < 0.7 for _ in ranks]
        self.early_before_products, self.kept = early_before_products, [None for _ in ranks]

    def check(self, ok, what):
        if not ok:
            raise Wrong(what)

    # ---- roles
    def weights(self, r):
        w, full, empty = self.c["w"], self.wfull[r], self.wempty[r]

        def load(slot, u):
            def land():
                self.check(self.wread[r][slot] == 0, "weights overwritten while somebody reads them")
                self.wslot[r][slot], self.wread[r][slot] = u, WARPS + (EPI if self.c["defer"] else 0)
                full[slot].arrive()
            self.flying.append(land)
        for i in range(min(w, self.u1 - self.u0)):
            load(i, self.u0 + i)
        ring = Ring(w)
        ring.use = 1
        for u in range(self.u0 + w, self.u1):
            yield lambda: empty[ring.slot].over(ring.use ^ 1)
            load(ring.slot, u)
            ring.step(1)

    def rows(self, r):
        full, free = self.xfull[r], (self.dread if self.c["defer"] else self.xdone)[r]
        ring = Ring(self.c["x"])
        for u in range(self.u0, self.u1):
            yield lambda: free[ring.slot].over(ring.use ^ 1)

            def land(slot=ring.slot, u=u):
                self.check(self.xbusy[slot] == 0, "activations overwritten under a product")
                self.xslot[r][slot] = u
                full[slot].arrive()
            self.flying.append(land)
            ring.step(1)

    def peer(self):
        ring = Ring(self.c["x"])
        for u in range(self.u0, self.u1):
            yield lambda: self.xfull[1][ring.slot].over(ring.use)
            self.xpeer[0][ring.slot].arrive()
            ring.step(1)

    def issue(self, mw):
        c, n = self.c, self.c["n_mma"]
        x, a, d = Ring(c["x"], mw), Ring(c["a"], mw), Ring(c["d"])
        u = self.u0
        while u < self.u1:
            end, tile = min(self.u1, (u // self.ku + 1) * self.ku), u // self.ku
            if not c["defer"]:
                yield lambda: self.dempty[0][d.slot].over(d.use ^ 1)
                fresh = True
            if n == 2 and (u - self.u0) % 2 != mw:
                u += 1
            while u < end:
                yield lambda: self.afull[0][a.slot].over(a.use)
                yield lambda: self.xfull[0][x.slot].over(x.use)
                if c["pair"]:
                    yield lambda: self.xpeer[0][x.slot].over(x.use)
                xs, as_, ds = x.slot, a.slot, d.slot
                self.abusy[as_] += 1
                self.xbusy[xs] += 1

                def product(u=u, xs=xs, as_=as_, ds=ds, fresh=c["defer"] or fresh, mw=mw):
                    for r in self.ranks:
                        self.check(self.xslot[r][xs] == u, f"product {u} meets activations of {self.xslot[r][xs]}")
                        self.check(self.aslot[r][as_] == [u] * WARPS, f"product {u} meets weights of {self.aslot[r][as_]}")
                    if c["defer"]:
                        self.check(self.dslot[xs] is None, "an accumulator that nobody has read is written")
                        self.dslot[xs] = [u, EPI]
                    else:
                        if fresh:
                            self.dbuf[ds][mw].clear()
                        self.dbuf[ds][mw].add(u)
                    self.abusy[as_] -= 1
                    self.xbusy[xs] -= 1
                    for r in self.ranks:
                        self.adone[r][as_].arrive()
                        self.xdone[r][xs].arrive()
                self.queue[mw].append(product)
                fresh = False
                u += n
                x.step(n)
                a.step(n)
            u = end
            if not c["defer"]:
                if fresh:   # nothing of this tile: whatever the buffer holds is not looked at
                    pass

                def commit(ds=d.slot):
                    for r in self.ranks:
                        self.dfull[r][ds].arrive()
                self.queue[mw].append(commit)
                d.step(1)

    def dequant(self, r, s, warp):
        c = self.c
        w, a = Ring(c["w"], s), Ring(c["a"], s)

        def fetch(u):
            if u >= self.u1:
                return
            if self.a_first:
                yield lambda: self.adone[r][a.slot].over(a.use ^ 1)
            yield lambda: self.wfull[r][w.slot].over(w.use)
            self.check(self.wslot[r][w.slot] == u, f"dequant of {u} meets weights of {self.wslot[r][w.slot]}")
            self.wread[r][w.slot] -= 1
        u = self.u0 + s
        yield from fetch(u)
        while u < self.u1:
            self.wempty[r][w.slot].arrive()
            yield lambda: self.adone[r][a.slot].over(a.use ^ 1)
            self.check(r != 0 or self.abusy[a.slot] == 0, "operand overwritten under a product")
            self.aslot[r][a.slot][warp] = u
            full = self.afull[0][a.slot]
            w.step(2)
            a.step(2)
            if c["defer"] and not self.a_first:
                yield from fetch(u + 2)
            full.arrive()
            if not c["defer"] or self.a_first:
                yield from fetch(u + 2)
            u += 2

    def epilogue(self, r, warp):
        c = self.c
        d, x, w = Ring(c["d"]), Ring(c["x"]), Ring(c["w"])
        u, t = self.u0, self.u0 // self.ku
        while u < self.u1:
            end = min(self.u1, (t + 1) * self.ku)
            if c["defer"]:
                while u < end:
                    for bar, ring in ((self.wfull, w), (self.xfull, x), (self.xdone, x)):
                        yield lambda bar=bar, ring=ring: bar[r][ring.slot].over(ring.use)
                    self.check(self.wslot[r][w.slot] == u, "parameters of another unit")
                    self.check(self.xslot[r][x.slot] == u, "sums of another unit")
                    self.check(self.dslot[x.slot] is not None and self.dslot[x.slot][0] == u, "accumulator of another unit")
                    self.wread[r][w.slot] -= 1
                    self.dslot[x.slot][1] -= 1
                    if self.dslot[x.slot][1] == 0:
                        self.dslot[x.slot] = None
                    self.dread[r][x.slot].arrive()
                    self.wempty[r][w.slot].arrive()
                    x.step(1)
                    w.step(1)
                    u += 1
            else:
                last = self.stays[r] and end == self.u1
                if not (last and self.early_before_products):
                    yield lambda: self.dfull[r][d.slot].over(d.use)
                if last:   # the tile is left where it is: buffer and, with one unit, whose accumulator (as the kernel works them out at the end)
                    slot = (t - self.u0 // self.ku) % c["d"]
                    self.check(slot == d.slot, "another buffer than the epilogue's")
                    self.kept[r] = (slot, t * self.ku, end, (t * self.ku - self.u0) & 1)
                    break
                self.drained(d.slot, t, u, end, (u - self.u0) & 1)
                self.dempty[0][d.slot].arrive()
                d.step(1)
                u = end
            t += 1
        self.done_tiles[r].append(warp)

    def drained(self, slot, t, u, end, parity):
        n = self.c["n_mma"]
        two = n == 2 and end - u > 1
        got = set()
        for mw in ((0, 1) if two else (parity,) if n == 2 else (0,)):
            got |= self.dbuf[slot][mw]
        self.check(got == set(range(u, end)), f"tile {t} has units {got}, not {u} .. {end - 1}")

    def meet(self, r):
        # all warps of the CTA, as soon as each is through with its own part
        slot, u, end, parity = self.kept[r]
        self.drained(slot, u // self.ku, u, end, parity)

    def run(self):
        roles = [self.weights(r) for r in self.ranks] + [self.rows(r) for r in self.ranks] + [self.issue(m) for m in range(self.c["n_mma"])]
        roles += [self.dequant(r, s, k) for r in self.ranks for s in range(2) for k in range(WARPS)]
        roles += [self.epilogue(r, k) for r in self.ranks for k in range(EPI)]
        if self.c["pair"]:
            roles.append(self.peer())
        mine = {r: [g for g in roles if g.gi_frame.f_locals.get("r", 0 if g.gi_code.co_name != "peer" else 1) == r] for r in self.ranks}
        # a role's speed: now and then one of them, or a copy, is held back for long
        waits = {}
        for g in roles:
            try:
                waits[g] = next(g)
            except StopIteration:
                pass
        weight = {g: self.rng.choice([1, 1, 5, 40]) for g in roles}
        lazy_copies, lazy_products = self.rng.choice([1, 10, 60]), self.rng.choice([1, 10, 60])
        met = set()
        while waits or self.flying or any(self.queue):
            for r in self.ranks:   # the CTA's own roles are over (what its issuing warp has asked for may be under way)
                if self.kept[r] and r not in met and not any(g in waits for g in mine[r]):
                    met.add(r)
                    self.meet(r)
            ready = [g for g in waits if waits[g]()]
            choices = [(g, weight[g]) for g in ready]
            choices += [("copy", 40 / lazy_copies)] if self.flying else []
            choices += [(q, 40 / lazy_products) for q in range(len(self.queue)) if self.queue[q]]
            if not choices:
                raise Wrong("everybody waits")
            pick = self.rng.choices([k for k, _ in choices], [v for _, v in choices])[0]
            if pick == "copy":
                self.flying.pop(self.rng.randrange(len(self.flying)))()
            elif isinstance(pick, int):
                self.queue[pick].pop(0)()
            else:
                try:
                    waits[pick] = next(pick)
                except StopIteration:
                    del waits[pick]
        for r in self.ranks:
            self.check(len(self.done_tiles[r]) == EPI, "an epilogue warp did not finish")
            if self.kept[r]:
                self.meet(r)   # (nothing has written there since)


def _plans():
    seen = {}
    for group in (0, 32, 64, 128, 256):
        for m in list(range(1, 1030)) + [2048, 4096]:
            for np_ in (16384, 8192, 4096, 2048):   # above 8192 outputs activations are staged; from 512 rows on they are read in place up to 2048, 4096 or 8192
                c = plan(m, group, np_)
                seen.setdefault(tuple(sorted(c.items())), (m, group, c))
    return list(seen.values())


PLANS = _plans()


def test_plans_cover_short_odd_and_even_rings_one_and_two_issuers():
    kinds = {(c["w"] % 2, c["w"] < c["a"] + 2, c["n_mma"], c["defer"], c["pair"]) for _, _, c in PLANS}
    assert any(w and short for w, short, *_ in kinds) and any(not w and n == 2 for w, _, n, *_ in kinds)
    for _, _, c in PLANS:
        assert c["w"] >= 2 and 2 <= c["a"] <= max(c["w"], A_SLOTS) and (c["n_mma"] == 1 or (c["w"] % 2 == 0 and c["x"] % 2 == 0 and c["a"] % 2 == 0))


@pytest.mark.parametrize("m,group,cfg", PLANS, ids=[f"{m} rows, group {g}" for m, g, _ in PLANS])
def test_every_order_of_the_roles_keeps_units_apart(m, group, cfg):
    for seed in range(12):
        rng = random.Random(seed)
        ku = rng.choice([1, 2, 3, 5, 8, 64])
        Model(rng, cfg, rng.randint(1, 40), ku, first=rng.randint(0, 2 * ku)).run()


@pytest.mark.parametrize("m,group,cfg", [p for p in PLANS if not p[2]["defer"]], ids=[f"{m} rows, group {g}" for m, g, c in PLANS if not c["defer"]])
def test_a_last_tile_may_stay_in_its_accumulators(m, group, cfg):
    for seed in range(12):
        rng = random.Random(1000 + seed)
        ku = rng.choice([2, 3, 5, 8, 64])
        Model(rng, cfg, rng.choice([rng.randint(1, 40), ku + 1, 2 * ku + 1, ku + 2]), ku, first=rng.choice([0, 0, rng.randint(0, 2 * ku)]), early=True).run()


def _found(cfg, **kw):
    for seed in range(300):
        rng = random.Random(seed)
        try:
            Model(rng, cfg, 40, 64 if "early" not in kw else 9, **kw).run()
        except Wrong:
            return True
    return False


def test_the_model_sees_what_the_rules_prevent():
    # three weight slots without waiting for the operand slot first; an odd ring under two issuing warps
    short = dict(w=3, x=3, a=3, n_mma=1, d=1, defer=False, pair=True)
    assert _found(short, a_first=False) and not _found(short)
    assert _found(dict(w=5, x=8, a=4, n_mma=2, d=2, defer=False, pair=False), a_first=False)
    # a last tile that is taken without waiting for its products
    even = plan(64, 128)
    assert _found(even, early=True, early_before_products=True) and not _found(even, early=True)


def _first(c, worker):
    return (worker * c.base + min(worker, c.rem)) * c.quantum


SHAPES = [(m, np_, kp, g) for m in (1, 16, 17, 32, 33, 64, 100, 128, 129, 600, 5000) for np_ in (128, 256, 1024, 1152, 4096, 14336, 28672)
          for kp in (64, 128, 256, 512, 768, 1024, 1280, 1792, 2304, 2816, 3328, 4096, 4160, 9472, 16384) for g in (0, 128)]


def test_every_unit_is_dealt_to_one_worker():
    for m, np_, kp, g in SHAPES:
        c = cut(m, np_, kp, g)
        ku = -(-kp // c.unit_k)   # (small weights: up to an eighth more, of zeros, so that owners divide them)
        assert ku <= c.units_per_tile <= ku + (ku + 7) // 8 * (c.unit_k == 256) and c.row_tiles * c.rows_per_tile >= m
        assert c.tiles == c.row_tiles * -(-np_ // (256 if c.pair else 128))
        assert 1 <= c.workers <= 148 // (2 if c.pair else 1) and _first(c, 0) == 0 and _first(c, c.workers) == c.tiles * c.units_per_tile
        assert c.base >= 1   # nobody goes without: the roles of a worker without units would wait for each other


def test_small_weights_are_cut_at_the_ends_of_tiles():
    """Fewer than four units of 256 k for each SM, and up to 16 in a tile: a worker's units are all of one tile"""
    met = 0
    for m, np_, kp, g in SHAPES:
        c = cut(m, np_, kp, g)
        sms = 148 // (2 if c.pair else 1)
        if c.unit_k != 256 or kp > 4096 or c.tiles > sms or c.tiles * -(-kp // 256) >= 4 * sms:
            continue
        ku, met = c.units_per_tile, met + 1
        assert all(_first(c, i) // ku == (_first(c, i + 1) - 1) // ku for i in range(c.workers)), (m, np_, kp, g)
    assert met > 400


@pytest.mark.parametrize("group,np_,tiles", [(0, 2048, (176, 208, 224, 240, 256)), (0, 2176, (224, 240, 256)), (0, 4096, (224, 240, 256)), (0, 4224, (240, 256)),
                                             (0, 8192, (240, 256)), (128, 4096, (176, 208, 224, 240, 256)), (128, 8192, (208, 224, 240, 256)), (128, 8320, ())])
def test_activations_are_read_in_place_where_the_products_of_a_tile_cover_the_turn(group, np_, tiles):
    for m in (511, 513, 528, 600, 640, 700, 768, 800, 1000, 1040, 2048):
        c = cut(m, np_, 4096, group)
        assert bool(c.in_place) == (m >= 512 and c.rows_per_tile in tiles), m
