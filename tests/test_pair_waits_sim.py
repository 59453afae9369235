"""The waits of the pair kernel (csrc/pair.cuh), replayed on the CPU: per cluster the scheduler, the weight producer, the
activations, the MMA issuer and the four groups of decode warps, each walking the units it is handed in the order of the
kernel and standing still until what it waits for has happened. Units are drawn from one counter by clusters that run at
different speeds or start late. Ring sizes and the rule when accumulators are drained are compiled from the kernel's own
header (csrc/pair_sched.h). Checked: every cluster reaches the end of the list, for any number of token tiles, any reduction
length and any number of clusters.

What a role waits for only ever becomes true, so with the same units drawn the order in which the roles run decides nothing;
what varies is which cluster draws which unit. The two CTAs of a cluster run the same program and wait for the same events:
one stands for both."""
import ctypes
import os
import random
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "muse-spark-kernels_b200", "csrc")
NAMES = ("PAIR_BH", "PAIR_SLOT_K", "PAIR_NSLOT", "PAIR_GROUPS", "PAIR_NST", "PAIR_UNITS", "PAIR_MARKS")


@pytest.fixture(scope="module")
def sched(tmp_path_factory):
    d = tmp_path_factory.mktemp("pair_sched")
    src, so = d / "shim.cpp", d / "shim.so"
    src.write_text('#include "pair_sched.h"\nextern "C" {\n'
                   "int tile_rows(int c, int n) { return msk::pair_tile_rows(c, n); }\n"
                   "int b_waits_for(int s, int c, int w) { return (int)msk::pair_b_waits_for(s, c, w); }\n"
                   "int b_place(int s, int c) { return (int)msk::pair_b_place(s, c); }\n"
                   "int cols(int rows) { return msk::pair_cols(rows); }\n"
                   "int before_drain(int a, int b, int c, int d) { return msk::pair_slots_before_drain(a, b, c, d); }\n"
                   + "".join(f"int c_{n}() {{ return msk::{n}; }}\n" for n in NAMES) + "}\n")
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-I", CSRC, "-o", str(so), str(src)], check=True)
    return ctypes.CDLL(str(so))


class Cluster:
    """One cluster; unit: (phase, tile, columns, slots). Slots are numbered through all units."""

    def __init__(self, c, deal, before_drain, b_waits_for):
        self.c, self.deal, self.before_drain, self.b_waits_for = c, deal, before_drain, b_waits_for
        self.units = []                 # as handed out, the end marker last
        self.first = []                 # number of each unit's first slot
        self.slots = 0                  # slots of the units handed out
        self.announced = 0              # units whose stores were announced (or need not be)
        self.done = False
        self.act_unit = self.act_slots = 0              # activations: unit walked, slots filled,
        self.wide_end = 0                               # number behind the last stage of a wide tile
        self.raw_unit = self.raw_stages = 0             # weights: unit walked, stages issued
        self.mma_unit = self.mma_slots = 0              # MMAs: unit walked, slots read and handed back
        G = c["PAIR_GROUPS"]
        self.dec_unit = [0] * G                         # decode groups: unit walked,
        self.filled = [0] * G                           # slots filled,
        self.drained = [0] * G                          # units drained
        self.ahead = [None] * G                         # slots to fill before the owed unit is drained
        self.bufs, self.next_buf = [], 0                # accumulator buffers of each unit
        self.roles = [self.schedule, self.produce, self.activate, self.mma] + [lambda g=g: self.decode(g) for g in range(G)]

    def slot_filled(self, n):
        G = self.c["PAIR_GROUPS"]
        return self.filled[n % G] > n // G

    def schedule(self):
        """Hands out the next unit once its place in the list is free; announces stored gate/up units in order on the way."""
        if self.done:
            return False
        i, U = len(self.units), self.c["PAIR_UNITS"]
        if i >= U:
            old = i - U                                 # the unit whose place this one takes
            if min(self.drained) <= old or min(self.act_unit, self.raw_unit, self.mma_unit) < old:
                return False
        while i >= U and self.announced <= i - U:
            self.announce()
        u = self.deal.draw()
        self.units.append(u)
        self.first.append(self.slots)
        self.slots += u[3] if u else 0
        self.done = u is None
        return True

    def announce(self):
        u = self.units[self.announced]
        if u and u[0] == 0:
            self.deal.stored[u[1]] += 1
        self.announced += 1

    def tail(self):
        """Behind the end of the list the stores of the last gate/up units are announced as they are made."""
        while self.done and self.announced < len(self.units) - 1 and min(self.drained) > self.announced:
            self.announce()

    def produce(self):
        if self.raw_unit >= len(self.units) or self.units[self.raw_unit] is None:
            return False
        n = self.raw_stages - self.c["PAIR_NST"]        # the stage whose place the next one takes
        if n >= 0 and not (self.slot_filled(2 * n) and self.slot_filled(2 * n + 1)):
            return False
        self.raw_stages += 1
        if 2 * self.raw_stages == self.first[self.raw_unit] + self.units[self.raw_unit][3]:
            self.raw_unit += 1
        return True

    def activate(self):
        if self.act_unit >= len(self.units) or self.units[self.act_unit] is None:
            return False
        phase, tile, cols, nsl = self.units[self.act_unit]
        if phase == 1 and self.act_slots == self.first[self.act_unit] and not self.deal.complete(tile):
            return False
        if self.b_waits_for(self.act_slots // 2, cols, self.wide_end) >= self.mma_slots:
            return False
        self.act_slots += 2                             # a stage, two slots, at a time
        if self.act_slots == self.first[self.act_unit] + nsl:
            self.act_unit += 1
            if cols > self.c["PAIR_BH"]:
                self.wide_end = self.act_slots // 2
        return True

    def mma(self):
        i = self.mma_unit
        if i >= len(self.units) or self.units[i] is None:
            return False
        if self.mma_slots == self.first[i]:             # the accumulators have to be drained by every group
            if i == len(self.bufs):
                self.bufs.append(self.take(self.units[i][2]))
            last = max((j for j in range(max(0, i - 2), i) if self.bufs[j] & self.bufs[i]), default=-1)
            if min(self.drained) <= last:
                return False
        n = self.mma_slots                              # a stage, two slots, at a time
        if not (self.act_slots >= n + 2 and self.slot_filled(n) and self.slot_filled(n + 1)):
            return False
        self.mma_slots += 2
        if self.mma_slots == self.first[i] + self.units[i][3]:
            self.mma_unit += 1
        return True

    def take(self, cols):
        """Accumulator buffers of the next unit: one of two in turn, or both (PairBuffers)."""
        wide = cols > self.c["PAIR_BH"]
        used = {0, 1} if wide else {self.next_buf}
        self.next_buf = 0 if wide else self.next_buf ^ 1
        return used

    def decode(self, g):
        i, G = self.dec_unit[g], self.c["PAIR_GROUPS"]
        if i >= len(self.units):
            return False
        u = self.units[i]
        nsl = u[3] if u else 0
        n = self.filled[g] * G + g                      # this group's next slot
        has_slot = n < self.first[i] + nsl
        owes = self.drained[g] < i
        if self.ahead[g] is None:
            o = self.units[i - 1] if i else (0, 0, 0, 0)
            self.ahead[g] = self.before_drain(o[0], o[2], u[0] if u else -1, u[2] if u else 0)
        if owes and (not has_slot or self.ahead[g] <= 0):
            if self.mma_unit < i:                       # the MMAs of the owed unit
                return False
            self.drained[g] += 1
            return True
        if has_slot:
            if self.raw_stages <= n // 2 or n - self.c["PAIR_NSLOT"] >= self.mma_slots:
                return False
            self.filled[g] += 1
            self.ahead[g] -= 1
            return True
        if u is None:
            return False
        self.dec_unit[g] += 1
        self.ahead[g] = None
        return True

    def run(self, budget, draws):
        """Up to `budget` steps of each role in turn and up to `draws` units drawn; False when none of them can move."""
        moved = False
        for role in self.roles:
            for _ in range(draws if role == self.schedule else budget):
                if not role():
                    break
                moved = True
        before = self.announced
        self.tail()
        return moved or self.announced != before

    def finished(self):
        return self.done and min(self.drained) == len(self.units) - 1 and self.announced == len(self.units) - 1


class Deal:
    """The counter that units are drawn from, and the gate/up units stored per tile."""

    def __init__(self, c, tiles, H, inter):
        self.n_pairs = (inter // 128, H // 256)
        self.order = [(phase, t, cols, (H, inter)[phase] // c["PAIR_SLOT_K"])
                      for phase in (0, 1) for t, cols in enumerate(tiles) for _ in range(self.n_pairs[phase])]
        self.at = 0
        self.stored = [0] * len(tiles)

    def draw(self):
        self.at += 1
        return self.order[self.at - 1] if self.at <= len(self.order) else None

    def complete(self, tile):
        return self.stored[tile] == self.n_pairs[0]


def ends(c, before_drain, b_waits_for, tiles, H, inter, clusters, seed):
    """True when every cluster reaches the end of the list. seed 0: all clusters at one speed, drawing in turn; others: each
    at a speed of its own, some starting late."""
    rng = random.Random(seed)
    deal = Deal(c, tiles, H, inter)
    cl = [Cluster(c, deal, before_drain, b_waits_for) for _ in range(clusters)]
    speed = [2 if seed == 0 else rng.choice((1, 2, 4, 8)) for _ in cl]
    draws = [1 if seed == 0 else rng.choice((1, 1, 2, 4)) for _ in cl]
    late = [0 if seed == 0 else rng.choice((0, 0, 1, 5, 40)) for _ in cl]
    tick = 0
    alive = list(range(clusters))
    while alive:
        moved = False
        for i in alive:
            if late[i] <= tick:
                moved |= cl[i].run(speed[i], draws[i])
        if not moved and all(late[i] <= tick for i in alive):
            return False
        alive = [i for i in alive if not cl[i].finished()]
        tick += 1
    return True


def old_rule(c):
    """Without regard to phases: the rule the kernel must not have."""
    return lambda owed_phase, owed_cols, phase, cols: 1 if max(cols, owed_cols) > c["PAIR_BH"] else 2


def _constants(sched):
    return {n: getattr(sched, "c_" + n)() for n in NAMES}


def _tiles(kind, n, seed):
    rng = random.Random(seed)
    return [{"narrow": 64, "wide": 256}.get(kind) or rng.choice((16, 48, 64, 112, 128, 144, 240, 256)) for _ in range(n)]


@pytest.mark.parametrize("H,inter,clusters", [(4096, 256, 74), (4096, 512, 74), (4096, 768, 74), (4096, 1536, 74), (4096, 4096, 74),
                                              (7168, 2048, 74), (2048, 1024, 74), (256, 768, 74), (2048, 14336, 37), (4096, 1536, 1),
                                              (1024, 4096, 2), (4096, 1536, 19)])
def test_every_cluster_reaches_the_end(sched, H, inter, clusters):
    c = _constants(sched)
    counts = (1, 2, 3, 4, 6, 8) if inter > 4096 else (1, 2, 3, 4, 5, 6, 8, 10, 13, 20, 40)
    for n in counts:
        for kind in ("narrow", "wide", "mixed"):
            for seed in range(1 if n > 8 else 3):
                assert ends(c, sched.before_drain, sched.b_waits_for, _tiles(kind, n, n + seed), H, inter, clusters, seed), (n, kind, seed)


@pytest.mark.parametrize("H,inter,clusters,tiles,seeds", [(4096, 1536, 74, 4, 1), (4096, 1536, 74, 5, 1), (4096, 1536, 74, 6, 1),
                                                          (4096, 4096, 74, 2, 1), (7168, 2048, 74, 4, 1), (4096, 1536, 1, 1, 1),
                                                          (4096, 1536, 74, 8, 12), (2048, 1024, 74, 8, 12)])
def test_the_model_sees_a_drain_behind_the_down_units_mmas(sched, H, inter, clusters, tiles, seeds):
    """Not vacuous: with the drain always behind the second slot of narrow tiles the same loads stand still."""
    c = _constants(sched)
    assert not all(ends(c, old_rule(c), sched.b_waits_for, [64] * tiles, H, inter, clusters, seed) for seed in range(seeds))


def overwrites_only_read_rows(c, sched, waits_for):
    """The ring of token rows, place by place, over units of random widths: whether, when a stage's copy starts, the MMAs of every stage that
    last used one of its places are done (MMAs are done in order), and the barrier waited for has not come round again."""
    for seed in range(40):
        rng = random.Random(seed)
        user = [-1] * c["PAIR_NSLOT"]
        stage = wide_end = 0
        for _ in range(60):
            cols = sched.cols(rng.randint(129, 256) if rng.random() < (0.5, 0.1, 0.9)[seed % 3] else rng.randint(1, 128))
            wide = cols > c["PAIR_BH"]
            for _ in range(rng.choice((1, 1, 2, 3, 5, 8))):
                at = sched.b_place(stage, cols)
                places = (at, at + 1) if wide else (at,)
                # the four sub-tiles of 64 K, 128 bytes a row, fit what the stage takes
                assert places[-1] < c["PAIR_NSLOT"] and 4 * 128 * (cols // 2) <= len(places) * c["PAIR_BH"] * 2 * c["PAIR_SLOT_K"]
                waits = waits_for(stage, cols, wide_end)
                if max(user[p] for p in places) >= 0 and 2 * max(user[p] for p in places) + 1 > waits:
                    return False
                if not 2 * stage - c["PAIR_MARKS"] <= waits < 2 * stage:
                    return False
                for p in places:
                    user[p] = stage
                stage += 1
            if wide:
                wide_end = stage
    return True


def test_token_rows_overwrite_only_what_the_mmas_have_read(sched):
    """With the places and the waits of the kernel's own header; and the replay sees waits that are too short."""
    c = _constants(sched)
    assert overwrites_only_read_rows(c, sched, sched.b_waits_for)
    narrow = lambda cols: cols <= c["PAIR_BH"]  # noqa: E731
    assert not overwrites_only_read_rows(c, sched, lambda s, cols, w: 2 * (s - (4 if narrow(cols) else 2)) + 1)     # no regard to wide tiles before
    assert not overwrites_only_read_rows(c, sched, lambda s, cols, w: sched.b_waits_for(s, cols, w) - 1)             # a stage's first slot
    assert not overwrites_only_read_rows(c, sched, lambda s, cols, w: sched.b_waits_for(s, cols, max(w - 1, 0)))     # a stage too early


def test_the_kernel_takes_places_and_waits_from_the_header():
    """Copies and MMAs both ask pair_b_place, and the copies wait for pair_b_waits_for as it stands."""
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "pair.cuh")).read())
    assert len(re.findall(r"\bpair_b_place\(st, u\.nmma\) \* C::B_SLOT_BYTES", src)) == src.count("pair_b_place(") == 2
    assert re.findall(r"before = (pair_b_waits_for\([^;]*);\s*if \(!mbar_wait_inline\(&ctl\.empty\[before & 7u\], \(before >> 3\) & 1u", src) == ["pair_b_waits_for(st, u.nmma, wide_end)"]


def test_columns_are_whole_rows_of_either_cta(sched):
    for rows in range(1, 257):
        cols = sched.cols(rows)
        assert rows <= cols < rows + 16 and cols % 16 == 0 and cols <= 256


def test_tile_rows_share_an_expert_evenly(sched):
    c = _constants(sched)
    top = 2 * c["PAIR_BH"]
    for rows in range(1, 3 * top + 70):
        n = -(-rows // top)
        per = sched.tile_rows(rows, n)
        shares = [min(per, rows - i * per) for i in range(n)]
        assert per <= top and per % 32 == 0 and min(shares) > 0 and sum(shares) == rows, rows
