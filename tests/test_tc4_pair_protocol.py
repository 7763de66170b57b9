"""The barrier protocol of the CTA pairs of the 4-bit tensor GEMM
(parpar_gb300/csrc/k_tc4.cu: k_tc4_gemm), checked on the CPU.

The source test holds every signal between the two CTAs of a pair to cluster
scope: an arrival or a wait at CTA scope orders nothing between them.  The model
runs the warps of a pair in random order over every ring layout that the planner
gives: no stage may be read before it is whole or overwritten before it has been
read, every tile is written once by every read-out warp, and nothing may wait for
ever.  It takes commits to arrive in their order, as the tensor core runs them."""
import ctypes
import os
import random
import re

import pytest

from parpar_gb300 import _lib

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "parpar_gb300", "csrc", "k_tc4.cu")

# who gives a barrier's signals: its own CTA alone, either CTA (or MMAs that
# read the shared memory of both), or accumulators changing hands
OWN = {"QFULL", "QEMPTY", "BFULL"}
PAIR = {"READY", "EMPTY", "IDFULL", "IDEMPTY"}
TMEM = {"TFULL", "TEMPTY"}


def source():
    with open(SRC) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    # adjacent string literals are one string
    return re.sub(r'"\s*\n\s*"', "", text)


def test_signals_between_the_ctas_of_a_pair_have_cluster_scope():
    text = source()
    # arrivals that can reach the other CTA
    arrivals = re.findall(r"[^\"]*mbarrier\.arrive[a-z_:.]*shared::cluster\.b64 _[^\"]*", text)
    assert arrivals
    for a in arrivals:
        assert "mbarrier.arrive.release.cluster." in a or (
            "fence.release.sync_restrict::shared::cta.cluster;" in a and "mbarrier.arrive.relaxed.cluster." in a), a
    # waits, by the barrier they wait for
    waits = re.findall(r"t4_wait_ab(<[^>]*>)?\([^;]*?T4B_([A-Z]+)", text)
    assert {b for _, b in waits} == OWN | PAIR | TMEM
    for kind, b in waits:
        assert kind == ("" if b in OWN else "<T4_PAIR>" if b in PAIR else "<T4_TMEM>"), (kind, b)
    body = text[text.index("bool t4_try("):text.index("uint32_t t4_test_pair(")]
    near, far = body[body.index("if(BY != T4_CTA)"):].split("else", 1)
    assert "try_wait.parity.relaxed.cluster." in near and "try_wait.parity.shared::cta" in far
    body = text[text.index("bool t4_wait_ab("):]
    assert re.search(r"if\(t4_try<BY>\(bar, parity\)\) \{\s*if\(BY == T4_PAIR\) t4_acquire_pair\(\);\s*return true;", body)
    assert "fence.acquire.sync_restrict::shared::cluster.cluster;" in text
    # a stage found ready by the look ahead is acquired where its wait is skipped
    assert re.search(r"if\(seen\) t4_acquire_pair\(\);\s*else if\(.*T4B_READY", text)
    assert "test_wait.parity.relaxed.cluster." in text
    # the accumulators' signals stand between the tcgen05 fences
    for b in TMEM:
        m = re.search(r"t4_wait_ab<T4_TMEM>\([^;]*T4B_%s[^;]*;\s*(break; \}|)\s*([^;]*;)" % b, text)
        assert m and "tcgen05.fence::after_thread_sync" in m.group(2), (b, m)


# ------------------------------------------------------------------ the model
# One pair of CTAs (and its share of the tiles) as generators, one per warp, with
# the waits, arrivals and slot arithmetic of the kernel.  A generator yields False
# where it polled a barrier in vain and True after a step.  What the hardware does
# by itself is a list of events taken in any order (bulk copies, tile numbers on
# their way) or, for the tensor core, in the order of issue: its MMAs read both
# CTAs' slots when they run, not when they are issued, and a commit signals once
# all before it have run.  Slots hold the stage that was written to them.
TR, EG, EXP, EPI = 4, 3, 12, 8


class Bar:
    def __init__(self, count):
        self.count, self.pending, self.tx, self.phase = count, count, 0, 0

    def _turn(self):
        if self.pending == 0 and self.tx == 0:
            self.phase, self.pending = self.phase + 1, self.count

    def arrive(self):
        self.pending -= 1
        assert self.pending >= 0, "an arrival too many"
        self._turn()

    def expect(self):
        self.tx += 1
        self.arrive()

    def complete(self):
        self.tx -= 1
        self._turn()

    def passed(self, parity):
        return (self.phase & 1) != parity


class Layout:
    """passes: of a tile's words and columns; spr: stages of a run; pps: whole passes of a stage (0: a pass is a
    run of stages); splits: tiles that share the passes."""

    def __init__(self, nA, nB, nQ, passes, spr, pps, PG, nGrp, splits=1):
        self.nA, self.nB, self.nQ, self.spr, self.pps, self.PG, self.nGrp = nA, nB, nQ, spr, pps, PG, nGrp
        self.all_passes, self.splits = passes, splits

    def span(self, t):
        """First pass of tile t, and the first that is not its own."""
        part = t % self.splits
        return part * self.all_passes // self.splits, (part + 1) * self.all_passes // self.splits

    def stages_of(self, t):
        n = self.span(t)[1] - self.span(t)[0]
        return -(-n // self.pps) if self.pps else n * self.spr


def wait(bar, parity):
    while not bar.passed(parity):
        yield False
    yield True


class Pair:
    def __init__(self, lay, n_tiles, counter, written, events):
        self.lay, self.n_tiles, self.counter, self.written, self.events = lay, n_tiles, counter, written, events
        self.queue = []                              # of the tensor core
        L = lay
        both = lambda n, count: [[Bar(count) for _ in range(n)] for _ in range(2)]
        lead = lambda n, count: [Bar(count) for _ in range(n)]
        self.qfull, self.qempty, self.bfull = both(L.nQ, 1), both(L.nQ, 4), both(L.nB, 1)
        self.ready, self.empty = lead(L.nB, 10), both(L.nB, 1)
        self.tfull, self.tempty = both(L.nGrp, 1), lead(L.nGrp, 2 * EPI)
        self.idfull, self.idempty = both(TR, 1), lead(TR, 2 * (EPI + EXP + 3) + 1)
        self.ids = [[None] * TR for _ in range(2)]
        self.Q = [[None] * L.nQ for _ in range(2)]
        self.B = [[None] * L.nB for _ in range(2)]
        self.A = [[[None] * 4 for _ in range(L.nA)] for _ in range(2)]
        self.acc = [[None] * L.PG for _ in range(L.nGrp)]

    def roles(self):
        out = [self.mma()]
        for r in range(2):
            out += [self.copy_b(r), self.copy_q(r), self.relay(r)]
            out += [self.expander(r, w // 4, w % 4) for w in range(EXP)] + [self.epilogue(r, w) for w in range(EPI)]
        return out

    def next_tile(self, r, j):
        yield from wait(self.idfull[r][j % TR], (j // TR) & 1)
        t = self.ids[r][j % TR]
        assert t is not None and t[0] == j, "a tile number of another turn"
        yield True
        self.idempty[j % TR].arrive()
        return t[1]

    def copy_b(self, r):
        L, g = self.lay, 0
        ahead = None

        def fetch():
            t = self.counter[0]
            self.counter[0] += 1
            return t if t < self.n_tiles else -1

        def publish(j, t):
            if j >= TR:
                yield from wait(self.idempty[j % TR], (j // TR - 1) & 1)

            def land(c):
                self.ids[c][j % TR] = (j, t)
                self.idfull[c][j % TR].complete()
            for c in range(2):
                self.events.append(lambda c=c: land(c))
            yield True

        if r == 0:
            ahead = fetch()
            yield from publish(0, ahead)
            if ahead >= 0:
                ahead = fetch()
        j = 0
        while True:
            self.idfull[r][j % TR].expect()
            t = yield from self.next_tile(r, j)
            if t < 0:
                break
            if r == 0:
                yield from publish(j + 1, ahead)
                if ahead >= 0:
                    ahead = fetch()
            for _ in range(L.stages_of(t)):
                s = g % L.nB
                if g >= L.nB:
                    yield from wait(self.empty[r][s], (g // L.nB - 1) & 1)
                self.bfull[r][s].expect()

                def land(s=s, g=g):
                    self.B[r][s] = g
                    self.bfull[r][s].complete()
                self.B[r][s] = None                  # being written from now on
                self.events.append(land)
                g += 1
                yield True
            j += 1
        for h in range(max(0, g - L.nB), g):
            yield from wait(self.empty[r][h % L.nB], (h // L.nB) & 1)

    def copy_q(self, r):
        L, g, j = self.lay, 0, 0
        while True:
            t = yield from self.next_tile(r, j)
            if t < 0:
                break
            for _ in range(L.stages_of(t)):
                s = g % L.nQ
                if g >= L.nQ:
                    yield from wait(self.qempty[r][s], (g // L.nQ - 1) & 1)
                self.qfull[r][s].expect()

                def land(s=s, g=g):
                    self.Q[r][s] = g
                    self.qfull[r][s].complete()
                self.Q[r][s] = None
                self.events.append(land)
                g += 1
                yield True
            j += 1
        for h in range(max(0, g - L.nQ), g):
            yield from wait(self.qfull[r][h % L.nQ], (h // L.nQ) & 1)

    def relay(self, r):
        L, s, ph, j = self.lay, 0, 0, 0
        while True:
            t = yield from self.next_tile(r, j)
            if t < 0:
                return
            for _ in range(L.stages_of(t)):
                yield from wait(self.bfull[r][s], ph)
                self.ready[s].arrive()
                s += 1
                if s == L.nB:
                    s, ph = 0, ph ^ 1
            j += 1

    def expander(self, r, grp, quarter):
        L = self.lay
        turn, qs, qph, sa, sb = 0, grp, 0, grp % L.nA, grp % L.nB
        seq, eb, eph, base, j = grp, 0, 0, 0, 0
        while True:
            t = yield from self.next_tile(r, j)
            if t < 0:
                return
            e = grp - turn if grp >= turn else grp + EG - turn
            stages = L.stages_of(t)
            turn = (turn + stages) % EG
            while e < stages:
                stage = base + e
                yield from wait(self.qfull[r][qs], qph)
                for _ in range(2):                   # the read takes a while
                    assert self.Q[r][qs] == stage, ("compact A", self.Q[r][qs], stage)
                    yield True
                self.qempty[r][qs].arrive()
                qs += EG
                if qs >= L.nQ:
                    qs, qph = qs - L.nQ, qph ^ 1
                if seq >= L.nA:
                    yield from wait(self.empty[r][eb], eph)
                    eb += EG
                    if eb >= L.nB:
                        eb, eph = eb - L.nB, eph ^ 1
                else:
                    seq += EG
                    if seq >= L.nA:
                        eb = seq - L.nA
                self.A[r][sa][quarter] = None
                yield True
                self.A[r][sa][quarter] = stage
                self.ready[sb].arrive()
                sa, sb, e = sa + EG, sb + EG, e + EG
                if sa >= L.nA:
                    sa -= L.nA
                if sb >= L.nB:
                    sb -= L.nB
                yield True
            base += stages
            j += 1

    def mma(self):
        L = self.lay
        sa = sb = ph_b = grp = kg = np_ = 0
        ph_t, g, j, seen = 1, 0, 0, False

        def run_pass(g, sa, sb, at, v):              # of a stage, or the part of it that a stage holds
            for c in range(2):
                assert self.A[c][sa] == [g] * 4, ("A", c, self.A[c][sa], g)
                assert self.B[c][sb] == g, ("B", c, self.B[c][sb], g)
            self.acc[at[0]][at[1]] = v

        while True:
            t = yield from self.next_tile(0, j)
            if t < 0:
                return
            p, last = L.span(t)
            for e in range(L.stages_of(t)):
                if not seen:
                    yield from wait(self.ready[sb], ph_b)
                seen = False
                slot_a, slot_b = sa, sb
                sa, sb = (sa + 1) % L.nA, sb + 1
                if sb == L.nB:
                    sb, ph_b = 0, ph_b ^ 1
                if L.pps:
                    peek = self.ready[sb].passed(ph_b)
                for k in range(L.pps or 1):
                    if p >= last:
                        break
                    if kg == 0 and (L.pps or e % L.spr == 0):
                        if np_ < L.nGrp:
                            np_ += 1
                        else:
                            yield from wait(self.tempty[grp], ph_t)
                    self.queue.append(lambda g=g, a=slot_a, b=slot_b, at=(grp, kg), v=(t, p): run_pass(g, a, b, at, v))
                    if L.pps or e % L.spr == L.spr - 1:
                        p += 1
                        kg += 1
                        if kg == L.PG or p == last:
                            self.queue.append(lambda gr=grp: [self.tfull[c][gr].arrive() for c in range(2)])
                            kg, grp = 0, grp + 1
                            if grp == L.nGrp:
                                grp, ph_t = 0, ph_t ^ 1
                self.queue.append(lambda b=slot_b: [self.empty[c][b].arrive() for c in range(2)])
                if L.pps:
                    seen = peek
                g += 1
                yield True
            j += 1

    def epilogue(self, r, w):
        L, grp, ph, j = self.lay, 0, 0, 0
        while True:
            t = yield from self.next_tile(r, j)
            if t < 0:
                return
            p, last = L.span(t)
            while p < last:
                yield from wait(self.tfull[r][grp], ph)
                for k in range(min(L.PG, last - p)):
                    assert self.acc[grp][k] == (t, p), ("accumulator", self.acc[grp][k], t, p)
                    p += 1
                    yield True
                self.tempty[grp].arrive()
                grp += 1
                if grp == L.nGrp:
                    grp, ph = 0, ph ^ 1
            self.written.append((t, r, w))
            j += 1


def run(lay, n_tiles, pairs, rng):
    counter, written, events = [0], [], []
    ps = [Pair(lay, n_tiles, counter, written, events) for _ in range(pairs)]
    alive = [g for p in ps for g in p.roles()]
    slow = rng.choice([None, None] + alive)          # one warp that hardly gets its turn
    idle = 0
    while alive or events or any(p.queue for p in ps):
        idle += 1
        x = rng.random()
        if events and x < 0.15:
            events.pop(rng.randrange(len(events)))()
            idle = 0
        elif x < 0.4 and any(p.queue for p in ps):
            rng.choice([p for p in ps if p.queue]).queue.pop(0)()
            idle = 0
        elif alive:
            g = rng.choice(alive)
            if g is slow and rng.random() < 0.9:
                continue
            for _ in range(rng.choice((1, 2, 12))):
                try:
                    if not next(g):
                        break
                    idle = 0
                except StopIteration:
                    alive.remove(g)
                    idle = 0
                    break
        if idle > 500 and not events and not any(p.queue for p in ps):
            for g in list(alive):                    # every warp once: one of them has to get on
                try:
                    if next(g):
                        idle = 0
                except StopIteration:
                    alive.remove(g)
                    idle = 0
            assert idle == 0, "deadlock"
    assert sorted(written) == sorted((t, r, w) for t in range(n_tiles) for r in range(2) for w in range(EPI))
    assert counter[0] == n_tiles + pairs


def layouts():
    """Every ring layout the planner gives for tiles of 16 to 240 columns and passes of 1 to 4 and of more units."""
    lib = _lib.load()
    out = {}
    for R in range(1, 61):
        for n in (20, 40, 60, 80, 110, 250, 500):
            words = 4096
            plan = _lib.Fp4Plan()
            sb = lib.par2cuda_tensor_fp4_scratch_bytes(R, n, words)
            assert lib.par2cuda_tensor_fp4_plan(R, n, words, sb, 76, ctypes.byref(plan)) == 0, lib.par2cuda_last_error()
            pps = 5 // plan.units if plan.units < 5 else 0
            spr = 1 if pps else -(-plan.units // 5)
            nGrp = min(8, 480 // (plan.group_passes * plan.columns))
            key = (plan.slots_a, plan.slots_b, plan.slots_q, 7, min(spr, 3), pps, plan.group_passes, nGrp)
            out.setdefault(key, set()).add(plan.columns)
    return out


def test_planned_ring_layouts_keep_the_rules_of_the_rings():
    found = layouts()
    assert {k[5] for k in found} == {0, 1, 2, 5} and set().union(*found.values()) == set(range(16, 241, 16))
    for (nA, nB, nQ, _, _, _, PG, nGrp), columns in found.items():
        # a slot of compact A belongs to one group of expanders, who otherwise wait for phases
        # they have not seen begin; A's slots are freed by phases of B's barriers
        assert nQ % EG == 0 and nB > EG and nB >= nA >= 3 and nGrp >= 2 and nGrp * PG * max(columns) <= 480, (nA, nB, nQ, PG, nGrp)


def test_pair_protocol():
    for k, key in enumerate(sorted(layouts())):
        for seed in range(2):
            rng = random.Random(100 * k + seed)
            run(Layout(*key), rng.randint(1, 6), rng.randint(1, 2), rng)


def test_pair_protocol_of_split_passes():
    # tiles of one to four passes, of unlike lengths, one after another
    for k, key in enumerate(sorted(key for key in layouts() if not key[5])):
        for splits in (2, 3, 4, 5, 7):
            rng = random.Random(1000 * k + splits)
            run(Layout(*key, splits), splits * rng.randint(1, 3), rng.randint(1, 2), rng)


def test_passes_are_split_only_where_pairs_would_idle():
    lib = _lib.load()

    def splits(n, R, words, pairs=76):
        plan = _lib.Fp4Plan()
        sb = lib.par2cuda_tensor_fp4_scratch_bytes(R, n, words)
        assert lib.par2cuda_tensor_fp4_plan(R, n, words, sb, pairs, ctypes.byref(plan)) == 0
        assert plan.pass_splits == 1 or (plan.form == 4 and plan.units >= 13 and plan.chunks == 1)
        return plan.pass_splits

    assert splits(10000, 60, 2052) == 7              # 9 tiles
    assert splits(10000, 60, 2053) == 1              # an odd number of words
    assert splits(288, 60, 2052) == 1 and splits(289, 60, 2052) == 7    # 12 units and 13
    assert splits(3000, 30, 256 * 10) == 7 and splits(3000, 30, 256 * 19) == 4 and splits(3000, 30, 256 * 20) == 1
    assert splits(3000, 61, 256 * 9) == 4 and splits(3000, 61, 256 * 10) == 1    # two column tiles
    assert splits(2000, 200, 1 << 20) == 1 and splits(777, 133, 700006) == 1
    for n in (120, 500, 4096):
        for R in (1, 60, 61, 300):
            for words in (2, 256, 4096, 19456, 40000, 200000):
                splits(n, R, words)


def test_pair_protocol_of_63_passes():
    # single-bit passes: an accumulator a pass, several stages a pass
    for seed, (nA, nB, nQ, spr) in enumerate([(3, 4, 3, 1), (3, 4, 3, 2), (4, 5, 6, 1)]):
        run(Layout(nA, nB, nQ, 63, spr, 0, 1, 2), 2, 1, random.Random(seed))


@pytest.mark.parametrize("nA,nB,nQ", [(3, 4, 4), (3, 4, 5), (6, 4, 6)])
def test_layouts_against_the_rules_fail(nA, nB, nQ):
    with pytest.raises(AssertionError):
        for seed in range(60):
            run(Layout(nA, nB, nQ, 7, 1, 0, 1, 2), 4, 1, random.Random(seed))
