"""CPU model of the tensor-core kernel's roles (csrc/kernels_tc.cu, tc_grm_kernel): the
producer, the MMA warp and the unpack warps of one CTA as coroutines over its run of
segments, with mbarrier phases, copies that land and MMAs that complete at any later time.

A random scheduler runs them for every kind of ring shape the host accepts and checks that
they always end (also when a wait gives up anywhere), with no copy, MMA or commit still in
flight; that a parity wait never passes on the wrong phase; that no operand slot, load slot
or accumulator is overwritten while it is still read; and that the segments of all CTAs
cover every tile once."""
import random

import pytest

GROUPS, WARPS = 4, 4  # unpack groups and their warps


def unit_begin(units, c, grid):
    return units * c // grid


MIN_SAVED = 24


def work(tiles, nk, sms, min_saved=MIN_SAVED):
    """tc_work: (grid, whole tiles per CTA, CTAs with one more, first shared tile, its units)."""
    grid, whole = sms, tiles // sms
    rest = tiles - whole * sms
    share = -(-rest * nk // sms)
    if rest > 0 and nk - share >= min_saved:
        return grid, whole, 0, whole * sms, rest * nk
    return (rest if whole == 0 else grid), whole, rest, whole * sms, 0


def segments(w, nk, c):
    grid, whole, extra, tail_tile, units = w
    for i in range(whole + (c < extra)):
        yield c + i * grid, 0, nk
    u, end = unit_begin(units, c, grid), unit_begin(units, c + 1, grid)
    while u < end:
        q = u // nk
        k0 = u - q * nk
        k1 = min(nk, k0 + end - u)
        yield tail_tile + q, k0, k1
        u += k1 - k0


def part_slot(w, nk, tile):
    grid, whole, extra, tail_tile, units = w
    first = (tile - tail_tile) * nk
    c = first * grid // units
    while unit_begin(units, c, grid) <= first:
        c += 1
    return c - 1


class Mbar:
    def __init__(self, count=1):
        self.count, self.have = count, 0
        self.done = 0  # completed phases

    def arrive(self):
        self.have += 1
        if self.have == self.count:
            self.have, self.done = 0, self.done + 1

    def passes(self, parity):
        return (self.done - 1) & 1 == parity


class Cta:
    def __init__(self, segs, nk, sub, sl, sa, rng, abort_at=None):
        self.segs, self.nk, self.sub, self.sl, self.sa, self.rng = segs, nk, sub, sl, sa, rng
        self.full = [Mbar() for _ in range(sl)]
        self.ldone = [Mbar() for _ in range(sl)]
        self.afull = [Mbar(WARPS) for _ in range(GROUPS)]
        self.adone = [Mbar() for _ in range(GROUPS)]
        self.accf, self.afree = Mbar(), Mbar(GROUPS * WARPS)
        self.psum, self.plast = Mbar(GROUPS * WARPS), Mbar()
        self.abort = False
        self.budget = abort_at  # polls until a wait gives up (None: never)
        self.loads = []         # landing copies
        self.tensor = []        # MMAs and commits in issue order, not completed yet
        self.holds = {}         # operand slot -> [sub-stage, warps that filled it]
        self.load_slot = {}     # load slot -> (load stage, first sub-stage, count, landed)
        self.acc_of = None      # segment in the accumulators
        self.acc_reads = {}
        self.finished = []

    def wait(self, mbar, parity, phase):
        """A bounded wait for a phase: True, or False when it gives up."""
        while not mbar.passes(parity):
            if self.abort:
                return False
            if self.budget is not None:
                self.budget -= 1
                if self.budget < 0:
                    self.abort = True
                    return False
            yield
        assert mbar.done > phase and phase & 1 == parity, "a parity wait passed too early"
        return True

    def drain(self, mbar, parity, phase):
        while not mbar.passes(parity):
            yield
        assert mbar.done > phase and phase & 1 == parity

    # ---- roles ----
    def producer(self):
        S = J = ph = 0
        live = True
        for tile, k0, k1 in self.segs:
            for k in range(k0, k1, self.sub):
                if J >= self.sl:
                    live = yield from self.wait(self.ldone[S], ph ^ 1, J // self.sl - 1)
                    if not live:
                        break
                assert not any(x[0] == "mma" and x[2] == S for x in self.tensor)
                self.load_slot[S] = (J, k, min(self.sub, k1 - k), False)
                self.loads.append(S)
                J += 1
                S += 1
                if S == self.sl:
                    S, ph = 0, ph ^ 1
                yield
            if not live:
                break
        for j in range(max(0, J - self.sl), J):
            yield from self.drain(self.full[j % self.sl], (j // self.sl) & 1, j // self.sl)

    def mma(self):
        t = s = ab = grp = ph_a = K = J = n_seg = 0
        live, ready = True, False
        for i, (tile, k0, k1) in enumerate(self.segs):
            if n_seg > 0:
                live = yield from self.wait(self.afree, (n_seg - 1) & 1, n_seg - 1)
            k = k0
            while live and k < k1:
                if not ready:
                    live = yield from self.wait(self.afull[grp], ph_a, K // GROUPS)
                if not live:
                    break
                assert self.afull[grp].done > K // GROUPS
                stage_end = t == self.sub - 1 or k == k1 - 1
                assert self.holds[ab] == [K, WARPS], "operand slot does not hold this sub-stage"
                j, base, cnt, landed = self.load_slot[s]
                assert landed and base + t == k and t < cnt and j == J
                if k == k0:
                    assert i == 0 or self.acc_reads[i - 1] == GROUPS * WARPS
                    self.acc_of = i
                self.tensor.append(("mma", ab, s))
                yield
                ready = self.afull[(grp + 1) % GROUPS].passes(ph_a ^ (grp == GROUPS - 1))
                self.tensor.append(("mma", ab, s))
                self.tensor.append(("adone", grp))
                if stage_end:
                    self.tensor.append(("ldone", s))
                K, t = K + 1, t + 1
                if stage_end:
                    t, J, s = 0, J + 1, (s + 1) % self.sl
                ab = (ab + 1) % self.sa
                grp += 1
                if grp == GROUPS:
                    grp, ph_a = 0, ph_a ^ 1
                k += 1
                yield
            if not live:
                break
            self.tensor.append(("accf",))
            n_seg += 1
        for ls in range(min(self.sl, J)):
            f = (J - 1 - (J - 1 - ls) % self.sl) // self.sl
            yield from self.drain(self.ldone[ls], f & 1, f)
        for g in range(min(GROUPS, K)):
            f = (K - 1 - (K - 1 - g) % GROUPS) // GROUPS
            yield from self.drain(self.adone[g], f & 1, f)
        if n_seg:
            yield from self.drain(self.accf, (n_seg - 1) & 1, n_seg - 1)
        assert not self.tensor, "an MMA or commit is still in flight"

    def unpack(self, grp, warp):
        lsub = self.sub >> 1
        K0 = s0 = ph0 = J0 = ph_part = n_part = 0
        for i, (tile, k0, k1) in enumerate(self.segs):
            n = k1 - k0
            x = (grp - K0) & (GROUPS - 1)
            s, ab, t, ph_l = s0 + (x >> lsub), (K0 + x) % self.sa, x & (self.sub - 1), ph0
            while s >= self.sl:
                s, ph_l = s - self.sl, ph_l ^ 1
            while x < n:
                K, J = K0 + x, J0 + (x >> lsub)
                assert s == J % self.sl and ph_l == (J // self.sl) & 1 and ab == K % self.sa
                if K >= self.sa:
                    f = (K - self.sa) // GROUPS
                    ok = yield from self.wait(self.adone[(K - self.sa) % GROUPS], f & 1, f)
                    if not ok:
                        return
                ok = yield from self.wait(self.full[s], ph_l, J // self.sl)
                if not ok:
                    return
                assert not any(y[0] == "mma" and y[1] == ab for y in self.tensor)
                j, base, cnt, landed = self.load_slot[s]
                assert landed and j == J and base + t == k0 + x
                if self.holds.get(ab, [None])[0] != K:
                    self.holds[ab] = [K, 0]
                yield
                assert self.holds[ab][0] == K
                self.holds[ab][1] += 1
                self.afull[grp].arrive()
                s += GROUPS >> lsub
                while s >= self.sl:
                    s, ph_l = s - self.sl, ph_l ^ 1
                if self.sa == 3:
                    ab = (ab + 1) % 3
                x += GROUPS
            K0 += n
            stages = (n + self.sub - 1) >> lsub
            J0 += stages
            s1 = s0 + stages
            s0, ph0 = s1 % self.sl, ph0 ^ ((s1 // self.sl) & 1)
            ok = yield from self.wait(self.accf, i & 1, i)
            if not ok:
                return
            assert self.acc_of == i, "the accumulators hold another segment"
            yield
            assert self.acc_of == i
            self.acc_reads[i] = self.acc_reads.get(i, 0) + 1
            self.afree.arrive()
            if (k0, k1) != (0, self.nk):
                self.psum.arrive()
                if grp == 0 and warp == 0:
                    ok = yield from self.wait(self.psum, ph_part, n_part)
                    if not ok:
                        return
                    self.plast.arrive()
                ok = yield from self.wait(self.plast, ph_part, n_part)
                if not ok:
                    return
                ph_part, n_part = ph_part ^ 1, n_part + 1
            if grp == 0 and warp == 0:
                self.finished.append((tile, k0, k1))

    # ---- asynchronous hardware ----
    def hardware(self):
        if self.loads and self.rng.random() < 0.5:
            S = self.loads.pop(self.rng.randrange(len(self.loads)))
            self.load_slot[S] = self.load_slot[S][:3] + (True,)
            self.full[S].arrive()
        elif self.tensor:
            op = self.tensor.pop(0)
            if op[0] == "adone":
                self.adone[op[1]].arrive()
            elif op[0] == "ldone":
                self.ldone[op[1]].arrive()
            elif op[0] == "accf":
                self.accf.arrive()

    def run(self):
        roles = [self.producer(), self.mma()]
        roles += [self.unpack(g, w) for g in range(GROUPS) for w in range(WARPS)]
        idle = 0
        while roles:
            before = len(roles)
            if self.rng.random() < 0.4:
                self.hardware()
            r = self.rng.choice(roles)
            try:
                next(r)
            except StopIteration:
                roles.remove(r)
            idle = 0 if len(roles) < before else idle + 1
            assert idle < 400000, "the roles wait for one another"
        assert not self.tensor and not self.loads
        if not self.abort:
            assert self.finished == self.segs


SHAPES = [(sub, sl, sa) for sub in (1, 2, 4) for sl in (2, 3, 5) for sa in (2, 3, 4)
          if (sl - 1) * sub + 1 >= sa]


# tiles, sub-stages, CTAs, saving from which the rest is shared
WORKS = ((1, 3, 1, 1), (3, 7, 2, 1), (5, 4, 3, 1), (2, 30, 4, 1), (7, 1, 3, 1), (7, 9, 3, 99))


@pytest.mark.parametrize("sub,sl,sa", SHAPES)
def test_roles_end_and_never_overtake(sub, sl, sa):
    rng = random.Random(100 * sub + 10 * sl + sa)
    for tiles, nk, sms, saved in WORKS:
        w = work(tiles, nk, sms, saved)
        for c in range(w[0]):
            Cta(list(segments(w, nk, c)), nk, sub, sl, sa, rng).run()


@pytest.mark.parametrize("sub,sl,sa", SHAPES)
def test_roles_end_when_a_wait_gives_up(sub, sl, sa):
    rng = random.Random(7 + 100 * sub + 10 * sl + sa)
    for abort_at in (0, 1, 3, 10, 30, 80, 200):
        for tiles, nk, sms in ((3, 7, 2), (4, 5, 3)):
            w = work(tiles, nk, sms, 1)
            for c in range(w[0]):
                Cta(list(segments(w, nk, c)), nk, sub, sl, sa, rng, abort_at=abort_at).run()


@pytest.mark.parametrize("tiles,nk", [(1, 1), (40, 16), (164, 72), (72, 164), (17, 447),
                                      (1173, 1563), (149, 1), (148, 5), (296, 30), (150, 400)])
def test_segments_cover_every_tile_and_shared_tiles_have_their_own_slot(tiles, nk):
    w = work(tiles, nk, 148)
    covered, slots, most = {}, {}, 0
    for c in range(w[0]):
        mine = 0
        for tile, k0, k1 in segments(w, nk, c):
            assert 0 <= tile < tiles and 0 <= k0 < k1 <= nk
            covered.setdefault(tile, []).append((k0, k1))
            mine += k1 - k0
            if (k0, k1) != (0, nk):
                slot = part_slot(w, nk, tile)
                assert 0 <= slot < 148
                assert slots.setdefault(slot, tile) == tile
        most = max(most, mine)
    for tile in range(tiles):
        parts = sorted(covered[tile])
        assert parts[0][0] == 0 and parts[-1][1] == nk
        assert all(a[1] == b[0] for a, b in zip(parts, parts[1:]))
    assert most <= -(-tiles * nk // 148) + max(MIN_SAVED, 1)
