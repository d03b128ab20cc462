"""The tensor-memory matmul (csrc/pie_qmt.cuh) on the CPU: its operand arithmetic over every scale significand and code, the barriers of
its ring under random schedules, and the shares of its CTAs."""
import os
import random
import re

import numpy as np
import pytest
import torch

HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "proxy_inference_engine_b200", "csrc", "pie_qmt.cuh")
COLS, STAGE, SMEM = 72, 128 * 160, 226 * 1024      # kQtCols, kQtStage, kQtSmem


def geometry(np_):
    """(turn size, stages) as launch_qmt takes them."""
    per = 2 if 2 * np_ + 6 * COLS <= 512 else 1
    fixed = 1024 + 3 * per * np_ * 288 + 4096 + 512 + (np_ * 512 if np_ == 32 else 0)
    stages = min(12, (SMEM - fixed) // STAGE)
    assert 2 * np_ + 3 * per * COLS <= 512 and fixed + stages * STAGE <= SMEM
    return per, stages


def test_the_constants_are_the_kernels():
    with open(HEADER) as f:
        text = f.read()
    assert "constexpr int kQtCols = 72;" in text and re.search(r"kQtPacked = 128 \* 128;", text) and "kQtPacked + 2 * 128 * 16;" in text
    assert "constexpr int kQtSmem = 226 * 1024;" in text and "1024 + 3 * per * a.np * 288 + 4096 + kQtMaxRows * 4 + (a.totals_smem ? a.np * 512 : 0)" in text


def test_operands_are_exact():
    """S q - E by both instruction sequences: equal, and numbers fp16 has, for every significand, exponent and code."""
    h = np.float16
    q = np.arange(16, dtype=np.float64)
    for k in range(-24, 3):
        s = np.arange(256, dtype=np.float64) * 2.0 ** k
        s = s[np.abs(s) <= 896]
        assert np.array_equal(s.astype(h).astype(np.float64), s)
        c = (s * -72).astype(h).astype(np.float64)                     # rounds once
        me = s * 64 + c
        assert np.array_equal(me.astype(h).astype(np.float64), me)
        two = s[:, None] * q + me[:, None]                             # (1024 + q) - 1024, then one multiply-add
        one = s[:, None] * (64 + q) + c[:, None]
        assert np.array_equal(two, one) and np.array_equal(two.astype(h).astype(np.float64), two)


class Bar:
    def __init__(self, count):
        self.count = self.pending = count
        self.phase = 0

    def arrive(self):
        self.pending -= 1
        assert self.pending >= 0
        if self.pending == 0:
            self.phase, self.pending = self.phase + 1, self.count

    def passed(self, parity):                                           # mbarrier.try_wait.parity
        return (self.phase & 1) != parity


def walk(np_, stages, rng):
    per, nw = geometry(np_)
    turns = stages * 2 // per
    wf, we = [Bar(1) for _ in range(nw)], [Bar(8 // per) for _ in range(nw)]
    af, ae = [Bar(5) for _ in range(3)], [Bar(1) for _ in range(3)]
    words, operand, xs = [None] * nw, [[None] * 4 for _ in range(3)], [None] * 3
    landing, mmas = [], []

    def packed():
        slot, phase = 0, 1
        for i in range(stages):
            while not we[slot].passed(phase):
                yield
            landing.append(lambda i=i, slot=slot: (words.__setitem__(slot, i), wf[slot].arrive()))
            slot = (slot + 1) % nw
            phase ^= slot == 0
            yield

    def prepared():
        for t in range(turns):
            while not ae[t % 3].passed(1 ^ (t // 3 & 1)):
                yield
            landing.append(lambda t=t: (xs.__setitem__(t % 3, t), af[t % 3].arrive()))
            yield

    def mma():
        for t in range(turns):
            while not af[t % 3].passed(t // 3 & 1):
                yield
            assert operand[t % 3] == [t] * 4 and xs[t % 3] == t
            mmas.append(t)
            yield

    def dequantise(s, quad):
        ws, wph, aph = s * per // 2, 0, 1
        for t in range(s, turns, 3):
            i = t * per // 2
            while not wf[ws].passed(wph):
                yield
            assert words[ws] == i                                       # neither early nor late
            while not ae[s].passed(aph):
                yield
            assert ae[s].phase == t // 3
            yield
            operand[s][quad] = t
            assert words[ws] == i
            af[s].arrive()
            we[ws].arrive()
            yield
            aph ^= 1
            ws += 3 if per == 2 else 1 + (t & 1)
            if ws >= nw:
                ws, wph = ws - nw, wph ^ 1

    threads = [packed(), prepared(), mma()] + [dequantise(s, quad) for s in range(3) for quad in range(4)]
    speed, alive, steps = [rng.choice([1, 1, 3, 20]) for _ in threads], set(range(len(threads))), 0
    while alive or mmas or landing:
        r = rng.random()
        if r < 0.25 and landing and rng.random() < 0.5:
            landing.pop(rng.randrange(len(landing)))()
        elif r < 0.4 and mmas and rng.random() < 0.7:
            ae[mmas.pop(0) % 3].arrive()
        elif alive:
            k = rng.choice(sorted(alive))
            for _ in range(speed[k]):
                try:
                    next(threads[k])
                except StopIteration:
                    alive.discard(k)
                    break
        steps += 1
        assert steps < 200000                                           # a wait that stays


@pytest.mark.parametrize("np_", range(16, 129, 16))
def test_no_wait_passes_early_or_stays(np_):
    rng = random.Random(np_)
    for _ in range(25):
        walk(np_, rng.randint(1, 40), rng)


def shares(ntiles, ks, sms=148):
    """[(first, end) stage of each CTA], and of each tile the (CTA, part) its finisher adds, as the kernel computes them."""
    total = ntiles * ks
    even, grid, split = -(-total // sms), min(total, sms), 0
    if ntiles <= sms:
        p = min(sms // ntiles, ks)
        if -(-ks // p) <= even + 1:
            split, grid = p, ntiles * p
    if split:
        cut = [(c // split * ks + c % split * ks // split, c // split * ks + (c % split + 1) * ks // split) for c in range(grid)]
    else:
        cut = [(c * total // grid, (c + 1) * total // grid) for c in range(grid)]
    parts = {}
    for t in range(ntiles):
        if split:
            c0, n, second = t * split, split, 0
        else:
            c0 = ((t * ks + 1) * grid - 1) // total
            n = ((t + 1) * ks * grid - 1) // total - c0 + 1
            second = int(c0 * total // grid < t * ks)
        parts[t] = [(c0, 2 * c0 + second)] + [(c, 2 * c) for c in range(c0 + 1, c0 + n)]
    return cut, parts


def test_shares_cover_the_work_and_parts_are_found_again():
    rng = random.Random(1)
    for case in range(600):
        ntiles, ks = rng.choice([rng.randint(1, 40), rng.randint(1, 1100)]), 2 * rng.randint(1, 64)
        cut, parts = shares(ntiles, ks)
        assert cut[0][0] == 0 and cut[-1][1] == ntiles * ks and all(a[1] == b[0] for a, b in zip(cut, cut[1:]))
        assert len(cut) <= 148 and all(a < b for a, b in cut)
        stored = {}
        for c, (lo, hi) in enumerate(cut):
            for t in range(lo // ks, (hi - 1) // ks + 1):
                if max(lo, t * ks) > t * ks or min(hi, (t + 1) * ks) < (t + 1) * ks:      # not the whole tile
                    stored.setdefault(t, []).append((c, 2 * c + int(lo < t * ks)))
        slots = [s for v in stored.values() for _, s in v]
        assert len(slots) == len(set(slots)) and all(0 <= s < 2 * 148 for s in slots)
        for t, v in stored.items():
            assert parts[t] == v


def test_accumulators_change_hands_at_the_same_turns():
    """The MMA warp's count of turns and the result warps' count of accumulators of a tile: the same runs, in the same order, whatever a CTA's share."""
    rng = random.Random(2)
    with open(HEADER) as f:
        text = f.read()
    assert "a.run = a.np <= 64 ? 8 / per : 1 << 30;" in text and "const int before = dry ? 0 : (take * (2 / PER) - 1) / a.run;" in text
    for np_ in range(16, 129, 16):
        per, _ = geometry(np_)
        run = 8 // per if np_ <= 64 else 1 << 30
        assert (3 * np_ + 3 * per * COLS > 512) == (np_ == 32 or np_ > 96) and per == (2 if np_ <= 32 else 1)    # totals of 32 rows: in shared memory
        for _ in range(60):
            ks = 2 * rng.randint(1, 64)
            lo = rng.randint(0, 5 * ks - 1)
            hi = rng.randint(lo + 1, 5 * ks)
            turns, tile_turns = (hi - lo) * 2 // per, ks * 2 // per
            mma, rest, n = [], tile_turns - lo % ks * 2 // per, 0
            left = min(rest, run)
            rest -= left
            for t in range(turns):
                left, n = left - 1, n + 1
                if left == 0 or t + 1 == turns:
                    mma.append((t + 1, n))
                    n, rest = 0, rest or tile_turns
                    left = min(rest, run)
                    rest -= left
            results, done, kk, todo = [], 0, lo % ks, hi - lo
            while todo:
                take = min(todo, ks - kk)
                before = (take * 2 // per - 1) // run
                sizes = [run] * before + [take * 2 // per - before * run]
                for size in sizes:
                    done += size
                    results.append((done, size))
                todo, kk = todo - take, 0
            assert mma == results and all(0 < n <= run for _, n in mma)


@pytest.mark.skipif(torch.cuda.is_available(), reason="the pointers are none")
@pytest.mark.parametrize("M", [40, 77])
def test_calls_go_on_where_no_tensor_map_can_be_made(M, monkeypatch):
    """Without a driver none can: the call goes on to the kernels that need none, and fails at their launch for want of a device."""
    from proxy_inference_engine_b200 import _lib
    L, at = _lib.load(), 1 << 20
    monkeypatch.setenv("PIE_QMT", "2")
    monkeypatch.setenv("PIE_QMM_TC", "0" if M < 64 else "1")
    n0 = L.pie_launch_count()
    assert L.pie_qmt(at, 4096, at, 4096, M, 4096, (_lib.QmvSeg * 1)(_lib.QmvSeg(at, at, at, 4096)), 1, 64, 4, None, 0.0, 0, None, at, 1 << 30, None) == _lib.EUNSUPPORTED
    assert L.pie_launch_count() == n0
    L.pie_qmm(at, at, at, at, at, M, 4096, 4096, 64, 4, at, 1 << 30, None)
    assert L.pie_launch_count() > n0 or b"NotSupported" not in L.pie_last_cuda_error()
