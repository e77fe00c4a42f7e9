"""Planned DFA batches (an explicit item length): the strings' shares of the planning CTAs,
against the oracle."""

import numpy as np
import pytest

from trex_b200.workloads import random_dfa

pytestmark = pytest.mark.gpu


def _check(torch, oracle, dfas, data, off, ids, seg_len):
    from trex_b200.engine import DFASet
    s = DFASet(dfas)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    fs, ac, _ = s.run(up(data), up(off), up(ids), seg_len=seg_len)
    torch.cuda.synchronize()
    assert s.last_error_word() == 0
    s.close()
    rfs, rac = oracle.dfa_walk([d.tmap for d in dfas], [d.n_states for d in dfas], [d.start for d in dfas],
                               [d.accept for d in dfas], data, off, ids)
    assert np.array_equal(fs.cpu().numpy(), rfs)
    assert np.array_equal(ac.cpu().numpy(), rac)


# fewer tiles of 1024 strings than CTAs, as many, a few more, uneven shares
@pytest.mark.parametrize("n", [1, 1024, 1025, 148 * 1024 - 1, 148 * 1024, 148 * 1024 + 1, 333333])
def test_shares_of_the_planning_ctas(cuda, oracle, n):
    rng = np.random.default_rng(n)
    dfas = [random_dfa(k, np.arange(256), rng) for k in (5, 12, 40)]
    lens = rng.integers(0, 24, size=n)
    lens[rng.integers(0, n, size=50)] = 700   # a few of several items
    off = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(lens, out=off[1:])
    data = rng.integers(0, 256, size=int(off[-1]), dtype=np.uint8)
    ids = rng.integers(0, len(dfas), size=n).astype(np.int32)
    _check(cuda, oracle, dfas, data, off, ids, 256)


# shares by weight (more than four tiles a CTA): long strings together at one end, spread, equal strings,
# empty ones, and offsets that are out of order in one place (the others' results stay)
@pytest.mark.parametrize("order", ["down", "up", "mixed", "equal", "empty", "out_of_order"])
def test_weighted_shares_of_the_planning_ctas(cuda, oracle, order):
    rng = np.random.default_rng(len(order))
    n = 4 * 148 * 1024 + 1025
    dfas = [random_dfa(k, np.arange(256), rng) for k in (6, 16)]
    lens = rng.integers(0, 6, size=n) if order != "empty" else np.zeros(n, dtype=np.int64)
    if order == "equal":
        lens[:] = 3
    else:
        lens[rng.integers(0, n, size=3000)] = rng.integers(200, 9000, size=3000)
        lens = {"down": np.sort(lens)[::-1], "up": np.sort(lens)}.get(order, lens)
    off = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(lens, out=off[1:])
    data = rng.integers(0, 256, size=int(off[-1]), dtype=np.uint8)
    ids = rng.integers(0, 2, size=n).astype(np.int32)
    want, wacc = oracle.dfa_walk([d.tmap for d in dfas], [d.n_states for d in dfas], [0, 0], [d.accept for d in dfas],
                                 data, off, ids)
    bad = np.zeros(n, dtype=bool)
    o = off.copy()
    if order == "out_of_order":
        for k, v in ((n // 3, data.size + 5), (n // 2, -7)):   # strings k - 1 and k each
            o[k] = v
            bad[[k - 1, k]] = True
    from trex_b200.engine import DFASet
    s = DFASet(dfas)
    fs = cuda.full((n,), 99, dtype=cuda.uint8, device="cuda")
    s.run(cuda.from_numpy(data).cuda(), cuda.from_numpy(o).cuda(), cuda.from_numpy(ids).cuda(), final_state=fs, seg_len=256)
    assert s.last_error_word() == (1 if bad.any() else 0)
    fs = fs.cpu().numpy()
    assert np.array_equal(fs[~bad], want[~bad]) and np.all(fs[bad] == 99)
    every = s.run_all(cuda.from_numpy(data).cuda(), cuda.from_numpy(off).cuda(), seg_len=256)[0].cpu().numpy()
    s.close()
    assert np.array_equal(np.where(ids == 0, every[0], every[1]), want)


# Long strings together may not cost more than the same strings spread (their items were listed by one
# planning CTA: 1.09 times the whole batch).
def test_batch_in_order_of_length_is_not_slower(cuda):
    from trex_b200.engine import DFASet
    rng = np.random.default_rng(1)
    s = DFASet([random_dfa(k, np.arange(256), rng) for k in (8, 12, 16) * 5])
    n = 700000
    lens = np.clip(np.rint(np.exp(rng.normal(np.log(1024), 1.18, n))), 16, 65536).astype(np.int64)
    data = cuda.randint(0, 256, (int(lens.sum()),), dtype=cuda.uint8, device="cuda")
    ids = cuda.arange(n, device="cuda", dtype=cuda.int32) % 15
    best = {}
    for name in ("spread", "down", "spread", "down"):
        off = np.zeros(n + 1, dtype=np.int64)
        np.cumsum(lens if name == "spread" else np.sort(lens)[::-1], out=off[1:])
        off = cuda.from_numpy(off).cuda()
        for _ in range(6):
            t0, t1 = (cuda.cuda.Event(enable_timing=True) for _ in range(2))
            t0.record()
            s.run(data, off, ids)
            t1.record()
            t1.synchronize()
            best[name] = min(best.get(name, 1e9), t0.elapsed_time(t1))
    s.close()
    assert best["down"] < 1.05 * best["spread"], best


# the shared-memory table of each layout: its fewest and most states, and a partial last word
@pytest.mark.parametrize("n_states", [1, 3, 7, 8, 9, 13, 16, 17, 31, 32, 33, 62, 64, 65])
def test_tables_of_each_layout(cuda, oracle, n_states):
    rng = np.random.default_rng(n_states)
    dfas = [random_dfa(n_states, np.arange(256), rng) for _ in range(2)]
    off = np.arange(0, 4001, dtype=np.int64) * 300
    data = rng.integers(0, 256, size=int(off[-1]), dtype=np.uint8)
    ids = rng.integers(0, 2, size=4000).astype(np.int32)
    _check(cuda, oracle, dfas, data, off, ids, 256)


# Queues shared out to a CTA's warps: fewer batches than CTAs, one more than a share, one automaton
# with most of the items among many with a few, letters of 16 (32 items a claim), large automata.
@pytest.mark.parametrize("case", ["one_short", "a_share_and_one", "uneven", "letters", "large"])
def test_short_queues(cuda, oracle, case):
    from trex_b200.engine import DFASet
    rng = np.random.default_rng(len(case))
    letters = np.arange(65, 81, dtype=np.uint8)
    sizes, n = {"one_short": ([40], 50), "a_share_and_one": ([16], 64 * 149), "uneven": ([8, 16, 64] * 20, 9000),
                "letters": ([12], 9000), "large": ([100, 250, 7], 3000)}[case]
    dfas = [random_dfa(k, letters if case == "letters" else np.arange(256), rng) for k in sizes]
    lens = rng.integers(0, 3000, size=n)
    off = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(lens, out=off[1:])
    data = rng.integers(0, 256, size=int(off[-1]), dtype=np.uint8)
    if case == "letters":
        data = letters[data & 15]
    ids = np.where(rng.random(n) < 0.7, 0, rng.integers(0, len(dfas), size=n)).astype(np.int32)
    s = DFASet(dfas, kgram=0 if case == "letters" else None)
    for seg in (512, 2048):
        fs, ac, _ = s.run(*(cuda.from_numpy(x).cuda() for x in (data, off, ids)), seg_len=seg)
        want, wacc = oracle.dfa_walk([d.tmap for d in dfas], [d.n_states for d in dfas], [0] * len(dfas),
                                     [d.accept for d in dfas], data, off, ids)
        assert s.last_error_word() == 0
        assert np.array_equal(fs.cpu().numpy(), want) and np.array_equal(ac.cpu().numpy(), wacc)
    s.close()
