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
