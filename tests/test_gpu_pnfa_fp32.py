"""FP32 probabilistic NFA with the tables on the SM (up to 20 symbols) and through L1 (more),
against the FP64 oracle and against each other."""

import numpy as np
import pytest

from trex_b200.workloads import random_prob_nfa

pytestmark = pytest.mark.gpu


def _run(torch, T, start, acc, data, off):
    from trex_b200.engine import PNFA
    m = PNFA(T, start, acc)
    d = torch.from_numpy(np.ascontiguousarray(data)).cuda()
    ll, ac = m.run(d, torch.from_numpy(off).cuda(), "fp32")
    torch.cuda.synchronize()
    err = m.error_word()
    m.close()
    return ll.cpu().numpy(), ac.cpu().numpy(), err


# one symbol, warps shared by few symbols, all warps a symbol each, the first past the rule;
# one string, fewer than an SM's groups, more strings than slots
@pytest.mark.parametrize("sigma", [1, 2, 3, 7, 11, 20, 21])
@pytest.mark.parametrize("n", [1, 100, 12000])
def test_fp32_rings(cuda, oracle, sigma, n):
    rng = np.random.default_rng(sigma * 31 + n)
    T, start, acc = random_prob_nfa(rng, 64 if sigma % 2 else 37, sigma)
    T, start, acc = (x.astype(np.float32) for x in (T, start, acc))
    lens = rng.integers(0, 30, size=n) if n > 1 else np.array([3000])
    off = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(lens, out=off[1:])
    data = rng.integers(0, sigma, size=int(off[-1]), dtype=np.uint8)
    if n > 1:   # bytes outside the alphabet are skipped, strings of nothing else too
        data[rng.random(data.size) < 0.1] = 200
    ll, ac, err = _run(cuda, T, start, acc, data, off)
    assert err == 0
    ref = oracle.pnfa_fp64(T, start, acc, data, off)
    # one rounding of a 64-term sum a step: 64 half-ulps at most, far fewer in the mean
    k = np.diff(off)
    assert np.array_equal(np.isinf(ll), np.isinf(ref))
    ok = np.isfinite(ref)
    assert np.all(np.abs(ll - ref)[ok] <= np.maximum(1e-5 * np.abs(ref), 1e-7 * (k + 1))[ok])
    assert np.array_equal(ac.astype(bool), ref > np.log(0.5))


def test_fp32_same_states_with_and_without_an_unused_symbol(cuda):
    # 20 symbols run on the rings, the same automaton with a 21st symbol that no string
    # uses on the plain kernel; both add a row's products in the same order, so the states are
    # the same bits and only the last sum's contraction into FMAs may differ: one rounding of
    # each of two products and their sum, 2^-23 relative, in the dot product
    rng = np.random.default_rng(5)
    T, start, acc = (x.astype(np.float32) for x in random_prob_nfa(rng, 64, 20))
    off = np.arange(0, 501, dtype=np.int64) * 200
    data = rng.integers(0, 20, size=int(off[-1]), dtype=np.uint8)
    a, _, ea = _run(cuda, T, start, acc, data, off)
    b, _, eb = _run(cuda, np.concatenate([T, T[:1]]), start, acc, data, off)
    assert ea == eb == 0
    assert np.all(np.abs(a - b) <= 2.0 ** -22)


def test_fp32_hand_off_gives_up(cuda):
    from trex_b200 import _lib
    torch = cuda
    from trex_b200.engine import PNFA
    rng = np.random.default_rng(6)
    m = PNFA(*random_prob_nfa(rng, 64, 20))
    off = torch.arange(0, 401, dtype=torch.int64).cuda() * 100
    data = torch.from_numpy(rng.integers(0, 20, size=40000, dtype=np.uint8)).cuda()
    lib = _lib.load()
    try:
        _lib.check(lib.trex_set_wait_limits(0, 1), "trex_set_wait_limits")
        m.run(data, off, "fp32")
        torch.cuda.synchronize()
        assert m.error_word() & 4
    finally:
        _lib.check(lib.trex_set_wait_limits(0, 0), "trex_set_wait_limits")
    ll, _ = m.run(data, off, "fp32")
    torch.cuda.synchronize()
    assert m.error_word() == 0 and bool(torch.isfinite(ll).all())
    m.close()


def test_fp32_long_skipped_runs_are_work(cuda, oracle):
    # runs of 16 MiB outside the alphabet, at a string's start and inside it, take many times the
    # wait limit set here; skipping is not a stalled hand-off
    from trex_b200 import _lib
    rng = np.random.default_rng(8)
    T, start, acc = (x.astype(np.float32) for x in random_prob_nfa(rng, 64, 20))
    run, tail = 16 << 20, 37
    off = np.array([0, run + tail, 2 * run + 2 * tail, 2 * run + 2 * tail + 500], dtype=np.int64)
    data = np.full(int(off[-1]), 200, dtype=np.uint8)
    data[run:run + tail] = rng.integers(0, 20, size=tail)                  # skipped bytes first
    data[off[1]:off[1] + 9] = rng.integers(0, 20, size=9)                  # between symbols
    data[off[2] - 21:off[2] - 1] = rng.integers(0, 20, size=20)            # (and one at the end)
    data[off[2]:] = rng.integers(0, 20, size=500)
    lib = _lib.load()
    try:
        _lib.check(lib.trex_set_wait_limits(0, 4_000_000), "trex_set_wait_limits")
        ll, ac, err = _run(cuda, T, start, acc, data, off)
    finally:
        _lib.check(lib.trex_set_wait_limits(0, 0), "trex_set_wait_limits")
    assert err == 0
    ref = oracle.pnfa_fp64(T, start, acc, data, off)
    assert np.all(np.abs(ll - ref) <= 1e-5 * np.abs(ref))   # at most 500 symbols, as above
    assert np.array_equal(ac.astype(bool), ref > np.log(0.5))


# runs of skipped bytes around the words and lines that they are read by, at every alignment of the string
@pytest.mark.parametrize("run", [1, 3, 4, 5, 63, 64, 65, 67, 127, 128, 131, 300])
def test_fp32_skipped_runs_at_every_alignment(cuda, oracle, run):
    rng = np.random.default_rng(run)
    T, start, acc = (x.astype(np.float32) for x in random_prob_nfa(rng, 64, 7))
    parts, off = [], [0]
    for lead in range(70):
        s = [np.full(lead % 3, 9), rng.integers(0, 7, size=lead), np.full(run, 200), rng.integers(0, 7, size=lead % 2),
             np.full(run * (lead % 2), 255)]
        parts.append(np.concatenate(s).astype(np.uint8))
        off.append(off[-1] + len(parts[-1]))
    data, off = np.concatenate(parts), np.array(off, dtype=np.int64)
    ll, _, err = _run(cuda, T, start, acc, data, off)
    ref = oracle.pnfa_fp64(T, start, acc, data, off)
    fin = np.isfinite(ref)
    assert err == 0 and np.array_equal(np.isfinite(ll), fin)
    assert np.all(np.abs(ll - ref)[fin] <= 1e-6 + 1e-5 * np.abs(ref[fin]))   # at most 70 symbols, as above
