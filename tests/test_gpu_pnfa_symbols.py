"""Tensor-core NFA forms with a symbol's table a warp (5 to 28 symbols): alphabets around
the warps a symbol gets, string lengths around the 16-symbol blocks, strings off the
16-byte grid, skipped bytes, more strings than slots; against the oracle."""

import numpy as np
import pytest

from trex_b200.workloads import random_bool_nfa, random_prob_nfa

pytestmark = pytest.mark.gpu

EDGES = [0, 1, 2, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 100]


def _automaton(rng, n, sigma, mode):
    # sparse for the Boolean forms: both outcomes occur
    T, start, acc = (random_bool_nfa(rng, n, sigma, density=1.5 / n) if mode.startswith("bool")
                     else random_prob_nfa(rng, n, sigma))
    return T.astype(np.float32), np.asarray(start, np.float32), np.asarray(acc, np.float32)


def _case(rng, sigma, lens, lead, skip):
    off = np.zeros(len(lens) + 1, dtype=np.int64)
    np.cumsum(lens, out=off[1:])
    off += lead
    data = rng.integers(0, sigma, size=int(off[-1]), dtype=np.uint8)
    if skip:
        data[rng.random(data.size) < skip] = sigma + rng.integers(0, 255 - sigma)
    return data, off


def _run(torch, T, start, acc, data, off, mode):
    from trex_b200.engine import PNFA
    m = PNFA(T, start, acc)
    ll, ac = m.run(torch.from_numpy(data).cuda(), torch.from_numpy(off).cuda(), mode)
    torch.cuda.synchronize()
    err = m.error_word()
    m.close()
    return ll.cpu().numpy(), ac.cpu().numpy(), err


def _check(oracle, T, start, acc, data, off, mode, ll, ac):
    if mode.startswith("bool"):
        _, ref = oracle.nfa_bool(T != 0, start, acc, data, off, unknown_rejects=False)
        assert np.array_equal(ac.astype(bool), ref.astype(bool))
        return
    ref = oracle.pnfa_fp64(T, start, acc, data, off)
    # 16-bit rounding of table and state: half a unit in the last place a step at most, and never as
    # much as half a power of two (an exponent lost by the rescaling is ln 2); long strings by the
    # relative bound of the benchmark
    u = {"bf16": 2.0 ** -8, "fp16": 2.0 ** -11}[mode]
    fin = np.isfinite(ref)
    assert np.array_equal(np.isfinite(ll), fin)
    tol = np.maximum(1e-4 * np.abs(ref), np.minimum(u * (np.diff(off) + 1), np.log(2) / 2))
    assert np.all(np.abs(ll - ref)[fin] <= tol[fin])
    clear = fin & (np.abs(ref - np.log(0.5)) > tol)
    assert np.array_equal(ac.astype(bool)[clear], ref[clear] > np.log(0.5)) and not ac[~fin].any()


# 20 warps: 4 a symbol, 2, 1 with a spare, 1 each; then several symbols a warp
@pytest.mark.parametrize("sigma", [5, 7, 10, 11, 19, 20, 21, 28])
@pytest.mark.parametrize("mode", ["bf16", "fp16", "bool", "bool8"])
def test_alphabets(cuda, oracle, sigma, mode):
    rng = np.random.default_rng(sigma)
    T, start, acc = _automaton(rng, 64, sigma, mode)
    lens = rng.permutation(np.array(EDGES * 40))
    data, off = _case(rng, sigma, lens, 3, 0.03)
    ll, ac, err = _run(cuda, T, start, acc, data, off, mode)
    assert err == 0
    _check(oracle, T, start, acc, data, off, mode, ll, ac)


@pytest.mark.parametrize("mode", ["bf16", "bool8"])
@pytest.mark.parametrize("shape", ["one", "few", "refills", "one_symbol", "only_skipped"])
def test_shapes(cuda, oracle, mode, shape):
    rng = np.random.default_rng(len(shape))
    T, start, acc = _automaton(rng, 50, 20, mode)
    lens = {"one": np.array([5000]), "few": np.array([700, 3, 1200]),
            "refills": rng.integers(0, 40, size=200000),      # more strings than all slots, mostly short
            "one_symbol": np.full(4000, 90), "only_skipped": np.array(EDGES)}[shape]
    data, off = _case(rng, 20, lens, 0, 0.0)
    if shape == "one_symbol":   # every string in one warp's list
        data[:] = 13
    if shape == "only_skipped":
        data[:] = 255
    ll, ac, err = _run(cuda, T, start, acc, data, off, mode)
    assert err == 0
    _check(oracle, T, start, acc, data, off, mode, ll, ac)


def test_growing_states_are_rescaled(cuda, oracle):
    # row sums of about 600: a rescale at every step; and of 12: every fourth
    for scale in (600.0, 12.0):
        rng = np.random.default_rng(3)
        T = rng.random((6, 64, 64)).astype(np.float32) * np.float32(scale / 32)
        start = np.ones(64, dtype=np.float32)
        acc = np.ones(64, dtype=np.float32)
        data, off = _case(rng, 6, np.array([500, 17, 300]), 0, 0.0)
        for mode in ("bf16", "fp16"):
            ll, ac, err = _run(cuda, T, start, acc, data, off, mode)
            assert err == 0
            _check(oracle, T, start, acc, data, off, mode, ll, ac)


def test_int8_tables_of_two_symbols_a_warp_stay_in_registers(cuda):
    # one symbol more than warps costs the eight-string groups of a second list, not a table's
    # load a step (which was 22 times the time of 20 symbols)
    from trex_b200.engine import PNFA
    ms = {}
    for sigma in (20, 21):
        rng = np.random.default_rng(sigma)
        m = PNFA(*_automaton(rng, 64, sigma, "bool8"))
        off = cuda.arange(0, 8193, dtype=cuda.int64, device="cuda") * 256
        data = cuda.from_numpy(rng.integers(0, sigma, size=8192 * 256, dtype=np.uint8)).cuda()
        for _ in range(6):
            t0, t1 = (cuda.cuda.Event(enable_timing=True) for _ in range(2))
            t0.record()
            m.run(data, off, "bool8")
            t1.record()
            t1.synchronize()
            ms[sigma] = min(ms.get(sigma, 1e9), t0.elapsed_time(t1))
        m.close()
    assert ms[21] < 4 * ms[20], ms
