"""Tensor-core NFA forms with a string on each TMEM lane (one to four symbols): string counts
around the tiles of 128, lanes that take a next string, skipped bytes; against the oracle."""

import numpy as np
import pytest

from trex_b200.workloads import random_bool_nfa, random_prob_nfa

pytestmark = pytest.mark.gpu


# one string, a tile but one, a tile, two tiles begun, one CTA's four tiles and one more, refills
@pytest.mark.parametrize("sigma,n", [(1, 1), (2, 127), (2, 128), (3, 129), (2, 513), (4, 20000), (2, 100000)])
@pytest.mark.parametrize("mode", ["bf16", "fp16", "bool", "bool8"])
def test_tiles(cuda, oracle, sigma, n, mode):
    from trex_b200.engine import PNFA
    rng = np.random.default_rng(sigma * 1000 + n)
    boolean = mode.startswith("bool")
    T, start, acc = (random_bool_nfa(rng, 64, sigma, density=0.03) if boolean
                     else random_prob_nfa(rng, 64, sigma))
    T, start, acc = (np.asarray(x, np.float32) for x in (T, start, acc))
    lens = rng.integers(0, 60, size=n) if n > 1 else np.array([2000])
    off = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(lens, out=off[1:])
    data = rng.integers(0, sigma, size=int(off[-1]), dtype=np.uint8)
    if n > 1:
        data[rng.random(data.size) < 0.05] = 200
    m = PNFA(T, start, acc)
    ll, ac = m.run(cuda.from_numpy(data).cuda(), cuda.from_numpy(off).cuda(), mode)
    cuda.cuda.synchronize()
    assert m.error_word() == 0
    m.close()
    ll, ac = ll.cpu().numpy(), ac.cpu().numpy().astype(bool)
    if boolean:
        _, ref = oracle.nfa_bool(T != 0, start, acc, data, off, unknown_rejects=False)
        assert np.array_equal(ac, ref.astype(bool))
        return
    ref = oracle.pnfa_fp64(T, start, acc, data, off)
    # 16-bit rounding of table and state: half a unit in the last place a step at most, and never as
    # much as half a power of two (an exponent lost by the rescaling is ln 2)
    u = {"bf16": 2.0 ** -8, "fp16": 2.0 ** -11}[mode]
    fin = np.isfinite(ref)
    assert np.array_equal(np.isfinite(ll), fin)
    tol = np.maximum(1e-4 * np.abs(ref), np.minimum(u * (np.diff(off) + 1), np.log(2) / 2))
    assert np.all(np.abs(ll - ref)[fin] <= tol[fin])
    clear = fin & (np.abs(ref - np.log(0.5)) > tol)
    assert np.array_equal(ac[clear], ref[clear] > np.log(0.5)) and not ac[~fin].any()
