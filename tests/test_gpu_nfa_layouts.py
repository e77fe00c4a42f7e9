"""Table layouts of the bit-parallel NFA (group widths, 16-, 32- and 64-state words)
against the C oracle."""

import numpy as np
import pytest

from trex_b200.workloads import random_bool_nfa

pytestmark = pytest.mark.gpu


def _run(torch, T, start, acc, data, off, rejects):
    from trex_b200.engine import NFA
    nfa = NFA(T, start, acc, unknown_rejects=rejects)
    d = torch.from_numpy(np.ascontiguousarray(data)).cuda()
    fm, ac = nfa.run(d, torch.from_numpy(off).cuda())
    torch.cuda.synchronize()
    err = nfa.error_word()
    nfa.close()
    return fm.cpu().numpy().view(np.uint64), ac.cpu().numpy(), err


def _batch(lens, sigma, rng, lead=0):
    off = np.zeros(len(lens) + 1, dtype=np.int64)
    np.cumsum(lens, out=off[1:])
    off += lead
    return rng.integers(0, sigma, size=int(off[-1]), dtype=np.uint8), off


def _check(torch, oracle, T, start, acc, data, off, rejects):
    fm, ac, err = _run(torch, T, start, acc, data, off, rejects)
    rfm, rac = oracle.nfa_bool(T, start, acc, data, off, unknown_rejects=rejects)
    assert err == 0
    assert np.array_equal(fm, rfm) and np.array_equal(ac, rac)


# the last alphabet of every layout and the first of the next: 64 states in 8 to 16 groups and
# from global memory, 32 states in 4 to 7 groups, 16 states in 2
@pytest.mark.parametrize("n,sigma", [(64, s) for s in (12, 13, 21, 22, 30, 31, 43, 44, 54, 55, 69, 70, 109, 110)] +
                         [(33, 20), (32, 54), (32, 55), (32, 124), (32, 125), (32, 219), (32, 220),
                          (17, 255), (16, 109), (16, 110), (9, 3)])
def test_layouts(cuda, oracle, n, sigma):
    rng = np.random.default_rng(1000 * n + sigma)
    T, start, acc = random_bool_nfa(rng, n, sigma, min(0.5, 2.5 / n))
    data, off = _batch(rng.integers(0, 90, size=300), min(256, sigma + 1), rng)
    _check(cuda, oracle, T, start, acc, data, off, rejects=False)
