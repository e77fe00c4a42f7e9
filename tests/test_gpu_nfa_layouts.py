"""Table layouts of the bit-parallel NFA (group widths, 16-, 32- and 64-state words)
and strings cut into units, against the C oracle."""

import numpy as np
import pytest

from trex_b200.workloads import random_bool_nfa

pytestmark = pytest.mark.gpu


def _run(torch, T, start, acc, data, off, rejects):
    from trex_b200.engine import NFA
    nfa = NFA(T, start, acc, unknown_rejects=rejects)
    d = torch.from_numpy(np.ascontiguousarray(data)).cuda()
    fm, ac = nfa.run(d, torch.from_numpy(off).cuda())
    fm2, _ = nfa.run(d, torch.from_numpy(off).cuda())   # the handle's units again
    torch.cuda.synchronize()
    err = nfa.error_word()
    nfa.close()
    assert torch.equal(fm, fm2)
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


def _shift_nfa(n, sigma):
    """Every symbol rotates the states: the sets from all states never shrink, no guess holds."""
    T = np.zeros((sigma, n, n), dtype=np.int8)
    for c in range(sigma):
        for j in range(n):
            T[c, (j + 1 + c) % n, j] = 1
    start = np.zeros(n, dtype=np.int8)
    start[0] = 1
    acc = np.zeros(n, dtype=np.int8)
    acc[: n // 3 + 1] = 1
    return T, start, acc


def _late_nfa(n, sigma):
    """Symbol 0 rotates, the others reset to state 0: guesses hold only after a reset, so some
    units of a string are walked again."""
    T, start, acc = _shift_nfa(n, sigma)
    T[1:] = 0
    T[1:, 0, :] = 1
    return T, start, acc


# around the shortest unit (512 bytes past the first 16-byte boundary), several units, one long
LENS = {"edges": [0, 1, 15, 16, 511, 512, 513, 526, 527, 528, 529, 1023, 1024, 1025, 1040, 1537, 5000] * 4,
        "one": [200003], "mixed": [20] * 500 + [30000, 4097, 700] * 3 + [300] * 400}


@pytest.mark.parametrize("kind", ["random", "shift", "late", "dies"])
@pytest.mark.parametrize("shape", sorted(LENS))
@pytest.mark.parametrize("n", [64, 20])
def test_strings_cut_into_units(cuda, oracle, kind, shape, n):
    rng = np.random.default_rng(n + len(kind) + len(shape))
    sigma = 6
    data, off = _batch(np.array(LENS[shape], dtype=np.int64), sigma, rng, lead=5)
    if kind == "random":
        T, start, acc = random_bool_nfa(rng, n, sigma, 3.0 / n)
    elif kind == "shift":
        T, start, acc = _shift_nfa(n, sigma)
    else:
        T, start, acc = _late_nfa(n, sigma)
        data = np.where(rng.random(data.size) < 0.002, data, 0).astype(np.uint8)
    rejects = kind == "dies"   # a byte outside the alphabet empties the set
    if rejects:
        data[rng.integers(0, data.size, size=3)] = sigma + 1
    _check(cuda, oracle, T, start, acc, data, off, rejects)


def test_cut_string_past_four_billion(cuda, oracle):
    # a cut string whose index needs more than 32 bits (its units are found by that index)
    from trex_b200.engine import NFA
    if cuda.cuda.mem_get_info()[0] < 100 << 30:
        pytest.skip("needs 75 GB of device memory")
    rng = np.random.default_rng(9)
    T, start, acc = random_bool_nfa(rng, 64, 20, density=0.05)
    n, L = (1 << 32) + 3, 200003
    data = rng.integers(0, 20, size=L, dtype=np.uint8)
    off = cuda.zeros(n + 1, dtype=cuda.int64, device="cuda")
    off[-2:] = L                                   # string 2^32 + 1; the one after it is empty
    m = NFA(T, start, acc, unknown_rejects=False)
    mask, ok = m.run(cuda.from_numpy(data).cuda(), off)
    assert m.error_word() == 0
    want, wacc = oracle.nfa_bool(T, start, acc, data, np.array([0, L, L]), unknown_rejects=False)
    m.close()
    for i, k in ((n - 2, 0), (n - 1, 1), (0, 1), (1, 1), (n - 3, 1)):
        assert int(mask[i].item()) & (1 << 64) - 1 == int(np.uint64(want[k])) and int(ok[i].item()) == int(wacc[k])
    del off, mask, ok
    cuda.cuda.empty_cache()
