"""Small batches at the default item length run as one launch (a lane or a warp a
string, or pieces of it on several CTAs): every form against the C oracle and the planned path (an explicit
item length), bit-exact."""

import numpy as np
import pytest

from trex_b200.workloads import ByteDFA, random_dfa

pytestmark = pytest.mark.gpu


def _permutation_dfa(n, rng):
    """Every byte permutes the states: two chains never meet, so every guess but one fails."""
    t = np.stack([rng.permutation(n) for _ in range(256)]).astype(np.uint8)
    acc = np.zeros(n, dtype=np.uint8)
    acc[0] = 1
    return ByteDFA(n_states=n, tmap=np.ascontiguousarray(t.reshape(-1)), accept=acc, start=n - 1)


def _batch(lens, rng, lead=0):
    off = np.zeros(len(lens) + 1, dtype=np.int64)
    np.cumsum(lens, out=off[1:])
    off += lead
    return rng.integers(0, 256, size=int(off[-1]), dtype=np.uint8), off


def _run(torch, s, data, off, ids, seg_len):
    d = torch.from_numpy(data).cuda()
    i = None if ids is None else torch.from_numpy(ids.astype(np.int32)).cuda()
    fs, ac, ai = s.run(d, torch.from_numpy(off).cuda(), i, seg_len=seg_len,
                       want=("final_state", "accept", "accept_i32"))
    torch.cuda.synchronize()
    return fs.cpu().numpy(), ac.cpu().numpy(), ai.cpu().numpy(), s.last_error_word()


def _expect(oracle, dfas, data, off, ids):
    fs, _ = oracle.dfa_walk([d.tmap for d in dfas], [d.n_states for d in dfas], [d.start for d in dfas],
                            [d.accept for d in dfas], data, off, np.asarray(ids, dtype=np.int32))
    return fs


# lengths at the edges of the windows, of the lane / warp / CTA rule and of the shares
EDGES = [0, 1, 15, 31, 32, 33, 63, 64, 65, 96, 127, 129, 1000, 1023, 1024, 1025, 1056, 2048, 4100]
SHAPES = {
    "edges": EDGES * 3,
    "one": [777],
    "one_long": [300001],                       # pieces on several CTAs
    # either side of the long-string rule, and of one, two and three pieces
    "long_edge": [16383, 16384, 16385, 32730, 32768, 32769, 65529, 65536, 65560, 98304, 98305],
    "many_short": [5, 40, 64, 90, 200] * 4000,  # several strings a warp, a string a lane
    "long_among_short": [40] * 6000 + [5000, 33000, 70001] + [17] * 6000 + [200000],
    "most_bytes": [2] * 3 + [(8 << 20) - 13],   # the largest batch of the path, and the most pieces
}


@pytest.mark.parametrize("shape", sorted(SHAPES))
@pytest.mark.parametrize("states", [(5,), (8, 16, 12), (17, 64), (200, 3), (250, 255, 256)])
def test_small_batch_matches_oracle_and_planned_path(cuda, oracle, shape, states):
    rng = np.random.default_rng(sum(states) + len(shape))
    lens = np.array(SHAPES[shape], dtype=np.int64)
    dfas = [random_dfa(n, np.arange(256), rng) for n in states]
    data, off = _batch(lens, rng, lead=7)   # the first string starts off the window grid
    ids = rng.integers(0, len(dfas), size=len(lens))
    from trex_b200.engine import DFASet
    s = DFASet(dfas)
    fs, ac, ai, err = _run(cuda, s, data, off, ids, 0)
    assert err == 0
    pf, pa, pi, perr = _run(cuda, s, data, off, ids, 2048)
    s.close()
    want = _expect(oracle, dfas, data, off, ids)
    assert perr == 0 and np.array_equal(pf, want)
    assert np.array_equal(fs, want)
    assert np.array_equal(ac, pa) and np.array_equal(ai, pi)


@pytest.mark.parametrize("n_states", [2, 16, 17, 40])
@pytest.mark.parametrize("lens", [[3000] * 40, [100000, 20000, 33000]], ids=["warp", "pieces"])
def test_small_batch_automata_that_never_synchronise(cuda, oracle, n_states, lens):
    rng = np.random.default_rng(n_states)
    dfa = _permutation_dfa(n_states, rng)
    data, off = _batch(np.array(lens, dtype=np.int64), rng)
    from trex_b200.engine import DFASet
    s = DFASet([dfa])
    fs, _, _, err = _run(cuda, s, data, off, None, 0)
    s.close()
    assert err == 0
    assert np.array_equal(fs, _expect(oracle, [dfa], data, off, np.zeros(len(lens), dtype=int)))


def _keep_state_dfa(n):
    """No byte changes the state: only the lane beside the start is wrong, then the next one."""
    acc = np.zeros(n, dtype=np.uint8)
    acc[n - 1] = 1
    return ByteDFA(n_states=n, tmap=np.tile(np.arange(n, dtype=np.uint8), 256), accept=acc, start=n - 1)


# state maps of whole pieces: shares of 8 to 256 states, one piece, odd ends, many pieces
@pytest.mark.parametrize("n_states", [1, 2, 8, 9, 16, 17, 100, 129, 256])
@pytest.mark.parametrize("make", [_permutation_dfa, lambda n, rng: _keep_state_dfa(n)], ids=["permutes", "keeps"])
def test_small_batch_pieces_as_state_maps(cuda, oracle, n_states, make):
    rng = np.random.default_rng(n_states)
    dfas = [make(n_states, rng), random_dfa(5, np.arange(256), rng)]
    lens = np.array([16385, 32768, 32769, 70001, 400, 16000, 131072 + 5, 900, 300003], dtype=np.int64)
    data, off = _batch(lens, rng, lead=13)
    ids = np.array([0, 0, 0, 0, 0, 0, 0, 1, 0])
    from trex_b200.engine import DFASet
    s = DFASet(dfas)
    fs, ac, ai, err = _run(cuda, s, data, off, ids, 0)
    assert err == 0
    assert np.array_equal(fs, _expect(oracle, dfas, data, off, ids))
    assert np.array_equal(ac, ai) and np.array_equal(ac, [dfas[d].accept[f] for d, f in zip(ids, fs)])
    every, _ = s.run_all(cuda.from_numpy(data).cuda(), cuda.from_numpy(off).cuda())
    s.close()
    for d in (0, 1):
        assert np.array_equal(every[d].cpu().numpy(), _expect(oracle, dfas, data, off, np.full(len(lens), d)))


# The one launch may not cost automata that never synchronise what it saves the others: against the
# planned path on the same batch (the forms differ by far more than the tolerance where one degenerates).
@pytest.mark.parametrize("n_states", [8, 24, 100, 256])
@pytest.mark.parametrize("shape", [(30, 100000), (200, 40000), (8000, 1000)])
def test_small_batch_never_synchronising_is_not_slower(cuda, n_states, shape):
    torch = cuda
    from trex_b200.engine import DFASet
    rng = np.random.default_rng(n_states)
    s = DFASet([_permutation_dfa(n_states, rng)])
    data, off = (torch.from_numpy(x).cuda() for x in _batch(np.full(shape[0], shape[1]), rng))
    best = {}
    for seg in (0, 2048, 0, 2048):
        for _ in range(6):
            t0, t1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            t0.record()
            s.run(data, off, seg_len=seg)
            t1.record()
            t1.synchronize()
            best[seg] = min(best.get(seg, 1e9), t0.elapsed_time(t1))
    s.close()
    assert best[0] <= 1.5 * best[2048], best


def test_small_batch_every_automaton(cuda, oracle):
    torch = cuda
    rng = np.random.default_rng(3)
    dfas = [random_dfa(n, np.arange(256), rng) for n in (3, 8, 16, 33)]
    data, off = _batch(np.array(EDGES * 5 + [20000, 90001, 17], dtype=np.int64), rng)
    from trex_b200.engine import DFASet
    s = DFASet(dfas)
    fs, _ = s.run_all(torch.from_numpy(data).cuda(), torch.from_numpy(off).cuda())
    fs = fs.cpu().numpy()
    s.close()
    n = len(off) - 1
    for d in range(len(dfas)):
        assert np.array_equal(fs[d], _expect(oracle, dfas, data, off, np.full(n, d)))


def test_small_batch_malformed_strings_are_flagged_and_skipped(cuda, oracle):
    torch = cuda
    rng = np.random.default_rng(4)
    dfas = [random_dfa(n, np.arange(256), rng) for n in (8, 16)]
    data, off = _batch(np.array([50, 60, 70, 800, 40], dtype=np.int64), rng)
    from trex_b200.engine import DFASet
    s = DFASet(dfas)
    want = _expect(oracle, dfas, data, off, np.array([0, 1, 0, 1, 0]))
    for case, bad, bit in (("id", [1], 2), ("offset", [1, 2], 1)):
        o, ids = off.copy(), np.array([0, 1, 0, 1, 0])
        if case == "id":
            ids[1] = 2
        else:
            o[2] = data.size + 5   # string 1 ends past the batch, string 2 is reversed
        out = []
        for seg in (0, 2048):   # the same bits and the same strings left alone on both paths
            d, do = torch.from_numpy(data).cuda(), torch.from_numpy(o).cuda()
            fs = torch.full((5,), 99, dtype=torch.uint8, device="cuda")
            s.run(d, do, torch.from_numpy(ids.astype(np.int32)).cuda(), final_state=fs, seg_len=seg)
            torch.cuda.synchronize()
            out.append((fs.cpu().numpy(), s.last_error_word()))
        assert out[0][1] == out[1][1] == bit
        good = [i for i in range(5) if i not in bad]
        for fs, _ in out:
            assert np.array_equal(fs[good], want[good]) and np.all(fs[bad] == 99)
    s.close()
