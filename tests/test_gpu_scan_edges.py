"""Per-position scan at its edges: automata of either table layout, batches off the word
grid, empty strings among more strings than the planning block has threads, automata
that never synchronise."""

import numpy as np
import pytest

from trex_b200.workloads import ByteDFA, random_dfa

pytestmark = pytest.mark.gpu


def _dfa(n, rng, permutation):
    if not permutation:
        return random_dfa(n, np.arange(256), rng)
    t = np.stack([rng.permutation(n) for _ in range(256)]).astype(np.uint8)
    acc = np.zeros(n, dtype=np.uint8)
    acc[n // 2] = 1
    return ByteDFA(n_states=n, tmap=np.ascontiguousarray(t.reshape(-1)), accept=acc, start=0)


# lengths around the 16-byte steps of the sync phase and the tile length, and none
LENS = {"edges": [0, 1, 3, 15, 16, 17, 31, 33, 63, 64, 65, 127, 129, 0, 500, 1023, 1024, 1025, 2049],
        "many": [0, 1, 7, 40] * 700 + [3000]}


@pytest.mark.parametrize("n,permutation", [(3, False), (8, False), (8, True), (9, False), (16, False), (16, True)])
@pytest.mark.parametrize("shape", sorted(LENS))
@pytest.mark.parametrize("lead", [0, 5])
@pytest.mark.parametrize("tile", [0, 64, 100])
def test_scan_edges(cuda, oracle, n, permutation, shape, lead, tile):
    torch = cuda
    from trex_b200.engine import DFASet
    rng = np.random.default_rng(n + lead + tile)
    dfa = _dfa(n, rng, permutation)
    off = np.zeros(len(LENS[shape]) + 1, dtype=np.int64)
    np.cumsum(LENS[shape], out=off[1:])
    data = rng.integers(0, 256, size=int(off[-1]), dtype=np.uint8)
    # the batch starts `lead` bytes into its allocation and ends at the allocation's end
    whole = torch.from_numpy(np.concatenate([np.zeros(lead, np.uint8), data])).cuda()
    s = DFASet([dfa])
    st, fs, ac, scratch = s.scan(whole[lead:], torch.from_numpy(off).cuda(), tile_len=tile)
    torch.cuda.synchronize()
    assert s.scan_error_word(scratch, len(off) - 1, data.size, tile) == 0
    s.close()
    ref = oracle.dfa_positions(dfa.tmap, n, 0, data, off)
    assert np.array_equal(st.cpu().numpy(), ref)
    want = np.array([ref[off[i + 1] - 1] if off[i + 1] > off[i] else 0 for i in range(len(off) - 1)])
    assert np.array_equal(fs.cpu().numpy(), want)
    assert np.array_equal(ac.cpu().numpy(), dfa.accept[want])
