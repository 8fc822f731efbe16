"""Prune and merge at the list lengths where their teams of warps change (32, 64, 128 entries), strict
and not, on lists with tombs, the node itself, repeated ids and equal rows: pruned lists, reverse
lists, merged rows and evaluation counts equal the oracle's."""
import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOMB = 0xFFFFFFFF


@pytest.fixture(scope="module")
def pg():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import paragraph_gb300
    paragraph_gb300.lib()
    return paragraph_gb300


def _dev(a):
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda()


def _u32(t):
    return t.cpu().numpy().view(np.uint32)


def _data(n, d, c):
    rng = np.random.default_rng(100 * c + d)
    base = rng.standard_normal((n, d)).astype(np.float32)
    base *= rng.uniform(0.3, 2.0, (n, 1)).astype(np.float32)
    base[n // 2:n // 2 + 50] = base[:50]
    graph = rng.integers(0, n, (n, c)).astype(np.uint32)
    graph[rng.random((n, c)) < 0.5 * rng.random((n, 1))] = TOMB
    graph[::5, c // 2] = np.arange(0, n, 5)  # the node itself
    graph[::7] = graph[::7, :1]  # one id all along
    graph[::11] = TOMB
    graph[3::11, 1:] = TOMB  # the node alone
    graph[3::11, 0] = np.arange(3, n, 11)
    return base, graph


@pytest.mark.parametrize("d", [8, 200, 260])
@pytest.mark.parametrize("c,p,r", [(2, 2, 5), (32, 15, 17), (33, 9, 23), (64, 32, 94),
                                   (65, 55, 71), (128, 15, 111), (128, 100, 28)])
@pytest.mark.parametrize("strict", [True, False])
def test_prune_and_merge_equal_oracle(pg, d, c, p, r, strict):
    n = 610
    base, graph = _data(n, d, c)
    degree = max(2, (p + r) // 3)
    ref = oracle.prune_reverse(base, graph, p, r, strict)
    want, want_ev = oracle.merge_prune(base, ref, degree, strict)
    pruned = torch.full((n, p), -1, dtype=torch.int32, device="cuda")
    rev = torch.full((n, r), -1, dtype=torch.int32, device="cuda")
    pnum, rnum = torch.empty((2, n), dtype=torch.int32, device="cuda")
    out = torch.empty((n, degree), dtype=torch.int32, device="cuda")
    with pg.Handle(0) as h:
        b = _dev(base)
        ev = h.prune_reverse(b, _dev(graph), pruned, pnum, rev, rnum, strict)
        mev = h.merge_prune(b, pruned, pnum, rev, rnum, out, strict)
    assert np.array_equal(_u32(pnum), ref.pruned_num)
    assert np.array_equal(_u32(rnum), ref.reverse_num)
    for i in range(n):
        k, m = ref.pruned_num[i], ref.reverse_num[i]
        assert np.array_equal(_u32(pruned)[i, :k], ref.pruned[i, :k]), i
        assert np.array_equal(_u32(rev)[i, :m], ref.reverse[i, :m]), i
    assert ev == ref.evals
    assert np.array_equal(_u32(out), want)
    assert mev == want_ev


@pytest.mark.parametrize("n", [1, 31, 1025, 4096, 4097, 8193])  # one-block scans and tiled ones
@pytest.mark.parametrize("r", [7, 111])
def test_reverse_lists_of_hubs_equal_oracle(pg, n, r):
    rng = np.random.default_rng(n)
    base = rng.standard_normal((n, 8)).astype(np.float32)
    base[0] *= 50.0  # a hub: nearest for about half of the nodes
    graph = rng.integers(0, n, (n, 6)).astype(np.uint32)
    graph[:, 2] = 0
    graph[rng.permutation(n), 3] = rng.integers(0, max(1, n // 50), n)
    ref = oracle.prune_reverse(base, graph, 6, r, False)
    pruned = torch.full((n, 6), -1, dtype=torch.int32, device="cuda")
    rev = torch.full((n, r), -1, dtype=torch.int32, device="cuda")
    pnum, rnum = torch.empty((2, n), dtype=torch.int32, device="cuda")
    with pg.Handle(0) as h:
        for _ in range(2):  # the second call finds the workspace that the first one left
            h.prune_reverse(_dev(base), _dev(graph), pruned, pnum, rev, rnum, False)
    assert np.array_equal(_u32(pnum), ref.pruned_num)
    assert np.array_equal(_u32(rnum), ref.reverse_num)
    want = np.where(np.arange(r)[None, :] < ref.reverse_num[:, None], ref.reverse, 0)
    got = np.where(np.arange(r)[None, :] < ref.reverse_num[:, None], _u32(rev), 0)
    assert np.array_equal(got, want)
