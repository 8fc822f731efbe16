"""The beam search at the edges of its kernel shapes -- row lengths around every K-step boundary,
each beam width, both pass sizes, few and many queries, distances that overflow to infinity -- against the oracle, id for
id with equal evaluation and iteration counts."""
import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pg():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import paragraph_gb300
    paragraph_gb300.lib()
    return paragraph_gb300


def _case(n, d, degree, huge):
    rng = np.random.default_rng(1000 * d + n)
    base = rng.standard_normal((n, d)).astype(np.float32)
    base[n // 2:n // 2 + n // 8] = base[:n // 8]  # equal rows: ties decided by position
    if huge:  # one coordinate near the end of the float range: inner products of both infinities
        rows = rng.choice(n, n // 6, replace=False)
        base[rows, 0] = np.float32(3e38) * rng.choice([-1.0, 1.0], len(rows)).astype(np.float32)
        base[rows, 1:] *= np.float32(1e-3)
    graph = rng.integers(0, n, (n, degree)).astype(np.uint32)
    graph[rng.random((n, degree)) < 0.3] = 0xFFFFFFFF
    return base, graph


@pytest.mark.parametrize("d", [4, 32, 200, 224, 228, 256, 260, 512])
@pytest.mark.parametrize("km,rows", [(32, 8), (32, 16), (64, 8), (96, 8)])
@pytest.mark.parametrize("n", [700, 1500])  # a few queries per SM, and enough to share its registers
def test_search_equals_oracle(pg, d, km, rows, n):
    n, degree = n + d // 4, 16
    base, graph = _case(n, d, degree, huge=d in (32, 260))
    ids, ev, it, _ = oracle.search(base, graph, km=km)
    out = torch.full((n, km + 32), -1, dtype=torch.int32, device="cuda")
    with pg.Handle(0) as h:
        t = h.get_tuning()
        t.search_rows = rows
        h.set_tuning(t)
        b = torch.from_numpy(base).cuda()
        g = torch.from_numpy(graph.view(np.int32)).cuda()
        gev, git = h.search(b, g, out, km=km)
        # the query search takes its pass size from the tuning; its ids are the rows' first ones
        q = torch.from_numpy(base[:257].copy()).cuda()
        qout = torch.full((257, 20), -1, dtype=torch.int32, device="cuda")
        h.query_search(b, g, q, qout, km=km, reset_iter=15)
    got = out.cpu().numpy().view(np.uint32)
    assert np.array_equal(got, ids)
    assert (gev, git) == (ev, it)
    assert np.array_equal(qout.cpu().numpy().view(np.uint32), ids[:257, :20])
