"""Merges whose rows are longer than their lists, over lists that hold an id several times and keep
every one of its entries: the fill then lists more ids than the merged list has entries.  Rows and
evaluation counts equal the oracle's."""
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


# merged lists of 32 (one warp) and 128 entries (four warps), every id `times` times
@pytest.mark.parametrize("p,r,degree", [(16, 16, 33), (16, 16, 40), (16, 16, 126), (64, 64, 126),
                                        (64, 64, 129), (64, 64, 260)])
@pytest.mark.parametrize("times", [2, 4, 16])
def test_repeated_ids_kept_more_than_once(pg, p, r, degree, times):
    n, d = 300, 16
    rng = np.random.default_rng(p + times)
    base = np.abs(rng.standard_normal((n, d))).astype(np.float32)
    base[:20] *= 50.0  # long rows: no short row lies closer to a short row than they do
    ids = np.array([rng.choice(np.arange(20, n), (p + r) // times, replace=False)
                    for _ in range(n)], dtype=np.uint32)
    lists = np.repeat(ids, times, axis=1)
    pr = oracle.PruneResult(lists[:, :p].copy(), np.full(n, p, np.uint32), lists[:, p:].copy(),
                            np.full(n, r, np.uint32), None, 0)
    want, want_ev = oracle.merge_prune(base, pr, degree, False)
    listed = (want != TOMB).sum(axis=1)
    kept = p + r  # every entry, then the repeats once more
    assert (listed[:20] == min(degree, 2 * kept - kept // times)).all()
    out = torch.full((n, degree), -1, dtype=torch.int32, device="cuda")
    with pg.Handle(0) as h:
        ev = h.merge_prune(_dev(base), _dev(pr.pruned), _dev(pr.pruned_num), _dev(pr.reverse),
                           _dev(pr.reverse_num), out, False)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
    assert ev == want_ev
