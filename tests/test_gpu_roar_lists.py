"""MatchSup, FusionNN and FusionFinal with lists on both sides of the one-warp limit, narrow and wide
prunes, rows with every tail of the distance order, tombs, repeated ids and equal rows: ids equal the
oracle's list for list."""
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


def _dev(a):
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda()


def _rows(out, cnt):
    o, k = out.cpu().numpy().view(np.uint32), cnt.cpu().numpy().view(np.uint32)
    return [o[i, :k[i]] for i in range(len(k))]


def _csr(off, ids):
    return [ids[off[i]:off[i + 1]] for i in range(len(off) - 1)]


def _u32(*shape):
    return torch.full(shape, -1, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("d", [4, 28, 40, 200])
@pytest.mark.parametrize("m_nn,m_final,gt_k", [(4, 9, 34), (20, 33, 128), (40, 70, 40), (64, 128, 200)])
def test_lists_equal_oracle(pg, d, m_nn, m_final, gt_k):
    n, q, rounds = 900, 2500, min(256 // m_nn, 5)
    rng = np.random.default_rng(d + m_nn)
    base = rng.standard_normal((n, d)).astype(np.float32)
    base *= rng.uniform(0.2, 3.0, (n, 1)).astype(np.float32)  # hubs
    base[n // 2:n // 2 + 60] = base[:60]
    queries = rng.standard_normal((q, d)).astype(np.float32)
    gt = np.argsort(-(queries @ base.T), axis=1, kind="stable")[:, :gt_k].astype(np.uint32)
    gt[::9, gt_k // 2:] = 0xFFFFFFFF
    gt[::11, 3] = gt[::11, 2]  # a repeated id
    sup = _u32(rounds, n, m_nn)
    supc = _u32(rounds, n)
    ref = []
    with pg.Handle(0) as h:
        db, dg = _dev(base), _dev(gt)
        for r in range(rounds):
            h.match_sup(db, dg, r + 1, sup[r], supc[r], m_nn=m_nn)
            ref.append(oracle.match_sup(base, gt, r + 1, m_nn))
            got = _rows(sup[r], supc[r])
            for i, want in enumerate(_csr(*ref[r])):
                assert np.array_equal(got[i], want), (r, i)
        out, cnt = _u32(n, 2 * m_nn), _u32(n)
        h.fusion_nn(db, sup, supc, out, cnt, m_nn=m_nn)
        fnn = oracle.fusion_nn(base, ref, m_nn)
        for i, (a, b) in enumerate(zip(_rows(out, cnt), _csr(*fnn))):
            assert np.array_equal(a, b), i
        link = rng.integers(0, n, (n, 48)).astype(np.uint32)
        link[rng.random((n, 48)) < rng.random((n, 1))] = 0xFFFFFFFF
        link[::7, 5] = np.arange(0, n, 7)  # the node itself
        proj = rng.integers(0, n, (n, 16)).astype(np.uint32)
        proj[::2] = 0xFFFFFFFF
        stride = 2 * m_nn + m_final
        fin, fcnt = _u32(n, stride), _u32(n)
        h.fusion_final(db, _dev(proj), _dev(link), fin, fcnt, bip_rows=out, bip_cnt=cnt,
                       m_final=m_final)
        want = _csr(*oracle.fusion_final(base, proj, fnn, link, m_final))
        for i, (a, b) in enumerate(zip(_rows(fin, fcnt), want)):
            assert np.array_equal(a, b), i
