"""Builds large enough to work on the relocated copy of the base (32 MB and more): graph,
projection and evaluation counts equal the oracle's, and a batched build equals building each
sub-index alone, below the limit.  The data hold equal rows (ties), hubs whose reverse lists
overflow, and ground truth padded with tombs."""
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


def _data(n, d, q, seed, cosine=False):
    from paragraph_gb300 import datagen
    base, gt, _ = datagen.make_dataset_cuda(n, d, q, seed=seed, cosine=cosine, return_queries=True)
    base, gt = base.cpu().numpy(), gt.cpu().numpy().view(np.uint32).copy()
    base[n // 2:n // 2 + n // 50] = base[:n // 50]
    base[7] *= 3.0  # a hub
    gt[::3, 90:] = TOMB
    gt[::5, 0] = 7
    return base, gt


def _dev(a):
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda()


def _build(pg, base, gt, params):
    graph = torch.full((base.shape[0], params.degree), -1, dtype=torch.int32, device="cuda")
    proj = torch.full((base.shape[0], 16), -1, dtype=torch.int32, device="cuda")
    with pg.Handle(0) as h:
        st = h.build_device(_dev(base), _dev(gt), graph, proj, params)
    return graph.cpu().numpy().view(np.uint32), proj.cpu().numpy().view(np.uint32), st


@pytest.mark.parametrize("n,d,q,degree,beam,screen,cosine", [
    (42_001, 200, 30_000, 32, 64, 3, False),
    (16_501, 512, 16_501, 48, 96, 1, True),
    (20_011, 420, 25_000, 55, 64, 0, True),
])
def test_relocated_build_equals_oracle(pg, n, d, q, degree, beam, screen, cosine):
    assert n * d * 4 >= 32 << 20
    base, gt = _data(n, d, q, seed=d, cosine=cosine)
    ref = oracle.build_graph(base, gt, degree=degree, beam=beam)
    graph, proj, st = _build(pg, base, gt, pg.default_params(degree, beam, screen=screen))
    assert np.array_equal(graph, ref["graph"])
    assert np.array_equal(proj, ref["proj"])
    assert st.evals_total == ref["stats"]["evals_total"]


@pytest.mark.parametrize("count", [3, 70])  # two seeds per locality key; one above 64 sub-indexes
def test_relocated_batched_equals_alone(pg, count):
    d, total = 512, 16_600
    rng = np.random.default_rng(count)
    cuts = np.sort(rng.choice(np.arange(150, total - 150, 150), count - 1, replace=False))
    off = np.concatenate([[0], cuts, [total]])
    parts = [_data(int(b - a), d, int(b - a), seed=900 + i) for i, (a, b) in
             enumerate(zip(off[:-1], off[1:]))]
    assert total * d * 4 >= 32 << 20
    base = np.concatenate([p[0] for p in parts])
    gt = np.concatenate([p[1] for p in parts])
    graph = torch.full((total, 32), -1, dtype=torch.int32, device="cuda")
    proj = torch.full((total, 16), -1, dtype=torch.int32, device="cuda")
    b_dev, g_dev = _dev(base), _dev(gt)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with pg.Handle(0, stream=stream) as h:
        for flags in (0, pg.FLAG_CUDA_GRAPH, pg.FLAG_CUDA_GRAPH):  # eager, capture, replay
            graph.fill_(-1)
            proj.fill_(-1)
            torch.cuda.synchronize()
            st = h.build_batched(b_dev, g_dev, off, off, graph, proj,
                                 pg.default_params(32, 64, screen=3, flags=flags))
            g_all = graph.cpu().numpy().view(np.uint32)
            p_all = proj.cpu().numpy().view(np.uint32)
            evals = 0
            for i, (b, g) in enumerate(parts):
                ga, pa, sa = _build(pg, b, g, pg.default_params(32, 64, screen=3))
                evals += sa.evals_total
                assert np.array_equal(g_all[off[i]:off[i + 1]], ga), i
                assert np.array_equal(p_all[off[i]:off[i + 1]], pa), i
            assert st.evals_total == evals
