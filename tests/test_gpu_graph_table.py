"""A captured batched build copies its sub-index table from pinned memory that the handle owns.  A
build with a longer table moves that memory, so the captured build must not be replayed after it."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pg():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import paragraph_gb300
    paragraph_gb300.lib()
    return paragraph_gb300


def test_longer_table_between_replays(pg):
    d, total = 64, 7000
    rng = np.random.default_rng(17)
    base = torch.from_numpy(rng.standard_normal((total, d)).astype(np.float32)).cuda()
    gt = torch.from_numpy(rng.integers(0, 100, (total, 128)).astype(np.int32)).cuda()
    few = np.array([0, 3000, 3500, total])
    many = np.arange(0, total + 1, 100)
    graph, eager, small = torch.full((3, total, 32), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    plain = pg.default_params(32, 64)
    captured = pg.default_params(32, 64, flags=pg.FLAG_CUDA_GRAPH)
    with pg.Handle(0, stream=stream) as h:
        # wider lists first: the workspace then holds either table's build, only the table grows
        wide = torch.full((total, 48), -1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        h.build_batched(base, gt, few, few, wide, None, pg.default_params(48, 96))
        h.build_batched(base, gt, few, few, eager, None, plain)
        want = h.build_batched(base, gt, few, few, graph, None, captured).evals_total
        assert torch.equal(graph, eager)
        for _ in range(2):
            h.build_batched(base, gt, many, many, small, None, plain)
            graph.fill_(-1)
            torch.cuda.synchronize()
            assert h.build_batched(base, gt, few, few, graph, None, captured).evals_total == want
            assert torch.equal(graph, eager)
