"""Calls with few queries over long rows: on both sides of the row length and of the query count from
which later rows are sent to L2 ahead, rows starting inside a 128-byte line.  Ids and counts equal the
oracle's."""
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


@pytest.mark.parametrize("d", [320, 324, 484, 512])
@pytest.mark.parametrize("km", [32, 96])
def test_few_queries_equal_oracle(pg, d, km):
    n = 3000
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(d + km)
    base = rng.standard_normal((n, d)).astype(np.float32)
    graph = rng.integers(0, n, (n, 16)).astype(np.uint32)
    queries = rng.standard_normal((2 * sms + 1, d)).astype(np.float32)
    want, _, _ = oracle.query_search(base, graph, queries, topk=10, km=km, reset_iter=4)
    flat = torch.zeros(n * d + 4, dtype=torch.float32, device="cuda")
    b = flat[4:].view(n, d)
    b.copy_(torch.from_numpy(base))
    g, q = torch.from_numpy(graph.view(np.int32)).cuda(), torch.from_numpy(queries).cuda()
    with pg.Handle(0) as h:
        for nq in (1, 2 * sms, 2 * sms + 1):
            out = torch.full((nq, 10), -1, dtype=torch.int32, device="cuda")
            _, ev, it = oracle.query_search(base, graph, queries[:nq], topk=10, km=km, reset_iter=4)
            got = h.query_search(b, g, q[:nq].contiguous(), out, km=km, reset_iter=4)
            assert np.array_equal(out.cpu().numpy().view(np.uint32), want[:nq])
            assert tuple(got) == (ev, it)
