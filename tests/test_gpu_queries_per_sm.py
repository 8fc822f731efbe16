"""The beam search's kernels for different numbers of queries per SM: on both sides of each limit, ids
and counts equal the oracle's."""
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


@pytest.mark.parametrize("d", [4, 224, 256, 260, 512])
@pytest.mark.parametrize("km", [32, 64, 96])
def test_queries_per_sm_equal_oracle(pg, d, km):
    n = 3000
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(3 * d + km)
    base = rng.standard_normal((n, d)).astype(np.float32)
    base[n // 2:n // 2 + n // 8] = base[:n // 8]  # equal rows: ties decided by position
    graph = rng.integers(0, n, (n, 16)).astype(np.uint32)
    queries = rng.standard_normal((16 * sms + 1, d)).astype(np.float32)
    want, ev, it = oracle.query_search(base, graph, queries, topk=10, km=km, reset_iter=4)
    b, q = torch.from_numpy(base).cuda(), torch.from_numpy(queries).cuda()
    g = torch.from_numpy(graph.view(np.int32)).cuda()
    with pg.Handle(0) as h:
        for nq in (8 * sms, 8 * sms + 1, 12 * sms, 12 * sms + 1, 16 * sms, 16 * sms + 1):
            out = torch.full((nq, 10), -1, dtype=torch.int32, device="cuda")
            got = h.query_search(b, g, q[:nq].contiguous(), out, km=km, reset_iter=4)
            assert np.array_equal(out.cpu().numpy().view(np.uint32), want[:nq])
        assert tuple(got) == (ev, it)
