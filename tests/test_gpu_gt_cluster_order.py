"""Ground truth of a base stored cluster by cluster.  The sampled threshold of a query whose cluster
misses the sample lets through more rows than its list holds, and such queries are filtered again, next
to queries of the same tile that are not.  Ids equal the FP64 oracle's."""
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


# part: the share of queries near a cluster; the others see no order.  0.01: a few tiles are filtered
# again, and tiles without any such query are passed over
@pytest.mark.parametrize("part", [1.0, 0.3, 0.01])
@pytest.mark.parametrize("n,nq,d,k,clusters", [(140_001, 700, 16, 10, 450), (270_000, 300, 32, 10, 900),
                                               (140_001, 129, 16, 64, 130)])
def test_cluster_order_equals_oracle(pg, part, n, nq, d, k, clusters):
    rng = np.random.default_rng(n + nq + k)
    centers = rng.standard_normal((clusters, d))
    label = np.sort(rng.integers(0, clusters, n))
    base = (centers[label] + 0.2 * rng.standard_normal((n, d))).astype(np.float32)
    queries = rng.standard_normal((nq, d))
    near = rng.random(nq) < part
    queries[near] = 3 * centers[rng.integers(0, clusters, near.sum())]
    queries = (queries + 0.1 * rng.standard_normal((nq, d))).astype(np.float32)
    out = torch.full((nq, k), -1, dtype=torch.int32, device="cuda")
    with pg.Handle(0) as h:
        h.ground_truth(torch.from_numpy(base).cuda(), torch.from_numpy(queries).cuda(), out)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), oracle.ground_truth(base, queries, k))
