"""Ground-truth selection where its parts can go wrong: long candidate lists, runs of equal and of
nearly equal scores, one maximum far above the rest, odd group counts, rows off a 16-byte boundary,
a sample of the base that misses the nearest rows.
Ids equal the FP64 oracle's."""
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


def _base(kind, n, d, rng):
    base = rng.standard_normal((n, d)).astype(np.float32)
    if kind == "copies":  # every score shared by many rows: order by id inside long runs
        base = base[rng.integers(0, 9, n)]
    elif kind == "close":  # neighbours differ in the last bits of one coordinate
        base[1::2] = base[0:n - n % 2:2]
        base[1::2, 0] = np.nextafter(base[1::2, 0], np.float32(9))
    elif kind == "missed":  # the sampled tiles of a large base hold none of the nearest rows
        base[(np.arange(n) // 256) % 8 != 0] *= 2.0
    elif kind == "outlier":  # the other maxima fall into one step of the first division
        base[n // 3] *= 20.0
    return np.ascontiguousarray(base)


@pytest.mark.parametrize("kind", ["plain", "copies", "close", "outlier", "missed"])
@pytest.mark.parametrize("n,nq,d,k", [(701, 33, 36, 256), (5003, 129, 200, 100),
                                      (20_481, 9, 64, 128), (140_000, 3, 16, 10),
                                      (270_000, 5, 8, 128)])
@pytest.mark.parametrize("shift", [0, 1])
def test_selection_equals_oracle(pg, kind, n, nq, d, k, shift):
    if kind == "copies":
        n = min(n, 900)  # more equal scores than the selection holds are refused
    rng = np.random.default_rng(n + d)
    base = _base(kind, n, d, rng)
    queries = rng.standard_normal((nq, d)).astype(np.float32)
    flat = torch.zeros(n * d + 4, dtype=torch.float32, device="cuda")
    b = flat[shift:shift + n * d].view(n, d)
    b.copy_(torch.from_numpy(base))
    out = torch.full((nq, k), -1, dtype=torch.int32, device="cuda")
    with pg.Handle(0) as h:
        h.ground_truth(b, torch.from_numpy(queries).cuda(), out)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), oracle.ground_truth(base, queries, k))
