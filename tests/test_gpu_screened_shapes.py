"""Screened builds at the edges of the tensor-core prune's tiles: row lengths around the 16- and
64-column steps, one and two nodes per tile, an odd node count, both operand types; lists full of
near-ties, equal rows and rows of one direction (every test inside the 16-bit margin).  Graph,
projection and evaluation counts equal the oracle's."""
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


@pytest.mark.parametrize("d", [4, 60, 64, 68, 144, 260, 512])
@pytest.mark.parametrize("beam,degree,screen", [(64, 32, 3), (64, 3, 1), (96, 48, 3), (128, 16, 1)])
def test_screened_build_equals_oracle(pg, d, beam, degree, screen):
    n, q = 615, 500
    rng = np.random.default_rng(d * 1000 + beam)
    base = rng.standard_normal((n, d)).astype(np.float32)
    base[100:140] = base[60:100]
    base[200:300] = base[200] * rng.uniform(0.999, 1.001, (100, 1)).astype(np.float32)
    base[300:420] = base[300] + 1e-4 * rng.standard_normal((120, d)).astype(np.float32)
    queries = (base[rng.integers(0, n, q)] + 0.3 * rng.standard_normal((q, d))).astype(np.float32)
    gt = np.argsort(-(queries @ base.T), axis=1, kind="stable")[:, :128].astype(np.uint32)
    over = {} if degree >= 16 else {"kp": 32, "kd": 1, "km": beam - 32}  # kd <= degree
    params = pg.default_params(degree, beam, screen=screen, **over)
    ref = oracle.build_graph(base, gt, degree=degree, beam=beam, **over)
    graph = torch.full((n, degree), -1, dtype=torch.int32, device="cuda")
    proj = torch.full((n, 16), -1, dtype=torch.int32, device="cuda")
    with pg.Handle(0) as h:
        st = h.build_device(torch.from_numpy(base).cuda(),
                            torch.from_numpy(gt.view(np.int32)).cuda(), graph, proj, params)
    assert np.array_equal(graph.cpu().numpy().view(np.uint32), ref["graph"])
    assert np.array_equal(proj.cpu().numpy().view(np.uint32), ref["proj"])
    assert st.evals_total == ref["stats"]["evals_total"]
