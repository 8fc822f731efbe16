"""The autotuner searches from the library's own defaults: what it does not try keeps them."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_untried_stages_keep_the_default():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import paragraph_gb300 as pg
    n = 2000
    rng = np.random.default_rng(8)
    base = torch.from_numpy(rng.standard_normal((n, 32)).astype(np.float32)).cuda()
    gt = torch.from_numpy(rng.integers(0, n, (n, 128)).astype(np.int32)).cuda()
    with pg.Handle(0) as h:
        # a plain build has no screened prune: its ring depth is not tried
        _, t = h.autotune(base, gt, pg.default_params(32, 64))
    assert t.screen_stages in (0, 3)
