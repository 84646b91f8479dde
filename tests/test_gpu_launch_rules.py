"""Launch shapes that set the order of FP32 sums follow the sizes alone: the same bits with the autotuner and
without it.  Sizes on both sides of each line of the rules, up to 1,024 chains."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from numpyro_gb300 import NUTS, models  # noqa: E402


def _both(model, z, monkeypatch):
    out = []
    for autotune in ("0", "1"):
        monkeypatch.setenv("GBN_AUTOTUNE", autotune)
        k = NUTS(model, num_chains=z.shape[0])
        out.append([t.cpu().numpy() for t in k.potential_and_grad(torch.as_tensor(z, device="cuda"))])
        k.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("n,p,C", [(8192, 13, 128), (8193, 55, 64), (10011, 55, 1024), (20011, 13, 4), (20011, 32, 12),
                                   (25000, 13, 64), (60000, 5, 300), (300000, 13, 1024)])
def test_logreg_row_groups(n, p, C, monkeypatch):
    rng = np.random.default_rng(n + C)
    X = rng.standard_normal((n, p)).astype(np.float32)
    y = (rng.random(n) < 0.4).astype(np.float32)
    _both(models.LogisticRegression(X, y), (0.1 * rng.standard_normal((C, p))).astype(np.float32), monkeypatch)
