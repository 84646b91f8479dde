"""Launch shapes that set the order of FP32 sums follow the sizes alone: the same bits with the autotuner and
without it.  Sizes on both sides of each line of the rules, up to 1,024 chains."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from numpyro_gb300 import NUTS, datasets, models  # noqa: E402


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


@pytest.mark.gpu
@pytest.mark.parametrize("n,p,C", [(64, 20, 3), (65, 50, 3), (200, 30, 128), (201, 96, 2), (1000, 1000, 127), (1000, 1000, 128)])
def test_horseshoe_tiles(n, p, C, monkeypatch):
    X, y, _ = datasets.horseshoe_data(seed=n, n=n, p=p, nonzero=5)
    z = (0.1 * np.random.default_rng(C).standard_normal((C, 2 * p + 2))).astype(np.float32)
    _both(models.HorseshoeRegression(X, y), z, monkeypatch)


def _logreg(n, p, seed):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, p)).astype(np.float32)
    return X, (rng.random(n) < 0.4).astype(np.float32), rng


@pytest.mark.gpu
@pytest.mark.parametrize("n,p,C", [(64, 3, 1025), (200, 5, 3000), (1000, 33, 2049), (8192, 13, 1100), (8193, 4, 5000)])
def test_many_points_vs_fp64(n, p, C):
    """Several tiles a row group and a warp a point for the sums.  Bounds as in test_gpu_logreg_fp32, with chains of n rows
    for the gradient; every point."""
    X, y, rng = _logreg(n, p, n + C)
    z = (0.3 * rng.standard_normal((C, p))).astype(np.float32)
    k = NUTS(models.LogisticRegression(X, y), num_chains=C)
    pe, g = k.potential_and_grad(torch.as_tensor(z, device="cuda"))
    k.close()
    U = 2.0 ** -24
    X, y, z = (torch.as_tensor(v, device="cuda", dtype=torch.float64) for v in (X, y, z))
    l, el = z @ X.T, p * U * (z.abs() @ X.abs().T)
    soft, e = torch.nn.functional.softplus(l), torch.sigmoid(l) - y
    ref = (soft - y * l).sum(1) + 0.5 * (z * z).sum(1) + 0.5 * p * np.log(2.0 * np.pi)
    assert bool(((pe - ref).abs() <= (el + 8 * U * (soft + l.abs())).sum(1) + 1e-9 * ref.abs()).all())
    bound = (0.25 * el + 4 * U + (n + 2) * U * e.abs()) @ X.abs() + 4 * U * z.abs()
    assert bool(((g - (e @ X + z)).abs() <= bound).all())


@pytest.mark.gpu
@pytest.mark.parametrize("n", [65, 200, 1100, 8192])
def test_small_data_sets_have_one_gradient(n):
    """Up to 8,192 rows and 1,024 points a point's gradient does not depend on how many there are."""
    X, y, rng = _logreg(n, 13, n)
    z = torch.as_tensor((0.3 * rng.standard_normal((1024, 13))).astype(np.float32), device="cuda")
    k = NUTS(models.LogisticRegression(X, y), num_chains=1024)
    g = k.potential_and_grad(z)[1]
    for C in (1, 9, 65, 511, 600):
        assert torch.equal(k.potential_and_grad(z[:C].contiguous())[1], g[:C]), C
    k.close()


@pytest.mark.gpu
def test_many_chains_need_little_memory():
    """Partial gradients of 65,536 chains: 128 row groups would take 2.2 GB."""
    X, y, _ = _logreg(8192, 5, 0)
    k = NUTS(models.LogisticRegression(X, y), num_chains=65536)
    z = torch.zeros(65536, 5, device="cuda")
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    k.potential_and_grad(z)
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] < 5e8
    k.close()
