"""The FP32 logistic potential at the edges of its tiles (64 rows; 8, 16, 64 and 128 chains; 32 and 64
feature words; rows of whole 16-byte words or not; one row group a tile or several tiles a group)
against the FP64 closed form.

Bounds: every FP32 operation rounds by at most u = 2^-24 of its result.  A logit is a chain of p fused
multiply-adds, so it is off by at most p u sum|x b|; softplus and sigmoid add a few u of their value (4 here)
and pass the logit's error on with slope at most 1 and 1/4.  A gradient entry is a chain of additions over
the rows of a group and over the groups; the potential's row sums are 4 rows long, then compensated.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from numpyro_gb300 import NUTS, models  # noqa: E402
from oracle import potentials_ref as PR  # noqa: E402

U = 2.0 ** -24
CASES = [(1, 1, 1), (3, 64, 8), (63, 3, 9), (64, 4, 16), (65, 31, 17), (200, 32, 1024), (130, 33, 129), (8192, 8, 3),
         (8193, 13, 4), (9999, 5, 16), (9800, 36, 64), (10011, 55, 65), (20000, 64, 128), (20001, 30, 200)]


@pytest.mark.gpu
@pytest.mark.parametrize("n,p,C", CASES)
def test_logreg_fp32_vs_oracle(n, p, C):
    rng = np.random.default_rng(n + 7 * p + C)
    X = rng.standard_normal((n, p)).astype(np.float32)
    y = (rng.random(n) < 0.4).astype(np.float32)
    z = (0.3 * rng.standard_normal((C, p))).astype(np.float32)
    k = NUTS(models.LogisticRegression(X, y), num_chains=C)
    pe, g = [t.cpu().numpy() for t in k.potential_and_grad(torch.as_tensor(z, device="cuda"))]
    again = [t.cpu().numpy() for t in k.potential_and_grad(torch.as_tensor(z, device="cuda"))]
    few, few_g = [t.cpu().numpy() for t in k.potential_and_grad(torch.as_tensor(z[:1], device="cuda"))]
    k.close()
    np.testing.assert_array_equal(pe, again[0])
    np.testing.assert_array_equal(g, again[1])
    X64, y64 = X.astype(np.float64), y.astype(np.float64)
    for c in sorted({0, C // 2, C - 1}):
        zc = z[c].astype(np.float64)
        el = p * U * (np.abs(X64) @ np.abs(zc))  # error of each logit
        sig = 1.0 / (1.0 + np.exp(-(X64 @ zc)))
        soft = np.logaddexp(0.0, X64 @ zc)
        ref, gref = PR.logreg_potential(zc, X64, y64), PR.logreg_grad(zc, X64, y64)
        bound = np.sum(el + 8 * U * (soft + np.abs(X64 @ zc))) + 1e-9 * abs(ref)
        chain = (n if n > 8192 else 64 + n // 64) + 2  # the longest chain of additions
        gbound = (np.abs(X64).T @ (0.25 * el + 4 * U * np.maximum(sig, 1.0)) + chain * U * (np.abs(X64).T @ np.abs(sig - y64))
                  + 4 * U * np.abs(zc))
        assert abs(pe[c] - ref) <= bound, (c, pe[c], ref, bound)
        assert np.all(np.abs(g[c] - gref) <= gbound), (c, np.max(np.abs(g[c] - gref) / gbound))
        if c == 0:  # another number of points: another launch shape
            assert abs(few[0] - ref) <= bound and np.all(np.abs(few_g[0] - gref) <= gbound)
