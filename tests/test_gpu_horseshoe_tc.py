"""The tensor-core horseshoe GEMMs at the edges of their tiles (128 chains, 64 rows or features, K blocks of
64: fewer K blocks than the two operand buffers, than the copy stages, and more; split-K ranges that are
empty, one block and several) against the FP64 closed form.

Bounds (u = 2^-24): an operand is the sum of three bf16 terms to u of it and the dropped products of terms are
below u of a product: 4 u a product.  A tensor core step adds 16 products to an FP32 sum with none of its 17
operands rounded to nearest: 34 u of what is summed.  The leading products take 4 steps before they are drained
into FP32 sums (K / 64 of them, u each); the corrections, 5 x 2^-8 of the products, take K / 16 steps.  So a
contraction over K is off by (140 + K / 64 + 0.042 K) u sum|a b|.  R passes its error on to sum R^2 and X^T R;
what is computed in FP32 outside the contractions is off by at most 32 u of the magnitudes that it adds, the sums
over the features by one u more for each.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from numpyro_gb300 import NUTS, models  # noqa: E402
from oracle import potentials_ref as PR  # noqa: E402

U = 2.0 ** -24
CASES = [(1, 1, 1), (63, 64, 127), (64, 65, 128), (65, 63, 129), (200, 130, 3), (257, 400, 40), (900, 449, 130),
         (9800, 20, 10)]


@pytest.mark.gpu
@pytest.mark.parametrize("noncentered", [False, True])
@pytest.mark.parametrize("n,p,C", CASES)
def test_horseshoe_tc_gemms_vs_oracle(n, p, C, noncentered):
    rng = np.random.default_rng(n + 5 * p + C)
    X = rng.standard_normal((n, p)).astype(np.float32)
    y = rng.standard_normal(n).astype(np.float32)
    model = models.HorseshoeRegression(X, y, noncentered=noncentered)
    z = (0.3 * rng.standard_normal((C, 2 * p + 2))).astype(np.float32)
    k = NUTS(model, num_chains=C, precision="bf16x3")
    pe, g = [t.cpu().numpy() for t in k.potential_and_grad(torch.as_tensor(z, device="cuda"))]
    again = [t.cpu().numpy() for t in k.potential_and_grad(torch.as_tensor(z, device="cuda"))]
    k.close()
    np.testing.assert_array_equal(pe, again[0])
    np.testing.assert_array_equal(g, again[1])
    X64, y64 = X.astype(np.float64), y.astype(np.float64)
    ref = PR.make_potential("horseshoe_nc" if noncentered else "horseshoe", X64, y64)

    def contraction(K):
        return (140 + K / 64 + 0.042 * K) * U

    for c in sorted({0, C // 2, C - 1}):
        zc = z[c].astype(np.float64)
        pr, gr = ref(zc)
        if noncentered:
            llam, lsig, ltau, eta = zc[:p], zc[p], zc[p + 1], zc[p + 2:]
            scale = np.exp(ltau + llam)
            beta = scale * eta
        else:
            beta, llam, lsig, ltau = zc[:p], zc[p:2 * p], zc[2 * p], zc[2 * p + 1]
            scale = np.exp(ltau + llam)
        prec, absx, r = np.exp(-2 * lsig), np.abs(X64), y64 - X64 @ beta
        e_r = (contraction(p) + 8 * U) * (absx @ np.abs(beta)) + 2 * U * (np.abs(r) + np.abs(y64))
        rr = np.sum(r * r)
        e_rr = np.sum(2 * np.abs(r) * e_r + e_r * e_r) + 32 * U * rr
        xr = absx.T @ np.abs(r)
        e_gx = prec * (absx.T @ e_r + (contraction(n) + 32 * U) * xr)  # error of X^T R / sigma^2
        e_sig = prec * e_rr + 32 * U * (prec * rr + np.exp(2 * lsig) + 1 + n)
        e_tau_prior = (32 + p) * U * 3
        if noncentered:
            gx = np.abs(X64.T @ r) * prec
            bg = np.abs(beta) * (gx + e_gx)
            e_lam = np.abs(beta) * e_gx + 32 * U * (bg + 2)
            e_tau = np.sum(np.abs(beta) * e_gx) + (32 + p) * U * np.sum(bg) + e_tau_prior
            e_eta = scale * e_gx + 32 * U * (scale * gx + np.abs(eta))
            bound = np.concatenate([e_lam, [e_sig, e_tau], e_eta])
            q = eta ** 2
        else:
            q = (beta / scale) ** 2
            e_beta = e_gx + 32 * U * np.abs(beta) / scale ** 2
            e_tau = (32 + p) * U * np.sum(q + 1) + e_tau_prior
            bound = np.concatenate([e_beta, 32 * U * (q + 3), [e_sig, e_tau]])
        e_pe = 0.5 * prec * e_rr + 32 * U * (prec * rr + np.sum(q + 3 * np.abs(llam) + 3) + n * (1 + abs(lsig)) + 10)
        assert abs(pe[c] - pr) <= e_pe, (c, pe[c], pr, e_pe)
        assert np.all(np.abs(g[c] - gr) <= bound), (c, np.max(np.abs(g[c] - gr) / bound))
