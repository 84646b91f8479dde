"""The stochastic-volatility potential at the walk lengths where its kernels' instances and rows change (steps a
thread, partly filled last steps, the first length past the register instances) against the FP64 closed form.

Bounds (u = 2^-24): the walk and every sum are compensated, so what is left are a few FP32 operations an element,
32 u of the magnitudes that they add; y^2 = r^2 e^(-2 h) is off by a few u (1 + |h|) of itself, which the terms in it pass
on with a factor of at most nu + 2.
"""
import numpy as np
import pytest
from scipy.special import digamma

torch = pytest.importorskip("torch")

from gpu_helpers import typical_points  # noqa: E402
from numpyro_gb300 import NUTS, datasets, models  # noqa: E402
from oracle import potentials_ref as PR  # noqa: E402

U = 2.0 ** -24


@pytest.mark.gpu
@pytest.mark.parametrize("noncentered", [False, True])
@pytest.mark.parametrize("T", [2, 31, 255, 256, 257, 513, 1023, 1025, 1537, 2305, 3073, 4096, 4097])
def test_sv_potential_vs_oracle(T, noncentered):
    name = "sv_nc" if noncentered else "sv"
    r, _ = datasets.sv_returns(seed=T, T=T)
    model = models.StochasticVolatility(r, noncentered=noncentered)
    z = typical_points(name, model, np.random.default_rng(T), 5)
    k = NUTS(model, num_chains=5)
    pe, g = [t.cpu().numpy() for t in k.potential_and_grad(torch.as_tensor(z, device="cuda"))]
    k.close()
    r64 = np.asarray(r, np.float32).astype(np.float64)
    ref = PR.make_potential(name, r64)
    for c in (0, 4):
        zc = z[c].astype(np.float64)
        pr, gr = ref(zc)
        nu, s, w = np.exp(zc[T]), np.exp(zc[T + 1]), zc[:T]
        S = np.cumsum(w)
        h = s * S if noncentered else w
        b = (nu + 2) * (1 + np.abs(h))
        y2 = (r64 * np.exp(-h)) ** 2
        d = np.diff(w, prepend=0.0)
        walk = np.sum(w * w) if noncentered else np.sum(d * d) / s ** 2
        l1p, frac = np.sum(np.log1p(y2 / nu)), np.sum(y2 / (nu + y2))
        assert abs(pe[c] - pr) <= 32 * U * (walk + (nu + 1) * l1p + np.sum(b) + 10), (c, pe[c], pr)
        if noncentered:
            head = np.abs(w) + s * np.cumsum(b[::-1])[::-1]
            tail = s * np.sum(b * np.abs(S)) + 10 * s + 1
        else:
            head = (np.abs(d) + np.abs(np.append(d[1:], 0.0))) / s ** 2 + b
            tail = walk + T + 10 * s + 1
        scale = nu * (l1p + (nu + 1) / nu * (frac + 1e-3 * T) + T / nu + T * (abs(digamma(nu / 2)) + abs(digamma(nu / 2 + 0.5)))
                      + 1) + np.sum(b) + 1
        bound = 32 * U * np.concatenate([head, [scale, tail]])
        assert np.all(np.abs(g[c] - gr) <= bound), (c, np.max(np.abs(g[c] - gr) / bound), np.argmax(np.abs(g[c] - gr) / bound))
