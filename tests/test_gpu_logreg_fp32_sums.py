"""The FP32 logistic potential adds its four-row sums in FP64, in every instance of the kernel.

A model of four equal rows gives one such sum for each point, and a model whose rows are those points gives their
total: l is the same product both times.  All rows in one row group (GBN_TUNE), so a thread adds a sum of each
tile of 64 rows.  Bound, in units u = 2^-53 of the total: the m = n / 64 additions of a thread round independently by at
most u of a sum that grows to a sixteenth of the total, a standard deviation of sqrt(m) u / 3 for a thread and
sqrt(m) u / 12 for sixteen of them; eight of these and 4 u for the few additions across lanes, warps and prior are less
than (sqrt(m) + 4) u.  Taking the prior off in FP64 adds two roundings of each four-row sum's potential, again independent.
"""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from numpyro_gb300 import NUTS, models  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("n,C", [(8192, 1), (8192, 16), (8192, 128), (19520, 128)])
def test_four_row_sums_are_added_in_fp64(n, C, monkeypatch):
    monkeypatch.setenv("GBN_TUNE", "lr_rg=1")
    l = np.random.default_rng(n + C).uniform(-12.0, 6.0, n // 4).astype(np.float32)
    zero = np.zeros(n, np.float32)
    k = NUTS(models.LogisticRegression(np.ones((4, 1), np.float32), zero[:4]), num_chains=n // 4)
    pe = k.potential_and_grad(torch.as_tensor(l[:, None], device="cuda"))[0].cpu().numpy()
    k.close()
    const = 0.5 * math.log(2.0 * math.pi)
    prior = 0.5 * l.astype(np.float64) ** 2 + const
    total = math.fsum(pe - prior) + 0.5 + const
    off = 8 * math.sqrt(2 * math.fsum((np.abs(pe) + prior) ** 2)) * 2.0 ** -53
    k = NUTS(models.LogisticRegression(np.repeat(l, 4)[:, None], zero), num_chains=C)
    got = k.potential_and_grad(torch.ones(C, 1, device="cuda"))[0].cpu().numpy()
    assert k.tuning() == "logreg_row_groups=1"
    k.close()
    bound = (math.sqrt(n / 64) + 4) * 2.0 ** -53 * total + off
    assert np.all(np.abs(got - total) <= bound), (got[0] - total, bound)
