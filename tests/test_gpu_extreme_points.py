"""Chains at the ends of the FP32 range: overflowing scales, infinities, NaN.  The register engines decide as the
tick engine does, bit for bit, and in the FP32 logistic kernel, where chains share threads and tiles, a bad point stays
in its own row."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from numpyro_gb300 import HMC, NUTS, datasets, models  # noqa: E402

NAN, INF = float("nan"), float("inf")


def _run(model, engine, z, **more):
    k = NUTS(model, num_chains=z.shape[0], step_size=0.05, engine=engine, max_tree_depth=6, **more)
    st = k.init(1, 5, z)
    draws = k.run_device(st, 8, collect=("z",))["z"]
    out = [t.cpu().numpy() for t in (st.z, st.z_grad, st.potential_energy, st.energy, st.accept_prob, st.num_steps,
                                     st.diverging, st.adapt_state.step_size, draws)]
    k.close()
    return out


def _same(model, z, **more):
    for a, b in zip(_run(model, "fused", z, **more), _run(model, "ticks", z, **more)):
        np.testing.assert_array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("groups,dense", [(8, False), (8, True), (40, False), (40, True)])
def test_hierarchical(groups, dense):
    rng = np.random.default_rng(groups)
    z = 0.5 * rng.standard_normal((13, groups + 2))
    z[1] *= 1e19
    z[2:8, 1] = [-200, -90, 45, 88.5, 100, NAN]  # log tau
    z[8, 0], z[9, 0], z[10, 5], z[11, 3], z[12, 2:] = INF, -1e25, 1e30, NAN, 1e18
    model = models.HierarchicalNormal((5 * rng.standard_normal(groups)).astype(np.float32),
                                      (1 + 4 * rng.random(groups)).astype(np.float32))
    _same(model, z.astype(np.float32), dense_mass=dense)


@pytest.mark.gpu
@pytest.mark.parametrize("noncentered", [False, True])
@pytest.mark.parametrize("T", [5, 300])
def test_stochastic_volatility(T, noncentered):
    r, h = datasets.sv_returns(seed=1, T=T)
    r = np.array(r)
    r[1] = 0.0
    z = np.empty((19, T + 2))
    z[:, :T] = 0.3 * np.random.default_rng(T).standard_normal((19, T)) + (0.0 if noncentered else h)
    z[:, T:] = [2.0, np.log(0.05)]
    z[1:9, T] = [100, 85, -88, -89, -95, -100, NAN, INF]  # log nu: from overflow to no FP32 reciprocal and to zero
    z[9:14, T + 1] = [100, 43, -50, -100, NAN]  # log s
    z[14, 3], z[15, 3], z[16, 0], z[17, T - 1], z[18, :T] = 1e4, -1e4, NAN, INF, 1e20
    _same(models.StochasticVolatility(r, noncentered=noncentered), z.astype(np.float32))


@pytest.mark.gpu
@pytest.mark.parametrize("n,C", [(65, 8), (300, 16), (300, 130), (12000, 64), (20000, 130)])
def test_logreg_fp32_rows_are_apart(n, C):
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, 13)).astype(np.float32)
    y = (rng.random(n) < 0.4).astype(np.float32)
    z = torch.as_tensor((0.1 * rng.standard_normal((C, 13))).astype(np.float32), device="cuda")
    k = NUTS(models.LogisticRegression(X, y), num_chains=C)
    pe, g = k.potential_and_grad(z)
    bad = z.clone()
    bad[1, 0], bad[2, 3], bad[4, 12], bad[6] = NAN, INF, -INF, 1e30
    pe2, g2 = k.potential_and_grad(bad)
    k.close()
    good = [c for c in range(C) if c not in (1, 2, 4, 6)]
    assert torch.equal(pe[good], pe2[good]) and torch.equal(g[good], g2[good])
    assert bool(pe2[1].isnan()) and bool(g2[1].isnan().all())
    for c, d in ((2, 3), (4, 12)):  # sigmoids of 0 and 1, an infinite prior term
        assert not bool(pe2[c].isfinite()) and bool(g2[c, d].isinf())
        assert bool(g2[c, [j for j in range(13) if j != d]].isfinite().all())
    assert float(pe2[6]) > 1e30 and bool(g2[6].isfinite().all())


@pytest.mark.gpu
@pytest.mark.parametrize("T", [4820, 4826, 4832])
def test_walks_at_the_end_of_shared_memory(T):
    """Twelve rows of such a walk and the kernel's static shared memory are just too much for a block: the state machine
    takes its rows from global memory."""
    r, h = datasets.sv_returns(seed=1, T=T)
    z = np.concatenate([h, [2.0, -3.0]])[None].repeat(2, 0).astype(np.float32)
    out = []
    for engine in ("fused", "ticks"):
        k = HMC(models.StochasticVolatility(r), num_chains=2, num_steps=3, trajectory_length=None, step_size=1e-3,
                engine=engine, adapt_step_size=False, adapt_mass_matrix=False)
        out.append(k.sample(k.init(0, 0, z)).z.cpu().numpy())
        k.close()
    np.testing.assert_array_equal(*out)
