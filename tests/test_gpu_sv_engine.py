"""The stochastic-volatility family's on-chip engine against the tick engine, bit for bit, at the walk
lengths where its layout changes: elements per thread, log nu and log s in one warp or two, in the
last element row or a row of their own, and the first lengths beyond its range.  Small steps, so that
trees grow past 32 leaves."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from numpyro_gb300 import NUTS, datasets, models  # noqa: E402

FIELDS = ("z", "z_grad", "potential_energy", "energy", "num_steps", "accept_prob", "diverging")


def _run(T, noncentered, engine, chains, warmup, draws, init_step, **more):
    r, h = datasets.sv_returns(seed=T, T=T)
    k = NUTS(models.StochasticVolatility(r, noncentered=noncentered), engine=engine, num_chains=chains,
             step_size=init_step, **more)
    rng = np.random.default_rng(T)
    z = np.empty((chains, T + 2))
    z[:, :T] = 0.3 * rng.standard_normal((chains, T)) + (0.0 if noncentered else h)
    z[:, T:] = [np.log(8.0), np.log(0.3)]
    st = k.init(11, warmup, z)
    out = k.run_device(st, warmup + draws, collect=("z", "num_steps"))
    got = {f: getattr(st, f).cpu().numpy() for f in FIELDS}
    got.update({"draw_" + f: v.cpu().numpy() for f, v in out.items()})
    got["step_size"] = st.adapt_state.step_size.cpu().numpy()
    got["inverse_mass_matrix"] = st.adapt_state.inverse_mass_matrix.cpu().numpy()
    k.close()
    return got


@pytest.mark.gpu
@pytest.mark.parametrize("noncentered", [False, True])
@pytest.mark.parametrize("T", [2, 3, 31, 253, 254, 255, 287, 510, 511, 1000, 1279, 2303, 4095, 4096, 4097, 4350, 4351])
def test_on_chip_engine_is_the_tick_engine(T, noncentered):
    step = 0.05 / T ** 0.5 if noncentered else 0.004
    args = dict(chains=3, warmup=0, draws=3, init_step=step, adapt_step_size=False, adapt_mass_matrix=False,
                max_tree_depth=6)
    a, b = _run(T, noncentered, "fused", **args), _run(T, noncentered, "ticks", **args)
    assert a["draw_num_steps"].max() > 40  # past the first block of 32 leaves at depth 5
    for f in a:
        np.testing.assert_array_equal(a[f], b[f], err_msg=f)


@pytest.mark.gpu
@pytest.mark.parametrize("searches", [False, True])
@pytest.mark.parametrize("noncentered", [False, True])
def test_on_chip_engine_warmup_is_the_tick_engine(noncentered, searches):
    """Adaptation with turns, divergences and early stops; more chains than SMs."""
    args = dict(chains=170, warmup=25, draws=2, init_step=0.1, find_heuristic_step_size=searches, max_tree_depth=6)
    a, b = _run(100, noncentered, "fused", **args), _run(100, noncentered, "ticks", **args)
    assert a["draw_num_steps"].max() > 8
    for f in a:
        np.testing.assert_array_equal(a[f], b[f], err_msg=f)
