"""The hierarchical family's register engine against the tick engine, bit for bit, at the sizes where
its lane layout changes: a lane's element count, full and nearly empty last elements, and the first
dimension beyond its range.  Small steps, so that trees grow past 32 leaves."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from numpyro_gb300 import NUTS, models  # noqa: E402

FIELDS = ("z", "z_grad", "potential_energy", "energy", "num_steps", "accept_prob", "diverging")


def _run(model, engine, chains, warmup, draws, **more):
    k = NUTS(model, engine=engine, num_chains=chains, **more)
    st = k.init(11, warmup)
    out = k.run_device(st, warmup + draws, collect=("z", "num_steps"))
    got = {f: getattr(st, f).cpu().numpy() for f in FIELDS}
    got.update({"draw_" + f: v.cpu().numpy() for f, v in out.items()})
    got["step_size"] = st.adapt_state.step_size.cpu().numpy()
    got["inverse_mass_matrix"] = st.adapt_state.inverse_mass_matrix.cpu().numpy()
    k.close()
    return got


def _model(sizes):
    rng = np.random.default_rng(sum(sizes))
    return models.HierarchicalNormal(datasets=[(3.0 * rng.standard_normal(J), rng.uniform(1.0, 9.0, J)) for J in sizes])


@pytest.mark.gpu
@pytest.mark.parametrize("J", [1, 2, 29, 30, 31, 62, 63, 94, 95, 158, 159, 222, 223, 286, 287])
def test_register_engine_is_the_tick_engine(J):
    model = _model([J])
    args = dict(chains=6, warmup=0, draws=4, step_size=0.02, adapt_step_size=False, adapt_mass_matrix=False,
                max_tree_depth=7)
    a, b = _run(model, "fused", **args), _run(model, "ticks", **args)
    assert a["draw_num_steps"].max() > 64  # past the first block of 32 leaves at depth 6
    for f in a:
        np.testing.assert_array_equal(a[f], b[f], err_msg=f)


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [[4, 200, 33, 1, 90], [30] * 200])
def test_register_engine_warmup_is_the_tick_engine(sizes):
    """Window ends with their step-size searches, uneven models; more chains than SMs."""
    model = _model(sizes)
    args = dict(chains=3 * len(sizes), warmup=30, draws=2, find_heuristic_step_size=True)
    a, b = _run(model, "fused", **args), _run(model, "ticks", **args)
    for f in a:
        np.testing.assert_array_equal(a[f], b[f], err_msg=f)


@pytest.mark.gpu
@pytest.mark.parametrize("J,chains", [(1, 3), (8, 5), (30, 5), (31, 200), (62, 4), (63, 4), (94, 310), (95, 3)])
def test_register_engine_dense_mass_is_the_tick_engine(J, chains):
    """Dense mass matrices through a window end (their factors change), one to three elements a lane."""
    args = dict(chains=chains, warmup=24, draws=3, dense_mass=True, max_tree_depth=6)
    a, b = _run(_model([J]), "fused", **args), _run(_model([J]), "ticks", **args)
    assert a["draw_num_steps"].max() > 3
    for f in a:
        np.testing.assert_array_equal(a[f], b[f], err_msg=f)
