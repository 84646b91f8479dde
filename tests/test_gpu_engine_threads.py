"""Two kernels that share an instance of a persistent engine but need different amounts of shared memory,
run from two host threads at once: distinct handles are independent, so every call succeeds and each chain
ends where it ends when its kernel runs alone."""
import ctypes
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from numpyro_gb300 import HMC, NUTS, _lib, datasets, models  # noqa: E402

FIXED = dict(adapt_step_size=False, adapt_mass_matrix=False)


def _hier(groups, chains, **more):
    rng = np.random.default_rng(groups)
    model = models.HierarchicalNormal(rng.standard_normal(groups).astype(np.float32), np.ones(groups, np.float32))
    return NUTS(model, num_chains=chains, step_size=0.1, max_tree_depth=2, **FIXED, **more), groups + 2


def _sv(T, chains, hmc=False):
    model = models.StochasticVolatility(datasets.sv_returns(seed=1, T=T)[0])
    more = dict(num_chains=chains, step_size=0.004, **FIXED)
    return (HMC(model, num_steps=2, trajectory_length=None, **more) if hmc else NUTS(model, max_tree_depth=1, **more)), T + 2


# (the larger kernel, more chains than SMs; the smaller one): dynamic shared memory per CTA in KB
PAIRS = {
    "hier dense": (lambda: _hier(94, 200, dense_mass=True), lambda: _hier(64, 2, dense_mass=True)),  # 80, 27
    "sv on chip": (lambda: _sv(4090, 160), lambda: _sv(3400, 2)),  # 87, 72
    "sv state machine": (lambda: _sv(4000, 2, hmc=True), lambda: _sv(1100, 2, hmc=True)),  # 188, 52
}


def _transitions(kernel, state, more):
    """gbn_sample on this thread's own stream and a copy of the state while more(calls made); (z, calls, errors)."""
    lib, state = _lib.load(), kernel.copy_state(state)
    fields, stream = kernel._cstate(state), torch.cuda.Stream()
    stream.wait_stream(torch.cuda.default_stream())
    calls, errors = 0, []
    while more(calls):
        if lib.gbn_sample(kernel._handle, ctypes.c_void_p(stream.cuda_stream), ctypes.byref(fields)) != 0:
            errors.append(lib.gbn_last_error(kernel._handle))
        calls += 1
    stream.synchronize()
    return state.z.cpu().numpy(), calls, errors


@pytest.mark.gpu
@pytest.mark.parametrize("pair", PAIRS)
def test_two_threads_two_sizes(pair):
    kernels, starts, got, done = [], [], [None, None], threading.Event()
    for make in PAIRS[pair]:
        kernel, dim = make()
        rng = np.random.default_rng(dim)
        kernels.append(kernel)
        starts.append(kernel.init(5, 0, (0.1 * rng.standard_normal((kernel._num_chains, dim))).astype(np.float32)))
    torch.cuda.synchronize()

    def small():
        got[1] = _transitions(kernels[1], starts[1], lambda n: not done.is_set())

    thread = threading.Thread(target=small)
    thread.start()
    got[0] = _transitions(kernels[0], starts[0], lambda n: n < 2000)
    done.set()
    thread.join()
    for i in range(2):
        z, calls, errors = got[i]
        assert not errors, (len(errors), calls, errors[0])
        np.testing.assert_array_equal(z, _transitions(kernels[i], starts[i], lambda n: n < calls)[0])
        kernels[i].close()
