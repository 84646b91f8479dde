"""The non-centred walk past the register instances, where eight steps' loads go together: chunks of whole eights
and with each kind of remainder, and a last thread with none, against the FP64 closed form at the bounds of
test_gpu_sv_potential."""
import pytest

from test_gpu_sv_potential import test_sv_potential_vs_oracle as _check


@pytest.mark.gpu
@pytest.mark.parametrize("T", [4352, 6144, 6145, 7000, 7681, 10001, 20000])
def test_long_walk_vs_oracle(T):
    _check(T, True)
