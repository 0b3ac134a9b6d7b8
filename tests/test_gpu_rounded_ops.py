"""The branch-free reciprocal and quotient of the RK5 step, exhaustively, and states outside the
range they cover: the step then divides as before."""
import ctypes

import numpy as np
import pytest

import nestgpu as ngpu
import oracle as orc

pytestmark = pytest.mark.gpu


def test_reciprocal_and_quotient_correctly_rounded():
    f = ngpu._lib.NGPU_TestRoundedOps
    f.restype = ctypes.c_longlong
    assert f() == 0


@pytest.mark.parametrize("model", ["aeif_cond_beta_multisynapse", "aeif_psc_exp_multisynapse"])
@pytest.mark.parametrize("scale", [1e30, 3e37, 3e38])
def test_states_beyond_the_range_match_oracle(model, scale):
    """Input weights that drive the error scale past 2^126, to infinity and to NaN."""
    def run(api):
        n = api.Create(model, 4, 1)
        sg = api.Create("spike_generator")
        api.SetStatus(sg, {"spike_times": [0.5, 1.0, 2.0]})
        for i in range(4):
            api.Connect(sg, [n[i]], {"rule": "one_to_one"}, {"weight": float(scale * (i - 1)), "delay": 0.3, "receptor": 0})
        api.Simulate(1.6)
        return np.asarray(api.GetStatus(n, "V_m"), dtype=np.float32), np.asarray(api.GetStatus(n, "w"), dtype=np.float32)
    ngpu.Reset()
    ngpu.SetVerbosityLevel(0)
    got = run(ngpu)
    ngpu.Reset()
    want = run(orc.Oracle())
    for a, b in zip(got, want):
        assert np.array_equal(a, b, equal_nan=True)
