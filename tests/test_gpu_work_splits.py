"""GPU tests of how matmuls and attention are cut into work: two teams of a CTA behind one panel."""
import numpy as np
import pytest

from tests.conftest import synth_module
from tests.test_gpu_prefill import _weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wtype,m,k", [("q4_0", 9664, 2624), ("q4_K", 9664, 2816), ("q4_0", 2400, 4160), ("q4_0", 9664, 5120)])
@pytest.mark.parametrize("M", [5, 8])
def test_two_teams_of_a_cta(lg, port_built, wtype, m, k, M):
    """More items than SMs and two panels; 151 items leave the last team idle, 150 do not.  Rows equal the one-panel launch's."""
    s = synth_module()
    rng = np.random.default_rng(m + k)
    raw, t, w = _weights(s, rng, wtype, m, k)
    x = rng.standard_normal((M, k)).astype(np.float32)
    got = lg.gemv(t, raw, m, k, x)
    want = x.astype(np.float64) @ w.astype(np.float64).T
    # activations: 16-bit integers of their 32-group (2^-16 of its largest); f32 sums
    assert np.abs(got - want).max() / np.abs(want).max() < 2e-4
    assert np.array_equal(got[:4], lg.gemv(t, raw, m, k, x[:4]))
