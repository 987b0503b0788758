"""GPU tests of the small-M matmul's tiled copies: enough row tiles for two and four per stage, k ranges that end inside a stage at
the matrix's edge (positions past it arrive as zeros) and at a slice's edge (bulk copies)."""
import numpy as np
import pytest

from tests.conftest import model_files, synth_module
from tests.test_gpu_prefill import _weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wtype,m,k,slices", [("q4_0", 9472, 4160, 0), ("q4_0", 18944, 2112, 0), ("q4_K", 9472, 4352, 0),
                                               ("q4_0", 4736, 8320, 2)])
@pytest.mark.parametrize("M", [1, 8])
def test_stages_of_several_row_tiles(lg, port_built, wtype, m, k, slices, M):
    s = synth_module()
    rng = np.random.default_rng(m + k)
    raw, t, w = _weights(s, rng, wtype, m, k)
    x = rng.standard_normal((M, k)).astype(np.float32)
    got = lg.gemv(t, raw, m, k, x, kslices=slices) if slices else lg.gemv(t, raw, m, k, x)
    got = got.sum(axis=0) if got.ndim == 3 else got
    want = x.astype(np.float64) @ w.astype(np.float64).T
    # activations: 16-bit integers of their 32-group (2^-16 of its largest); f32 sums
    assert np.abs(got - want).max() / np.abs(want).max() < 2e-4


@pytest.mark.parametrize("tname,m,k", [("Q8_0", 9472, 4160), ("Q8_0", 18944, 1088), ("Q6_K", 9472, 2304), ("Q3_K", 18944, 1280),
                                       ("Q5_K", 9472, 2304), ("Q5_K", 18944, 1280)])
@pytest.mark.parametrize("M", [1, 8])
def test_stages_of_several_row_tiles_i8(lg, port_built, tname, m, k, M):
    """1024-byte tiles in stages of 2 x 8 and 4 x 4; q5_K brings a fourth array."""
    from oracle.pyref import PortOracle
    s = synth_module()
    t = getattr(s, tname)
    rng = np.random.default_rng(m + k + t)
    raw = s.quantize_q8_0(rng.standard_normal(m * k).astype(np.float32) * 0.02) if t == s.Q8_0 else s.random_k_blocks(rng, m * k, t)
    o = PortOracle(model_files("tiny")[0], None, 64)
    w = o.dequant(t, raw, m * k).reshape(m, k).astype(np.float64)
    o.close()
    x = rng.standard_normal((M, k)).astype(np.float32)
    want = x.astype(np.float64) @ w.T
    # activations: 16-bit integers of their 32-group (2^-16 of its largest); f32 sums
    assert np.abs(lg.gemv(t, raw, m, k, x) - want).max() / np.abs(want).max() < 2e-4
