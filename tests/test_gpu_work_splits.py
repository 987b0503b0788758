"""GPU tests of how matmuls and attention are cut into work: two teams of a CTA behind one panel, spans merged by a launch of their
own, several tiles per CTA of the dense prompt matmul, k slices of a cluster."""
import numpy as np
import pytest

from tests.conftest import model_files, synth_module
from tests.test_gpu_prefill import _weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wtype,m,k,teams", [("q4_0", 9664, 2624, 2), ("q4_K", 9664, 2816, 2), ("q4_0", 2400, 4160, 2), ("q4_0", 9664, 5120, 1)])
@pytest.mark.parametrize("M", [5, 8])
def test_two_teams_of_a_cta(lg, port_built, wtype, m, k, teams, M):
    """More items than SMs and two panels; 151 items leave the last team idle, 150 do not.  The panels of 5120 columns leave no room for a
    second team.  Rows equal the one-panel launch's."""
    s = synth_module()
    rng = np.random.default_rng(m + k)
    raw, t, w = _weights(s, rng, wtype, m, k)
    assert lg.load().lg_debug_matmul_teams(t, m, k, M) == teams and lg.load().lg_debug_matmul_teams(t, m, k, 4) == 1
    x = rng.standard_normal((M, k)).astype(np.float32)
    got = lg.gemv(t, raw, m, k, x)
    want = x.astype(np.float64) @ w.astype(np.float64).T
    # activations: 16-bit integers of their 32-group (2^-16 of its largest); f32 sums
    assert np.abs(got - want).max() / np.abs(want).max() < 2e-4
    assert np.array_equal(got[:4], lg.gemv(t, raw, m, k, x[:4]))


@pytest.mark.parametrize("depth", [100, 128 * 8 - 2, 128 * 8 + 5, 128 * 65 + 1])
def test_span_merge(lg, depth):
    """Spans of two tiles of 64 keys: a single one, eight (one per warp of the merge), nine, and more than eight per warp.  The two
    decompositions add the same f32 terms in another order: 1e-4 of the logits' range is some 50 times what that makes."""
    s = synth_module()
    tp, _ = model_files("mid")
    out = []
    for spans in (False, True):
        lg.set_attn_deep(64 if spans else 1 << 30, 2 if spans else 0)
        try:
            with lg.Session(tp, None, 8704) as g:
                toks = s.prompt_ids(depth + 4, g.n_vocab, seed=61)
                g.prefill(toks[:depth], 0)
                out.append(np.stack([g.forward(int(toks[depth + i]), depth + i) for i in range(4)]))
        finally:
            lg.set_attn_deep()
    assert np.abs(out[0] - out[1]).max() / (out[0].max() - out[0].min()) < 1e-4


@pytest.mark.parametrize("n", [4, 8])
def test_spans_where_no_cluster_fits(lg, n):
    """A cache too long for a cluster and too short for spans that fill the GPU: spans of two tiles against one tile per CTA, and a
    speculative stream that equals the plain one."""
    s = synth_module()
    tp, _ = model_files("mid")
    out = []
    for min_seq in (-1, 1 << 30):
        lg.set_attn_deep(min_seq, 0)
        try:
            with lg.Session(tp, None, 8300, mtp_n=n) as g:
                prompt = s.prompt_ids(700, g.n_vocab, seed=63)
                g.prefill(prompt[:-1], 0)
                out.append(g.forward(int(prompt[-1]), len(prompt) - 1))
        finally:
            lg.set_attn_deep()
    assert np.abs(out[0] - out[1]).max() / (out[0].max() - out[0].min()) < 1e-4        # as above
    with lg.Session(tp, None, 8300, mtp_n=n) as g:
        plain, _ = g.generate_device(prompt, 200, 0)
    with lg.Session(tp, None, 8300, mtp_n=n) as g:
        mtp, _ = g.generate_device(prompt, 200, 2, s.replay_drafts(plain, g.n_vocab, 0.7))
    assert np.array_equal(plain[:200], mtp[:200])


@pytest.mark.parametrize("m,k,n", [(2400, 150, 2000), (4128, 320, 2048), (2080, 64, 2300), (1312, 640, 4100)])
def test_dense_prompt_matmul_of_several_tiles_per_cta(lg, m, k, n):
    """More tiles than CTAs, ragged in tokens and rows, fewer and more blocks of k than ring stages."""
    rng = np.random.default_rng(m + k)
    bf = lambda a: (np.ascontiguousarray(a, np.float32).view(np.uint32) & 0xffff0000).view(np.float32)
    w, x = bf(rng.standard_normal((m, k)) * k ** -0.5), bf(rng.standard_normal((n, k)))
    want = x.astype(np.float64) @ w.T.astype(np.float64)
    # exact products, f32 sums of up to 640 terms
    assert np.abs(lg.dense_matmul(w, x) - want).max() / np.abs(want).max() < 2e-5


@pytest.mark.parametrize("m,k", [(1024, 4800), (1152, 11840)])
@pytest.mark.parametrize("M", [1, 6])
def test_cluster_slices_of_unequal_length(lg, port_built, m, k, M):
    """75 and 185 positions in four k slices: the ranks of a cluster hold panels of different lengths, yet send their sums to the
    same places of rank 0's shared memory."""
    from tests.test_gpu_kernels import _oracle, _resid_ref
    s = synth_module()
    rng = np.random.default_rng(m + k + M)
    o = _oracle()
    raw = s.quantize_q4_0(rng.standard_normal(m * k).astype(np.float32) * 0.02)
    w = o.dequant(s.Q4_0, raw, m * k).reshape(m, k)
    o.close()
    act, x = rng.standard_normal((M, k)).astype(np.float32), rng.standard_normal((M, m)).astype(np.float32)
    add_w, norm_w = ((1.0 + 0.3 * rng.standard_normal(m)).astype(np.float32) for _ in range(2))
    xn, y, cluster = lg.matmul_resid(s.Q4_0, raw, m, k, act, x, add_w, 1.0, norm_w, 1e-6)
    want_x, want_y = _resid_ref(w, act, x, add_w, 1.0, norm_w, 1e-6)
    assert cluster
    # 16-bit integers of the 32-group (2^-16 of its largest), f32 sums
    assert np.abs(xn - want_x).max() / np.abs(want_x).max() < 2e-4 and np.abs(y - want_y).max() / np.abs(want_y).max() < 2e-4
