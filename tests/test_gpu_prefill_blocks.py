"""GPU tests of the wide matmul's persistent form (an odd number of k blocks, so a last step of one; row blocks with fewer than
eight row tiles; several items per CTA, several token tiles) and of prompts of several token tiles, key tiles and blocks."""
import numpy as np
import pytest

from tests.conftest import model_files, synth_module
from tests.test_gpu_prefill import _weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k", [(16, 64), (48, 192), (272, 320), (2048, 448)])
@pytest.mark.parametrize("n", [1, 17, 241, 256])
def test_odd_k_blocks_and_ragged_rows(lg, port_built, m, k, n):
    s = synth_module()
    rng = np.random.default_rng(m + k + n)
    raw, t, w = _weights(s, rng, "q4_0", m, k)
    x = rng.standard_normal((n, k)).astype(np.float32)
    got = lg.prefill_matmul(t, raw, m, k, x)
    want = x.astype(np.float16).astype(np.float64) @ w.astype(np.float64).T
    # one f16 rounding per weight (2^-11 relative) and f32 sums
    bound = 2.0 ** -11 * (np.abs(x) @ np.abs(w.T)) + 1e-5 * np.abs(want).max()
    assert (np.abs(got - want) <= bound).all()


@pytest.mark.parametrize("wtype,k", [("q4_0", 448), ("q4_K", 512)])
@pytest.mark.parametrize("n,geglu", [(257, False), (521, True), (1001, False), (1024, True)])
def test_several_items_per_cta(lg, port_built, wtype, k, n, geglu):
    """149 row blocks (the last of four row tiles) x 2 to 4 token tiles: two to five items for each of the 148 CTAs, so that the
    accumulator is handed back between items and the rings of 3 stages run on through items of 4 steps."""
    s = synth_module()
    m = 19008
    rng = np.random.default_rng(n + k)
    x = rng.standard_normal((n, k)).astype(np.float32)
    x16 = x.astype(np.float16).astype(np.float64)
    if geglu:
        (raw, t, wg), (raw_u, _, wu) = _weights(s, rng, wtype, m // 2, k), _weights(s, rng, wtype, m // 2, k)
        got = lg.prefill_matmul(t, raw, m // 2, k, x, raw_up=raw_u)
        g, u = (x16 @ v.astype(np.float64).T for v in (wg, wu))
        want = 0.5 * g * (1.0 + np.tanh(0.7978845608028654 * (g + 0.044715 * g ** 3))) * u
        assert np.abs(got - want).max() / np.abs(want).max() < 5e-3      # f16 output + f16 weights, as of one item
        return
    raw, t, w = _weights(s, rng, wtype, m, k)
    got = lg.prefill_matmul(t, raw, m, k, x)
    want = x16 @ w.astype(np.float64).T
    if wtype == "q4_0":          # one f16 rounding per weight (2^-11 relative) and f32 sums
        assert (np.abs(got - want) <= 2.0 ** -11 * (np.abs(x16) @ np.abs(w.T)) + 1e-5 * np.abs(want).max()).all()
    else:                        # two f16 products and an f16 fma, as of one item
        assert np.abs(got - want).max() / np.abs(want).max() < 4e-3


@pytest.mark.parametrize("n", [257, 521, 1024, 1101])
def test_token_tiles_do_not_change_a_prompt(lg, n):
    """One call (tiles of equal shares, one block of up to 1024) against calls of 200 tokens (one tile each, other k slices)."""
    s = synth_module()
    tp, _ = model_files("mid")
    out = []
    for step in (n, 200):
        with lg.Session(tp, None, 1280) as g:
            toks = s.prompt_ids(n + 1, g.n_vocab, seed=31)
            for i in range(0, n, step):
                g.prefill(toks[i:min(n, i + step)], i)
            rows = [np.concatenate(g.kv_row(layer, p, 512)) for layer in range(2) for p in (0, 199, n - 40, n - 1)]
            out.append((rows, g.forward(int(toks[n]), n)))
    for a, b in zip(*[o[0] for o in out]):
        assert np.abs(a - b).max() <= 1e-2 * max(1.0, np.abs(b).max())
    a, b = out[0][1], out[1][1]
    assert np.abs(a - b).max() / (b.max() - b.min()) <= 1e-2


@pytest.mark.parametrize("name,n,step", [("tiny", 1500, 200), ("tiny", 1500, 64), ("mid", 330, 129)])
def test_prompt_attention_tiles_and_ring(lg, name, n, step):
    """Key tiles behind a wrapped sliding-window ring, first tiles that some rows do not see, query blocks that end inside a tile:
    one call against calls of `step` tokens."""
    s = synth_module()
    tp, _ = model_files(name)
    out = []
    for st in (n, step):
        with lg.Session(tp, None, 2048) as g:
            toks = s.prompt_ids(n + 1, g.n_vocab, seed=32)
            for i in range(0, n, st):
                g.prefill(toks[i:min(n, i + st)], i)
            out.append(g.forward(int(toks[n]), n))
    assert np.abs(out[0] - out[1]).max() / (out[1].max() - out[1].min()) <= 1e-2


@pytest.mark.parametrize("name", ["tiny", "mid"])
@pytest.mark.parametrize("n", [33, 65, 100])
def test_rows_behind_the_prompt_do_not_matter(lg, name, n):
    """A prompt over a cache that an earlier, longer one has filled gives the bits of a fresh cache."""
    s = synth_module()
    tp, _ = model_files(name)
    out = []
    for used in (False, True):
        with lg.Session(tp, None, 512) as g:
            if used:
                g.prefill(s.prompt_ids(400, g.n_vocab, seed=33), 0)
            toks = s.prompt_ids(n + 1, g.n_vocab, seed=34)
            g.prefill(toks[:n], 0)
            out.append(g.forward(int(toks[n]), n))
    assert np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32))


@pytest.mark.parametrize("n", [45, 330, 1001])
@pytest.mark.parametrize("pos0", [0, 21])
def test_a_prompt_that_fills_its_cache(lg, n, pos0):
    """No room for the pad rows of the last block: all whole groups of eight still take the wide pass (the bits of a cache with room
    for the padding, which the narrow path's 16-bit integer activations do not give), and the rows before the prompt stay."""
    s = synth_module()
    tp, _ = model_files("mid")
    out = []
    for room in (1, 600):
        with lg.Session(tp, None, pos0 + n + room) as g:
            toks = s.prompt_ids(pos0 + n + 1, g.n_vocab, seed=35)
            if pos0:
                g.prefill(toks[:pos0], 0)
            g.prefill(toks[pos0:pos0 + n], pos0)
            places = [p for p in (0, pos0 - 1, pos0, pos0 + n // 2, pos0 + n // 8 * 8 - 1) if p >= 0]
            rows = [np.concatenate(g.kv_row(layer, p, 512)) for layer in range(3) for p in places]
            out.append((rows, g.forward(int(toks[pos0 + n]), pos0 + n)))
    for a, b in zip(*[o[0] for o in out]):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    a, b = out[0][1], out[1][1]              # the last 1 to 7 rows come from the narrow path in one of the two
    assert np.abs(a - b).max() / (b.max() - b.min()) <= 1e-2


@pytest.mark.parametrize("n,step", [(45, 45), (300, 300), (300, 131)])
def test_head_size_128_without_groups_matches_oracle(lg, port_built, n, step):
    """128 tokens per attention CTA (one query head per KV head) in two column blocks, a window shorter than the prompt: most rows
    do not see the first key tiles of their CTA."""
    from oracle.pyref import PortOracle
    s = synth_module()
    tp, _ = model_files("hd128")
    o = PortOracle(tp, None, 512, True, 4)
    toks = s.prompt_ids(n + 3, o.n_vocab, seed=36)
    o.prefill(toks[:n], 0)
    with lg.Session(tp, None, 512) as g:
        for i in range(0, n, step):
            g.prefill(toks[i:min(n, i + step)], i)
        for layer in range(4):
            for pos in sorted({max(0, n - 60), n - 33, n - 9, n - 1}):          # the oracle's ring keeps the window's 64 rows
                for a, b in zip(g.kv_row(layer, pos, 4 * 128), o.kv_row(layer, pos, 4 * 128)):
                    assert np.abs(a - b).max() < 1e-2 * max(1.0, np.abs(b).max()), (layer, pos)
        for i in range(n, n + 3):
            want, got = o.forward(int(toks[i]), i), g.forward(int(toks[i]), i)
            assert np.abs(got - want).max() / (want.max() - want.min()) <= 1e-2
    o.close()


def test_timing_pass_takes_the_block_a_prompt_runs(lg):
    """The benchmark times the block that a prompt of its length runs, up to the largest one."""
    import bench
    s = synth_module()
    tp, _ = model_files("mid")
    with lg.Session(tp, None, 2048) as g:
        g.prefill(s.prompt_ids(1024, g.n_vocab, seed=37), 0)
        assert bench.block_of(929) == 936 and bench.block_of(5000) == bench.PF_BLOCK
        assert g.prefill_pass(bench.block_of(929), 0) > 0 and g.prefill_pass(bench.PF_BLOCK, 0) > 0
        assert g.prefill_pass(bench.PF_BLOCK + 1, 0) == -1
