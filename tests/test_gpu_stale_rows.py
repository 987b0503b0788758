"""GPU tests of cache rows behind a block: what an earlier use left there, not-a-numbers among it, is not seen."""
import numpy as np
import pytest

from tests.conftest import model_files, synth_module

pytestmark = pytest.mark.gpu


def _steps(g, prompt, spoil):
    """Logits of three tokens behind a prompt, successors of a block of 4 and of one of 8; rows 0 .. 127 hold NaN before the prompt."""
    n = len(prompt) - 16
    if spoil:
        g.prefill_embd(np.full((128, g.n_embd), np.nan, dtype=np.float32), 0)
        k, v = g.kv_row(g.n_layer - 1, 127, 512)
        assert np.isnan(k).all() and np.isnan(v).all()
    g.prefill(prompt[:n], 0)
    out = [g.forward(int(prompt[n + i]), n + i) for i in range(3)]
    for width in (4, 8):
        g.mtp_n = width
        g.L.lgs_set_mtp_n(g.h, width)
        out.append(g.spec(prompt[n + 3:n + 3 + width], n + 3)[1].copy())
    return out


# spans of two tiles of 64 keys, a cluster's tiles of 128; sliding-window layers
@pytest.mark.parametrize("name,rows", [("full", 8300), ("full", 4096), ("mid", 512)])
@pytest.mark.parametrize("n", [40, 57])
def test_rows_behind_a_block_are_not_seen(lg, name, rows, n):
    s = synth_module()
    tp, _ = model_files(name)
    got = []
    for spoil in (False, True):
        with lg.Session(tp, None, rows) as g:
            got.append(_steps(g, s.prompt_ids(n + 16, g.n_vocab, seed=81), spoil))
    for clean, spoiled in zip(*got):
        assert np.array_equal(clean, spoiled)
