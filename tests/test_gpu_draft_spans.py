"""GPU tests of the draft head over caches that no cluster per KV head holds: span attention with borrowed K / V rows, queries one
position ahead of the last row they see, launches that are called off."""
import ctypes as C

import numpy as np
import pytest

from tests.conftest import model_files, synth_module

pytestmark = pytest.mark.gpu

LONG = 8300                                   # rows: one more than 64 tiles of 128, the most that a cluster takes


def test_scratch_grows_with_a_later_longer_cache(lg):
    """One head over a short cache, then over a long one: drafts as with the long cache alone."""
    s = synth_module()
    tp, hp = model_files("mid")
    out = []
    for rows in (512, LONG):
        with lg.Session(tp, hp, rows, mtp_n=4) as g:
            prompt = s.prompt_ids(60, g.n_vocab, seed=91)
            g.prefill(prompt[:-1], 0)
            g.next(int(prompt[-1]), 59)                           # leaves the hidden row that the draft starts from
            first = g.draft(int(prompt[0]), 60)
            if rows == LONG:
                out.append([first, g.draft_chain(1, 61)])
                continue
            kv = C.create_string_buffer(256)                      # struct kvcache: 64 bytes
            model, head = C.c_void_p(g.model), C.c_void_p(g.head)
            assert g.L.kvcache_init(kv, model, LONG) == 0
            g.L.model_prefill(model, kv, prompt.ctypes.data_as(C.c_void_p), len(prompt) - 1, 0)
            g.L.model_forward_next(model, kv, int(prompt[-1]), 59)
            out.append([g.L.mtp_draft_device(head, model, kv, int(prompt[0]), 60), g.L.mtp_draft_chain_device(head, model, kv, 1, 61)])
            g.L.kvcache_free(kv)
    assert out[0] == out[1]
