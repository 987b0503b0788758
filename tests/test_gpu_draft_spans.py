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


# queries around the borders of a tile of 64 keys and of a span of two: the last row they see is one position before them
PLACES = [1, 5, 62, 63, 64, 65, 66, 126, 127, 128, 129, 130, 255, 256, 257, 300]


def _drafts(g, stream, places):
    """(draft, chained draft, chained draft) at each of the places, each behind its own step."""
    out = []
    for p in places:
        g.prefill(stream[:p - 1], 0)
        g.next(int(stream[p - 1]), p - 1)
        d = [g.draft(int(stream[p]), p)]
        for j in (1, 2):
            d.append(g.draft_chain(d[-1], p + j))
        out.append(d)
    return out


def test_drafts_of_spans_equal_those_of_single_tiles(lg):
    """The two decompositions add the same f32 terms in another order, 1e-6 of a logit: no draft changes.  A span, a border or a mask
    that were wrong would change most of them."""
    s = synth_module()
    tp, hp = model_files("mid")
    out = []
    for min_seq in (-1, 1 << 30):
        lg.set_attn_deep(min_seq, 0)
        try:
            with lg.Session(tp, hp, LONG, mtp_n=4) as g:
                out.append(_drafts(g, s.prompt_ids(400, g.n_vocab, seed=92), PLACES))
        finally:
            lg.set_attn_deep()
    assert out[0] == out[1]
    assert len({tuple(d) for d in out[0]}) > len(PLACES) // 2      # and they tell the places apart


def test_drafts_of_spans_match_the_oracle(lg, port_built):
    from oracle.pyref import PortOracle
    s = synth_module()
    tp, hp = model_files("mid")
    o = PortOracle(tp, hp, LONG, True, 4)
    stream = s.prompt_ids(140, o.n_vocab, seed=93)
    same = total = 0
    with lg.Session(tp, hp, LONG, mtp_n=4) as g:
        for i in range(len(stream) - 1):
            o.forward(int(stream[i]), i)
            g.next(int(stream[i]), i)
            if i >= 4:
                total += 1
                same += int(g.draft(int(stream[i + 1]), i + 1) == o.draft(int(stream[i + 1]), i + 1))
    o.close()
    print(f"draft tokens over spans equal to the oracle's: {same}/{total}")
    assert same >= total * 0.8                          # as for the other attention kernels


def test_drafts_do_not_see_rows_at_or_behind_their_position(lg):
    s = synth_module()
    tp, hp = model_files("mid")
    for rows in (LONG, 512):                            # spans, clusters
        out = []
        for spoil in (False, True):
            with lg.Session(tp, hp, rows, mtp_n=4) as g:
                if spoil:
                    g.prefill_embd(np.full((128, g.n_embd), np.nan, dtype=np.float32), 0)
                stream = s.prompt_ids(100, g.n_vocab, seed=94)
                g.prefill(stream[:57], 0)
                g.next(int(stream[57]), 57)
                d = [g.draft(int(stream[58]), 58)]
                out.append(d + [g.draft_chain(d[0], 59)])
        assert out[0] == out[1]


@pytest.mark.parametrize("margin", [0.0, 0.05, 1e30])
def test_stream_with_drafts_over_spans_equals_plain(lg, margin):
    """The head's own drafts, all of them, some or none of the chained ones called off: both launches of the spans leave."""
    s = synth_module()
    tp, hp = model_files("mid")
    with lg.Session(tp, hp, LONG, mtp_n=4) as g:
        prompt = s.prompt_ids(50, g.n_vocab, seed=95)
        plain, _ = g.generate_device(prompt, 100, 0)
    with lg.Session(tp, hp, LONG, mtp_n=4) as g:
        g.set_draft_margin(margin)
        dev, st = g.generate_device(prompt, 100, 1)
        skipped = g.drafts_skipped()
    assert np.array_equal(dev[:100], plain[:100])
    rounds = st[0] // 3
    assert rounds > 0 and (skipped == 0 if margin == 0 else skipped == 2 * rounds if margin > 1 else 0 < skipped < 2 * rounds)
