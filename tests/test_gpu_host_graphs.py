"""GPU tests of the graphs that the host waits for: what enters through their imports and what leaves with the status word."""
import numpy as np
import pytest

from tests.conftest import model_files, synth_module

pytestmark = pytest.mark.gpu


def test_nothing_starts_before_an_import_has_ended(lg):
    """The attention of the target reads the position ahead of its dependency wait.  A missing trigger in the import is not enough for
    that: the edge behind it has to be a full one, in every graph that begins with an import."""
    s = synth_module()
    tp, hp = model_files("mid")
    with lg.Session(tp, hp, 512, mtp_n=4) as g:
        early = np.full(1, -1, dtype=np.int32)
        prompt = s.prompt_ids(41, g.n_vocab, seed=71)
        edges = []
        for step in (lambda: g.forward(int(prompt[0]), 0), lambda: g.next(int(prompt[1]), 1),          # one token, with and without logits
                     lambda: g.prefill_logits(prompt, 0, [40]),                                         # the last token of a prompt
                     lambda: g.spec(prompt[:4], 41), lambda: g.draft(int(prompt[0]), 45)):              # a verify block, a whole round
            step()
            edges.append(g.L.lg_debug_import_edges(g.model, early))
            assert early[0] == 0
        assert edges == [1, 2, 3, 4, 5]                          # every one of them began with an import


@pytest.mark.parametrize("family", ["hybrid", "latent"])
def test_nothing_starts_before_an_import_has_ended_in_plan_models(lg, family):
    from tests import hybrid_models, latent_models
    shape, _, path = hybrid_models.model("deep") if family == "hybrid" else latent_models.model("mixed")
    toks = synth_module().prompt_ids(8, shape.vocab, seed=72)
    early = np.full(1, -1, dtype=np.int32)
    with lg.Session(path, None, 64, mtp_n=4) as g:
        g.forward(int(toks[0]), 0), g.next(int(toks[1]), 1), g.spec(toks[2:6], 2)
        assert g.L.lg_debug_import_edges(g.model, early) == 3 and early[0] == 0
