"""k_cand's tables in shared memory are refilled group of rows by group of rows
and lot of neighbours by lot of neighbours: a run repeated on the same inputs
gives the same bits, in its sums as in its records."""
import numpy as np
import pytest

from cipsi_gb300 import engine, synth

pytestmark = pytest.mark.gpu

ANSWER = ("e2mp", "e2vp", "e2b", "psimp", "psivp", "tabmp", "tabvp", "nom", "nam", "dpivot", "ietat", "n_processed",
          "n_selected", "n_candidates")


@pytest.mark.parametrize("kw", [
    # hundreds of neighbours a block: many lots of 32, lists beyond shared memory
    dict(norb=18, nocc=4, ncf=400, ranks=(1, 2)),
    # rows by sixteens, several groups a block
    dict(norb=40, nocc=4, ncf=300, ranks=(1, 2, 3), nsym=4, metat=2),
    dict(norb=70, nocc=3, ncf=300, ranks=(1, 2), metat=3),
], ids=["lots", "groups", "two_words"])
def test_repeated_runs_same_bits(tmp_path, engine_lib, kw):
    cfg = synth.SynthConfig("r", **dict(dict(ncholesky=10, metat=1, tau=0.01, seed=3, coef_mode="gauss005",
                                             virt_shift=3.0), **kw))
    wd = str(tmp_path / "in")
    synth.generate(cfg, wd)
    inp = engine.Inputs(wd)
    with engine.Context(inp.dims) as ctx:
        ctx.upload(inp)
        first = None
        for _ in range(4):
            r = ctx.run(inp.opts)
            rec = ctx.selection_raw(r["n_selected"])
            got = [np.asarray(r[k]) for k in ANSWER] + [rec[k] for k in ("bits", "owner", "xam", "evp")]
            if first is None:
                assert r["n_selected"] > 0
                first = [x.copy() for x in got]
            for a, b in zip(first, got):
                assert np.array_equal(a, b)
