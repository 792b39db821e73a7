"""A batch stays valid while its contexts run on their own, as long as no buffer
that its graph refers to is replaced."""
import numpy as np
import pytest

from cipsi_gb300 import engine, synth

pytestmark = pytest.mark.gpu

ANSWER = ("e2mp", "e2vp", "e2b", "psimp", "psivp", "tabmp", "tabvp", "nom", "nam", "ietat", "n_processed", "n_selected")


@pytest.mark.parametrize("members", [1, 4])
def test_batch_after_larger_plain_runs(tmp_path, engine_lib, members):
    pairs = []
    for i in range(members):
        cfg = synth.SynthConfig(f"v{i}", norb=20, nocc=5, ncholesky=10, ncf=600, metat=1, tau=0.01, ranks=(1, 2, 3),
                                seed=20 + i, coef_mode="gauss005", virt_shift=3.0)
        wd = str(tmp_path / cfg.name)
        synth.generate(cfg, wd)
        inp = engine.Inputs(wd)
        ctx = engine.Context(inp.dims)
        ctx.upload(inp)
        # a shard of the generators first: fewer units than the whole run has
        mask = (np.arange(inp.dims.ncf) % 3 == 0).astype(np.uint8)
        ctx.run(inp.opts, gen_mask=mask, run_pertu=False)
        pairs.append((ctx, inp.opts))
    ctxs, opts = [c for c, _ in pairs], [o for _, o in pairs]
    with engine.Batch(ctxs, opts) as b:
        b.run()
        b.wait()
        first = b.fetch_all(allow_overflow=False)
        plain = [c.run(o) for c, o in pairs]
        b.run()
        b.wait()
        second = b.fetch_all(allow_overflow=False)
    for x, y, z in zip(first, plain, second):
        for k in ANSWER:
            assert np.array_equal(x[k], z[k]), k
            np.testing.assert_allclose(x[k], y[k], rtol=1e-12, err_msg=k)
    for c in ctxs:
        c.close()
