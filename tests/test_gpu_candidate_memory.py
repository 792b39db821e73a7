"""The buffer between the two forward kernels: runs that go through it in parts,
contexts that share it, and the memory that many contexts keep."""
import numpy as np
import pytest

from cipsi_gb300 import CipsiError, engine, synth

pytestmark = pytest.mark.gpu

ANSWER = ("e2mp", "e2vp", "e2b", "psimp", "psivp", "tabmp", "tabvp", "nom", "nam", "dpivot", "ietat", "n_processed",
          "n_selected", "n_candidates")
# 64-bit strings, one root, 6 MB; two words, two roots, 0.5 GB
SYSTEMS = [dict(norb=20, nocc=5, ncf=60, ranks=(1, 2)), dict(norb=66, nocc=5, ncf=200, ranks=(1, 2, 3), metat=2)]


def load(tmp_path, **kw):
    cfg = synth.SynthConfig("m", **dict(dict(ncholesky=10, metat=1, tau=0.01, seed=7, coef_mode="gauss005",
                                             virt_shift=3.0, energy="diagonal"), **kw))
    wd = str(tmp_path / f"in{cfg.seed}")
    synth.generate(cfg, wd)
    inp = engine.Inputs(wd)
    ctx = engine.Context(inp.dims)
    ctx.upload(inp)
    return ctx, inp.opts


def answer(res):
    return [np.asarray(res[k]) for k in ANSWER]


def records(ctx, res):
    rec = ctx.selection_raw(res["n_selected"])
    return [rec[k] for k in ("bits", "owner", "xam", "evp")]


def same(a, b):
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info(0)[0]


@pytest.mark.parametrize("kw", SYSTEMS, ids=["one_word", "two_words"])
def test_parts_give_the_same_bits(tmp_path, engine_lib, kw):
    ctx, opts = load(tmp_path, **kw)
    with ctx:
        whole = ctx.run(opts)
        assert whole["launches"] == 5  # both kernels once
        recs = records(ctx, whole)
        assert len(recs[1]) > 0
        for limit in (1, 1 << 20, 3 << 20):
            ctx.set_candidate_bytes(limit)
            part = ctx.run(opts)
            assert part["launches"] > 5
            same(answer(part), answer(whole))
            same(records(ctx, part), recs)
            same(answer(ctx.run_stream(opts)), answer(whole))
            with engine.Batch([ctx], [opts]) as b:
                b.run()
                b.wait()
                got = b.fetch_all(allow_overflow=False)[0]
                same(answer(got), answer(whole))
                same(records(ctx, got), recs)
        ctx.set_candidate_bytes(0)
        assert ctx.run(opts)["launches"] == 5
        with pytest.raises(CipsiError):
            ctx.set_candidate_bytes(-1)


def test_contexts_take_turns(tmp_path, engine_lib):
    """Runs of several contexts in flight at once, each more than a context's
    own buffer holds."""
    pairs = [load(tmp_path, **dict(SYSTEMS[1], seed=s)) for s in (1, 2, 3, 4)]
    alone = [(answer(c.run(o)), c) for c, o in pairs]
    for _ in range(2):
        for c, o in pairs:
            c.run_async(o)
        for a, c in alone:
            same(answer(c.fetch()), a)
    for c, _ in pairs:
        c.close()


def test_memory_of_many_contexts(tmp_path, engine_lib):
    """Two dozen contexts whose candidates take 1.1 GB each: a process that
    holds them all keeps one buffer, and a few hundred MB a context for lists
    and records."""
    kw = dict(norb=45, nocc=9, ncf=450, ranks=(1, 2))
    first, opts = load(tmp_path, **kw)
    ref = answer(first.run(opts))
    shared = free_bytes()  # code, local memory, the shared buffer and one context's own
    ctxs = [first] + [load(tmp_path, **kw)[0] for _ in range(23)]
    for c in ctxs:
        same(answer(c.run(opts)), ref)
    assert shared - free_bytes() < 23 * (300 << 20)
    for c in ctxs:
        c.close()
    assert free_bytes() > shared
