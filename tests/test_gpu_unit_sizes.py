"""The forward kernels over the sizes of their work units: from six blocks of
removed electrons on, a warp takes whole blocks; below, several share one.

Runs large enough for units of sixteen blocks, and of six, against the CPU
oracle (the comparison and its tolerances are those of test_gpu_parity), and
units of every kind against each other: every sum and record is the same bits."""
import numpy as np
import pytest

from cipsi_gb300 import engine, synth
from test_gpu_parity import check, run_both

pytestmark = pytest.mark.gpu

CASES = [
    dict(norb=20, nocc=5, ncf=1300, ranks=(1, 2, 3)),
    dict(norb=20, nocc=5, ncf=1300, ranks=(1, 2, 3), metat=2),
    dict(norb=66, nocc=7, ncf=240, ranks=(1, 2, 3)),
    dict(norb=66, nocc=7, ncf=240, ranks=(2,), metat=2),
]


def config(kw):
    return synth.SynthConfig("u", **dict(dict(ncholesky=10, metat=1, tau=0.02, seed=11, coef_mode="gauss005",
                                              virt_shift=3.0), **kw))


def unit_blocks(inp, r_chunk):
    """Blocks per work unit, by the engine's rule: r_chunk itself below six,
    else 8/3 of it, but no more than leaves six units per thread block."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    gens = int((inp.array("ygen").astype(bool) & ~inp.array("ysaut").astype(bool)).sum())
    nel = 2 * inp.dims.noca
    blocks = gens * nel * (nel + 1) // 2
    return r_chunk if r_chunk < 6 else max(2, min(8 * r_chunk // 3, blocks // (12 * sms)))


@pytest.mark.parametrize("kw", CASES, ids=["one_root", "two_roots", "two_words", "two_words_two_roots"])
def test_whole_blocks_against_oracle(tmp_path, oracle_exe, engine_lib, kw):
    cfg = config(kw)
    wd = str(tmp_path / "plan")
    synth.generate(cfg, wd)
    assert unit_blocks(engine.Inputs(wd), 6) >= (16 if cfg.norb <= 64 else 6)
    check(*run_both(tmp_path, cfg), variant="cipsym")


@pytest.mark.parametrize("kw", CASES[1:3], ids=["two_roots", "two_words"])
def test_every_unit_size_same_bits(tmp_path, engine_lib, kw):
    wd = str(tmp_path / "in")
    synth.generate(config(kw), wd)
    inp = engine.Inputs(wd)
    sizes = {r: unit_blocks(inp, r) for r in (6, 5, 4, 3, 2, 1)}
    assert len(set(sizes.values())) == len(sizes)
    first = None
    with engine.Context(inp.dims) as ctx:
        ctx.upload(inp)
        for r in sizes:
            ctx.set_tuning(r_chunk=r)
            a = ctx.run(inp.opts)
            rec = ctx.selection_raw(a["n_selected"])
            got = [np.asarray(a[k]) for k in ("e2mp", "e2vp", "e2b", "psimp", "psivp", "tabmp", "tabvp", "nom", "nam",
                                              "dpivot", "ietat", "n_processed", "n_selected", "n_candidates")]
            got += [rec[k] for k in ("bits", "owner", "xam", "evp")]
            first = first or [x.copy() for x in got]
            for x, y in zip(first, got):
                assert np.array_equal(x, y), r
