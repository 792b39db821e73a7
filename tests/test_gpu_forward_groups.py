"""k_cand at the edges of its row groups, list capacities and block sharing,
against the CPU oracle (the comparison and its tolerances are those of
test_gpu_parity)."""
import numpy as np
import pytest

from cipsi_gb300 import engine, synth
from test_gpu_parity import check, run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [
    # fewer than 256 neighbours: the reference's lone blocks copied by every warp
    dict(norb=14, nocc=3, ncf=60, ranks=(1, 2)),
    # 256 and more: built once for all warps; lists longer than shared memory holds
    dict(norb=18, nocc=4, ncf=400, ranks=(1, 2)),
    # sparse rows: sixteen in a group
    dict(norb=24, nocc=5, ncf=120, ranks=(1, 2, 3), nsym=4),
    # two electrons of a spin at most, rows nearly as long as the 64 places of one-word strings
    dict(norb=64, nocc=2, ncf=40, ranks=(1, 2)),
    # the same with four roots' shorter places, and two words: rows of more than 64 columns
    dict(norb=62, nocc=2, ncf=40, ranks=(1, 2), metat=3),
    dict(norb=100, nocc=2, ncf=60, ranks=(1, 2), metat=2),
    dict(norb=70, nocc=3, ncf=300, ranks=(1, 2), metat=5),
], ids=lambda kw: "-".join(f"{v}" for v in kw.values()).replace(" ", ""))
def test_edges_against_oracle(tmp_path, oracle_exe, engine_lib, kw):
    kw = dict(dict(ncholesky=10, metat=1, tau=0.02, seed=11, coef_mode="gauss005", virt_shift=3.0), **kw)
    check(*run_both(tmp_path, synth.SynthConfig("g", **kw)), variant="cipsym")


@pytest.mark.parametrize("r_chunk", [1, 2, 3, 5, 6, 40])
def test_unit_sizes_agree(tmp_path, engine_lib, r_chunk):
    # how many warps share a block follows the unit's size: every sum and record
    # is the same bits
    cfg = synth.SynthConfig("u", norb=22, nocc=4, ncholesky=10, ncf=300, ranks=(1, 2, 3), metat=2, tau=0.01, seed=5)
    wd = str(tmp_path / "in")
    synth.generate(cfg, wd)
    inp = engine.Inputs(wd)
    with engine.Context(inp.dims) as ctx:
        ctx.upload(inp)
        o = inp.opts
        a = ctx.run(o)
        ra = ctx.selection_raw(a["n_selected"])
        ctx.set_tuning(r_chunk=r_chunk)
        b = ctx.run(o)
        rb = ctx.selection_raw(b["n_selected"])
    for k in ("e2mp", "e2vp", "e2b", "psimp", "psivp", "tabmp", "tabvp", "nom", "nam", "n_candidates", "n_processed", "ietat", "dpivot"):
        assert np.array_equal(a[k], b[k]), k
    key = lambda r: sorted(zip(map(bytes, np.ascontiguousarray(r["bits"])), r["owner"].tolist(), r["xam"].tolist()))
    assert key(ra) == key(rb)
