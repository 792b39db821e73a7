"""The forward run's sums hold terms of any size: coefficients scaled by a power
of two scale every coupling b, and every term b^2 / d, exactly, so E2 and the
norms of the scaled run are those of the plain one times that power, to the
rounding of the sums.

A sum holds every bit of its terms from 2^-127 to 2^62.  Up to 32 terms below
2^-64 are added up in FP64 first (five additions), and a result adds four parts:
2^-49 covers both sides.  Beyond that range terms are added one by one, or by
32, in FP64: 2^-53 for each perturber."""
import numpy as np
import pytest

from cipsi_gb300 import engine, synth

pytestmark = pytest.mark.gpu

SUMS = ("e2mp", "e2vp", "e2b", "psimp", "psivp")


def _load(tmp_path, **kw):
    cfg = synth.SynthConfig("s", **dict(dict(norb=20, nocc=5, ncholesky=20, ncf=80, metat=1, tau=0.02, ranks=(1, 2, 3),
                                             coef_mode="gauss005", seed=9, virt_shift=3.0), **kw))
    wd = str(tmp_path / "in")
    synth.generate(cfg, wd)
    inp = engine.Inputs(wd)
    return inp, {k: inp.array(k) for k in ("c", "e", "eb", "emp", "teste", "taum", "fmpb")}


@pytest.mark.parametrize("kw", [dict(), dict(norb=70, nocc=4, metat=3), dict(ityper=1, metat=2)],
                         ids=["one_root", "three_roots_two_words", "mp_alone"])
def test_terms_of_any_size(tmp_path, engine_lib, kw):
    inp, roots = _load(tmp_path, **kw)
    with engine.Context(inp.dims) as ctx:
        ctx.upload(inp)
        base = ctx.run(inp.opts)
        n = base["n_processed"]
        for k in (0, -8, -16, -24, -32, -36, -48, -64, -100, 8, 12, 20, 40, 100):
            ctx.set_roots(**dict(roots, c=roots["c"] * 2.0 ** k))
            got = ctx.run(inp.opts)
            assert got["n_processed"] == n
            exact = -36 <= k <= 20
            for q in SUMS:
                np.testing.assert_allclose(np.array(got[q]) * 2.0 ** (-2 * k), base[q], atol=0.0,
                                           rtol=2.0 ** -49 if exact else n * 2.0 ** -53, err_msg=f"{q} at 2^{k}")


def test_infinite_and_undefined_terms(tmp_path, engine_lib):
    inp, roots = _load(tmp_path)
    with engine.Context(inp.dims) as ctx:
        ctx.upload(inp)
        base = ctx.run(inp.opts)
        # infinite EN denominators, by division: no EN terms, the MP ones as they were
        ctx.set_roots(**dict(roots, e=roots["e"] + np.inf))
        got = ctx.run(inp.opts)
        assert got["e2vp"] == [0.0] and got["psivp"] == [0.0]
        np.testing.assert_allclose(got["e2mp"], base["e2mp"], rtol=2.0 ** -49)
        # and undefined ones
        ctx.set_roots(**dict(roots, e=roots["e"] * np.nan))
        got = ctx.run(inp.opts)
        assert np.isnan(got["e2vp"][0]) and np.isnan(got["psivp"][0])
        assert got["n_processed"] == base["n_processed"]


def test_zero_denominators(tmp_path, engine_lib):
    """A root whose MP energy is exactly a perturber's: infinite MP sums, EN sums
    and the set of perturbers as they were."""
    inp, roots = _load(tmp_path)
    opts = engine.Opts.from_buffer_copy(inp.opts)
    opts.tau, opts.ywdeg = -1.0, 0  # a record of every perturber
    fmpb = np.round(roots["fmpb"] * 1024) / 1024  # sums of these are exact
    with engine.Context(inp.dims) as ctx:
        ctx.upload(inp)
        ctx.set_roots(**dict(roots, fmpb=fmpb))
        base = ctx.run(opts)
        bits = ctx.selection_raw(base["n_selected"])["bits"]
        norb, nocc = inp.dims.norb, inp.dims.noca
        occ = np.unpackbits(np.ascontiguousarray(bits).view(np.uint8), axis=1, bitorder="little")
        occ = np.concatenate([occ[:, :norb], occ[:, 64:64 + norb]], axis=1).astype(float)
        hmp = (occ - np.tile(np.arange(norb) < nocc, 2)) @ fmpb
        ctx.set_roots(**dict(roots, fmpb=fmpb, emp=hmp[len(hmp) // 2:][:1]))
        got = ctx.run(opts)
    assert np.isinf(got["e2mp"][0]) and np.isinf(got["psimp"][0])
    assert got["n_processed"] == base["n_processed"] and got["n_selected"] == base["n_selected"]
    for q in ("e2vp", "e2b", "psivp"):
        np.testing.assert_allclose(got[q], base[q], rtol=2.0 ** -49, atol=0.0)
