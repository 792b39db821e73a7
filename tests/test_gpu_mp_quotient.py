"""The Moller-Plesset partition alone (ityper = 1): a record's value is the
coefficient <I|H|Psi> / (E - hmp(I)), correctly rounded as the reference's own
division is.

Orbital energies and the root's (lowered by 64, so that no perturber comes near
it) are rounded to 2^-10, so that every denominator is exact whatever the order
of its sum; a first run with denominators of -1 gives the couplings themselves."""
import numpy as np
import pytest

from cipsi_gb300 import engine, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [dict(norb=20, nocc=5, ncf=60), dict(norb=68, nocc=3, ncf=40)], ids=["one_word", "two_words"])
def test_coefficients_are_quotients(tmp_path, engine_lib, kw):
    cfg = synth.SynthConfig("q", **dict(dict(ncholesky=12, metat=1, tau=0.01, ityper=1, ranks=(1, 2), seed=17,
                                             coef_mode="gauss005", virt_shift=3.0), **kw))
    wd = str(tmp_path / "in")
    synth.generate(cfg, wd)
    inp = engine.Inputs(wd)
    roots = {k: inp.array(k) for k in ("c", "e", "eb", "emp", "teste", "taum", "fmpb")}
    roots["taum"] = np.ones(1)
    opts = engine.Opts.from_buffer_copy(inp.opts)
    opts.tau, opts.ywdeg = -1.0, 0  # every perturber, its own value
    with engine.Context(inp.dims) as ctx:
        ctx.upload(inp)

        def values(emp, fmpb):
            ctx.set_roots(**dict(roots, emp=emp, fmpb=fmpb))
            n = ctx.run(opts)["n_selected"]
            return ctx.selection_raw(n)

        b = values(-np.ones(1), 0.0 * roots["fmpb"])
        fmpb, emp = np.round(roots["fmpb"] * 1024) / 1024, np.round(roots["emp"] * 1024) / 1024 - 64.0
        got = values(emp, fmpb)
    assert np.array_equal(b["bits"], got["bits"]) and len(got["xam"]) > 10000
    W, norb = got["bits"].shape[1] // 2, cfg.norb
    occ = np.unpackbits(np.ascontiguousarray(got["bits"]).view(np.uint8), axis=1, bitorder="little")
    occ = np.concatenate([occ[:, :norb], occ[:, 64 * W:64 * W + norb]], axis=1).astype(float)
    ref = np.tile(np.arange(norb) < cfg.nocc, 2).astype(float)
    denominators = np.abs(emp[0] - (occ - ref) @ fmpb)
    assert denominators.min() > 0.05
    assert np.array_equal(got["xam"], b["xam"] / denominators)
