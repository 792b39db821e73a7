"""The Hamiltonian's pair scan at the edges of its column segments and row
blocks: the columns of every row against a numpy degree test, the elements of
a sample of rows against the Slater-Condon rules (synth.SlaterCondon)."""
import ctypes

import numpy as np
import pytest

from cipsi_gb300 import engine, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norb,ncf,jmax", [(16, 1, -1), (16, 127, -1), (20, 1023, -1), (20, 1025, -1),
                                           (20, 2049, 1100), (70, 1030, -1), (20, 1500, 0)])
def test_scan_edges(tmp_path, engine_lib, norb, ncf, jmax):
    cfg = synth.SynthConfig("h", norb=norb, nocc=4, ncholesky=12, ncf=ncf, metat=1, tau=0.02, ranks=(1, 2, 3), seed=3,
                            energy="diagonal")
    wd = str(tmp_path / "in")
    synth.generate(cfg, wd)
    inp = engine.Inputs(wd)
    rng = np.random.default_rng(cfg.seed)
    h, L, irrep = synth.make_integrals(cfg, rng)
    dets, _ = synth.build_space(cfg, rng, irrep)
    n = inp.dims.ncf
    bits = [synth.det_from_lists(a, b, norb, cfg.nocc) for a, b in dets]
    m64 = (1 << 64) - 1
    M = np.array([[a & m64, a >> 64, b & m64, b >> 64] for a, b in bits], dtype=np.uint64)
    lib = engine._lib()
    P, I64 = ctypes.c_void_p, ctypes.c_int64
    lib.cipsi_hamiltonian_build.argtypes = [P, P, ctypes.c_int32, ctypes.POINTER(I64)]
    lib.cipsi_hamiltonian_get.argtypes = [P, ctypes.c_int32, ctypes.c_int32, P, P, P]
    with engine.Context(inp.dims) as ctx:
        if n == 1:  # S of the reference determinant alone has no hole list: the upload refuses it
            with pytest.raises(engine.CipsiError, match="null array"):
                ctx.upload(inp)
            return
        ctx.upload(inp)
        for _ in range(2):  # the second build reuses the workspace
            npairs = I64()
            ctx._check(lib.cipsi_hamiltonian_build(ctx._c, None, jmax, ctypes.byref(npairs)), "build")
            rp, col, val = np.zeros(n + 1, np.int64), np.zeros(max(npairs.value, 1), np.int32), \
                np.zeros(max(npairs.value, 1))
            ctx._check(lib.cipsi_hamiltonian_get(ctx._c, 0, n, rp.ctypes.data, col.ctypes.data, val.ctypes.data), "get")
            want = []
            for i in range(n):
                top = min(i, n if jmax < 0 else jmax)
                d = np.bitwise_count(M[:top] ^ M[i]).sum(axis=1)
                want.append(np.nonzero(d <= 4)[0])
            assert np.array_equal(np.diff(rp), [len(w) for w in want])
            assert npairs.value == rp[n]
            assert np.array_equal(col[:npairs.value], np.concatenate(want) if want else [])
    sc = synth.SlaterCondon(h, L, norb, cfg.nocc)
    sg = [synth.cip_phase(a, b, norb, cfg.nocc) for a, b in dets]
    for i in range(0, n, max(1, n // 12)):
        for t in list(range(rp[i], rp[i + 1]))[::5]:
            j = int(col[t])
            ref = sg[i] * sg[j] * sc.offdiag(*bits[i], *bits[j])
            # integrals are stored as real*4 (2^-24 relative), up to about 20 of them, each below 10, in an element
            assert abs(val[t] - ref) <= 20 * 10 * 2.0 ** -24, (i, j, val[t], ref)
