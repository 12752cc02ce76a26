"""The fused FFT / products kernel over its (E, G) plans: one evaluation against the oracle.

A thread takes the column pair (k1, G - k1) of one row: pair 0 holds the two columns that are their
own mirrors, an even E has a bin that is its own mirror (P2 / 2, in column 0), an odd E has it in
column G / 2, and G = 1 has one column.  The orders M give E = 3, 6, 9, 12, 18 with G = 1 .. 16 (P2 = 3 M / 2 =
E G); odd theta counts add the equator row.  Every product set: Boussinesq, with composition,
anelastic with and without it.  The tuner's plans of G = 8 and 4 likewise; from E = 18 on their products
run as the default plan's, bit for bit.

Tolerance: the nonlinear terms of one evaluation, 1e-11 of the largest coefficient, as at the
ordinary sizes.
"""
import importlib

import numpy as np
import pytest

import oracle_lib as ol

pkg = importlib.import_module("leeds-code_b200")
capi = pkg.capi
syn = pkg.synthetic


@pytest.mark.gpu
@pytest.mark.parametrize("anelastic", [False, True])
@pytest.mark.parametrize("comp", [0, 1])
@pytest.mark.parametrize("L,M", [(3, 2), (9, 4), (11, 6), (17, 8), (25, 12), (24, 24), (33, 32), (49, 48), (64, 64),
                                 (97, 96), (129, 128), (192, 192)])
def test_products_plans(L, M, comp, anelastic):
    kw = dict(L=L, M=M, N=6, KL=2, comp_tstep=comp)
    cfg = syn.config_anelastic(**kw) if anelastic else syn.config_parity(Ra_comp=80.0, Sc=1.5, **kw)
    g, o = pkg.Context(cfg), ol.Oracle(cfg)
    if anelastic:
        prof = syn.polytrope_reference_state(cfg.N)
        g.set_reference_state(prof)
        o.set_reference_state(prof)
    for f, (re, im) in syn.boussinesq_state(cfg, seed=L, composition=bool(comp)).items():
        g.set_coll(f, re, im)
        o.set_coll(f, re, im)
    g.nonlinear()
    o.nonlinear()
    for f in range(6 if comp else 5):
        a, b = np.stack(g.get_nonlinear(f)), np.stack(o.get_nonlinear(f))
        assert np.abs(a - b).max() <= 1e-11 * max(np.abs(b).max(), 1e-300), f
    g.close()
    o.close()


@pytest.mark.gpu
@pytest.mark.parametrize("anelastic", [False, True])
@pytest.mark.parametrize("comp", [0, 1])
@pytest.mark.parametrize("L,M", [(24, 24), (33, 32), (48, 48), (64, 64), (97, 96), (128, 128), (192, 192)])
def test_products_tuner_plans(L, M, comp, anelastic):
    kw = dict(L=L, M=M, N=6, KL=2, comp_tstep=comp)
    cfg = syn.config_anelastic(**kw) if anelastic else syn.config_parity(Ra_comp=80.0, Sc=1.5, **kw)
    g = pkg.Context(cfg)
    if anelastic:
        g.set_reference_state(syn.polytrope_reference_state(cfg.N))
    state = syn.boussinesq_state(cfg, seed=L, composition=bool(comp))
    first = None
    for E, G in pkg.lsd.tune_candidates(cfg)["fft"]:
        g.set_tuning(fft_E=E, fft_G=G)
        for f, (re, im) in state.items():  # stress-free walls: an evaluation adjusts the state
            g.set_coll(f, re, im)
        g.nonlinear()
        got = [np.stack(g.get_nonlinear(f)) for f in range(6 if comp else 5)]
        first = first or got
        for a, b in zip(got, first):
            if E >= 18:
                assert np.array_equal(a, b), (E, G)
            assert np.abs(a - b).max() <= 1e-11 * max(np.abs(b).max(), 1e-300), (E, G)
    g.close()
