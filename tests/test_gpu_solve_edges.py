"""The streamed banded solves at the edges of their tiles: two steps (predictor and corrector
solves of every field) against the oracle, and the same bits for every CTA size.

A warp takes 32 degrees of one order, a CTA 1, 2 or 4 orders, a ring stage 4 rows.  The sizes put
the last block of degrees at 1, 31, 8 and 1 degrees, orders that start inside a block, orders that
are no multiple of a CTA's, every half-width KL, the fewest rows (N = 2 KL + 2), row counts that
are no multiple of a stage, and the inner core's smallest and largest mesh.  Infinite and overflowing
right-hand sides give the infinities and NaN of the divisions they stand for.

Tolerance: FP64 on both sides in different orders; the toroidal velocity amplifies rounding most (the
oracle's own change under last-bit perturbations of its initial state is 6e-11 of the largest
coefficient at lmax 127 after 3 steps), so 1e-10 of each field's largest coefficient.
"""
import importlib

import numpy as np
import pytest

import oracle_lib as ol

pkg = importlib.import_module("leeds-code_b200")
capi = pkg.capi
syn = pkg.synthetic

CASES = [dict(L=33, M=8, Mp=4, N=6, KL=2), dict(L=31, M=24, Mp=1, N=23, KL=5), dict(L=40, M=16, Mp=2, N=14, KL=6),
         dict(L=65, M=64, Mp=1, N=18, KL=4, comp_tstep=1, vel_bc=2), dict(L=16, M=16, Mp=1, N=17, KL=3, vel_bc=4),
         dict(L=33, M=16, Mp=2, N=19, KL=3, Nic=7, rot_tstep=1), dict(L=20, M=8, Mp=2, N=13, KL=2, Nic=13, rot_tstep=1)]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join("%s%s" % kv for kv in c.items()))
def test_steps_at_tile_edges(case):
    cfg = syn.config_parity(**dict(dict(timestep=1e-5, Ra_comp=80.0, Sc=1.5), **case))
    o = ol.Oracle(cfg)
    state = syn.boussinesq_state(cfg, seed=5, composition=bool(cfg.comp_tstep))
    fields = list(state) + ([capi.MAG_IC_TOR, capi.MAG_IC_POL] if cfg.Nic > 1 else [])
    for f, (re, im) in state.items():
        o.set_coll(f, re, im)
    so = o.step(2)
    first = None
    for threads in (128, 64, 32):
        g = pkg.Context(cfg)
        g.set_tuning(solve_threads=threads)
        for f, (re, im) in state.items():
            g.set_coll(f, re, im)
        sg = g.step(2)
        assert sg.steps_done == so.steps_done and sg.correctors == so.correctors
        got = [np.stack(g.get_coll(f)) for f in fields]
        g.close()
        if first is None:
            first = got
            for f, a in zip(fields, got):
                b = np.stack(o.get_coll(f))
                assert np.abs(a - b).max() <= 1e-10 * max(np.abs(b).max(), 1e-300), f
        else:
            assert all(np.array_equal(a, b) for a, b in zip(first, got)), threads
    o.close()


def ieee_solve(ab, ipiv, kl, b):
    """dgbtrs on the factors, without its tests for zero"""
    n, b = b.size, b.copy()
    for j in range(n):
        p = ipiv[j] - 1
        b[j], b[p] = b[p], b[j]
        for i in range(1, min(kl, n - 1 - j) + 1):
            b[j + i] -= ab[2 * kl + i, j] * b[j]
    for j in range(n - 1, -1, -1):
        b[j] = b[j] / ab[2 * kl, j]
        for t in range(1, min(2 * kl, j) + 1):
            b[j - t] -= b[j] * ab[2 * kl - t, j]
    return b


@pytest.mark.gpu
def test_infinite_right_hand_sides():
    import torch
    cfg = capi.template_config(L=8, M=8, Mp=1, N=16, KL=3, timestep=1e-5, cod_bc=2)
    g, o = pkg.Context(cfg), ol.Oracle(cfg)
    l, _, _ = o.harmonics()
    fields, lu = (capi.COD_C, capi.MAG_POL), (3, 5)
    # rows of Re and Im of a harmonic: an infinity just inside the outer wall (it reaches the wall's row
    # and its quotient), the largest magnitude there, an infinity in the middle, ordinary values
    kinds = [(14, np.inf), (14, -np.inf), (14, np.finfo(float).max), (7, np.inf), (7, 1.0)]
    b = np.ones((len(fields), cfg.N, g.H, 2))
    b[:, [0, -1]] = 0.0
    for nh in range(g.H):
        for part in range(2):
            row, v = kinds[(nh + 2 * part) % len(kinds)]
            b[:, row, nh, part] = v
    d = torch.tensor(b, device="cuda")
    torch.cuda.synchronize()
    g.operator_solve_device(list(fields), d.data_ptr())
    g.synchronize()
    x = d.cpu().numpy()
    seen = 0
    with np.errstate(all="ignore"):
        for k, f in enumerate(fields):
            for nh in range(g.H):
                if f != capi.COD_C and l[nh] == 0:
                    continue
                ab, ipiv = o.operator_lu(lu[k], int(l[nh]))
                for part in range(2):
                    want, got = ieee_solve(ab, ipiv, cfg.KL, b[k, :, nh, part]), x[k, :, nh, part]
                    assert np.array_equal(np.isnan(want), np.isnan(got)), (f, nh, part)
                    inf = np.isinf(want)
                    assert np.array_equal(inf, np.isinf(got)) and np.array_equal(want[inf], got[inf]), (f, nh, part)
                    seen += inf.sum()
                    fin = np.isfinite(want)
                    if fin.all():
                        assert np.abs(want - got).max() <= 1e-10 * np.abs(want).max(), (f, nh, part)
    assert seen > 0
    g.close()
    o.close()
