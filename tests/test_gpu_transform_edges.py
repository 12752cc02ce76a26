"""The transforms at the edges of their tiles, every tra_* against the oracle.

The FP64 contraction takes 48 theta rows (synthesis) or 48 harmonics of one parity (analysis),
16 or 32 shells and 8 + 8 K values at a time; the grid transforms take 4 or 8 half-rows.  The
sizes put remainders everywhere: an odd theta count (the equator row is its own mirror, and an
odd half grid misaligns the tables' rows to 8 bytes), half grids just below and above a tile,
orders with a single harmonic, more than 48 harmonics of a parity, shell counts that are no
multiple of a tile, and every (E, G) family of the FFT lengths 3 2^a and 9 2^a.

Tolerance: both sides sum K <= 2 Th2 = 196 products in FP64, so they differ by at most
2 K 2^-53 = 4.4e-14 of sum |terms|, a few times the largest output here; 1e-12 of the
largest magnitude, as for the transforms at the ordinary sizes.
"""
import importlib

import numpy as np
import pytest

import oracle_lib as ol

pkg = importlib.import_module("leeds-code_b200")
capi = pkg.capi


def relerr(a, b):
    return float(np.abs(np.asarray(a) - np.asarray(b)).max() / max(np.abs(np.asarray(b)).max(), 1e-300))


@pytest.mark.gpu
@pytest.mark.parametrize("L,M,Mp,N", [(3, 2, 1, 6), (9, 4, 2, 7), (17, 12, 1, 6), (33, 6, 4, 17), (37, 16, 2, 9),
                                      (63, 48, 1, 33), (65, 64, 1, 6), (96, 96, 1, 6), (130, 128, 1, 7),
                                      (131, 24, 5, 18)])
def test_transforms_at_tile_edges(L, M, Mp, N):
    cfg = capi.template_config(L=L, M=M, Mp=Mp, N=N, KL=2, timestep=1e-5)
    g, o = pkg.Context(cfg), ol.Oracle(cfg)
    rng = np.random.default_rng(L + M + N)
    _, m, _ = o.harmonics()

    def spec():
        re, im = rng.standard_normal((2, N, o.H))
        im[:, m == 0] = 0
        return re, im

    q, s, t = spec(), spec(), spec()
    grid = [rng.standard_normal((N, o.Ph, o.Th)) for _ in range(3)]
    assert relerr(g.tra_spec2phys(*q), o.spec2phys(*q)) < 1e-12
    assert relerr(g.tra_phys2spec(grid[0]), o.phys2spec(grid[0])) < 1e-12
    for x, y in zip(g.tra_qst2rtp(q, s, t), o.qst2rtp(q, s, t)):
        assert relerr(x, y) < 1e-12
    for x, y in zip(g.tra_rtp2qst(*grid), o.rtp2qst(*grid)):
        assert relerr(x, y) < 1e-12
    for x, y in zip(g.tra_grad(*q), o.grad(*q)):
        assert relerr(x, y) < 1e-12
    g.close()
    o.close()
