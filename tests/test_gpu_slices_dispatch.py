"""LSD_PREC_OZAKI contexts on either side of the lines between the int8-slice contraction and the
FP64 tensor instruction (int8: up to 5 slices, and 8; at 6 and 7 from a number of harmonics per order
on, each direction for itself): every transform against the oracle, with odd theta counts and
partial tiles.

Tolerance: S slices carry 8 S - 2 bits of each operand's row or column maximum.  Measured over all
transforms, three seeds and 13 shapes: 6.5e-4 of the largest output at S = 2, 3.0e-6 (3), 1.2e-8 (4),
5.8e-11 (5), 2.9e-13 (6), some 215 times per slice.  The bounds are 2.8e-3 / 215^(S - 2), 4 to 5
times that, and 1e-12 from S = 7 on and where the FP64 instruction runs.
"""
import importlib
from fractions import Fraction

import numpy as np
import pytest

import oracle_lib as ol

pkg = importlib.import_module("leeds-code_b200")
capi = pkg.capi


def relerr(a, b):
    return float(np.abs(np.asarray(a) - np.asarray(b)).max() / max(np.abs(np.asarray(b)).max(), 1e-300))


def route(g):
    """(synthesis, analysis) run on the slices: a slicing pass and a GEMM, two launches, where the FP64
    contraction is one; a scalar transform has one more launch, the phi FFT."""
    n0 = g.kernel_launches()
    phys = g.tra_spec2phys(*np.zeros((2, g.N, g.H)))
    n1 = g.kernel_launches()
    g.tra_phys2spec(phys)
    n2 = g.kernel_launches()
    assert {n1 - n0, n2 - n1} <= {2, 3}
    return n1 - n0 == 3, n2 - n1 == 3


@pytest.mark.gpu
@pytest.mark.parametrize("L,M,Mp,S,int8", [
    # FP64 took 1.04 .. 1.50 times the slices' time at these
    (208, 32, 1, 6, (True, True)), (256, 64, 1, 6, (True, True)), (160, 96, 1, 6, (True, False)),
    (192, 96, 1, 6, (True, True)), (256, 64, 1, 7, (True, True)), (208, 64, 1, 7, (True, True)),
    (208, 32, 1, 7, (True, True)), (204, 128, 1, 7, (True, True)),
    # and 0.4 .. 1.02 times at these
    (128, 16, 1, 6, (False, False)), (192, 192, 1, 6, (False, False)), (192, 32, 6, 6, (False, False)),
    (256, 256, 1, 6, (False, True)), (256, 256, 1, 7, (False, False)), (192, 96, 1, 7, (False, False)),
    (256, 32, 8, 7, (False, False)), (192, 64, 1, 7, (False, True)), (153, 48, 1, 7, (True, False)),
    (64, 16, 4, 7, (False, False)),
    (64, 16, 4, 5, (True, True)), (64, 16, 4, 8, (True, True))])
def test_faster_side_of_the_dispatch(L, M, Mp, S, int8):
    """also: lsd_create makes the three (synthesis) and two (analysis) digit tables of the directions
    that read them"""
    kw = dict(L=L, M=M, Mp=Mp, N=6, KL=2, timestep=1e-5)
    f = pkg.Context(capi.template_config(**kw))
    g = pkg.Context(capi.template_config(precision=capi.PREC_OZAKI, ozaki_slices=S, **kw))
    assert g.kernel_launches() - f.kernel_launches() == 3 * int8[0] + 2 * int8[1]
    assert route(g) == int8
    f.close()
    g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("L,M,S", [(17, 8, 2), (79, 64, 3), (113, 64, 4), (128, 16, 5), (33, 32, 6), (192, 32, 6),
                                   (193, 32, 6), (200, 64, 6), (200, 64, 7), (64, 64, 8), (128, 16, 2), (17, 8, 3),
                                   (160, 24, 6), (192, 16, 7)])
def test_transforms_across_the_dispatch(L, M, S):
    kw = dict(L=L, M=M, Mp=1, N=7, KL=2, timestep=1e-5)
    g, o = pkg.Context(capi.template_config(precision=capi.PREC_OZAKI, ozaki_slices=S, **kw)), ol.Oracle(
        capi.template_config(**kw))
    int8_s, int8_a = route(g)
    tol_s, tol_a = (max(2.8e-3 / 215.0 ** (S - 2), 1e-12) if int8 else 1e-12 for int8 in (int8_s, int8_a))
    rng = np.random.default_rng(L + M + S)
    _, m, _ = o.harmonics()

    def spec():
        re, im = rng.standard_normal((2, o.N, o.H))
        im[:, m == 0] = 0
        return re, im

    q, s, t = spec(), spec(), spec()
    grid = [rng.standard_normal((o.N, o.Ph, o.Th)) for _ in range(3)]
    assert relerr(g.tra_spec2phys(*q), o.spec2phys(*q)) < tol_s
    for x, y in zip(g.tra_qst2rtp(q, s, t), o.qst2rtp(q, s, t)):
        assert relerr(x, y) < tol_s
    for x, y in zip(g.tra_grad(*q), o.grad(*q)):
        assert relerr(x, y) < tol_s
    assert relerr(g.tra_phys2spec(grid[0]), o.phys2spec(grid[0])) < tol_a
    for x, y in zip(g.tra_rtp2qst(*grid), o.rtp2qst(*grid)):
        assert relerr(x, y) < tol_a
    g.close()
    o.close()


@pytest.mark.gpu
def test_eight_slices_exceed_fp64():
    """Eight slices carry 62 bits of the power of two above each operand's row or column maximum and
    sum digit products exactly; the diagonals are joined by Horner's rule in FP64, whose last two
    steps exceed 53 bits.  A sum of K products is off by at most 2 x 2^-53 |sum| for these two
    roundings, K (2 x 2^-63 + 9 x 2^-62) of the powers' product for the operands' rounding and the
    dropped digit pairs, and 2^-53 K / 60 of it for the part of the lower diagonals in the sums that
    are rounded.  A chain of FP64 multiply-adds exceeds that here, where the partial sums are far
    larger than the sum.  The phi transform is exact for these inputs: m = 0 alone,
    and a grid with one phi sample."""
    L, M, N = 64, 16, 7
    g = pkg.Context(capi.template_config(L=L, M=M, Mp=1, N=N, KL=2, timestep=1e-5, precision=capi.PREC_OZAKI,
                                         ozaki_slices=8))
    rng = np.random.default_rng(8)
    l, m, _ = g.harmonics()

    def rise_and_fall(k):
        return np.where(np.arange(k) < k // 2, 1.0, -1.0) * (0.99 - 0.25 * rng.random((N, k)))

    def check(got, c, T):  # got[n, i] = sum_k c[n, k] T[i, k]
        a = c.shape[1] * (10.0 / 512.0 + 1.0 / 60.0)
        cf = [[Fraction(v) for v in row] for row in c.tolist()]
        above = lambda v: 2.0 ** int(np.frexp(np.abs(v).max())[1])
        for i, row in enumerate(T.tolist()):
            tf = [Fraction(v) for v in row]
            for n in range(N):
                x = sum(u * v for u, v in zip(cf[n], tf))
                err = abs(float(Fraction(float(got[n, i])) - x))
                assert err <= 2.0 ** -53 * (2.0 * abs(float(x)) + a * above(c[n]) * above(T[i])), (n, i)

    idx = np.flatnonzero((m == 0) & (l % 2 == 0))
    re, im = np.zeros((2, N, g.H))
    re[:, idx] = rise_and_fall(idx.size)
    phys = g.tra_spec2phys(re, im)
    assert np.array_equal(phys, np.broadcast_to(phys[:, :1, :], phys.shape))
    check(phys[:, 0, :g.Th2], re[:, idx], g.legendre_table(capi.LEG_P)[:, idx])

    grid = np.zeros((N, g.Ph, g.Th))
    grid[:, 0, :g.Th2] = rise_and_fall(g.Th2)
    re, im = g.tra_phys2spec(grid)
    idx = np.flatnonzero(m == 0)
    check(re[:, idx], grid[:, 0, :g.Th2] * (1.0 / g.Ph), g.legendre_table(capi.LEG_GWP)[:, idx].T)
    g.close()
