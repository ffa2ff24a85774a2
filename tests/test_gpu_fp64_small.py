"""The small-tile kernels of the FP64 form: the 16 x 16 GEMM and the 8 x 8
energy, around their tile edges and around the sizes where the 64 x 64 kernels
take over.

GEMM bound per element: k FP64 FMAs, (k + 2) 2^-53 sum|a||b| plus the rounding
of alpha, beta.  Energies against the oracle: the FP64 bound of the repository,
1e-12 relative.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [
    (1, 1, 1), (1, 17, 5), (16, 16, 32), (17, 15, 33), (24, 24, 24), (31, 1, 64), (64, 64, 64),
    (65, 63, 31), (100, 70, 1), (2000, 24, 24), (13824, 24, 24), (300, 300, 90), (900, 800, 40),
])
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_gemm(ctx, m, n, k, ta, tb):
    r = O.rng(m + 3 * n + 7 * k)
    A, B, C0 = r.standard_normal((m, k)), r.standard_normal((k, n)), r.standard_normal((m, n))
    for alpha, beta in ((1.0, 0.0), (-0.7, 1.3)):
        C = ctx.dgemm(np.ascontiguousarray(A.T) if ta else A,
                      np.ascontiguousarray(B.T) if tb else B, transa=bool(ta), transb=bool(tb),
                      alpha=alpha, beta=beta, out=C0.copy())
        ex = alpha * (A @ B) + beta * C0
        bound = (k + 2) * 2.0 ** -52 * abs(alpha) * (np.abs(A) @ np.abs(B)) + \
            2.0 ** -50 * np.abs(beta * C0)
        assert (np.abs(C - ex) <= bound + 1e-300).all()


@pytest.mark.parametrize("o,v,x", [
    (1, 1, 1), (1, 7, 3), (2, 8, 4), (3, 9, 5), (5, 19, 76), (4, 16, 17), (7, 33, 50),
    (9, 64, 31), (12, 40, 90), (20, 20, 40), (40, 12, 21), (1, 130, 40),
])
def test_energy(ctx, o, v, x):
    B, eps = O.synth_rimp2(o, v, x, o + 10 * v + 100 * x)
    e, ref = ctx.rimp2_energy(B, eps, o, v, x, "fp64"), O.rimp2_energy(B, eps, o, v)
    for got, want in zip((e.e_ss, e.e_os, e.e_total), ref):
        assert abs(got - want) <= 1e-12 * max(abs(ref[2]), abs(want))


def test_non_finite_and_zero_denominator_are_refused(ctx):
    import corr_gb300

    B, eps = O.synth_rimp2(3, 9, 20, 1)
    for where in ("nan", "inf", "denominator"):
        Bx, ex = B.copy(), eps.copy()
        if where == "denominator":
            ex[:] = 0.0
        else:
            Bx[3, 1, 2] = float(where)
        with pytest.raises(corr_gb300.CorrError):
            ctx.rimp2_energy(Bx, ex, 3, 9, 20, "fp64")
