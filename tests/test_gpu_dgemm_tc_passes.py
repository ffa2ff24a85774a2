"""The digit GEMM where the operands' magnitudes change over K: every 512 of K has its
own scales, so that the error of a pass is that of its own rows and columns.

Bound per element, from an extended-precision product of every pass: the digit GEMM's
8 2^-53 sqrt(512) max|row| max|column| of the pass, summed over the passes, and
2^-52 of the partial sums per FP64 accumulation.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble
PASS = 512


def _scales(kind, k):
    """Factors of A's and B's elements over K."""
    s = np.array([1.0, 1e6, 1e-5, 1e11])[(np.arange(k) // PASS) % 4]
    if kind == "opposed":
        return s, 1.0 / s
    if kind == "alike":
        return s, s
    if kind == "one":
        return s, np.ones(k)
    z = (np.arange(k) // PASS) % 2  # passes of zeros in A, where B is large
    return 1.0 - z, np.where(z, 1e30, 1e-30)


def _bound_and_ref(A, B, C0):
    ref, parts = C0.astype(LD), np.abs(C0).astype(LD)
    tol = np.zeros(ref.shape, LD)
    npass = 0
    for k0 in range(0, A.shape[1], PASS):
        a, b = A[:, k0:k0 + PASS], B[:, k0:k0 + PASS]
        p = a.astype(LD) @ b.astype(LD).T
        tol += 8 * 2.0 ** -53 * np.sqrt(PASS) * np.outer(np.abs(a).max(1), np.abs(b).max(1))
        ref = ref + p
        parts = parts + np.abs(p)
        npass += 1
    return ref, tol + npass * LD(2) ** -52 * parts


# one tile split over K, a few tiles, tiles of several waves (no split), two launches of K
@pytest.mark.parametrize("m,n,k", [(40, 30, 513), (130, 70, 1024), (130, 70, 2048),
                                   (200, 150, 1536), (1500, 1000, 1100), (1500, 1000, 2047),
                                   (140, 70, 4133)])
@pytest.mark.parametrize("kind", ["opposed", "alike", "one", "zero"])
def test_scales_over_k(ctx, m, n, k, kind):
    r = np.random.default_rng(m + n + k)
    sa, sb = _scales(kind, k)
    A, B = r.standard_normal((m, k)) * sa, r.standard_normal((n, k)) * sb
    rows, cols = (np.sort(r.choice(x, min(x, 24), replace=False)) for x in (m, n))
    for beta in (0.0, 1.0):
        C0 = r.standard_normal((m, n)) * (beta * np.abs(A[0]).max() * np.abs(B[0]).max())
        ref, tol = _bound_and_ref(A[rows], B[cols], C0[np.ix_(rows, cols)])
        for ta in (False, True):  # k adjacent in memory, and rows adjacent
            a, b = (np.ascontiguousarray(x.T) if ta else x for x in (A, B))
            C = ctx.dgemm(a, b, transa=ta, transb=not ta, beta=beta, out=C0.copy(),
                          tensor_cores=True)
            assert (np.abs(C[np.ix_(rows, cols)] - ref) <= tol).all(), (beta, ta)
