"""The Cholesky factor and its inverse by recursive halves (chol.cu), directly.

Bounds from the standard error analysis of blocked factorisation and substitution
(N. J. Higham, Accuracy and Stability of Numerical Algorithms, ch. 8 and 10), whose
constants grow with the order m: |L L^T - J| <= 4 m 2^-53 max J (|L| |L^T| is at most
max J for a positive definite J, and the digit GEMM adds its row and column maxima),
|X L - I| <= 4 m 2^-53 max (|X| |L|).  Orders around the blocks of 64, and on both
sides of the 1e7 multiply-adds from which the products run on the digit GEMM (384, 448).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _metric(m, cond, seed):
    r = np.random.default_rng(seed)
    q, _ = np.linalg.qr(r.standard_normal((m, m)))
    J = (q * np.geomspace(1.0, 1.0 / cond, m)) @ q.T
    return 0.5 * (J + J.T)


@pytest.mark.parametrize("m", [1, 2, 63, 64, 65, 127, 128, 129, 191, 257, 384, 448, 577, 1100])
@pytest.mark.parametrize("cond", [10.0, 1e6])
def test_residuals(ctx, m, cond):
    J = _metric(m, cond, m)
    L, X = ctx.selftest_factor(J)
    assert not np.triu(L, 1).any() and not np.triu(X, 1).any()
    rows = np.sort(np.random.default_rng(1).choice(m, min(m, 40), replace=False))
    Ll, Xl = L.astype(np.longdouble), X.astype(np.longdouble)
    u = 4 * m * 2.0 ** -53
    assert np.abs(Ll[rows] @ Ll.T - J[rows]).max() <= u * np.abs(J).max()
    R = Xl[rows] @ Ll
    R[np.arange(len(rows)), rows] -= 1
    assert np.abs(R).max() <= u * (np.abs(X[rows]) @ np.abs(L)).max()


@pytest.mark.parametrize("m", [40, 65, 130, 500])
@pytest.mark.parametrize("bad", ["negative", "zero", "first", "last", "nan", "inf", "indefinite"])
def test_refused(ctx, m, bad):
    import corr_gb300

    J = _metric(m, 10.0, m)
    if bad in ("negative", "zero"):
        J *= -1.0 if bad == "negative" else 0.0
    elif bad == "indefinite":  # one eigenvalue below zero
        v = np.linalg.eigh(J)[1][:, 0]
        J -= 0.5 * np.outer(v, v)
    else:
        i = 0 if bad == "first" else m - 1
        J[i, i] = {"nan": np.nan, "inf": np.inf}.get(bad, -1e-3)
    with pytest.raises(corr_gb300.CorrError):
        ctx.selftest_factor(J)
    J = _metric(m, 10.0, m)  # and the context still works
    L, _ = ctx.selftest_factor(J)
    assert np.abs(L @ L.T - J).max() <= 4 * m * 2.0 ** -53 * np.abs(J).max()


@pytest.mark.parametrize("bad", ["negative", "nan", "zero"])
@pytest.mark.parametrize("precision", ["split_fp16", "split_bf16", "fp64"])
def test_pipeline_refuses_the_metric(ctx, bad, precision):
    import corr_gb300

    n, o, x = 40, 9, 150
    r = np.random.default_rng(5)
    J, P = _metric(x, 10.0, 5), 0.01 * r.standard_normal((x, n, n))
    P = 0.5 * (P + P.transpose(0, 2, 1))
    mos = np.linalg.qr(r.standard_normal((n, n)))[0]
    eps = np.concatenate([np.sort(r.uniform(-1.5, -0.3, o)), np.sort(r.uniform(0.05, 3, n - o))])
    good, _ = ctx.rimp2_energy_from_3index(2 * o, mos, eps, J, P, precision)
    K = -J if bad == "negative" else 0.0 * J
    if bad == "nan":
        K = J.copy()
        K[100, 20] = K[20, 100] = np.nan
    with pytest.raises(corr_gb300.CorrError):
        ctx.rimp2_energy_from_3index(2 * o, mos, eps, K, P, precision)
    again, _ = ctx.rimp2_energy_from_3index(2 * o, mos, eps, J, P, precision)
    assert again.as_tuple() == good.as_tuple()
