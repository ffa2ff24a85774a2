"""The Cholesky factorisation with its inverse (blocks of 64, recursive halves)
through the 3-index pipeline: sizes around the blocks, ill-conditioned metrics,
and metrics that it has to refuse.

The precision forms use the factor's inverse: their energies within 1e-7 of the
exact one (the digits of B alone deviate by about 1e-8; a wrong block would be far
off).  The plain form factors and substitutes: 1e-12 relative for well-conditioned
metrics; an ill-conditioned one (condition number k) may move the energy by k 2^-53
times a modest factor (16 here).
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _inputs(x, n, o, seed, cond=10.0):
    r = O.rng(seed)
    q, _ = np.linalg.qr(r.standard_normal((x, x)))
    J = (q * np.geomspace(1.0, 1.0 / cond, x)) @ q.T
    J = 0.5 * (J + J.T)
    P = r.standard_normal((x, n, n)) * 0.01
    P = 0.5 * (P + P.transpose(0, 2, 1))
    mos = np.linalg.qr(r.standard_normal((n, n)))[0]
    eps = np.concatenate([np.sort(r.uniform(-1.5, -0.3, o)), np.sort(r.uniform(0.05, 3, n - o))])
    return mos, eps, J, P


def _both(ctx, x, n, o, seed, cond):
    mos, eps, J, P = _inputs(x, n, o, seed, cond)
    got, cut = ctx.rimp2_energy_from_3index(2 * o, mos, eps, J, P, "fp64")
    ref, cut2 = ctx.rimp2_energy_from_3index(2 * o, mos, eps, J, P, "split_bf16")
    w, v = np.linalg.eigh(J)
    keep = w / w.max() >= 1e-10
    B = ((v[:, keep] / np.sqrt(w[keep])).T @ np.einsum("im,pmn,an->pia", mos[:o], P, mos[o:],
                                                        optimize=True).reshape(x, -1))
    exact = O.rimp2_energy(np.ascontiguousarray(B).reshape(-1, o, n - o), eps, o, n - o)[2]
    return got.e_total, ref.e_total, exact, cut, cut2


@pytest.mark.parametrize("x", [63, 64, 65, 127, 128, 129, 191, 200, 257, 400, 577])
def test_sizes_around_the_blocks(ctx, x):
    n = 60 if x < 300 else 70
    got, ref, exact, cut, cut2 = _both(ctx, x, n, 12, x, 10.0)
    assert cut == cut2 == 0
    assert abs(got - exact) <= 1e-12 * abs(exact) and abs(ref - exact) <= 1e-7 * abs(exact)


@pytest.mark.parametrize("cond", [1e4, 1e7])
def test_ill_conditioned(ctx, cond):
    got, ref, exact, cut, cut2 = _both(ctx, 330, 64, 12, 9, cond)
    assert cut == cut2 == 0
    assert abs(got - exact) <= 16 * cond * 2.0 ** -53 * abs(exact)
    assert abs(ref - exact) <= (1e-7 + 16 * cond * 2.0 ** -53) * abs(exact)


@pytest.mark.parametrize("x,zero", [(130, 3), (200, 1)])
def test_rank_deficient_takes_the_cutoff(ctx, x, zero):
    mos, eps, J, P = _inputs(x, 60, 12, 3)
    r = O.rng(4)
    q, _ = np.linalg.qr(r.standard_normal((x, x)))
    w = np.concatenate([np.zeros(zero), np.geomspace(0.1, 1.0, x - zero)])
    J = (q * w) @ q.T
    J = 0.5 * (J + J.T)
    _, cut = ctx.rimp2_energy_from_3index(24, mos, eps, J, P, "fp64")
    _, cut16 = ctx.rimp2_energy_from_3index(24, mos, eps, J, P, "split_fp16")
    assert cut == cut16 == zero


@pytest.mark.parametrize("bad", ["negative", "nan", "zero"])
def test_refused_metrics(ctx, bad):
    import corr_gb300

    mos, eps, J, P = _inputs(150, 60, 12, 5)
    if bad == "negative":
        J = -J
    elif bad == "zero":
        J = np.zeros_like(J)
    else:
        J[100, 20] = J[20, 100] = np.nan
    with pytest.raises(corr_gb300.CorrError):
        ctx.rimp2_energy_from_3index(24, mos, eps, J, P, "fp64")
