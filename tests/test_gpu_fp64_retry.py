"""Calls that the digit GEMM's range guard sends back to the FP64 pipe: a part of B
below 2^-958 or subnormal among normal values.  The repeated call gives what a strict
context gives (energies bit for bit; gradients to rounding, their sums are atomic), and
it has run: the launches of both routes are counted.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

O_, V, X = 10, 70, 700  # (o v)^2 x = 3.4e8: energies on panels, two passes of 512


def _small_parts(kind, B):
    B = B.copy()
    if kind == "row":              # (i, a) of all Q
        B[:, 3, 20] *= 1e-300
    elif kind == "subnormal row":
        B[:, 9, 69] = 3e-310
    elif kind == "segment":        # (i, a) of the second 256 of Q alone
        B[256:512, 0, 5] *= 1e-300
    elif kind == "second pass":
        B[512:, 4, 0] *= 1e-300
    else:                          # one Q of all (i, a): a row of the gradient's products
        B[5] *= 1e-300
    return B


def _run(ctx, call, strict=False):
    """Result and launches of a call."""
    ctx.set_fp64_strict(strict)
    try:
        n = ctx.timing().launches_total
        out = call()
        return out, ctx.timing().launches_total - n
    finally:
        ctx.set_fp64_strict(False)


@pytest.mark.parametrize("kind", ["row", "subnormal row", "segment", "second pass"])
def test_energy(ctx, kind):
    B, eps = O.synth_rimp2(O_, V, X, 1)
    _, digits = _run(ctx, lambda: ctx.rimp2_energy(B, eps, O_, V, X, "fp64"))
    S = _small_parts(kind, B)
    got, n = _run(ctx, lambda: ctx.rimp2_energy(S, eps, O_, V, X, "fp64"))
    ref, fp64 = _run(ctx, lambda: ctx.rimp2_energy(S, eps, O_, V, X, "fp64"), strict=True)
    assert n == digits + fp64 and got.as_tuple() == ref.as_tuple()
    e = O.rimp2_energy(S, eps, O_, V)[2]
    assert abs(got.e_total - e) <= 1e-12 * abs(e)


@pytest.mark.parametrize("kind", ["row", "subnormal row", "segment", "second pass", "one Q"])
def test_gradient(ctx, kind):
    B, eps = O.synth_rimp2(O_, V, X, 2)
    _, digits = _run(ctx, lambda: ctx.rimp2_gradient(B, eps, O_, V, X))
    S = _small_parts(kind, B)
    got, n = _run(ctx, lambda: ctx.rimp2_gradient(S, eps, O_, V, X))
    ref, fp64 = _run(ctx, lambda: ctx.rimp2_gradient(S, eps, O_, V, X), strict=True)
    assert n == digits + fp64
    assert abs(got[0] - ref[0]) <= 1e-13 * abs(ref[0])
    for a, b in zip(got[1:], ref[1:]):
        assert np.abs(a - b).max() <= 1e-13 * np.abs(b).max()


def test_pipeline(ctx):
    n, o, x = 60, 10, 190
    r = O.rng(3)
    L = r.standard_normal((x, x))
    J = L @ L.T / x + 0.5 * np.eye(x)
    P = r.standard_normal((x, n, n)) * 0.01
    P = 0.5 * (P + P.transpose(0, 2, 1))
    mos = np.linalg.qr(r.standard_normal((n, n)))[0]
    eps = np.concatenate([np.sort(r.uniform(-1.5, -0.3, o)), np.sort(r.uniform(0.05, 3, n - o))])
    call = lambda m: ctx.rimp2_energy_from_3index(2 * o, m, eps, J, P, "fp64")
    _, digits = _run(ctx, lambda: call(mos))
    small = mos.copy()
    small[4] *= 1e-300  # (P|ia) and B of one occupied orbital
    (got, cut), launches = _run(ctx, lambda: call(small))
    (ref, cut2), fp64 = _run(ctx, lambda: call(small), strict=True)
    assert launches == digits + fp64 and cut == cut2 == 0
    assert got.as_tuple() == ref.as_tuple()


def test_output_over_an_input(ctx):
    """dE/d eps over eps: refused on either route, as eps is cleared before it is read."""
    import torch

    import corr_gb300

    B, eps = O.synth_rimp2(O_, V, 40, 4)
    dB = torch.from_numpy(B).cuda()
    for strict in (False, True):
        de = torch.from_numpy(eps).cuda()
        with pytest.raises(corr_gb300.CorrError):
            _run(ctx, lambda: ctx.rimp2_gradient(dB, de, O_, V, 40, deps=de), strict)
    ctx.rimp2_gradient(dB, torch.from_numpy(eps).cuda(), O_, V, 40)  # the context still works
