"""The plain form's routes: the energy and the gradient from FP64-accurate panels on
the digit GEMM (the default; the energy from 3e7 multiply-adds on) against the FP64
pipe (set_fp64_strict) and the oracle, on both sides of the rule's line, and the
transforms and metric products, which stay on the FP64 pipe.

Tolerances: the repository's FP64 bounds, 1e-12 relative for energies and 1e-11
of the largest component for gradients; transforms 1e-13 of the largest element
per factor (two factors), as in the transform tests.
"""
import contextlib

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def strict(ctx):
    ctx.set_fp64_strict(True)
    try:
        yield
    finally:
        ctx.set_fp64_strict(False)


def _same_energy(a, b, tol=1e-12):
    for x, y in ((a.e_ss, b.e_ss), (a.e_os, b.e_os), (a.e_total, b.e_total)):
        assert abs(x - y) <= tol * max(abs(y), abs(b.e_total)), (x, y)


# (o v)^2 naux around the rule; nvir around the 32-wide panel tiles and the 64-wide
# column tiles; two panels of 512 MiB in the last
@pytest.mark.parametrize("o,v,x", [
    (10, 100, 29), (10, 100, 30), (10, 100, 31), (1, 640, 120), (64, 10, 90), (33, 31, 40),
    (16, 32, 130), (17, 33, 130), (13, 97, 2049), (8, 129, 4100), (50, 180, 24),
])
def test_energy(ctx, o, v, x):
    B, eps = O.synth_rimp2(o, v, x, o + v + x)
    got = ctx.rimp2_energy(B, eps, o, v, x, "fp64")
    with strict(ctx):
        ref = ctx.rimp2_energy(B, eps, o, v, x, "fp64")
    _same_energy(got, ref)
    if o * v <= 1300:
        ess, eos, e = O.rimp2_energy(B, eps, o, v)
        assert abs(got.e_total - e) <= 1e-12 * abs(e) and abs(got.e_ss - ess) <= 1e-12 * abs(e)


def test_energy_of_wide_ranges(ctx):
    """Rows over twelve decades, elements over eight inside each: every element
    of (ia|jb) keeps the accuracy of its row scales, and so does the energy."""
    o, v, x = 12, 90, 150
    r = O.rng(3)
    B, eps = O.synth_rimp2(o, v, x, 4)
    B = B * 10.0 ** r.uniform(-12, 0, (1, o, v)) * 10.0 ** r.uniform(-8, 0, (x, o, v))
    got = ctx.rimp2_energy(B, eps, o, v, x, "fp64")
    with strict(ctx):
        _same_energy(got, ctx.rimp2_energy(B, eps, o, v, x, "fp64"))


@pytest.mark.parametrize("value", ["nan", "inf", "denominator"])
def test_energy_refuses_what_it_refused(ctx, value):
    import corr_gb300

    o, v, x = 12, 90, 150
    B, eps = O.synth_rimp2(o, v, x, 5)
    if value == "denominator":
        eps = np.zeros_like(eps)
    else:
        B[7, 3, 20] = float(value)
    for run in (lambda: ctx.rimp2_energy(B, eps, o, v, x, "fp64"),
                lambda: ctx.rimp2_gradient(B, eps, o, v, x)):
        with pytest.raises(corr_gb300.CorrError):
            run()
    B, eps = O.synth_rimp2(o, v, x, 5)  # and the context still works
    ctx.rimp2_energy(B, eps, o, v, x, "fp64")


def test_rows_below_the_splitting_take_the_fp64_pipe(ctx):
    """A row of subnormals: bit for bit what the FP64 pipe gives."""
    r = O.rng(6)
    J, P = r.standard_normal((300, 300)), r.standard_normal((300, 21, 21))
    J[4] = 3e-310
    got = ctx.ri_build_bpq(J, P)
    with strict(ctx):
        ref = ctx.ri_build_bpq(J, P)
    assert (got == ref).all() and (got[4] != 0).any()


def test_infinities_propagate_as_on_the_fp64_pipe(ctx):
    r = O.rng(7)
    J, P = r.standard_normal((300, 300)), r.standard_normal((300, 21, 21))
    P[5, 2, 3] = np.inf
    P[9, 7, 7] = np.nan
    got = ctx.ri_build_bpq(J, P)
    with strict(ctx):
        ref = ctx.ri_build_bpq(J, P)
    assert np.array_equal(got, ref, equal_nan=True) and np.isfinite(got).any()


@pytest.mark.parametrize("o,v,x", [(3, 7, 9), (9, 64, 70), (11, 65, 40), (5, 131, 2050),
                                   (60, 200, 16), (1, 5300, 5)])
def test_gradient(ctx, o, v, x):
    B, eps = O.synth_rimp2(o, v, x, 7 * o + v + x)
    got = ctx.rimp2_gradient(B, eps, o, v, x)
    got_tc = ctx.rimp2_gradient(B, eps, o, v, x, tensor_cores=True)
    with strict(ctx):
        ref = ctx.rimp2_gradient(B, eps, o, v, x)
    for g in (got, got_tc):
        assert abs(g[0] - ref[0]) <= 1e-12 * max(1.0, abs(ref[0]))
        for a, b in zip(g[1:], ref[1:]):
            assert np.abs(a - b).max() <= 1e-11 * np.abs(b).max()


@pytest.mark.parametrize("n,o,x", [(40, 9, 90), (61, 13, 70), (64, 64 // 4, 130), (130, 1, 33)])
def test_transform_ri_not_symmetric(ctx, n, o, x):
    r = O.rng(n + o + x)
    mos, b = r.standard_normal((n, n)), r.standard_normal((x, n, n))  # b[Q] not symmetric
    got = ctx.transform_ri(2 * o, mos, b)
    ref = np.einsum("im,qmn,an->qia", mos[:o], b, mos[o:], optimize=True)
    assert np.abs(got - ref).max() <= 2e-13 * np.abs(ref).max()
    with strict(ctx):
        s = ctx.transform_ri(2 * o, mos, b)
    assert np.abs(got - s).max() <= 2e-13 * np.abs(ref).max()


def test_metric_products_and_fock(ctx):
    r = O.rng(11)
    J, P = r.standard_normal((210, 210)), r.standard_normal((210, 37, 37))
    ref = (J @ P.reshape(210, -1)).reshape(P.shape)
    assert np.abs(ctx.ri_build_bpq(J, P) - ref).max() <= 1e-13 * np.abs(ref).max()
    assert np.abs(ctx.ri_apply_metric(J, P) - ref).max() <= 1e-13 * np.abs(ref).max()
    C, F = r.standard_normal((290, 290)), r.standard_normal((290, 290))
    ref = C @ F @ C.T
    assert np.abs(ctx.build_fmo(C, F) - ref).max() <= 2e-13 * np.abs(ref).max()
    import torch

    dC, dF = torch.from_numpy(C).cuda(), torch.from_numpy(F).cuda()
    ctx.build_fmo(dC, dF, out=dF)  # the output may be the input
    assert np.abs(dF.cpu().numpy() - ref).max() <= 2e-13 * np.abs(ref).max()


@pytest.mark.parametrize("n", [28, 29, 33, 40])
def test_motrans(ctx, n):
    eri, _ = O.synth_eri(n, n)
    pk = O.pack_eri(eri)
    mos = np.linalg.qr(O.rng(n).standard_normal((n, n)))[0]
    ref = np.einsum("ia,jb,kc,ld,abcd->ijkl", mos, mos, mos, mos, eri, optimize=True)
    got = ctx.motrans(2 * (n // 5), mos, pk)
    assert np.abs(got - ref).max() <= 4e-13 * np.abs(ref).max()
    o = n // 5
    got = ctx.motrans_ovov(2 * o, mos, pk)
    assert np.abs(got - ref[:o, o:, :o, o:]).max() <= 4e-13 * np.abs(ref).max()


@pytest.mark.parametrize("n,o,x", [(24, 5, 70), (60, 12, 190), (75, 15, 240)])
def test_pipeline(ctx, n, o, x):
    r = O.rng(n)
    L = r.standard_normal((x, x))
    J = L @ L.T / x + 0.5 * np.eye(x)
    P = r.standard_normal((x, n, n)) * 0.01
    P = 0.5 * (P + P.transpose(0, 2, 1))
    mos = np.linalg.qr(r.standard_normal((n, n)))[0]
    eps = np.concatenate([np.sort(r.uniform(-1.5, -0.3, o)), np.sort(r.uniform(0.05, 3, n - o))])
    got, cut = ctx.rimp2_energy_from_3index(2 * o, mos, eps, J, P, "fp64")
    with strict(ctx):
        ref, cut2 = ctx.rimp2_energy_from_3index(2 * o, mos, eps, J, P, "fp64")
    _same_energy(got, ref)
    assert cut == cut2 == 0
