"""corr_dgemm_tc at the edges of its K passes, K chunks and epilogue branches,
against an extended-precision product.

Bound per element, derived from the splitting: operands rounded at 2^-57 of a
row's (column's) scale, levels below 2^-56 dropped and one rounding to FP64
give 8 * 2^-53 * sqrt(k) * max|row| * max|column| (the module's bound), plus
one FP64 rounding of the running sum per further K chunk of 2048.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(C, A, B, alpha=1.0, C0=None, extra=0):
    k = A.shape[1]
    ex = alpha * (A.astype(np.longdouble) @ B.astype(np.longdouble))
    if C0 is not None:
        ex = ex + C0
    bound = 8.0 * 2.0 ** -53 * np.sqrt(k) * abs(alpha) * np.outer(np.abs(A).max(1),
                                                                  np.abs(B).max(0))
    bound = bound + (1 + extra) * 2.0 ** -52 * np.abs(ex).astype(np.float64)
    err = np.abs(C - ex).astype(np.float64)
    assert (err <= bound).all(), (err / bound).max()


@pytest.mark.parametrize("m,n,k", [
    (130, 66, 512), (130, 66, 513), (70, 70, 1024), (65, 129, 2047), (65, 129, 2048),
    (65, 129, 2049), (40, 33, 4100), (257, 63, 31),
])
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 1)])
def test_pass_and_chunk_edges(ctx, m, n, k, ta, tb):
    r = O.rng(m + n + k)
    A, B = r.standard_normal((m, k)), r.standard_normal((k, n))
    C = ctx.dgemm(np.ascontiguousarray(A.T) if ta else A, np.ascontiguousarray(B.T) if tb else B,
                  transa=bool(ta), transb=bool(tb), tensor_cores=True)
    _check(C, A, B, extra=(k - 1) // 2048)


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("k", [480, 1536, 2100])
def test_large_level_sums(ctx, sign, k):
    """Every product of one sign and near the row scale: level sums above the
    2^22 of the epilogue's fast conversion, integer sums near their largest."""
    r = O.rng(5 + k)
    A, B = r.uniform(0.96, 1.0, (140, k)), sign * r.uniform(0.96, 1.0, (k, 70))
    C = ctx.dgemm(A, B, tensor_cores=True)
    _check(C, A, B, extra=(k - 1) // 2048)
    A[3] *= 1e-9                      # one small row beside the large ones
    A[7, ::2] *= -1.0                 # and one whose sum cancels
    C = ctx.dgemm(A, B, tensor_cores=True)
    _check(C, A, B, extra=(k - 1) // 2048)


@pytest.mark.parametrize("alpha", [1.0, -1.0, 2.0, -0.125, 3.0])
def test_alpha_in_the_exponent(ctx, alpha):
    r = O.rng(17)
    A, B, C0 = r.standard_normal((75, 90)), r.standard_normal((90, 45)), r.standard_normal((75, 45))
    C = ctx.dgemm(A, B, alpha=alpha, beta=1.0, out=C0.copy(), tensor_cores=True)
    _check(C, A, B, alpha, C0, extra=1)


@pytest.mark.parametrize("scale", [2.0 ** -520, 2.0 ** -537, 2.0 ** 500])
def test_extreme_scales(ctx, scale):
    """Results near and below the smallest normal value (rounded as FP64 does,
    to within one subnormal step) and near the largest."""
    r = O.rng(23)
    A, B = r.standard_normal((20, 40)), r.standard_normal((40, 30))
    C = ctx.dgemm(A * scale, B * scale, tensor_cores=True)
    ex = (A.astype(np.longdouble) @ B.astype(np.longdouble)) * np.longdouble(scale) ** 2
    bound = 8.0 * 2.0 ** -53 * np.sqrt(40) * np.outer(np.abs(A).max(1), np.abs(B).max(0))
    bound = bound.astype(np.longdouble) * np.longdouble(scale) ** 2 + np.longdouble(2.0) ** -1074
    assert (np.abs(C - ex) <= bound).all()


def test_misaligned_device_operands(ctx):
    """Rows at odd 8-byte addresses take the scalar loads of the slicing."""
    import torch

    r = O.rng(29)
    base = torch.from_numpy(r.standard_normal(1 + 61 * 77)).cuda()
    A = base[1:].view(61, 77)
    B = torch.from_numpy(r.standard_normal((77, 40))).cuda()
    C = ctx.dgemm(A, B, tensor_cores=True)
    _check(C.cpu().numpy(), A.cpu().numpy(), B.cpu().numpy())


@pytest.mark.parametrize("m,n,k", [
    (128, 64, 64), (129, 65, 200), (100, 64, 2048), (256, 256, 500), (700, 700, 700),
    (700, 260, 1030), (1300, 900, 33), (128, 64, 4099),
])
def test_tiles_split_over_k(ctx, m, n, k):
    """Few tiles: each is summed by several CTAs.  Same bound, the same bits on
    every run, and the same integers whatever part arrives last."""
    import torch

    r = O.rng(m + n + 2 * k)
    A, B = r.standard_normal((m, k)), r.standard_normal((k, n))
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    C = ctx.dgemm(dA, dB, tensor_cores=True)
    _check(C.cpu().numpy(), A, B, extra=(k - 1) // 2048)
    for _ in range(5):
        assert torch.equal(ctx.dgemm(dA, dB, tensor_cores=True), C)
