"""Device memory of the digit GEMM's callers: an operand's digit planes stay within 1 GiB
(the product runs in blocks of its columns), and the blocks give the whole product.

Bounds on what a context may take: the panel (512 MiB for the energy, one occupied
orbital's for the gradient), 1 GiB of column planes, the block's row planes and 31 MB
of split sums, times the workspace's 9/8.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GIB = 1 << 30


def _normal(shape, seed, scale):
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float64) * scale


def _eps(o, v, seed):
    import torch

    r = np.random.default_rng(seed)
    return torch.from_numpy(np.concatenate([r.uniform(-1.5, -0.3, o),
                                            r.uniform(0.05, 3.0, v)])).cuda()


def _taken(call):
    """What `call` of a new context returns, and the device memory it took."""
    import torch

    import corr_gb300

    with corr_gb300.Context(0) as c:
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        out = call(c)
        torch.cuda.synchronize()
        return out, free - torch.cuda.mem_get_info()[0]


def test_energy(ctx):
    o, v, x = 20, 1000, 13600  # B 2.2 GB, its digit planes 4.4 GB
    B, eps = _normal((x, o, v), 1, 0.01), _eps(o, v, 1)
    e, taken = _taken(lambda c: c.rimp2_energy(B, eps, o, v, x, "fp64"))
    assert taken <= (512 << 20) * 9 / 8 + 9 / 8 * (GIB + 160e6) + 64e6
    ctx.set_fp64_strict(True)
    try:
        ref = ctx.rimp2_energy(B, eps, o, v, x, "fp64")
    finally:
        ctx.set_fp64_strict(False)
    for a, b in ((e.e_ss, ref.e_ss), (e.e_os, ref.e_os)):
        assert abs(a - b) <= 1e-12 * abs(ref.e_total)


def test_gradient(ctx):
    o, v, x = 160, 1000, 8  # a panel of one orbital 1.28 GB, planes of 160000 columns 2.6 GB
    B, eps = _normal((x, o, v), 2, 0.1), _eps(o, v, 2)
    (e, dB, de), taken = _taken(lambda c: c.rimp2_gradient(B, eps, o, v, x))
    assert taken <= 9 / 8 * (8.0 * v * (o * v + 64) + GIB + 160e6) + 64e6
    ctx.set_fp64_strict(True)
    try:
        ref = ctx.rimp2_gradient(B, eps, o, v, x)
    finally:
        ctx.set_fp64_strict(False)
    assert abs(e - ref[0]) <= 1e-12 * abs(ref[0])
    for a, b in ((dB, ref[1]), (de, ref[2])):
        assert float((a - b).abs().max()) <= 1e-11 * float(b.abs().max())


@pytest.mark.parametrize("m,n,k", [(130, 40000, 2049), (70, 33000, 4100), (40000, 40000, 33)])
@pytest.mark.parametrize("tb", [False, True])
@pytest.mark.parametrize("beta", [0.0, 1.0])
def test_product_in_blocks(ctx, m, n, k, tb, beta):
    """Columns around the blocks' ends against an extended-precision product (the bound
    of the digit GEMM's tests, per pass of 512)."""
    A, B = _normal((m, k), 3, 1.0), _normal((n, k) if tb else (k, n), 4, 1.0)
    C = _normal((m, n), 5, beta)
    cols = np.r_[0:20, 16376:16392, 32760:32776, n - 20:n]
    rows = np.r_[0:20, m - 20:m]
    C0 = C[rows][:, cols].cpu().numpy().astype(np.longdouble)
    C = ctx.dgemm(A, B, transb=tb, beta=beta, out=C, tensor_cores=True)
    a = A[rows].cpu().numpy()
    b = (B[cols] if tb else B[:, cols].T.contiguous()).cpu().numpy()
    ref = C0 + a.astype(np.longdouble) @ b.T.astype(np.longdouble)
    passes = (k + 511) // 512
    tol = passes * 8 * 2.0 ** -53 * np.sqrt(512) * np.outer(np.abs(a).max(1), np.abs(b).max(1))
    tol = tol + passes * 2.0 ** -52 * (np.abs(C0) + np.abs(a) @ np.abs(b).T)
    assert (np.abs(C[rows][:, cols].cpu().numpy() - ref) <= tol).all()
