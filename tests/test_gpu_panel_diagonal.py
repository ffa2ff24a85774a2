"""The plain form's energy where (ia|ia) dominates: the digit products a digit GEMM
leaves out include squares, which add up instead of cancelling.

Every row of B has one element of 1 at a Q of its own and 511 of up to 2^-6, so that
(ia|ia) is near 1 and every other (ia|jb) below 0.1.  512 left-out squares of a digit
uniform in [-64, 64] (1365 on average), each at 2^-70 of the row scale 2 squared, bias
(ia|ia) by 2.4e-15, the energy by 4.7e-15.  Bound: 4 2^-53 relative, the rounding of a few FP64 sums whose errors have
no common sign.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_energy_of_dominant_diagonal(ctx, seed):
    v, x = 256, 512
    r = O.rng(seed)
    B = r.uniform(-1.0, 1.0, (x, 1, v)) / 64
    B[r.permutation(x)[:v], 0, np.arange(v)] = 1.0
    eps = np.concatenate([[-0.7], r.uniform(0.05, 3.0, v)])
    L = B.reshape(x, v).astype(np.longdouble)
    M, e = L.T @ L, eps.astype(np.longdouble)
    E = -(M * M / (e[1:, None] + e[None, 1:] - 2 * e[0])).sum()
    got = [ctx.rimp2_energy(B, eps, 1, v, x, "fp64").e_total,
           ctx.rimp2_gradient(B, eps, 1, v, x)[0],
           ctx.rimp2_gradient(B, eps, 1, v, x, tensor_cores=True)[0]]
    for g in got:
        assert abs(g - E) <= 4 * 2.0 ** -53 * abs(E), float((g - E) / E)
