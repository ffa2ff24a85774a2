"""Shells that share primitives (corr_basis: poff is free): integrals equal, bit for
bit, those of the same shells with primitives of their own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EXPS, COEFS = [8.0, 2.0, 0.7, 0.3], [0.2, 0.5, 0.4, 1.0]
A, B, C = (0.0, 0.0, 0.0), (1.1, -0.4, 0.3), (-0.7, 0.8, 1.9)
# (l, nprim, poff, centre): parts of another shell's range, whole ranges at other
# angular momenta
SAME_L = [(1, 3, 0, A), (1, 1, 2, B), (1, 2, 1, C)]
MIXED_L = [(0, 3, 0, A), (1, 3, 0, A), (2, 2, 1, B), (3, 1, 3, C)]
ORBITAL = [(0, 2, 0, A), (1, 2, 0, A), (0, 1, 3, B), (2, 1, 2, C)]
PLAIN = [(0, 2, 0, A), (0, 1, 3, B)]


def _basis(shells, shared):
    import corr_gb300

    l, n, off, cen = zip(*shells)
    if shared:
        return corr_gb300.Basis(l, n, off, cen, EXPS, COEFS)
    own = [k for _, m, p, _ in shells for k in range(p, p + m)]
    return corr_gb300.Basis(l, n, np.cumsum((0,) + n[:-1]), cen, [EXPS[k] for k in own],
                            [COEFS[k] for k in own])


@pytest.mark.parametrize("aux,orbital", [(SAME_L, PLAIN), (MIXED_L, PLAIN), (SAME_L, ORBITAL),
                                         (MIXED_L, ORBITAL)])
def test_shared_ranges(ctx, aux, orbital):
    got, ref = (ctx.ri_integrals(_basis(orbital, s), _basis(aux, s), device="cpu")
                for s in (True, False))
    for a, b in zip(got, ref):
        assert np.array_equal(np.asarray(a), np.asarray(b)) and np.abs(b).max() > 0.1
