"""Integrals with a centre that is not finite: NaN in the blocks of that shell,
whatever the NaN's sign and payload (the Boys table is indexed by the low bits of its
argument), and every other block as without the shell."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [0x7FF8000000000000, 0xFFF8000000000000, 0xFFF8000000000F00,
                                  0xFFFFFFFFFFFFFFFF, 0x7FF0000000000000, 0xFFF0000000000000])
def test_centre_not_finite(ctx, bits):
    import corr_gb300

    l, exps, coefs = [0, 2, 1], [3.0, 0.9, 0.5], [1.0, 1.0, 1.0]
    cen = np.array([[0.0, 0.0, 0.0], [0.3, -0.2, 0.8], [0.0, 0.9, 0.1]])
    obs = corr_gb300.Basis([0, 1], [1, 1], [0, 1], cen[[0, 2]], [1.1, 0.4], [1.0, 1.0])

    def run(shells, c):
        aux = corr_gb300.Basis([l[s] for s in shells], [1] * len(shells), range(len(shells)),
                               c[shells], [exps[s] for s in shells], [coefs[s] for s in shells])
        return ctx.ri_integrals(obs, aux, device="cpu")

    bad = cen.copy()
    bad[1, 0] = np.array([bits], dtype=np.uint64).view(np.float64)[0]
    J, P = run([0, 1, 2], bad)
    J0, P0 = run([0, 2], cen)
    keep = [0, 6, 7, 8]  # functions of shells 0 and 2
    assert np.array_equal(J[np.ix_(keep, keep)], J0) and np.array_equal(P[keep], P0)
    assert np.isnan(J[1:6, keep]).any() and not np.isfinite(J[1:6, 1:6]).all()
    assert np.isnan(P[1:6]).any()
