"""The fast kernels at the sizes where they can go wrong: tile and warp edges,
remainders, the smallest and the largest of their ranges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 32, 33, 65])
def test_contact_table_tile_edges(n, engine_lib):
    """table sizes around the product's 32 x 32 tiles against adaptive
    quadrature, with the golden test's tolerance"""
    pytest.importorskip("scipy")
    from oracle import contact_table as CT
    from pimc.engine import contact_table
    g0, tau, rng_ = 2.0, 1.0 / 16, 4.0
    tab = contact_table(g0, tau, rng_, n)
    np.testing.assert_array_equal(tab, tab.T)
    r = CT.grid(rng_, n)
    big = np.abs(tab).max()
    idx = sorted({0, 1, n // 2, max(n - 2, 0), n - 1})
    for i in idx:
        for j in idx:
            if i <= j:
                v = CT.entry(float(r[i]), float(r[j]), g0, tau)
                assert abs(tab[i, j] - v) <= 1e-10 * abs(v) + 1e-13 * big, (i, j, tab[i, j], v)


def test_contact_table_in_several_ranges_of_nodes(engine_lib):
    """a table whose node rows outgrow the scratch (38 k nodes x 608 radii) has
    the entries of a small table of the same quadrature: the 601 grid's every
    200th radius.  Both sum the same terms, |terms| within a few times the
    largest entry, in another order: 38 k rounding errors of 1.1e-16 stay
    below 1e-11 of it"""
    from pimc.engine import contact_table
    big = contact_table(2.0, 1.0 / 2000, 13.0, 601)
    small = contact_table(2.0, 1.0 / 2000, 13.0, 4)
    np.testing.assert_allclose(big[::200, ::200], small, rtol=0, atol=1e-11 * np.abs(small).max())
