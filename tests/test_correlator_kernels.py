"""The correlator and slab kernels at the edges of their blocks.  Without
updates the two-level estimator is the single-level multihit correlator: every
sub-update has the same slab products, and a product of slab products over time
is the Polyakov loop's.  Both are FP64 sums of the same FP32 links, so they agree
to FP64 rounding (about 1e-14 of the largest term; 1e-12 asked)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from latticeu1_b200 import Context
    return Context(0)


# sub-updates: one, a full batch, one more, several batches; extents: r beyond a
# direction's extent, partial blocks of columns and lines, a line longer than a block
@pytest.mark.parametrize("N", [(4, 2, 2, 4), (12, 4, 2, 8), (10, 6, 14, 4), (24, 16, 20, 12), (2, 2, 2, 36),
                               (4, 520, 2, 4), (1030, 2, 4, 4)])
@pytest.mark.parametrize("n2", [1, 16, 17, 35])
def test_multilevel_without_updates_is_the_multihit_correlator(ctx, N, n2):
    from latticeu1_b200 import Lattice, Rng
    lat = Lattice(ctx, 4, N, 0.9, 1.3)
    rng = Rng(ctx, 5)
    lat.hot_start(rng)
    single = lat.poly_corr(True)
    multi = lat.multilevel(rng, 2, 0, n2, 0, 1, 1)
    lat.close()
    assert np.abs(multi - single).max() <= 1e-12 * np.abs(single).max()


@pytest.mark.parametrize("dims,N", [(2, (6, 0, 0, 4)), (2, (70, 0, 0, 34)), (3, (8, 6, 0, 2)), (3, (34, 10, 0, 50)),
                                    (4, (6, 4, 10, 18)), (4, (20, 14, 6, 32))])
def test_poly_corr_matches_float64(ctx, dims, N):
    """The plain correlator from the links themselves in 64 bits (products of Nt
    FP32 links: relative error about Nt * 6e-8 each, averaged; 1e-5 asked)."""
    from latticeu1_b200 import Lattice, Rng
    lat = Lattice(ctx, dims, N, 1.0)
    lat.hot_start(Rng(ctx, 11))
    th = lat.export_angles()
    got = lat.poly_corr(False)
    ext = lat.grid[:dims]
    V = lat.V
    lex = np.arange(V)
    par, r = np.zeros(V, int), lex.copy()
    for e in ext:
        par, r = par + r % e, r // e
    t = th.reshape(dims, V)[dims - 1][(lex >> 1) + (par & 1) * (V // 2)].reshape(ext[::-1])
    P = np.exp(1j * t.sum(axis=0))
    want = np.array([sum((P * np.roll(P, -k, axis=dims - 2 - d).conj()).mean() for d in range(dims - 1)) / (dims - 1)
                     for k in range(1, ext[0] // 2 + 1)])
    lat.close()
    assert np.abs(got - want).max() < 1e-5
