"""The MI adjoint's contraction at the edges of its 128 x 128 tiles and 16-deep slices, with the FP64
oracle, and its slab form (Q larger than its buffer) against the one-slab form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,bins,order", [(2, 5, 10, 3), (13, 127, 10, 3), (26, 128, 10, 3), (39, 129, 10, 3),
                                            (64, 64, 2, 1), (35, 257, 12, 4), (19, 130, 10, 2)])
def test_tile_edges_vs_fp64(gpu, port, built_lib, n, m, bins, order):
    rng = np.random.default_rng(n * m)
    X = built_lib.synth_grn(n, m, seed=n + 3 * m)
    G = rng.normal(size=(n, n)).astype(np.float32)
    got = gpu.bspline_mi_bwd(X, G, bins, order)
    want = port.mi_bwd(X.astype(np.float64), G.astype(np.float64), bins, order)
    # the FP32 adjoint's tolerance elsewhere: 1e-3 of the largest entry
    assert np.abs(got - want).max() <= 1e-3 * max(np.abs(want).max(), 1e-30)


def test_slabs_equal_one_slab(gpu, built_lib):
    """4,600 genes x 10 bins exceed the one-slab buffer.  With a gradient on 200 of them, those genes
    get what they get alone and the others exactly zero."""
    n, m = 4600, 40
    rng = np.random.default_rng(1)
    X = built_lib.synth_grn(n, m, seed=5)
    pick = np.r_[0:100, 4500:4600]
    Gs = rng.normal(size=(200, 200)).astype(np.float32)
    G = np.zeros((n, n), np.float32)
    G[np.ix_(pick, pick)] = Gs
    got = gpu.bspline_mi_bwd(X, G)
    alone = gpu.bspline_mi_bwd(X[pick], Gs)
    rest = np.setdiff1d(np.arange(n), pick)
    assert not got[rest].any()
    # same chains of multiply-adds with zeros between them; only the pair sums' order differs
    assert np.abs(got[pick] - alone).max() <= 1e-5 * np.abs(alone).max()
