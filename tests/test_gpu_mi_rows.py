"""FP32 B-spline MI, 10 bins / order 3 (three weight rows per sample): edges of its gene tiles,
sample chunks and CTA widths against the FP64 oracle, and its bits against the all-rows form that an
irregular sample (NaN input) selects."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(1, 1), (2, 3), (31, 63), (32, 64), (33, 65), (97, 129), (190, 64), (260, 191),
                                 (401, 100)])
def test_sizes_match_the_fp64_oracle(gpu, built_lib, port, n, m):
    X = built_lib.synth_grn(n, m, seed=n * 1000 + m)
    got, H = gpu.bspline_mi(X, 10, 3, "fp32", return_H=True)
    want = port.bspline_mi(X.astype(np.float64))
    assert np.array_equal(got, got.T)
    # float sums of <= 191 samples and 100 float terms: the bound the FP32 form is held to elsewhere
    assert np.abs(got - want).max() <= 2e-5
    assert H.shape == (n,)


@pytest.mark.parametrize("n,m", [(40, 130), (300, 257)])
def test_same_bits_as_all_rows(gpu, built_lib, n, m):
    """One gene with a NaN sample makes every row of every pair be multiplied; the other genes' pairs
    must not change by a bit."""
    X = built_lib.synth_grn(n, m, seed=7)
    clean = gpu.bspline_mi(X, 10, 3, "fp32")
    X2 = np.concatenate([X, X[:1]])
    X2[n, m // 2] = np.nan
    mixed = gpu.bspline_mi(X2, 10, 3, "fp32")
    assert np.array_equal(mixed[:n, :n].view(np.uint32), clean.view(np.uint32))


def test_constant_and_two_valued_genes(gpu, port):
    """Samples on the ends of the range (one nonzero weight) and genes without a range."""
    rng = np.random.default_rng(3)
    X = rng.integers(0, 2, (37, 70)).astype(np.float32)
    X[5] = 0.5
    got = gpu.bspline_mi(X, 10, 3, "fp32")
    assert np.abs(got - port.bspline_mi(X.astype(np.float64))).max() <= 2e-5
