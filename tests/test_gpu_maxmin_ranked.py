"""The max-min products with ordered candidates (from 256 rows and candidates up) against the
exhaustive definition, bit for bit: tile and list edges, inputs on which the ordered form gives up
(ties, NaN), both layouts of an API call, and stream capture."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def keys(a):
    """Order-preserving integers of float32 (-0 below +0): max.f32 / min.f32 order for NaN-free data."""
    u = np.ascontiguousarray(a, np.float32).view(np.int32)
    return u ^ ((u >> 31) & 0x7FFFFFFF)


def exhaustive(A, B):
    a, b = keys(A), keys(B)
    out = np.empty((A.shape[0], B.shape[0]), np.int32)
    for i in range(A.shape[0]):
        out[i] = np.minimum(a[i][None, :], b).max(1)
    return (out ^ ((out >> 31) & 0x7FFFFFFF)).view(np.float32)


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def data(kind, rows, k, rng):
    if kind == "uniform":
        a = rng.random((rows, k))
    elif kind == "skewed":      # rows of very different strength, as hubs beside isolated genes
        a = rng.random((rows, k)) ** 8 * np.exp(2.0 * rng.standard_normal((rows, 1)))
    elif kind == "signed":
        a = rng.standard_normal((rows, k))
    elif kind == "ties":        # five values: the lists cannot separate them
        a = rng.integers(0, 5, (rows, k)) / 4.0
    elif kind == "zeros":       # +0, -0 and a few others
        a = np.where(rng.random((rows, k)) < 0.98, rng.choice([0.0, -0.0], (rows, k)), rng.standard_normal((rows, k)))
    elif kind == "constant":
        a = np.full((rows, k), 0.25)
    elif kind == "chain":       # min(i, k): every candidate beyond the output's own counts
        a = np.minimum(np.arange(rows)[:, None], np.arange(k)[None, :]) + 0.5
    else:                       # infinities
        a = rng.random((rows, k))
        a[rng.random((rows, k)) < 0.05] = np.inf
        a[rng.random((rows, k)) < 0.05] = -np.inf
        a[3] = -np.inf
    return a.astype(np.float32)


KINDS = ["uniform", "skewed", "signed", "ties", "zeros", "constant", "chain", "inf"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("rows,cols,k", [(256, 256, 256), (257, 259, 1021), (9, 384, 300), (8, 257, 2049)])
def test_products_equal_the_exhaustive_form(gpu, kind, rows, cols, k):
    rng = np.random.default_rng(rows * 7 + k + KINDS.index(kind))
    A, B = data(kind, rows, k, rng), data(kind, cols, k, rng)
    assert np.array_equal(bits(gpu.maxmin(A, B)), bits(exhaustive(A, B)))
    assert np.array_equal(bits(gpu.maxmin(B)), bits(exhaustive(B, B)))  # symmetric form, rectangular operand


@pytest.mark.parametrize("where", ["A", "B"])
def test_nan_operands_take_the_exhaustive_form(gpu, where):
    rng = np.random.default_rng(5)
    A, B = rng.random((300, 320)).astype(np.float32), rng.random((290, 320)).astype(np.float32)
    (A if where == "A" else B)[7, ::3] = np.nan
    want = np.empty((300, 290), np.float32)
    for i in range(300):
        want[i] = np.fmax.reduce(np.fmin(A[i][None, :], B), axis=1)
    assert np.array_equal(bits(gpu.maxmin(A, B)), bits(want))


@pytest.mark.parametrize("n", [255, 256, 301])
@pytest.mark.parametrize("kind", ["skewed", "ties"])
def test_ensemble_chain(gpu, n, kind):
    """M1, M2 = A (x) M1, M3 = M1 (x) M1 and one ratio, on padded device views."""
    import torch
    rng = np.random.default_rng(n)
    A = data(kind, n, n, rng)
    A = np.maximum(A, A.T)
    big = torch.zeros((n, n + 5), device="cuda")
    big[:, 1:n + 1] = torch.from_numpy(A).cuda()
    out = {k: torch.full((n, n + 3), -1.0, device="cuda") for k in ("M1", "M2", "M3", "R3")}
    gpu.maxmins_dev(big[:, 1:n + 1], **{k: v[:, :n] for k, v in out.items()})
    gpu.synchronize()
    M1 = exhaustive(A, A)
    want = {"M1": M1, "M2": exhaustive(A, M1), "M3": exhaustive(M1, M1)}
    for k, w in want.items():
        assert np.array_equal(bits(out[k][:, :n].cpu().numpy()), bits(w)), k
        assert (out[k][:, n:] == -1.0).all()
    assert np.array_equal(bits(out["R3"][:, :n].cpu().numpy()), bits(gpu.ratio(A, want["M2"])))


@pytest.mark.parametrize("warm", [False, True])
def test_products_under_stream_capture(built_lib, warm):
    """With its scratch in place the ordered form is captured; a first call inside a capture, which
    cannot allocate, is captured as the exhaustive form."""
    import torch
    rng = np.random.default_rng(11)
    A = torch.from_numpy(data("skewed", 320, 320, rng)).cuda()
    C = torch.empty((320, 320), device="cuda")
    s = torch.cuda.Stream()
    h = built_lib.Handle(0)
    try:
        h.set_stream(s.cuda_stream)
        torch.cuda.synchronize()
        if warm:
            h.maxmin_dev(A, A, C)
            torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            h.maxmin_dev(A, A, C)
        for _ in range(2):
            A.copy_(torch.from_numpy(data("skewed", 320, 320, rng)))
            C.zero_()
            g.replay()
            torch.cuda.synchronize()
            a = A.cpu().numpy()
            assert np.array_equal(bits(C.cpu().numpy()), bits(exhaustive(a, a)))
    finally:
        h.close()


@pytest.mark.parametrize("n,tol", [(256, 0.1), (301, 0.0), (517, 0.15), (300, 1.0)])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("symmetric", [True, False])
def test_dpi_equals_the_reference_loop(gpu, port, kind, n, tol, symmetric):
    rng = np.random.default_rng(n + KINDS.index(kind))
    A = data(kind, n, n, rng)
    if symmetric:
        A = np.maximum(A, A.T)
    with np.errstate(all="ignore"):
        out, mask, removed = gpu.dpi(A, tol, want_mask=True)
        oo, om, orem = port.dpi(A, tol)
    # at tol = 1 a zero entry's threshold is 0 * inf = NaN: the library keeps such an entry (as its product form
    # does), the reference's loop clears it; it is a zero of either sign in both
    defined = slice(None) if tol < 1.0 else A != 0.0
    assert np.array_equal(mask[defined], om[defined])
    assert np.array_equal(bits(out)[defined], bits(oo)[defined])
    assert removed == orem


def test_dpi_on_a_nan_matrix_takes_the_product_form(gpu):
    """The deletions of a matrix with NaN entries outside some pairs' rows: those pairs decide as without."""
    rng = np.random.default_rng(2)
    n = 300
    A = data("skewed", n, n, rng)
    A = np.maximum(A, A.T)
    B = np.zeros((n + 1, n + 1), np.float32)
    B[:n, :n] = A
    B[n, 1:n:2] = B[1:n:2, n] = np.nan
    clean, cmask, _ = gpu.dpi(A, 0.1, want_mask=True)
    out, mask, _ = gpu.dpi(B, 0.1, want_mask=True)
    even = np.arange(0, n, 2)  # rows without a NaN: the extra gene adds min(0, 0) as a candidate only
    pos = A[np.ix_(even, even)] > 0
    assert np.array_equal(mask[np.ix_(even, even)][pos], cmask[np.ix_(even, even)][pos])
    assert np.array_equal(out[np.ix_(even, even)][pos], clean[np.ix_(even, even)][pos])


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("rows,cols,k", [(256, 256, 256), (301, 260, 517), (8, 300, 1030)])
def test_witnesses_equal_the_first_attaining_candidate(gpu, kind, rows, cols, k):
    rng = np.random.default_rng(rows + k + KINDS.index(kind))
    A, B = data(kind, rows, k, rng), data(kind, cols, k, rng)
    for X, Y, args in ((A, B, (A, B)), (B, B, (B,))):
        C, K = gpu.maxmin_witness(*args)
        for i in range(X.shape[0]):
            v = np.minimum(X[i][None, :], Y)
            first = v.argmax(1)  # the first of equal values
            value = v[np.arange(Y.shape[0]), first]
            want = np.where(value == -np.inf, -1, first)
            assert np.array_equal(K[i], want), i
            assert np.array_equal(C[i], value), i


def test_dpi_thresholds_at_rounding_ties(gpu, port):
    """Entries over the float range, powers of two and their neighbours, where the product's rounding is
    decided in its last bits; and a matrix large enough for the symmetry check."""
    rng = np.random.default_rng(4)
    n = 300
    e = np.exp2(rng.integers(-40, 30, (n, n)).astype(np.float32)) * (1 + rng.integers(-3, 4, (n, n)) * np.float32(2.0 ** -23))
    A = np.maximum(e, e.T).astype(np.float32)
    for tol in (0.1, 0.2, 0.25, 0.5, 1.0 - 2.0 ** -20):
        out, mask, removed = gpu.dpi(A, tol, want_mask=True)
        oo, om, orem = port.dpi(A, tol)
        assert np.array_equal(mask, om) and np.array_equal(bits(out), bits(oo)) and removed == orem


@pytest.mark.parametrize("symmetric", [True, False])
def test_dpi_above_the_symmetry_check(gpu, port, symmetric):
    rng = np.random.default_rng(8)
    n = 4100
    A = (rng.random((n, n), dtype=np.float32) ** 4) * np.exp(rng.standard_normal((n, 1))).astype(np.float32)
    if symmetric:
        A = np.maximum(A, A.T)
    out, mask, _ = gpu.dpi(A, 0.1, want_mask=True)
    rows = np.r_[0:20, 2000:2020, n - 20:n].astype(np.int64)
    oo, om, _ = port.dpi_rows(A, rows, 0.1)
    assert np.array_equal(mask[rows], om)
    assert np.array_equal(bits(out[rows]), bits(oo))
