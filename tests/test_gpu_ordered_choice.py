"""Two-operand max-min products choose on the device which operand's rows own the lists: the bits of the
exhaustive definition whichever it is, and no give-up with the operands the other way round."""
import numpy as np
import pytest

from test_gpu_maxmin_ranked import bits, data, exhaustive
from test_gpu_ordered_routes import gave_up, h, product  # noqa: F401

pytestmark = pytest.mark.gpu


def similarity(n, rng):
    a = data("skewed", n, n, rng)
    a = np.maximum(a, a.T)
    np.fill_diagonal(a, 0.0)
    return a


@pytest.mark.parametrize("n", [256, 513, 1500])
def test_own_product_first(h, n):  # noqa: F811
    """M1 (x) A: M1's rows have no pronounced largest values, and the product used to give up."""
    a = similarity(n, np.random.default_rng(n))
    m1, _ = product(h, a, None)
    for x, y in ((m1, a), (a, m1)):
        c, s = product(h, x, y)
        assert s["enqueued"] and not gave_up(s)
        assert np.array_equal(bits(c), bits(exhaustive(x, y)))


# flat: nearly equal values in every row, so only the other operand's lists settle
@pytest.mark.parametrize("rows,cols,k", [(8, 256, 256), (256, 1000, 300), (1000, 257, 301), (700, 2100, 1030),
                                         (2100, 384, 515)])
@pytest.mark.parametrize("flat", ["first", "second", "neither", "both"])
def test_rectangles(h, rows, cols, k, flat):  # noqa: F811
    rng = np.random.default_rng(rows + k)
    a, b = data("skewed", rows, k, rng), data("skewed", cols, k, rng)
    top = np.float32(2 * max(a.max(), b.max()))
    if flat in ("first", "both"):
        a = top + rng.random((rows, k), dtype=np.float32)
    if flat in ("second", "both"):
        b = top + rng.random((cols, k), dtype=np.float32)
    c, s = product(h, a, b)
    assert s["enqueued"]
    assert np.array_equal(bits(c), bits(exhaustive(a, b)))
    if flat in ("first", "second"):
        assert not gave_up(s)


def test_neither_operand_settles(h):  # noqa: F811
    """Rising rows against falling ones: the exhaustive kernel runs."""
    rng = np.random.default_rng(6)
    k = 1200
    ramp = np.arange(k, dtype=np.float32) / k
    a = ramp + 1e-4 * rng.random((600, 1), dtype=np.float32)
    b = 1 - ramp + 1e-4 * rng.random((500, 1), dtype=np.float32)
    c, s = product(h, a.astype(np.float32), b.astype(np.float32))
    assert gave_up(s)
    assert np.array_equal(bits(c), bits(exhaustive(a.astype(np.float32), b.astype(np.float32))))


@pytest.mark.parametrize("first,second", [(True, False), (False, True)])
def test_nan_in_either_operand(h, first, second):  # noqa: F811
    import torch
    rng = np.random.default_rng(8)
    a, b = data("uniform", 300, 400, rng), data("uniform", 500, 400, rng)
    b += np.float32(1.0)
    (a if first else b)[17, 399] = np.nan
    for x, y in ((a, b), (b, a)):
        c, s = product(h, x, y)
        assert s["nan"]
        X, Y = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
        out = torch.empty(c.shape, device="cuda")
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        h.set_stream(stream.cuda_stream)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):  # the exhaustive kernel
            h.maxmin_dev(X, Y, out)
        g.replay()
        torch.cuda.synchronize()
        h.set_stream(torch.cuda.current_stream().cuda_stream)
        assert np.array_equal(bits(c), bits(out.cpu().numpy()))


@pytest.mark.parametrize("rows,cols,k", [(300, 300, 300), (259, 1100, 400), (1100, 260, 401)])
@pytest.mark.parametrize("swap", [False, True])
def test_witnesses(h, rows, cols, k, swap):  # noqa: F811
    """The first candidate that attains the product, whichever operand owns; values on a grid tie often."""
    import torch
    rng = np.random.default_rng(cols)
    a = np.floor(100 * rng.random((rows, k), dtype=np.float32))
    b = 50 + np.floor(1000 * rng.random((cols, k), dtype=np.float32))
    if swap:
        a, b = b, a
    A, B = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    C = torch.empty((len(a), len(b)), device="cuda")
    K = torch.empty((len(a), len(b)), dtype=torch.int32, device="cuda")
    h.maxmin_witness_dev(A, B, C, K)
    assert not gave_up(h.ordered_stats())
    for i in range(0, len(a), 37):
        mins = np.minimum(a[i][None], b)
        assert np.array_equal(C[i].cpu().numpy(), mins.max(1))
        assert np.array_equal(K[i].cpu().numpy(), mins.argmax(1))


def test_general_mask(h):  # noqa: F811
    import torch
    n = 300
    rng = np.random.default_rng(2)
    a = similarity(n, rng)
    m1, _ = product(h, a, None)
    mask = np.linspace(0.01, float(m1.max()), n).astype(np.float32)
    for x, y in ((m1, a), (a, m1)):
        got = h.maxmin_masked(np.ascontiguousarray(x), np.ascontiguousarray(y), mask)
        assert np.array_equal(bits(got), bits(exhaustive(np.minimum(x, mask), y)))
