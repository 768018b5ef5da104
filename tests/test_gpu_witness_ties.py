"""Witnesses of matrices with many equal values: the first candidate that attains each output, without the
exhaustive kernel, and where ties begin beyond the scanned candidates."""
import numpy as np
import pytest

from test_gpu_ordered_routes import h  # noqa: F401

pytestmark = pytest.mark.gpu


def check(h, a, b):  # noqa: F811
    import torch
    A = torch.from_numpy(a).cuda()
    B = A if b is a else torch.from_numpy(b).cuda()
    C = torch.empty((len(a), len(b)), device="cuda")
    K = torch.full((len(a), len(b)), -7, dtype=torch.int32, device="cuda")
    h.maxmin_witness_dev(A, B, C, K)
    stats = h.ordered_stats()
    C, K = C.cpu().numpy(), K.cpu().numpy()
    for i in range(len(a)):
        mins = np.minimum(a[i][None], b)
        top = mins.max(1)
        assert np.array_equal(C[i], top)
        # nothing attains -inf
        assert np.array_equal(K[i], np.where(top == -np.inf, -1, mins.argmax(1)))
    return stats


def tied(kind, rows, k, rng):
    if kind == "constant":
        a = np.full((rows, k), 0.5)
    elif kind == "five":
        a = rng.integers(0, 5, (rows, k)) / 4.0
    elif kind == "rare":        # one value in 100 is 1, so the first common one lies some hundreds in, or nowhere
        a = rng.random((rows, k)) < 0.01
    elif kind == "sparse":
        a = np.where(rng.random((rows, k)) < 3.0 / k, rng.random((rows, k)), 0.0)
    else:                       # "late": distinct small values first, ties in the last quarter only
        a = rng.random((rows, k)) / 8
        a[:, -(k // 4):] = 1.0
        a[::3, -(k // 4):] = 0.5
    return a.astype(np.float32)


@pytest.mark.parametrize("kind", ["constant", "five", "rare", "sparse", "late"])
@pytest.mark.parametrize("rows,cols,k", [(257, 257, 257), (300, 261, 511), (130, 260, 513), (260, 129 * 2, 700)])
def test_first_of_many_ties(h, kind, rows, cols, k):  # noqa: F811
    rng = np.random.default_rng(rows + k)
    a = tied(kind, rows, k, rng)
    check(h, a, a)
    check(h, a, tied(kind, cols, k, rng))


@pytest.mark.parametrize("rows", [8, 256])
def test_negative_infinity(h, rows):  # noqa: F811
    a = np.full((rows, 300), -np.inf, np.float32)
    b = np.zeros((300, 300), np.float32)
    a[::2, 150:] = 2.0
    check(h, a, b)
    check(h, b, b)


@pytest.mark.parametrize("kind", ["constant", "five", "sparse"])
def test_no_exhaustive_kernel(h, kind):  # noqa: F811
    """The pending witnesses stay below their list's capacity."""
    import torch
    n = 2000
    a = tied(kind, n, n, np.random.default_rng(1))
    A = torch.from_numpy(np.maximum(a, a.T)).cuda()
    C = torch.empty((n, n), device="cuda")
    K = torch.empty((n, n), dtype=torch.int32, device="cuda")

    def best(f):
        t = []
        for _ in range(6):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            f()
            e[1].record()
            torch.cuda.synchronize()
            t.append(e[0].elapsed_time(e[1]))
        return min(t)

    ordered = best(lambda: h.maxmin_witness_dev(A, A, C, K))
    s = torch.cuda.Stream()
    h.set_stream(s.cuda_stream)
    g = torch.cuda.CUDAGraph()
    K2, C2 = torch.empty_like(K), torch.empty_like(C)
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s):  # the exhaustive kernel
        h.maxmin_witness_dev(A, A, C2, K2)
    exhaustive = best(g.replay)
    h.set_stream(torch.cuda.current_stream().cuda_stream)
    assert torch.equal(K, K2) and torch.equal(C.view(torch.int32), C2.view(torch.int32))
    assert ordered < exhaustive
