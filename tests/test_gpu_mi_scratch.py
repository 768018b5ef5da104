"""Device scratch of the FP32 MI and its adjoint: calls that fit without the row-skipping form's
buffers run without them, with the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def up(a, b):
    return (a + b - 1) // b * b


@pytest.mark.parametrize("n,m", [(40, 64), (300, 257)])
def test_fp32_mi_within_the_dense_forms_scratch(built_lib, n, m):
    import torch
    X = torch.from_numpy(built_lib.synth_grn(n, m, seed=3)).cuda()
    MI = torch.empty((n, n), device="cuda")
    dense = up(m, 16) * up(n, 16) * 10 * 4 + 8 * n  # weights and entropies
    got = []
    for limit in (0, dense, dense + (1 << 16)):
        with built_lib.Handle(0) as h:
            h.set_stream(torch.cuda.current_stream().cuda_stream)
            h.limit_scratch(limit)
            for _ in range(2):
                MI.zero_()
                h.bspline_mi_dev(X, MI)
                got.append(MI.cpu().view(torch.int32))
    assert all(torch.equal(g, got[0]) for g in got)


def test_fp32_mi_captured_in_the_dense_forms_scratch(built_lib):
    """Scratch in place from a call of another spline order, which has no row-skipping form: a capture does not
    allocate."""
    import torch
    n, m = 64, 100
    X = torch.from_numpy(built_lib.synth_grn(n, m, seed=4)).cuda()
    MI, want = torch.empty((n, n), device="cuda"), torch.empty((n, n), device="cuda")
    s = torch.cuda.Stream()
    with built_lib.Handle(0) as h:
        h.bspline_mi_dev(X, want)
        h.synchronize()
    with built_lib.Handle(0) as h:
        h.set_stream(s.cuda_stream)
        h.bspline_mi_dev(X, MI, 10, 4)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            h.bspline_mi_dev(X, MI)
        MI.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(MI.view(torch.int32), want.view(torch.int32))


@pytest.mark.parametrize("n,m,order", [(200, 1000, 3), (200, 1000, 4), (600, 64, 3)])
def test_adjoint_within_less_scratch(built_lib, n, m, order):
    """From the scratch of one copy of the weights, one slab of Q and dW (the dense form's) down to slabs of 32
    genes, and up to what the row-skipping form takes.  Every element of Q and of the contraction is the same
    chain of operations in all of them."""
    import torch
    X = torch.from_numpy(built_lib.synth_grn(n, m, seed=6)).cuda()
    G = torch.randn((n, n), generator=torch.Generator("cuda").manual_seed(1), device="cuda")
    dX = torch.empty((n, m), device="cuda")
    w, q = 4 * up(m, 16) * up(n, 16) * 10, 4 * (up(n, 16) * 10) ** 2
    least = 4 * up(m, 16) * up(n, 16) * 10 + 4 * n * 10 * up(m, 128) + 320 * 4 * up(m, 4) + n * 10 * 384 * 4 + 12 * n
    got = []
    for limit in (0, least, (least + 2 * w + q) // 2, 2 * w + q, 3 * w + q, 6 * w + q):
        with built_lib.Handle(0) as h:
            h.set_stream(torch.cuda.current_stream().cuda_stream)
            h.limit_scratch(limit)
            for _ in range(2):
                dX.zero_()
                h.bspline_mi_bwd_dev(X, G, dX, 10, order)
                got.append(dX.cpu().view(torch.int32))
    assert all(torch.equal(g, got[0]) for g in got)


@pytest.mark.parametrize("n,m", [(2, 20), (37, 129)])
@pytest.mark.parametrize("order,launches", [(3, 6), (4, 5)])
def test_adjoint_launches(built_lib, port, n, m, order, launches):
    """Both copies of the weights come from one pass over the samples: weights, pair sums, Q, contraction, dX,
    and the entries of the row-skipping form."""
    X = built_lib.synth_grn(n, m, seed=8)
    G = np.random.default_rng(n).normal(size=(n, n)).astype(np.float32)
    with built_lib.Handle(0) as h:
        before = h.kernel_launches
        got = h.bspline_mi_bwd(X, G, 10, order)
        assert h.kernel_launches - before == launches
    want = port.mi_bwd(X.astype(np.float64), G.astype(np.float64), 10, order)
    # the FP32 adjoint's tolerance elsewhere: 1e-3 of the largest entry
    assert np.abs(got - want).max() <= 1e-3 * max(np.abs(want).max(), 1e-30)


@pytest.mark.parametrize("n,m,launches", [(1, 1, 2), (8, 48, 2), (8, 49, 3), (299, 48, 2), (299, 49, 3), (300, 32, 2),
                                          (300, 33, 3), (599, 32, 2), (600, 16, 2), (600, 17, 3)])
def test_few_samples_take_the_dense_form(built_lib, n, m, launches):
    """At the rule's edges: weights and contraction, or with entries between; the bits of the dense kernel."""
    import torch
    X = torch.from_numpy(built_lib.synth_grn(n, m, seed=9)).cuda()
    MI, want = torch.empty((n, n), device="cuda"), torch.empty((n, n), device="cuda")
    with built_lib.Handle(0) as h:
        h.set_stream(torch.cuda.current_stream().cuda_stream)
        before = h.kernel_launches
        h.bspline_mi_dev(X, MI)
        assert h.kernel_launches - before == launches
    rc = built_lib.lib().mcpg_bspline_mi_fp32_noalloc(X.data_ptr(), n, m, m, 10, 3, want.data_ptr(), n, None,
                                                      torch.cuda.current_stream().cuda_stream)
    assert rc == built_lib.OK
    assert torch.equal(MI.view(torch.int32), want.view(torch.int32))
