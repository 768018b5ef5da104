"""The MI adjoint in more than one slab of Q: shown by the launches, with the bits of other slab sizes and forms and
the FP64 oracle's gradient."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def adjoint(M, X, G, order, limit=0):
    """dX and the number of slabs (Q, contraction and dX kernels each; before them weights, entries of the
    row-skipping form, pair sums)."""
    import torch
    dX = torch.full_like(X, np.nan)
    with M.Handle(0) as h:
        h.set_stream(torch.cuda.current_stream().cuda_stream)
        h.limit_scratch(limit)
        before = h.kernel_launches
        h.bspline_mi_bwd_dev(X, G, dX, 10, order)
        launches = h.kernel_launches - before
    return dX.cpu(), launches


def on_picked(n, pick, Gs):
    import torch
    G = np.zeros((n, n), np.float32)
    G[np.ix_(pick, pick)] = Gs
    return torch.from_numpy(G).cuda()


def test_row_skipping_slabs(built_lib, port):
    """4,700 genes x 10 bins: Q is 8.9 GB, above the one-slab limit of 8 GiB, so five slabs of up to 1,120 genes."""
    import torch
    n, m = 4700, 40
    Xh = built_lib.synth_grn(n, m, seed=11)
    X = torch.from_numpy(Xh).cuda()
    # the dense form's slabs: no room for the entries and the longer weights
    dense = 12 * n + 48 * 47040 * 4 + n * 10 * 128 * 4 + 11200 * 40 * 4 + n * 10 * 11264 * 4
    G = torch.randn((n, n), generator=torch.Generator("cuda").manual_seed(2), device="cuda")
    a, la = adjoint(built_lib, X, G, 3)
    b, lb = adjoint(built_lib, X, G, 3, dense + (2 << 20))
    assert (la, lb) == (3 + 3 * 5, 2 + 3 * 5)
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    del G, b
    pick = np.r_[0:20, 1110:1130, 4460:4490, 4690:4700]  # both sides of the slabs' edges
    Gs = np.random.default_rng(3).normal(size=(len(pick), len(pick))).astype(np.float32)
    got, launches = adjoint(built_lib, X, on_picked(n, pick, Gs), 3)
    assert launches == 3 + 3 * 5
    got = got.numpy()
    want = port.mi_bwd(Xh[pick].astype(np.float64), Gs.astype(np.float64))
    # the FP32 adjoint's tolerance elsewhere: 1e-3 of the largest entry
    assert np.abs(got[pick] - want).max() <= 1e-3 * np.abs(want).max()
    assert not got[np.setdiff1d(np.arange(n), pick)].any()


def test_dense_slabs(built_lib, port):
    """Order 4 has no row-skipping form: above 2 GiB of Q, slabs of up to 2,208 of 2,400 genes."""
    import torch
    n, m = 2400, 40
    Xh = built_lib.synth_grn(n, m, seed=12)
    X = torch.from_numpy(Xh).cuda()
    pick = np.r_[0:20, 1100:1120, 2200:2220, 2390:2400]
    Gs = np.random.default_rng(4).normal(size=(len(pick), len(pick))).astype(np.float32)
    G = on_picked(n, pick, Gs)
    a, la = adjoint(built_lib, X, G, 4)
    b, lb = adjoint(built_lib, X, G, 4, 1500 << 20)
    assert la == 2 + 3 * 2 and lb > la
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    want = port.mi_bwd(Xh[pick].astype(np.float64), Gs.astype(np.float64), 10, 4)
    assert np.abs(a.numpy()[pick] - want).max() <= 1e-3 * np.abs(want).max()
