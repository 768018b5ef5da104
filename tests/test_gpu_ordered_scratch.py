"""The ordered max-min form's device scratch: captured graphs, streams, allocation failures and
what a call waits for."""
import numpy as np
import pytest

from test_gpu_maxmin_ranked import bits, data, exhaustive

pytestmark = pytest.mark.gpu


def symmetric(n, seed, kind="skewed"):
    a = data(kind, n, n, np.random.default_rng(seed))
    return np.maximum(a, a.T)


@pytest.mark.parametrize("close", [False, True])
def test_captured_products_outlive_the_scratch(built_lib, close):
    """Graphs of products on aligned operands, captured with the scratch in place: replayed after larger
    calls have replaced it, and after the handle is gone."""
    import torch
    n = 320
    A = torch.from_numpy(symmetric(n, 1)).cuda()
    o = {k: torch.empty((n, n), device="cuda") for k in ("C", "W", "M", "R", "M1", "M2", "M3")}
    K = torch.empty((n, n), dtype=torch.int32, device="cuda")
    big = torch.rand((1500, 1500), device="cuda")
    big_out = torch.empty_like(big)
    s = torch.cuda.Stream()
    h = built_lib.Handle(0)

    def calls():
        h.maxmin_dev(A, A, o["C"])
        h.maxmin_witness_dev(A, A, o["W"], K)
        h.mcp_dev(A, 2, M=o["M"], R=o["R"])
        h.maxmins_dev(A, M1=o["M1"], M2=o["M2"], M3=o["M3"])

    h.set_stream(s.cuda_stream)
    torch.cuda.synchronize()
    calls()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        before = h.kernel_launches
        calls()
        launches = h.kernel_launches - before
    assert launches == 6  # one exhaustive kernel per product
    h.maxmins_dev(big, M3=big_out)  # grows every buffer
    h.maxmin_witness_dev(big, big, big_out, torch.empty((1500, 1500), dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    if close:
        h.close()
    for seed in (2, 3):
        a = symmetric(n, seed)
        A.copy_(torch.from_numpy(a))
        for v in o.values():
            v.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        m1 = exhaustive(a, a)
        want = {"C": m1, "W": m1, "M": m1, "M1": m1, "M2": exhaustive(a, m1), "M3": exhaustive(m1, m1)}
        for k, w in want.items():
            assert np.array_equal(bits(o[k].cpu().numpy()), bits(w)), k
    h.close()
