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


def test_products_on_two_streams(built_lib):
    """A handle moved to another stream while its product is still pending on the first: neither takes the
    other's lists."""
    import torch
    n = 1000
    a = [symmetric(n, 10 + i, kind) for i, kind in enumerate(("skewed", "uniform"))]
    A = [torch.from_numpy(x).cuda() for x in a]
    C = [torch.empty((n, n), device="cuda") for _ in a]
    streams = [torch.cuda.Stream() for _ in a]
    with built_lib.Handle(0) as h:
        h.maxmin_dev(A[0], A[0], C[0])  # scratch in place
        h.synchronize()
        want = [exhaustive(x, x) for x in a]
        for _ in range(5):
            for i, s in enumerate(streams):
                C[i].zero_()
                s.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(streams[0]):
                torch.cuda._sleep(2_000_000)  # about a millisecond
            for i, s in enumerate(streams):
                h.set_stream(s.cuda_stream)
                h.maxmin_dev(A[i], A[i], C[i])
            torch.cuda.synchronize()
            for c, w in zip(C, want):
                assert np.array_equal(bits(c.cpu().numpy()), bits(w))


@pytest.mark.parametrize("n", [256, 300, 1024])
def test_dpi_without_a_count_is_asynchronous_and_captured(built_lib, port, n):
    """Up to 1,024 genes nothing has to be read back: the call returns while the stream is still busy, on
    matrices the ordered form settles and on those it gives up on (NaN), and it can be captured."""
    import torch
    good = symmetric(n, n)
    bad = good.copy()
    bad[5, 7] = bad[7, 5] = np.nan
    s = torch.cuda.Stream()
    with built_lib.Handle(0) as h:
        h.set_stream(s.cuda_stream)

        def dpi(A, out, mask):
            h._check(h._L.mcpg_dpi_dev(h._h, A.data_ptr(), n, n, 0.1, out.data_ptr(), n, mask.data_ptr(), None), "dpi_dev")

        for a in (good, bad):
            A = torch.from_numpy(a).cuda()
            out, mask = torch.empty_like(A), torch.empty((n, n), dtype=torch.uint8, device="cuda")
            want, wmask = torch.empty_like(A), torch.empty_like(mask)
            h.dpi_dev(A, want, tol=0.1, mask=wmask)  # with a count
            dpi(A, out, mask)  # scratch in place, kernels loaded
            torch.cuda.synchronize()
            with torch.cuda.stream(s):
                torch.cuda._sleep(200_000_000)  # about 0.1 s
            dpi(A, out, mask)
            assert not s.query()
            torch.cuda.synchronize()
            assert torch.equal(mask, wmask) and np.array_equal(bits(out.cpu().numpy()), bits(want.cpu().numpy()))
        oo, om, _ = port.dpi(good, 0.1)
        A.copy_(torch.from_numpy(good))
        g = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(g, stream=s):
            dpi(A, out, mask)
        out.zero_()
        mask.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(mask.cpu().numpy(), om) and np.array_equal(bits(out.cpu().numpy()), bits(oo))


def test_products_of_several_threads(built_lib):
    """A handle per thread, one with rows that need a large row buffer and three with small ones: no launch
    sees another thread's buffer size."""
    import threading
    import torch
    errors = []

    def work(n, calls):
        try:
            with torch.cuda.stream(torch.cuda.Stream()), built_lib.Handle(0) as h:
                h.set_stream(torch.cuda.current_stream().cuda_stream)
                A = torch.rand((n, 256), device="cuda")
                C = torch.empty((n, n), device="cuda")
                torch.cuda.current_stream().synchronize()
                for _ in range(calls):
                    h.maxmin_dev(A, A, C)
                    h.dpi_dev(C, C, tol=0.1)
                h.synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(f"{n}: {e}")

    threads = [threading.Thread(target=work, args=a) for a in ((13000, 60), (300, 1500), (301, 1500), (257, 1500))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("call", ["maxmin", "dpi", "mcp4", "maxmin_two", "witness"])
def test_scratch_is_what_the_call_can_use(built_lib, call):
    """The transposed operand, the product, the lists and the pending outputs that the call's kind may leave
    (1/64 of the outputs, with two operands 1/4), and nothing for the forms it does not take."""
    import torch
    n = 4096
    A, B, C = (torch.rand((n, n), device="cuda") for _ in range(3))
    K = torch.empty((n, n), dtype=torch.int32, device="cuda")
    lists = n * (4 * 64 * 8 + 5 * 4)
    two = call == "maxmin_two"
    want = 2 * 4 * n * n + (1 + (call == "mcp4") + two) * lists + n * n // (4 if two else 64) * 12
    want += 4 * n * n * (call in ("mcp4", "witness"))  # M1; the witnesses
    with built_lib.Handle(0) as h:
        h.set_stream(torch.cuda.current_stream().cuda_stream)
        tiny = torch.rand((256, 256), device="cuda")
        run = {"maxmin": lambda a, b: h.maxmin_dev(a, a, C), "dpi": lambda a, b: h.dpi_dev(a, C),
               "mcp4": lambda a, b: h.mcp_dev(a, 4, M=C), "maxmin_two": lambda a, b: h.maxmin_dev(a, b, C),
               "witness": lambda a, b: h.maxmin_witness_dev(a, a, C, K)}[call]
        run(tiny, tiny.clone())  # kernels loaded
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        run(A, B)
        torch.cuda.synchronize()
        used = before - torch.cuda.mem_get_info()[0]
    assert used <= want + (8 << 20), (used, want)


def products_case(call, n):
    """(run(h, operand, outputs), the scratch the exhaustive form needs)."""
    import torch
    ld = (n + 31) // 32 * 32
    nn = 4 * n * ld
    return {
        "maxmin": (lambda h, a, o: h.maxmin_dev(a, a, o["C"]), 0),
        "mcp2": (lambda h, a, o: h.mcp_dev(a, 2, M=o["C"]), 0),
        "mcp3": (lambda h, a, o: h.mcp_dev(a, 3, M=o["C"]), nn),
        "mcp3_symmetrized": (lambda h, a, o: h.mcp_dev(a, 3, M=o["C"], symmetrize=True), 2 * nn),
        "mcp4": (lambda h, a, o: h.mcp_dev(a, 4, M=o["C"]), nn),
        "maxmins": (lambda h, a, o: h.maxmins_dev(a, M2=o["C"], M3=o["D"]), nn),
        "witness": (lambda h, a, o: h.maxmin_witness_dev(a, a, o["C"], o["D"].view(torch.int32)), 0),
    }[call]


@pytest.mark.parametrize("call", ["maxmin", "mcp2", "mcp3", "mcp3_symmetrized", "mcp4", "maxmins", "witness"])
def test_no_call_needs_the_ordered_scratch(built_lib, call):
    """From the scratch the exhaustive form needs up to all that the ordered one takes, on a new handle and on
    one whose ordered scratch fills the limit: the same bits."""
    import torch
    n = 512
    run, need = products_case(call, n)
    A = torch.from_numpy(symmetric(n, 21)).cuda()
    big = torch.from_numpy(symmetric(1024, 22)).cuda()
    o = {k: torch.zeros((n, n), device="cuda") for k in "CD"}
    big_out = torch.empty_like(big)
    with built_lib.Handle(0) as h:
        h.set_stream(torch.cuda.current_stream().cuda_stream)
        run(h, A, o)
        want = {k: v.cpu() for k, v in o.items()}
    for limit in [max(need, 1)] + [need + s for s in (1 << 20, 2 << 20, 3 << 20, 4 << 20, 64 << 20)]:
        for warm in (False, True):
            with built_lib.Handle(0) as h:
                h.set_stream(torch.cuda.current_stream().cuda_stream)
                if warm:  # 1,024 genes' ordered scratch takes most of 12 MB
                    h.maxmin_dev(big, big, big_out)
                    limit = max(limit, 12 << 20)
                h.limit_scratch(limit)
                for v in o.values():
                    v.zero_()
                run(h, A, o)
                h.synchronize()
            for k in o:
                assert torch.equal(o[k].cpu().view(torch.int32), want[k].view(torch.int32)), (limit, warm, k)
