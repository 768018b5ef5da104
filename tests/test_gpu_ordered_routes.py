"""Which way the ordered max-min products and DPI go (their device counters), with the bits of the
exhaustive definition on each."""
import numpy as np
import pytest

from test_gpu_maxmin_ranked import bits, data, exhaustive

pytestmark = pytest.mark.gpu


@pytest.fixture
def h(built_lib):
    import torch
    with built_lib.Handle(0) as hh:
        hh.set_stream(torch.cuda.current_stream().cuda_stream)
        yield hh


def product(h, a, b):
    """C = a (x) b (b None: a (x) a) on the device, and how it went."""
    import torch
    A = torch.from_numpy(a).cuda()
    B = A if b is None else torch.from_numpy(b).cuda()
    C = torch.empty((A.shape[0], B.shape[0]), device="cuda")
    h.maxmin_dev(A, B, C)
    return C.cpu().numpy(), h.ordered_stats()


def gave_up(s):
    return s["nan"] or s["pending"] > s["pending_cap"] or (s["full_cap"] and s["full"] > s["full_cap"])


def test_too_small_or_too_narrow(h):
    a = data("uniform", 300, 255, np.random.default_rng(0))
    assert product(h, a, None)[1]["enqueued"] == 0
    b = data("uniform", 7, 300, np.random.default_rng(0))
    assert product(h, b, data("uniform", 300, 300, np.random.default_rng(1)))[1]["enqueued"] == 0


@pytest.mark.parametrize("kind", ["uniform", "skewed", "signed"])
def test_settled_by_the_lists(h, kind):
    a = data(kind, 600, 700, np.random.default_rng(3))
    c, s = product(h, a, None)
    assert s["enqueued"] and not gave_up(s)
    assert np.array_equal(bits(c), bits(exhaustive(a, a)))


def test_nan_gives_up(h):
    a = data("uniform", 300, 300, np.random.default_rng(4))
    a[5, 6] = np.nan
    assert product(h, a, None)[1]["nan"]


def test_pending_outputs_read_whole_rows_without_the_other_lists(h):
    """500 candidates: reading a column's pending outputs is cheaper than building its list."""
    import torch
    n, t = 2000, 500
    rng = np.random.default_rng(1)
    a = data("skewed", n, n, rng)
    a = np.maximum(a, a.T)
    tfs = np.full(n, -np.inf, np.float32)
    rows = np.sort(rng.permutation(n)[:t])
    tfs[rows] = np.inf
    M1 = torch.empty((t, n), device="cuda")
    h.maxmins_tf_dev(torch.from_numpy(a).cuda(), tfs, M1=M1)
    s = h.ordered_stats()
    assert t * n // 256 < s["pending"] and s["lists_above"] == 0 and not gave_up(s)
    assert np.array_equal(bits(M1.cpu().numpy()), bits(exhaustive(a[np.ix_(rows, rows)], np.ascontiguousarray(a[:, rows]))))


def test_the_other_operands_lists_settle_what_pends(h):
    """A tenth of the owners have large values everywhere: nothing in their lists tells the columns apart."""
    rng = np.random.default_rng(5)
    a, b = data("uniform", 2000, 2000, rng), data("uniform", 1900, 2000, rng)
    a[::10] = 1e6 + rng.random((200, 2000), dtype=np.float32)
    c, s = product(h, a, b)
    assert s["lists_above"] < s["pending"] <= s["pending_cap"] and s["full"] < s["full_cap"] and not gave_up(s)
    assert np.array_equal(bits(c), bits(exhaustive(a, b)))


def test_gives_up_where_no_list_settles(h):
    """Rising rows against falling ones: half of either row lies above the maximum of the minima."""
    rng = np.random.default_rng(6)
    k = 2000
    ramp = np.arange(k, dtype=np.float32) / k
    a, b = data("uniform", 2000, k, rng), data("uniform", 1900, k, rng)
    a[:1000] = ramp + 1e-4 * rng.random((1000, 1), dtype=np.float32)
    b[:700] = 1 - ramp + 1e-4 * rng.random((700, 1), dtype=np.float32)
    c, s = product(h, a, b)
    assert s["pending"] <= s["pending_cap"] and s["full"] > s["full_cap"]
    assert np.array_equal(bits(c), bits(exhaustive(a, b)))
