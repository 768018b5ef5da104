"""The two products of the MCP3 gradient in one call: the bits and witnesses of the two calls."""
import numpy as np
import pytest

from test_gpu_maxmin_ranked import data
from test_gpu_ordered_routes import h  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["skewed", "signed", "ties", "zeros", "inf", "chain"])
@pytest.mark.parametrize("n,pitch", [(1, 1), (255, 255), (256, 256), (257, 259), (700, 700)])
def test_equal_to_two_calls(h, built_lib, kind, n, pitch):  # noqa: F811
    import torch
    if n < 4 and kind == "inf":
        pytest.skip("needs four rows")
    a = data(kind, n, n, np.random.default_rng(n))
    A = torch.from_numpy(np.maximum(a, a.T)).cuda()
    M = [torch.full((n, pitch), -5.0, device="cuda")[:, :n] for _ in range(4)]
    K = [torch.full((n, pitch), -7, dtype=torch.int32, device="cuda")[:, :n] for _ in range(4)]
    h.maxmin_witness_dev(A, A, M[0], K[0])
    h.maxmin_witness_dev(A, M[0], M[1], K[1])
    rc = built_lib.lib().mcpg_maxmins_witness_dev(
        h._h, A.data_ptr(), n, n, M[2].data_ptr(), pitch, K[2].data_ptr(), pitch, M[3].data_ptr(), pitch,
        K[3].data_ptr(), pitch)
    assert rc == built_lib.OK
    for one, both in ((0, 2), (1, 3)):
        assert torch.equal(M[one].contiguous().view(torch.int32), M[both].contiguous().view(torch.int32))
        assert torch.equal(K[one], K[both])
