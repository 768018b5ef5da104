"""FP32 MI, 10 bins / order 3, of genes with NaN or infinite samples: the row-skipping form gives the dense kernel's
bits, those genes' pairs included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(40, 130), (300, 257), (700, 64)])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_irregular_genes_equal_the_dense_kernel(built_lib, n, m, bad):
    import torch
    X = built_lib.synth_grn(n, m, seed=13)
    for g, s in ((0, 0), (n // 2, m // 3), (n - 1, m - 1)):
        X[g, s] = bad
    X = torch.from_numpy(X).cuda()
    MI, want = torch.empty((n, n), device="cuda"), torch.empty((n, n), device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    with built_lib.Handle(0) as h:
        h.set_stream(stream)
        before = h.kernel_launches
        h.bspline_mi_dev(X, MI)
        assert h.kernel_launches - before == 3  # weights, entries, contraction
    rc = built_lib.lib().mcpg_bspline_mi_fp32_noalloc(X.data_ptr(), n, m, m, 10, 3, want.data_ptr(), n, None, stream)
    assert rc == built_lib.OK
    torch.cuda.synchronize()
    assert torch.equal(torch.isnan(MI), torch.isnan(want))
    number = ~torch.isnan(want)
    assert torch.equal(MI[number].view(torch.int32), want[number].view(torch.int32))
