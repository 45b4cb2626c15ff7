"""Device memory of a plan of many small replicas (GPU)."""
import pytest

pytestmark = pytest.mark.gpu


def test_many_small_replicas():
    # 4096 grids of 12 x 6: 10 planes and 3 half spectra are 33 MB, and the partial
    # sums of their kernels are to be small beside them
    import torch
    from mgkmc_b200.linear_elastic_simulator import Ls2dBatch
    Ls2dBatch([(12, 6)])
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    plan = Ls2dBatch([(12, 6)] * 4096)
    used = before - torch.cuda.mem_get_info()[0]
    assert plan is not None and used < 64 << 20
