"""What the kernels' host side answers in a process that has no CUDA device."""
import pytest
import torch

pytestmark = pytest.mark.skipif(torch.cuda.is_available(), reason="a CUDA device is there")


def test_no_kernel_has_run_so_none_gave_up_a_wait():
    from titan_b200 import kernels as K
    assert K.wait_errors() == {}


@pytest.mark.parametrize("N,Kd,M", [(5632, 1024, 8), (2048, 2048, 32), (130, 512, 1)])
def test_products_of_whole_sums_take_one_slice_where_no_cluster_is_placed(N, Kd, M):
    from titan_b200 import kernels as K
    assert K.tlib().tb_gemm_tc_normed_slices(N, Kd, K.EPI_SWIGLU, M, 0) == 1
