"""What the kernels' host side answers in a process that has no CUDA device."""
import pytest
import torch

pytestmark = pytest.mark.skipif(torch.cuda.is_available(), reason="a CUDA device is there")


def test_no_kernel_has_run_so_none_gave_up_a_wait():
    from titan_b200 import kernels as K
    assert K.wait_errors() == {}
