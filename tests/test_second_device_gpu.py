"""Several GPUs in one process: what a launch needs is set up on each of them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 3, 37, 100, 300, 2000])
def test_products_on_every_device(M):
    """One row, few rows, single-CTA tiles and CTA pairs, whose shared memory a device has to grant each by itself."""
    from megalodon_b200.ops import cuda_ops
    if torch.cuda.device_count() < 2:
        pytest.skip("needs 2 GPUs")
    for dev in range(torch.cuda.device_count()):
        torch.manual_seed(M)
        x = torch.randn(M, 1024, device=f"cuda:{dev}").bfloat16()
        w = (torch.randn(512, 1024, device=f"cuda:{dev}") / 32).bfloat16()
        y, _ = cuda_ops.gemm(x, w)
        ref = x.double() @ w.double().t()
        assert ((y.double() - ref).norm() / ref.norm()).item() < 2.0 ** -8
    cuda_ops.check_kernel_errors()
