"""Launch-shape choices of the kernels at the sizes where they change: results against plain PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(BF)


@pytest.mark.parametrize("m,n,k", [(256, 256, 64), (257, 136, 65), (768, 768, 8192), (2304, 768, 1096), (64, 256, 20000), (3072, 768, 4099)])
def test_weight_gradient_split(m, n, k):
    """Products added with red.add, whatever number of K ranges is chosen. The bound: a range is at most K / 64 blocks of
    four instructions, each of which truncates to 24 bits: 4 * K / 64 * 2**-23 of the sum of absolute values' scale."""
    from tnn_b200.ops.gemm import gemm
    torch.manual_seed(0)
    a, b = _rand(k, m), _rand(k, n)
    out = torch.ones(m, n, device="cuda")
    gemm(a, b, a_t=True, b_t=True, out=out, atomic=True)
    ref = 1 + a.double().t() @ b.double()
    err = (out.double() - ref).norm() / ref.norm()
    assert float(err) < 4 * ((k + 63) // 64 + 1) * 2.0 ** -23
