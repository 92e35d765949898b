"""FP32 products take scratch that the SIMT kernels did not: on a device that is nearly full,
what fitted without it still runs."""
import pytest

pytestmark = pytest.mark.gpu

N = 4096
BLOCK = 4 * N * N   # one f32 block
PLANES = 6 * N * N  # its planes


@pytest.fixture(scope="module")
def T(cuda):
    import torch
    from bbts_b200 import lib, ops, runtime
    assert lib.bbx_matmul_f32_route(N, N, N, 1) == 1
    return torch, ops, runtime, lib


def test_other_allocators_get_the_scratch_back(T):
    torch, ops, runtime, lib = T
    a, b, c = (torch.randn(N, N, device="cuda") for _ in range(3))
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    lib.bbx_trim_scratch()
    before = torch.cuda.mem_get_info()[0]
    ops.matmul_f32(a, b, c)
    torch.cuda.synchronize()
    kept = before - torch.cuda.mem_get_info()[0]
    assert 0 < kept <= 512 << 20
    lib.bbx_trim_scratch()
    assert torch.cuda.mem_get_info()[0] == before
