"""FP32 products take scratch that the SIMT kernels did not: on a device that is nearly full,
what fitted without it still runs. The device is filled from the host, but for a stated rest."""
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


class _Filled:
    """All device memory but `rest` bytes taken (in whole 2 MiB pieces)."""

    def __init__(self, torch, lib, rest):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        lib.bbx_trim_scratch()
        free = torch.cuda.mem_get_info()[0]
        assert free > rest
        self.torch = torch
        self.block = torch.empty((free - rest) >> 21 << 21, dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.torch.cuda.synchronize()
        self.block = None
        self.torch.cuda.empty_cache()


def _simt(torch, ops, a, b):
    c = torch.empty(N, N, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):  # a captured call runs the SIMT kernel
        ops.matmul_f32(a, b, c)
    graph.replay()
    torch.cuda.synchronize()
    return c


# nine operands' planes (864 MiB) and eight results (512): everything fits; the arena fits but not the results after
# it; not even the arena
@pytest.mark.parametrize("rest,planes", [(2 << 30, True), (1100 << 20, False), (700 << 20, False)])
def test_compiled_list_without_room_for_planes(T, rest, planes):
    torch, ops, runtime, lib = T
    rt = runtime.Runtime()
    g = torch.Generator(device="cuda").manual_seed(1)
    x = [torch.randn(N, N, device="cuda", generator=g) for _ in range(9)]
    for t, v in enumerate(x):
        rt.put_dense(t, v.cpu().numpy())
    mm = rt.impl("matrix_mult", ["dense"] * 2, ["dense"])
    for j in range(8):
        rt.apply(mm, [0, 1 + j], [100 + j])
    simt, got = _simt(torch, ops, x[0], x[8]), torch.empty(N, N, device="cuda")
    tc = torch.empty(N, N, device="cuda")
    ops.matmul_f32(x[0], x[8], tc)
    with _Filled(torch, lib, rest):
        dag = rt.build_dag()
        dag.launch()
        dag.fetch(107, got.data_ptr(), BLOCK, on_device=True)
    assert torch.equal(got, tc if planes else simt)
    dag.close()
    rt.close()


def test_commands_whose_scratch_is_still_queued(T):
    """Products one after another, nothing waited for: a block's allocation that the queued products'
    scratch stands in the way of waits for it."""
    torch, ops, runtime, lib = T
    rt = runtime.Runtime()
    g = torch.Generator(device="cuda").manual_seed(2)
    a, b = torch.randn(N, N, device="cuda", generator=g), torch.randn(N, N, device="cuda", generator=g)
    rt.put_dense(0, a.cpu().numpy())
    rt.put_dense(1, b.cpu().numpy())
    mm = rt.impl("matrix_mult", ["dense"] * 2, ["dense"])
    count = 8
    for j in range(count):
        rt.apply(mm, [0, 1], [100 + j])
    simt = _simt(torch, ops, a, b)
    with _Filled(torch, lib, count * BLOCK + PLANES):  # the blocks, and half of one product's scratch
        rt.run()
    ref = a.double() @ b.double()
    for j in range(count):  # each on the tensor cores or, without room for its planes, on the SIMT kernel
        got = torch.from_numpy(rt.get_dense(100 + j)).cuda()
        assert torch.equal(got, simt) or ((got.double() - ref).norm() < 1e-6 * ref.norm())
    rt.close()


def test_other_allocators_get_the_scratch_back(T):
    torch, ops, runtime, lib = T
    a, b, c = (torch.randn(N, N, device="cuda") for _ in range(3))
    ops.matmul_f32(a, b, c)  # loads the kernels
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
