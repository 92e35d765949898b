"""Kernels that start before their predecessor has finished (programmatic dependent
launch): long chains on one stream, with nothing waiting in between, give the
results of the same calls with a synchronisation after each."""
import pytest

pytestmark = pytest.mark.gpu


def _chain(torch, ops, x, sync):
    """tensor-core product -> grouped streams -> reduce -> f32 product -> contraction, each reading the one before."""
    n = x.shape[0]
    wait = torch.cuda.synchronize if sync else (lambda: None)
    b = torch.empty(n, n, device="cuda", dtype=torch.bfloat16)
    c, s, r, f, z = [torch.empty(n, n, device="cuda") for _ in range(5)]
    out = []
    for i in range(6):
        ops.stream_group([ops.stream_op(ops.S_CAST, [x.view(-1)], b.view(-1))])
        wait()
        ops.matmul_tc([ops.tc_problem(b, b, c, alpha=1.0 / n)])
        wait()
        ops.stream_group([ops.stream_op(ops.S_BINARY, [c.view(-1), x.view(-1)], s.view(-1), op=ops.B_SUB)])
        wait()
        ops.reduce([s, c, x], r)
        wait()
        ops.matmul_f32(r, s, f, alpha=1.0 / n)
        wait()
        ops.contraction(f.view(-1), [n, n], [0, 1], s.view(-1), [n, n], [1, 2], z.view(-1), [0, 2], alpha=1.0 / n,
                        precision=i % 2)
        wait()
        out.append(z.clone())
        x = z + x
        wait()
    return torch.stack(out)


@pytest.mark.parametrize("n", [64, 200, 520, 1032])
def test_chain_of_calls(cuda, n):
    import torch
    from bbts_b200 import ops
    x = torch.randn(n, n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n))
    want = _chain(torch, ops, x, True)
    for _ in range(5):
        assert torch.equal(_chain(torch, ops, x, False), want)


@pytest.mark.parametrize("dtype", ["bf16", "f32"])
@pytest.mark.parametrize("n,split", [(256, 2), (1536, 3)])
def test_replays_back_to_back(cuda, n, split, dtype):
    """Replays of a compiled chain of single-group waves with new inputs between them, none waited for."""
    import torch
    from bbts_b200 import runtime, workloads
    rt = runtime.Runtime()
    info = workloads.bmm(rt, n=n, split=split, dtype=dtype, host=False)
    dag = rt.build_dag()
    bs, tdt = n // split, torch.bfloat16 if dtype == "bf16" else torch.float32
    g = torch.Generator(device="cuda").manual_seed(3)
    blocks = [torch.randn(bs, bs, device="cuda", generator=g).to(tdt) for _ in range(8)]
    key = (0, split - 1)
    got = [torch.empty(bs, bs, device="cuda") for _ in blocks]
    want = [torch.empty(bs, bs, device="cuda") for _ in blocks]
    torch.cuda.synchronize()
    for outs, wait in ((want, True), (got, False)):
        for x, o in zip(blocks, outs):
            dag.write(info["A"][(0, 0)], x.data_ptr(), x.numel() * x.element_size(), on_device=True)
            dag.launch()
            dag.fetch(info["C"][key], o.data_ptr(), o.numel() * 4, on_device=True)
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert not torch.equal(want[0], want[1])
