"""The 2-SM pair of e4m3 operands (taken by the size rule for K-major operands and
long K): exact integer products at the edges of its 256 x 256 tiles and its
128-deep K steps, grouped, and against the 1-SM tile's bits."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,count", [(4096, 4096, 1536, 1), (2064, 1040, 1552, 4), (272, 4112, 2064, 5),
                                         (256, 256, 4096, 150)])
def test_e4m3_pair_integer_exact(cuda, m, n, k, count):
    import torch
    from bbts_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(m + k)
    a = [torch.randint(-4, 5, (m, k), device="cuda", generator=g).float() for _ in range(count)]
    b = [torch.randint(-4, 5, (n, k), device="cuda", generator=g).float() for _ in range(count)]
    qa, qb = [x.to(torch.float8_e4m3fn) for x in a], [x.to(torch.float8_e4m3fn) for x in b]
    c = [torch.full((m, n), float("nan"), device="cuda") for _ in range(count)]
    d = [torch.empty(m, n, device="cuda") for _ in range(count)]
    plan = ops.TcPlan([ops.tc_problem(qa[i], qb[i], c[i], trans_b=True, alpha=0.5) for i in range(count)], in_dtype=ops.E4M3)
    assert plan.tile_n == 512
    plan.launch()
    one = ops.TcPlan([ops.tc_problem(qa[i], qb[i], d[i], trans_b=True, alpha=0.5) for i in range(count)], in_dtype=ops.E4M3,
                     tile_n=256)
    one.launch()
    for i in range(count):
        # sums of at most 4096 integers of magnitude 16: exact in f32
        assert torch.equal(c[i].double(), 0.5 * (a[i].double() @ b[i].double().T))
        assert torch.equal(c[i], d[i])


def test_e4m3_pair_is_refused_by_name(cuda):
    import torch
    from bbts_b200 import BbxError, ops
    x = torch.zeros(4096, 4096, device="cuda").to(torch.float8_e4m3fn)
    c = torch.empty(4096, 4096, device="cuda")
    with pytest.raises(BbxError):
        ops.TcPlan([ops.tc_problem(x, x, c, trans_b=True)], in_dtype=ops.E4M3, tile_n=512)


@pytest.mark.parametrize("rows,cols", [(16, 8), (128, 64), (144, 72), (112, 200), (272, 136)])
@pytest.mark.parametrize("bf16", [False, True])
def test_transposed_quantisation_tile_edges(cuda, rows, cols, bf16):
    """The transposed kernel's 128 x 64 tiles against the row-major kernel's bytes, transposed."""
    import torch
    from bbts_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, cols, device="cuda", generator=g)
    x = x.bfloat16() if bf16 else x
    q, t = torch.empty(rows, cols, device="cuda", dtype=torch.float8_e4m3fn), torch.empty(cols, rows, device="cuda", dtype=torch.float8_e4m3fn)
    s = torch.empty(2, device="cuda")
    ops.quantize_e4m3(x, q, s[:1])
    ops.quantize_e4m3(x, t, s[1:], transpose=True)
    assert torch.equal(q.view(torch.uint8).T, t.view(torch.uint8)) and s[0].item() == s[1].item()
