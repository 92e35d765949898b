"""FP32 products and contractions at sizes that the size rule gives to the tensor cores (asserted
in each test): tile and chunk edges in every layout on both tile shapes, batches with every epilogue
term, operands over the whole f32 range and of one sign, every contraction lowering, and sources
at each of the four alignments whose neighbours in memory are NaN.

Bound, element by element, against FP64: a chunk of 64 ends in four MMAs that each truncate the
accumulator by less than 2 ulp (8 * 2^-23), chunks are added with one rounding each
(K / 64 * 2^-24), the dropped products are below 3 * 2^-27, and alpha, beta and bias round once
each: less than (16 + K / 64) * 2^-23 of sum |a||b| (+ |beta c| + |bias|).
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def T(cuda):
    import torch
    from bbts_b200 import lib, ops
    return torch, ops, lib


def _bound(k, mag):
    return (16 + k / 64) * 2.0 ** -23 * mag


def _check(torch, a, b, c, extra=0.0, ref_extra=0.0):
    """c against a @ b + ref_extra."""
    a, b = a.double(), b.double()
    over = (c.double() - (a @ b + ref_extra)).abs() - _bound(a.shape[-1], a.abs() @ b.abs() + extra)
    assert over.max().item() <= 2.0 ** -140, over.max().item()  # f32's own smallest values


def _guarded(torch, x, offset):
    """x's values at a view `offset` elements into an allocation that is NaN everywhere else, flat."""
    buf = torch.full((x.numel() + 16,), float("nan"), device="cuda")
    v = buf[4 + offset:4 + offset + x.numel()]
    v.copy_(x.reshape(-1))
    return v


SIZES = [(128, 128, 192), (129, 255, 193), (257, 130, 320), (16, 2000, 250), (1000, 264, 200), (2049, 2300, 136),
         (4000, 3900, 72)]  # the last one on the 256 pair


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("m,n,k", SIZES)
def test_sizes_and_layouts(T, m, n, k, ta, tb):
    torch, ops, lib = T
    assert lib.bbx_matmul_f32_route(m, n, k, 1) == 1
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn((k, m) if ta else (m, k), device="cuda", generator=g)
    b = torch.randn((n, k) if tb else (k, n), device="cuda", generator=g)
    c = torch.full((m, n), float("nan"), device="cuda")
    ops.matmul_f32(a, b, c, bool(ta), bool(tb))
    _check(torch, a.T if ta else a, b.T if tb else b, c)


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_unaligned_operands_between_nans(T, ta, tb, offset):
    """The split reads whole 16-byte pieces around its elements: nothing beside the operand may count."""
    torch, ops, lib = T
    m, n, k = 203, 149, 301
    assert lib.bbx_matmul_f32_route(m, n, k, 1) == 1
    g = torch.Generator(device="cuda").manual_seed(offset)
    a = torch.randn((k, m) if ta else (m, k), device="cuda", generator=g)
    b = torch.randn((n, k) if tb else (k, n), device="cuda", generator=g)
    av, bv = _guarded(torch, a, offset).view(a.shape), _guarded(torch, b, 3 - offset).view(b.shape)
    c = _guarded(torch, torch.zeros(m, n, device="cuda"), offset)
    ops.matmul_f32(av, bv, c.view(m, n), bool(ta), bool(tb))
    _check(torch, a.T if ta else a, b.T if tb else b, c.view(m, n))
    buf = c._base
    assert buf[:4 + offset].isnan().all() and buf[4 + offset + m * n:].isnan().all()


@pytest.mark.parametrize("pad", [0, 3, 4])
@pytest.mark.parametrize("m,n,k,nb", [(200, 181, 200, 5), (130, 260, 450, 3)])
def test_batch_pitch_and_epilogue(T, m, n, k, nb, pad):
    torch, ops, lib = T
    assert lib.bbx_matmul_f32_route(m, n, k, nb) == 1
    g = torch.Generator(device="cuda").manual_seed(pad)
    wide = lambda r, c: torch.randn((nb, r, c + pad), device="cuda", generator=g)
    a, b, c = wide(m, k), wide(k, n), wide(m, n)
    a[:, :, k:], b[:, :, :pad] = float("nan"), float("nan")
    av, bv, cv = a[:, :, :k], b[:, :, pad:], c[:, :, :n]
    c0, bias = c.clone(), torch.randn(n, device="cuda", generator=g)
    ops.matmul_f32(av, bv, cv, alpha=2.0, beta=-0.5, bias=bias)
    _check(torch, 2.0 * av, bv, cv, extra=(0.5 * c0[:, :, :n]).abs().double() + bias.abs().double(),
           ref_extra=-0.5 * c0[:, :, :n].double() + bias.double())
    assert torch.equal(c[:, :, n:], c0[:, :, n:])  # the pitch padding of C is left alone
    d = torch.empty(nb, m, n, device="cuda")
    ops.matmul_f32(av[:1].expand(nb, m, k), bv, d)  # one A for the whole batch: stride 0
    _check(torch, av[:1].expand(nb, m, k), bv, d)


@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 1)])
def test_whole_range_of_f32(T, ta, tb):
    """Rows of A and columns of B from 2^-130 (subnormal) to 2^40, each output relative to its own terms."""
    torch, ops, lib = T
    n, k = 320, 260
    assert lib.bbx_matmul_f32_route(n, n, k, 1) == 1
    g = torch.Generator(device="cuda").manual_seed(5)
    ea = torch.tensor([-130.0, -120, -100, -60, -20, 0, 20, 40], device="cuda", dtype=torch.float64).repeat(n // 8)
    eb = torch.tensor([40.0, 30, 20, 10, 40], device="cuda", dtype=torch.float64).repeat(n // 5)
    a = (torch.randn(n, k, device="cuda", generator=g).double() * 2.0 ** ea[:, None]).float()
    b = (torch.randn(k, n, device="cuda", generator=g).double() * 2.0 ** eb[None, :]).float()
    c = torch.empty(n, n, device="cuda")
    ops.matmul_f32(a.T.contiguous() if ta else a, b.T.contiguous() if tb else b, c, bool(ta), bool(tb))
    _check(torch, a, b, c)


@pytest.mark.parametrize("values", ["normal", "uniform", "negative", "around one"])
@pytest.mark.parametrize("m,n,k", [(256, 256, 192), (500, 300, 450), (512, 512, 2048)])
def test_error_is_below_the_fma_chains(T, values, m, n, k):
    """Of both signs and of one, where the tensor core's truncation adds up: Frobenius error against FP64,
    here and on the SIMT kernel (which a captured call runs)."""
    torch, ops, lib = T
    assert lib.bbx_matmul_f32_route(m, n, k, 1) == 1
    g = torch.Generator(device="cuda").manual_seed(k)

    def draw(r, c):
        if values == "normal":
            return torch.randn(r, c, device="cuda", generator=g)
        u = torch.rand(r, c, device="cuda", generator=g)
        return {"uniform": u, "negative": -0.5 - u, "around one": 1 + 1e-3 * u}[values]
    a, b = draw(m, k), draw(k, n)
    c, d = torch.empty(m, n, device="cuda"), torch.empty(m, n, device="cuda")
    ops.matmul_f32(a, b, c)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.matmul_f32(a, b, d)
    graph.replay()
    _check(torch, a, b, c)
    ref = a.double() @ b.double()
    assert (c.double() - ref).norm() <= (d.double() - ref).norm()


# modes and extents: K- and MN-major sources, a batch mode, summed modes, two contracted modes apart, outputs
# in another order
FORMS = [("ijk,kl->ijl", dict(i=70, j=5, k=260, l=190)), ("ijk,lk->ilj", dict(i=130, j=5, k=192, l=129)),
         ("kij,kl->lij", dict(k=300, i=20, j=60, l=150)), ("ijb,jkb->ikb", dict(i=150, j=256, k=130, b=3)),
         ("iks,kl->il", dict(i=300, k=261, s=3, l=140)), ("ikjb,bkl->ijl", dict(i=40, k=33, j=9, b=8, l=170)),
         ("ki,skl->li", dict(k=250, i=203, s=2, l=301))]


@pytest.mark.parametrize("form,ext", FORMS)
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("bf16", [False, True])
def test_contraction_lowerings(T, form, ext, offset, bf16):
    torch, ops, lib = T
    lhs, rest = form.split(",")
    rhs, out = rest.split("->")
    num = {c: i for i, c in enumerate("ijklbs")}
    shape, code = lambda s: [ext[c] for c in s], lambda s: [num[c] for c in s]

    def size(names):
        n = 1
        for c in names:
            n *= ext[c]
        return n
    batch = [c for c in ext if c in lhs and c in rhs and c in out]
    k = size([c for c in lhs if c in rhs and c not in out])
    assert lib.bbx_matmul_f32_route(size([c for c in lhs if c in out and c not in batch]),
                                    size([c for c in rhs if c in out and c not in batch]), k, size(batch)) == 1
    g = torch.Generator(device="cuda").manual_seed(9)
    x, y = torch.randn(size(lhs), device="cuda", generator=g), torch.randn(size(rhs), device="cuda", generator=g)
    xv, yv, z = _guarded(torch, x, offset), _guarded(torch, y, 3 - offset), _guarded(torch, torch.zeros(size(out), device="cuda"), offset)
    ops.contraction(xv, shape(lhs), code(lhs), yv, shape(rhs), code(rhs), z, code(out), alpha=0.5,
                    precision=ops.BF16 if bf16 else ops.F32)
    summed = "s" in lhs + rhs and "s" not in out
    if bf16 and not summed:
        x, y = x.bfloat16(), y.bfloat16()
    ein = "%s,%s->%s" % (lhs[::-1], rhs[::-1], out[::-1])
    X, Y = 0.5 * x.double().view(shape(lhs)[::-1]), y.double().view(shape(rhs)[::-1])
    ref, mag = torch.einsum(ein, X, Y).reshape(-1), torch.einsum(ein, X.abs(), Y.abs()).reshape(-1)
    if bf16:  # one accumulator of truncating additions (2 ulp each, 16 steps at a time); summed modes round to bf16 after the sum
        bound = (4 + k / 8) * 2.0 ** -23 * mag + (2.0 ** -7 * mag if summed else 0)
    else:  # a summed mode is one f32 sum first
        bound = _bound(k, mag) + (size(["s"]) * 2.0 ** -24 * mag if summed else 0)
    assert ((z.double() - ref).abs() <= bound).all(), ((z.double() - ref).abs() / mag).max().item()
    buf = z._base
    assert buf[:4 + offset].isnan().all() and buf[4 + offset + z.numel():].isnan().all()


@pytest.mark.parametrize("tile_n", [128, 256, 512])
@pytest.mark.parametrize("kind", ["f32 short", "f32 long", "bf16", "f32 columns", "bf16 columns"])
@pytest.mark.parametrize("m,n", [(256, 256), (272, 264), (40, 520), (301, 259)])
def test_tensor_core_stores(T, tile_n, kind, m, n):
    """Every way C leaves a bf16 product (swizzled and plain boxes, staged rows, columns from registers):
    whole numbers that f32 and (at most 256) bf16 hold, a guard around C."""
    torch, ops, lib = T
    k = 640 if kind == "f32 long" else 256
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a = torch.randint(-1, 2, (m, k), device="cuda", generator=g).bfloat16()
    b = torch.randint(-1, 2, (k, (n + 7) // 8 * 8), device="cuda", generator=g).bfloat16()[:, :n]
    cols, dt = "columns" in kind, torch.bfloat16 if "bf16" in kind else torch.float32
    r, w = (n, m) if cols else (m, n)
    for pad in (0, 8, 5):
        buf = torch.full((r + 2, w + pad), float("nan"), device="cuda", dtype=dt)
        c = buf[1:r + 1, :w]
        ops.matmul_tc([ops.tc_problem(a, b, c, c_colmajor=cols)], tile_n=tile_n)
        ref = a.double() @ b.double()
        assert torch.equal(c.double(), ref.T if cols else ref)
        c.fill_(float("nan"))
        assert buf.isnan().all()
