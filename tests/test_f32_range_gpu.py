"""FP32 products whose operands leave the range of the tensor-core scheme: infinities, NaN,
sums near overflow, products that are all tiny. They are the FMA chain's, bit for bit (which a
captured call runs, on the SIMT kernel), on both tile shapes, alone and beside products in
range, without running out any bounded wait, and take about the SIMT kernel's time.
Every size here is one that the size rule gives to the tensor cores."""
import pytest

pytestmark = pytest.mark.gpu

KINDS = ("inf", "nan", "largest", "tiny")


@pytest.fixture(scope="module")
def T(cuda):
    import torch
    from bbts_b200 import lib, ops
    return torch, ops, lib


def _out_of_range(torch, kind, a, b):
    if kind == "inf":
        a.view(-1)[a.numel() // 3], b.view(-1)[7] = float("inf"), float("-inf")
    elif kind == "nan":
        b.view(-1)[b.numel() - 1] = float("nan")
    elif kind == "largest":
        a.view(-1)[0], a.view(-1)[a.numel() - 1] = torch.finfo(torch.float32).max, -1e38
    else:  # down to f32's smallest values, themselves and as products
        a *= 2.0 ** -60
        a.view(-1)[::5] *= 2.0 ** -85
        b *= 2.0 ** -60


def _captured(torch, f):
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        f()
    return graph


def _same(torch, x, y):
    assert torch.equal(x.isnan(), y.isnan())
    same = (x.view(torch.int32) == y.view(torch.int32)) | x.isnan()
    assert same.all(), (x[~same][:4], y[~same][:4], int((~same).sum()))


def _status(lib):
    assert lib.bbx_check_device_status(None, None) == 0


# 128 tiles with edges inside and at their ends; a size whose 256 tiles fill the chip
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("m,n,k", [(257, 300, 205), (640, 129, 256), (3900, 4001, 77)])
def test_alone(T, kind, ta, tb, m, n, k):
    torch, ops, lib = T
    assert lib.bbx_matmul_f32_route(m, n, k, 1) == 1
    g = torch.Generator(device="cuda").manual_seed(k)
    a = torch.randn((k, m) if ta else (m, k), device="cuda", generator=g)
    b = torch.randn((n, k) if tb else (k, n), device="cuda", generator=g)
    _out_of_range(torch, kind, a, b)
    c, d = torch.full((m, n), 7.0, device="cuda"), torch.full((m, n), 7.0, device="cuda")
    ops.matmul_f32(a, b, c, bool(ta), bool(tb))
    _captured(torch, lambda: ops.matmul_f32(a, b, d, bool(ta), bool(tb))).replay()
    _same(torch, c, d)
    _status(lib)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("pad", [0, 3])
def test_batch_pitch_and_epilogue(T, kind, pad):
    torch, ops, lib = T
    m, n, k, nb = 300, 261, 250, 3
    assert lib.bbx_matmul_f32_route(m, n, k, nb) == 1
    g = torch.Generator(device="cuda").manual_seed(pad)
    wide = lambda r, c: torch.randn((nb, r, c + pad), device="cuda", generator=g)
    a, b, c = wide(m, k), wide(k, n), wide(m, n)
    _out_of_range(torch, kind, a[1], b[1])  # one of the batch; the maxima are the call's
    d, bias = c.clone(), torch.randn(n, device="cuda", generator=g)
    call = lambda out: ops.matmul_f32(a[:, :, :k], b[:, :, pad:], out[:, :, :n], alpha=2.0, beta=-0.5, bias=bias)
    if kind == "tiny":  # all of it
        a *= 2.0 ** -60
        b *= 2.0 ** -60
    graph = _captured(torch, lambda: call(d))
    call(c)
    graph.replay()
    _same(torch, c, d)
    _status(lib)


@pytest.mark.parametrize("form,dims", [("ijk,kl->ijl", (70, 5, 260, 190)), ("ijk,lk->ilj", (130, 5, 192, 129)),
                                       ("kij,kl->lij", (300, 20, 60, 150)), ("ijb,jkb->ikb", (150, 256, 130, 3))])
@pytest.mark.parametrize("kind", ["inf", "tiny"])
def test_contractions(T, form, dims, kind):
    """Against FP64: non-finite outputs where they belong, the others within the FMA chain's K ulp."""
    torch, ops, lib = T
    lhs, rest = form.split(",")
    rhs, out = rest.split("->")
    ext = dict(zip("ijkb" if "b" in form else "kijl" if lhs == "kij" else "ijkl", dims))
    num = {c: i for i, c in enumerate("ijklb")}
    shape, code = lambda s: [ext[c] for c in s], lambda s: [num[c] for c in s]
    size = lambda names: int(torch.tensor([ext[c] for c in names] or [1]).prod())
    batch = [c for c in ext if c in lhs and c in rhs and c in out]
    k = size([c for c in lhs if c in rhs and c not in out])
    assert lib.bbx_matmul_f32_route(size([c for c in lhs if c in out and c not in batch]),
                                    size([c for c in rhs if c in out and c not in batch]), k, size(batch)) == 1
    g = torch.Generator(device="cuda").manual_seed(9)
    x, y = torch.randn(size(lhs), device="cuda", generator=g), torch.randn(size(rhs), device="cuda", generator=g)
    if kind == "inf":
        x[size(lhs) // 2] = float("inf")
    else:
        _out_of_range(torch, kind, x, y)
    z = torch.empty(size(out), device="cuda")
    ops.contraction(x, shape(lhs), code(lhs), y, shape(rhs), code(rhs), z, code(out))
    ein = "%s,%s->%s" % (lhs[::-1], rhs[::-1], out[::-1])
    X, Y = x.double().view(shape(lhs)[::-1]), y.double().view(shape(rhs)[::-1])
    ref, mag = torch.einsum(ein, X, Y).reshape(-1), torch.einsum(ein, X.abs(), Y.abs()).reshape(-1)
    assert torch.equal(z.isinf(), ref.isinf()) and torch.equal(z.isnan(), ref.isnan())
    ok = ref.isfinite()
    # one rounding a step: K half-ulps of the terms' magnitudes, or K / 2 of f32's smallest value
    assert ((z.double() - ref).abs() <= k * (2.0 ** -24 * mag + 2.0 ** -150))[ok].all()
    _status(lib)


@pytest.mark.parametrize("bs", [200, 1100])
def test_beside_products_in_range(T, bs):
    """One compiled group of products in and out of range, small tiles and (at 1100) pairs: those in
    range as if alone, the others the FMA chain's."""
    torch, ops, lib = T
    from bbts_b200 import runtime
    assert lib.bbx_matmul_f32_route(bs, bs, bs, 1) == 1
    g = torch.Generator(device="cuda").manual_seed(bs)
    x = [torch.randn(bs, bs, device="cuda", generator=g) for _ in range(7)]
    x[3].view(-1)[bs + 3] = float("inf")
    x[4].view(-1)[5] = float("nan")
    x[5].view(-1)[bs * bs - 1] = torch.finfo(torch.float32).max
    x[6] *= 2.0 ** -60  # in range with x[0..2], not with itself
    rt = runtime.Runtime()
    for t, v in enumerate(x):
        rt.put_dense(t, v.cpu().numpy())
    mm = rt.impl("matrix_mult", ["dense"] * 2, ["dense"])
    pairs = [(i, j) for i in range(7) for j in range(7)]
    for q, (i, j) in enumerate(pairs):
        rt.apply(mm, [i, j], [100 + q], params=[bool(q & 1), bool(q & 2)])
    dag = rt.build_dag()
    dag.launch()
    for q, (i, j) in enumerate(pairs):
        got = torch.empty(bs, bs, device="cuda")
        dag.fetch(100 + q, got.data_ptr(), 4 * bs * bs, on_device=True)
        torch.cuda.synchronize()
        want = torch.empty(bs, bs, device="cuda")
        call = lambda: ops.matmul_f32(x[i], x[j], want, bool(q & 1), bool(q & 2))
        if {3, 4, 5} & {i, j} or i == j == 6:
            _captured(torch, call).replay()
        else:
            call()
        torch.cuda.synchronize()
        _same(torch, got, want)
    _status(lib)


def test_one_infinity_costs_about_the_simt_time(T):
    """1024^3: measured 105 us on the SIMT kernel."""
    torch, ops, lib = T
    a, b, c = (torch.randn(1024, 1024, device="cuda") for _ in range(3))
    a[3, 5] = float("inf")
    graph = _captured(torch, lambda: ops.matmul_f32(a, b, c))

    def us(f):
        t = []
        for _ in range(7):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            f()
            e[1].record()
            torch.cuda.synchronize()
            t.append(1e3 * e[0].elapsed_time(e[1]))
        return sorted(t)[3]
    simt, here = us(graph.replay), us(lambda: ops.matmul_f32(a, b, c))
    assert here < 4 * simt, (here, simt)
