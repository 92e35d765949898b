"""FP32 products on the tensor cores (csrc/gemm_f32tc.cuh): sizes at the edges of
the 64-deep chunks and the 128 / 256 tiles, every layout, batches, epilogues,
operands over the whole f32 range, and the FP32 form that takes over outside it.

Bound, element by element, against FP64: a chunk of 64 ends in four MMAs that
each truncate the accumulator by less than 2 ulp (8 * 2^-23), chunks are added
with one rounding each (K / 64 * 2^-24), the dropped products are below 3 * 2^-27,
and alpha, beta and bias round once each: less than (16 + K / 64) * 2^-23 of
sum |a||b| (+ |beta c| + |bias|).
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def T(cuda):
    import torch
    from bbts_b200 import ops
    return torch, ops


def _bound(k, mag):
    return (16 + k / 64) * 2.0 ** -23 * mag


def _check(torch, a, b, c, ta=False, tb=False, extra=None, ref_extra=0.0):
    A = a.double().transpose(-1, -2) if ta else a.double()
    B = b.double().transpose(-1, -2) if tb else b.double()
    ref = A @ B + ref_extra
    mag = A.abs() @ B.abs() + (0 if extra is None else extra)
    over = (c.double() - ref).abs() - _bound(A.shape[-1], mag)
    assert over.max().item() <= 2.0 ** -140, over.max().item()  # f32's own smallest values


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("m,n,k", [(64, 64, 64), (65, 127, 66), (128, 129, 127), (257, 255, 129), (300, 520, 64),
                                   (1000, 264, 200), (2049, 2300, 72)])
def test_sizes_and_layouts(T, m, n, k, ta, tb):
    torch, ops = T
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn((k, m) if ta else (m, k), device="cuda", generator=g)
    b = torch.randn((n, k) if tb else (k, n), device="cuda", generator=g)
    c = torch.full((m, n), float("nan"), device="cuda")
    ops.matmul_f32(a, b, c, bool(ta), bool(tb))
    _check(torch, a, b, c, ta, tb)


@pytest.mark.parametrize("pad", [0, 3, 4])
def test_batch_pitch_and_epilogue(T, pad):
    torch, ops = T
    m, n, k, nb = 130, 197 if pad == 3 else 196, 100, 3
    g = torch.Generator(device="cuda").manual_seed(pad)
    wide = lambda r, c: torch.randn((nb, r, c + pad), device="cuda", generator=g)
    a, b, c = wide(m, k), wide(k, n), wide(m, n)
    av, bv, cv = a[:, :, :k], b[:, :, pad:], c[:, :, :n]
    c0, bias = c.clone(), torch.randn(n, device="cuda", generator=g)
    ops.matmul_f32(av, bv, cv, alpha=2.0, beta=-0.5, bias=bias, relu=False)
    _check(torch, 2.0 * av, bv, cv, extra=(0.5 * c0[:, :, :n]).abs().double() + bias.abs().double(),
           ref_extra=-0.5 * c0[:, :, :n].double() + bias.double())
    assert torch.equal(c[:, :, n:], c0[:, :, n:])  # the pitch padding of C is left alone
    ops.matmul_f32(av, bv, cv, relu=True)
    assert cv.min().item() == 0.0


@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 1)])
def test_whole_range_of_f32(T, ta, tb):
    """Rows of A and columns of B from 2^-130 (subnormal) to 2^40, each output relative to its own terms."""
    torch, ops = T
    n, k = 160, 192
    g = torch.Generator(device="cuda").manual_seed(5)
    ea = torch.tensor([-130.0, -120, -100, -60, -20, 0, 20, 40], device="cuda", dtype=torch.float64).repeat(n // 8)
    eb = torch.tensor([40.0, 30, 20, 10, 40], device="cuda", dtype=torch.float64).repeat(n // 5)
    a = (torch.randn(n, k, device="cuda", generator=g).double() * 2.0 ** ea[:, None]).float()
    b = (torch.randn(k, n, device="cuda", generator=g).double() * 2.0 ** eb[None, :]).float()
    c = torch.empty(n, n, device="cuda")
    ops.matmul_f32(a.T.contiguous() if ta else a, b.T.contiguous() if tb else b, c, bool(ta), bool(tb))
    _check(torch, a, b, c)


@pytest.mark.parametrize("kind", ["inf", "nan", "largest", "tiny", "zero"])
@pytest.mark.parametrize("m,n,k", [(96, 200, 80), (700, 64, 130)])
def test_out_of_range_is_the_fma_chain(T, kind, m, n, k):
    """Operands outside the range give the SIMT kernel's bits (which a captured call runs)."""
    torch, ops = T
    g = torch.Generator(device="cuda").manual_seed(k)
    a = torch.randn(m, k, device="cuda", generator=g)
    b = torch.randn(k, n, device="cuda", generator=g)
    if kind == "inf":
        a[3, 5], b[7, 11] = float("inf"), float("-inf")
    elif kind == "nan":
        b[2, 1] = float("nan")
    elif kind == "largest":
        a[0, 0], a[5, :] = torch.finfo(torch.float32).max, 1e38
    elif kind == "tiny":
        a *= 2.0 ** -60
        b *= 2.0 ** -60
    else:
        a.zero_()
    c = torch.full((m, n), 7.0, device="cuda")
    d = torch.full((m, n), 7.0, device="cuda")
    ops.matmul_f32(a, b, c)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.matmul_f32(a, b, d)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(c.isnan(), d.isnan())
    assert torch.equal(c.nan_to_num(nan=0.0, posinf=1e30, neginf=-1e30), d.nan_to_num(nan=0.0, posinf=1e30, neginf=-1e30))


@pytest.mark.parametrize("form,dims", [("ijk,kl->ijl", (70, 3, 65, 90)), ("ijk,lk->ilj", (66, 5, 64, 129)),
                                       ("kij,kl->lij", (40, 11, 100, 64)), ("ijb,jkb->ikb", (72, 64, 80, 3))])
def test_contraction_forms(T, form, dims):
    torch, ops = T
    ext = dict(zip("ijklb" if "b" not in form else "ijkb", dims))
    num = {c: i for i, c in enumerate("ijklb")}
    lhs, rest = form.split(",")
    rhs, out = rest.split("->")
    shape = lambda s: [ext[c] for c in s]
    numel = lambda s: int(torch.tensor(shape(s)).prod())
    g = torch.Generator(device="cuda").manual_seed(9)
    x, y = torch.randn(numel(lhs), device="cuda", generator=g), torch.randn(numel(rhs), device="cuda", generator=g)
    z = torch.empty(numel(out), device="cuda")
    code = lambda s: [num[c] for c in s]
    ops.contraction(x, shape(lhs), code(lhs), y, shape(rhs), code(rhs), z, code(out), alpha=0.5)
    ein = "%s,%s->%s" % (lhs[::-1], rhs[::-1], out[::-1])
    X, Y = 0.5 * x.double().view(shape(lhs)[::-1]), y.double().view(shape(rhs)[::-1])
    ref, mag = torch.einsum(ein, X, Y).reshape(-1), torch.einsum(ein, X.abs(), Y.abs()).reshape(-1)
    summed = [c for c in "ijklb" if c in lhs and c in rhs and c not in out]
    k = 1
    for c in summed:
        k *= ext[c]
    assert ((z.double() - ref).abs() <= _bound(k, mag)).all()


def test_many_streams_share_the_scratch_pool(T):
    """Products on several streams at once: each call's planes are its own."""
    torch, ops = T
    g = torch.Generator(device="cuda").manual_seed(1)
    streams = [torch.cuda.Stream() for _ in range(4)]
    work = []
    for i in range(12):
        a = torch.randn(200 + i, 300, device="cuda", generator=g)
        b = torch.randn(300, 260, device="cuda", generator=g)
        work.append((a, b, torch.empty(200 + i, 260, device="cuda")))
    torch.cuda.synchronize()
    for r in range(3):
        for i, (a, b, c) in enumerate(work):
            with torch.cuda.stream(streams[(i + r) % 4]):
                ops.matmul_f32(a, b, c)
        torch.cuda.synchronize()
    for a, b, c in work:
        _check(torch, a, b, c)


@pytest.mark.parametrize("bs", [96, 201])
def test_pre_activations_keep_the_fma_chain(T, bs):
    """Products that reach a ReLU through adds give the SIMT kernel's bits, per command and in a grouped
    DAG launch (whose packed FMAs round alike); the others run on the tensor cores in both."""
    torch, ops = T
    import numpy as np
    from bbts_b200 import runtime
    rng = np.random.default_rng(bs)
    n = 4 * bs
    x = [rng.standard_normal((n, n)).astype(np.float32) for _ in range(4)]
    got = {}
    for path in ("per_op", "dag"):
        rt = runtime.Runtime()
        for t, v in enumerate(x):
            rt.put_dense(t, v)
        mm, add = rt.impl("matrix_mult", ["dense"] * 2, ["dense"]), rt.impl("matrix_add", ["dense"] * 2, ["dense"])
        relu = rt.impl("matrix_relu", ["dense"], ["dense"])
        rt.apply(mm, [0, 1], [10])
        rt.apply(mm, [2, 3], [11], params=[True, False])
        rt.apply(add, [10, 11], [12])
        rt.apply(relu, [12], [13])
        rt.apply(mm, [0, 3], [14], params=[False, True])
        if path == "dag":
            dag = rt.build_dag()
            dag.launch()
            got[path] = [dag.read_bytes(t, 4 * n * n).view(np.float32).reshape(n, n) for t in (10, 11, 13, 14)]
        else:
            rt.run()
            got[path] = [rt.get_dense(t) for t in (10, 11, 13, 14)]
    for p, d in zip(got["per_op"], got["dag"]):
        assert np.array_equal(p, d)
    dev = [torch.from_numpy(v).cuda() for v in x]
    want = []
    for a, b, ta in ((dev[0], dev[1], False), (dev[2], dev[3], True)):
        c = torch.empty(n, n, device="cuda")
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):  # a captured call runs the SIMT kernel
            ops.matmul_f32(a, b, c, ta)
        graph.replay()
        torch.cuda.synchronize()
        want.append(c.cpu().numpy())
    assert np.array_equal(got["dag"][0], want[0]) and np.array_equal(got["dag"][1], want[1])
    _check(torch, dev[0], dev[3], torch.from_numpy(got["dag"][3]).cuda(), tb=True)
