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


@pytest.mark.parametrize("n,h,w,c,k,s,p", [(1, 1, 1, 1, 1, 1, 0), (3, 17, 19, 3, 7, 2, 3), (2, 8, 8, 16, 5, 1, 0), (5, 32, 33, 3, 3, 1, 1),
                                           (1, 7, 300, 24, 3, 2, 2), (2, 28, 28, 1, 5, 1, 0), (2, 9, 700, 64, 3, 1, 1), (1, 12, 12, 8, 4, 4, 5),
                                           (3, 40, 16, 7, 16, 1, 8)])
def test_im2col_rows(n, h, w, c, k, s, p):
    """Patch matrix, bit for bit: rows with and without whole 16-byte vectors, padding wider than the filter needs, a last
    block of fewer output rows, more than 256 column groups."""
    from tnn_b200.ops import conv
    torch.manual_seed(0)
    x = _rand(n, h, w, c)
    oh, ow = (h + 2 * p - k) // s + 1, (w + 2 * p - k) // s + 1
    cols, K = conv.im2col(x, k, k, (s, s), (p, p), oh, ow)
    u = torch.nn.functional.unfold(x.permute(0, 3, 1, 2).float(), k, padding=p, stride=s)       # [n, c*k*k, oh*ow]
    ref = u.view(n, c, k * k, oh * ow).permute(0, 3, 2, 1).reshape(n * oh * ow, K)
    assert torch.equal(cols[:, :K].float(), ref)


@pytest.mark.parametrize("n,h,w,c,k,s,p", [(2, 7, 7, 40, 7, 1, 0), (3, 9, 11, 8, 3, 2, 1), (1, 5, 300, 64, 2, 2, 0), (4, 8, 8, 24, 5, 3, 2),
                                           (2, 16, 16, 16, 4, 1, 0), (1, 3, 3, 8, 3, 1, 2),
                                           (2, 10, 9, 16, 4, 2, 1), (1, 7, 12, 72, 3, 2, 0), (2, 5, 6, 8, 1, 2, 0), (1, 9, 9, 8, 2, 2, 1)])
@pytest.mark.parametrize("mode", ["max", "avg"])
def test_pool_rows(n, h, w, c, k, s, p, mode):
    """Pooling forward (values and positions) and backward against the CPU reference: short and long rows, windows that
    reach over every edge, the shared-window average."""
    from tnn_b200.ops import raw
    torch.manual_seed(0)
    x = _rand(n, h, w, c)
    y, idx = raw.pool2d_fwd(x, mode, (k, k), (s, s), (p, p), True)
    yr, ir = raw.pool2d_fwd(x.cpu(), mode, (k, k), (s, s), (p, p), True)
    if mode == "max":
        assert torch.equal(y.cpu(), yr) and torch.equal(idx.cpu().int(), ir.int())
    else:
        assert torch.allclose(y.cpu().float(), yr.float(), rtol=2.0 ** -8, atol=1e-6)  # one bf16 rounding
    dy = _rand(*y.shape)
    dx = raw.pool2d_bwd(dy, idx, x.shape, mode, (k, k), (s, s), (p, p))
    dr = raw.pool2d_bwd(dy.cpu(), ir, x.shape, mode, (k, k), (s, s), (p, p))
    assert torch.allclose(dx.cpu().float(), dr.float(), rtol=2.0 ** -7, atol=2.0 ** -7 * float(dr.float().abs().max()) / 4)


@pytest.mark.parametrize("n,hw,c,k,p", [(3, 8, 2048, 8, 0), (140, 4, 512, 4, 0), (300, 4, 1024, 4, 0), (2, 19, 64, 4, 0), (5, 16, 8, 15, 0),
                                        (7, 7, 2048, 7, 0), (3, 9, 40, 5, 2)])
def test_average_adds_in_window_order(n, hw, c, k, p):
    """The elements of a window are added row by row in fp32, whatever kernel does it: bit for bit where the division is by a
    power of two, else to one bf16 rounding (2**-8)."""
    from tnn_b200.ops import raw
    torch.manual_seed(0)
    x = _rand(n, hw, hw, c)
    x[:, 0, 0] = 2.0 ** 20   # with its opposite at the end: what is left depends on the order
    x[:, k - 1, k - 1] = -2.0 ** 20
    y, _ = raw.pool2d_fwd(x, "avg", (k, k), (1, 1), (p, p))
    f = torch.nn.functional.pad(x.float(), (0, 0, p, p, p, p))
    inside = torch.nn.functional.pad(torch.ones(hw, hw, device="cuda"), (p, p, p, p))
    o = y.shape[1]
    total, count = torch.zeros(y.shape, device="cuda"), torch.zeros(o, o, device="cuda")
    for kh in range(k):
        for kw in range(k):
            total += f[:, kh:kh + o, kw:kw + o]
            count += inside[kh:kh + o, kw:kw + o]
    ref = (total / count[:, :, None]).to(BF)
    if p == 0 and k in (4, 8):
        assert torch.equal(y, ref)
    else:
        assert torch.allclose(y.float(), ref.float(), rtol=2.0 ** -7, atol=1e-6)


@pytest.mark.parametrize("mode", ["max", "avg"])
@pytest.mark.parametrize("n,c", [(0, 8), (3, 0)])
def test_empty_pools_and_patches(mode, n, c):
    from tnn_b200.ops import conv, raw
    x = torch.empty(n, 6, 6, c, dtype=BF, device="cuda")
    y, idx = raw.pool2d_fwd(x, mode, (2, 2), (2, 2), (0, 0), True)
    assert y.shape == (n, 3, 3, c)
    assert raw.pool2d_bwd(y, idx, x.shape, mode, (2, 2), (2, 2), (0, 0)).shape == x.shape
    assert conv.im2col(x, 3, 3, (1, 1), (1, 1), 6, 6)[0].shape == (n * 36, 9 * c)


def test_pool_of_more_rows_than_31_bits():
    """2**31 + 6144 rows of one pixel: the batch goes in two parts. A window of one element copies its input."""
    from tnn_b200.ops import raw
    if torch.cuda.mem_get_info()[0] < 100 << 30:
        pytest.skip("needs 75 GB")
    x = torch.empty(2 ** 20 + 3, 2048, 1, 8, dtype=BF, device="cuda").uniform_()
    same = lambda a: all(torch.equal(p, q) for p, q in zip(a.split(2 ** 16), x.split(2 ** 16)))
    y, _ = raw.pool2d_fwd(x, "avg", (1, 1), (1, 1), (0, 0))
    assert same(y)
    y.zero_()
    del y
    dx = raw.pool2d_bwd(x, None, x.shape, "avg", (1, 1), (1, 1), (0, 0))
    assert same(dx)
    del x, dx
    torch.cuda.empty_cache()


@pytest.mark.parametrize("o,kh,kw,c,khs,kws", [(64, 3, 3, 64, [2, 1, 0], [2, 1, 0]), (128, 1, 1, 64, [0], [0]), (64, 3, 3, 192, [2, 0], [1]),
                                               (192, 5, 2, 64, [4, 2, 0], [1, 0]), (64, 4, 7, 128, [3, 1], [5, 2])])
def test_dgrad_filter(o, kh, kw, c, khs, kws):
    from tnn_b200.ops import conv
    torch.manual_seed(0)
    w = _rand(o, kh, kw, c)
    ref = w[:, khs][:, :, kws].permute(3, 1, 2, 0).contiguous()
    assert torch.equal(conv._dgrad_filter(w, khs, kws), ref)
    assert torch.equal(conv._dgrad_filter(w.transpose(0, 3).contiguous().transpose(0, 3), khs, kws), ref)  # strided weights


@pytest.mark.parametrize("rows,c", [(1, 8), (7, 256), (300, 264), (65, 512), (1030, 768), (9, 776), (600, 1024), (33, 1280), (40, 2048)])
@pytest.mark.parametrize("p,with_delta,affine", [(0.0, True, True), (0.1, True, True), (0.0, False, True), (0.0, False, False)])
def test_layernorm_widths(rows, c, p, with_delta, affine):
    """Every register width of the forward kernel, with lanes that hold fewer chunks than others, against the CPU path.
    The bound is one bf16 rounding of the result (2**-8 of its size) on both sides."""
    from tnn_b200.ops import raw
    torch.manual_seed(0)
    x, d = _rand(rows, c), _rand(rows, c) if with_delta else None
    g, b = (1 + _rand(c, scale=0.1), _rand(c, scale=0.1)) if affine else (None, None)
    xo, h, mean, rstd = raw.layernorm_fwd(x, d, g, b, 1e-5, p, 11)
    cpu = [t.cpu() if t is not None else None for t in (x, d, g, b)]
    xr, hr, mr, rr = raw.layernorm_fwd(*cpu, 1e-5, p, 11)
    if p == 0.0:
        assert torch.equal(xo.cpu(), xr)
    else:  # d * (1 / (1 - p)) against d / (1 - p): one fp32 rounding, which can move the bf16 rounding by one unit
        assert torch.allclose(xo.cpu().float(), xr.float(), rtol=2.0 ** -7, atol=2.0 ** -16)
    one_unit = 0.0 if p == 0.0 else 2.0 ** -7 * float(xr.float().abs().max())  # of an element of the sum
    assert torch.allclose(mean.cpu(), mr, rtol=0, atol=1e-5 + one_unit / c)
    assert torch.allclose(rstd.cpu(), rr, rtol=1e-5 + one_unit / c * 4, atol=0)
    assert torch.allclose(h.cpu().float(), hr.float(), rtol=2.0 ** -7, atol=2.0 ** -7 + one_unit * float(rr.max()))


@pytest.mark.parametrize("rows,c", [(1, 8), (7, 256), (300, 264), (1500, 512), (2030, 768), (9, 776), (600, 1024), (33, 1280), (40, 2048)])
@pytest.mark.parametrize("dres,ddelta,dbias", [(True, True, True), (True, True, False), (False, False, False)])
def test_layernorm_backward_widths(rows, c, dres, ddelta, dbias):
    """Every register width of the backward kernel: rows against the CPU path to one bf16 rounding, column sums against fp64.
    A sum adds the rows of a warp, the eight warps of a block and the blocks, one after another in fp32: each of these
    additions rounds a partial sum, which is about the root of the sum of squares, by 2**-24 of it; the normalised values
    in the terms carry three roundings of their own. A row that is left out changes a sum by about 1."""
    from tnn_b200.ops import raw
    torch.manual_seed(0)
    x, dh, g = _rand(rows, c), _rand(rows, c), 1 + _rand(c, scale=0.1)
    res = _rand(rows, c) if dres else None
    mean, rstd = x.float().mean(1), torch.rsqrt(x.float().var(1, unbiased=False) + 1e-5)
    def run(dev):
        acc = [torch.full((c,), 0.5, device=dev) for _ in range(3)]
        to = lambda t: t.to(dev) if t is not None else None
        dx, dd = raw.layernorm_bwd(to(dh), to(x), to(mean), to(rstd), to(g), to(res), ddelta, 0.0, 0, acc[0], acc[1],
                                   dbias=acc[2] if dbias else None)
        return [dx] + ([dd] if ddelta else []), acc
    (got, sums), (ref, _) = run("cuda"), run("cpu")
    for a, b in zip(got, ref):
        assert torch.allclose(a.cpu().float(), b.float(), rtol=2.0 ** -7, atol=2.0 ** -7)
    blocks = min(-(-rows // 8), 148 * 3)
    depth = -(-rows // (8 * blocks)) + 8 + blocks + 3
    xhat = (x.double() - mean.double()[:, None]) * rstd.double()[:, None]
    terms = [dh.double() * xhat, dh.double()] + ([got[-1].double()] if dbias else [])  # dbias sums the rows as they are stored
    for total, t in zip(sums, terms):
        bound = depth * 2.0 ** -24 * (0.25 + t.square().sum(0)).sqrt()
        assert bool(((total.double() - 0.5 - t.sum(0)).abs() <= bound).all())
    if not dbias:
        assert bool((sums[2] == 0.5).all())


@pytest.mark.parametrize("rows,c", [(1, 8), (9, 256), (3553, 264), (3600, 768), (2369, 1024), (1185, 2048)])
def test_layernorm_backward_last_rows(rows, c):
    """Only the last rows have a gradient, whole numbers whose sums are exact: a remainder that is skipped shows."""
    from tnn_b200.ops import raw
    last = min(rows, 3)
    x, dh = torch.zeros(rows, c, dtype=BF, device="cuda"), torch.zeros(rows, c, dtype=BF, device="cuda")
    x[-last:] = 2
    dh[-last:] = torch.arange(1, last + 1, device="cuda", dtype=BF)[:, None]
    acc = [torch.zeros(c, device="cuda") for _ in range(2)]
    raw.layernorm_bwd(dh, x, torch.ones(rows, device="cuda"), torch.ones(rows, device="cuda"), torch.ones(c, dtype=BF, device="cuda"),
                      None, False, 0.0, 0, acc[0], acc[1])
    want = last * (last + 1) / 2
    assert bool((acc[0] == want).all()) and bool((acc[1] == want).all())


@pytest.mark.parametrize("rows,cols,pad", [(1, 1, 0), (5, 203, 5), (333, 1024, 0), (64, 50257, 7), (3, 8, 8)])
def test_scale_by(rows, cols, pad):
    from tnn_b200.ops import raw
    torch.manual_seed(0)
    x = _rand(rows, cols + pad)[:, :cols]
    f = torch.tensor(0.3712, device="cuda")
    assert torch.equal(raw.scale_by(x, f), (x.float() * f).to(BF))


@pytest.mark.parametrize("shape,strides", [((1, 40), (8, 1)), ((1, 40), (0, 1)), ((3, 40), (0, 1)), ((3, 40), (16, 1)), ((40, 3), (1, 40))])
def test_scale_by_strides(shape, strides):
    """Rows that overlap, repeat, or have a stride that is never used."""
    from tnn_b200.ops import raw
    torch.manual_seed(0)
    x = _rand(256).as_strided(shape, strides)
    f = torch.tensor(0.3712, device="cuda")
    assert torch.equal(raw.scale_by(x, f), (x.float() * f).to(BF))


def _colsum_rows(m, n):
    """Rows per block and blocks of the column sums."""
    want = -(-4 * 148 // -(-n // 64))
    if m < 65536:
        want = min(want, 64)
    rows = -(--(-m // want) // 128) * 128
    return rows, -(-m // rows)


@pytest.mark.parametrize("m,n", [(65535, 64), (65536, 64), (70001, 8), (70001, 72), (300, 3072)])
def test_colsum_tall(m, n):
    """A sum adds the rows of a lane, the 32 lanes of a block and the blocks, one after another in fp32: each of these
    additions rounds a partial sum, which is about the root of the sum of squares, by 2**-24 of it. A row that is left out
    changes a sum by about 1, a hundred times the bound."""
    from tnn_b200.ops import raw
    torch.manual_seed(0)
    x, out = _rand(m, n), torch.zeros(n, device="cuda")
    raw.colsum_accum(x, out)
    rows, blocks = _colsum_rows(m, n)
    x = x.double()
    assert bool(((out.double() - x.sum(0)).abs() <= (rows // 32 + 32 + blocks) * 2.0 ** -24 * x.square().sum(0).sqrt()).all())


@pytest.mark.parametrize("m,n", [(1, 8), (129, 64), (65535, 64), (65536, 64), (70001, 8), (70001, 72)])
def test_colsum_last_rows(m, n):
    """Only the last row of each block and of the matrix holds anything, whole numbers whose sums are exact."""
    from tnn_b200.ops import raw
    rows, blocks = _colsum_rows(m, n)
    x, out = torch.zeros(m, n, dtype=BF, device="cuda"), torch.zeros(n, device="cuda")
    ends = torch.tensor([min(m, (k + 1) * rows) - 1 for k in range(blocks)], device="cuda")
    x[ends] = (1 + torch.arange(blocks, device="cuda") % 5).to(BF)[:, None] * (1 + torch.arange(n, device="cuda") % 3).to(BF)
    raw.colsum_accum(x, out)
    assert torch.equal(out.double(), x.double().sum(0))


@pytest.mark.parametrize("b,h,s,d", [(1, 1, 1, 8), (2, 3, 33, 32), (3, 2, 130, 48), (2, 4, 96, 80), (2, 2, 257, 96), (1, 3, 200, 128), (2, 1, 64, 136)])
@pytest.mark.parametrize("causal", [True, False])
def test_attention_heads_in_place(b, h, s, d, causal, monkeypatch):
    """Head sizes without a flash kernel, also when the heads are taken in groups that cut through a sequence, and from a
    buffer that starts off a 16-byte boundary. Probabilities and their gradients pass through bf16 (2**-9 relative each)
    before the second product: bound 2**-7 of the largest value."""
    from tnn_b200.ops import raw
    torch.manual_seed(s)
    qkv, do = _rand(b * s, 3 * h * d), _rand(b * s, h * d)
    orf, lrf = raw.attn_fwd(qkv.cpu(), b, s, h, d, causal, d ** -0.5)
    drf = raw.attn_bwd(qkv.cpu(), orf, do.cpu(), lrf, b, s, h, d, causal, d ** -0.5)
    close = lambda x, y: float((x.cpu().float() - y.float()).abs().max()) <= 2.0 ** -7 * max(1.0, float(y.float().abs().max()))
    for group in (None, 2):
        if group:
            monkeypatch.setattr(raw, "_group", lambda BH, S: min(BH, group))
            odd = torch.empty(qkv.numel() + 1, dtype=BF, device="cuda")[1:].view_as(qkv)
            qkv = odd.copy_(qkv)
        o, lse = raw.attn_fwd(qkv, b, s, h, d, causal, d ** -0.5)
        assert close(o, orf) and torch.allclose(lse.cpu(), lrf, rtol=0, atol=1e-3)
        assert close(raw.attn_bwd(qkv, o, do, lse, b, s, h, d, causal, d ** -0.5), drf)


def test_attention_backward_with_an_fp32_output():
    """The output is only multiplied with its gradient: kept in fp32 it gives the same result as the bf16 values it holds, but
    for the order of a sum of 40 products (2**-18 of its terms), which a bf16 rounding (2**-8) covers."""
    from tnn_b200.ops import raw
    torch.manual_seed(0)
    b, h, s, d = 2, 3, 70, 40
    qkv, do = _rand(b * s, 3 * h * d), _rand(b * s, h * d)
    o, lse = raw.attn_fwd(qkv, b, s, h, d, True, d ** -0.5)
    ref = raw.attn_bwd(qkv, o, do, lse, b, s, h, d, True, d ** -0.5).float()
    got = raw.attn_bwd(qkv, o.float(), do, lse, b, s, h, d, True, d ** -0.5).float()
    assert torch.allclose(got, ref, rtol=2.0 ** -7, atol=2.0 ** -8 * float(ref.abs().max()))


@pytest.mark.parametrize("g,m,n,k", [(3, 5, 7, 64), (2, 130, 33, 72), (1, 128, 256, 8)])
def test_batched_gemm_odd_outputs(g, m, n, k):
    from tnn_b200.ops.gemm import gemm_batched
    torch.manual_seed(0)
    a, b = _rand(g, m, k), _rand(g, n, k)
    out = gemm_batched(a, b, out_dtype=torch.float32)
    ref = a.double() @ b.double().transpose(1, 2)
    assert float((out.double() - ref).abs().max()) <= k * 2.0 ** -22 * float((a.double().abs() @ b.double().abs().transpose(1, 2)).max())


@pytest.mark.parametrize("n,pitch,off,dtype", [(31, 40, 1, BF), (8, 8, 3, BF), (31, 32, 1, torch.float32), (40, 43, 1, BF), (33, 47, 3, torch.float32)])
def test_batched_gemm_outputs_off_a_vector(n, pitch, off, dtype):
    """Outputs that start off a 16-byte boundary: narrower than the groups of 32 columns that are stored as vectors, or with
    a pitch that rules vectors out. Nothing beside them is written."""
    from tnn_b200.ops.gemm import gemm_batched
    torch.manual_seed(0)
    a, b = _rand(3, 20, 64), _rand(3, n, 64)
    buf = torch.full((3 * 20 * pitch + 8,), 7.0, dtype=dtype, device="cuda")
    out = buf[off:off + 3 * 20 * pitch].view(3, 20, pitch)[:, :, :n]
    gemm_batched(a, b, out=out)
    ref = a.double() @ b.double().transpose(1, 2)
    assert torch.allclose(out.double(), ref, rtol=2.0 ** -8, atol=1e-4)
    out.fill_(7.0)
    assert bool((buf == 7).all())


@pytest.mark.parametrize("n,pitch,off,dtype", [(32, 40, 1, BF), (64, 64, 1, torch.float32)])
def test_batched_gemm_refuses_what_it_cannot_store(n, pitch, off, dtype):
    from tnn_b200.ops.gemm import gemm_batched
    out = torch.empty(20 * pitch + 8, dtype=dtype, device="cuda")[off:off + 20 * pitch].view(1, 20, pitch)[:, :, :n]
    with pytest.raises(RuntimeError):
        gemm_batched(_rand(1, 20, 64), _rand(1, n, 64), out=out)


@pytest.mark.parametrize("heads,seqs,first,count", [(1, 1, 0, 1), (3, 2, 0, 6), (3, 4, 2, 5), (2, 3, 5, 1)])
@pytest.mark.parametrize("m,n,k", [(40, 24, 72), (130, 264, 64), (5, 8, 136)])
@pytest.mark.parametrize("a_t,b_t,dtype", [(False, False, BF), (False, True, torch.float32), (True, True, BF)])
def test_products_of_packed_heads(heads, seqs, first, count, m, n, k, a_t, b_t, dtype):
    """Heads read from and written into packed [sequence, row, head, column] tensors, from any head on: the items asked for
    and nothing else. fp32 sums of at most 136 products, rounded to the output's type."""
    from tnn_b200.ops.gemm import Heads, gemm_heads
    if (a_t and m % 8) or (b_t and n % 8):
        pytest.skip("operand pitch")
    torch.manual_seed(0)

    def packed(r, c):
        t = _rand(seqs, r, heads, c)
        return t, Heads(t.view(seqs * r, heads * c), 0, heads * c, heads, seqs, first, c, r * heads * c)

    (a, ha), (b, hb) = packed(*((k, m) if a_t else (m, k))), packed(*((k, n) if b_t else (n, k)))
    out = torch.full((seqs, m, heads, n), 7.0, dtype=dtype, device="cuda")
    gemm_heads(ha, hb, Heads(out.view(seqs * m, heads * n), 0, heads * n, heads, seqs, first, n, m * heads * n), m, n, k, count,
               a_t=a_t, b_t=b_t)
    ref = torch.full((seqs, m, heads, n), 7.0, dtype=torch.float64, device="cuda")
    for i in range(first, first + count):
        x, y = a[i // heads, :, i % heads].double(), b[i // heads, :, i % heads].double()
        ref[i // heads, :, i % heads] = (x.t() if a_t else x) @ (y if b_t else y.t())
    assert torch.allclose(out.double(), ref, rtol=2.0 ** -8 if dtype == BF else 0, atol=k * 2.0 ** -20)


def test_packed_heads_that_are_refused():
    """Layouts outside the tensor, pitches and addresses that the copies cannot take: an error before any launch."""
    from tnn_b200.ops.gemm import Heads, gemm_heads
    t = _rand(64, 96)
    good = lambda **kw: Heads(*[{**dict(t=t, offset=0, ld=96, heads=3, seqs=2, first=0, stride_h=32, stride_b=32 * 96), **kw}[x]
                                for x in ("t", "offset", "ld", "heads", "seqs", "first", "stride_h", "stride_b")])
    out = lambda **kw: good(t=torch.empty(64, 96, dtype=BF, device="cuda"), **kw)
    gemm_heads(good(), good(), out(), 32, 32, 32, 6)
    for bad in (dict(first=1), dict(first=-1), dict(heads=0), dict(seqs=1), dict(ld=92), dict(stride_h=36), dict(stride_b=3076), dict(offset=4)):
        with pytest.raises(RuntimeError):
            gemm_heads(good(**bad), good(), out(), 32, 32, 32, 6)
        with pytest.raises(RuntimeError):
            gemm_heads(good(), good(**bad), out(), 32, 32, 32, 6)
    for bad in (dict(first=1), dict(heads=0), dict(seqs=1), dict(stride_h=36), dict(stride_b=3076), dict(offset=4)):
        with pytest.raises(RuntimeError):
            gemm_heads(good(), good(), out(**bad), 32, 32, 32, 6)


@pytest.mark.parametrize("m,n,k", [(129, 129, 64), (1218, 256, 72), (1536, 1536, 200), (1664, 1537, 64), (4736, 256, 136), (4737, 1024, 64),
                                   (300, 4000, 1000)])
@pytest.mark.parametrize("a_t,b_t", [(False, False), (False, True)])
def test_gemm_one_wave_shapes(m, n, k, a_t, b_t):
    """Around the tile counts at which the kernel changes (148 tiles of 128 x 128 or 128 x 256): the same product, bit for
    bit, as every kernel gives when it is forced, and a bf16 rounding (2**-8) from the fp64 one."""
    from tnn_b200.ops.gemm import gemm
    torch.manual_seed(0)
    a, b = _rand(m, k), (_rand(k, n) if b_t else _rand(n, k))
    bias, res = _rand(n), _rand(m, (n + 7) // 8 * 8)[:, :n]
    out = lambda: torch.empty(m, (n + 7) // 8 * 8, dtype=BF, device="cuda")[:, :n]
    if k % 8 or (b_t and n % 8):
        pytest.skip("operand pitch")
    y = gemm(a, b, b_t=b_t, bias=bias, residual=res, out=out())
    for bn in (128, 256, 512):
        assert torch.equal(y, gemm(a, b, b_t=b_t, bias=bias, residual=res, out=out(), force_bn=bn))
    ref = a.double() @ (b.double() if b_t else b.double().t()) + bias.double() + res.double()
    assert torch.allclose(y.double(), ref, rtol=2.0 ** -8, atol=2.0 ** -8)


def _bn_block_sums(v, per_sm):
    """Sum of ``v [M, C]`` over its rows in the order of the batch-norm kernels: a row lane adds every 256 / cl-th row of its
    block, the block adds its row lanes one after another, all in fp32; the blocks are added in fp64."""
    m, c = v.shape
    cl = 32
    while cl > c // 8:
        cl //= 2
    gy = -(-per_sm * 148 // (-(-(c // 8) // cl)))
    lanes = 256 // cl
    rpb = max(-(-m // gy), 4 * lanes)
    total = torch.zeros(c, dtype=torch.float64, device=v.device)
    for r0 in range(0, m, rpb):
        rows = v[r0:min(m, r0 + rpb)]
        part = torch.zeros(lanes, c, device=v.device)
        for j in range(0, rows.shape[0], lanes):
            part[:rows[j:j + lanes].shape[0]] += rows[j:j + lanes]
        acc = torch.zeros(c, device=v.device)
        for lane in part:
            acc = acc + lane
        total += acc.double()
    return total


@pytest.mark.parametrize("m,c", [(300, 8), (1029, 24), (4096, 64), (3137, 128), (2000, 200), (777, 512), (5, 1024)])
def test_batchnorm_sum_order(m, c):
    """Statistics bit for bit as the sums in the kernels' stated order give them: an ulp of a mean is enough to move the
    gradients of a deep stack of layers."""
    from tnn_b200.ops import raw
    torch.manual_seed(m)
    x, dy = _rand(m, c) + 0.3, _rand(m, c)
    run_mean, run_var = torch.zeros(c, device="cuda"), torch.zeros(c, device="cuda")
    _, mean, rstd = raw.batchnorm_fwd_train(x, None, None, run_mean, run_var, 1e-5, 1.0, False)
    ref = _bn_block_sums(x.float(), 3) / m
    var = (_bn_block_sums(x.float().square(), 3) / m - ref * ref).float()
    assert torch.equal(mean, ref.float())
    assert torch.equal(run_var, var * torch.tensor(m / (m - 1), device="cuda"))
    dgamma, dbeta = torch.zeros(c, device="cuda"), torch.zeros(c, device="cuda")
    raw.batchnorm_bwd(dy, x, None, mean, rstd, torch.ones(c, dtype=BF, device="cuda"), dgamma, dbeta, False)
    assert torch.equal(dbeta, _bn_block_sums(dy.float(), 2).float())


def _captured(fn):
    """``fn`` in a CUDA graph, where every launch is a plain one, and its outputs."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        fn()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = fn()
    return graph, out


def _check_chain(fn, inputs, exact):
    """Launches one by one, each of which may be set up while the one before still writes, against the same launches in
    plain order: new values in the same buffers every time. ``exact`` outputs bit for bit; the others are sums of
    fp32 adds in the order in which blocks finish, a few ulps apart."""
    graph, plain = _captured(fn)
    for trial in range(25):
        torch.manual_seed(trial)
        for t in inputs:
            t.copy_(torch.randn(t.shape, device="cuda") * (1 + trial % 3))
        early = fn()
        graph.replay()
        for k, (a, b) in enumerate(zip(early, plain)):
            if k in exact:
                assert torch.equal(a, b), (trial, k)
            else:
                assert float((a.float() - b.float()).norm()) <= 2e-6 * float(b.float().norm()), (trial, k)


@pytest.mark.parametrize("rows,width", [(64, 256), (1500, 768), (4100, 512)])
def test_chain_of_dense_layers(rows, width):
    from tnn_b200.ops import raw
    from tnn_b200.ops.gemm import gemm
    x, w1, w2 = _rand(rows, width), _rand(width, width, scale=width ** -0.5), _rand(width, width, scale=width ** -0.5)
    g, b = _rand(width), _rand(width)

    def chain():
        h = gemm(x, w1, bias=b)
        s, h, mean, rstd = raw.layernorm_fwd(x, h, g, b, 1e-5, 0.1, 3)
        y = gemm(h, w2, bias=b, residual=s)
        dg, db, dbias = (torch.zeros(width, device="cuda") for _ in range(3))
        dx, dd = raw.layernorm_bwd(y, s, mean, rstd, g, x, True, 0.1, 3, dg, db, dbias=dbias)
        dw = torch.zeros(width, width, device="cuda")
        gemm(dd, x, a_t=True, b_t=True, out=dw, atomic=True)
        col = torch.zeros(width, device="cuda")
        raw.colsum_accum(dd, col)
        return s, h, mean, rstd, y, dx, dd, dg, db, dbias, dw, col

    _check_chain(chain, (x, w1, w2, g, b), range(7))


@pytest.mark.parametrize("b,s,h,d", [(2, 333, 3, 64), (1, 1024, 12, 64), (2, 130, 2, 96)])
def test_chain_around_attention(b, s, h, d):
    from tnn_b200.ops import raw
    from tnn_b200.ops.gemm import gemm
    e = h * d
    x, w, do = _rand(b * s, e), _rand(3 * e, e), _rand(b * s, e)

    def chain():
        _, n, _, _ = raw.layernorm_fwd(x, None, None, None, 1e-5)
        qkv = gemm(n, w)
        o, lse = raw.attn_fwd(qkv, b, s, h, d, True, 1.0 / d)
        d2 = gemm(do, w[:e])
        dqkv = raw.attn_bwd(qkv, o, d2, lse, b, s, h, d, True, 1.0 / d)
        return n, qkv, o, lse, d2, dqkv[:, e:].contiguous(), gemm(dqkv[:, e:], w[e:], b_t=True)

    _check_chain(chain, (x, w, do), range(7))


@pytest.mark.parametrize("n,hw,c", [(2, 9, 64), (16, 28, 128)])
def test_chain_around_batchnorm(n, hw, c):
    """The sums of the statistics are added in fp64 in the order in which blocks finish: equal after rounding to fp32 but for
    a chance of about 1e-8 per channel."""
    from tnn_b200.ops import raw
    x, w, dy = _rand(n, hw, hw, c), _rand(c, 3, 3, c, scale=c ** -0.5), _rand(n, hw, hw, c)
    g, b = _rand(c), _rand(c)
    rm, rv = torch.zeros(c, device="cuda"), torch.ones(c, device="cuda")

    def chain():
        y = raw.conv2d_fwd(x, w, None, (1, 1), (1, 1))
        z, mean, rstd = raw.batchnorm_fwd_train(y, g, b, rm, rv, 1e-5, 0.0, True)
        u = raw.conv2d_fwd(z, w, None, (1, 1), (1, 1))
        dg, db = torch.zeros(c, device="cuda"), torch.zeros(c, device="cuda")
        dz = raw.conv2d_dgrad(dy, w, tuple(z.shape), (1, 1), (1, 1))
        dyy = raw.batchnorm_bwd(dz, y, z, mean, rstd, g, dg, db, True, beta=b)
        dx = raw.conv2d_dgrad(dyy, w, tuple(x.shape), (1, 1), (1, 1))
        return y, z, mean, rstd, u, dz, dyy, dx, dg, db

    _check_chain(chain, (x, w, dy, g, b), range(10))


def test_batchnorm_mean_is_the_quotient():
    """The sum of 49 rows over 49 is half way between two fp32 numbers; times 1 / 49 in fp64 it is not. One block has the
    large values, the other the small one, so that the sum is exact."""
    from tnn_b200.ops import raw
    c = 2048
    x = torch.zeros(49, c, dtype=BF, device="cuda")
    x[3], x[20], x[40] = 48 * 2.0 ** 25, 2.0 ** 25, -49
    run_mean, run_var = torch.zeros(c, device="cuda"), torch.zeros(c, device="cuda")
    _, mean, _ = raw.batchnorm_fwd_train(x, None, None, run_mean, run_var, 1e-5, 1.0, False)
    assert bool((mean == 2.0 ** 25).all())
