"""sm_100a kernels vs the fp32 PyTorch oracle (zorse_b200.ops.ref on CPU)."""
import math
import os

import pytest
import torch

pytestmark = pytest.mark.gpu

from zorse_b200.ops import ref


@pytest.fixture(scope="module")
def k():
    from zorse_b200.ops import sm100

    sm100.lib()
    return sm100


def _rand(*shape, scale=1.0, seed=0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(torch.bfloat16)


def _close(got, want, atol, rtol):
    got = got.float().cpu()
    want = want.float().cpu()
    err = (got - want).abs()
    tol = atol + rtol * want.abs()
    bad = (err > tol).float().mean().item()
    assert bad == 0.0, f"max err {err.max().item():.4g}, frac bad {bad:.4g}"


GEMM_SHAPES = [
    (128, 128, 64), (128, 256, 64), (256, 512, 256), (200, 136, 72), (1, 8, 8),
    (384, 1376, 512), (512, 512, 2048), (1000, 1000, 264),
]


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES)
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("bn", [128, 256])
def test_gemm_layouts(k, M, N, K, a_mn, b_mn, bn):
    if (a_mn and M % 8) or (b_mn and N % 8):
        pytest.skip("MN-major operand needs a 16-byte aligned row stride")
    a = _rand(M, K, seed=1)
    b = _rand(N, K, seed=2)
    want = a.float() @ b.float().t()
    ad = (a.t().contiguous() if a_mn else a).cuda()
    bd = (b.t().contiguous() if b_mn else b).cuda()
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    k.gemm(ad, bd, out, a_mn=a_mn, b_mn=b_mn, bn=bn)
    k.check_status()
    _close(out, want, atol=0.02 * math.sqrt(K), rtol=1e-2)


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (512, 768, 256), (300, 520, 200), (1024, 1280, 4096), (4096, 1024, 512)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_gemm_pair_kernel(k, M, N, K, a_mn, b_mn):
    if (a_mn and M % 8) or (b_mn and N % 8):
        pytest.skip("MN-major operand needs a 16-byte aligned row stride")
    a = _rand(M, K, seed=1)
    b = _rand(N, K, seed=2)
    want = a.float() @ b.float().t()
    ad = (a.t().contiguous() if a_mn else a).cuda()
    bd = (b.t().contiguous() if b_mn else b).cuda()
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    k.gemm(ad, bd, out, a_mn=a_mn, b_mn=b_mn, kernel="2cta")
    k.check_status()
    _close(out, want, atol=0.02 * math.sqrt(K), rtol=1e-2)
    acc = torch.ones(M, N, dtype=torch.float32, device="cuda")
    k.gemm(ad, bd, acc, a_mn=a_mn, b_mn=b_mn, kernel="2cta", accumulate=True)
    k.check_status()
    _close(acc, want + 1, atol=0.02 * math.sqrt(K), rtol=1e-2)


@pytest.mark.parametrize("M,N,K", [(264, 264, 72), (1018, 1544, 520), (520, 1088, 1000),          # 256 x 128 tiles
                                   (4104, 1032, 264), (2312, 1800, 2056)])                        # 256 x 256 tiles
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_gemm_pair_kernel_tile_widths(k, M, N, K, a_mn, b_mn):
    """Both tile widths of the pair kernel at ragged edges, bf16 and fp32 outputs, added to what is there.  Bounds: the
    operands are bf16 (exact products), so fp32 sums of K terms of unit variance are off by at most K * 2^-24 * sqrt(K)
    in the worst order; bf16 outputs add half an ulp, 2^-9 relative, doubled for the rounding of the comparison."""
    if (a_mn and M % 8) or (b_mn and N % 8):
        pytest.skip("MN-major operand needs a 16-byte aligned row stride")
    a, b = _rand(M, K, seed=1), _rand(N, K, seed=2)
    want = (a.cuda().double() @ b.cuda().double().t()).cpu()
    ad = (a.t().contiguous() if a_mn else a).cuda()
    bd = (b.t().contiguous() if b_mn else b).cuda()
    old = _rand(M, N, seed=3).cuda()
    for dtype in (torch.float32, torch.bfloat16):
        out = old.to(dtype, copy=True)
        k.gemm(ad, bd, out, a_mn=a_mn, b_mn=b_mn, kernel="2cta", accumulate=True)
        plain = torch.full((M, N), 7.0, dtype=dtype, device="cuda")
        k.gemm(ad, bd, plain, a_mn=a_mn, b_mn=b_mn, kernel="2cta")
        k.check_status()
        rtol = 0.0 if dtype == torch.float32 else 2.0 ** -8
        atol = K * math.sqrt(K) * 2.0 ** -24 + 1e-5
        _close(out, want + old.cpu().double(), atol=atol, rtol=rtol)
        _close(plain, want, atol=atol, rtol=rtol)


@pytest.mark.parametrize("M,N,K", [(300, 520, 8200), (264, 264, 8200), (256, 504, 20008), (1018, 504, 12296), (2500, 2040, 4104), (2560, 2048, 4096),
                                   (4096, 1288, 6152)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_gemm_split_last_wave(k, M, N, K, a_mn, b_mn):
    """Products whose last tiles are cut along K (all of them, or those behind one to two full waves), ragged in every
    direction, through every epilogue.  Bounds as in test_gemm_pair_kernel_tile_widths."""
    if (a_mn and M % 8) or (b_mn and N % 8):
        pytest.skip("MN-major operand needs a 16-byte aligned row stride")
    assert k._gemm2_workspace(M, N, K, 0) > 0
    a, b = _rand(M, K, seed=1).cuda(), _rand(N, K, seed=2).cuda()
    want = a.double() @ b.double().t()
    ad, bd = (a.t().contiguous() if a_mn else a), (b.t().contiguous() if b_mn else b)
    old, bias = _rand(M, N, seed=3).cuda(), _rand(N, seed=4).cuda()
    atol = K * math.sqrt(K) * 2.0 ** -24 + 1e-5
    for dtype, rtol in ((torch.float32, 0.0), (torch.bfloat16, 2.0 ** -8)):
        acc = old.to(dtype, copy=True)
        k.gemm(ad, bd, acc, a_mn=a_mn, b_mn=b_mn, kernel="2cta", accumulate=True)
        out = torch.full((M, N), 7.0, dtype=dtype, device="cuda")
        k.gemm(ad, bd, out, a_mn=a_mn, b_mn=b_mn, kernel="2cta")
        again = torch.full((M, N), 5.0, dtype=dtype, device="cuda")
        k.gemm(ad, bd, again, a_mn=a_mn, b_mn=b_mn, kernel="2cta")
        k.check_status()
        _close(acc, want + old.double(), atol=atol, rtol=rtol)
        _close(out, want, atol=atol, rtol=rtol)
        assert torch.equal(out, again)
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    k.gemm(ad, bd, out, a_mn=a_mn, b_mn=b_mn, kernel="2cta", bias=bias, addend=old)
    _close(out, want + bias.double() + old.double(), atol=atol, rtol=2.0 ** -8)
    k.gemm(ad, bd, out, a_mn=a_mn, b_mn=b_mn, kernel="2cta", bias=bias, act="relu")
    _close(out, (want + bias.double()).clamp(min=0), atol=atol, rtol=2.0 ** -8)
    k.check_status()


@pytest.mark.parametrize("M,K", [(300, 256), (1100, 2056), (300, 8200)])
@pytest.mark.parametrize("N", [1029, 1030, 1032, 1036])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gemm_writes_only_its_columns(k, M, N, K, dtype):
    """An output that is the left part of a wider matrix, its rows ending on a 16-byte boundary or not: what follows the last
    column, and the last row, stays as it was.  Plain, accumulated, with an addend; whole tiles and a split last wave."""
    a, b = _rand(M, K, seed=1).cuda(), _rand(N, K, seed=2).cuda()
    want = a.double() @ b.double().t()
    rtol = 0.0 if dtype == torch.float32 else 2.0 ** -8
    atol = K * math.sqrt(K) * 2.0 ** -24 + 1e-5
    add = _rand(M, 1040, seed=3).cuda()[:, :N]
    for kw, more in (({}, 0.0), ({"accumulate": True}, 3.0), ({"addend": add}, add.double())):
        full = torch.full((M + 1, 1048), 3.0, dtype=dtype, device="cuda")
        k.gemm(a, b, full[:M, :N], kernel="2cta", **kw)
        k.check_status()
        _close(full[:M, :N], want + more, atol=atol, rtol=rtol)
        assert bool((full[:M, N:] == 3.0).all()) and bool((full[M] == 3.0).all())


@pytest.mark.parametrize("M,N,K", [(300, 520, 8200), (2500, 2040, 4104)])
@pytest.mark.parametrize("room", [-16, -4, 0])
def test_gemm_split_stays_inside_its_workspace(k, M, N, K, room):
    """A workspace smaller than the plan needs is left alone (the product runs in whole tiles); one of the right size is
    not written past its end.  Guard bytes on both sides."""
    need = k._gemm2_workspace(M, N, K, 0)
    assert need > 0
    a, b = _rand(M, K, seed=1).cuda(), _rand(N, K, seed=2).cuda()
    out = torch.full((M, N), 7.0, device="cuda")
    buf = torch.full((need + 8192,), 0x5a, dtype=torch.uint8, device="cuda")
    rc = k.lib().zb_gemm2_split_bf16(a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, K, K, N, 0, 0, 0, 0, 0, k.GEMM_OUT_F32,
                                     buf.data_ptr() + 4096, need + room, k.status_word().data_ptr(), k._stream())
    k._check(rc, "gemm2_split")
    k.check_status()
    _close(out, a.double() @ b.double().t(), atol=K * math.sqrt(K) * 2.0 ** -24 + 1e-5, rtol=0.0)
    assert bool((buf[:4096] == 0x5a).all()) and bool((buf[4096 + need:] == 0x5a).all())
    assert bool((buf == 0x5a).all()) == (room < 0)


@pytest.mark.parametrize("M,N,K", [(512, 768, 256), (300, 520, 4104), (2500, 2040, 4104)])
def test_gemm_addend_forms(k, M, N, K):
    """Every form of addend the pair kernel accepts, with and without a split last wave: own rows, a row stride of its own,
    one row for all (stride 0), rows that are not 16-byte aligned, and the output itself.  Bounds as in
    test_gemm_pair_kernel_tile_widths."""
    a, b = _rand(M, K, seed=1).cuda(), _rand(N, K, seed=2).cuda()
    want = a.double() @ b.double().t()
    wide = _rand(M, N + 24, seed=3).cuda()
    atol = K * math.sqrt(K) * 2.0 ** -24 + 1e-5
    for add in (wide[:, :N].contiguous(), wide[:, 8:8 + N], wide[:1, :N].expand(M, N), wide[:, 3:3 + N]):
        for dtype, rtol in ((torch.float32, 0.0), (torch.bfloat16, 2.0 ** -8)):
            out = torch.full((M, N), 7.0, dtype=dtype, device="cuda")
            k.gemm(a, b, out, addend=add, kernel="2cta")
            _close(out, want + add.double(), atol=atol, rtol=rtol)
    out = wide[:, :N].contiguous()
    k.gemm(a, b, out, addend=out, kernel="2cta")
    _close(out, want + wide[:, :N].double(), atol=atol, rtol=2.0 ** -8)
    k.check_status()


def test_gemm_reads_a_bias_written_by_the_kernel_before(k):
    """The pair kernel starts under the tail of its predecessor; here that one writes the bias (other values each time, into
    the same place, from a kernel that lets its successor start at once).  fp32 outputs of exact small whole numbers."""
    M, N, K = 512, 2048, 256
    a = torch.ones(M, K, dtype=torch.bfloat16, device="cuda")
    b = torch.ones(N, K, dtype=torch.bfloat16, device="cuda")
    bias = torch.zeros(N, dtype=torch.bfloat16, device="cuda")
    dy = torch.ones(4096, N, dtype=torch.bfloat16, device="cuda") / 4096
    out = torch.empty(M, N, dtype=torch.float32, device="cuda")
    bad = torch.zeros((), dtype=torch.int64, device="cuda")
    for i in range(50):
        k.colsum_accumulate(dy, bias)                       # bias += 1
        k.gemm(a, b, out, bias=bias, kernel="2cta")
        bad += (out != K + i + 1).any()
    k.check_status()
    assert int(bad) == 0


def test_gemm_epilogues(k):
    M, N, K = 300, 520, 192
    a, b = _rand(M, K, seed=3), _rand(N, K, seed=4)
    bias, res = _rand(N, seed=5), _rand(M, N, seed=6)
    base = a.float() @ b.float().t()
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    k.gemm(a.cuda(), b.cuda(), out, bias=bias.cuda(), addend=res.cuda())
    _close(out, base + bias.float() + res.float(), atol=0.3, rtol=1e-2)
    # fp32 accumulate, twice
    acc = torch.zeros(M, N, dtype=torch.float32, device="cuda")
    k.gemm(a.cuda(), b.cuda(), acc, accumulate=True)
    k.gemm(a.cuda(), b.cuda(), acc, accumulate=True)
    _close(acc, 2 * base, atol=0.05, rtol=2e-3)
    # bf16 accumulate
    acc16 = res.cuda().clone()
    k.gemm(a.cuda(), b.cuda(), acc16, accumulate=True)
    _close(acc16, base + res.float(), atol=0.3, rtol=1e-2)
    # gelu after bias
    k.gemm(a.cuda(), b.cuda(), out, bias=bias.cuda(), act="gelu")
    _close(out, torch.nn.functional.gelu(base + bias.float(), approximate="tanh"), atol=0.3, rtol=1e-2)
    k.check_status()


def test_gemm_large_vs_fp32(k):
    M, N, K = 1024, 2048, 4096
    a, b = _rand(M, K, seed=7, scale=0.5), _rand(N, K, seed=8, scale=0.5)
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    k.gemm(a.cuda(), b.cuda(), out)
    k.check_status()
    want = a.double() @ b.double().t()
    _close(out, want, atol=0.15, rtol=1e-2)


@pytest.mark.parametrize("bwd_version", [1, 2])
@pytest.mark.parametrize("T,H", [(5, 512), (300, 4096), (64, 2048), (33, 5120), (1000, 4096)])
@pytest.mark.parametrize("ln", [False, True])
def test_norm(k, T, H, ln, bwd_version):
    x, w, b = _rand(T, H, seed=1), (_rand(H, seed=2) * 0.1 + 1).to(torch.bfloat16), _rand(H, seed=3, scale=0.1)
    dy, dres = _rand(T, H, seed=4), _rand(T, H, seed=5)
    xr = x.float().requires_grad_(True)
    wr = w.float().requires_grad_(True)
    br = b.float().requires_grad_(True)
    if ln:
        yr = torch.nn.functional.layer_norm(xr, (H,), wr, br, 1e-5)
    else:
        yr = xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + 1e-5) * wr
    yr.backward(dy.float())
    y, stats = k.norm_fwd(x.cuda(), w.cuda(), b.cuda() if ln else None, 1e-5, ln, version=bwd_version)
    _close(y, yr.detach(), atol=2e-2, rtol=1e-2)
    for gdt in (torch.float32, torch.bfloat16):
        dw = torch.ones(H, dtype=gdt, device="cuda")
        db = torch.ones(H, dtype=gdt, device="cuda")
        dx = k.norm_bwd(dy.cuda(), x.cuda(), w.cuda(), stats, dres.cuda(), dw, db if ln else None, ln,
                        version=bwd_version)
        _close(dx, xr.grad + dres.float(), atol=5e-2, rtol=2e-2)
        tol = 0.02 * math.sqrt(T) + (0.3 if gdt == torch.bfloat16 else 0)
        _close(dw, wr.grad + 1, atol=tol, rtol=2e-2)
        if ln:
            _close(db, br.grad + 1, atol=tol, rtol=2e-2)


@pytest.mark.parametrize("H", [8, 264, 512, 768, 1024, 1032, 1536, 2056, 3072, 4104, 6144, 8192])
@pytest.mark.parametrize("T", [1, 3, 2500])
@pytest.mark.parametrize("ln", [False, True])
def test_norm_row_widths(k, T, H, ln):
    """Every split of a CTA into rows and chunks per thread, with and without the residual gradient, against fp64.  Bounds:
    bf16 results to two ulp (2^-7) of values of a few units; weight gradients are fp32 sums of T products, each rounded
    to 2^-22 relative at worst (statistics included), of values below 30."""
    x, w, b = _rand(T, H, seed=1).cuda(), (_rand(H, seed=2) * 0.1 + 1).cuda(), _rand(H, seed=3, scale=0.1).cuda()
    dy, dres = _rand(T, H, seed=4).cuda(), _rand(T, H, seed=5).cuda()
    xr, wr, br = (t.double().requires_grad_(True) for t in (x, w, b))
    if ln:
        yr = torch.nn.functional.layer_norm(xr, (H,), wr, br, 1e-5)
    else:
        yr = xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + 1e-5) * wr
    yr.backward(dy.double())
    y, stats = k.norm_fwd(x, w, b if ln else None, 1e-5, ln)
    _close(y, yr.detach(), atol=1e-3, rtol=2.0 ** -7)
    for res in (None, dres):
        dw, db = torch.ones(H, device="cuda"), torch.ones(H, device="cuda")
        dx = k.norm_bwd(dy, x, w, stats, res, dw, db if ln else None, ln)
        _close(dx, xr.grad + (0 if res is None else res.double()), atol=4e-3, rtol=2.0 ** -7)
        _close(dw, wr.grad + 1, atol=T * 30 * 2.0 ** -22 + 1e-4, rtol=1e-5)
        if ln:
            _close(db, br.grad + 1, atol=T * 30 * 2.0 ** -22 + 1e-5, rtol=1e-5)


def test_colsum(k):
    dy = _rand(777, 520, seed=1)
    out = torch.zeros(520, dtype=torch.float32, device="cuda")
    k.colsum_accumulate(dy.cuda(), out)
    _close(out, dy.float().sum(0), atol=1e-2, rtol=1e-3)


@pytest.mark.parametrize("T", [1, 7, 9, 300, 4100, 8192, 8193, 9000])
@pytest.mark.parametrize("N,width", [(8, 8), (264, 264), (260, 260), (512, 1536), (4096, 4096), (4104, 4104), (5120, 5120)])
def test_colsum_sizes(k, T, N, width):
    """Sizes at the edges of the split over CTAs and rows and of the rule for one launch (8192 rows, 4096 columns); 260 columns take the kernel for unaligned rows, 512 of 1536 a
    strided matrix.  Bound: fp32 sums of T bf16 values of unit variance, any order; half an ulp of a bf16 result, doubled
    for the rounding of the comparison."""
    dy = _rand(T, width, seed=T + N).cuda()[:, :N]
    for dtype, rtol in ((torch.float32, 0.0), (torch.bfloat16, 2.0 ** -8)):
        out = torch.ones(N, dtype=dtype, device="cuda")
        k.colsum_accumulate(dy, out)
        _close(out, dy.double().sum(0) + 1, atol=T * math.sqrt(T) * 2.0 ** -24 + 2e-6, rtol=rtol)


@pytest.mark.parametrize("d,hq,hkv", [(64, 4, 2), (128, 2, 2)])
def test_rope(k, d, hq, hkv):
    B, S = 2, 96
    qkv = _rand(B * S, (hq + 2 * hkv) * d, seed=1)
    cs = ref.rope_table(S, d, 10000.0)
    want = ref.rope(qkv.float(), cs, S, hq + hkv, d)
    got = k.rope_(qkv.cuda().clone(), cs.cuda(), S, hq + hkv, d)
    _close(got, want, atol=2e-2, rtol=1e-2)
    wantb = ref.rope(qkv.float(), cs, S, hq + hkv, d, backward=True)
    gotb = k.rope_(qkv.cuda().clone(), cs.cuda(), S, hq + hkv, d, backward=True)
    _close(gotb, wantb, atol=2e-2, rtol=1e-2)


def test_swiglu_and_act(k):
    T, F_ = 130, 1376
    gu, dout = _rand(T, 2 * F_, seed=1), _rand(T, F_, seed=2)
    gr = gu.float().requires_grad_(True)
    o = torch.nn.functional.silu(gr[:, :F_]) * gr[:, F_:]
    o.backward(dout.float())
    _close(k.swiglu_fwd(gu.cuda()), o.detach(), atol=2e-2, rtol=1e-2)
    _close(k.swiglu_bwd(gu.cuda(), dout.cuda()), gr.grad, atol=3e-2, rtol=2e-2)
    for kind, name in ((k.ACT_GELU_TANH, "gelu"), (k.ACT_RELU, "relu"), (k.ACT_GELU_ERF, "gelu_erf")):
        x = _rand(T, F_, seed=3)
        xr = x.float().requires_grad_(True)
        y = ref.activation(xr, name)
        y.backward(dout.float())
        _close(k.act_fwd(x.cuda(), kind), y.detach(), atol=2e-2, rtol=1e-2)
        _close(k.act_bwd(x.cuda(), dout.cuda(), kind), xr.grad, atol=3e-2, rtol=2e-2)


@pytest.mark.parametrize("B,C,H,W,p", [(1, 3, 32, 32, 16), (2, 3, 24, 40, 8), (3, 1, 10, 6, 2), (2, 3, 28, 42, 14),
                                       (1, 3, 33, 35, 16)])
def test_patches(k, B, C, H, W, p):
    """Bit for bit the rows that unfolding the image gives, padded to a multiple of 8 columns; sizes with a rest, patches
    whose rows are no multiple of 8, an image that is not contiguous or not 16-byte aligned."""
    kdim = (C * p * p + 7) // 8 * 8
    for img in (torch.randn(B, C, H, W), torch.randn(B, C, W, H).transpose(2, 3), torch.randn(B * C * H * W + 1)[1:].view(B, C, H, W)):
        pt = torch.nn.functional.unfold(img[:, :, :H // p * p, :W // p * p], p, stride=p).transpose(1, 2).reshape(-1, C * p * p)
        want = torch.nn.functional.pad(pt, (0, kdim - C * p * p)).to(torch.bfloat16)
        dev = torch.empty(img.numel() + 1, device="cuda")[1:].view(B, C, H, W) if img.storage_offset() else None
        got = k.patches(img.cuda() if dev is None else dev.copy_(img), p, kdim)
        assert torch.equal(got.cpu(), want)


def test_embedding(k):
    V, H, S, B = 1000, 512, 16, 3
    table, pos = _rand(V, H, seed=1), _rand(S + 2, H, seed=2)
    ids = torch.randint(0, V, (B * S,), generator=torch.Generator().manual_seed(0))
    want = ref.embedding(ids, table.float(), pos.float(), S, 2)
    got = k.embedding_fwd(ids.cuda(), table.cuda(), pos.cuda(), S, 2)
    _close(got, want, atol=2e-2, rtol=1e-2)
    dout = _rand(B * S, H, seed=3)
    for gdt in (torch.float32, torch.bfloat16):
        dt = torch.zeros(V, H, dtype=gdt, device="cuda")
        dp = torch.zeros(S + 2, H, dtype=gdt, device="cuda")
        k.embedding_bwd(ids.cuda(), dout.cuda(), dt, dp, S, 2)
        wt = torch.zeros(V, H).index_add_(0, ids, dout.float())
        wp = torch.zeros(S + 2, H).index_add_(0, torch.arange(B * S) % S + 2, dout.float())
        _close(dt, wt, atol=5e-2, rtol=2e-2)
        _close(dp, wp, atol=5e-2, rtol=2e-2)


@pytest.mark.parametrize("offset", [0, 2])     # gradient tables 16-byte aligned, or not
@pytest.mark.parametrize("gdt", [torch.float32, torch.bfloat16])
def test_embedding_bwd_alignment(k, offset, gdt):
    """Both forms of the scatter-add; each id at most twice and small whole numbers, so every sum is exact."""
    V, H, S, B = 40, 264, 10, 2
    ids = torch.randperm(V, generator=torch.Generator().manual_seed(1))[:S].repeat(B)
    dout = torch.randint(-8, 9, (B * S, H), generator=torch.Generator().manual_seed(2)).to(torch.bfloat16)
    dt = torch.ones(V * H + offset, dtype=gdt, device="cuda")[offset:].view(V, H)
    dp = torch.ones((S + 2) * H + offset, dtype=gdt, device="cuda")[offset:].view(S + 2, H)
    k.embedding_bwd(ids.cuda(), dout.cuda(), dt, dp, S, 2)
    assert torch.equal(dt.float().cpu(), torch.ones(V, H).index_add_(0, ids, dout.float()))
    assert torch.equal(dp.float().cpu(), torch.ones(S + 2, H).index_add_(0, torch.arange(B * S) % S + 2, dout.float()))


@pytest.mark.parametrize("V", [4104, 32000, 1001])
def test_cross_entropy_in_place_gives_the_loss_of_the_logits(k, V):
    """The gradient is written over the logits by all threads of a row while one of them forms the loss.  Targets in the
    columns that are written first; the loss is that of separate buffers bit for bit, and so is the gradient."""
    T = 4096
    logits = (torch.randn(T, V, device="cuda", generator=torch.Generator("cuda").manual_seed(V)) * 2).to(torch.bfloat16)
    targets = (torch.arange(T, device="cuda") * 8) % min(V, 4096)
    targets[5] = -100
    grad = torch.empty_like(logits)
    want = k.cross_entropy(logits, targets, 0.5, grad)
    for _ in range(10):
        x = logits.clone()
        got = k.cross_entropy(x, targets, 0.5, x)
        assert torch.equal(got, want) and torch.equal(x, grad)


@pytest.mark.parametrize("T,V", [(9, 32000), (64, 50272), (4, 1001)])
def test_cross_entropy(k, T, V):
    logits = _rand(T, V, seed=1, scale=2.0)
    tg = torch.randint(0, V, (T,), generator=torch.Generator().manual_seed(1))
    lr = logits.float().requires_grad_(True)
    rows = torch.nn.functional.cross_entropy(lr, tg, reduction="none")
    (rows.sum() * 0.125).backward()
    d = torch.empty_like(logits, device="cuda")
    got = k.cross_entropy(logits.cuda(), tg.cuda(), 0.125, dlogits=d)
    _close(got, rows.detach(), atol=2e-3, rtol=1e-3)
    _close(d, lr.grad, atol=2e-3, rtol=2e-2)


@pytest.mark.parametrize("T,V", [(3, 8), (700, 16376), (290, 16384), (300, 16392), (310, 120000)])
def test_cross_entropy_against_64_bits(k, T, V):
    """A row of one piece, rows that end inside, at and just behind a round of pieces, both numbers of CTAs per SM, logits of
    minus infinity (whole rounds of a thread among them) and far below the others.  fp32 sums of V probabilities and two
    exponentials: 2^-16 of the loss' terms; the gradient half a unit in the last of 8 bits on top of 2^-16 of the largest."""
    logits = (torch.randn(T, V, device="cuda", generator=torch.Generator("cuda").manual_seed(V)) * 2).to(torch.bfloat16)
    if V > 8:
        logits[1, : V - 8] = -float("inf")
        logits[2, : V // 2] = -200.0
    tg = torch.randint(V - 8, V, (T,), device="cuda")
    d = torch.empty_like(logits)
    got = k.cross_entropy(logits, tg, 1.0, dlogits=d)
    want = torch.logsumexp(logits.double(), 1) - logits.double().gather(1, tg[:, None])[:, 0]
    torch.testing.assert_close(got.double(), want, rtol=2.0 ** -16, atol=2.0 ** -16 * 8)
    grad = torch.softmax(logits.double(), 1)
    grad.scatter_add_(1, tg[:, None], torch.full((T, 1), -1.0, device="cuda", dtype=torch.float64))
    torch.testing.assert_close(d.double(), grad, rtol=2.0 ** -8, atol=2.0 ** -16)


def test_cross_entropy_ignored_rows(k):
    """Rows whose target is the ignore index (-100) give zero loss and a zero gradient row."""
    T, V = 64, 1000
    logits = _rand(T, V, seed=3, scale=2.0)
    tg = torch.randint(0, V, (T,), generator=torch.Generator().manual_seed(3))
    tg[::4] = -100
    lr = logits.float().requires_grad_(True)
    rows = torch.nn.functional.cross_entropy(lr, tg, reduction="none", ignore_index=-100)
    rows.sum().backward()
    d = torch.empty_like(logits, device="cuda")
    got = k.cross_entropy(logits.cuda(), tg.cuda(), 1.0, dlogits=d)
    _close(got, rows.detach(), atol=2e-3, rtol=1e-3)
    _close(d, lr.grad, atol=2e-3, rtol=2e-2)
    assert float(d[::4].float().abs().max()) == 0.0 and float(got[::4].abs().max()) == 0.0


@pytest.mark.parametrize("gdt", [torch.float32, torch.bfloat16])
def test_adam(k, gdt):
    n = 100_003
    g0 = torch.Generator().manual_seed(0)
    p = torch.randn(n, generator=g0)
    grads = [torch.randn(n, generator=g0).to(gdt) for _ in range(3)]
    pr = p.clone().requires_grad_(True)
    opt = torch.optim.Adam([pr], lr=1e-3, betas=(0.9, 0.999), eps=1e-8)
    pd, m, v = p.cuda(), torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    p16 = torch.empty(n, dtype=torch.bfloat16, device="cuda")
    for step, g in enumerate(grads, 1):
        pr.grad = g.float() * 0.5
        opt.step()
        gd = g.cuda()
        k.adam_step(pd, m, v, gd, p16, lr=1e-3, beta1=0.9, beta2=0.999, eps=1e-8, weight_decay=0.0, step=step,
                    grad_scale=0.5, zero_grad=True)
        assert float(gd.float().abs().max()) == 0.0
    _close(pd, pr.detach(), atol=2e-6, rtol=1e-5)
    _close(p16, pr.detach(), atol=1e-2, rtol=1e-2)


ATTN_CASES = [
    (1, 300, 2, 1, 64, True, 0),
    (1, 640, 1, 1, 128, True, 200),
    # B, S, Hq, Hkv, D, causal, window
    (1, 128, 1, 1, 128, True, 0),
    (1, 128, 1, 1, 64, True, 0),
    (2, 256, 4, 2, 128, True, 0),
    (1, 384, 4, 1, 64, True, 0),
    (1, 200, 2, 2, 128, True, 0),
    (1, 512, 2, 1, 128, True, 192),
    (1, 256, 2, 2, 64, False, 0),
    (1, 1024, 2, 2, 128, True, 0),
]


# (version, flags)
FWD_VERSIONS = [(1, 0), (2, 0), (4, 0), (4, 1), (4, 2)]


@pytest.mark.parametrize("version,flags", FWD_VERSIONS)
@pytest.mark.parametrize("B,S,Hq,Hkv,D,causal,window", ATTN_CASES)
def test_flash_fwd(k, B, S, Hq, Hkv, D, causal, window, version, flags):
    qkv = _rand(B * S, (Hq + 2 * Hkv) * D, seed=1)
    want = ref.attention(qkv.float(), B, S, Hq, Hkv, D, causal, window)
    out, lse = k.flash_fwd(qkv.cuda(), B, S, Hq, Hkv, D, causal, window, version=version, flags=flags)
    k.check_status()
    _close(out, want, atol=2e-2, rtol=2e-2)
    # log-sum-exp against the oracle's scores
    x = qkv.float().reshape(B, S, Hq + 2 * Hkv, D)
    q = x[:, :, :Hq].permute(0, 2, 1, 3)
    kk = x[:, :, Hq:Hq + Hkv].permute(0, 2, 1, 3).repeat_interleave(Hq // Hkv, dim=1)
    s = (q @ kk.transpose(-1, -2)) / math.sqrt(D)
    i = torch.arange(S)[:, None]
    j = torch.arange(S)[None, :]
    mask = torch.ones(S, S, dtype=torch.bool)
    if causal:
        mask &= j <= i
    if window:
        mask &= (i - j) < window
    want_lse = torch.logsumexp(s.masked_fill(~mask, float("-inf")), dim=-1)
    _close(lse, want_lse, atol=2e-2, rtol=1e-2)


def test_flash_default_versions_on_a_large_problem(k):
    """The size-based default picks the two-tile forward here (20 heads x 8 pairs of query tiles, 160 CTAs);
    forward and backward defaults against the fp32 oracle, grouped-query heads, 2048 tokens."""
    B, S, Hq, Hkv, D = 1, 2048, 20, 4, 128
    assert k._auto_fwd_version(B, S, Hq, D) == 4
    qkv = _rand(B * S, (Hq + 2 * Hkv) * D, seed=11)
    do = _rand(B * S, Hq * D, seed=12)
    q = qkv.float().requires_grad_(True)
    want_o = ref.attention(q, B, S, Hq, Hkv, D, True, 0)
    (want,) = torch.autograd.grad(want_o, q, do.float())
    out, lse = k.flash_fwd(qkv.cuda(), B, S, Hq, Hkv, D, True, 0)
    got = k.flash_bwd(do.cuda(), qkv.cuda(), out, lse, B, S, Hq, Hkv, D, True, 0)
    k.check_status()
    _close(out, want_o.detach(), atol=2e-2, rtol=2e-2)
    _close(got, want, atol=4e-2, rtol=3e-2)


def test_flash_fwd_version_rule(k):
    """Both sides of both thresholds: CTAs of two query tiles, 64 at head size 128 and 148 at 64."""
    assert k._auto_fwd_version(1, 1000, 16, 128) == 4 and k._auto_fwd_version(1, 1024, 16, 128) == 4      # 64 CTAs
    assert k._auto_fwd_version(1, 768, 21, 128) == 1 and k._auto_fwd_version(9, 256, 7, 128) == 1         # 63
    assert k._auto_fwd_version(1, 1000, 37, 64) == 4 and k._auto_fwd_version(4, 256, 37, 64) == 4         # 148
    assert k._auto_fwd_version(1, 768, 49, 64) == 1 and k._auto_fwd_version(1, 1000, 16, 64) == 1         # 147, 64


@pytest.mark.parametrize("B,S,Hq,Hkv,causal,window", [(1, 1000, 16, 4, True, 0), (2, 600, 12, 12, True, 200), (1, 900, 20, 20, False, 0),
                                                      (3, 300, 16, 8, True, 0), (1, 1030, 25, 5, True, 0)])
def test_flash_fwd_default_at_few_ctas(k, B, S, Hq, Hkv, causal, window):
    """Head size 128 at 64 to 125 CTAs of two query tiles, where the default is the two-tile kernel: output and log-sum-exp
    through the default dispatch, ragged lengths, one of them (300 and 1030 tokens) with an empty or nearly empty second
    tile.  Bounds as in test_flash_fwd."""
    D = 128
    assert 64 <= B * Hq * ((S + 255) // 256) < 148 and k._auto_fwd_version(B, S, Hq, D) == 4
    qkv = _rand(B * S, (Hq + 2 * Hkv) * D, seed=51).cuda()
    out, lse = k.flash_fwd(qkv, B, S, Hq, Hkv, D, causal, window)
    one, lse1 = k.flash_fwd(qkv, B, S, Hq, Hkv, D, causal, window, version=1)
    k.check_status()
    _close(out, ref.attention(qkv.float(), B, S, Hq, Hkv, D, causal, window), atol=2e-2, rtol=2e-2)
    _close(lse, lse1, atol=1e-3, rtol=1e-4)       # both fp32 sums of the same exponentials, in another order
    _close(out, one, atol=2e-2, rtol=2e-2)


BWD_VERSIONS = [1, 2, 3]


@pytest.mark.parametrize("version", BWD_VERSIONS)
@pytest.mark.parametrize("B,S,Hq,Hkv,D,causal,window", ATTN_CASES)
def test_flash_bwd(k, B, S, Hq, Hkv, D, causal, window, version):
    qkv = _rand(B * S, (Hq + 2 * Hkv) * D, seed=1)
    do = _rand(B * S, Hq * D, seed=2)
    q = qkv.float().requires_grad_(True)
    want_o = ref.attention(q, B, S, Hq, Hkv, D, causal, window)
    (want,) = torch.autograd.grad(want_o, q, do.float())
    out, lse = k.flash_fwd(qkv.cuda(), B, S, Hq, Hkv, D, causal, window)
    for _ in range(2):  # second call checks that the scratch accumulator was left clean
        got = k.flash_bwd(do.cuda(), qkv.cuda(), out, lse, B, S, Hq, Hkv, D, causal, window, version=version)
    k.check_status()
    _close(got, want, atol=4e-2, rtol=3e-2)


@pytest.mark.parametrize("B,S,Hq,Hkv,causal,window", [(1, 130, 4, 1, True, 0), (1, 640, 8, 2, True, 0), (2, 600, 8, 2, True, 200),
                                                      (1, 300, 4, 2, False, 0), (1, 2100, 6, 3, True, 0), (3, 1300, 8, 4, False, 0),
                                                      (1, 1000, 12, 4, True, 0)])
@pytest.mark.parametrize("D", [64, 128])
def test_flash_bwd_grouped_heads(k, B, S, Hq, Hkv, D, causal, window):
    """Key tiles shared by clusters of one, two and four CTAs (by the number of tiles and the heads of a group), one to many
    query tiles per head.  Bounds as in test_flash_bwd; a second call gives the same bits (sums in rank order)."""
    qkv = _rand(B * S, (Hq + 2 * Hkv) * D, seed=21).cuda()
    do = _rand(B * S, Hq * D, seed=22).cuda()
    q = qkv.float().requires_grad_(True)
    want_o = ref.attention(q, B, S, Hq, Hkv, D, causal, window)
    (want,) = torch.autograd.grad(want_o, q, do.float())
    out, lse = k.flash_fwd(qkv, B, S, Hq, Hkv, D, causal, window)
    got = k.flash_bwd(do, qkv, out, lse, B, S, Hq, Hkv, D, causal, window)
    again = k.flash_bwd(do, qkv, out, lse, B, S, Hq, Hkv, D, causal, window)
    k.check_status()
    _close(got, want, atol=4e-2, rtol=3e-2)
    assert torch.equal(got, again)


@pytest.mark.parametrize("window", [300, 301, 4096, 2 ** 31 - 1, 2 ** 40])
@pytest.mark.parametrize("D", [64, 128])
def test_flash_window_no_shorter_than_the_sequence(k, D, window):
    """Such a window hides no key: outputs and gradients have the bits of the call without one, in every version."""
    B, S, Hq, Hkv = 1, 300, 4, 2
    qkv, do = _rand(B * S, (Hq + 2 * Hkv) * D, seed=41).cuda(), _rand(B * S, Hq * D, seed=42).cuda()
    for fwd, bwd in ((1, 2), (2, 3), (4, 3)):
        want, lse = k.flash_fwd(qkv, B, S, Hq, Hkv, D, True, 0, version=fwd)
        got, lse2 = k.flash_fwd(qkv, B, S, Hq, Hkv, D, True, window, version=fwd)
        assert torch.equal(got, want) and torch.equal(lse, lse2)
        g0 = k.flash_bwd(do, qkv, want, lse, B, S, Hq, Hkv, D, True, 0, version=bwd)
        g1 = k.flash_bwd(do, qkv, want, lse, B, S, Hq, Hkv, D, True, window, version=bwd)
        kv = slice(Hq * D, None) if bwd == 2 else slice(None)     # version 2 adds dQ with atomics
        assert torch.equal(g0[:, kv], g1[:, kv])
    k.check_status()


@pytest.mark.parametrize("B,S,Hq,Hkv", [(1, 640, 8, 2), (1, 2048, 32, 8), (1, 2560, 16, 8), (2, 1000, 12, 12)])
def test_flash_bwd_narrow_heads_beside_a_busy_stream(k, B, S, Hq, Hkv):
    """200 backward passes at head size 64 (clusters of four, two and one CTA per key tile, grouped and single heads) while
    an optimizer saturates memory on another stream: the issuer and the compute warps run against each other at other
    speeds than on an idle GPU.  Every pass gives the bits of the first, and no wait runs out."""
    D = 64
    qkv = _rand(B * S, (Hq + 2 * Hkv) * D, seed=31).cuda()
    do = _rand(B * S, Hq * D, seed=32).cuda()
    out, lse = k.flash_fwd(qkv, B, S, Hq, Hkv, D, True, 0)
    q = qkv.float().requires_grad_(True)
    (want,) = torch.autograd.grad(ref.attention(q, B, S, Hq, Hkv, D, True, 0), q, do.float())
    n = 1 << 25
    p, m, v = (torch.zeros(n, device="cuda") for _ in range(3))
    g, p16 = torch.ones(n, device="cuda"), torch.empty(n, dtype=torch.bfloat16, device="cuda")
    k.status_word()
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    first, bad = None, torch.zeros((), dtype=torch.int64, device="cuda")
    for i in range(200):
        if i % 2 == 0:      # about one update per two backward passes keeps the other stream busy throughout
            with torch.cuda.stream(side):
                k.adam_step(p, m, v, g, p16, lr=1e-3, beta1=0.9, beta2=0.999, eps=1e-8, weight_decay=0.0, step=i + 1)
        got = k.flash_bwd(do, qkv, out, lse, B, S, Hq, Hkv, D, True, 0)
        if first is None:
            first = got
        else:
            bad += (got.view(torch.int16) != first.view(torch.int16)).any()
    torch.cuda.synchronize()
    k.check_status()
    assert int(bad) == 0
    _close(first, want, atol=4e-2, rtol=3e-2)


def test_attention_traces_run(k):
    """The in-kernel phase traces terminate, leave the status word clean and record plausible clocks."""
    from zorse_b200.profiler import attn_trace

    for kern in ("fwd4", "bwd2"):
        attn_trace.main(["--kernel", kern, "--S", "1024", "--heads", "2", "--kv_heads", "2", "--ctas", "2"])
        k.check_status()


def test_a_wait_that_runs_out_reports_and_leaves_the_context_usable(k):
    """Failure detection on the device: a wait on a flag that nothing sets gives up after its (short)
    limit, the kernel returns, the host reads which wait it was, and the next launches work.  Nothing
    here faults, traps or spins without bound."""
    from zorse_b200.ops.sm100 import KernelError

    flags = torch.zeros(8, dtype=torch.int32, device="cuda")
    k.check_status()
    k.wait_flags(flags, 2, 0, 1, wait_seconds=0.05)        # flags[0..1] never reach epoch 1
    torch.cuda.synchronize()
    with pytest.raises(KernelError, match="status"):
        k.check_status()
    k.check_status()                                        # the word was cleared by the report
    flags[:2] = 1
    k.wait_flags(flags, 2, 0, 1, wait_seconds=0.05)        # satisfied at once
    k.check_status()
    x = torch.arange(8, device="cuda", dtype=torch.float32)
    assert float(x.sum().item()) == 28.0


@pytest.mark.parametrize("M,N,K,a_mn,b_mn", [(512, 768, 1024, True, True), (304, 520, 256, True, True),
                                              (512, 512, 512, False, False), (256, 1000, 384, False, True),
                                              (300, 1032, 2056, False, False)])
def test_accumulate_prefetch_gemm_matches_the_default(k, M, N, K, a_mn, b_mn):
    """The epilogue that requests the old C tile ahead of the accumulators by TMA gives the bits of the one that reads it
    from global memory, which rows that are not 16-byte aligned take (same arithmetic, same order), ragged edges included,
    twice in a row; columns behind the last one stay as they were."""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randn((K, M) if a_mn else (M, K), device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randn((K, N) if b_mn else (N, K), device="cuda", generator=g).to(torch.bfloat16)
    c0 = torch.randn(M, N, device="cuda", generator=g).to(torch.bfloat16)
    rows = torch.full((M, (N + 15) // 8 * 8), 7.0, dtype=torch.bfloat16, device="cuda")
    got = rows[:, :N].copy_(c0)
    want = torch.empty(M, N + 9 + N % 2, dtype=torch.bfloat16, device="cuda")[:, 3:3 + N].copy_(c0)
    assert want.stride(0) % 2 == 1 and got.stride(0) % 8 == 0
    for _ in range(2):
        k.gemm(a, b, want, a_mn=a_mn, b_mn=b_mn, accumulate=True, kernel="2cta")
        k.gemm(a, b, got, a_mn=a_mn, b_mn=b_mn, accumulate=True, kernel="2cta")
    k.check_status()
    assert torch.equal(got, want) and bool((rows[:, N:] == 7.0).all())


def test_checking_build_gives_the_same_results_and_a_clean_status():
    """The debug build (-DZB_DEBUG_BOUNDS=1: kernels verify tile coordinates, shard offsets and flag indices and
    report through the status word) runs a GEMM with ragged edges and attention forward + backward in a child
    process and must agree with the fp32 oracle with no check tripped."""
    import subprocess
    import sys

    code = r'''
import math, torch
from zorse_b200.ops import sm100 as k
assert str(k.lib()._name).endswith("libzorse_sm100_dbg.so"), k.lib()._name
g = torch.Generator().manual_seed(3)
rnd = lambda *s: (torch.randn(*s, generator=g) * 0.5).to(torch.bfloat16)
a, b = rnd(300, 520), rnd(1320, 520)
out = torch.empty(300, 1320, dtype=torch.bfloat16, device="cuda")
k.gemm(a.cuda(), b.cuda(), out)
k.check_status()
want = a.float() @ b.float().t()
assert (out.float().cpu() - want).abs().max() < 0.15
B, S, Hq, Hkv, D = 1, 600, 4, 2, 128
qkv, do = rnd(B * S, (Hq + 2 * Hkv) * D).cuda(), rnd(B * S, Hq * D).cuda()
o1, l1 = k.flash_fwd(qkv, B, S, Hq, Hkv, D, True, 0, version=1)
o4, l4 = k.flash_fwd(qkv, B, S, Hq, Hkv, D, True, 0, version=4)
d1 = k.flash_bwd(do, qkv, o1, l1, B, S, Hq, Hkv, D, True, 0, version=1)
d3 = k.flash_bwd(do, qkv, o1, l1, B, S, Hq, Hkv, D, True, 0, version=3)
k.check_status()
assert (o1.float() - o4.float()).abs().max() < 3e-2 and (d1.float() - d3.float()).abs().max() < 6e-2
print("CHECKING_BUILD_OK")
'''
    env = dict(os.environ, ZORSE_DEBUG_BOUNDS="1")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600, env=env,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0 and "CHECKING_BUILD_OK" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]
