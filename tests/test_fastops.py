"""The native calls of csrc/host/fastops.cpp against the wrappers of ops/sm100.py: same results, bit for bit, for every form
of argument they take, and everything else declined (the wrapper then takes or refuses it)."""
import pytest
import torch

from zorse_b200.ops import build
from zorse_b200.ops import sm100 as k


def _module():
    import importlib.util

    spec = importlib.util.spec_from_file_location("zorse_fastops", build.build_fast())
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_declines_what_is_not_on_a_gpu():
    m = _module()
    x, w = torch.zeros(4, 8, dtype=torch.bfloat16), torch.zeros(16, 8, dtype=torch.bfloat16)
    g, v = torch.zeros(16, 8), torch.zeros(8)
    calls = [(m.linear_fwd, (x, w, None, None)), (m.linear_dgrad, (x, x, None)), (m.linear_wgrad, (x, x, g, None, None)),
             (m.norm_fwd, (x, v, None, 1e-5, False)), (m.norm_bwd, (x, x, v, g, None, v, None, False, None)),
             (m.rope, (x, g, 4, 1, 8, False)), (m.swiglu_fwd, (x,)), (m.swiglu_bwd, (x, x)), (m.act_fwd, (x, 0)),
             (m.act_bwd, (x, x, 0)), (m.attn_fwd, (x, 1, 4, 1, 1, 64, True, 0, 1)),
             (m.attn_bwd, (x, x, x, g, 1, 4, 1, 1, 64, True, 0))]
    for fn, args in calls:
        assert fn(*args) is None
        assert fn(*[None] * len(args)) is None and fn(*["x"] * len(args)) is None
        with pytest.raises(TypeError):
            fn(*args, None)
    with pytest.raises(ValueError):
        m.init((1, 2), RuntimeError)


def test_entry_points_stand_in_the_order_of_the_table():
    """`init` fills the table by position: as many names as members, each member named like its entry point."""
    import re

    src = build.FAST_SRC.read_text()
    body = src[src.index("struct Entry {"):src.index("Entry lib;")]
    members = re.findall(r"\(\*(\w+)\)", body)
    names = [n[len("zb_"):] for n in k._FAST_ENTRIES]
    same = {"gemm_bf16": "gemm", "gemm2_bf16": "gemm2", "gemm2_split_bf16": "gemm2_split",
            "flash_bwd2_stats_floats": "flash_stats_floats"}
    assert [same.get(n, n) for n in names] == members
    # and each member takes what the C function takes
    for name, member in zip(k._FAST_ENTRIES, members):
        if name not in k._SIGNATURES:
            continue
        params = re.search(r"\(\*" + member + r"\)\(([^)]*)\)", body).group(1).split(",")
        kinds = "".join("p" if "*" in p or "cudaStream_t" in p else {"int": "i", "long": "l", "float": "f"}[p.split()[-1]]
                        for p in params)
        assert kinds == k._SIGNATURES[name], name


@pytest.fixture
def ops():
    from zorse_b200.ops.api import get_ops

    o = get_ops("sm100")
    k.status_word(0)
    return o


def _rand(*shape, seed=0, dtype=torch.bfloat16):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(dtype).cuda()


@pytest.mark.gpu
@pytest.mark.parametrize("T,K,N", [(300, 512, 768), (64, 264, 72), (1018, 512, 1544), (300, 8200, 520), (1, 8, 8)])
@pytest.mark.parametrize("wide", [False, True])      # rows of a wider matrix
def test_linear(ops, T, K, N, wide):
    pad = 8 if wide else 0
    x, w = _rand(T, K + pad, seed=1)[:, :K], _rand(N, K + pad, seed=2)[:, :K]
    b, add = _rand(N, seed=3), _rand(T, N + pad, seed=4)[:, :N]
    dy = _rand(T, N + pad, seed=5)[:, :N]

    def wrap(a, c, M, n, **kw):
        return k.gemm(a, c, torch.empty(M, n, dtype=torch.bfloat16, device="cuda"), **kw)

    before = k.launch_count()
    assert k._fast.linear_fwd(x, w, b, add) is not None and k.launch_count() > before
    for bias in (None, b):
        for addend in (None, add):
            assert torch.equal(ops.linear_fwd(x, w, bias, addend), wrap(x, w, T, N, bias=bias, addend=addend))
    addk = _rand(T, K, seed=6)
    for addend in (None, addk):
        assert torch.equal(ops.linear_dgrad(dy, w, addend), wrap(dy, w, T, K, b_mn=True, addend=addend))
    for dt in (torch.float32, torch.bfloat16):
        for bias in (False, True):
            g = [torch.ones(N, K, dtype=dt, device="cuda") for _ in range(2)]
            gb = [torch.ones(N, dtype=dt, device="cuda") for _ in range(2)]
            assert k._fast.linear_wgrad(dy, x, g[0], gb[0] if bias else None, None) is True
            k.gemm(dy, x, g[1], a_mn=True, b_mn=True, accumulate=True)
            if bias:
                k.colsum_accumulate(dy, gb[1])
            assert torch.equal(g[0], g[1]) and torch.equal(gb[0], gb[1])
    k.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("T,H", [(1, 8), (300, 512), (33, 1032), (5, 8192)])
@pytest.mark.parametrize("ln", [False, True])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_norms(ops, T, H, ln, dt):
    x, dy, w, b = _rand(T, H, seed=1), _rand(T, H, seed=2), _rand(H, seed=3), _rand(H, seed=4)
    y, st = ops.norm_fwd(x, w, b if ln else None, 1e-5, ln)
    y2, st2 = k.norm_fwd(x, w, b if ln else None, 1e-5, ln)
    assert torch.equal(y, y2) and torch.equal(st, st2)
    for dres in (None, _rand(T, H, seed=5)):
        g = [torch.ones(4, H, dtype=dt, device="cuda") for _ in range(1)][0]
        assert k._fast.norm_bwd(dy, x, w, st, dres, g[0], g[1] if ln else None, ln, None) is not None
        dx2 = k.norm_bwd(dy, x, w, st, dres, g[2], g[3] if ln else None, ln)
        assert torch.equal(g[0], g[2]) and torch.equal(g[1], g[3])
        assert torch.equal(ops.norm_bwd(dy, x, w, st, dres, g[0], g[1] if ln else None, ln), dx2)
    k.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("T,widths", [(1, [8, 512]), (7, [72, 64, 520]), (300, [768, 3072, 768, 2304]), (2503, [1032, 8, 200]),
                                      (4616, [768] * 6)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_finish_of_a_layer_in_one_launch(ops, T, widths, dt):
    """Bias gradients of matrices of several widths (one a slice of wider rows) and the gradients of two norms: fewer and more
    than fit one launch, against 64 bits, and the same bits each time.  Bounds: fp32 sums of T terms in chains of at most T / 256
    + 40 additions, of numbers whose absolute sum is `mass`; bf16 gradients round once more."""
    H = 512
    x, dyn, w = _rand(T, H, seed=1), _rand(T, H, seed=2), _rand(H, seed=3)
    _, st = k.norm_fwd(x, w, w, 1e-5, True)
    dys = [_rand(T, n + 8 * (i == 1), seed=10 + i)[:, :n] for i, n in enumerate(widths)]
    x16 = x[:, :16].contiguous()

    def run():
        later, outs = ops.collect(), [torch.ones(n, dtype=dt, device="cuda") for n in widths]
        gw = [torch.zeros(n, 16, dtype=dt, device="cuda") for n in widths]
        norm = [torch.ones(H, dtype=dt, device="cuda") for _ in range(4)]
        before = k.launch_count()
        for dy, g, o in zip(dys, gw, outs):
            ops.linear_wgrad(dy, x16, g, o, later=later)
        for i in (0, 2):
            ops.norm_bwd(dyn, x, w, st, None, norm[i], norm[i + 1], True, later)
        assert len(later) == len(widths) + 2 and all(bool((o == 1).all()) for o in outs + norm)
        ops.finish(later)
        assert not later and k.launch_count() - before == len(widths) + 2 + -(-(len(widths) + 4) // 8)
        return outs + norm

    got, again = run(), run()
    k.check_status()
    xh = (x.double() - st[:, :1].double()) * st[:, 1:].double()
    srcs = [d.double() for d in dys] + [dyn.double() * xh, dyn.double()] * 2
    for o, o2, src in zip(got, again, srcs):
        assert torch.equal(o, o2)
        mass = 1 + src.abs().sum(0)
        tol = mass * (T / 256 + 40) * 2.0 ** -24 + (0 if dt == torch.float32 else 2.0 ** -8) * (1 + src.sum(0)).abs()
        assert bool(((o.double() - 1 - src.sum(0)).abs() <= tol + 1e-6).all())


@pytest.mark.gpu
@pytest.mark.parametrize("T,sizes", [(300, [(1536, 512), (512, 512), (2048, 512), (512, 2048)]), (4616, [(2304, 768), (768, 768)]),
                                     (3072, [(768, 768)]), (8200, [(520, 264), (264, 520), (1032, 1000)]), (64, [(304, 256), (72, 512)])])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_weight_gradients_that_start_under_one_another(ops, T, sizes, dt):
    """A layer's products without a wait between them, behind a kernel that has just written their operands, several times into
    the same gradients: the bits of the same products one after the other (whole tiles: the same sums in the same order; the
    last one is cut along K as it would be alone), and bias gradients of operands written just before."""
    dys = [torch.zeros(T, n, dtype=torch.bfloat16, device="cuda") for n, _ in sizes]
    xs = [_rand(T, m, seed=20 + i) for i, (_, m) in enumerate(sizes)]
    fresh = [[_rand(T, n, seed=40 + 10 * r + i) for i, (n, _) in enumerate(sizes)] for r in range(3)]
    new = lambda *shape: [torch.zeros(*shape, dtype=dt, device="cuda") for _ in range(2)]
    gw, gb = [new(n, m) for n, m in sizes], [new(n) for n, _ in sizes]
    for r in range(3):
        for i, dy in enumerate(dys):
            k.lib().zb_act_fwd(fresh[r][i].data_ptr(), dy.data_ptr(), dy.numel(), 1, k._stream())   # relu, launched like a step's
        later = ops.collect()
        for i, dy in enumerate(dys):
            ops.linear_wgrad(dy, xs[i], gw[i][0], gb[i][0], later=later)
        ops.finish(later)
    for r in range(3):
        for i in range(len(sizes)):
            dy = fresh[r][i].clamp(min=0)
            torch.cuda.synchronize()
            if i + 1 < len(sizes) and T > 3000 and min(sizes[i]) >= 256:      # not cut along K there
                rc = k.lib().zb_gemm2_bf16(dy.data_ptr(), xs[i].data_ptr(), gw[i][1].data_ptr(), *sizes[i], T, sizes[i][0], sizes[i][1],
                                           sizes[i][1], 1, 1, 0, 0, 0, k.GEMM_ACCUMULATE | (k.GEMM_OUT_F32 if dt == torch.float32 else 0),
                                           0, k.status_word(0).data_ptr(), k._stream())
                k._check(rc, "gemm2")
            else:
                k.gemm(dy, xs[i], gw[i][1], a_mn=True, b_mn=True, accumulate=True)
            gb[i][1] += dy.double().sum(0).to(dt)
    k.check_status()
    for i in range(len(sizes)):
        assert torch.equal(gw[i][0], gw[i][1]), i
        torch.testing.assert_close(gb[i][0].double(), gb[i][1].double(), rtol=1e-5 if dt == torch.float32 else 2.0 ** -6, atol=1e-2)


@pytest.mark.gpu
@pytest.mark.parametrize("B,S,Hq,Hkv,D,causal,window", [(2, 150, 8, 8, 64, True, 0), (1, 600, 4, 2, 128, True, 200),
                                                        (3, 129, 2, 1, 64, False, 0), (1, 1, 1, 1, 128, True, 5)])
def test_attention(ops, B, S, Hq, Hkv, D, causal, window):
    """The backward's statistics live in memory as the allocator hands it out: their padding is written by the kernel (NaN in
    what the allocator will hand out next would show)."""
    qkv, do = _rand(B * S, (Hq + 2 * Hkv) * D, seed=1), _rand(B * S, Hq * D, seed=2)
    out, lse = k.flash_fwd(qkv, B, S, Hq, Hkv, D, causal, window, version=4)
    got = k._fast.attn_fwd(qkv, B, S, Hq, Hkv, D, causal, window, k.ATTN_FWD4_FLAGS)
    assert torch.equal(got[0], out) and torch.equal(got[1], lse)
    want = k.flash_bwd(do, qkv, out, lse, B, S, Hq, Hkv, D, causal, window)
    for _ in range(3):
        for n in (2 * B * Hq * ((S + 127) // 128 * 128), qkv.numel() // 2):
            torch.full((n,), float("nan"), device="cuda")
        assert torch.equal(k._fast.attn_bwd(do, qkv, out, lse, B, S, Hq, Hkv, D, causal, window), want)
    k.check_status()


@pytest.mark.gpu
def test_passes(ops):
    q, h = _rand(300, 1536, seed=1), _rand(300, 768, seed=2)
    cs = ops.rope_table(150, 64, 1e4, "cuda")
    for backward in (False, True):
        assert torch.equal(ops.rope_(q.clone(), cs, 150, 16, 64, backward), k.rope_(q.clone(), cs, 150, 16, 64, backward))
    assert torch.equal(ops.swiglu_fwd(q), k.swiglu_fwd(q)) and torch.equal(ops.swiglu_bwd(q, h), k.swiglu_bwd(q, h))
    for name, kind in (("gelu", 0), ("relu", 1), ("gelu_erf", 2)):
        assert torch.equal(ops.act_fwd(h, name), k.act_fwd(h, kind)) and torch.equal(ops.act_bwd(h, h + 1, name), k.act_bwd(h, h + 1, kind))


@pytest.mark.gpu
def test_what_is_declined_and_what_is_refused(ops):
    x, w = _rand(64, 512), _rand(256, 512)
    f = k._fast
    for args in ((x.float(), w, None, None), (x, w.t(), None, None), (x.t(), w, None, None), (x, w.cpu(), None, None),
                 (x[0], w, None, None), (x, w, w[0], None), (x, w, None, x), (x[:0], w, None, None)):
        assert f.linear_fwd(*args) is None
    with pytest.raises(AssertionError):
        ops.linear_fwd(x, w.t())
    with pytest.raises(TypeError):
        ops.linear_fwd(x.float(), w)
    with pytest.raises(k.KernelError, match="H=12 unsupported"):
        ops.norm_fwd(_rand(4, 12), _rand(12), None, 1e-5, False)

    class Marked(torch.Tensor):
        pass

    assert f.swiglu_fwd(_rand(8, 64).as_subclass(Marked)) is None
    assert f.rope(_rand(8, 64), torch.zeros(4, 64, device="cuda"), 8, 1, 64, False) is None      # a table of fewer positions
    out = torch.empty(8, 64, dtype=torch.bfloat16, device="cuda")
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):                       # launches follow the current stream
        a = _rand(4096, 4096, seed=7)
        for _ in range(20):
            a = ops.linear_fwd(a, _rand(4096, 4096, seed=8)) * 0.01
        b = ops.linear_fwd(a, w.repeat(1, 8))
    side.synchronize()
    assert torch.equal(b, ops.linear_fwd(a, w.repeat(1, 8))) and out.shape == (8, 64)


def _mlp_reference(x, w, b, act, pre=None, d=None):
    """The pre-activations and the activation in fp64, or the gradient of the pre-activations for `d`."""
    h = (x.double() @ w.double().t() + (0 if b is None else b.double())).bfloat16() if pre is None else pre
    h = h.double().requires_grad_(True)
    f = torch.nn.functional
    a = {"swiglu": lambda: f.silu(h[:, :h.shape[1] // 2]) * h[:, h.shape[1] // 2:], "relu": lambda: f.relu(h),
         "gelu": lambda: f.gelu(h, approximate="tanh"), "gelu_erf": lambda: f.gelu(h)}[act]()
    if d is None:
        return a.detach(), h.detach()
    return torch.autograd.grad(a, h, d.double())[0]


@pytest.mark.gpu
@pytest.mark.parametrize("T,K,F", [(256, 512, 256), (300, 512, 1376), (1018, 264, 520), (2500, 768, 3080), (520, 4104, 1032),
                                   (4104, 2048, 2056)])
@pytest.mark.parametrize("act", ["swiglu", "gelu", "relu", "gelu_erf"])
def test_activation_in_the_epilogue(ops, T, K, F, act):
    """Both directions at ragged edges of the tiles (rows, columns, columns of one half of a gated unit), both tile widths and
    both splits of shared memory (K below and from 2048 on).  The product is rounded to bf16 ahead of the activation, as a pass
    of its own would find it, and the result once more: 2^-8 of the value covers a flip of the first rounding (a slope of at
    most 1.13) and the second; the absolute part the same for values near a zero of the activation, whose argument is off by
    2^-9 of its size, and the fast exponentials and tanh (2^-11 of 1)."""
    rows = 2 * F if act == "swiglu" else F
    x, w = _rand(T, K, seed=1), (_rand(rows, K, seed=2).float() / K ** 0.5).bfloat16()
    b = None if act == "swiglu" else _rand(rows, seed=3)
    kind = {"gelu": 0, "relu": 1, "gelu_erf": 2, "swiglu": 3}[act]
    both, keep = k._fast.act_linear_fwd(x, w, b, kind, False), k._fast.act_linear_fwd(x, w, b, kind, True)
    assert both[1] is None and torch.equal(both[0], keep[0])
    a, pre = keep
    assert torch.equal(pre, ops.linear_fwd(x, w, b))
    plain = k.swiglu_fwd(pre) if act == "swiglu" else k.act_fwd(pre, kind)
    want, _ = _mlp_reference(x, w, b, act, pre=None)
    torch.testing.assert_close(a.double(), plain.double(), rtol=2.0 ** -7, atol=1e-6)
    torch.testing.assert_close(a.double(), want, rtol=2.0 ** -6, atol=0.04)
    down = (_rand(512, F, seed=4).float() / 512 ** 0.5).bfloat16()
    dy = _rand(T, 512, seed=5)
    got = k._fast.act_linear_dgrad(dy, down, pre, kind)
    da = ops.linear_dgrad(dy, down)
    plain = k.swiglu_bwd(pre, da) if act == "swiglu" else k.act_bwd(pre, da, kind)
    torch.testing.assert_close(got.double(), plain.double(), rtol=2.0 ** -7, atol=1e-6)
    torch.testing.assert_close(got.double(), _mlp_reference(x, w, b, act, pre=pre, d=da), rtol=2.0 ** -6, atol=0.02)
    k.check_status()


@pytest.mark.gpu
def test_activation_products_that_are_not_for_the_epilogue(ops):
    """Few rows, few or odd columns: declined, and the two calls they stand for give the result."""
    for T, K, F in ((255, 512, 512), (300, 512, 248), (300, 512, 516)):
        x, w = _rand(T, K, seed=1), (_rand(F, K, seed=2).float() / K ** 0.5).bfloat16()
        assert k._fast.act_linear_fwd(x, w, None, 1, True) is None
        if F % 8 == 0:
            a, pre = ops.act_linear_fwd(x, w, None, "relu", True)
            assert torch.equal(pre, ops.linear_fwd(x, w)) and torch.equal(a, pre.clamp(min=0))
            d = ops.act_linear_dgrad(_rand(T, 512, seed=3), _rand(512, F, seed=4), pre, "relu")
            assert d.shape == pre.shape
    x = _rand(300, 512)
    assert k._fast.act_linear_fwd(x, _rand(512, 512), _rand(512), 3, True) is None         # a gated unit with a bias
    assert k._fast.act_linear_dgrad(x, _rand(512, 512), _rand(300, 512), 3) is None        # pre-activations of half the width


@pytest.mark.gpu
@pytest.mark.parametrize("T,K,S", [(256, 256, 256), (301, 520, 43), (1030, 2048, 515), (2500, 768, 2500), (4104, 2056, 1026)])
@pytest.mark.parametrize("Hq,Hkv,d,bias", [(4, 4, 64, False), (5, 1, 64, True), (2, 1, 128, True), (9, 3, 128, False)])
def test_rotation_in_the_epilogue(ops, T, K, S, Hq, Hkv, d, bias):
    """Ragged rows and columns, rows that start again at position 0 inside a tile, value heads that stay as they are, both tile
    widths and both splits of shared memory.  The product is rounded ahead of the rotation, as the pass it stands for finds it:
    against that pass one flip of the second rounding (2^-7, or 2^-22 of the pair where its terms cancel); against 64 bits 2^-8
    of either of a pair, then 2^-8 of the result."""
    x, w = _rand(T, K, seed=1), (_rand((Hq + 2 * Hkv) * d, K, seed=2).float() / K ** 0.5).bfloat16()
    b = _rand((Hq + 2 * Hkv) * d, seed=3) if bias else None
    cs = ops.rope_table(S, d, 1e4, "cuda")
    got = k._fast.linear_rope_fwd(x, w, b, cs, S, Hq + Hkv, d)
    y = x.double() @ w.double().t() + (0 if b is None else b.double())
    c, sn = cs.double()[torch.arange(T, device="cuda") % S].view(T, 1, 2, d // 2).unbind(2)
    heads = y.view(T, -1, 2, d // 2)
    lo, hi = heads[:, :Hq + Hkv].unbind(2)
    rot = torch.stack((lo * c - hi * sn, hi * c + lo * sn), 2)
    want = torch.cat((rot, heads[:, Hq + Hkv:]), 1).reshape(T, -1)
    pair = heads.abs().sum(2, keepdim=True).expand(-1, -1, 2, -1).reshape(T, -1)
    two = ops.rope_(ops.linear_fwd(x, w, b), cs, S, Hq + Hkv, d)
    assert ((got.double() - two.double()).abs() <= 2.0 ** -7 * two.double().abs() + 2.0 ** -22 * pair).all()
    assert ((got.double() - want).abs() <= 2.0 ** -8 * 1.01 * (want.abs() + pair)).all()
    assert torch.equal(got.view(T, -1, d)[:, Hq + Hkv:], two.view(T, -1, d)[:, Hq + Hkv:])
    k.check_status()


@pytest.mark.gpu
def test_projections_whose_rotation_stays_a_pass(ops):
    """Few rows, heads of other widths, columns that are no whole heads, more heads than columns, a table for other heads or
    too few positions: declined; where the two calls take it, they give the result."""
    x, w = _rand(300, 512), _rand(512, 512, seed=2)
    cs = {d: ops.rope_table(300, d, 1e4, "cuda") for d in (32, 64, 128)}
    f = k._fast.linear_rope_fwd
    assert f(x[:255], w, None, cs[64], 300, 8, 64) is None and f(x, w[:248], None, cs[64], 300, 2, 64) is None
    assert f(x, w, None, cs[32], 300, 8, 32) is None and f(x, w, None, cs[64], 300, 9, 64) is None
    assert f(x, w[:320], None, cs[128], 300, 2, 128) is None
    assert f(x, w, None, cs[128], 300, 8, 64) is None and f(x, w, None, cs[64], 301, 8, 64) is None
    assert f(x, w, None, cs[64].bfloat16(), 300, 8, 64) is None
    assert torch.equal(ops.linear_rope_fwd(x, w, None, cs[32], 300, 8, 32), ops.rope_(ops.linear_fwd(x, w), cs[32], 300, 8, 32))


@pytest.mark.gpu
def test_gelu_erf_over_all_arguments(ops):
    """Every bf16 argument against 64 bits.  In fp32 the value is off by a few 2^-24 of itself (the tail is never a difference
    of larger numbers; the derivative has a zero near -0.75 and is off by a few 2^-24 there), so what is left is the rounding
    to bf16: half a unit of 8 bits, 2^-8 of the value at most."""
    x = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16).cuda()
    xd = x.double()
    phi = torch.exp(-xd * xd / 2) / (2 * torch.pi) ** 0.5
    cdf = 0.5 * torch.erfc(-xd / 2 ** 0.5)
    y, dy = k.act_fwd(x, 2), k.act_bwd(x, torch.ones_like(x), 2)
    for got, want in ((y, xd * cdf), (dy, cdf + xd * phi)):
        m = torch.isfinite(xd) & torch.isfinite(want) & (want.abs() > 1e-30)
        assert bool(((got.double() - want).abs()[m] <= (2.0 ** -8 + 1e-6) * want.abs()[m] + 2e-7 * (want.abs()[m] < 0.5)).all())
    at = lambda t, bits: float(t[bits])
    assert at(y, 0x7f80) == float("inf") and at(y, 0x0000) == 0.0 and at(y, 0x7f7f) == float(x[0x7f7f]) and at(y, 0xff7f) == 0.0
    assert torch.isnan(y[0x7fc0]) and torch.isnan(y[0xff80]) and torch.isnan(dy[0x7fc0])       # as before: -inf times 0
    assert at(dy, 0x0000) == 0.5 and at(dy, 0x7f7f) == 1.0 and at(dy, 0xff7f) == 0.0
