"""Weight gradients that a schedule holds back: the same bits as without, layer by layer."""
import pytest
import torch

from zorse_b200.parallel.stage import DeferredWgrad


def test_a_flush_finishes_what_a_layer_had_collected_together():
    calls = []

    class Ops:
        def collect(self):
            return []

        def finish(self, later):
            calls.append(("finish", list(later)))

        def linear_wgrad(self, *a, **k):
            calls.append(("wgrad", *a))
            if k.get("later") is not None:
                k["later"].append(a[0])

    d = DeferredWgrad(Ops())
    d.active = True
    d.linear_wgrad("head")
    for layer in ("b1", "b0"):                       # equal (empty) lists, and yet two layers
        later = d.collect()
        d.linear_wgrad(layer + ".down", 0, 0, None, later=later)
        d.linear_wgrad(layer + ".up", 0, 0, None, later)
        d.finish(later)
    d.linear_wgrad("emb")
    assert calls == [("finish", []), ("finish", [])]
    d.active = False
    d.flush()
    assert calls[2:] == [("wgrad", "head"),
                         ("wgrad", "b1.down", 0, 0, None), ("wgrad", "b1.up", 0, 0, None), ("finish", ["b1.down", "b1.up"]),
                         ("wgrad", "b0.down", 0, 0, None), ("wgrad", "b0.up", 0, 0, None), ("finish", ["b0.down", "b0.up"]),
                         ("wgrad", "emb")]


@pytest.mark.gpu
@pytest.mark.parametrize("model,B,S", [("deepspeedbert_base", 8, 390), ("deepspeedgpt_test", 2, 509), ("tiny_llama", 5, 700),
                                       ("opt_125m", 2, 2048)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_held_back_gradients_of_blocks_are_the_same_bits(model, B, S, dt):
    """Two blocks, two microbatches, with and without biases, up to 4096 tokens."""
    from zorse_b200.models import registry
    from zorse_b200.ops import sm100 as k
    from zorse_b200.ops.api import get_ops

    ops, spec = get_ops("sm100"), registry.get_spec(model)
    blocks, buckets = [], []
    for i in range(2):
        blk = registry.make_block(spec)
        _, n = blk.layout()
        flat = torch.empty(n, dtype=torch.float32, device="cuda")
        blk.init_flat(flat, 3 + i)
        blocks.append((blk, flat.to(torch.bfloat16)))
    rand = lambda seed: torch.randn(B * S, spec.hidden, generator=torch.Generator().manual_seed(seed)).mul(0.5).bfloat16().cuda()
    for hold in (False, True):
        front = DeferredWgrad(ops)
        front.active = hold
        grads = [torch.zeros(w.numel(), dtype=dt, device="cuda") for _, w in blocks]
        for mb in range(2):
            x, dy, ctx, saved = rand(10 + mb), rand(20 + mb), {"B": B, "S": S}, [{}, {}]
            for (blk, w), g, sv in zip(blocks, grads, saved):
                blk.bind(w, g)
                x = blk.forward(x, ctx, ops, sv)
            for (blk, _), sv in zip(reversed(blocks), reversed(saved)):
                dy = blk.backward(dy, ctx, front, sv)
        front.active = False
        front.flush()
        buckets.append(grads)
    k.check_status()
    for a, b in zip(*buckets):
        assert bool(a.any()) and torch.equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("T,sizes", [(8192, [(512, 1376), (2752, 512), (512, 512), (1536, 512)]), (5600, [(768, 3072), (768, 768), (2304, 768)]),
                                     (6200, [(2048, 8192), (2048, 2048), (3072, 2048), (512, 512)]), (4600, [(4096, 3072), (6144, 4096), (512, 512)])])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_collected_products_are_cut_like_those_alone(T, sizes, dt):
    """Reductions long enough to be cut for most of these: the bits of each product alone, behind kernels that have just written
    the operands, twice into the same gradients."""
    from zorse_b200.ops import sm100 as k
    from zorse_b200.ops.api import get_ops

    ops = get_ops("sm100")
    rand = lambda *shape, seed: torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).bfloat16().cuda()
    src, xs = [rand(T, n, seed=i) for i, (n, _) in enumerate(sizes)], [rand(T, m, seed=10 + i) for i, (_, m) in enumerate(sizes)]
    got, want = ([torch.zeros(n, m, dtype=dt, device="cuda") for n, m in sizes] for _ in range(2))
    for _ in range(2):
        later, dys = ops.collect(), [ops.act_fwd(s, "relu") for s in src]
        for dy, x, g in zip(dys, xs, got):
            ops.linear_wgrad(dy, x, g, later=later)
        ops.finish(later)
        torch.cuda.synchronize()
        for dy, x, g in zip(dys, xs, want):
            ops.linear_wgrad(dy, x, g)
    k.check_status()
    assert any(k._gemm2_workspace(n, m, T, 0) for n, m in sizes[:-1])
    for g, w in zip(got, want):
        assert torch.equal(g, w)
