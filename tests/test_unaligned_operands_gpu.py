"""Dense views that do not start on a 16-byte boundary: what reads 16 bytes at a time refuses them on the host, and what has
another way declines them."""
import pytest
import torch


def _shifted(t):
    """The same values, one element behind an aligned address."""
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    flat[1:] = t.flatten()
    return flat[1:].view(t.shape)


@pytest.mark.gpu
def test_unaligned_operands_are_declined_or_refused():
    from zorse_b200.ops import sm100 as k
    from zorse_b200.ops.api import get_ops

    ops = get_ops("sm100")
    rand = lambda *shape: torch.randn(*shape, device="cuda").bfloat16()
    k.status_word(0)
    dy, w, pre, gu = rand(300, 512), rand(512, 256), rand(300, 256), rand(300, 512)
    assert k._fast.act_linear_dgrad(dy, w, pre, 1) is not None and k._fast.act_linear_dgrad(dy, w, gu, 3) is not None
    assert k._fast.act_linear_dgrad(dy, w, _shifted(pre), 1) is None and k._fast.act_linear_dgrad(dy, w, _shifted(gu), 3) is None
    cs = ops.rope_table(300, 64, 1e4, "cuda")
    assert k._fast.linear_rope_fwd(dy, rand(512, 512), None, cs, 300, 4, 64) is not None
    assert k._fast.linear_rope_fwd(dy, rand(512, 512), None, _shifted(cs), 300, 4, 64) is None
    for call in (lambda: ops.act_linear_dgrad(dy, w, _shifted(pre), "relu"), lambda: ops.act_linear_dgrad(dy, w, _shifted(gu), "swiglu"),
                 lambda: ops.linear_rope_fwd(dy, rand(512, 512), None, _shifted(cs), 300, 4, 64),
                 lambda: ops.act_fwd(_shifted(pre), "relu"), lambda: k.act_fwd(_shifted(pre), 0),
                 lambda: ops.act_bwd(pre, _shifted(pre), "gelu"), lambda: ops.swiglu_fwd(_shifted(gu)),
                 lambda: ops.swiglu_bwd(gu, _shifted(pre)), lambda: ops.rope_(_shifted(gu), cs, 300, 4, 64)):
        with pytest.raises(k.KernelError, match="not 16-byte aligned"):
            call()
    torch.cuda.synchronize()
    k.check_status()
