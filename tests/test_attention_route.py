"""The op layer has one attention forward, whichever way a call takes: native, or by the wrapper what the native call declines."""
import pytest
import torch

from zorse_b200.ops import sm100 as k


@pytest.mark.parametrize("forced,entry", [(0, "zb_flash_fwd4"), (1, "zb_flash_fwd"), (4, "zb_flash_fwd4")])
@pytest.mark.parametrize("B,S,Hq,Hkv,D", [(1, 128, 4, 2, 64), (1, 256, 2, 2, 128), (4, 256, 37, 37, 64)])
def test_a_declined_call_gets_the_same_version(monkeypatch, forced, entry, B, S, Hq, Hkv, D):
    from zorse_b200.ops.api import Sm100Ops

    calls = []

    class Lib:
        def __getattr__(self, name):
            return lambda *a: calls.append(name) or 0

    monkeypatch.setattr(k, "_lib", Lib())
    monkeypatch.setattr(k, "_bf16", lambda t, name: None)
    monkeypatch.setattr(k, "status_word", lambda device=None: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(k, "_stream", lambda: None)
    monkeypatch.setattr(k, "ATTN_FWD_VERSION", forced)
    qkv = torch.zeros(B * S, (Hq + 2 * Hkv) * D, dtype=torch.bfloat16)       # (not on a GPU: declined)
    Sm100Ops().attn_fwd(qkv, B, S, Hq, Hkv, D)
    assert calls == [entry]


@pytest.mark.gpu
@pytest.mark.parametrize("B,S,Hq,Hkv,D", [(2, 128, 8, 2, 64), (2, 509, 8, 8, 64), (1, 700, 4, 2, 128), (1, 2048, 12, 12, 64)])
def test_the_first_call_on_a_device_gives_the_bits_of_the_next(B, S, Hq, Hkv, D):
    """The native call declines while the device's status word is unknown to it, as in the first call of a program."""
    from zorse_b200.ops.api import get_ops

    ops = get_ops("sm100")
    word = k.status_word(0)
    gen = torch.Generator().manual_seed(1)
    qkv = torch.randn(B * S, (Hq + 2 * Hkv) * D, generator=gen).bfloat16().cuda()
    later = ops.attn_fwd(qkv, B, S, Hq, Hkv, D)
    k._fast.set_status(0, 0)
    try:
        first = ops.attn_fwd(qkv, B, S, Hq, Hkv, D)
    finally:
        k._fast.set_status(0, word.data_ptr())
    k.check_status()
    assert torch.equal(first[0], later[0]) and torch.equal(first[1], later[1])
