"""The erf GELU against 64 bits, argument by argument."""
import pytest
import torch


def _rounded(want):
    """64-bit values to the nearest bf16, ties to even (not by way of fp32, which would round twice)."""
    f = want.float()
    tie = (f.double() != want) & ((f.view(torch.int32) & 0xffff) == 0x8000)
    away = torch.where(want > f.double(), torch.full_like(f, float("inf")), torch.full_like(f, float("-inf")))
    return torch.where(tie, torch.nextafter(f, away), f).bfloat16()


@pytest.mark.gpu
def test_gelu_erf_is_the_rounded_value():
    """Every normal bf16 argument whose result is at least 2^-124 (numbers below 2^-126 are flushed, those of the derivative's
    exponential a little earlier)."""
    from zorse_b200.ops import sm100 as k

    x = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16).cuda()
    xd = x.double()
    cdf = 0.5 * torch.erfc(-xd / 2 ** 0.5)
    phi = torch.exp(-xd * xd / 2) / (2 * torch.pi) ** 0.5
    for got, want in ((k.act_fwd(x, 2), xd * cdf), (k.act_bwd(x, torch.ones_like(x), 2), cdf + xd * phi)):
        m = torch.isfinite(xd) & torch.isfinite(want) & (xd.abs() >= 2.0 ** -126) & (want.abs() >= 2.0 ** -124)
        assert int(m.sum()) > 48000 and int((got[m] != _rounded(want[m])).sum()) == 0
