"""Two calls for one parameter in one list (a layer that applies a weight twice)."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("T,N,K", [(300, 512, 768), (2048, 2048, 2048), (1018, 264, 1544), (64, 72, 8)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_a_gradient_that_two_calls_of_a_list_add_to(T, N, K, dt):
    """The second product reads what the first has written, whole or in part (a view of its rows): the bits of the calls one
    after the other (no reduction here is long enough to be cut).  Bias and norm gradients, which the list adds up in one
    launch otherwise, against 64 bits: 2^-20 of the sum of magnitudes for fp32, a rounding per addition for bf16."""
    from zorse_b200.ops import sm100 as k
    from zorse_b200.ops.api import get_ops

    ops = get_ops("sm100")
    rand = lambda *shape, seed: torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).bfloat16().cuda()
    dys, xs = [rand(T, N, seed=i) for i in range(4)], [rand(T, K, seed=10 + i) for i in range(4)]
    rows = N // 16 * 8
    got, want = (torch.ones(N, K, dtype=dt, device="cuda") for _ in range(2))
    gb, norm = torch.ones(N, dtype=dt, device="cuda"), torch.ones(2, K, dtype=dt, device="cuda")
    w = rand(K, seed=30)
    _, st = ops.norm_fwd(xs[0], w, w, 1e-5, True)
    for _ in range(3):
        later = ops.collect()
        ops.linear_wgrad(dys[0], xs[0], got, gb, later=later)
        ops.linear_wgrad(dys[1], xs[1], got, gb, later=later)
        ops.norm_bwd(xs[1], xs[0], w, st, None, norm[0], norm[1], True, later)
        ops.linear_wgrad(dys[2][:, :rows], xs[2], got[:rows], gb[:rows], later=later)
        ops.norm_bwd(xs[2], xs[0], w, st, None, norm[0], norm[1], True, later)
        ops.linear_wgrad(dys[3], xs[3], got, gb, later=later)
        ops.finish(later)
        for dy, x, rs in zip(dys, xs, (N, N, rows, N)):
            ops.linear_wgrad(dy[:, :rs], x, want[:rs])
    torch.cuda.synchronize()
    k.check_status()
    assert torch.equal(got, want)
    bias = [dy.double() for dy in dys]
    bias[2] = torch.cat((bias[2][:, :rows], torch.zeros_like(bias[2][:, rows:])), 1)
    xh = (xs[0].double() - st[:, :1].double()) * st[:, 1:].double()
    for out, srcs in ((gb, bias), (norm[0], [xs[1].double() * xh, xs[2].double() * xh]), (norm[1], [xs[1].double(), xs[2].double()])):
        exact, mass = 1 + 3 * sum(s.sum(0) for s in srcs), 1 + 3 * sum(s.abs().sum(0) for s in srcs)
        # (bf16: each of at most twelve additions rounds a value no larger than the mass)
        bound = mass * (2.0 ** -20 if dt == torch.float32 else 12 * 2.0 ** -9)
        assert bool(((out.double() - exact).abs() <= bound + 1e-6).all())
