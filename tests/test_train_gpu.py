"""End-to-end training steps on a GPU through the sm_100a kernels vs the fp32 PyTorch oracle."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from zorse_b200.config.training_config import parse_pipeline_dict


def _cfg(model="tiny_llama", gbs=4, mbs=2, seq=256, vocab=2048, schedule=None, reduce="float32", layers=(0, 4), **kw):
    d = {"model_name": model, "global_batch_size": gbs, "microbatch_size": mbs, "sequence_length": seq,
         "vocab_size": vocab, "autocast_dtype": "bfloat16", "reduce_dtype": reduce,
         "pipeline_config": [{"gpu_ranks": [0], "num_microbatches_per_rank": [gbs // mbs],
                              "layer_partition": list(layers), "zero_config": [[0]]}]}
    d.update(kw)
    return parse_pipeline_dict(d)


def _oracle_from(tr, cfg, overrides=None):
    """Oracle initialised from the trainer's own fp32 master weights (rounded to bf16 as the
    compute copy is), so both start from identical parameters."""
    from zorse_b200.utils.oracle import OracleTrainer

    orc = OracleTrainer(cfg, model_overrides=overrides)
    with torch.no_grad():
        for u, f in zip(tr.stages[0].engine.units, orc.flats):
            f.copy_(u.full_master()[: f.numel()].cpu())
    return orc


@pytest.mark.parametrize("schedule,recompute", [("zero2", True), ("1f1b", False), ("layer_major", True)])
@pytest.mark.parametrize("model,overrides", [("tiny_llama", {}), ("deepspeedmistral_toy", {}),
                                             ("toygpt", {"heads": 4, "hidden": 256}), ("opt_125m", {"layers": 2})])
def test_loss_and_grads_match_oracle(schedule, recompute, model, overrides):
    from zorse_b200.trainer import Trainer, TrainerOptions

    nl = overrides.get("layers", 4)
    cfg = _cfg(model=model, layers=(0, nl), seq=128 if model == "toygpt" else 256)
    tr = Trainer(cfg, TrainerOptions(schedule=schedule, ops="sm100", activation_recompute=recompute,
                                     model_overrides=overrides, lr=0.0))
    batch = tr.synthetic_batch()
    orc = _oracle_from(tr, cfg, overrides)
    want_loss, want_grads = orc.grads({k: v for k, v in batch.items()})
    # lr = 0: parameters stay put, Adam's first moment after one step is (1 - beta1) * grad
    loss = tr.train_step_from_host(batch)
    tr.check_kernels()
    assert abs(loss - want_loss) < 0.03 * max(1.0, abs(want_loss)), (loss, want_loss)
    for u, wg in zip(tr.stages[0].engine.units, want_grads):
        got = (u.m[: wg.numel()] / (1 - 0.9)).float().cpu()
        denom = wg.abs().max().item() + 1e-6
        err = (got - wg).abs().max().item() / denom
        cos = torch.nn.functional.cosine_similarity(got.flatten(), wg.flatten(), dim=0).item()
        assert cos > 0.99 and err < 0.08, f"unit {u.gid} ({u.layer.kind}): rel err {err:.4f}, cosine {cos:.5f}"


def test_loss_decreases_and_bf16_reduce():
    from zorse_b200.trainer import Trainer, TrainerOptions

    cfg = _cfg(reduce="bfloat16", gbs=8, mbs=2)
    tr = Trainer(cfg, TrainerOptions(schedule="zero2", ops="sm100", optimizer_in_backward=True))
    batch = tr.synthetic_batch()
    losses = [tr.train_step_from_host(batch) for _ in range(8)]
    tr.check_kernels()
    assert losses[-1] < losses[0] - 0.5, losses


@pytest.mark.parametrize("schedule", ["layer_major", "zero2"])
def test_parameter_offload_trains_like_the_resident_run(schedule):
    """`offload_model_params` (bf16 shards parked in pinned host memory, copied in on a copy stream before a
    unit is gathered; needs optimizer-in-backward, reference zorse.py:264-267) gives the same losses as the
    same job with resident parameters."""
    from zorse_b200.trainer import Trainer, TrainerOptions

    cfg = _cfg(gbs=4, mbs=2)
    losses = {}
    for off in (False, True):
        tr = Trainer(cfg, TrainerOptions(schedule=schedule, ops="sm100", optimizer_in_backward=True,
                                         offload_model_params=off))
        batch = tr.synthetic_batch()
        losses[off] = [tr.train_step_from_host(batch) for _ in range(3)]
        tr.check_kernels()
        if off:
            assert all(u.cfg.offload_params for u in tr.stages[0].engine.units)
        del tr
    assert losses[True] == pytest.approx(losses[False], rel=2e-3, abs=2e-3), losses


@pytest.mark.parametrize("schedule", ["layer_major", "zero2", "1f1b"])
def test_masters_on_their_way_to_the_optimizer_take_few_buffers(schedule, monkeypatch):
    """Parked fp32 masters travel to the GPU ahead of the optimizer.  With the communication stream held up, so that the host
    runs a whole backward pass ahead of it, a step needs at most two more units' masters of device memory than one that
    fetches none ahead (three buffers against the one of its optimizer); a unit that was updated already is not fetched again; every copy is counted once."""
    from zorse_b200.engine.zero import ZeroUnit
    from zorse_b200.trainer import Trainer, TrainerOptions

    def peak(ahead):
        with monkeypatch.context() as m:
            if not ahead:
                m.setattr(ZeroUnit, "_fetch_master", lambda self: None)
            torch.cuda.synchronize()
            torch.cuda.empty_cache()
            before = torch.cuda.memory_stats()["active_bytes.all.current"]
            tr = Trainer(_cfg(model="opt_125m", gbs=1, mbs=1, seq=128, layers=(0, 12)),
                         TrainerOptions(schedule=schedule, ops="sm100", optimizer_in_backward=True, offload_model_params=True))
            batch = tr.synthetic_batch()
            units = tr.stages[0].engine.units
            counters = tr.stages[0].engine.counters
            masters = sum(u.host_master.numel() * 4 for u in units)
            got, losses = [], []
            for _ in range(3):
                h2d, d2h = counters.h2d_bytes, counters.d2h_bytes
                torch.cuda.synchronize()
                torch.cuda.reset_peak_memory_stats()
                with torch.cuda.stream(tr.streams.comm):
                    torch.cuda._sleep(200_000_000)       # about 0.1 s
                losses.append(tr.train_step_from_host(batch))
                got.append(torch.cuda.memory_stats()["active_bytes.all.peak"] - before)
                assert (counters.h2d_bytes - h2d - masters) % 2 == 0
                bf16 = (counters.h2d_bytes - h2d - masters) / (masters / 2)
                assert 1 <= bf16 <= 2, "bf16 copies in: one per pass at most, masters once"
                assert counters.d2h_bytes - d2h == masters + masters // 2
            tr.check_kernels()
            if ahead:
                lower, upper = units[3], units[4]
                lower.step_count += 1                     # as after its update in this step
                upper.grad_views()
                upper.reduce_grads()
                torch.cuda.synchronize()
                assert lower.master_slot is None and units[3].below.master_slot is None
            return max(got), max(u.shard_n for u in units) * 4, losses

    (without, _, want), (with_, unit, losses) = peak(False), peak(True)
    assert with_ - without <= 2 * unit + (1 << 20), (with_, without, unit)
    assert losses == pytest.approx(want, rel=1e-3)


def test_activation_offload_to_pinned_host_matches_the_resident_stash():
    """Layer inputs parked in pinned host buffers between forward and backward (copy stream both ways)
    against the same recomputing schedule with the stash kept on the device."""
    from zorse_b200.trainer import Trainer, TrainerOptions

    cfg = _cfg(gbs=4, mbs=2)
    losses = {}
    for off in (False, True):
        tr = Trainer(cfg, TrainerOptions(schedule="layer_major", ops="sm100", activation_recompute=True,
                                         activation_offload=off))
        batch = tr.synthetic_batch()
        losses[off] = [tr.train_step_from_host(batch) for _ in range(3)]
        tr.check_kernels()
        if off:
            st = tr.stages[0].stash
            assert st.offload and st.d2h_bytes > 0 and st.h2d_bytes > 0, "activations were not parked on the host"
        del tr
    assert losses[True] == pytest.approx(losses[False], rel=2e-3, abs=2e-3), losses


def test_a_kernel_that_gave_up_ends_the_step_it_was_part_of(monkeypatch):
    """train_step_from_host reads the kernels' status word with the loss.  The word is set from the host here, as a kernel
    does whose wait ran out; a rank that has no loss to wait for raises at its next call."""
    from zorse_b200.ops.sm100 import KernelError
    from zorse_b200.trainer import Trainer, TrainerOptions

    tr = Trainer(_cfg(), TrainerOptions(schedule="1f1b", ops="sm100"))
    batch = tr.synthetic_batch()
    first = tr.train_step_from_host(batch)
    word = tr.ops.k.status_word(tr.device)
    word.fill_(3)
    with pytest.raises(KernelError, match="accumulator never completed"):
        tr.train_step_from_host(batch)
    assert tr.train_step_from_host(batch) < first            # reported once, and the trainer goes on
    monkeypatch.setattr(tr, "train_step", lambda inputs, targets: None)
    word.fill_(7)
    assert tr.train_step_from_host(batch) is None
    torch.cuda.synchronize()
    with pytest.raises(KernelError, match="wait ran out"):
        tr.train_step_from_host(batch)
    assert tr.train_step_from_host(batch) is None
    tr.check_kernels()


def test_smoke_entry():
    import __graft_entry__ as g

    g.smoke()


@pytest.mark.parametrize("buffers", [1, 5])
def test_backward_shards_come_from_the_masters(buffers, monkeypatch):
    """A parked unit that is fetched again for its backward pass gets its bf16 shard from the landed fp32 master: the same
    bits as the parked copy's (both are the master rounded to nearest), so the losses are those of a run that fetches every
    shard, and the bf16 copies cross the link once.  With one landing buffer, which the unit above holds, they
    are fetched as before."""
    from zorse_b200.engine.zero import MasterLanding, ZeroUnit
    from zorse_b200.trainer import Trainer, TrainerOptions

    def run(from_master):
        with monkeypatch.context() as m:
            m.setattr(MasterLanding, "BUFFERS", buffers)
            if not from_master:
                m.setattr(ZeroUnit, "_shard_from_master", lambda self: False)
            tr = Trainer(_cfg(gbs=4, mbs=2), TrainerOptions(schedule="layer_major", ops="sm100", optimizer_in_backward=True,
                                                            offload_model_params=True))
            batch = tr.synthetic_batch()
            counters = tr.stages[0].engine.counters
            losses = [tr.train_step_from_host(batch) for _ in range(3)]
            before = counters.h2d_bytes
            losses.append(tr.train_step_from_host(batch))
            units = tr.stages[0].engine.units
            tr.check_kernels()
            torch.cuda.synchronize()
            for u in units:
                assert u.master_slot is None
                assert torch.equal(u.host_p, u.host_master.to(torch.bfloat16))
            return losses, counters.h2d_bytes - before, [u.host_p.numel() for u in units]

    losses, moved, n = run(True)
    want, every, _ = run(False)
    assert losses == pytest.approx(want, rel=1e-3), (losses, want)
    assert every == sum(n) * 6 + sum(n[:-1]) * 2             # every master and shard, all shards but the head's again
    assert moved == every - (2 * sum(n[:-1]) if buffers == 5 else 0)
