"""The work this framework is timed on: whole training steps through `Trainer`, and single transformer blocks
forward and backward as the layer profiler and the pipeline stages run them.

Every case is a dict of plain values.  Two kinds:

* ``step``  one optimizer step of a one-GPU job through `Trainer.train_step_from_host`: copy of the step's inputs
  from pinned host memory, every microbatch forward and backward, Adam, the loss read back.  Outputs: the loss, and
  of every unit the fp32 master weights and both Adam moments.
* ``block`` one transformer block on one microbatch: forward (``backward: False``, the pass a schedule with
  recomputation makes first), or forward and backward with the weight gradients added to the block's bucket.
"""
from __future__ import annotations

import math

import torch

from zorse_b200.config.training_config import parse_pipeline_dict
from zorse_b200.models import registry
from zorse_b200.ops.api import get_ops
from zorse_b200.trainer import Trainer, TrainerOptions


def _step(name, model, layers, seq, mbs, microbatches, vocab, schedule, reduce, in_backward=False, offload=False):
    return {"name": name, "kind": "step", "model": model, "layers": layers, "seq": seq, "microbatch": mbs,
            "microbatches": microbatches, "vocab": vocab, "schedule": schedule, "reduce": reduce,
            "in_backward": in_backward, "offload": offload}


def _block(name, model, seq, mbs, reduce, backward=True):
    return {"name": name, "kind": "block", "model": model, "seq": seq, "microbatch": mbs, "reduce": reduce,
            "backward": backward}


def listed():
    return [
        # a test or debugging job: the tiny decoder of the first benchmark configuration, 8 sequences of 128 tokens.
        # Its kernels take a few microseconds each, so launches and host work count.
        _step("step_tiny_llama", "tiny_llama", 4, 128, 2, 4, 32000, "1f1b", "float32"),
        # a small GPT (LayerNorm, GELU, biases, learned positions) on sequences cut to an odd length, with the
        # reference's ZeRO-2 schedule: activations are recomputed in the backward pass
        _step("step_gpt_test_ragged", "deepspeedgpt_test", 12, 509, 2, 4, 49152, "zero2", "float32"),
        # BERT pre-training: post-LayerNorm, erf-GELU, short sequences in larger microbatches
        _step("step_bert_base", "deepspeedbert_base", 12, 384, 8, 2, 30528, "1f1b", "bfloat16"),
        # ViT on 384 x 384 images: 577 tokens per image, bidirectional attention, a classifier head on one token
        _step("step_vit", "deepspeedvit_default", 12, 577, 8, 2, 32000, "1f1b", "float32"),
        # OPT with parameters parked in pinned host memory between uses and the optimizer inside the backward pass,
        # layer-major: the plan of the offloading configuration, on the smallest model of that family
        _step("step_opt_offload", "opt_125m", 12, 2048, 1, 4, 50272, "layer_major", "float32", True, True),
        # the 1B model of the second configuration as it stands: grouped-query heads of 64, a vocabulary of 128256
        _step("step_llama_1b", "llama3.2_1b", 16, 2048, 1, 4, 128256, "zero2", "bfloat16", True),
        # the headline model: four blocks of Llama-2-7B between embedding and head, microbatches of one 4096-token
        # sequence, 1F1B without recomputation
        _step("step_llama_7b_4layers", "llama2_7b", 4, 4096, 1, 4, 32000, "1f1b", "bfloat16"),
        # one block of the same model, forward and backward: what the layer profiler times for the planner
        _block("block_llama_7b", "llama2_7b", 4096, 1, "float32"),
        # the forward a schedule with recomputation runs first, at a length between two powers of two
        _block("block_forward_llama_1b", "llama3.2_1b", 1500, 2, "bfloat16", False),
        # long sequences with a sliding window (8192 tokens, window 4096, grouped-query heads)
        _block("block_mistral_7b_window", "mistral_7b", 8192, 1, "bfloat16"),
        # wide LayerNorm / GELU block with biases, the 13B model of the offloading configuration
        _block("block_opt_13b", "opt_13b", 2048, 1, "bfloat16"),
    ]


# families a case may be drawn from: (model, sequence lengths, largest tokens per microbatch)
_STEP_MODELS = [("tiny_llama", (64, 2048), 4096), ("deepspeedmistral_toy", (64, 2048), 4096),
                ("deepspeedgpt_test", (64, 2048), 4096), ("opt_125m", (128, 2048), 4096),
                ("deepspeedbert_base", (64, 512), 4096), ("deepspeedvit_default", (577, 577), 4616),
                ("deepspeedbert_330m", (64, 512), 4096), ("opt_350m", (128, 2048), 4096),
                ("llama3.2_1b", (256, 4096), 4096), ("llama2_7b", (512, 4096), 4096),
                ("mistral_7b", (512, 4608), 4608)]
_BLOCK_MODELS = [("tiny_llama", (64, 4096), 8192), ("deepspeedgpt_1.3b", (128, 2048), 8192),
                 ("deepspeedgpt_6.7b", (128, 2048), 4096), ("opt_350m", (128, 2048), 8192),
                 ("opt_13b", (128, 2048), 4096), ("deepspeedbert_large", (64, 512), 8192),
                 ("deepspeedvit_5b", (577, 577), 4616), ("llama3.2_1b", (128, 8192), 8192),
                 ("llama2_7b", (128, 6144), 6144), ("mistral_7b", (128, 8192), 8192)]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    if rng.random() < 0.5:
        model, (lo, hi), most = rng.choice(_STEP_MODELS)
        seq = _log_uniform(rng, lo, hi)
        mbs = _log_uniform(rng, 1, max(1, min(8, most // seq)))
        large = registry.get_spec(model).hidden >= 2048
        layers = min(registry.get_spec(model).layers, rng.randint(1, 3) if large else rng.randint(2, 12))
        reduce = rng.choice(["float32", "bfloat16"])
        schedule = rng.choice(["1f1b", "zero2", "layer_major"])
        in_backward = rng.random() < 0.5
        offload = in_backward and not large and rng.random() < 0.25
        vocab = 8 * _log_uniform(rng, 1000, 6300)
        return {k: v for k, v in _step("", model, layers, seq, mbs, rng.randint(1, 3), vocab, schedule, reduce,
                                       in_backward, offload).items() if k != "name"}
    model, (lo, hi), most = rng.choice(_BLOCK_MODELS)
    seq = _log_uniform(rng, lo, hi)
    mbs = _log_uniform(rng, 1, max(1, min(8, most // seq)))
    return {k: v for k, v in _block("", model, seq, mbs, rng.choice(["float32", "bfloat16"]),
                                    rng.random() < 0.7).items() if k != "name"}


def prepare(case, seed):
    if case["kind"] == "step":
        return _prepare_step(case, seed)
    return _prepare_block(case, seed)


def _overrides(case):
    """ViT classifies into 1000 classes here: the kernels need a class count that is a multiple of 8."""
    vit = registry.get_spec(case["model"]).family == "vit"
    return {"layers": case["layers"], **({"classes": 1000} if vit else {})}


def _prepare_step(case, seed):
    M = case["microbatches"]
    cfg = parse_pipeline_dict({
        "model_name": case["model"], "global_batch_size": M * case["microbatch"],
        "microbatch_size": case["microbatch"], "sequence_length": case["seq"], "vocab_size": case["vocab"],
        "autocast_dtype": "bfloat16", "reduce_dtype": case["reduce"],
        "pipeline_config": [{"gpu_ranks": [0], "num_microbatches_per_rank": [M],
                             "layer_partition": [0, case["layers"]], "zero_config": [[0]]}]})
    tr = Trainer(cfg, TrainerOptions(schedule=case["schedule"], ops="sm100", lr=1e-4, seed=seed,
                                     optimizer_in_backward=case["in_backward"], offload_model_params=case["offload"],
                                     model_overrides=_overrides(case)))
    return {"case": case, "trainer": tr, "batch": tr.synthetic_batch(seed)}


def _prepare_block(case, seed):
    spec = registry.get_spec(case["model"])
    blk = registry.make_block(spec)
    _, n = blk.layout()
    flat = torch.empty(n, dtype=torch.float32, device="cuda")
    blk.init_flat(flat, seed)
    grads = None
    if case["backward"]:
        grads = torch.zeros(n, dtype=getattr(torch, case["reduce"]), device="cuda")
    blk.bind(flat.to(torch.bfloat16), grads)
    T = case["microbatch"] * case["seq"]
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    x = torch.randn(T, spec.hidden, device="cuda", generator=gen).mul_(0.5).to(torch.bfloat16)
    dy = torch.randn(T, spec.hidden, device="cuda", generator=gen).mul_(0.5).to(torch.bfloat16)
    return {"case": case, "block": blk, "grads": grads, "x": x, "dy": dy, "ops": get_ops("sm100"),
            "ctx": {"B": case["microbatch"], "S": case["seq"]}}


def run(state):
    if state["case"]["kind"] == "step":
        tr = state["trainer"]
        loss = tr.train_step_from_host(state["batch"])
        return {"loss": loss, "state": [u.state_tensors() for st in tr.stages for u in st.engine.units]}
    blk, ctx, ops = state["block"], state["ctx"], state["ops"]
    if not state["case"]["backward"]:
        return blk.forward(state["x"], ctx, ops, None)
    saved: dict = {}
    y = blk.forward(state["x"], ctx, ops, saved)
    dx = blk.backward(state["dy"], ctx, ops, saved)
    return {"y": y, "dx": dx, "grads": state["grads"]}


def _score_pairs(spec, seq):
    """Visible (query, key) pairs of one sequence and head."""
    if not spec.causal:
        return seq * seq
    w = min(spec.window or seq, seq)
    return w * (w + 1) // 2 + (seq - w) * w


def work(case):
    spec = registry.get_spec(case["model"])
    blk = registry.make_block(spec)
    seq = case["seq"]
    n_blk = blk.num_params()
    pairs = _score_pairs(spec, seq) * spec.heads * spec.head_dim
    gb = 4 if case["reduce"] == "float32" else 2
    if case["kind"] == "block":
        T = case["microbatch"] * seq
        if not case["backward"]:
            # weights and x in, y out; 2 flops per weight and token, 2 products of 2 flops per visible pair
            return {"bytes": 2.0 * n_blk + 4.0 * T * spec.hidden,
                    "flops": 2.0 * n_blk * T + 4.0 * pairs * case["microbatch"]}
        # weights, x and dy in, y and dx out, the gradient bucket read and written; backward: 5 products per pair
        return {"bytes": (2.0 + 2 * gb) * n_blk + 8.0 * T * spec.hidden,
                "flops": 6.0 * n_blk * T + 14.0 * pairs * case["microbatch"]}
    seqs = case["microbatch"] * case["microbatches"]
    spec = registry.get_spec(case["model"], vocab=case["vocab"], **_overrides(case))
    head = registry.make_head(spec).num_params()
    emb = registry.make_embedding(spec, seq).num_params()
    total = n_blk * case["layers"] + head + emb
    head_rows = seqs * (1 if spec.pool else seq)
    patches = 4.0 * emb * seqs * seq if spec.family == "vit" else 0.0
    # master weights and both moments read and written in fp32, the bf16 copy read and written
    return {"bytes": 28.0 * total,
            "flops": (6.0 * n_blk * seq + 14.0 * pairs) * case["layers"] * seqs + 6.0 * head * head_rows + patches}


def tolerance(case):
    """About four times the largest relative difference seen against the same path on plain PyTorch in fp32 with bf16
    results: blocks 0.006 in every output; steps, in the second moment (twice the gradient's), 0.019 for the narrow
    models, 0.024 for four wide layers and 0.05 for the sixteen of the 1B model (rounding grows with depth)."""
    if case["kind"] == "block":
        return {"rel": 0.025}
    if registry.get_spec(case["model"]).hidden < 2048:
        return {"rel": 0.07}
    return {"rel": 0.1 if case["layers"] <= 4 else 0.2}
