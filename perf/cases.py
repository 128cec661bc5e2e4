"""What the framework is timed on: the passes that a pre-training job on one GPU consists of.

``listed()`` are the standing cases, ``draw(rng)`` gives more of the same ranges, ``prepare(case, seed)`` builds what a user's
program holds before the pass (model, gradient buckets, optimizer, token ids), ``run(state)`` is one pass through the public
entry points, ``work(case)`` the bytes and operations a pass cannot do without, ``tolerance(case)`` how far the results of
another correct implementation at the same precision may be off.

Kinds of passes:

``train``    gradient accumulation: the buckets are cleared, then forward + backward of ``micro`` micro-batches; gives the
             loss and the whole fp32 gradient buffer.
``step``     an eager optimizer step: one micro-batch, AdamW, bucket reset; gives the loss and every weight.
``trainer``  ``Trainer.step`` as ``train.py`` calls it (data loader, ``micro`` accumulation micro-batches, AdamW).
``update``   the end of a step on its own: global-norm clipping and AdamW over given gradients; gives weights and moments.
``eval``     validation loss of a batch, no gradients.
``logits``   the forward pass that greedy decoding makes for every token; gives the logits.
"""
import math

import torch

from picotron_b200.config import ModelConfig
from picotron_b200.models.llama import Llama
from picotron_b200.optim import FusedAdamW, clip_grad_norm_
from picotron_b200.parallel.data_parallel import DataParallelBucket
from picotron_b200.trainer import build_trainer

# hidden, intermediate, query heads, key/value heads, layers, vocabulary, rope theta: the shapes of the package's presets and,
# first, of its smoke test
SHAPES = {
    "smoke": (512, 1024, 8, 4, 2, 2048, 10000.0),
    "135m": (576, 1536, 9, 3, 30, 49152, 10000.0),
    "360m": (960, 2560, 15, 5, 32, 49152, 10000.0),
    "1.7b": (2048, 8192, 32, 32, 24, 49152, 10000.0),
    "1b": (2048, 8192, 32, 8, 16, 128256, 500000.0),
    "7b": (4096, 11008, 32, 32, 32, 32000, 10000.0),
    "8b": (4096, 14336, 32, 8, 32, 128256, 500000.0),
}


def _case(name, kind, shape, batch, seq, micro=1, layers=None):
    hidden, inter, heads, kv, depth, vocab, theta = SHAPES[shape]
    return {"name": name, "kind": kind, "hidden": hidden, "inter": inter, "heads": heads, "kv": kv,
            "layers": layers or depth, "vocab": vocab, "theta": theta, "batch": batch, "seq": seq, "micro": micro}


def listed():
    return [
        # the smallest job: a model for trying things out, where launches and host work are everything
        _case("tiny_step", "step", "smoke", 2, 256),
        # one forward pass of greedy decoding with a small model, a prompt of a few hundred tokens
        _case("decode_forward", "logits", "135m", 1, 256),
        # short sequences (a five-layer cut of the 1.7B shape, 4 x 128 tokens, two micro-batches): weights and gradients weigh
        # more than tokens
        _case("short_sequences", "train", "1.7b", 4, 128, micro=2, layers=5),
        # a small model with sample lengths that fit no tile
        _case("small_ragged", "train", "135m", 3, 601, layers=16),
        # a small model, an ordinary batch
        _case("small_train", "train", "135m", 8, 1024, layers=16),
        # the command a user runs: Trainer.step with gradient accumulation, the depth of the default configuration
        _case("trainer_step", "trainer", "360m", 4, 1024, micro=4, layers=16),
        # the micro-batch of the headline benchmark, with the 15 layers of the data-parallel example
        _case("headline_train", "train", "1.7b", 4, 1024, layers=15),
        # a validation batch of the same model, all its layers
        _case("headline_eval", "eval", "1.7b", 4, 1024),
        # one pipeline stage's worth of a 7B model (head dimension 128)
        _case("stage_7b", "train", "7b", 4, 1024, layers=4),
        # the same for an 8B model at 8192 tokens, grouped-query attention, large vocabulary
        _case("stage_8b", "train", "8b", 1, 8192, layers=3),
        # long context, head dimension 64, grouped-query attention
        _case("long_context", "train", "1b", 1, 32768, layers=4),
        # clipping and AdamW over a stage of a 7B model
        _case("update_7b", "update", "7b", 1, 128, layers=2),
    ]


def draw(rng):
    largest = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choice(["step", "logits", "train", "train", "train", "train", "trainer", "update", "eval"])
        if kind == "step":
            c = _case("", kind, "smoke", rng.randint(1, 8), int(64 * 2 ** rng.uniform(0, 4)), layers=rng.randint(1, 4))
        elif kind == "logits":
            c = _case("", kind, rng.choice(["135m", "360m"]), rng.randint(1, 4), int(32 * 2 ** rng.uniform(0, 5)))
        elif kind == "update":
            c = _case("", kind, rng.choice(["360m", "1.7b", "7b"]), 1, 128, layers=rng.randint(1, 2))
            c["inter"] = 8 * rng.randint(c["hidden"] // 8, c["hidden"] // 2)
        elif kind == "trainer":
            c = _case("", kind, rng.choice(["135m", "360m"]), rng.randint(1, 6), 8 * int(32 * 2 ** rng.uniform(0, 3)),
                      micro=rng.randint(1, 4))
        else:
            shape = rng.choice(["135m", "360m", "1.7b", "1b", "7b", "8b"])
            depth = {"7b": 8, "8b": 6}.get(shape, 16)
            seq = int(128 * 2 ** rng.uniform(0, 7))
            seq = seq if rng.random() < 0.3 else max(128, seq // 128 * 128)
            c = _case("", kind, shape, max(1, min(8, int(8192 * rng.random()) // seq)), seq, micro=rng.randint(1, 2),
                      layers=rng.randint(max(2, depth // 4), depth))
            if kind == "eval":
                c["micro"] = 1
        if c["batch"] * c["seq"] * c["micro"] > 32768 or work(c)["flops"] > 0.7 * largest:
            continue
        del c["name"]
        return c


def _model_config(case):
    return ModelConfig(hidden_size=case["hidden"], intermediate_size=case["inter"], num_hidden_layers=case["layers"],
                       num_attention_heads=case["heads"], num_key_value_heads=case["kv"], vocab_size=case["vocab"],
                       rope_theta=case["theta"], max_position_embeddings=case["seq"])


def _tokens(case, gen):
    window = torch.randint(0, case["vocab"], (case["batch"], case["seq"] + 1), device="cuda", generator=gen)
    return window[:, :-1].contiguous(), window[:, 1:].contiguous()


class _State(dict):
    """A pass's state. The gradient-ready hooks of a wrapped model refer to the model through C++, where Python's garbage
    collector does not see them, so they are taken off with the state: a run has one model, here many are made."""

    def __del__(self):
        model = self["trainer"].model if "trainer" in self else self["model"]
        for handle in getattr(model, "_hook_handles", ()):
            handle.remove()
        for p in model.parameters():
            p.__dict__.pop("_grad_ready_cb", None)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "trainer":
        trainer = build_trainer({
            "distributed": {"tp_size": 1, "cp_size": 1, "pp_size": 1, "dp_size": 1, "use_cpu": False},
            "model": {"name": "custom", "hidden_size": case["hidden"], "intermediate_size": case["inter"],
                      "num_hidden_layers": case["layers"], "num_attention_heads": case["heads"],
                      "num_key_value_heads": case["kv"], "vocab_size": case["vocab"], "rope_theta": case["theta"]},
            "training": {"seed": seed, "learning_rate": 3e-4, "total_train_steps": 10 ** 9, "seq_length": case["seq"],
                         "micro_batch_size": case["batch"], "gradient_accumulation_steps": case["micro"], "num_samples": None},
            "dataset": {"name": "synthetic"}}, init_dist=False)
        return _State(kind=kind, trainer=trainer, params=list(trainer.model.parameters()))
    gen = torch.Generator(device="cuda").manual_seed(seed)
    torch.manual_seed(seed)
    with torch.device("cuda"):
        model = Llama(_model_config(case), init="reference")
    model = model.to(torch.bfloat16)
    state = _State(kind=kind, model=model)
    if kind in ("train", "step", "update"):
        state["model"] = model = DataParallelBucket(model)
    if kind in ("step", "update"):
        state["optimizer"] = FusedAdamW(model.parameters(), lr=3e-4)
        state["params"] = list(model.parameters())
    if kind == "update":
        # gradients of a late training step, moments of the step before it
        model.bucket_manager.flat.normal_(0.0, 1e-3, generator=gen)
        state["optimizer"].step()
        model.bucket_manager.flat.normal_(0.0, 1e-3, generator=gen)
    else:
        state["batches"] = [_tokens(case, gen) for _ in range(case["micro"])]
    return state


def run(state):
    kind = state["kind"]
    if kind == "trainer":
        loss = state["trainer"].step()
        # one tensor: the model has more weight tensors than a result may have
        return {"loss": loss, "weights": torch.cat([p.detach().reshape(-1) for p in state["params"]])}
    model = state["model"]
    if kind == "train":
        model.reset()
        n = len(state["batches"])
        total = 0.0
        for i, (ids, targets) in enumerate(state["batches"]):
            model.require_backward_grad_sync = i == n - 1
            loss = model(input_ids=ids, target_ids=targets, loss_scale=1.0 / n)
            loss.backward()
            total = total + loss.detach()
        return {"loss": total, "grads": model.bucket_manager.flat}
    if kind == "step":
        ids, targets = state["batches"][0]
        loss = model(input_ids=ids, target_ids=targets)
        loss.backward()
        state["optimizer"].step()
        model.reset()
        return {"loss": loss.detach(), "weights": [p.detach() for p in state["params"]]}
    if kind == "update":
        norm = clip_grad_norm_(model, 1.0)
        opt = state["optimizer"]
        opt.step()
        return {"norm": norm, "weights": [p.detach() for p in state["params"]],
                "exp_avg": [opt.state[p]["exp_avg"] for p in state["params"]],
                "exp_avg_sq": [opt.state[p]["exp_avg_sq"] for p in state["params"]]}
    with torch.no_grad():
        ids, targets = state["batches"][0]
        return model(input_ids=ids, target_ids=targets) if kind == "eval" else model(input_ids=ids)


def work(case):
    h, i, layers, v, kind = case["hidden"], case["inter"], case["layers"], case["vocab"], case["kind"]
    kv = case["kv"] * (h // case["heads"])
    matrices = layers * (2 * h * h + 2 * kv * h + 3 * h * i) + v * h       # what every token is multiplied with
    params = matrices + v * h + (2 * layers + 1) * h
    tokens = case["batch"] * case["seq"] * case["micro"]
    # causal attention: each token meets half of the sequence, twice (scores, values); the backward pass costs twice the forward
    forward = 2.0 * matrices * tokens + 2.0 * layers * h * case["seq"] * tokens
    if kind == "update":
        # gradients read, scaled and written back by the clipping; then gradient, moments and master weight in, all but the
        # gradient and a bf16 weight out
        return {"bytes": params * (4 + 4 + 3 * 4 + 3 * 4 + 2), "flops": 16.0 * params}
    if kind in ("eval", "logits"):
        return {"bytes": 2.0 * params + 16.0 * tokens + (2.0 * v * tokens if kind == "logits" else 0.0), "flops": forward}
    adam = params * (4 + 3 * 4 + 3 * 4 + 2) if kind in ("step", "trainer") else 0
    return {"bytes": 2.0 * params + 4.0 * params + 16.0 * tokens + adam, "flops": 3.0 * forward}


def tolerance(case):
    """Four times (rounded, and at most 0.03) what was measured between the path and itself with its roundings moved: RoPE
    tables off by 2e-6, or the separate kernels instead of the fused epilogues. Any such change moves every later bf16 rounding
    of a deep model, so the figures are those of bf16 itself."""
    kind = case["kind"]
    if kind == "update":
        # fp32 throughout, the weights rounded to bf16 once: a weight next to a rounding boundary may land on the other side
        return {"rel": 2e-4, "max": 1e-2}
    if kind in ("step", "trainer"):
        # bf16 weights after the update. AdamW's first updates have the size of the learning rate whatever the gradient, so an
        # element whose gradient is lost in the noise may move the other way
        return {"rel": 5e-3, "max": 0.15} if kind == "step" else {"rel": 4e-4, "max": 2e-2}
    if kind == "eval":
        return {"rel": 5e-5}
    if kind == "logits":
        return {"rel": 0.03, "max": 0.4}
    # gradients: 0.0035 (largest element 0.24) with 4 layers, 0.012 (0.7) with 24
    return {"rel": 0.015 if case["layers"] <= 4 else 0.03, "max": 0.99}
