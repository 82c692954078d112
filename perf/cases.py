"""Performance cases: what users of the framework have it do, through its public entry points.

Four kinds of work, each with its own sizes:

* `train`: one optimizer step of a model (`ScheduleRunner.run_step`): host batches from the data loader, forward, backward,
  gradient accumulation over micro-batches, clipping and the Adam update.  Dense, packed-document, LoRA and hybrid decoders.
* `moe`: forward and backward of a dropless mixture-of-experts layer, stand-alone (behind an attention layer the last bit of
  a bf16 activation decides between two experts, so a whole model's outputs could not be compared).
* `score`: prompt log-likelihoods through the Hugging Face wrapper: one forward pass over left-padded rows, logits out.
* `generate`: a request through the Hugging Face wrapper with its key / value cache: the prompt, then one call per new token.
  The tokens are given (as in scoring an answer), so that a tie between two logits does not change the rest of the text.
"""

import itertools
import math

import torch

import fast_llm_b200.models.auto  # noqa: F401
from fast_llm_b200.data.document import LanguageModelBatch, LanguageModelDocument
from fast_llm_b200.engine.inference.huggingface import HuggingfaceGPTModelForCausalLM
from fast_llm_b200.engine.multi_stage.config import StageMode
from fast_llm_b200.engine.optimizer.optimizer import Optimizer
from fast_llm_b200.engine.schedule.runner import ScheduleRunner
from fast_llm_b200.engine.schedule.schedule import Schedule
from fast_llm_b200.layers.moe import MoEMLPConfig
from fast_llm_b200.models.gpt.config import GPTModelConfig
from fast_llm_b200.models.gpt.model import GPTModel
from fast_llm_b200.models.gpt.trainer import GPTTrainerConfig
from fast_llm_b200.parallel.distributed import Distributed
from fast_llm_b200.parallel.topology import DistributedConfig, PhaseType
from fast_llm_b200.tensor import TensorDim


def _train(name=None, **sizes):
    case = {
        "kind": "train", "mixers": "attention", "layers": 2, "hidden": 1024, "heads": 8, "kv_heads": 4, "head_size": 128, "ffn": 4096,
        "vocab": 32000, "window": 0, "tokens": 4096, "documents": 1, "micro_batches": 1, "lora_rank": 0,
    }
    return {**({} if name is None else {"name": name}), **case, **sizes}


def _inference(kind, name=None, **sizes):
    case = {
        "kind": kind, "mixers": "attention", "layers": 8, "hidden": 2048, "heads": 16, "kv_heads": 4, "head_size": 128, "ffn": 8192,
        "vocab": 32000, "window": 0, "rows": 8, "prompt": 512,
    }
    return {**({} if name is None else {"name": name}), **case, **sizes}


def listed():
    return [
        # The tiny Llama-style decoder of the example configuration, on a GPU: debugging runs and unit-size experiments, where
        # launches and host work are everything.
        _train("train_tiny", hidden=256, heads=8, kv_heads=4, head_size=32, ffn=1024, vocab=8192, tokens=1024, documents=2),
        # A small pre-training run (ablations, scaling-law points): many short kernels, an odd number of packed documents.
        _train("train_small", layers=8, hidden=1024, heads=16, kv_heads=4, head_size=64, ffn=2816, tokens=4096, documents=5),
        # The headline configuration at a depth that fits three times: Mistral-7B blocks, 8192-token micro-batches, 4096-token
        # documents, window 4096.
        _train("train_mistral", layers=4, hidden=4096, heads=32, kv_heads=8, ffn=14336, window=4096, tokens=8192, documents=2),
        # Instruction fine-tuning of a Llama-3-8B shape: packed conversations of ragged lengths, its 128k vocabulary, two
        # micro-batches of an odd number of tokens accumulated into one step.
        _train("train_packed", layers=1, hidden=4096, heads=32, kv_heads=8, ffn=14336, vocab=128256, tokens=4099, documents=23, micro_batches=2),
        # The same with adapters: frozen base weights, LoRA on the attention projections.
        _train("train_lora", layers=4, hidden=4096, heads=32, kv_heads=8, ffn=14336, tokens=2048, documents=9, lora_rank=16),
        # Hybrid decoders, attention alternating with a recurrent mixer: Mamba, gated DeltaNet, Kimi delta attention.
        _train("train_mamba", mixers="attention,mamba", hidden=4096, heads=32, kv_heads=8, ffn=8192, tokens=8192, documents=2),
        _train("train_gdn", mixers="attention,gdn", hidden=4096, heads=32, kv_heads=8, ffn=8192, tokens=8192, documents=4),
        _train("train_kda", mixers="kda", hidden=2048, heads=16, kv_heads=16, ffn=5632, tokens=4096, documents=7),
        # A Mixtral-8x7B layer: 8 experts of 14336, two per token.
        {"name": "moe_mixtral", "kind": "moe", "hidden": 4096, "ffn": 14336, "experts": 8, "top_k": 2, "tokens": 4096},
        # One user's short request: latency of every token.
        _inference("generate", "generate_one", rows=1, prompt=100, new=24),
        # A batch of requests with prompts of different lengths.
        _inference("generate", "generate_batch", rows=8, prompt=512, new=24),
        # Evaluation harness: log-likelihoods of a batch of left-padded rows.
        _inference("score", "score_batch", rows=8, prompt=1000),
    ]


_MAX_FLOPS = 6e13  # of a drawn case: just below the largest listed one
_MAX_PARAMETERS = 1.2e9


def draw(rng):
    def log_uniform(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    while True:
        kind = rng.choice(["train", "train", "train", "hybrid", "hybrid", "moe", "generate", "score"])
        hidden = rng.choice([256, 512, 1024, 2048, 4096])
        head_size = rng.choice([64, 128])
        heads = max(hidden // head_size, 2)
        kv_heads = max(heads // rng.choice([1, 2, 4]), 1)
        ffn = 64 * max(log_uniform(2 * hidden, 4 * hidden) // 64, 1)
        layers = rng.randint(1, 8)
        vocab = rng.choice([8192, 32000, 32000, 128256])
        window = rng.choice([0, 0, 1024, 4096])
        tokens = log_uniform(256, 8192)
        shape = dict(layers=layers, hidden=hidden, heads=heads, kv_heads=kv_heads, head_size=head_size, ffn=ffn, vocab=vocab)
        if kind == "train":
            case = _train(**shape, window=window, tokens=tokens, documents=rng.randint(1, max(tokens // 128, 1)), micro_batches=rng.choice([1, 1, 2]),
                          lora_rank=rng.choice([0, 0, 0, 16]))
        elif kind == "hybrid":
            mixer = rng.choice(["mamba", "gdn", "kda"])
            prefix = "attention," if layers > 1 and rng.random() < 0.5 else ""
            case = _train(**shape, mixers=prefix + mixer, tokens=tokens, documents=rng.randint(1, max(tokens // 256, 1)))
            if mixer == "kda" and tokens * hidden * layers > 4096 * 2048 * 2:
                continue
            if mixer != "kda" and tokens * hidden * layers > 8192 * 4096 * 2:
                continue
        elif kind == "moe":
            case = {"kind": "moe", "hidden": hidden, "ffn": ffn, "experts": rng.choice([4, 8, 16]), "top_k": rng.choice([1, 2, 4]), "tokens": tokens}
        elif kind == "generate":
            case = _inference("generate", **shape, rows=log_uniform(1, 16), prompt=log_uniform(16, 1024), new=rng.randint(8, 32))
        else:
            case = _inference("score", **shape, rows=log_uniform(1, 16), prompt=log_uniform(16, 1024))
        if work(case)["flops"] <= _MAX_FLOPS and _parameters(case) <= _MAX_PARAMETERS:
            return case


# ----------------------------------------------------------------------------------------------------------------------
# models
# ----------------------------------------------------------------------------------------------------------------------
def _mixer(case, name):
    hidden, heads, head_size = case["hidden"], case["heads"], case["head_size"]
    if name == "attention":
        mixer = {"type": "attention", "rotary": {"type": "default", "theta": 10000}, "heads": heads, "head_groups": case["kv_heads"], "head_size": head_size,
                 "add_linear_biases": False}
        return {**mixer, "window_size": case["window"]} if case["window"] else mixer
    if name == "mamba":
        return {"type": "mamba", "d_inner": hidden, "d_xb": hidden // 4, "state_size": 16, "dt_rank": max(hidden // 16, 16), "add_linear_biases": False}
    if name == "gdn":
        return {"type": "gdn", "value_heads": heads, "key_heads": heads // 2, "key_head_dim": head_size, "value_head_dim": head_size}
    return {"type": "kda", "heads": heads, "head_dim": head_size}


def _base_model(case):
    norm = {"type": "rms_norm", "epsilon": 1e-5}

    def block(name):
        return {"mixer": _mixer(case, name), "normalization": norm,
                "mlp": {"intermediate_size": case["ffn"], "add_linear_biases": False, "gated": True, "activation": "silu"}}

    names = case["mixers"].split(",")
    if len(names) == 1:
        decoder = {"num_blocks": case["layers"], "block": block(names[0])}
    else:
        decoder = {"type": "pattern", "num_blocks": case["layers"], "pattern": names, "blocks": {n: block(n) for n in names}}
    model = {"embeddings": {"vocab_size": case["vocab"]}, "decoder": decoder, "head": {"normalization": norm}, "hidden_size": case["hidden"],
             "tied_embedding_weight": False}
    if case.get("lora_rank"):
        model["peft"] = {"type": "lora", "rank": case["lora_rank"], "alpha": 2.0 * case["lora_rank"]}
    return model


def _distributed(seed):
    return {"compute_dtype": "bf16", "seed": seed, "world_size": 1, "rank": 0, "local_world_size": 1}


def _document_lengths(total, count, generator):
    """`count` ragged lengths that add up to `total`."""
    cuts = (torch.randperm(total - 1, generator=generator)[: count - 1] + 1).sort().values.tolist()
    ends = [0, *cuts, total]
    return [b - a for a, b in zip(ends, ends[1:])]


def _prepare_train(case, seed):
    config = GPTTrainerConfig.from_dict({
        "model": {"base_model": _base_model(case), "distributed": _distributed(seed)},
        "optimizer": {"learning_rate": {"base": 1e-5}, "weight_decay": 0.1, "beta_1": 0.9, "beta_2": 0.95},
        "schedule": {"depth_first_micro_batches": case["micro_batches"]},
        "data": {"datasets": {"training": {"type": "random"}}, "micro_batch_size": case["tokens"]},
    })
    config.validate()
    distributed = Distributed(config.model.distributed)
    model = GPTModel(config.model, optimizer_state_names=config.optimizer.state_names, verbose=False)
    model.setup(distributed, mode=StageMode.training)
    groups = model.get_param_groups()
    optimizer = Optimizer(config.optimizer, groups, model.get_grad_norm_slices(), distributed, compute_dtype=torch.bfloat16,
                          weight_arena=model.weight_arena, grad_norm_partials=model.grad_norm_partials)
    runner = ScheduleRunner(config=config.schedule, multi_stage=model, distributed_config=config.model.distributed)
    runner.setup(distributed, optimizer)
    model.initialize_weights()
    optimizer.reset_state()
    schedule = Schedule(model, config.schedule, config.model.distributed, PhaseType.training)
    # what the data loader hands over: packed micro-batches in pinned host memory
    generator = torch.Generator().manual_seed(seed)
    batches = []
    for _ in range(2 * case["micro_batches"]):
        documents = [LanguageModelDocument(tokens=torch.randint(0, case["vocab"], (n,), generator=generator))
                     for n in _document_lengths(case["tokens"] + 1, case["documents"], generator)]
        batch = LanguageModelBatch.from_documents(documents, case["tokens"] + 1)
        batches.append(batch.get_model_inputs(micro_batch_size=case["tokens"], pin=True))
    return {"kind": "train", "runner": runner, "schedule": schedule, "data": itertools.cycle(batches), "iteration": 0,
            "updated": {**model.shards, "gradients": [g["grads"] for g in groups]}}


def _prepare_moe(case, seed):
    config = MoEMLPConfig.from_dict({"type": "moe", "experts": case["experts"], "experts_per_token": case["top_k"], "intermediate_size": case["ffn"],
                                     "gated": True, "activation": "silu", "add_linear_biases": False, "auxiliary_loss_coefficient": 0.01})
    config.validate()
    distributed = DistributedConfig.from_dict(_distributed(seed))
    distributed.validate()
    layer = config.get_layer(distributed, TensorDim("hidden", case["hidden"]))
    layer.set_names("mlp.")
    layer.materialize(device=torch.device("cuda"), dtype=torch.bfloat16)
    generator = torch.Generator(device="cuda").manual_seed(seed)
    x, grad = (torch.randn(case["tokens"], case["hidden"], device="cuda", generator=generator).bfloat16() for _ in range(2))
    return {"kind": "moe", "layer": layer, "x": x, "grad": grad}


def _prepare_inference(case, seed):
    config = GPTModelConfig.from_dict({"base_model": _base_model(case), "distributed": _distributed(seed)})
    config.validate()
    model = GPTModel(config, verbose=False)
    model.setup(Distributed(config.distributed), mode=StageMode.inference)
    model.initialize_weights()
    rows, prompt, new = case["rows"], case["prompt"], case.get("new", 0)
    generator = torch.Generator().manual_seed(seed)
    ids = torch.randint(1, case["vocab"], (rows, prompt + new), generator=generator)
    mask = torch.ones(rows, prompt, dtype=torch.int64)
    for row in range(1, rows):  # the first row is the longest
        mask[row, : int(torch.randint(0, max(prompt // 2, 1), (1,), generator=generator))] = 0
    return {"kind": case["kind"], "model": HuggingfaceGPTModelForCausalLM(model), "prompt": ids[:, :prompt].cuda(), "mask": mask.cuda(),
            "tokens": [t.cuda() for t in ids[:, prompt:].split(1, dim=1)] if new else []}


def prepare(case, seed):
    if case["kind"] == "train":
        return _prepare_train(case, seed)
    return _prepare_moe(case, seed) if case["kind"] == "moe" else _prepare_inference(case, seed)


# ----------------------------------------------------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------------------------------------------------
def run(state):
    if state["kind"] == "train":
        state["iteration"] += 1
        losses, _, _ = state["runner"].run_step(state["data"], state["schedule"], iteration=state["iteration"])
        return {**losses, **state["updated"]}
    if state["kind"] == "moe":
        x = state["x"].detach().requires_grad_()
        out = state["layer"].forward(x, {"training": True})
        out.backward(state["grad"])
        gradients = [p.grad for p in state["layer"].parameters()]
        for p in state["layer"].parameters():
            p.grad = None
        return {"out": out.detach(), "input_gradient": x.grad, "weight_gradients": gradients}
    model = state["model"]
    with torch.no_grad():
        if state["kind"] == "score":
            return model(input_ids=state["prompt"], attention_mask=state["mask"], use_cache=False).logits
        out = model(input_ids=state["prompt"], attention_mask=state["mask"], use_cache=True)
        logits = [out.logits]
        for tokens in state["tokens"]:
            out = model(input_ids=tokens, past_key_values=out.past_key_values, use_cache=True)
            logits.append(out.logits)
    return logits


# ----------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------------------------------------------------
def _mixer_work(case, name):
    """(parameters, FLOPs per token beside the projections) of a mixer; attention scores are counted by `_attention_flops`."""
    h, heads, d = case["hidden"], case["heads"], case["head_size"]
    if name == "attention":
        return h * d * (2 * heads + 2 * case["kv_heads"]), 0
    if name == "mamba":
        rank = max(h // 16, 16)
        return h * (2 * h + h // 2 + rank) + rank * h + h * h, 9 * h * 16
    if name == "gdn":
        return h * d * 4 * heads + 2 * h * heads, 6 * heads * d * d
    return h * d * 4 * heads + 4 * h * d + h * heads, 6 * heads * d * d


def _block_names(case):
    names = case["mixers"].split(",")
    return [names[i % len(names)] for i in range(case["layers"])]


def _parameters(case):
    if case["kind"] == "moe":
        return 3 * case["experts"] * case["hidden"] * case["ffn"]
    blocks = sum(_mixer_work(case, name)[0] + 3 * case["hidden"] * case["ffn"] for name in _block_names(case))
    return blocks + 2 * case["vocab"] * case["hidden"]


def _attention_flops(case, length):
    """Causal scores and outputs of one document through every attention layer, forward."""
    window = min(case["window"] or length, length)
    pairs = window * (window + 1) / 2 + (length - window) * window
    return 4 * pairs * case["heads"] * case["head_size"] * _block_names(case).count("attention")


def work(case):
    if case["kind"] == "moe":
        t, h, f, weights = case["tokens"], case["hidden"], case["ffn"], _parameters(case)
        # weights read and their gradients written (bf16); input, its gradient, output and output gradient
        return {"bytes": 4 * weights + 8 * t * h, "flops": 18 * t * case["top_k"] * h * f}
    parameters, embedding = _parameters(case), case["vocab"] * case["hidden"]
    scan = sum(_mixer_work(case, name)[1] for name in _block_names(case))
    if case["kind"] == "train":
        tokens = case["tokens"] * case["micro_batches"]
        attention = case["micro_batches"] * case["documents"] * _attention_flops(case, case["tokens"] // case["documents"])
        if case["lora_rank"]:
            # frozen weights: read once, forward and input gradients; the embedding table takes no gradient and no matmul
            return {"bytes": 2 * parameters + 16 * tokens, "flops": 4 * tokens * (parameters - embedding) + 3.5 * attention + 3 * scan * tokens}
        # master weights and two moments read and written, gradients and compute-dtype weights written
        return {"bytes": 30 * parameters + 16 * tokens, "flops": 6 * tokens * (parameters - embedding) + 3.5 * attention + 3 * scan * tokens}
    rows, prompt, new = case["rows"], case["prompt"], case.get("new", 0)
    kv_bytes = 4 * case["kv_heads"] * case["head_size"] * _block_names(case).count("attention")
    flops = 2 * rows * (prompt + new) * (parameters - embedding) + rows * _attention_flops(case, prompt + new) + scan * rows * (prompt + new)
    # every call reads the weights and the rows' keys and values; logits are written
    nbytes = 2 * (1 + new) * (parameters - embedding) + new * rows * (prompt + new / 2) * kv_bytes + 2 * rows * (prompt + new) * case["vocab"]
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """bf16 activations and weights, fp32 accumulation and optimizer state.  Every layer rounds its outputs to 8 bits, so two
    summation orders differ by a few 2^-9 at the logits and, after the way back, by about 1e-2 in gradients and moments."""
    return {"rel": 0.02, "max": 0.9} if case["kind"] == "train" else {"rel": 0.015, "max": 0.9}
