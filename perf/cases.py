"""Performance cases: the work a user of this framework has the GPU do, through its public entry points.

Six kinds of pass, each at small, ordinary, large and ragged sizes:

  functional   ``clipped_grad`` -> ``gaussian_noise`` -> optimizer on a small fp32 network, the form of ``examples/train_dpsgd.py``
  accumulate   ``FusedDPEngine.accumulate``: forward, backward, per-example norms, clip-weighted weight gradients of one
               (micro)batch; what the trainers call for every batch of an accumulation
  step         ``FusedDPEngine.step``: the same, then noise, optimizer and parameter write-back, and the metrics read to the host
  eval         ``token_nll`` without gradients: evaluation and the reference log-probabilities of preference training

The models are the configurations of ``bench.py`` with random weights; the large ones are cut to fewer layers (as with its
``--layers``) where the fp32 training state of the whole model would not leave room for a second copy.  Token ids are uniform.
"""
from __future__ import annotations

import functools

import torch

from opaque_b200 import optimizers
from opaque_b200.dpsgd import clipped_grad, gaussian_noise
from opaque_b200.engine.fused import FusedDPEngine
from opaque_b200.functional import make_functional
from opaque_b200.models import (GPT2Config, GPT2LMHeadModel, LlamaConfig, LlamaForCausalLM, MoEConfig, MoEForCausalLM,
                                shift_labels)
from opaque_b200.parallel.sharded import DPStepConfig
from opaque_b200.random import key

# per model: vocabulary, noise multiplier and learning rate of its benchmark configuration, share of the positions that are scored
_RUNS = {
    "gpt2-small": dict(vocab=50257, sigma=0.8, lr=1e-4, scored=1.0),
    "llama32-1b": dict(vocab=128256, sigma=0.7, lr=2e-4, scored=0.5),
    "llama3-8b": dict(vocab=128256, sigma=0.7, lr=2e-4, scored=0.5),
    "moe": dict(vocab=151936, sigma=1.0, lr=1e-4, scored=1.0),
}
_BLT = {"kind": "blt", "scale": [0.31, 0.18, 0.09, 0.04], "decay": [0.55, 0.85, 0.96, 0.995]}


def _case(name, kind, model, batch, seq, **kw):
    case = dict(kind=kind, model=model, layers=0, batch=batch, seq=seq, lora_rank=0, clipping="fixed", noise="gaussian", graph=False)
    if name:
        case["name"] = name
    case.update(kw)
    return case


def listed():
    return [
        # the smallest network one trains privately: fp32 784-256-10, Poisson batches of 256 expected (examples/train_dpsgd.py)
        _case("mlp-functional-256", "functional", "mlp", 256, 784),
        # full-parameter DP-SGD of GPT-2 small, two short records: a step bound by its number of launches; microbatches as CUDA graphs
        _case("gpt2-step-2x64", "step", "gpt2-small", 2, 64, graph=True),
        # the benchmark's microbatch of the same model
        _case("gpt2-accumulate-32x512", "accumulate", "gpt2-small", 32, 512, graph=True),
        # a Poisson draw of odd size, sequences padded to the longest record rather than to a round length; AUTO-S clipping
        _case("gpt2-accumulate-11x333", "accumulate", "gpt2-small", 11, 333, clipping="auto"),
        # LoRA fine-tuning with two short records: eager launches, host-bound
        _case("llama1b-lora-step-2x128", "step", "llama32-1b", 2, 128, lora_rank=16),
        # LoRA with a ragged batch of medium length
        _case("llama1b-lora-step-7x777", "step", "llama32-1b", 7, 777, lora_rank=8),
        # the headline configuration: Llama-3-8B architecture, LoRA r=16, a step of one whole microbatch (the largest case)
        _case("llama8b-lora-step-16x1024", "step", "llama3-8b", 16, 1024, lora_rank=16),
        # full-parameter DP-FTRL with four correlated-noise buffers (half of the 16 layers), one microbatch and its step
        _case("llama1b-blt-step-8x1024", "step", "llama32-1b", 8, 1024, layers=8, noise="blt"),
        # full-parameter DP-SGD of the mixture of experts (2 of 24 layers), the benchmark's microbatch
        _case("moe-accumulate-4x2048", "accumulate", "moe", 4, 2048, layers=2),
        # the same on few, short, odd-length records with a clipping group of its own for the experts
        _case("moe-accumulate-3x199", "accumulate", "moe", 3, 199, layers=1, clipping="group"),
        # evaluation: forward only, loss of every token
        _case("llama8b-eval-8x1024", "eval", "llama3-8b", 8, 1024, layers=16),
        _case("gpt2-eval-5x257", "eval", "gpt2-small", 5, 257),
    ]


def _log(rng, lo, hi):
    """A whole number from lo to hi, spread evenly over its logarithm."""
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def _length(rng, lo, hi):
    """A sequence length: half of them whole multiples of 64, as packed data has them."""
    n = _log(rng, lo, hi)
    return max(64, n // 64 * 64) if rng.random() < 0.5 and hi >= 64 else n


def draw(rng):
    which = rng.choice(("functional", "gpt2", "gpt2", "lora-1b", "lora-8b", "full-1b", "moe", "eval"))
    clipping = rng.choice(("fixed", "fixed", "auto"))
    if which == "functional":
        return _case("", "functional", "mlp", _log(rng, 16, 2048), 784)
    if which == "gpt2":
        seq = _length(rng, 40, 1024)
        graph = rng.random() < 0.5
        return _case("", rng.choice(("step", "accumulate")), "gpt2-small", _log(rng, 2, max(2, 16384 // seq)), seq, clipping=clipping, graph=graph)
    if which == "lora-1b":
        seq = _length(rng, 64, 2048)
        return _case("", "step", "llama32-1b", _log(rng, 1, max(1, 16384 // seq)), seq, lora_rank=rng.choice((8, 16, 32)), clipping=clipping)
    if which == "lora-8b":
        seq = _length(rng, 128, 2048)
        return _case("", "step", "llama3-8b", _log(rng, 1, max(1, 16384 // seq)), seq, layers=rng.choice((8, 16, 32)), lora_rank=16)
    if which == "full-1b":
        seq = _length(rng, 128, 1024)
        return _case("", "step", "llama32-1b", _log(rng, 1, max(1, 8192 // seq)), seq, layers=rng.choice((4, 8)), noise=rng.choice(("blt", "gaussian")))
    if which == "moe":
        seq = _length(rng, 128, 2048)
        return _case("", "accumulate", "moe", _log(rng, 1, max(1, 8192 // seq)), seq, layers=1, clipping=rng.choice(("fixed", "group")))
    model = rng.choice(("gpt2-small", "llama32-1b", "llama3-8b"))
    seq = _length(rng, 64, 1024)
    return _case("", "eval", model, _log(rng, 1, max(1, 8192 // seq)), seq, layers=16 if model == "llama3-8b" else 0)


# ------------------------------------------------------------------------------------------------------------ states

def _build_model(case, device):
    name = case["model"]
    if name == "gpt2-small":
        cfg = GPT2Config.small()
        if case["layers"]:
            cfg.n_layer = case["layers"]
        return GPT2LMHeadModel(cfg, device=device)
    if name == "moe":
        cfg = MoEConfig()
        if case["layers"]:
            cfg.num_hidden_layers = case["layers"]
        return MoEForCausalLM(cfg, device=device)
    cfg = LlamaConfig.llama32_1b() if name == "llama32-1b" else LlamaConfig.llama3_8b()
    if case["layers"]:
        cfg.num_hidden_layers = case["layers"]
    return LlamaForCausalLM(cfg, device=device)


def _expert_group(name: str) -> str:
    return "experts" if ".experts." in name else "dense"


def _prepare_functional(case, seed, device):
    gen = torch.Generator(device=device).manual_seed(seed)
    torch.manual_seed(seed)
    model = torch.nn.Sequential(torch.nn.Linear(784, 256), torch.nn.ReLU(), torch.nn.Linear(256, 10)).to(device)
    fmodel, params = make_functional(model, disable_autograd_tracking=True)

    def loss_fn(p, x, y):
        return torch.nn.functional.cross_entropy(fmodel(p, x.unsqueeze(0)), y.unsqueeze(0))
    grad_fn, clip_state = clipped_grad(loss_fn, clipping_norm=1.0, normalize_by=float(case["batch"]), batch_argnums=(1, 2), return_aux=True)
    noise_fn, noise_state = gaussian_noise(noise_multiplier=1.0, key=key(seed + 1))
    opt = optimizers.sgd(lr=0.1)
    return dict(x=torch.randn(case["batch"], 784, device=device, generator=gen),
                y=torch.randint(0, 10, (case["batch"],), device=device, generator=gen),
                params=params, grad_fn=grad_fn, clip_state=clip_state, noise_fn=noise_fn, noise_state=noise_state, opt=opt,
                opt_state=opt.init(params))


def prepare(case, seed):
    device = torch.device("cuda", torch.cuda.current_device())
    if case["kind"] == "functional":
        return dict(_prepare_functional(case, seed, device), kind="functional")
    run_cfg = _RUNS[case["model"]]
    torch.manual_seed(seed)
    model = _build_model(case, device)
    gen = torch.Generator(device=device).manual_seed(seed)
    ids = torch.randint(0, run_cfg["vocab"], (case["batch"], case["seq"]), device=device, generator=gen)
    batch = {"input_ids": ids, "labels": shift_labels(ids, run_cfg["scored"])}
    state = dict(kind=case["kind"], batch=batch)
    if case["kind"] == "eval":
        return dict(state, model=model.requires_grad_(False))
    loss_fn = model.per_example_loss
    if case["lora_rank"]:
        model.add_lora(case["lora_rank"], 2.0 * case["lora_rank"])
        with torch.no_grad():                    # a run that is under way: the B factors have left their zero start
            for name, p in model.named_parameters():
                if name.endswith("lora_B"):
                    p.normal_(std=0.01, generator=gen)
        # completion-only fine-tuning with a known prompt length: the head runs on the scored rows alone
        loss_fn = functools.partial(loss_fn, scored_suffix=case["seq"] - int(case["seq"] * (1.0 - run_cfg["scored"])))
    grouped = case["clipping"] == "group"
    engine = FusedDPEngine(model, clipping_norm={"experts": 0.6, "dense": 0.8} if grouped else 1.0, noise_multiplier=run_cfg["sigma"],
                           normalize_by=float(case["batch"]), key=key(seed),
                           step_config=DPStepConfig(lr=run_cfg["lr"], noise_bias_correction=True), microbatch_size=case["batch"],
                           mechanism=_BLT if case["noise"] == "blt" else None,
                           clipping_mode="auto" if case["clipping"] == "auto" else "clip",
                           group_of=_expert_group if grouped else None, cuda_graph=case["graph"])
    if case["graph"]:
        engine.prepare_graphs(loss_fn, batch)
    return dict(state, engine=engine, loss_fn=loss_fn)


# ------------------------------------------------------------------------------------------------------------ passes

def run(state):
    if state["kind"] == "eval":
        with torch.no_grad():
            return state["model"].token_nll(**state["batch"])
    if state["kind"] == "functional":
        (grads, aux), state["clip_state"] = state["grad_fn"](state["params"], state["x"], state["y"], state=state["clip_state"])
        noisy, state["noise_state"] = state["noise_fn"](grads, state["noise_state"])
        updates, state["opt_state"] = state["opt"].update(noisy, state["opt_state"], params=state["params"])
        state["params"] = optimizers.apply_updates(state["params"], updates)
        return {"params": list(state["params"]), "losses": aux.loss_values, "norms": aux.grad_norms}
    engine = state["engine"]
    if state["kind"] == "accumulate":
        # the clipped sum grows from pass to pass as over the microbatches of one logical batch
        res = engine.accumulate(state["loss_fn"], state["batch"])
        return {"grad": engine.space.grad.local, "losses": res.losses, "norms": res.norms}
    # The moments are linear and quadratic in the noised gradient.  The weights themselves are not compared: with noise bias
    # correction the denominator sqrt(v - phi) passes through zero for coordinates that carry noise only, and there a last-bit
    # difference of the gradient changes an update by orders of magnitude.
    engine.step(state["loss_fn"], state["batch"])
    return {"m": engine.opt.space.m, "v": engine.opt.space.v}


# ------------------------------------------------------------------------------------------------------- work, tolerance

def _shape(case):
    """(matrix parameters of the layers that a token passes, all parameters, vocabulary rows, width, attention width, layers)."""
    if case["model"] == "gpt2-small":
        d, n, v = 768, case["layers"] or 12, 50304
        return n * 12 * d * d, n * 12 * d * d + v * d + 1024 * d, v, d, d, n
    if case["model"] == "moe":
        d, n, v, ffn = 2048, case["layers"] or 24, 151936, 1408
        attn, expert, shared = 4 * d * d, 3 * d * ffn, 3 * d * 4 * ffn
        return n * (attn + 4 * expert + shared), n * (attn + 60 * expert + shared) + 2 * v * d, v, d, d, n
    if case["model"] == "llama32-1b":
        d, ffn, kv, n, tied = 2048, 8192, 512, case["layers"] or 16, 1
    else:
        d, ffn, kv, n, tied = 4096, 14336, 1024, case["layers"] or 32, 2
    layer = 2 * d * d + 2 * d * kv + 3 * d * ffn
    return n * layer, n * layer + tied * 128256 * d, 128256, d, d, n


def _trained(case):
    """Number of trained parameters."""
    _, total, _, d, _, layers = _shape(case)
    if not case["lora_rank"]:
        return total
    kv = 512 if case["model"] == "llama32-1b" else 1024
    return layers * case["lora_rank"] * (4 * d + 2 * (d + kv))          # q and o: d -> d; k and v: d -> kv


def work(case):
    """Least bytes and operations of one pass.

    Training: forward and data-gradient products, weight gradients of what is trained, attention.  Per-example norms are not
    counted: an implementation that formed each record's gradient once would have them for nothing.
    """
    b = case["batch"]
    if case["kind"] == "functional":
        p = 784 * 256 + 256 + 256 * 10 + 10
        return {"bytes": 4.0 * (2 * p + b * 785 + 2 * b), "flops": 6.0 * b * (784 * 256 + 256 * 10)}
    body, total, vocab, width, attn, layers = _shape(case)
    tokens = b * case["seq"]
    scored = tokens * (_RUNS[case["model"]]["scored"] if case["lora_rank"] or case["kind"] == "eval" else 1.0)
    core = 2.0 * layers * b * case["seq"] ** 2 * attn              # causal QK' and PV: half of 2 * 2 * T^2 * width each
    forward = 2.0 * tokens * body + 2.0 * scored * vocab * width + core
    if case["kind"] == "eval":
        return {"bytes": 2.0 * total + 20.0 * tokens, "flops": forward}
    trained = _trained(case)
    # per trained parameter: its gradient; in a step also master, m, v (read and written), the bf16 weight and the noise buffers
    state_bytes = 4.0 if case["kind"] == "accumulate" else 34.0 + (32.0 if case["noise"] == "blt" else 0.0)
    backward = forward + core + 2.0 * tokens * trained * 3 if case["lora_rank"] else 2.0 * forward + 0.5 * core
    return {"bytes": 2.0 * total + state_bytes * trained + 16.0 * tokens, "flops": forward + backward}


def tolerance(case):
    """About four times what two correct bf16 implementations were seen to differ by (the layers' products rounded once, or once
    more after the bias and the low-rank term): gradients of whole models 0.4 %, of the experts 0.5 % (0.7 % with two layers, where
    router ties fall differently)."""
    if case["kind"] == "functional":
        return {"rel": 1e-5, "max": 1e-3}
    if case["kind"] == "eval":
        return {"rel": 7e-4, "max": 6e-3}
    if case["kind"] == "accumulate":
        return {"rel": 0.03 if case["layers"] == 2 else 0.02, "max": 0.99}
    # A step's moments are mostly noise: its norm is sigma * sqrt(parameters), the clipped sum's at most the batch size.  Over two
    # steps the implementations above differed by this share of that largest sum: GPT-2 1 %, 1B with BLT noise 4 %, LoRA 2 to 4 %
    # (its factors sit behind every layer's roundings).
    share = 0.05 if case["model"] == "gpt2-small" else 0.16
    noise = _RUNS[case["model"]]["sigma"] * _trained(case) ** 0.5
    return {"rel": share * case["batch"] / noise, "max": 0.05}
