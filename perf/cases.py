"""The work that users of this package have it do, as cases that can be timed and compared.

A case is one MoE block of one model shape and one batch of tokens, run through the package's public calls:

* ``forward``: ``fp8_moe_forward`` - router, experts and weighted sum; per-tensor scales, or 128x128 block scales
  (as Hugging Face checkpoints carry them), with the deterministic or the atomic sum;
* ``layer``:   ``fp8_moe_forward_shared`` - a DeepSeek layer with its always-on shared experts in one pipeline;
* ``cached``:  ``fp8_moe_forward_fastcache`` - routing done by the caller, experts taken from the slots of an
  expert-residency cache through its id -> slot table.

The shapes are the benchmark configurations of this repository.  The batch sizes run from one token (decode of a
single sequence) over decode batches and ragged prompt chunks to full prefill batches.
"""

import math

import numpy as np
import torch

import blackwell_moe_b200 as bw

# hidden size, expert intermediate size, experts, experts per token
MIXTRAL_8X7B = dict(D=4096, H=14336, E=8, K=2)
DEEPSEEK_V2_LITE = dict(D=2048, H=1408, E=64, K=6)
QWEN3_30B = dict(D=2048, H=768, E=128, K=8)
QWEN36_35B = dict(D=2048, H=512, E=256, K=8)


def _case(name, entry, T, shape, scales="tensor", shared=0, slots=0, zipf=False, combine="deterministic"):
    return dict(name=name, entry=entry, T=T, scales=scales, shared=shared, slots=slots, zipf=zipf, combine=combine, **shape)


def listed():
    return [
        # decode of one sequence: two large experts' weights are read for one token
        _case("mixtral-1", "forward", 1, MIXTRAL_8X7B),
        # a decode batch that reaches every expert
        _case("mixtral-16", "forward", 16, MIXTRAL_8X7B),
        # a chunk of a long prompt, of no round length
        _case("mixtral-1003", "forward", 1003, MIXTRAL_8X7B),
        # full prefill
        _case("mixtral-16384", "forward", 16384, MIXTRAL_8X7B),
        # decode of one sequence through a layer of small experts: launches and latency count most here
        _case("deepseek-layer-1", "layer", 1, DEEPSEEK_V2_LITE, shared=2),
        # a decode batch of a server
        _case("deepseek-layer-64", "layer", 64, DEEPSEEK_V2_LITE, shared=2),
        # prefill
        _case("deepseek-layer-4096", "layer", 4096, DEEPSEEK_V2_LITE, shared=2),
        # decode of one sequence from a block-scaled checkpoint
        _case("qwen3-block-1", "forward", 1, QWEN3_30B, scales="block", zipf=True),
        # prefill with skewed expert popularity: a few experts get most of the rows
        _case("qwen3-block-8192", "forward", 8192, QWEN3_30B, scales="block", zipf=True),
        # a decode batch that reaches nearly all of 256 small experts
        _case("qwen36-block-128", "forward", 128, QWEN36_35B, scales="block"),
        # full prefill over 256 experts: many rows, little work for each
        _case("qwen36-block-32768", "forward", 32768, QWEN36_35B, scales="block"),
        # an expert-residency cache's call: odd batch, three quarters of the experts resident
        _case("deepseek-cached-37", "cached", 37, DEEPSEEK_V2_LITE, slots=48),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _multiple(rng, unit, lo, hi):
    return max(1, round(_log_uniform(rng, lo, hi) / unit)) * unit


def draw(rng):
    """One more case: the listed models' shapes or another of the same range, any batch size, any option."""
    entry, scales, own = rng.choice([("forward", "tensor", MIXTRAL_8X7B), ("forward", "tensor", DEEPSEEK_V2_LITE),
                                     ("layer", "tensor", DEEPSEEK_V2_LITE), ("forward", "block", QWEN3_30B),
                                     ("forward", "block", QWEN36_35B), ("cached", "tensor", DEEPSEEK_V2_LITE),
                                     ("cached", "block", QWEN3_30B)])
    if rng.random() < 0.4:
        shape = dict(own)
    else:
        E = rng.choice([8, 16, 32, 64, 128, 256] if scales == "tensor" and entry == "forward" else [64, 96, 128, 160])
        # weights of at most 1.5 GB; hidden sizes in multiples of 64, as models have them, and ragged intermediates
        D = _multiple(rng, 64, 1024, 4096)
        H = _multiple(rng, 16 if scales == "tensor" else 64, 320, max(384, min(14336, 1.5e9 / (3.0 * D * E))))
        shape = dict(D=D, H=H, E=E, K=rng.randint(2, 8))
    shared = rng.choice([1, 2]) if entry == "layer" else 0
    slots = rng.choice([shape["E"] * 3 // 4, shape["E"]]) if entry == "cached" else 0
    per_token = 6.0 * (shape["K"] + shared) * shape["D"] * shape["H"]
    t_max = min({"forward": 16384, "layer": 16384, "cached": 2048}[entry], 3e12 / per_token)
    combine = "atomic" if entry == "forward" and scales == "tensor" and rng.random() < 0.25 else "deterministic"
    case = _case("", entry, max(1, _log_uniform(rng, 1, t_max)), shape, scales, shared, slots,
                 zipf=rng.random() < 0.3, combine=combine)
    del case["name"]
    return case


def _generator(seed, tensor):
    # one stream per tensor, made from the seed alone
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1009 + tensor)


def _experts(case, seed, stream, count, H):
    """``count`` experts of intermediate size ``H``: weights ~N(0, 0.02^2), quantised as a loader does."""
    quantise = bw.quantize_expert_weights if case["scales"] == "tensor" else bw.quantize_expert_weights_block
    out = []
    for n, (rows, cols) in enumerate(((case["D"], H), (case["D"], H), (H, case["D"]))):
        w = torch.empty((count, rows, cols), dtype=torch.bfloat16, device="cuda")
        w.normal_(0.0, 0.02, generator=_generator(seed, stream + n))
        out.append(quantise(w))
    (g, sg), (u, su), (d, sd) = out
    return g, u, d, sg, su, sd


def _gate(case, seed):
    """The router's weight, ~N(0, 0.02^2).  Skewed popularity (Zipf 1.1) comes in through a constant input feature
    and a row of the weight that holds the experts' log rank."""
    g = _generator(seed, 7)
    w = torch.randn((case["D"], case["E"]), generator=g, device="cuda") * 0.02
    if case["zipf"]:
        bias = -1.1 * torch.log(torch.randperm(case["E"], generator=g, device="cuda").float() + 1.0)
        w[0] = bias - bias.mean()
    return w.to(torch.bfloat16)


def prepare(case, seed):
    case = dict(case)
    T, D, H, E, K = (case[k] for k in ("T", "D", "H", "E", "K"))
    x = torch.randn((T, D), generator=_generator(seed, 8), device="cuda").to(torch.bfloat16)
    if case["zipf"]:
        x[:, 0] = 1.0
    state = dict(case=case, x=x)
    if case["entry"] == "cached":
        state["weights"] = _experts(case, seed, 10, case["slots"], H)
        # the resident experts in random slots, and a batch that was routed to experts the cache has fetched
        g = _generator(seed, 9)
        resident = torch.randperm(E, generator=g, device="cuda")[: case["slots"]]
        state["remap"] = torch.full((E,), -1, dtype=torch.int32, device="cuda")
        state["remap"][resident] = torch.arange(case["slots"], dtype=torch.int32, device="cuda")
        state["routing"], ids = bw.top_k_router(x, _gate(case, seed)[:, resident].contiguous(), K)
        state["ids"] = resident[ids.long()].to(torch.int32)
        return state
    state["weights"] = _experts(case, seed, 10, E, H)
    state["gate"] = _gate(case, seed)
    if case["entry"] == "layer":
        g, u, d, sg, su, sd = _experts(case, seed, 20, 1, case["shared"] * H)
        *stacked, n = bw.stack_shared_experts(*state["weights"], g[0], u[0], d[0], sg[0], su[0], sd[0])
        state["weights"] = tuple(stacked)
        assert n == case["shared"]
    return state


def run(state):
    case = state["case"]
    if case["entry"] == "cached":
        return bw.fp8_moe_forward_fastcache(state["x"], state["routing"], state["ids"], state["remap"], *state["weights"],
                                            n_slots=case["slots"], top_k=case["K"])
    if case["entry"] == "layer":
        return bw.fp8_moe_forward_shared(state["x"], state["gate"], *state["weights"], top_k=case["K"],
                                         n_shared=case["shared"], routed_scale=1.0)
    return bw.fp8_moe_forward(state["x"], state["gate"], *state["weights"], top_k=case["K"], combine=case["combine"])


def _experts_used(case):
    """Distinct experts that a batch reaches: counted on a random draw of the router's logits, which are
    N(0, 0.02^2 * D) plus, where popularity is skewed, the experts' log rank."""
    n = case["slots"] or case["E"]
    rng = np.random.default_rng(0)
    logits = rng.standard_normal((min(case["T"], 2048), n)) * 0.02 * math.sqrt(case["D"])
    if case["zipf"]:
        logits += -1.1 * np.log(rng.permutation(n) + 1.0)
    return len(np.unique(np.argpartition(-logits, case["K"] - 1, axis=1)[:, : case["K"]]))


def work(case):
    T, D, H, K, shared = (case[k] for k in ("T", "D", "H", "K", "shared"))
    used = _experts_used(case) + shared
    scales = 12 if case["scales"] == "tensor" else 12 * (-(-D // 128)) * (-(-H // 128))
    routed_by_caller = case["entry"] == "cached"
    return {
        # every used expert's weights, the router's weight (or the caller's routing), x in, the result out
        "bytes": used * (3.0 * D * H + scales) + (8.0 * T * K if routed_by_caller else 2.0 * D * case["E"]) + 4.0 * T * D,
        "flops": float(T) * (6.0 * (K + shared) * D * H + (0.0 if routed_by_caller else 2.0 * D * case["E"])),
    }


def tolerance(case):
    # Four times the largest distance seen between this package's results and the same recipe with its sums in fp64
    # (the same codes and rounding points; listed shapes and ten drawn ones).  A sum in another order moves a bf16
    # rounding of h here and there, which moves an E4M3 code, and where it moves the largest |h| of an expert's rows
    # it moves that expert's scale: rel 2e-5 to 4e-4, once 2.1e-3 (per-tensor scales); 2.5e-4 (block scales, whose
    # groups are too small for one of them to show).  Single values: 0.04 of the larger of value and RMS.
    if case["combine"] == "atomic":
        # K bf16 additions in order of arrival, each off by up to 2^-9: sqrt(8) * 2^-9 / sqrt(3) = 3.2e-3
        return {"rel": 1.2e-2, "max": 0.17}
    return {"rel": 8e-3 if case["scales"] == "tensor" else 1e-3, "max": 0.17}
