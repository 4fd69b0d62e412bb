"""The workloads this repository's speed is judged by: one pass of each is one call of the public API as a program that
trains, serves or dispatches to the MoE layer makes it.

A case is a dict of plain values.  `kind` says which use of the framework it is:

  train     forward + backward of the pre-routed expert compute (`run_sonic_moe`) for one micro-batch, weight gradients
            accumulated into the parameters' fp32 `main_grad` (what a training framework does between optimizer steps)
  payload   the same on the receiving side of an expert-parallel FP8 dispatch: e4m3 tokens + ue8m0 scales in, slots of
            experts that live on other ranks marked -1, the gradient of the output arriving as an FP8 payload too
  module    forward + backward of the `MoE` module (router, auxiliary loss, gradients left on the parameters in bf16)
  infer     forward of the `MoE` module in inference mode (decode: few tokens; prefill: many)
  metadata  the routing metadata alone, as a host framework asks for it after its dispatch
  weights   the FP8 copies of a layer's weights made anew, once per optimizer step

`layer` names the sizes (H, I, E, K) of the layer; they are those of the repository's benchmark and tests.  `T` is the
number of tokens, `E` (where given) replaces the layer's number of experts.  `skew` adds a Zipf(1.2) bias to the router logits (some experts busy, some idle or empty).
"""
import math
import os
import sys

import torch

sys.path.insert(1, os.path.join(os.getcwd(), "supersonic-moe_b200"))

import sonicmoe  # noqa: E402
from sonicmoe import MoE, run_sonic_moe  # noqa: E402
from sonicmoe.enums import ActivationType  # noqa: E402
from sonicmoe.ernie_compat import deepep_topk_to_sonic_metadata  # noqa: E402
from sonicmoe.functional import Fp8CombineGradHandle, drop_weight_fp8, precompute_weight_fp8, weight_fp8  # noqa: E402
from sonicmoe.quack_utils import quantize_activation_blockscaled_fast  # noqa: E402

# (H, I, E, K)
LAYERS = {
    "tiny": (256, 128, 8, 2),            # the smallest layer the repository runs (smoke test)
    "base": (3072, 1536, 8, 8),          # the headline layer
    "base_e16": (3072, 1536, 16, 8),     # the published expert-count sweep of the headline layer
    "base_e32": (3072, 1536, 32, 8),
    "wide": (4096, 4096, 8, 8),          # the peak-utilisation layer; H is no multiple of 384
    "fine": (2048, 768, 128, 8),         # fine-grained experts
    "large": (6144, 3072, 8, 8),         # one rank's 8 experts of the 64-expert layer
}
GLOBAL_EXPERTS = 64                      # of the layer "large": tokens choose among these, 8 of them are local


def listed():
    return [
        # routing metadata of one dispatch: integers only, launches count
        dict(name="metadata_16384", kind="metadata", layer="fine", T=16384, skew=True),
        # one decode step of a serving batch over 128 experts, four real rows per expert
        dict(name="decode_64", kind="infer", layer="fine", T=64, skew=False),
        # a prompt chunk through the headline layer
        dict(name="prefill_2048", kind="infer", layer="base", T=2048, skew=False),
        # the smallest training step: launch latency and host work
        dict(name="train_tiny", kind="train", layer="tiny", T=256, skew=False),
        # the published sweep over token counts starts here
        dict(name="train_1024", kind="train", layer="base", T=1024, skew=False),
        # the headline workload
        dict(name="train_8192", kind="train", layer="base", T=8192, skew=False),
        # the peak-utilisation workload
        dict(name="train_wide_8192", kind="train", layer="wide", T=8192, skew=False),
        # many small experts under a skewed router: short reductions, padding, idle experts
        dict(name="train_fine_skewed_16384", kind="train", layer="fine", T=16384, skew=True),
        # an nn.Module user: router and auxiliary loss included, bf16 gradients on the parameters
        dict(name="module_e32_4096", kind="module", layer="base_e32", T=4096, skew=False),
        # what one of eight expert-parallel ranks computes on the (odd number of) tokens it received
        dict(name="payload_3001", kind="payload", layer="large", T=3001, skew=False),
        # after every optimizer step
        dict(name="weights_fine", kind="weights", layer="fine", T=0, skew=False),
    ]


# token range of each kind, and the layers it is drawn with
RANGES = {
    "train": ((128, 16384), ("tiny", "base", "base_e16", "base_e32", "wide", "fine")),
    "module": ((128, 8192), ("tiny", "base", "base_e32", "fine")),
    "payload": ((256, 8192), ("large",)),
    "infer": ((1, 8192), ("tiny", "base", "base_e32", "wide", "fine")),
    "metadata": ((128, 65536), ("tiny", "base", "base_e32", "fine")),
    "weights": ((0, 0), ("base", "base_e32", "wide", "fine")),
}
# how often each use is drawn
KINDS = ("train",) * 4 + ("infer",) * 3 + ("module", "payload", "metadata", "weights")


def _sizes(case):
    H, I, E, K = LAYERS[case["layer"]]
    return H, I, case.get("E", E), K


def draw(rng):
    kind = rng.choice(KINDS)
    (lo, hi), layers = RANGES[kind]
    layer = rng.choice(layers)
    if layer == "wide":
        hi = min(hi, 8192)
    T = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) if hi else 0
    if T > 8 and rng.random() < 0.25:
        T = T // 8 * 8                    # round batch sizes are as usual as ragged ones
    case = dict(kind=kind, layer=layer, T=T, skew=layer == "fine" and rng.random() < 0.5)
    if kind == "weights":
        case.update(skew=False, E=int(round(math.exp(rng.uniform(math.log(2), math.log(32))))))
    return case


# ------------------------------------------------------------------------------------------------ inputs
def _route(g, T, E, K, skew):
    """Router decisions of T tokens: logits N(0,1) (+ log Zipf), top-K, softmax over the K selected."""
    logits = torch.randn(T, E, generator=g, device="cuda")
    if skew:
        p = torch.arange(1, E + 1, dtype=torch.float32, device="cuda") ** -1.2
        logits += torch.log(p / p.sum())[torch.randperm(E, generator=g, device="cuda")]
    vals, idx = logits.topk(K, dim=-1)
    return idx.to(torch.int32), torch.softmax(vals, dim=-1)


def _tokens(g, T, H):
    return torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)


def _weights(g, H, I, E):
    w1 = torch.randn(E, 2 * I, H, generator=g, device="cuda").mul_(0.02).to(torch.bfloat16)
    w2 = torch.randn(E, H, I, generator=g, device="cuda").mul_(0.02).to(torch.bfloat16)
    return w1.requires_grad_(True), w2.requires_grad_(True)


def _module(g, H, I, E, K, skew):
    with torch.device("cuda"):
        m = MoE(E, K, H, I, ActivationType.SWIGLU, add_bias=False, std=0.02).to(torch.bfloat16)
    with torch.no_grad():
        for p, std in ((m.router.weight, 1.0 / math.sqrt(H)), (m.c_fc.weight, 0.02), (m.c_proj.weight, 0.02)):
            p.copy_(torch.randn(p.shape, generator=g, device="cuda").mul_(std))
        if skew:          # tokens of a trained model lean towards some experts: the first columns carry the bias
            m.router.weight[:, :8] += (torch.arange(1, E + 1, device="cuda").float() ** -1.2).log()[:, None] / 8
    return m


def prepare(case, seed):
    kind, T = case["kind"], case["T"]
    H, I, E, K = _sizes(case)
    g = torch.Generator(device="cuda").manual_seed(seed)
    s = dict(kind=kind, T=T, E=E, K=K)
    if kind == "metadata":
        s["idx"], s["probs"] = _route(g, T, E, K, case["skew"])
        return s
    if kind in ("module", "infer"):
        s["m"] = _module(g, H, I, E, K, case["skew"])
        s["x"] = _tokens(g, T, H)
        if case["skew"]:
            s["x"][:, :8] = 1.0
        precompute_weight_fp8(s["m"].c_fc.weight, s["m"].c_proj.weight)
        if kind == "infer":
            s["m"].eval()
        else:
            s["x"].requires_grad_(True)
            s["dy"] = _tokens(g, T, H)
            s["daux"] = torch.tensor(0.01, device="cuda")
        return s
    s["w1"], s["w2"] = _weights(g, H, I, E)
    if kind == "weights":
        return s
    s["w1"].main_grad = torch.zeros(E, 2 * I, H, dtype=torch.float32, device="cuda")
    s["w2"].main_grad = torch.zeros(E, I, H, dtype=torch.float32, device="cuda")
    precompute_weight_fp8(s["w1"], s["w2"])
    s["x"], s["dy"] = _tokens(g, T, H), _tokens(g, T, H)
    if kind == "train":
        s["idx"], s["probs"] = _route(g, T, E, K, case["skew"])
        s["x"].requires_grad_(True)
        s["probs"].requires_grad_(True)
        return s
    # payload: a received token has at least one local expert; the other slots belong to other ranks
    idx, probs = _route(g, T, GLOBAL_EXPERTS, K, case["skew"])
    idx = torch.where(idx < E, idx, torch.full_like(idx, -1))
    none = (idx >= 0).sum(1) == 0
    idx[none, 0] = torch.randint(0, E, (int(none.sum()),), generator=g, device="cuda", dtype=torch.int32)
    s["idx"], s["probs"] = idx, probs.requires_grad_(True)
    s["x"], s["x_scale"] = quantize_activation_blockscaled_fast(s["x"])
    s["dy_q"], s["dy_scale"] = quantize_activation_blockscaled_fast(s["dy"])
    s["dy"] = torch.zeros((), dtype=torch.bfloat16, device="cuda").expand(T, H)       # carries the autograd edge only
    s["holder"] = torch.zeros(T, H, dtype=torch.bfloat16, device="cuda", requires_grad=True)      # receives dx
    return s


# ------------------------------------------------------------------------------------------------ one pass
def run(s):
    kind = s["kind"]
    if kind == "metadata":
        r = deepep_topk_to_sonic_metadata(s["idx"], s["probs"], None, s["E"], sync_free_sizing=True)
        return [t for t in r if isinstance(t, torch.Tensor)]
    if kind == "weights":
        w1, w2 = s["w1"], s["w2"]
        drop_weight_fp8(w1, w2)
        precompute_weight_fp8(w1, w2)
        return [weight_fp8(w, t) for w in (w1, w2) for t in (False, True)]
    if kind == "infer":
        with torch.no_grad():
            return s["m"](s["x"], is_inference_mode=True, use_fp8=True)[0]
    if kind == "module":
        m, x = s["m"], s["x"]
        m.zero_grad(set_to_none=True)
        x.grad = None
        out, aux = m(x, use_fp8=True)
        torch.autograd.backward((out, aux), (s["dy"], s["daux"]))
        return [out, aux, x.grad, m.router.weight.grad, m.c_fc.weight.grad, m.c_proj.weight.grad]
    w1, w2, probs = s["w1"], s["w2"], s["probs"]
    probs.grad = None
    if kind == "train":
        x = s["x"]
        x.grad = None
        out = run_sonic_moe(x, s["idx"], probs, s["K"], s["E"], w1, w2, fp8=True)
    else:
        x = s["holder"]
        x.grad = None
        handle = Fp8CombineGradHandle()
        handle.put(s["dy_q"].view(torch.uint8), s["dy_scale"])
        out = run_sonic_moe(s["x"], s["idx"], probs, s["K"], s["E"], w1, w2, fp8=True, fp8_scale=s["x_scale"],
                            fp8_combine_grad_handle=handle, sync_free_sizing=True, grad_holder=x)
    out.backward(s["dy"])
    return [out, x.grad, probs.grad, w1.main_grad, w2.main_grad]


# ------------------------------------------------------------------------------------------------ what a pass needs
def work(case):
    kind, T = case["kind"], case["T"]
    H, I, E, K = _sizes(case)
    W = 3 * E * H * I                                   # weights of the layer
    SC = 33 / 32                                        # e4m3 payload with its 1x32 scales
    if kind == "metadata":                              # indices and scores in; the eight index / score tables out
        TK = T * K
        return {"bytes": 8 * TK + 4 * (3 * (TK + 128 * E) + 2 * TK + T + E), "flops": 0}
    if kind == "weights":                               # bf16 in once, two e4m3 copies out
        return {"bytes": W * (2 + 2 * SC), "flops": 0}
    if kind == "infer":
        touched = E * (1 - (1 - K / E) ** T) if K < E else E
        return {"bytes": 4 * T * H + 2 * E * H + W * SC * touched / E, "flops": 6 * T * K * H * I + 2 * T * H * E}
    if kind == "module":                                # tokens and gradients in bf16, weights in e4m3, bf16 gradients out
        return {"bytes": 8 * T * H + W * SC + 2 * W + 4 * E * H, "flops": 18 * T * K * H * I + 6 * T * H * E}
    main_grad = 8 * W                                   # fp32, read and written
    if kind == "train":
        return {"bytes": 8 * T * H + 12 * T * K + W * SC + main_grad, "flops": 18 * T * K * H * I}
    pairs = T * max(1.2, K * E / GLOBAL_EXPERTS)        # local (token, expert) pairs of T received tokens
    return {"bytes": T * H * (2 * SC + 4) + 12 * T * K + W * SC + main_grad, "flops": 18 * pairs * H * I}


def tolerance(case):
    if case["kind"] in ("metadata", "weights"):
        return "exact"
    # e4m3 and bf16 intermediates: another order of the fp32 sums moves a few values across a rounding boundary.  With
    # H and I permuted in blocks of 32 (same groups, other order) the outputs of four layers moved by 3.7e-4 at most,
    # single values by 0.09
    return {"rel": 1.5e-3, "max": 0.35}
