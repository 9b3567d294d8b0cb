"""What a user of the MoE layer has it do, as timed cases: inference from one token to a prefill, training steps of
small, ordinary and large layers, and the options that programs really use (top-1 routing, token rounding, caller-supplied
pairs with a skewed load, FP8 experts, biases with another activation).

Sizes are the benchmark configurations of this repository (`bench.py`), the layer shapes of the published figures they
come from, and generic ones of the same kind.  Weights are N(0, 0.02), activations and upstream gradients N(0, 1).
"""

import math
import os
import sys

import torch

_PACKAGE = os.path.join(os.getcwd(), "sonic-moe_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import sonicmoe  # noqa: E402
from sonicmoe.enums import ActivationType, is_glu  # noqa: E402
from sonicmoe.functional import forward_token_choice_rounding, moe_general_routing_inputs  # noqa: E402
from sonicmoe.functional.fp8 import moe_fp8_softmax_topk_layer  # noqa: E402

AUX_WEIGHT = 0.01  # weight of the load-balancing loss in the training loss


def _case(kind, T, H, I, E, K, **more):
    """kind: "infer" / "train" (the `MoE` module), "rounding" (token-rounding router + general routing), "pairs"
    (general routing with caller-supplied pairs, Zipf-skewed load), "fp8_infer" / "fp8_train" (FP8 experts)."""
    return dict(kind=kind, T=T, H=H, I=I, E=E, K=K, activation="swiglu", bias=False, scales="", **more)


def listed():
    cases = [
        # one token of a small layer: the latency of a decode step at batch 1
        _case("infer", 1, 2048, 768, 64, 4, name="decode_1"),
        # a decode step of a batch of 64 on the benchmark layer: most experts get a few rows each
        _case("infer", 64, 4096, 1024, 128, 8, name="decode_64"),
        # a short ragged prompt on the finest-grained layer of the benchmark family: about 64 rows per expert
        _case("infer", 1027, 4096, 512, 256, 16, name="prefill_1027"),
        # a long prefill on the benchmark layer
        _case("infer", 8192, 4096, 1024, 128, 8, name="prefill_8192"),
        # a training step of the smallest configuration (few experts, small hidden size)
        _case("train", 2048, 768, 256, 8, 2, name="train_2048_small"),
        # a training step of a mid-size layer with fine-grained experts
        _case("train", 24576, 1536, 256, 128, 8, name="train_24576_mid"),
        # the headline training step
        _case("train", 32768, 4096, 1024, 128, 8, name="train_32768"),
        # top-1 routing, an odd number of tokens
        _case("train", 8197, 2048, 1024, 64, 1, name="train_8197_top1"),
        # every expert's count rounded to a multiple of 128 by the token-rounding router
        _case("rounding", 16384, 4096, 1024, 256, 8, name="rounding_16384"),
        # pairs from the caller's own router, load as skewed as log-rank biases make it
        _case("pairs", 65536, 2048, 768, 64, 4, name="pairs_zipf_65536"),
        # one rank's experts of an FP8 layer with a large hidden size
        dict(_case("fp8_train", 8192, 7168, 2048, 32, 8, name="fp8_train_8192"), scales="ue8m0"),
        # expert biases and a non-gated activation
        dict(_case("train", 8191, 1024, 512, 32, 4, name="train_8191_gelu_bias"), activation="gelu", bias=True),
    ]
    return cases


def _cost(case):
    """Rough seconds at the rates of one GPU, to keep drawn cases below the largest listed one."""
    w = work(case)
    return w["flops"] / 1.4e15 + w["bytes"] / 6e12


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# (H, I, E, K) of the benchmark configurations and published figures
_LAYERS = [
    (4096, 1024, 128, 8), (4096, 512, 256, 16), (4096, 2048, 64, 4), (4096, 1024, 64, 4), (4096, 512, 128, 8),
    (4096, 256, 256, 16), (1536, 256, 128, 8), (1536, 512, 64, 4), (1536, 1024, 32, 2), (768, 256, 128, 8),
    (768, 512, 64, 4), (768, 1024, 32, 2), (768, 256, 8, 2), (2048, 768, 64, 4), (4096, 1024, 256, 8),
]


def draw(rng):
    most = _cost(max(listed(), key=_cost))
    while True:
        kind = rng.choice(["infer", "infer", "infer", "train", "train", "train", "rounding", "pairs", "fp8_infer",
                           "fp8_train"])
        if rng.random() < 0.6:
            H, I, E, K = rng.choice(_LAYERS)
        else:  # any layer of the same range
            step = 128 if kind.startswith("fp8") else 64
            H = step * rng.randint(512 // step, 4096 // step)
            I = step * rng.randint(max(1, 128 // step), 2048 // step)
            E = rng.choice([8, 16, 32, 64, 96, 128, 192, 256])
            K = rng.choice([k for k in (1, 2, 4, 6, 8, 16) if 2 * k <= E])
        if kind in ("infer", "fp8_infer"):
            T = _log_uniform(rng, 1, 16384)
        elif kind == "rounding":
            T = _log_uniform(rng, 2048, 32768)
        else:
            T = _log_uniform(rng, 256, 65536)
        if T > 256 and rng.random() < 0.5:
            T = T // 64 * 64
        case = _case(kind, T, H, I, E, K)
        if kind.startswith("fp8"):
            case["scales"] = rng.choice(["ue8m0", "ue8m0", "fp32"])
        elif kind in ("train", "infer") and rng.random() < 0.2:
            case["activation"] = rng.choice(["swiglu", "geglu", "reglu", "gelu", "relu", "silu", "relu_sq"])
            case["bias"] = rng.random() < 0.5
            n1 = 2 * I if is_glu(ActivationType(case["activation"])) else I
            if n1 % 128:
                continue
        if kind == "rounding" and T * K < 128 * E:
            continue  # most experts would round to nothing
        if _cost(case) <= most:
            return case


def _weights(case):
    """(router, up, down, up bias, down bias) in parameter storage order."""
    T, H, I, E = case["T"], case["H"], case["I"], case["E"]
    n1 = 2 * I if is_glu(ActivationType(case["activation"])) else I

    def normal(*shape):
        return torch.empty(*shape, dtype=torch.bfloat16, device="cuda").normal_(0, 0.02)

    router, w1, w2 = normal(E, H), normal(E, n1, H), normal(E, H, I)
    b1, b2 = (normal(E, n1), normal(E, H)) if case["bias"] else (None, None)
    return router, w1, w2, b1, b2


def prepare(case, seed):
    torch.manual_seed(seed)
    T, H, I, E, K = (case[k] for k in ("T", "H", "I", "E", "K"))
    train = case["kind"] not in ("infer", "fp8_infer")
    router, w1, w2, b1, b2 = _weights(case)
    state = dict(case=case, train=train)
    if case["kind"] in ("infer", "train"):
        with torch.device("meta"):
            moe = sonicmoe.MoE(E, K, H, I, ActivationType(case["activation"]), case["bias"], 0.02)
        named = {"router.weight": router, "c_fc.weight": w1, "c_proj.weight": w2}
        if case["bias"]:
            named.update({"c_fc.bias": b1, "c_proj.bias": b2})
        moe.load_state_dict(named, assign=True)
        moe.train(train)
        state.update(moe=moe, params=[p.requires_grad_(train) for p in moe.parameters()])
    else:
        params = [p.requires_grad_(train) for p in (router, w1, w2)]
        state.update(params=params)
    x = torch.randn(T, H, dtype=torch.bfloat16, device="cuda")
    state["x"] = x.requires_grad_(train)
    if train:
        state["dout"] = torch.randn(T, H, dtype=torch.bfloat16, device="cuda")
        state["daux"] = torch.full((), AUX_WEIGHT, device="cuda")
    if case["kind"] == "pairs":
        # the caller's routing decision: random logits plus 2 log(1 / rank) for a random ranking of the experts
        rank = torch.randperm(E, device="cuda").float() + 1
        logits = torch.randn(T, E, device="cuda") - 2 * torch.log(rank)
        top, experts = logits.topk(K, dim=-1)
        state["scores"] = torch.softmax(top, -1).reshape(-1).requires_grad_(True)
        state["experts"] = experts.to(torch.int32).reshape(-1)
        state["tokens"] = torch.arange(T, dtype=torch.int32, device="cuda").repeat_interleave(K)
        state["params"] = state["params"][1:]
    return state


def run(state):
    case = state["case"]
    kind, E, K, x = case["kind"], case["E"], case["K"], state["x"]
    if kind == "infer":
        with torch.no_grad():
            out, aux = state["moe"](x, is_inference_mode=True)
        return dict(out=out)
    if kind == "train":
        out, aux = state["moe"](x)
        grads = torch.autograd.grad([out, aux], [x, *state["params"]], [state["dout"], state["daux"]])
        return dict(out=out.detach(), aux=aux.detach(), grads=grads)
    if kind == "pairs":
        w1, w2 = state["params"]
        out, count = moe_general_routing_inputs(
            x, state["scores"], state["tokens"], state["experts"], w1.permute(1, 2, 0), None, w2.permute(1, 2, 0), None, E)
        grads = torch.autograd.grad(out, [x, state["scores"], w1, w2], state["dout"])
        return dict(out=out.detach(), count=count, grads=grads)
    router, w1, w2 = state["params"]
    if kind == "rounding":
        scores, tokens, experts = forward_token_choice_rounding(x, router, E, K, 128, "nr")
        out, count = moe_general_routing_inputs(
            x, scores, tokens, experts, w1.permute(1, 2, 0), None, w2.permute(1, 2, 0), None, E)
        grads = torch.autograd.grad(out, [x, router, w1, w2], state["dout"])
        return dict(out=out.detach(), count=count, grads=grads)
    if kind == "fp8_infer":
        with torch.no_grad():
            out, _, count = moe_fp8_softmax_topk_layer(
                x, router, w1.permute(1, 2, 0), None, w2.permute(1, 2, 0), None, K, is_inference_mode_enabled=True,
                scale_format=case["scales"])
        return dict(out=out, count=count)
    out, _, count = moe_fp8_softmax_topk_layer(
        x, router, w1.permute(1, 2, 0), None, w2.permute(1, 2, 0), None, K, scale_format=case["scales"])
    grads = torch.autograd.grad(out, [x, router, w1, w2], state["dout"])
    return dict(out=out.detach(), count=count, grads=grads)


def work(case):
    """Inputs read once, outputs written once; the weights of experts that no token can reach are not counted.
    FLOPs: the experts' GEMMs and the router's."""
    T, H, I, E, K = (case[k] for k in ("T", "H", "I", "E", "K"))
    n1 = 2 * I if is_glu(ActivationType(case["activation"])) else I
    train = case["kind"] not in ("infer", "fp8_infer")
    routed = case["kind"] != "pairs"
    reached = E * (1 - (1 - K / E) ** T)  # experts with at least one token, expected for an even load
    expert = (n1 + I) * H * 2
    weights = reached * expert + (E * H * 2 if routed else 0)
    bytes_ = weights + 2 * T * H * 2
    flops = 2 * T * K * (n1 + I) * H + (2 * T * H * E if routed else 0)
    if train:
        bytes_ += E * expert + (E * H * 2 if routed else 0) + 2 * T * H * 2
        flops *= 3
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # bf16 results of fp32 sums.  Measured: 2.5e-3 to 4.1e-3 against an fp32 oracle; FP8 against a simulation with the
    # same quantisation points 2.7e-3.  The router's sums in another order (library GEMM instead of the fused kernel)
    # change a result by 1e-4 at most.
    return {"rel": 1e-2}


def _activate(name, z):
    gate, up = (z[:, 0::2], z[:, 1::2]) if is_glu(ActivationType(name)) else (z, None)
    act = {"swiglu": torch.nn.functional.silu, "silu": torch.nn.functional.silu, "geglu": torch.nn.functional.gelu,
           "gelu": torch.nn.functional.gelu, "reglu": torch.relu, "relu": torch.relu,
           "relu_sq": lambda v: torch.relu(v).square()}[name](gate)
    return act if up is None else act * up


def _experts64(case, x, w1, b1, w2, b2, tokens, experts, scores, dout):
    """Output of the experts and, with dout, the gradients of x, w1, b1, w2, b2 and scores, expert by expert."""
    train = dout is not None
    out = torch.zeros_like(x)
    dx, ds = (torch.zeros_like(x), torch.zeros_like(scores)) if train else (None, None)
    dw = [None if w is None else torch.zeros(w.shape, dtype=torch.float64, device=x.device) if train else None
          for w in (w1, b1, w2, b2)]
    for e in range(case["E"]):
        pairs = (experts == e).nonzero()[:, 0]
        if pairs.numel() == 0:
            continue
        rows, s = tokens[pairs].long(), scores[pairs, None]
        up, down, xe = w1[e].double(), w2[e].double(), x[rows]
        z = (xe @ up.T + (0 if b1 is None else b1[e].double())).requires_grad_(train)
        with torch.enable_grad():
            y1 = _activate(case["activation"], z)
        y2 = y1.detach() @ down.T + (0 if b2 is None else b2[e].double())
        out.index_add_(0, rows, s * y2)
        if train:
            dy2 = dout[rows]
            ds[pairs] = (dy2 * y2).sum(-1)
            dy2 = dy2 * s
            dz, = torch.autograd.grad(y1, z, dy2 @ down)
            dx.index_add_(0, rows, dz @ up)
            dw[0][e], dw[2][e] = dz.T @ xe, dy2.T @ y1.detach()
            if b1 is not None:
                dw[1][e], dw[3][e] = dz.sum(0), dy2.sum(0)
    return out, dx, dw, ds


@torch.no_grad()
def exact(case, seed):
    """The layer in 64 bits, routed on the logits rounded to the activations' type as the layer defines them (near-ties
    would otherwise go to other experts).  FP8 cases: the layer without quantisation, which is what they approximate.
    Token rounding has none: which pairs it keeps hangs on ties among 16-bit probabilities."""
    kind, T, E, K = case["kind"], case["T"], case["E"], case["K"]
    if kind == "rounding" or work(case)["flops"] > 3e13:
        return None
    state = prepare(case, seed)
    x = state["x"].detach().double()
    train = state["train"]
    dout = state["dout"].double() if train else None
    if kind == "pairs":
        w1, w2 = (p.detach() for p in state["params"])
        tokens, experts, scores = state["tokens"], state["experts"], state["scores"].detach().double()
        out, dx, dw, ds = _experts64(case, x, w1, None, w2, None, tokens, experts, scores, dout)
        return dict(out=out, count=torch.bincount(experts, minlength=E).int(), grads=(dx, ds, dw[0], dw[2]))
    if "moe" in state:
        named = {n: p.detach() for n, p in state["moe"].named_parameters()}
        order = [n for n, _ in state["moe"].named_parameters()]
    else:
        order = ["router.weight", "c_fc.weight", "c_proj.weight"]
        named = {n: p.detach() for n, p in zip(order, state["params"])}
    router = named["router.weight"].double()
    w1, b1, w2, b2 = (named.get(n) for n in ("c_fc.weight", "c_fc.bias", "c_proj.weight", "c_proj.bias"))
    logits = (x @ router.T).to(state["x"].dtype).double()
    top, chosen = logits.sort(dim=-1, descending=True, stable=True)
    top, chosen = top[:, :K], chosen[:, :K]
    scores = torch.softmax(top, -1)
    experts = chosen.reshape(-1)
    count = torch.bincount(experts, minlength=E)
    tokens = torch.arange(T, device=x.device).repeat_interleave(K)
    out, dx, dw, ds = _experts64(case, x, w1, b1, w2, b2, tokens, experts, scores.reshape(-1), dout)
    if not train:
        return dict(out=out) if kind == "infer" else dict(out=out, count=count.int())
    ds = ds.view(T, K)
    dlogits = torch.zeros_like(logits).scatter_(1, chosen, scores * (ds - (ds * scores).sum(-1, keepdim=True)))
    if kind == "train":
        # E <share, p> with p the mean of the full softmax over the tokens (its sum is 1) and share the tokens' shares
        share, probs = count / count.sum(), torch.softmax(logits, -1)
        aux = E * (probs.mean(0) * share).sum()
        dprobs = (AUX_WEIGHT * E / T) * (share - (probs.mean(0) * share).sum())
        dlogits += probs * (dprobs - (probs * dprobs).sum(-1, keepdim=True))
    dx += dlogits @ router
    grads = {"router.weight": dlogits.T @ x, "c_fc.weight": dw[0], "c_fc.bias": dw[1], "c_proj.weight": dw[2],
             "c_proj.bias": dw[3]}
    grads = (dx, *[grads[n] for n in order])
    if kind == "train":
        return dict(out=out, aux=aux, grads=grads)
    return dict(out=out, count=count.int(), grads=grads)
