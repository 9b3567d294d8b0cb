"""Functional / autograd layer of the MoE hot path, backed by libsonicmoe_b200.so.

Public entry points keep the reference's names and argument conventions
(sonicmoe/functional/__init__.py:423-562):

* ``moe_TC_softmax_topk_layer``  – router linear, top-k + softmax, routed experts (token-choice top-k);
* ``moe_general_routing_inputs`` – routed experts for caller-supplied (score, token, expert) pairs with a
  variable number of experts per token (token rounding uses this);
* ``TC_topk_router_metadata`` / ``general_routing_router_metadata`` – the grouped-row index vectors;
* ``forward_token_choice_rounding`` – the token-rounding router.

Everything runs on the tensors' CUDA device on the *current* stream; the ``stream_id`` arguments are
accepted for call compatibility and ignored (the reference requires them to equal the current stream).
What is saved for backward follows the reference's recompute policy: x, z (pre-activation), scores and
the index vectors are kept; gathered inputs, y1 and y2 are not.
"""

from __future__ import annotations

import os
from contextlib import contextmanager
from dataclasses import dataclass

import torch
import torch.nn.functional as F
from torch.autograd import forward_ad

from .. import _lib
from .._lib import check, lib, ptr, stream_ptr
from ..count_cumsum import count_cumsum
from ..enums import ActivationType, is_glu
from .token_rounding import forward_token_choice_rounding

__all__ = [
    "count_cumsum",
    "enable_quack_gemm",
    "is_using_quack_gemm",
    "moe_TC_softmax_topk_layer",
    "moe_general_routing_inputs",
    "TC_topk_router_metadata",
    "general_routing_router_metadata",
    "forward_token_choice_rounding",
    "topk_softmax",
    "set_fused_combine",
    "set_fused_router",
    "layer_router_logits",
]


# ------------------------------------------------------------------------------------------------
# toggles
# ------------------------------------------------------------------------------------------------
@contextmanager
def enable_quack_gemm(enable: bool = True):
    """Accepted for source compatibility with the reference (sonicmoe/functional/utils.py:12-25).

    The reference switches to its QuACK GEMMs here; this build has a single GEMM implementation, so the
    context manager changes nothing.
    """
    yield


def is_using_quack_gemm() -> bool:
    return False


# Down-projection epilogue: False = write y2 (TK,H) and reduce it with a deterministic gather-sum;
# True = scatter-reduce into an fp32 (T,H) accumulator from inside the GEMM epilogue (atomic adds).
_FUSED_COMBINE = os.getenv("SONICMOE_FUSED_COMBINE", "0") == "1"


def set_fused_combine(enable: bool) -> bool:
    """Select the fused scatter-reduce epilogue for the down projection; returns the previous setting."""
    global _FUSED_COMBINE
    prev, _FUSED_COMBINE = _FUSED_COMBINE, bool(enable)
    return prev


# ------------------------------------------------------------------------------------------------
# routing metadata
# ------------------------------------------------------------------------------------------------
@dataclass
class Route:
    """Index vectors of one routing decision (all int32, on the activations' device)."""

    expert_frequency: torch.Tensor         # (E,)   rows per expert
    expert_frequency_offset: torch.Tensor  # (E+1,) first grouped row of each expert
    x_gather_idx: torch.Tensor             # (TK,)  token of each grouped row
    s_scatter_idx: torch.Tensor            # (TK,)  flat (token, k) slot of each grouped row
    s_reverse_scatter_idx: torch.Tensor    # (TK,)  grouped row of each flat slot
    token_offset: torch.Tensor | None      # (T+1,) first flat slot of each token; None = fixed K per token
    K: int                                 # experts per token when token_offset is None
    # called in the backward pass with dx as soon as it exists (before the weight-gradient GEMMs are launched): an
    # expert-parallel caller starts sending dx back to the tokens' ranks while those GEMMs run
    on_dx: object = None
    # shared by the chunks of one batch whose rows reach the same experts in several calls (`WeightGradSum`)
    wgrad_sum: object = None


class WeightGradSum:
    """One pair of weight-gradient buffers for ``chunks`` calls of the routed experts on the same weights.

    The first backward pass to run stores its dW1 / dW2, every later one adds to them inside the weight-gradient
    GEMMs' epilogue (`smoe_*_weight_grad_accumulate`), and only the last returns gradients to autograd (the others
    return None).  The result is what autograd's own accumulation of per-chunk bf16 gradients gives (bit for bit
    with two chunks), without a full set of gradient tensors per chunk and the read-add-write pass that adds them.
    Every chunk's backward pass has to run (all chunk outputs feed the loss)."""

    def __init__(self, chunks: int):
        self.remaining = chunks
        self.dw1 = self.dw2 = None

    def buffers(self, w1e, w2e):
        """(dw1, dw2, accumulate?) for the chunk whose backward pass runs now."""
        first = self.dw1 is None
        if first:
            self.dw1, self.dw2 = torch.empty_like(w1e), torch.empty_like(w2e)
        return self.dw1, self.dw2, not first

    def finish_chunk(self):
        """The gradients if this was the last chunk, else (None, None)."""
        self.remaining -= 1
        if self.remaining > 0:
            return None, None
        dw1, dw2 = self.dw1, self.dw2
        self.dw1 = self.dw2 = None
        return dw1, dw2


def _one_row_per_token(route: "Route", T: int) -> bool:
    """Every token has exactly one routed row (top-1 routing, or the rows an expert-parallel rank received): the
    combine and the dX reduction are permutations, which the GEMM epilogues write directly."""
    return route.token_offset is None and route.K == 1 and route.x_gather_idx.numel() == T


def _route_metadata(expert_idx: torch.Tensor, token_idx: torch.Tensor | None, E: int, K: int) -> Route:
    dev = expert_idx.device
    _lib.require_cuda(expert_idx, "expert indices")
    n = expert_idx.numel()
    expert_idx = expert_idx.contiguous()
    if expert_idx.dtype != torch.int32:
        expert_idx = expert_idx.to(torch.int32)
    if token_idx is not None:
        token_idx = token_idx.contiguous()
        if token_idx.dtype != torch.int32:
            token_idx = token_idx.to(torch.int32)
    with torch.cuda.device(dev):
        freq = torch.empty(E, dtype=torch.int32, device=dev)
        off = torch.empty(E + 1, dtype=torch.int32, device=dev)
        idx3 = torch.empty(3, n, dtype=torch.int32, device=dev)
        ws = _lib.workspace(lib.smoe_route_metadata_workspace_bytes(E), dev)
        s_scatter, s_reverse, x_gather = idx3.unbind(0)
        rc = lib.smoe_route_metadata(
            expert_idx.data_ptr(), ptr(token_idx), n, E, max(K, 1), freq.data_ptr(), off.data_ptr(),
            s_scatter.data_ptr(), s_reverse.data_ptr(), x_gather.data_ptr(), ws.data_ptr(), stream_ptr(dev),
        )
        check(rc, "route_metadata")
    return Route(freq, off, x_gather, s_scatter, s_reverse, None, K)


def TC_topk_router_metadata(topk_router_indices: torch.Tensor, expert_frequency_offset: torch.Tensor, K: int):
    """Index vectors for token-choice top-k routing (reference: sonicmoe/functional/__init__.py:19-46).

    ``expert_frequency_offset`` is the inclusive cumsum the reference passes in; only its length (E) is
    used, the offsets are recomputed together with the sort.  Rows of one expert are ordered by flat slot
    (a stable sort; the reference's argsort leaves that order unspecified).
    Returns (expert_frequency_offset with leading 0, x_gather_idx, s_scatter_idx, s_reverse_scatter_idx,
    num_activated_expert_per_token_offset).
    """
    E = expert_frequency_offset.numel()
    r = _route_metadata(topk_router_indices.reshape(-1), None, E, K)
    T = topk_router_indices.shape[0]
    tok_off = torch.arange(0, T * K + 1, K, dtype=torch.int32, device=topk_router_indices.device)
    return r.expert_frequency_offset, r.x_gather_idx, r.s_scatter_idx, r.s_reverse_scatter_idx, tok_off


def _sorted_offsets(sorted_idx: torch.Tensor, T: int) -> torch.Tensor:
    dev = sorted_idx.device
    with torch.cuda.device(dev):
        out = torch.empty(T + 1, dtype=torch.int32, device=dev)
        check(lib.smoe_sorted_offsets(sorted_idx.data_ptr(), sorted_idx.numel(), T, out.data_ptr(), stream_ptr(dev)),
              "sorted_offsets")
    return out


def general_routing_router_metadata(
    router_scores_selected: torch.Tensor, sorted_selected_T: torch.Tensor, selected_E: torch.Tensor, T: int, E: int
):
    """Index vectors for caller-supplied pairs sorted by token (reference: functional/__init__.py:49-82).

    Returns (expert_frequency, expert_frequency_offset, x_gather_idx, s_scatter_idx, s_reverse_scatter_idx,
    num_activated_expert_per_token_offset).
    """
    tok = sorted_selected_T.contiguous().to(torch.int32)
    r = _route_metadata(selected_E, tok, E, 0)
    tok_off = _sorted_offsets(tok, T)
    return (r.expert_frequency, r.expert_frequency_offset, r.x_gather_idx, r.s_scatter_idx,
            r.s_reverse_scatter_idx, tok_off)


# ------------------------------------------------------------------------------------------------
# top-k + softmax
# ------------------------------------------------------------------------------------------------
class _TopkSoftmax(torch.autograd.Function):
    """scores (T,K) fp32 = softmax over the K largest logits of each row; indices (T,K) int32.

    Largest first; equal logits are ordered by lower expert id.  Reference:
    TC_Softmax_Topk_Router_Function (sonicmoe/functional/__init__.py:85-111).
    """

    @staticmethod
    def forward(ctx, router_logits: torch.Tensor, K: int):
        _lib.require_cuda(router_logits, "router_logits")
        if router_logits.dtype not in (torch.float32, torch.bfloat16):
            raise TypeError(f"router logits must be fp32 or bf16, got {router_logits.dtype}")
        logits = router_logits.contiguous()
        T, E = logits.shape
        dev = logits.device
        with torch.cuda.device(dev):
            scores = torch.empty(T, K, dtype=torch.float32, device=dev)
            indices = torch.empty(T, K, dtype=torch.int32, device=dev)
            check(lib.smoe_topk_softmax(logits.data_ptr(), _lib.dtype_code(logits.dtype), scores.data_ptr(),
                                        indices.data_ptr(), T, E, K, stream_ptr(dev)), "topk_softmax")
        ctx.save_for_backward(scores, indices)
        ctx.E = E
        ctx.logits_dtype = logits.dtype
        ctx.mark_non_differentiable(indices)
        return scores, indices

    @staticmethod
    def backward(ctx, dscores: torch.Tensor, _unused):
        scores, indices = ctx.saved_tensors
        T, K = scores.shape
        dev = scores.device
        dscores = dscores.contiguous().float()
        with torch.cuda.device(dev):
            dlogits = torch.empty(T, ctx.E, dtype=ctx.logits_dtype, device=dev)
            check(lib.smoe_softmax_topk_backward(dlogits.data_ptr(), _lib.dtype_code(ctx.logits_dtype),
                                                 dscores.data_ptr(), scores.data_ptr(), indices.data_ptr(),
                                                 T, ctx.E, K, stream_ptr(dev)), "softmax_topk_backward")
        return dlogits, None


def topk_softmax(router_logits: torch.Tensor, K: int) -> tuple[torch.Tensor, torch.Tensor]:
    return _TopkSoftmax.apply(router_logits, K)


# ------------------------------------------------------------------------------------------------
# fused routing front end
# ------------------------------------------------------------------------------------------------
_FUSED_ROUTER = os.getenv("SONICMOE_FUSED_ROUTER", "1") != "0"


def set_fused_router(enable: bool) -> bool:
    """Use the one-pass router kernel where it applies (default) or always the separate router linear + top-k;
    returns the previous setting."""
    global _FUSED_ROUTER
    prev, _FUSED_ROUTER = _FUSED_ROUTER, bool(enable)
    return prev


def fused_router_applies(x: torch.Tensor, router_w: torch.Tensor, K: int) -> bool:
    return (_FUSED_ROUTER and x.is_cuda and x.dtype == torch.bfloat16 and router_w.dtype == torch.bfloat16
            and not torch.compiler.is_compiling()
            and bool(lib.smoe_router_forward_supported(x.shape[1], router_w.shape[0], K)))


@torch.no_grad()
def layer_router_logits(x: torch.Tensor, router_w: torch.Tensor, K: int) -> torch.Tensor:
    """The router logits exactly as `moe_TC_softmax_topk_layer` computes them for these inputs (the fused kernel's
    where it applies, the router linear's otherwise) -- what a check of the routing decision must be run on."""
    if fused_router_applies(x, router_w, K):
        return _FusedRouter.apply(x, router_w, K)[0]
    return F.linear(x if x.dtype == router_w.dtype else x.to(router_w.dtype), router_w)


class _FusedRouter(torch.autograd.Function):
    """(logits (T,E) bf16, scores (T,K) fp32, indices (T,K) int32, expert_frequency (E) int32, prob_colsum (E) fp32,
    load-balancing loss () fp32) from one pass over x: router GEMM, top-K + softmax over the winners, token counts and
    the column sums of the full softmax, in one kernel, and the loss in the small one that adds up its CTAs' sums.
    Routing is decided on the bf16 logits this returns.  Backward: one kernel turns
    the gradients of logits, scores, prob_colsum and the loss into dlogits; the two router GEMMs stay library calls, as the
    forward one does in the reference (sonicmoe/functional/__init__.py:438-446, sonicmoe/moe.py:251-274)."""

    @staticmethod
    def forward(ctx, x, router_w, K: int):
        x = x.contiguous()
        router_w = router_w.contiguous()
        T, H = x.shape
        E = router_w.shape[0]
        dev = x.device
        st = _lib.device_state(dev)
        with torch.cuda.device(dev):
            logits = torch.empty(T, E, dtype=torch.bfloat16, device=dev)
            scores = torch.empty(T, K, dtype=torch.float32, device=dev)
            indices = torch.empty(T, K, dtype=torch.int32, device=dev)
            freq = torch.empty(E, dtype=torch.int32, device=dev)
            colsum = torch.empty(E, dtype=torch.float32, device=dev)
            aux = torch.empty((), dtype=torch.float32, device=dev)
            aux_grad = torch.empty(E, dtype=torch.float32, device=dev)
            ws = _lib.workspace(lib.smoe_router_forward_workspace_bytes(E), dev)
            check(lib.smoe_router_forward_aux(x.data_ptr(), router_w.data_ptr(), logits.data_ptr(), scores.data_ptr(),
                                              indices.data_ptr(), freq.data_ptr(), colsum.data_ptr(), aux.data_ptr(),
                                              aux_grad.data_ptr(), ws.data_ptr(), T, H, E, K, st.status.data_ptr(),
                                              stream_ptr(dev)), "router_forward")
        ctx.save_for_backward(x, router_w, logits, scores, indices, aux_grad)
        ctx.mark_non_differentiable(indices, freq)
        ctx.set_materialize_grads(False)
        return logits, scores, indices, freq, colsum, aux

    @staticmethod
    def backward(ctx, g_logits, g_scores, _gi, _gf, g_colsum, g_aux):
        x, router_w, logits, scores, indices, aux_grad = ctx.saved_tensors
        if g_logits is None and g_scores is None and g_colsum is None and g_aux is None:
            return None, None, None
        T, E = logits.shape
        K = scores.shape[1]
        dev = x.device
        if g_logits is not None:
            g_logits = g_logits.contiguous().to(torch.bfloat16)
        if g_scores is not None:
            g_scores = g_scores.contiguous().float()
        if g_colsum is not None:
            g_colsum = g_colsum.contiguous().float()
        if g_aux is not None:
            g_aux = g_aux.float()
        with torch.cuda.device(dev):
            dlogits = torch.empty_like(logits)
            check(lib.smoe_router_backward_aux(dlogits.data_ptr(), logits.data_ptr(), ptr(g_scores), scores.data_ptr(),
                                               indices.data_ptr(), ptr(g_colsum), ptr(g_logits), ptr(g_aux),
                                               aux_grad.data_ptr(), T, E, K, stream_ptr(dev)), "router_backward")
        dx = dlogits @ router_w if ctx.needs_input_grad[0] else None
        dw = dlogits.t() @ x if ctx.needs_input_grad[1] else None
        return dx, dw, None


def switch_loss_formula(probs: torch.Tensor, expert_frequency: torch.Tensor) -> torch.Tensor:
    """E <normalised mean of the rows of probs (T,E), normalised expert_frequency>."""
    share = F.normalize(expert_frequency.float(), p=1, dim=0)
    mean_prob = F.normalize(probs.sum(0), p=1, dim=0)
    return probs.size(-1) * (mean_prob * share).sum()


class _SwitchLoss(torch.autograd.Function):
    """The load-balancing loss of bf16 logits (T,E), E <= 256, and token counts that other kernels made.  A backward pass
    that is itself recorded (create_graph) differentiates the loss's formula instead, so that higher derivatives exist."""

    @staticmethod
    def forward(ctx, logits, freq):
        logits_in, logits = logits, logits.contiguous()
        T, E = logits.shape
        dev = logits.device
        with torch.cuda.device(dev):
            aux = torch.empty((), dtype=torch.float32, device=dev)
            aux_grad = torch.empty(E, dtype=torch.float32, device=dev)
            ws = _lib.workspace(lib.smoe_router_forward_workspace_bytes(E), dev)
            check(lib.smoe_switch_loss(logits.data_ptr(), freq.data_ptr(), aux.data_ptr(), aux_grad.data_ptr(),
                                       ws.data_ptr(), T, E, stream_ptr(dev)), "switch_loss")
        ctx.save_for_backward(logits_in, freq, aux_grad)
        return aux

    @staticmethod
    def backward(ctx, g_aux):
        logits, freq, aux_grad = ctx.saved_tensors
        if torch.is_grad_enabled():
            aux = switch_loss_formula(F.softmax(logits, dim=-1, dtype=torch.float32), freq)
            return torch.autograd.grad(aux, logits, g_aux, create_graph=True)[0], None
        logits = logits.contiguous()
        T, E = logits.shape
        dev = logits.device
        g_aux = g_aux.float()
        with torch.cuda.device(dev):
            dlogits = torch.empty_like(logits)
            check(lib.smoe_router_backward_aux(dlogits.data_ptr(), logits.data_ptr(), None, None, None, None, None,
                                               g_aux.data_ptr(), aux_grad.data_ptr(), T, E, 1, stream_ptr(dev)),
                  "router_backward")
        return dlogits, None


def switch_loss(logits: torch.Tensor, expert_frequency: torch.Tensor) -> torch.Tensor | None:
    """`switch_loss_formula` of softmax(logits) by kernels, or None where they do not apply."""
    if not (logits.is_cuda and logits.dtype == torch.bfloat16 and logits.dim() == 2 and logits.shape[1] <= 256
            and expert_frequency.dtype == torch.int32 and expert_frequency.device == logits.device
            and expert_frequency.is_contiguous() and not torch.compiler.is_compiling()):
        return None
    return _SwitchLoss.apply(logits, expert_frequency)


# ------------------------------------------------------------------------------------------------
# routed experts
# ------------------------------------------------------------------------------------------------
def _expert_major(w: torch.Tensor) -> torch.Tensor:
    """(out, in, E) view as passed by MoE.forward -> contiguous (E, out, in) storage (no copy if it is one)."""
    return w.permute(2, 0, 1).contiguous()


_ACT_CODE = {ActivationType.SWIGLU: 0, ActivationType.GEGLU: 1, ActivationType.REGLU: 2, ActivationType.RELU_SQ: 3,
             ActivationType.RELU: 4, ActivationType.GELU: 5, ActivationType.SILU: 6}


def _check_experts_args(x, w1, w2, b1, b2, activation_type, expert_major=False):
    """w1 (N1,H,E) and w2 (H,I,E), or (E,N1,H) and (E,H,I)."""
    if (b1 is None) != (b2 is None):
        raise AssertionError("b1 and b2 has to be None or not None at the same time!")
    if isinstance(activation_type, str):
        activation_type = ActivationType(activation_type)
    if activation_type not in _ACT_CODE:
        raise ValueError(f"unknown activation {activation_type}")
    _lib.require_cuda(x, "x")
    if x.dtype != torch.bfloat16 or w1.dtype != torch.bfloat16 or w2.dtype != torch.bfloat16:
        raise TypeError("the sm_100a kernels take bf16 activations and weights "
                        f"(got x {x.dtype}, w1 {w1.dtype}, w2 {w2.dtype})")
    H = x.shape[1]
    if expert_major:
        (e1, n1, h1), (e2, h2, I) = w1.shape, w2.shape
    else:
        (n1, h1, e1), (h2, I, e2) = w1.shape, w2.shape
    if h1 != H or h2 != H or I * (2 if is_glu(activation_type) else 1) != n1 or e1 != e2:
        raise ValueError(f"inconsistent shapes: x {tuple(x.shape)}, w1 {tuple(w1.shape)}, w2 {tuple(w2.shape)}")
    if H % 64 != 0 or I % 64 != 0:
        raise ValueError("hidden size and intermediate size must be multiples of 64")
    if (b1 is not None or activation_type != ActivationType.SWIGLU) and n1 % 128 != 0:
        raise ValueError("with a bias or a non-SwiGLU activation the up projection needs a multiple of 128 output rows")
    if b1 is not None and (b1.dtype != x.dtype or b2.dtype != x.dtype):
        raise TypeError("biases must have the activations' dtype")
    if b1 is not None and (b1.numel() < e1 * n1 or b2.numel() < e1 * H):  # the kernels read that many
        raise ValueError(f"inconsistent shapes: w1 {tuple(w1.shape)}, w2 {tuple(w2.shape)}, b1 {tuple(b1.shape)}, "
                         f"b2 {tuple(b2.shape)}")
    return activation_type


def _check_router_args(x, router_w, w1, expert_major=False):
    """The kernels take the number of experts from the router and read that many experts' weights."""
    if router_w.shape != (w1.shape[0 if expert_major else 2], x.shape[1]):
        raise ValueError(f"inconsistent shapes: x {tuple(x.shape)}, router {tuple(router_w.shape)}, w1 {tuple(w1.shape)}")


def _experts(x, w1, b1, w2, b2, scores_flat, route, T, inference, activation_type):
    """Routed experts: the tuned bias-free SwiGLU kernels, or the general ones for a bias / another activation."""
    if b1 is None and activation_type == ActivationType.SWIGLU:
        return _RoutedExperts.apply(x, w1, w2, scores_flat, route, T, inference)
    return _RoutedExpertsGeneral.apply(x, w1, b1, w2, b2, scores_flat, route, T, inference,
                                       _ACT_CODE[activation_type])


class _RoutedExperts(torch.autograd.Function):
    """o[t] = sum over the pairs (t, e) routed to token t of score * W2[e] swiglu(W1[e] x[t]).

    Forward: gather-fused up projection with the SwiGLU epilogue (z, y1), down projection, combine.
    Backward: dH GEMM with the fused dSwiGLU / ds / y1*s epilogue, the two weight-gradient GEMMs over the
    ragged token dimension, the dX GEMM and its reduction over each token's rows.
    Reference: _UpProjection + _DownProjection (sonicmoe/functional/__init__.py:114-420).
    """

    @staticmethod
    def forward(ctx, x, w1, w2, scores_flat, route: Route, T: int, inference: bool):
        dev = x.device
        x = x.contiguous()
        w1e = _expert_major(w1)  # (E, 2I, H)
        w2e = _expert_major(w2)  # (E, H, I)
        E, two_i, H = w1e.shape
        I = two_i // 2
        TK = route.x_gather_idx.numel()
        scores_flat = scores_flat.contiguous()
        st = _lib.device_state(dev)
        need_grad = not inference
        with torch.cuda.device(dev):
            stream = stream_ptr(dev)
            z = torch.empty(TK, two_i, dtype=x.dtype, device=dev) if need_grad else None
            y1 = torch.empty(TK, I, dtype=x.dtype, device=dev)
            check(lib.smoe_up_projection_forward(
                x.data_ptr(), w1e.data_ptr(), ptr(z), y1.data_ptr(), route.expert_frequency_offset.data_ptr(),
                route.x_gather_idx.data_ptr(), T, H, I, E, TK, st.status.data_ptr(), stream), "up_projection_forward")
            o = torch.empty(T, H, dtype=x.dtype, device=dev)
            if _one_row_per_token(route, T):
                check(lib.smoe_down_projection_forward_rows(
                    y1.data_ptr(), w2e.data_ptr(), o.data_ptr(), scores_flat.data_ptr(),
                    int(scores_flat.dtype == torch.bfloat16), route.expert_frequency_offset.data_ptr(),
                    route.x_gather_idx.data_ptr(), route.s_scatter_idx.data_ptr(), H, I, E, TK,
                    st.status.data_ptr(), stream), "down_projection_forward_rows")
            elif _FUSED_COMBINE:
                o_acc = torch.zeros(T, H, dtype=torch.float32, device=dev)
                check(lib.smoe_down_projection_forward_scatter(
                    y1.data_ptr(), w2e.data_ptr(), o_acc.data_ptr(), scores_flat.data_ptr(),
                    int(scores_flat.dtype == torch.bfloat16), route.expert_frequency_offset.data_ptr(),
                    route.x_gather_idx.data_ptr(), route.s_scatter_idx.data_ptr(), T, H, I, E, TK,
                    st.status.data_ptr(), stream), "down_projection_forward_scatter")
                check(lib.smoe_cast_f32_to_bf16(o_acc.data_ptr(), o.data_ptr(), T * H, stream), "cast")
            else:
                y2 = torch.empty(TK, H, dtype=x.dtype, device=dev)
                check(lib.smoe_down_projection_forward(
                    y1.data_ptr(), w2e.data_ptr(), y2.data_ptr(), route.expert_frequency_offset.data_ptr(),
                    H, I, E, TK, st.status.data_ptr(), stream), "down_projection_forward")
                check(lib.smoe_gather_sum(
                    y2.data_ptr(), o.data_ptr(), scores_flat.data_ptr(), _lib.dtype_code(scores_flat.dtype),
                    route.s_reverse_scatter_idx.data_ptr(), ptr(route.token_offset), T, H, max(route.K, 1), stream),
                    "gather_sum")
        if need_grad:
            ctx.save_for_backward(x, w1e, w2e, z, scores_flat)
            ctx.route = route
            ctx.dims = (T, H, I, E, TK)
            ctx.w_shapes = (w1.shape, w2.shape)
        return o

    @staticmethod
    def backward(ctx, dout):
        x, w1e, w2e, z, scores_flat = ctx.saved_tensors
        route: Route = ctx.route
        T, H, I, E, TK = ctx.dims
        dev = x.device
        dout = dout.contiguous()
        if dout.dtype != x.dtype:
            dout = dout.to(x.dtype)
        st = _lib.device_state(dev)
        off = route.expert_frequency_offset.data_ptr()
        gat = route.x_gather_idx.data_ptr()
        with torch.cuda.device(dev):
            stream = stream_ptr(dev)
            dz = torch.empty(TK, 2 * I, dtype=x.dtype, device=dev)
            y1s = torch.empty(TK, I, dtype=x.dtype, device=dev)
            ncols = lib.smoe_ds_partial_columns(I)
            ds_partial = torch.empty(ncols, TK, dtype=torch.float32, device=dev)
            check(lib.smoe_down_projection_backward_act(
                dout.data_ptr(), w2e.data_ptr(), z.data_ptr(), scores_flat.data_ptr(),
                int(scores_flat.dtype == torch.bfloat16), dz.data_ptr(), y1s.data_ptr(), ds_partial.data_ptr(),
                off, gat, route.s_scatter_idx.data_ptr(), T, H, I, E, TK, st.status.data_ptr(), stream),
                "down_projection_backward_act")
            ds = torch.empty_like(scores_flat)
            check(lib.smoe_ds_reduce(ds_partial.data_ptr(), route.s_scatter_idx.data_ptr(), ds.data_ptr(),
                                     _lib.dtype_code(ds.dtype), TK, ncols, stream), "ds_reduce")
            # dX first: nothing else depends on the weight gradients, and a caller that has to send dx somewhere
            # (expert parallelism) can do so while the two weight-gradient GEMMs run
            dx = torch.empty(T, H, dtype=x.dtype, device=dev)
            if _one_row_per_token(route, T):
                check(lib.smoe_up_projection_backward_dx_rows(
                    dz.data_ptr(), w1e.data_ptr(), dx.data_ptr(), off, gat, H, I, E, TK, st.status.data_ptr(), stream),
                    "up_projection_backward_dx_rows")
            else:
                dx_expanded = torch.empty(TK, H, dtype=x.dtype, device=dev)
                check(lib.smoe_up_projection_backward_dx(
                    dz.data_ptr(), w1e.data_ptr(), dx_expanded.data_ptr(), off, H, I, E, TK, st.status.data_ptr(),
                    stream), "up_projection_backward_dx")
                check(lib.smoe_gather_sum(
                    dx_expanded.data_ptr(), dx.data_ptr(), None, _lib.SMOE_F32,
                    route.s_reverse_scatter_idx.data_ptr(), ptr(route.token_offset), T, H, max(route.K, 1), stream),
                    "gather_sum")
                del dx_expanded
            if route.on_dx is not None:
                route.on_dx(dx)
            shared = route.wgrad_sum
            if shared is None:
                dw1, dw2, add = torch.empty_like(w1e), torch.empty_like(w2e), False
            else:
                dw1, dw2, add = shared.buffers(w1e, w2e)
            down = lib.smoe_down_projection_weight_grad_accumulate if add else lib.smoe_down_projection_weight_grad
            check(down(dout.data_ptr(), y1s.data_ptr(), dw2.data_ptr(), off, gat, T, H, I, E, TK,
                       st.status.data_ptr(), stream), "down_projection_weight_grad")
            del y1s, ds_partial
            up = lib.smoe_up_projection_weight_grad_accumulate if add else lib.smoe_up_projection_weight_grad
            check(up(x.data_ptr(), dz.data_ptr(), dw1.data_ptr(), off, gat, T, H, I, E, TK, st.status.data_ptr(),
                     stream), "up_projection_weight_grad")
            if shared is not None:
                dw1, dw2 = shared.finish_chunk()
                if dw1 is None:
                    return dx, None, None, ds, None, None, None
        # gradients in the layout of the (out, in, E) views the caller passed
        return dx, dw1.permute(1, 2, 0), dw2.permute(1, 2, 0), ds, None, None, None


class _RoutedExpertsGeneral(torch.autograd.Function):
    """`_RoutedExperts` with optional expert biases and any activation of ``ActivationType``.

    o[t] = sum score * (W2[e] act(W1[e] x[t] + b1[e]) + b2[e]).  Gradients also for b1, b2; the score gradient
    gains the term <dout[t], b2[e]>.  Reference: sonicmoe/functional/__init__.py:114-420 with b1/b2 and
    activation_type, bias kernels sonicmoe/functional/backward.py:36-168.
    """

    @staticmethod
    def forward(ctx, x, w1, b1, w2, b2, scores_flat, route: Route, T: int, inference: bool, act: int):
        dev = x.device
        x = x.contiguous()
        w1e = _expert_major(w1)  # (E, N1, H)
        w2e = _expert_major(w2)  # (E, H, I)
        E, n1, H = w1e.shape
        I = w2e.shape[2]
        TK = route.x_gather_idx.numel()
        scores_flat = scores_flat.contiguous()
        b1c = None if b1 is None else b1.contiguous()
        b2c = None if b2 is None else b2.contiguous()
        st = _lib.device_state(dev)
        off = route.expert_frequency_offset.data_ptr()
        with torch.cuda.device(dev):
            stream = stream_ptr(dev)
            z = torch.empty(TK, n1, dtype=x.dtype, device=dev) if not inference else None
            y1 = torch.empty(TK, I, dtype=x.dtype, device=dev)
            check(lib.smoe_up_projection_forward_act(
                x.data_ptr(), w1e.data_ptr(), ptr(b1c), ptr(z), y1.data_ptr(), off, route.x_gather_idx.data_ptr(),
                T, H, n1, E, TK, act, st.status.data_ptr(), stream), "up_projection_forward_act")
            y2 = torch.empty(TK, H, dtype=x.dtype, device=dev)
            check(lib.smoe_down_projection_forward_bias(
                y1.data_ptr(), w2e.data_ptr(), ptr(b2c), y2.data_ptr(), off, H, I, E, TK, st.status.data_ptr(),
                stream), "down_projection_forward_bias")
            o = torch.empty(T, H, dtype=x.dtype, device=dev)
            check(lib.smoe_gather_sum(
                y2.data_ptr(), o.data_ptr(), scores_flat.data_ptr(), _lib.dtype_code(scores_flat.dtype),
                route.s_reverse_scatter_idx.data_ptr(), ptr(route.token_offset), T, H, max(route.K, 1), stream),
                "gather_sum")
        if not inference:
            ctx.save_for_backward(x, w1e, w2e, z, scores_flat, b2c)
            ctx.route = route
            ctx.dims = (T, H, I, E, TK, n1)
            ctx.act = act
            ctx.has_bias = b1 is not None
        return o

    @staticmethod
    def backward(ctx, dout):
        x, w1e, w2e, z, scores_flat, b2c = ctx.saved_tensors
        route: Route = ctx.route
        T, H, I, E, TK, n1 = ctx.dims
        dev = x.device
        dout = dout.contiguous().to(x.dtype)
        st = _lib.device_state(dev)
        off = route.expert_frequency_offset.data_ptr()
        gat = route.x_gather_idx.data_ptr()
        sct = route.s_scatter_idx.data_ptr()
        sc_bf16 = int(scores_flat.dtype == torch.bfloat16)
        with torch.cuda.device(dev):
            stream = stream_ptr(dev)
            dz = torch.empty(TK, n1, dtype=x.dtype, device=dev)
            y1s = torch.empty(TK, I, dtype=x.dtype, device=dev)
            ncols = lib.smoe_ds_partial_columns(I)
            ds_partial = torch.empty(ncols, TK, dtype=torch.float32, device=dev)
            check(lib.smoe_down_projection_backward_dact(
                dout.data_ptr(), w2e.data_ptr(), z.data_ptr(), scores_flat.data_ptr(), sc_bf16, dz.data_ptr(),
                y1s.data_ptr(), ds_partial.data_ptr(), off, gat, sct, T, H, I, E, TK, ctx.act, st.status.data_ptr(),
                stream), "down_projection_backward_dact")
            ds = torch.empty_like(scores_flat)
            check(lib.smoe_ds_reduce(ds_partial.data_ptr(), sct, ds.data_ptr(), _lib.dtype_code(ds.dtype), TK, ncols,
                                     stream), "ds_reduce")
            db1 = db2 = None
            if ctx.has_bias:
                check(lib.smoe_ds_add_bias_term(dout.data_ptr(), b2c.data_ptr(), off, gat, sct, ds.data_ptr(),
                                                _lib.dtype_code(ds.dtype), E, H, TK, stream), "ds_add_bias_term")
                db2 = torch.empty(E, H, dtype=x.dtype, device=dev)
                check(lib.smoe_expert_column_sum(dout.data_ptr(), H, gat, scores_flat.data_ptr(),
                                                 _lib.dtype_code(scores_flat.dtype), sct, off, db2.data_ptr(), E, H,
                                                 stream), "expert_column_sum")
                db1 = torch.empty(E, n1, dtype=x.dtype, device=dev)
                check(lib.smoe_expert_column_sum(dz.data_ptr(), n1, None, None, 0, None, off, db1.data_ptr(), E, n1,
                                                 stream), "expert_column_sum")
            dw2 = torch.empty_like(w2e)
            check(lib.smoe_down_projection_weight_grad(
                dout.data_ptr(), y1s.data_ptr(), dw2.data_ptr(), off, gat, T, H, I, E, TK, st.status.data_ptr(),
                stream), "down_projection_weight_grad")
            # the two kernels below take the up projection's output rows as 2 * (their I argument)
            half = n1 // 2
            dw1 = torch.empty_like(w1e)
            check(lib.smoe_up_projection_weight_grad(
                x.data_ptr(), dz.data_ptr(), dw1.data_ptr(), off, gat, T, H, half, E, TK, st.status.data_ptr(),
                stream), "up_projection_weight_grad")
            dx_expanded = torch.empty(TK, H, dtype=x.dtype, device=dev)
            check(lib.smoe_up_projection_backward_dx(
                dz.data_ptr(), w1e.data_ptr(), dx_expanded.data_ptr(), off, H, half, E, TK, st.status.data_ptr(),
                stream), "up_projection_backward_dx")
            dx = torch.empty(T, H, dtype=x.dtype, device=dev)
            check(lib.smoe_gather_sum(
                dx_expanded.data_ptr(), dx.data_ptr(), None, _lib.SMOE_F32, route.s_reverse_scatter_idx.data_ptr(),
                ptr(route.token_offset), T, H, max(route.K, 1), stream), "gather_sum")
        return dx, dw1.permute(1, 2, 0), db1, dw2.permute(1, 2, 0), db2, ds, None, None, None, None


def moe_TC_softmax_topk_layer(
    x: torch.Tensor,
    router_w: torch.Tensor,
    w1: torch.Tensor,
    b1: torch.Tensor | None,
    w2: torch.Tensor,
    b2: torch.Tensor | None,
    K: int,
    stream_id: int = 0,
    activation_type: ActivationType | str = ActivationType.SWIGLU,
    is_inference_mode_enabled: bool = False,
) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """Token-choice top-K MoE layer: returns (o (T,H), router_logits (T,E), expert_frequency (E,) int32).

    x (T,H) bf16; router_w (E,H); w1 (2I,H,E) and w2 (H,I,E) are the ``permute(1,2,0)`` views of the
    (E,2I,H) / (E,H,I) parameters, gate/up rows of w1 interleaved.
    Reference: sonicmoe/functional/__init__.py:423-490.
    """
    o, router_logits, freq, _ = moe_TC_softmax_topk_layer_with_router_stats(
        x, router_w, w1, b1, w2, b2, K, stream_id, activation_type, is_inference_mode_enabled)
    return o, router_logits, freq


def moe_TC_softmax_topk_layer_with_router_stats(x, router_w, w1, b1, w2, b2, K, stream_id=0,
                                                activation_type=ActivationType.SWIGLU,
                                                is_inference_mode_enabled=False):
    """`moe_TC_softmax_topk_layer` plus a fourth result: the column sums (E,) fp32 of softmax(router_logits) when the
    fused routing kernel produced them (what the load-balancing loss needs), else None."""
    _check_router_args(x, router_w, w1)
    return _layer_with_aux(x, router_w, w1.permute(2, 0, 1), b1, w2.permute(2, 0, 1), b2, K, activation_type,
                           is_inference_mode_enabled)[:4]


def _layer_forward(x, router_w, w1, w2, K):
    """The results of `_layer_with_aux` for a bias-free SwiGLU layer with the fused router where no gradient is wanted:
    one call of the library, one piece of scratch."""
    dev = x.device
    T, H = x.shape
    E, _, I = w2.shape
    x, router_w, w1, w2 = x.contiguous(), router_w.contiguous(), w1.contiguous(), w2.contiguous()
    with _lib.on_device(dev):
        o = torch.empty_like(x)
        logits = torch.empty(T, E, dtype=torch.bfloat16, device=dev)
        freq = torch.empty(E, dtype=torch.int32, device=dev)
        colsum = torch.empty(E, dtype=torch.float32, device=dev)
        aux = torch.empty((), dtype=torch.float32, device=dev)
        scratch = _lib.workspace(lib.smoe_layer_forward_scratch_bytes(T, H, I, E, K), dev)
        check(lib.smoe_layer_forward(
            x.data_ptr(), router_w.data_ptr(), w1.data_ptr(), w2.data_ptr(), o.data_ptr(), logits.data_ptr(),
            freq.data_ptr(), colsum.data_ptr(), aux.data_ptr(), scratch.data_ptr(), T, H, I, E, K,
            _lib.device_state(dev).status.data_ptr(), stream_ptr(dev)), "layer_forward")
    return o, logits, freq, colsum, aux


class _Layer(torch.autograd.Function):
    """The whole layer as one node: router (or the top-K of given logits), routing metadata and routed experts, with four
    calls of the library in a training step where the separate functions make 17 in four nodes.

    Either router_w (the fused router) or logits_in (T,E) is given; training: a backward pass may follow.  Results: o (T,H), expert_frequency (E,) int32, and with
    router_w the logits, the column sums of their softmax and the load-balancing loss (else None).  The router's part of the
    gradient of x comes from a library GEMM, the experts' part is added to it by the kernel that adds up each token's rows.
    Same kernels, results and saved activations as `_FusedRouter` / `topk_softmax` and `_RoutedExperts(General)`."""

    @staticmethod
    def forward(ctx, x, router_w, logits_in, w1, b1, w2, b2, K: int, act: int, training: bool):
        dev = x.device
        x, w1, w2 = x.contiguous(), w1.contiguous(), w2.contiguous()
        b1 = None if b1 is None else b1.contiguous()
        b2 = None if b2 is None else b2.contiguous()
        T, H = x.shape
        E, n1, _ = w1.shape
        I = w2.shape[2]
        with _lib.on_device(dev):
            if router_w is not None:
                router_w = router_w.contiguous()
                logits = torch.empty(T, E, dtype=torch.bfloat16, device=dev)
                colsum = torch.empty(E, dtype=torch.float32, device=dev)
                aux = torch.empty((), dtype=torch.float32, device=dev)
            else:
                logits = logits_in.contiguous()
                colsum = aux = None
            o = torch.empty_like(x)
            z = torch.empty(T * K, n1, dtype=x.dtype, device=dev) if training else None
            freq = torch.empty(E, dtype=torch.int32, device=dev)
            meta = torch.empty(lib.smoe_layer_meta_words(T, E, K), dtype=torch.int32, device=dev)
            scratch_bytes = (lib.smoe_layer_train_forward_plain_scratch_bytes if b1 is None and act == 0
                             else lib.smoe_layer_train_forward_scratch_bytes)
            scratch = _lib.workspace(scratch_bytes(T, H, I, E, K), dev)
            check(lib.smoe_layer_train_forward(
                x.data_ptr(), ptr(router_w), logits.data_ptr(), _lib.dtype_code(logits.dtype), w1.data_ptr(), ptr(b1),
                w2.data_ptr(), ptr(b2), o.data_ptr(), ptr(z), meta.data_ptr(), freq.data_ptr(), ptr(colsum), ptr(aux),
                scratch.data_ptr(), T, H, I, n1, E, K, act, _lib.device_state(dev).status.data_ptr(), stream_ptr(dev)),
                "layer_train_forward")
        if training:
            fused = router_w is not None
            ctx.save_for_backward(x, w1, w2, b2, z, meta, router_w, logits if fused else None)
            ctx.layer = (T, H, I, n1, E, K, act, fused, logits.dtype)
            ctx.mark_non_differentiable(freq)
            ctx.set_materialize_grads(False)
        return o, freq, (logits if router_w is not None else None), colsum, aux

    @staticmethod
    def backward(ctx, dout, _freq, g_logits, g_colsum, g_aux):
        x, w1, w2, b2, z, meta, router_w, logits = ctx.saved_tensors
        T, H, I, n1, E, K, act, fused, logits_dtype = ctx.layer
        need_x, need_router, need_logits, need_w1, _, need_w2 = ctx.needs_input_grad[:6]
        if dout is None and (not fused or (g_logits is None and g_colsum is None and g_aux is None)):
            return (None,) * 10
        dev = x.device
        if dout is not None:
            dout = dout.contiguous().to(x.dtype)
        if g_logits is not None:
            g_logits = g_logits.contiguous().to(torch.bfloat16)
        if g_colsum is not None:
            g_colsum = g_colsum.contiguous().float()
        if g_aux is not None:
            g_aux = g_aux.float()
        dx = dw1 = dw2 = db1 = db2 = dlogits = d_router = None
        with _lib.on_device(dev):
            stream = stream_ptr(dev)
            status = _lib.device_state(dev).status.data_ptr()
            scratch = None
            if dout is not None:
                scratch = _lib.workspace(lib.smoe_layer_backward_scratch_bytes(T, I, n1, K), dev)
                if b2 is not None:
                    db1 = torch.empty(E, n1, dtype=x.dtype, device=dev)
                    db2 = torch.empty(E, H, dtype=x.dtype, device=dev)
            if need_logits or (fused and (need_x or need_router)):
                dlogits = torch.empty(T, E, dtype=logits_dtype, device=dev)
            check(lib.smoe_layer_backward_act(
                ptr(dout), w2.data_ptr(), ptr(b2), z.data_ptr(), meta.data_ptr(), ptr(logits),
                _lib.dtype_code(logits_dtype), fused, ptr(g_logits), ptr(g_colsum), ptr(g_aux), ptr(dlogits), ptr(db1),
                ptr(db2), ptr(scratch), T, H, I, n1, E, K, act, status, stream), "layer_backward_act")
            if fused:
                if need_x:
                    dx = (dlogits @ router_w).to(x.dtype)  # autocast may choose another type, and the experts' part is added below
                if need_router:
                    d_router = dlogits.t() @ x
            if dout is not None:
                # dX before the weight gradients, so that its rows are given back before those are allocated
                if need_x:
                    add = dx is not None
                    if not add:
                        dx = torch.empty(T, H, dtype=x.dtype, device=dev)
                    rows = torch.empty(T * K, H, dtype=x.dtype, device=dev) if K > 1 else None
                    check(lib.smoe_layer_backward_dx(w1.data_ptr(), meta.data_ptr(), scratch.data_ptr(), ptr(rows),
                                                     dx.data_ptr(), add, T, H, I, n1, E, K, status, stream),
                          "layer_backward_dx")
                    del rows
                if need_w1 or need_w2:
                    dw1, dw2 = torch.empty_like(w1), torch.empty_like(w2)
                    check(lib.smoe_layer_backward_weights(
                        x.data_ptr(), dout.data_ptr(), meta.data_ptr(), scratch.data_ptr(), dw1.data_ptr(),
                        dw2.data_ptr(), T, H, I, n1, E, K, status, stream), "layer_backward_weights")
        return dx, d_router, (None if fused else dlogits), dw1, db1, dw2, db2, None, None, None


def _layer_with_aux(x, router_w, w1, b1, w2, b2, K, activation_type, is_inference_mode_enabled):
    """(o, router_logits, expert_frequency, column sums of softmax(router_logits), load-balancing loss) with w1 (E,N1,H) and
    w2 (E,H,I); the last two are None where the fused routing kernel does not apply."""
    _check_router_args(x, router_w, w1, expert_major=True)
    activation_type = _check_experts_args(x, w1, w2, b1, b2, activation_type, expert_major=True)
    E = router_w.size(0)
    T = x.size(0)
    grad = torch.is_grad_enabled()
    inference = is_inference_mode_enabled or not grad
    fused = fused_router_applies(x, router_w, K)
    plain = b1 is None and activation_type == ActivationType.SWIGLU
    one_call = (T > 0 and not _FUSED_COMBINE and not torch.compiler.is_compiling() and not torch.jit.is_tracing()
                and forward_ad._current_level < 0)
    recorded = grad and any(t is not None and t.requires_grad for t in (x, router_w, w1, b1, w2, b2))
    if fused and plain and one_call and not recorded:
        return _layer_forward(x, router_w, w1, w2, K)
    if one_call and not (inference and recorded):
        act = _ACT_CODE[activation_type]
        if fused:
            o, freq, router_logits, colsum, aux = _Layer.apply(x, router_w, None, w1, b1, w2, b2, K, act, recorded)
            return o, router_logits, freq, colsum, aux
        router_logits = F.linear(x if x.dtype == router_w.dtype else x.to(router_w.dtype), router_w)
        if router_logits.dtype in (torch.float32, torch.bfloat16):
            o, freq, _, _, _ = _Layer.apply(x, None, router_logits, w1, b1, w2, b2, K, act, recorded)
            return o, router_logits, freq, None, None
    if fused:
        router_logits, scores, indices, _freq, colsum, aux = _FusedRouter.apply(x, router_w, K)
    else:
        colsum = aux = None
        # a router kept in fp32 (an extension over the reference) computes its logits in fp32
        router_logits = F.linear(x if x.dtype == router_w.dtype else x.to(router_w.dtype), router_w)
        if torch.compiler.is_compiling() and plain:
            # opaque custom ops instead of autograd functions with ctypes calls inside (torch.compile, fullgraph)
            from .compiled_ops import layer_with_custom_ops

            o, freq = layer_with_custom_ops(x, router_logits, w1.permute(1, 2, 0), w2.permute(1, 2, 0), K, E, inference)
            return o, router_logits, freq, None, None
        scores, indices = topk_softmax(router_logits, K)
    route = _route_metadata(indices.reshape(-1), None, E, K)
    o = _experts(x, w1.permute(1, 2, 0), b1, w2.permute(1, 2, 0), b2, scores.reshape(-1), route, T, inference,
                 activation_type)
    return o, router_logits, route.expert_frequency, colsum, aux


def moe_general_routing_inputs(
    x: torch.Tensor,
    router_scores: torch.Tensor,
    token_indices: torch.Tensor,
    expert_indices: torch.Tensor,
    w1: torch.Tensor,
    b1: torch.Tensor | None,
    w2: torch.Tensor,
    b2: torch.Tensor | None,
    E: int,
    stream_id: int = 0,
    activation_type: ActivationType | str = ActivationType.SWIGLU,
    is_inference_mode_enabled: bool = False,
) -> tuple[torch.Tensor, torch.Tensor]:
    """Routed experts for an arbitrary list of (score, token, expert) pairs; ``token_indices`` ascending.

    Returns (o (T,H), expert_frequency (E,) int32).  Gradients flow to x, w1, w2 and router_scores.
    Reference: sonicmoe/functional/__init__.py:497-562.
    """
    activation_type = _check_experts_args(x, w1, w2, b1, b2, activation_type)
    T = x.size(0)
    E = w2.size(-1)
    tok = token_indices.contiguous().to(torch.int32)
    route = _route_metadata(expert_indices, tok, E, 0)
    route.token_offset = _sorted_offsets(tok, T)
    inference = is_inference_mode_enabled or not torch.is_grad_enabled()
    o = _experts(x, w1, b1, w2, b2, router_scores, route, T, inference, activation_type)
    return o, route.expert_frequency
