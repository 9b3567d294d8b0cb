"""Host-side logic that needs no GPU: module surface, state-dict layout, eager backend vs oracle, errors."""

import os
import re

import numpy as np
import pytest
import torch

from conftest import ROOT
from oracle import moe_oracle as orc


def _module(E=8, K=2, H=128, I=64, seed=0):
    import sonicmoe
    from sonicmoe.enums import ActivationType

    inp = orc.make_inputs(96, H, I, E, K, seed=seed)
    m = sonicmoe.MoE(E, K, H, I, ActivationType.SWIGLU, False, 0.02)
    with torch.no_grad():
        m.router.weight.copy_(inp["router_w"])
        m.c_fc.weight.copy_(inp["w1"])
        m.c_proj.weight.copy_(inp["w2"])
    return m, inp


def test_public_surface(built_library):
    import sonicmoe
    from sonicmoe import KernelBackendMoE, MoE, count_cumsum, enable_quack_gemm, moe_TC_softmax_topk_layer  # noqa: F401
    from sonicmoe.enums import ActivationType, is_glu
    from sonicmoe.functional import count_cumsum as cc2, moe_general_routing_inputs  # noqa: F401

    assert KernelBackendMoE("sonicmoe") is KernelBackendMoE.sonicmoe
    assert ActivationType("swiglu") is ActivationType.SWIGLU
    assert is_glu(ActivationType.GEGLU) and not is_glu(ActivationType.RELU_SQ)
    with enable_quack_gemm(True):
        pass


def test_state_dict_layout(built_library):
    m, _ = _module()
    sd = m.state_dict()
    assert set(sd) == {"router.weight", "c_fc.weight", "c_proj.weight"}
    assert sd["router.weight"].shape == (8, 128)
    assert sd["c_fc.weight"].shape == (8, 128, 128)   # (E, 2I, H)
    assert sd["c_proj.weight"].shape == (8, 128, 64)  # (E, H, I)
    import sonicmoe
    from sonicmoe.enums import ActivationType

    mb = sonicmoe.MoE(4, 2, 64, 64, ActivationType.GELU, True, 0.02)
    assert mb.c_fc.weight.shape == (4, 64, 64) and mb.c_fc.bias.shape == (4, 64) and mb.c_proj.bias.shape == (4, 64)


def test_eager_backend_matches_oracle(built_library):
    from sonicmoe import KernelBackendMoE

    m, inp = _module()
    x = inp["x"].clone().requires_grad_(True)
    o, aux = m(x.view(2, 48, 128), kernel_backend_moe=KernelBackendMoE.torch)
    assert o.shape == (2, 48, 128)
    grads = torch.autograd.grad(o, [x, m.router.weight, m.c_fc.weight, m.c_proj.weight], inp["dout"].view(2, 48, 128))
    ref = orc.moe_layer(inp["x"], inp["router_w"], inp["w1"], inp["w2"], 2, dout=inp["dout"])
    for got, want in zip((o.reshape(96, 128), aux, *grads),
                         (ref["o"], ref["aux_loss"], ref["dx"], ref["drouter_w"], ref["dw1"], ref["dw2"])):
        assert (got.detach() - want).norm() <= 2e-5 * want.norm()


def test_cuda_backend_refuses_cpu_and_unsupported_inputs(built_library):
    from sonicmoe import _lib
    from sonicmoe.functional import moe_TC_softmax_topk_layer

    m, inp = _module()
    with pytest.raises(_lib.SonicMoEError):
        m(inp["x"])  # CPU tensor: no fallback
    w1 = m.c_fc.weight.permute(1, 2, 0)
    w2 = m.c_proj.weight.permute(1, 2, 0)
    with pytest.raises(AssertionError):
        moe_TC_softmax_topk_layer(inp["x"], m.router.weight, w1, torch.zeros(8, 128), w2, None, 2)
    with pytest.raises(ValueError):
        moe_TC_softmax_topk_layer(inp["x"], m.router.weight, w1, None, w2, None, 2, 0, "not-an-activation")
    with pytest.raises(_lib.SonicMoEError):  # a supported activation still has no CPU path
        moe_TC_softmax_topk_layer(inp["x"], m.router.weight, w1, None, w2, None, 2, 0, "gelu")
    with pytest.raises(ValueError):
        m(inp["x"], kernel_backend_moe=__import__("sonicmoe").KernelBackendMoE.scattermoe)


def test_rounded_counts():
    from sonicmoe.functional.token_rounding import rounded_counts

    f = torch.tensor([0, 1, 63, 64, 65, 127, 128, 191, 192, 193, 320, 448])
    assert rounded_counts(f, "down").tolist() == [0, 0, 0, 0, 0, 0, 128, 128, 128, 128, 256, 384]
    assert rounded_counts(f, "up").tolist() == [0, 128, 128, 128, 128, 128, 128, 256, 256, 256, 384, 512]
    # nearest, exact halves go to the even multiple (64 -> 0, 192 -> 256, 320 -> 256, 448 -> 512)
    assert rounded_counts(f, "nr").tolist() == [0, 0, 0, 0, 128, 128, 128, 128, 256, 256, 256, 512]
    assert torch.equal(rounded_counts(f, "nr"), orc.rounded_counts(f, "nr"))


def test_token_rounding_router_has_no_cpu_path():
    """The selection runs in the library's CUDA kernels only: CPU tensors are refused, unknown modes too."""
    from sonicmoe import _lib
    from sonicmoe.functional.token_rounding import forward_token_choice_rounding, select_pairs

    inp = orc.make_inputs(512, 64, 64, 8, 2, seed=11, dtype=torch.float32)
    with pytest.raises(_lib.SonicMoEError):
        forward_token_choice_rounding(inp["x"], inp["router_w"], 8, 2, 128, "nr")
    with pytest.raises(NotImplementedError):
        select_pairs(torch.zeros(4, 8), torch.zeros(4, 2, dtype=torch.int32), "sideways")


@pytest.mark.parametrize("name", ["state_dict_swiglu", "state_dict_gelu_bias"])
def test_reference_state_dict_loads_and_reproduces_reference_output(built_library, name):
    """Checkpoint interchange: the state dict of a module the reference constructed and initialised loads with
    strict=True into this build's `MoE`, and the eager backend then reproduces the reference's output, aux loss and
    every gradient (fixtures: tests/golden/make_golden.py, reference sonicmoe/moe.py:58-68, 186-204)."""
    import sonicmoe
    from conftest import golden
    from sonicmoe import KernelBackendMoE
    from sonicmoe.enums import ActivationType

    g = golden(name)
    T, H, I, E, K, _seed, add_bias = [int(v) for v in g["meta"]]
    state = {k[len("param."):]: torch.from_numpy(g[k]) for k in g.files if k.startswith("param.")}
    m = sonicmoe.MoE(E, K, H, I, ActivationType(str(g["activation"])), bool(add_bias), 0.02)
    missing = m.load_state_dict(state, strict=True)
    assert not missing.missing_keys and not missing.unexpected_keys
    x = torch.from_numpy(g["x"]).requires_grad_(True)
    o, aux = m(x, kernel_backend_moe=KernelBackendMoE.torch)
    names = [n for n, _ in m.named_parameters()]
    grads = torch.autograd.grad(o, [x] + list(m.parameters()), torch.from_numpy(g["dout"]))

    def close(a, b):
        b = torch.from_numpy(np.asarray(b))
        assert (a.detach() - b).norm() <= 2e-5 * b.norm() + 1e-12

    close(o, g["o"])
    close(aux, g["aux_loss"])
    close(grads[0], g["dx"])
    for n, got in zip(names, grads[1:]):
        close(got, g[f"grad.{n}"])


def test_fp8_layer_refuses_biases_and_other_activations(built_library):
    """The FP8 experts are bias-free SwiGLU: other configurations are refused, not silently mis-computed."""
    from sonicmoe.functional.fp8 import moe_fp8_softmax_topk_layer

    m, inp = _module()
    w1 = m.c_fc.weight.permute(1, 2, 0)
    w2 = m.c_proj.weight.permute(1, 2, 0)
    b1, b2 = torch.zeros(8, 128), torch.zeros(8, 128)
    with pytest.raises(NotImplementedError):
        moe_fp8_softmax_topk_layer(inp["x"], m.router.weight, w1, b1, w2, b2, 2)
    with pytest.raises(NotImplementedError):
        moe_fp8_softmax_topk_layer(inp["x"], m.router.weight, w1, None, w2, None, 2, 0, "geglu")


def test_weight_grad_sum_bookkeeping():
    """`WeightGradSum`: the first chunk gets fresh buffers and stores, later chunks get the same buffers and add, only
    the last chunk hands the gradients on, and the object is empty again afterwards."""
    import torch

    from sonicmoe.functional import WeightGradSum

    w1, w2 = torch.zeros(2, 4, 3), torch.zeros(2, 3, 2)
    shared = WeightGradSum(3)
    d1, d2, add = shared.buffers(w1, w2)
    assert not add and d1.shape == w1.shape and d2.shape == w2.shape
    assert shared.finish_chunk() == (None, None)
    e1, e2, add = shared.buffers(w1, w2)
    assert add and e1 is d1 and e2 is d2
    assert shared.finish_chunk() == (None, None)
    f1, f2, add = shared.buffers(w1, w2)
    assert add and f1 is d1
    out1, out2 = shared.finish_chunk()
    assert out1 is d1 and out2 is d2
    assert shared.dw1 is None and shared.dw2 is None and shared.remaining == 0


def test_router_and_expert_weights_must_agree(built_library):
    """One number of experts, one hidden size: checked before anything reads a weight."""
    from sonicmoe.functional import moe_TC_softmax_topk_layer
    from sonicmoe.functional.fp8 import moe_fp8_softmax_topk_layer

    x, w1, w2 = torch.zeros(4, 128), torch.zeros(256, 128, 32), torch.zeros(128, 128, 32)
    for layer in (moe_TC_softmax_topk_layer, moe_fp8_softmax_topk_layer):
        for router in (torch.zeros(64, 128), torch.zeros(16, 128), torch.zeros(32, 64), torch.zeros(32, 256)):
            with pytest.raises(ValueError):
                layer(x, router, w1, None, w2, None, 2)


@pytest.mark.parametrize("entry,position", [("route_metadata", 10), ("router_forward_aux", 9)])
def test_calls_that_overlap_have_workspaces_of_their_own(built_library, monkeypatch, entry, position):
    """A second call that runs inside the first, as one of another thread or stream may: their scratch must differ."""
    import contextlib

    from sonicmoe import _lib, functional as fn

    real, spaces = _lib.lib, []

    def call():
        if entry == "route_metadata":
            fn._route_metadata(torch.zeros(64, dtype=torch.int32), None, 32, 2)
        else:
            fn._FusedRouter.apply(torch.zeros(32, 64).bfloat16(), torch.zeros(32, 64).bfloat16(), 2)

    class Library:
        def __getattr__(self, name):
            if name != "smoe_" + entry:
                return getattr(real, name)

            def kernel(*args):
                spaces.append(args[position])
                if len(spaces) == 1:
                    call()
                return 0

            return kernel

    state = _lib._DeviceState(torch.device("cpu"))
    monkeypatch.setattr(fn, "lib", Library())
    monkeypatch.setattr(fn, "stream_ptr", lambda device: 0)
    monkeypatch.setattr(_lib, "require_cuda", lambda t, name: None)
    monkeypatch.setattr(_lib, "device_state", lambda device: state)
    monkeypatch.setattr(torch.cuda, "device", lambda device: contextlib.nullcontext())
    call()
    assert len(spaces) == 2 and all(spaces) and spaces[0] != spaces[1]


def test_recorded_backward_of_the_load_balancing_loss(built_library, monkeypatch):
    """Second derivatives through the loss that kernels compute, against those of its formula."""
    import contextlib

    from sonicmoe import _lib, functional as fn

    class Library:  # the kernels' results play no part in a recorded backward pass
        def __getattr__(self, name):
            return getattr(_lib.lib, name) if name.endswith("bytes") else lambda *args: 0

    monkeypatch.setattr(fn, "lib", Library())
    monkeypatch.setattr(fn, "stream_ptr", lambda device: 0)
    monkeypatch.setattr(torch.cuda, "device", lambda device: contextlib.nullcontext())
    T, E = 24, 8
    x = torch.randn(T, 16, generator=torch.Generator().manual_seed(0)).requires_grad_(True)
    w = torch.randn(E, 16, generator=torch.Generator().manual_seed(1)).requires_grad_(True)
    freq = torch.arange(E, dtype=torch.int32)
    results = []
    for loss in (fn._SwitchLoss.apply,
                 lambda logits, n: fn.switch_loss_formula(torch.softmax(logits, -1, dtype=torch.float32), n)):
        for logits in ((x @ w.T).bfloat16(), (w @ x.T).bfloat16().T):  # a transposed view as well
            first = torch.autograd.grad(loss(logits, freq), [x, w], create_graph=True)
            second = torch.autograd.grad(sum(g.square().sum() for g in first), [x, w])
            results.append([*first, *second])
    for got, want in zip(results[:2], results[2:]):
        for a, b in zip(got, want):
            assert b.abs().max() > 0 and torch.equal(a, b)


def test_own_load_balancing_loss_is_used(built_library, monkeypatch):
    """A subclass's (or an instance's) `_compute_switch_loss` takes the place of the loss kernels."""
    import sonicmoe.moe as module

    m, inp = _module()
    T, E = 96, 8
    layer = (torch.zeros(T, 128), torch.zeros(T, E), torch.full((E,), 24, dtype=torch.int32), None, None)
    monkeypatch.setattr(module, "_layer_with_aux", lambda *args: layer)
    monkeypatch.setattr(module, "switch_loss", lambda logits, freq: torch.tensor(1.0))
    assert m(inp["x"])[1].item() == 1.0

    class Own(module.MoE):
        def _compute_switch_loss(self, logits, probs, expert_frequency):
            return probs.sum() * 0 + 2.0

    m.__class__ = Own
    assert m(inp["x"])[1].item() == 2.0
    m._compute_switch_loss = lambda logits, probs, expert_frequency: torch.tensor(3.0)
    assert m(inp["x"])[1].item() == 3.0


def test_waits_of_whole_warps_have_one_answer():
    """A wait on an mbarrier is given up after a time limit, which the lanes of a warp may see at different polls.  Where a whole
    warp waits (and its loop goes on with warp-wide operations) that has to be by mbar_wait_warp; mbar_wait is for code that a
    single elected thread runs."""
    seen = 0
    csrc = os.path.join(ROOT, "sonic-moe_b200", "csrc")
    for name in sorted(os.listdir(csrc)):
        if name == "ptx.cuh":  # defines both
            continue
        text = open(os.path.join(csrc, name)).read()
        text = re.sub(r'/\*.*?\*/|//[^\n]*|"[^"\n]*"', lambda m: re.sub(r"[^\n]", " ", m[0]), text, flags=re.S)
        headers, start = [], 0  # what stands before each open brace
        for m in re.finditer(r"[{};]|\bmbar_wait\(", text):
            if m[0] == "mbar_wait(":
                seen += 1
                line = text.count("\n", 0, m.start()) + 1
                assert any(re.search(r"\belect(ed\b|_one\()", h) for h in headers), f"{name}:{line}"
                continue
            if m[0] == "{":
                headers.append(text[start:m.start()])
            elif m[0] == "}":
                headers.pop()
            start = m.end()
    assert seen > 10


def test_warps_that_meet_at_a_named_barrier_give_up_together():
    """Behind a wait that may be abandoned, warps that will meet at a named barrier decide together whether it was."""
    csrc = os.path.join(ROOT, "sonic-moe_b200", "csrc")
    for name in sorted(os.listdir(csrc)):
        text = open(os.path.join(csrc, name)).read()
        for m in re.finditer(r"\bbar\.sync %\d", text):
            before = text[:m.start()]
            wait = before.rfind("mbar_wait_warp(")
            assert "warps_agree(" in before[wait:], f"{name}:{before.count(chr(10)) + 1}"


def test_biases_of_another_size_are_refused(built_library, monkeypatch):
    """The kernels read E rows of both biases."""
    from sonicmoe import functional as fn

    monkeypatch.setattr(fn._lib, "require_cuda", lambda *args: None)
    E, H, I = 4, 64, 128

    def bf(*shape):
        return torch.zeros(shape, dtype=torch.bfloat16)

    x, w1, w2 = bf(8, H), bf(E, I, H), bf(E, H, I)
    good, views = (bf(E, I), bf(E, H)), (w1.permute(1, 2, 0), w2.permute(1, 2, 0))
    fn._check_experts_args(x, w1, w2, *good, "gelu", expert_major=True)
    fn._check_experts_args(x, *views, *good, "gelu")
    for b1, b2 in ((bf(E - 1, I), good[1]), (good[0], bf(H)), (bf(E, H), good[1])):
        with pytest.raises(ValueError):
            fn._check_experts_args(x, w1, w2, b1, b2, "gelu", expert_major=True)
        with pytest.raises(ValueError):
            fn._check_experts_args(x, *views, b1, b2, "gelu")
