"""Whole-layer parity on the GPU: the `sonicmoe.MoE` module and the functional entry points against the
CPU oracle and against the golden fixtures produced by the reference.

Tolerance: relative Frobenius error <= 1e-2 for every bf16 output and gradient (the bound stated for the
bf16 layer); routing (indices, expert frequencies) bit-exact on the same logits.
"""

import pytest
import torch

from conftest import golden
from oracle import moe_oracle as orc

pytestmark = pytest.mark.gpu

TOL = 1e-2


def rel(a, b):
    a = a.detach().float().cpu()
    b = torch.as_tensor(b).detach().float().cpu()
    return ((a - b).norm() / (b.norm() + 1e-30)).item()


def _module(T, H, I, E, K, seed, **kw):
    import sonicmoe
    from sonicmoe.enums import ActivationType

    inp = orc.make_inputs(T, H, I, E, K, seed=seed, dtype=torch.bfloat16, **kw)
    m = sonicmoe.MoE(E, K, H, I, ActivationType.SWIGLU, False, 0.02).cuda().to(torch.bfloat16)
    with torch.no_grad():
        m.router.weight.copy_(inp["router_w"])
        m.c_fc.weight.copy_(inp["w1"])
        m.c_proj.weight.copy_(inp["w2"])
    return m, inp


# reference test matrix shapes (tests/moe_test.py:25-38) scaled to sizes the CPU oracle finishes in seconds,
# plus ragged / tiny / single-expert-per-token cases
LAYER_SHAPES = [
    (512, 256, 128, 16, 4),
    (1024, 768, 256, 8, 2),
    (777, 768, 320, 32, 8),
    (640, 1536, 256, 64, 16),
    (64, 128, 64, 4, 1),
    (2048, 768, 256, 128, 8),
    (30, 256, 64, 256, 8),   # far fewer tokens than experts: most experts are empty
]


@pytest.mark.parametrize("T,H,I,E,K", LAYER_SHAPES)
@pytest.mark.parametrize("fused_combine", [False, True])
def test_module_forward_backward_vs_oracle(built_library, T, H, I, E, K, fused_combine):
    from sonicmoe import _lib, functional

    m, inp = _module(T, H, I, E, K, seed=T + E)
    prev = functional.set_fused_combine(fused_combine)
    try:
        x = inp["x"].cuda().requires_grad_(True)
        o, aux = m(x.view(1, T, H))
        assert o.shape == (1, T, H) and o.dtype == torch.bfloat16
        grads = torch.autograd.grad(o, [x, m.router.weight, m.c_fc.weight, m.c_proj.weight],
                                    inp["dout"].cuda().view(1, T, H))
    finally:
        functional.set_fused_combine(prev)
    torch.cuda.synchronize()
    _lib.check_status()

    logits = functional.layer_router_logits(x.detach(), m.router.weight.detach(), K)
    f32 = {k: v.float() for k, v in inp.items()}
    ref = orc.moe_layer(f32["x"], f32["router_w"], f32["w1"], f32["w2"], K, dout=f32["dout"],
                        logits=logits.float().cpu())
    # routing on the same logits tensor is bit-exact
    scores, idx = functional.topk_softmax(logits, K)
    assert torch.equal(idx.cpu(), ref["indices"])
    assert rel(o.view(T, H), ref["o"]) < TOL
    assert rel(aux, ref["aux_loss"]) < 1e-3
    # dx = expert path + router path; the router path is torch autograd on bf16 logits
    assert rel(grads[0], ref["dx"]) < TOL
    assert rel(grads[1], ref["drouter_w"]) < 2e-2  # dlogits are rounded to bf16 before the router GEMM
    assert rel(grads[2], ref["dw1"]) < TOL
    assert rel(grads[3], ref["dw2"]) < TOL
    assert grads[2].shape == m.c_fc.weight.shape and grads[3].shape == m.c_proj.weight.shape


@pytest.mark.parametrize("name", ["layer_small", "layer_ties", "layer_k1"])
def test_functional_layer_vs_reference_golden(built_library, name):
    """The device path against outputs of the reference's own eager layer (fp32 router, bf16 experts)."""
    from sonicmoe import _lib
    from sonicmoe.functional import moe_TC_softmax_topk_layer

    g = golden(name)
    T, H, I, E, K, seed, _ = [int(v) for v in g["meta"]]
    inp = orc.make_inputs(T, H, I, E, K, seed=seed, dtype=torch.bfloat16)
    x = inp["x"].cuda().requires_grad_(True)
    rw = inp["router_w"].float().cuda().requires_grad_(True)  # fp32 router: same logits as the reference run
    w1 = inp["w1"].cuda().requires_grad_(True)
    w2 = inp["w2"].cuda().requires_grad_(True)
    o, logits, freq = moe_TC_softmax_topk_layer(x, rw, w1.permute(1, 2, 0), None, w2.permute(1, 2, 0), None, K)
    grads = torch.autograd.grad(o, [x, rw, w1, w2], inp["dout"].cuda())
    torch.cuda.synchronize()
    _lib.check_status()
    assert torch.equal(freq.cpu(), torch.from_numpy(g["expert_frequency"]))
    assert rel(logits, g["logits"]) < 1e-5
    assert rel(o, g["o"]) < TOL
    for got, key in zip(grads, ("dx", "drouter_w", "dw1", "dw2")):
        assert rel(got, g[key]) < TOL, key


def test_inference_mode_matches_training_forward(built_library):
    m, inp = _module(512, 256, 128, 16, 4, seed=3)
    x = inp["x"].cuda()
    o_train, _ = m(x)
    m.eval()
    with torch.no_grad():
        o_eval, _ = m(x)
    o_flag, _ = m.train()(x, is_inference_mode=True)
    assert torch.equal(o_train, o_eval) and torch.equal(o_train, o_flag)


@pytest.mark.parametrize("routing", ["nr", "up", "down"])
@pytest.mark.parametrize("T,H,I,E,K", [(1024, 256, 128, 8, 2), (2048, 512, 128, 16, 4)])
def test_token_rounding_layer_vs_oracle(built_library, routing, T, H, I, E, K):
    """Token-rounding router + general-routing layer: selections bit-exact, outputs and gradients in tolerance."""
    from sonicmoe import _lib
    from sonicmoe.functional import forward_token_choice_rounding, moe_general_routing_inputs

    inp = orc.make_inputs(T, H, I, E, K, seed=T + E + len(routing), dtype=torch.bfloat16)
    x = inp["x"].cuda().requires_grad_(True)
    w1 = inp["w1"].cuda().requires_grad_(True)
    w2 = inp["w2"].cuda().requires_grad_(True)
    scores, tokens, experts = forward_token_choice_rounding(x.detach(), inp["router_w"].cuda(), E, K, 128, routing)
    logits = torch.nn.functional.linear(x.detach(), inp["router_w"].cuda())
    s_ref, t_ref, e_ref, _ = orc.token_rounding_route(logits.cpu(), K, routing, torch.bfloat16)
    assert torch.equal(tokens.cpu(), t_ref) and torch.equal(experts.cpu(), e_ref)
    assert torch.equal(scores.cpu(), s_ref)
    counts = torch.bincount(experts.long(), minlength=E)
    assert (counts % 128 == 0).all()

    sc = scores.detach().clone().requires_grad_(True)
    o, freq = moe_general_routing_inputs(x, sc, tokens, experts, w1.permute(1, 2, 0), None, w2.permute(1, 2, 0),
                                         None, E, 0, __import__("sonicmoe").ActivationType.SWIGLU)
    grads = torch.autograd.grad(o, [x, w1, w2, sc], inp["dout"].cuda())
    torch.cuda.synchronize()
    _lib.check_status()
    assert torch.equal(freq.cpu(), counts.cpu().int())
    f32 = {k: v.float() for k, v in inp.items()}
    ref = orc.general_routing_layer(f32["x"], f32["w1"], f32["w2"], s_ref.float(), t_ref, e_ref, dout=f32["dout"])
    assert rel(o, ref["o"]) < TOL
    assert rel(grads[0], ref["dx"]) < TOL
    assert rel(grads[1], ref["dw1"]) < TOL
    assert rel(grads[2], ref["dw2"]) < TOL
    assert grads[3].dtype == torch.bfloat16 and rel(grads[3], ref["ds"]) < TOL


def test_general_routing_with_empty_tokens_and_experts(built_library):
    from sonicmoe import ActivationType, _lib
    from sonicmoe.functional import moe_general_routing_inputs

    T, H, I, E = 200, 128, 64, 8
    inp = orc.make_inputs(T, H, I, E, 2, seed=5, dtype=torch.bfloat16, w_std=0.05)
    g = torch.Generator().manual_seed(1)
    n = 300
    tokens = torch.randint(0, T // 2, (n,), generator=g).sort().values.int()  # upper half of the tokens unused
    experts = torch.randint(0, E - 2, (n,), generator=g).int()                # two experts unused
    scores = torch.rand(n, generator=g)
    x = inp["x"].cuda().requires_grad_(True)
    w1 = inp["w1"].cuda().requires_grad_(True)
    w2 = inp["w2"].cuda().requires_grad_(True)
    sc = scores.cuda().requires_grad_(True)
    o, freq = moe_general_routing_inputs(x, sc, tokens.cuda(), experts.cuda(), w1.permute(1, 2, 0), None,
                                         w2.permute(1, 2, 0), None, E, 0, ActivationType.SWIGLU)
    grads = torch.autograd.grad(o, [x, w1, w2, sc], inp["dout"].cuda())
    torch.cuda.synchronize()
    _lib.check_status()
    f32 = {k: v.float() for k, v in inp.items()}
    ref = orc.general_routing_layer(f32["x"], f32["w1"], f32["w2"], scores, tokens, experts, dout=f32["dout"])
    assert (o[T // 2:] == 0).all() and (grads[0][T // 2:] == 0).all()
    assert (grads[1][E - 2:] == 0).all() and (grads[2][E - 2:] == 0).all()
    assert rel(o, ref["o"]) < TOL and rel(grads[0], ref["dx"]) < TOL
    assert rel(grads[1], ref["dw1"]) < TOL and rel(grads[2], ref["dw2"]) < TOL
    assert grads[3].dtype == torch.float32 and rel(grads[3], ref["ds"]) < 1e-2


def test_linearity_at_full_hidden_size(built_library):
    """Size-independent property at the benchmark's H and I: with the routing fixed, the layer output is linear in
    the routing scores, o(a*s1 + b*s2) = a*o(s1) + b*o(s2), and doubling dout doubles every gradient."""
    from sonicmoe import ActivationType, _lib
    from sonicmoe.functional import moe_general_routing_inputs

    T, H, I, E, K = 4096, 4096, 1024, 16, 2
    inp = orc.make_inputs(T, H, I, E, K, seed=1, dtype=torch.bfloat16)
    g = torch.Generator().manual_seed(2)
    experts = torch.stack([torch.randperm(E, generator=g)[:K] for _ in range(T)]).reshape(-1).int().cuda()
    tokens = torch.arange(T).repeat_interleave(K).int().cuda()
    s1 = torch.rand(T * K, generator=g).cuda()
    s2 = torch.rand(T * K, generator=g).cuda()
    x = inp["x"].cuda()
    w1 = inp["w1"].cuda().permute(1, 2, 0)
    w2 = inp["w2"].cuda().permute(1, 2, 0)

    def run(s):
        with torch.no_grad():
            return moe_general_routing_inputs(x, s, tokens, experts, w1, None, w2, None, E, 0,
                                              ActivationType.SWIGLU)[0].float()

    o1, o2, o12 = run(s1), run(s2), run(0.5 * s1 + 2.0 * s2)
    assert ((o12 - (0.5 * o1 + 2.0 * o2)).norm() / o12.norm()).item() < TOL
    torch.cuda.synchronize()
    _lib.check_status()


def test_torch_compile_fullgraph_matches_eager(built_library):
    """`torch.compile(fullgraph=True)` of the module (the reference compiles it in its tests and benchmarks,
    tests/moe_test.py:80-81): same output and gradients as the eager module."""
    from sonicmoe import _lib

    T, H, I, E, K = 512, 256, 128, 16, 4
    m, inp = _module(T, H, I, E, K, seed=9)
    x = inp["x"].cuda().requires_grad_(True)
    dout = inp["dout"].cuda()
    o_ref, aux_ref = m(x)
    g_ref = torch.autograd.grad(o_ref, [x, m.router.weight, m.c_fc.weight, m.c_proj.weight], dout)
    compiled = torch.compile(m, fullgraph=True)
    o, aux = compiled(x)
    g = torch.autograd.grad(o, [x, m.router.weight, m.c_fc.weight, m.c_proj.weight], dout)
    torch.cuda.synchronize()
    _lib.check_status()
    assert torch.equal(o, o_ref)
    assert rel(aux, aux_ref) < 1e-5
    for a, b in zip(g, g_ref):
        assert a.shape == b.shape and rel(a, b) < 1e-3


@pytest.mark.parametrize("act,bias", [("swiglu", True), ("geglu", False), ("reglu", True), ("gelu", True),
                                      ("relu", False), ("silu", True), ("relu_sq", False)])
def test_bias_and_activations_vs_oracle(built_library, act, bias):
    """Every activation of the layer, with and without expert biases (the reference test matrix has
    add_bias, tests/moe_test.py:25-56; activations are a benchmark flag, benchmarks/moe-cute.py:62-94)."""
    import sonicmoe
    from sonicmoe import _lib
    from sonicmoe.enums import ActivationType, is_glu

    T, H, I, E, K = 700, 256, 128, 8, 2
    kind = ActivationType(act)
    n1 = 2 * I if is_glu(kind) else I
    g = torch.Generator().manual_seed(len(act) + bias)
    m = sonicmoe.MoE(E, K, H, I, kind, bias, 0.05).cuda().to(torch.bfloat16)
    with torch.no_grad():
        m.router.weight.copy_(torch.randn(E, H, generator=g) * 0.05)
        if bias:
            m.c_fc.bias.copy_(torch.randn(E, n1, generator=g) * 0.1)
            m.c_proj.bias.copy_(torch.randn(E, H, generator=g) * 0.1)
    x = torch.randn(T, H, generator=g).bfloat16().cuda().requires_grad_(True)
    dout = torch.randn(T, H, generator=g).bfloat16().cuda()
    o, _aux = m(x)
    params = [m.c_fc.weight, m.c_proj.weight] + ([m.c_fc.bias, m.c_proj.bias] if bias else [])
    grads = torch.autograd.grad(o, [x] + params, dout)
    torch.cuda.synchronize()
    _lib.check_status()

    from sonicmoe.functional import layer_router_logits

    logits = layer_router_logits(x.detach(), m.router.weight.detach(), K).float().cpu()
    scores, idx = orc.topk_softmax(logits, K)
    route = orc.route_metadata(idx, E, T, K=K)
    f = lambda t: None if t is None else t.detach().float().cpu()
    ref = orc.experts_autograd(f(x), f(m.c_fc.weight), f(m.c_fc.bias), f(m.c_proj.weight), f(m.c_proj.bias),
                               scores.reshape(-1), route, act, f(dout))
    dlogits = orc.softmax_topk_backward(scores, idx, ref["ds"].reshape(T, K), E)
    dx_ref = ref["dx"] + dlogits @ f(m.router.weight)
    assert rel(o, ref["o"]) < TOL
    assert rel(grads[0], dx_ref) < TOL
    assert rel(grads[1], ref["dw1"]) < TOL
    assert rel(grads[2], ref["dw2"]) < TOL
    if bias:
        assert rel(grads[3], ref["db1"]) < TOL
        assert rel(grads[4], ref["db2"]) < TOL


def test_second_device_in_one_process(built_library):
    """Kernel attributes (dynamic shared memory) and the SM count are cached per device, not per process: a layer on
    cuda:1 of a process that already ran one on cuda:0 launches and gives the same result."""
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    from sonicmoe import _lib

    T, H, I, E, K = 512, 256, 128, 16, 4
    outs = []
    for d in (0, 1):
        m, inp = _module(T, H, I, E, K, seed=3)
        m = m.to(f"cuda:{d}")
        x = inp["x"].to(f"cuda:{d}").requires_grad_(True)
        o, _ = m(x)
        o.backward(inp["dout"].to(f"cuda:{d}"))
        torch.cuda.synchronize(d)
        _lib.check_status(torch.device("cuda", d))
        outs.append((o.detach().cpu(), x.grad.cpu(), m.c_fc.weight.grad.cpu()))
    for a, b in zip(*outs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("kind", ["bf16", "fp8"])
def test_chunks_share_weight_gradient_buffers(built_library, kind):
    """A batch processed as three chunks that share a `WeightGradSum`: the last chunk's backward pass hands autograd
    the sum of the chunks' weight gradients (accumulated in the GEMM epilogues), the others hand it nothing; the
    parameters' gradients match the whole batch's within bf16 accumulation error, and the two-chunk case equals
    autograd's own accumulation of per-chunk gradients bit for bit.  The `on_dx` hook sees each chunk's dx before
    the chunk's weight gradients are launched.  Same contract for the FP8 local experts."""
    from sonicmoe import _lib, functional as fn
    from sonicmoe.functional.fp8 import _RoutedExpertsFp8

    T, H, I, E, K = 1536, 512, 256, 8, 2
    g = torch.Generator(device="cuda").manual_seed(11)

    def rn(*shape, std):
        return (torch.randn(*shape, generator=g, device="cuda") * std).bfloat16()

    x0, dout = rn(T, H, std=1.0), rn(T, H, std=1.0)
    w1, w2 = rn(E, 2 * I, H, std=0.05).requires_grad_(True), rn(E, H, I, std=0.05).requires_grad_(True)
    logits = rn(T, E, std=1.0)
    scores, idx = fn.topk_softmax(logits, K)

    def run(bounds, share):
        w1.grad = w2.grad = None
        x = x0.clone().requires_grad_(True)
        shared = fn.WeightGradSum(len(bounds) - 1) if share else None
        outs, announced = [], []
        for a, b in zip(bounds[:-1], bounds[1:]):
            route = fn._route_metadata(idx[a:b].reshape(-1), None, E, K)
            route.wgrad_sum = shared
            route.on_dx = lambda dx, a=a, b=b: announced.append((a, b, dx.clone()))
            args = (x[a:b], w1.permute(1, 2, 0), w2.permute(1, 2, 0), scores[a:b].reshape(-1), route, b - a, False)
            outs.append(_RoutedExpertsFp8.apply(*args, "ue8m0") if kind == "fp8" else fn._RoutedExperts.apply(*args))
        torch.cat(outs).backward(dout)
        torch.cuda.synchronize()
        _lib.check_status()
        assert len(announced) == len(bounds) - 1
        for a, b, dx in announced:
            assert torch.equal(dx, x.grad[a:b])
        return w1.grad.clone(), w2.grad.clone()

    whole = run([0, T], False)
    tol = 1e-2  # FP8 too: activations are quantised row by row, so cutting the batch changes no quantised value
    for bounds in ([0, 700, T], [0, 100, 100, T]):  # uneven chunks; an empty one
        separate, shared = run(bounds, False), run(bounds, True)
        for a, b, c in zip(shared, separate, whole):
            assert rel(a, c) < tol and rel(b, c) < tol
            if len(bounds) == 3:
                assert torch.equal(a, b)


@pytest.mark.parametrize("T,E,K", [(1, 32, 1), (1, 64, 4), (130, 32, 1), (777, 64, 4), (3000, 32, 8)])
def test_forward_without_gradients_matches_training_forward(built_library, T, E, K):
    """The one-call inference forward against the forward pass of a training step: the same kernels, so the same bits."""
    import sonicmoe
    from sonicmoe import _lib
    from sonicmoe.enums import ActivationType

    H, I = 256, 128
    inp = orc.make_inputs(T, H, I, E, K, seed=T, dtype=torch.bfloat16)
    m = sonicmoe.MoE(E, K, H, I, ActivationType.SWIGLU, False, 0.05).cuda().to(torch.bfloat16)
    x = inp["x"].cuda()
    o_ref, aux_ref = m(x)
    assert o_ref.requires_grad
    with torch.no_grad():
        o, aux = m(x)
        side = torch.cuda.Stream()  # its scratch is its own: a second stream gives the same
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            o_side, _ = m(x)
        torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    _lib.check_status()
    assert torch.equal(o, o_ref) and torch.equal(aux, aux_ref) and torch.equal(o_side, o_ref)
    assert not o.requires_grad
    out, logits, freq = sonicmoe.moe_TC_softmax_topk_layer(
        x, m.router.weight.detach(), m.c_fc.weight.detach().permute(1, 2, 0), None,
        m.c_proj.weight.detach().permute(1, 2, 0), None, K, 0, ActivationType.SWIGLU, True)
    assert torch.equal(out, o_ref) and logits.shape == (T, E) and int(freq.sum()) == T * K


def test_training_steps_on_two_streams_at_a_time(built_library):
    """Forward and backward passes of two layers on two streams, not ordered with each other, against the same one after
    the other."""
    import sonicmoe
    from sonicmoe import _lib
    from sonicmoe.enums import ActivationType

    T, H, I, K, rounds = 2048, 256, 128, 4, 8
    layers = []
    for n, E in enumerate((32, 64)):  # the second needs larger workspaces
        inp = orc.make_inputs(T, H, I, E, K, seed=n, dtype=torch.bfloat16)
        m = sonicmoe.MoE(E, K, H, I, ActivationType.SWIGLU, False, 0.05).cuda().to(torch.bfloat16)
        layers.append((m, inp["x"].cuda().requires_grad_(True), inp["dout"].cuda()))

    def step(m, x, dout):
        o, aux = m(x)
        return [o, aux, *torch.autograd.grad([o, aux], [x, *m.parameters()], [dout, torch.ones_like(aux)])]

    want = [[t.detach() for t in step(*layer)] for layer in layers]
    streams = [torch.cuda.Stream() for _ in layers]
    for s in streams:
        s.wait_stream(torch.cuda.current_stream())
    got = [[], []]
    for _ in range(rounds):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i].append([t.detach() for t in step(*layers[i])])
    torch.cuda.synchronize()
    _lib.check_status()
    for i in range(2):
        for result in got[i]:
            for a, b in zip(result, want[i]):
                assert torch.equal(a, b)


@pytest.mark.parametrize("T,E,K,kernels", [
    (1, 32, 1, 7),       # router 2, sort 3, up, down
    (4, 64, 4, 8),       # and the combine
    (1030, 128, 8, 8),   # 64 rows per expert: projections in one launch each
    (9600, 32, 4, 8),    # 256 x 256 tiles
])
def test_launch_count(built_library, T, E, K, kernels):
    """The library's own count of its launches, over an inference forward."""
    import sonicmoe
    from sonicmoe import _lib
    from sonicmoe.enums import ActivationType

    m = sonicmoe.MoE(E, K, 256, 128, ActivationType.SWIGLU, False, 0.05).cuda().to(torch.bfloat16)
    x = torch.randn(T, 256, device="cuda").bfloat16()
    with torch.no_grad():
        before = _lib.launch_count()
        m(x)
        assert _lib.launch_count() - before == kernels
    torch.cuda.synchronize()
    _lib.check_status()


@pytest.mark.parametrize("T,E,K", [(3, 64, 4), (300, 32, 2), (9600, 32, 4)])
def test_chained_launches_under_graph_capture(built_library, T, E, K):
    """The launches may begin before the kernel in front of them has ended: a captured forward pass and training step, replayed
    back to back on changing inputs, give the bits of the same passes run one by one with a synchronisation after each."""
    import sonicmoe
    from sonicmoe import _lib
    from sonicmoe.enums import ActivationType

    H, I, rounds = 256, 128, 6
    m = sonicmoe.MoE(E, K, H, I, ActivationType.SWIGLU, False, 0.05).cuda().to(torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(T)
    inputs = [torch.randn(T, H, device="cuda", generator=g).bfloat16() for _ in range(rounds)]
    dout = torch.randn(T, H, device="cuda", generator=g).bfloat16()
    x = inputs[0].clone().requires_grad_(True)

    def step():
        with torch.no_grad():
            o = m(x, is_inference_mode=True)[0]
        y, aux = m(x)
        return [o, y.detach(), *torch.autograd.grad([y, aux], [x, *m.parameters()], [dout, torch.ones_like(aux)])]

    want = []
    for v in inputs:
        with torch.no_grad():
            x.copy_(v)
        torch.cuda.synchronize()
        want.append([t.clone() for t in step()])
        torch.cuda.synchronize()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = step()
    got = []
    for v in inputs:
        with torch.no_grad():
            x.copy_(v)
        graph.replay()
        got.append([t.clone() for t in captured])
    torch.cuda.synchronize()
    _lib.check_status()
    for a, b in zip(got, want):
        for s, t in zip(a, b):
            assert torch.equal(s, t)


@pytest.mark.parametrize("T,E,K,act,bias", [
    (1, 32, 1, "swiglu", False), (333, 64, 4, "swiglu", False), (2050, 32, 1, "swiglu", False),
    (300, 8, 2, "swiglu", False), (257, 8, 1, "gelu", True), (700, 96, 16, "geglu", True), (130, 32, 1, "relu", False),
])
def test_layer_in_one_node_matches_separate_functions(built_library, T, E, K, act, bias):
    """The layer as one autograd node against the router, the routing metadata and the experts as functions of their own: the
    same kernels, so the same bits, except for the gradient of x with the fused router and K > 1.  There the experts' part e
    and the router's r (rounded by its GEMM in both) are added before e is rounded instead of after: s = b(b(e) + r) against
    t = b(e + r), which differ by u (|e| + |s| + |t|) at most, u = 2^-8 the unit roundoff of bf16 (8 significant bits; 2 % more for
    the products of two roundings).  Strided inputs,
    gradients of single outputs, frozen inputs and passes without gradients among them."""
    from sonicmoe import _lib, functional as fn
    from sonicmoe.enums import ActivationType, is_glu

    H, I = 256, 128
    kind = ActivationType(act)
    n1 = 2 * I if is_glu(kind) else I
    g = torch.Generator(device="cuda").manual_seed(T + E)

    def normal(*shape, std=0.05):
        return (torch.randn(*shape, device="cuda", generator=g) * std).bfloat16()

    wide = normal(T, 2 * H, std=1.0)
    x = wide[:, ::2]                                      # strided
    router, w1, w2 = normal(E, H), normal(n1, H, E), normal(E, H, I)  # w1 stored as the view that the layer takes
    b1, b2 = (normal(E, n1), normal(E, H)) if bias else (None, None)
    dout, gl = normal(T, H, std=1.0).t().contiguous().t(), normal(T, E)
    ga = torch.full((), 0.3, device="cuda")

    def separate(x, router, w1, b1, w2, b2):
        if fn.fused_router_applies(x, router, K):
            logits, scores, indices, _, _, aux = fn._FusedRouter.apply(x, router, K)
        else:
            logits = torch.nn.functional.linear(x, router)
            scores, indices = fn.topk_softmax(logits, K)
            aux = None
        route = fn._route_metadata(indices.reshape(-1), None, E, K)
        o = fn._experts(x, w1, b1, w2, b2, scores.reshape(-1), route, T, False, kind)
        return o, logits, route.expert_frequency, aux

    def one_node(x, router, w1, b1, w2, b2):
        o, logits, freq, _, aux = fn._layer_with_aux(x, router, w1.permute(2, 0, 1), b1, w2.permute(2, 0, 1), b2, K, kind,
                                                     False)
        return o, logits, freq, aux

    given = [x, router, w1, b1, w2.permute(1, 2, 0), b2]
    scores, indices = fn.topk_softmax(fn.layer_router_logits(x, router, K), K)
    xe = x.detach().requires_grad_(True)
    oe = fn._experts(xe, *given[2:], scores.reshape(-1), fn._route_metadata(indices.reshape(-1), None, E, K), T, False, kind)
    experts_dx, = torch.autograd.grad(oe, xe, dout)
    for frozen in ((), (0,), (1,), (2, 4), (0, 1)):
        results = []
        for layer in (separate, one_node):
            inputs = [None if t is None else t.detach().requires_grad_(i not in frozen) for i, t in enumerate(given)]
            o, logits, freq, aux = layer(*inputs)
            outputs = [(o, dout), (logits, gl)] + ([(aux, ga)] if aux is not None else [])
            wanted = [t for t in inputs if t is not None and t.requires_grad]
            grads = []
            for chosen in (outputs, outputs[:1], outputs[1:]):
                chosen = [c for c in chosen if c[0].requires_grad]
                grads.append(torch.autograd.grad([c[0] for c in chosen], wanted, [c[1] for c in chosen], retain_graph=True,
                                                 allow_unused=True) if chosen else ())
            results.append((o, logits, freq, aux, grads, wanted))
        torch.cuda.synchronize()
        _lib.check_status()
        (o, logits, freq, aux, grads, _), (o2, logits2, freq2, aux2, grads2, wanted) = results
        assert torch.equal(o, o2) and torch.equal(logits, logits2) and torch.equal(freq, freq2)
        assert aux is None and aux2 is None or torch.equal(aux, aux2)
        for a, b in zip(grads, grads2):
            for i, (s, t) in enumerate(zip(a, b)):
                assert (s is None) == (t is None)
                if s is not None and i == 0 and 0 not in frozen and K > 1 and aux is not None:
                    e, s, t = experts_dx.float(), s.float(), t.float()
                    assert ((s - t).abs() <= 1.02 * 2.0 ** -8 * (e.abs() + s.abs() + t.abs())).all()
                elif s is not None:
                    assert torch.equal(s, t), (frozen, i)
    with torch.no_grad():
        assert torch.equal(one_node(*given)[0], o)


@pytest.mark.parametrize("train", [False, True])
def test_second_stream_gets_on_beside_the_launch_chain(built_library, train):
    """A row of small kernels on a second stream, enqueued behind passes of the layer, ends long before these: a kernel of the chain
    must not stand in front of them while it waits for room itself, or each of them waits for the end of one of the layer's."""
    import sonicmoe
    from sonicmoe import _lib
    from sonicmoe.enums import ActivationType

    T, H, I, E, K = 16384, 4096, 1024, 32, 8  # about 5 (15) ms of kernels and 0.1 (0.5) ms of launches a pass
    passes = 4 if train else 10  # fewer kernels than the second stream has
    m = sonicmoe.MoE(E, K, H, I, ActivationType.SWIGLU, False, 0.02).cuda().to(torch.bfloat16)
    x = torch.randn(T, H, device="cuda").bfloat16().requires_grad_(train)
    dout = torch.randn(T, H, device="cuda").bfloat16()
    small = torch.zeros(1 << 20, device="cuda")
    side = torch.cuda.Stream()

    def layer():
        with torch.set_grad_enabled(train):
            o, _ = m(x, is_inference_mode=not train)
            if train:
                torch.autograd.grad(o, [x, *m.parameters()], dout)

    for _ in range(2):
        layer()
        small.add_(1.0)
    torch.cuda.synchronize()
    begin, end, side_end = (torch.cuda.Event(enable_timing=True) for _ in range(3))
    begin.record()
    for _ in range(passes):
        layer()
    end.record()
    with torch.cuda.stream(side):
        for _ in range(300):
            small.add_(1.0)
        side_end.record()
    torch.cuda.synchronize()
    _lib.check_status()
    assert begin.elapsed_time(side_end) < 0.7 * begin.elapsed_time(end)


@pytest.mark.parametrize("K", [1, 4])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_backward_pass_under_autocast(built_library, K, dtype):
    """A backward pass that runs inside an autocast region: the router's GEMMs may come out in the region's type, and the experts'
    part of the gradient of x is added to the router's.  Three roundings of at most 2^-8 (bf16 has 8 significant bits; fp16 more) of
    parts no larger than the gradient tell the two apart: 3 2^-8 < 2^-6 of the norm."""
    import sonicmoe
    from sonicmoe import _lib
    from sonicmoe.enums import ActivationType

    T, H, I, E = 300, 256, 128, 32
    m = sonicmoe.MoE(E, K, H, I, ActivationType.SWIGLU, False, 0.05).cuda().to(torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(K)
    x = torch.randn(T, H, device="cuda", generator=g).bfloat16().requires_grad_(True)
    dout = torch.randn(T, H, device="cuda", generator=g).bfloat16()
    wanted = [x, *m.parameters()]
    o, aux = m(x)
    outputs, grads = [o, aux], [dout, torch.ones_like(aux)]
    plain = torch.autograd.grad(outputs, wanted, grads, retain_graph=True)
    with torch.autocast("cuda", dtype=dtype):
        cast = torch.autograd.grad(outputs, wanted, grads)
    torch.cuda.synchronize()
    _lib.check_status()
    for p, c in zip(plain, cast):
        assert p.dtype == c.dtype == torch.bfloat16
        assert (p.double() - c.double()).norm() <= 2.0 ** -6 * p.double().norm()
