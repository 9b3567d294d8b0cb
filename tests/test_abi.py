"""The C-ABI library loads without a GPU and exports exactly what include/sonicmoe_b200.h declares."""

import ctypes
import os
import re

from conftest import ROOT


def _declared():
    text = open(os.path.join(ROOT, "include", "sonicmoe_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(smoe_\w+)\s*\(", text)))


def test_header_symbols_are_exported(built_library):
    lib = ctypes.CDLL(built_library)
    names = _declared()
    assert len(names) >= 15
    for name in names:
        assert hasattr(lib, name), f"{name} is declared in the header but not exported"


def test_python_binding_covers_header(built_library):
    from sonicmoe import _lib

    assert sorted(_lib.SIGNATURES) == _declared()
    assert _lib.lib.smoe_abi_version() >= 1


def test_queries_and_argument_checks_without_gpu(built_library):
    """Entry points validate sizes before touching the device, so these calls are safe on a CPU-only box."""
    from sonicmoe import _lib

    lib = _lib.lib
    assert lib.smoe_ds_partial_columns(1024) == 8   # one row of partials per 128 accumulator columns
    assert lib.smoe_ds_partial_columns(64) == 2
    assert lib.smoe_route_metadata_workspace_bytes(128) >= 128 * 4
    # hidden size not a multiple of 64 -> shape error, nothing launched
    assert lib.smoe_up_projection_forward(None, None, None, None, None, None, 16, 100, 64, 8, 32, None, None) == -1
    assert lib.smoe_down_projection_forward(None, None, None, None, 128, 100, 8, 32, None, None) == -1
    # more experts than the kernels' tile table holds
    assert lib.smoe_up_projection_backward_dx(None, None, None, None, 128, 64, 5000, 32, None, None) == -1
    assert lib.smoe_topk_softmax(None, 0, None, None, 4, 8, 9, None) == -1      # K > E
    assert lib.smoe_topk_softmax(None, 7, None, None, 4, 8, 2, None) == -6      # unknown dtype
    assert lib.smoe_gather_sum(None, None, None, 0, None, None, 4, 12, 2, None) == -1  # H % 8
    # expert-parallel kernel: segment table checked on the host before anything is launched
    assert lib.smoe_gather_sum_to_peers(None, None, 0, None, None, 8, 64, 1, None, None, 0, 0, None) == -1
    assert lib.smoe_gather_sum_to_peers(None, None, 0, None, None, 8, 64, 1, None, None, 17, 0, None) == -1
    assert lib.smoe_router_forward_supported(4096, 128, 8) == 1
    assert lib.smoe_router_forward_supported(4096, 8, 2) == 0 and lib.smoe_router_forward_supported(4096, 128, 17) == 0
    # empty problems are no-ops
    assert lib.smoe_topk_softmax(None, 0, None, None, 0, 8, 2, None) == 0
    assert lib.smoe_up_projection_forward(None, None, None, None, None, None, 16, 128, 64, 8, 0, None, None) == 0


def test_block_quantiser_refuses_misaligned_pointers(built_library):
    """Refused before anything is launched (the addresses here belong to nothing)."""
    from sonicmoe._lib import lib

    for quantise in (lib.smoe_fp8_quantize_blocks, lib.smoe_mxfp8_quantize_blocks):
        assert quantise(4096 + 2, 8192, 8192, 1, 128, 128, None) == -2
        assert quantise(4096 + 4, 8192, 8192, 1, 128, 128, None) == -2
        assert quantise(4096, 8192 + 2, 8192, 1, 128, 128, None) == -2
    assert lib.smoe_fp8_quantize_blocks(4096, 8192, 8192 + 2, 1, 128, 128, None) == -2


def test_layer_forward_refuses_before_the_first_launch(built_library):
    """Sizes and pointers that only a later kernel of the call would refuse (the addresses here belong to nothing)."""
    from sonicmoe._lib import lib

    def call(T=4, H=128, I=64, E=32, K=2, **bad):
        names = ["x", "router_w", "w1", "w2", "o", "logits", "expert_count", "prob_colsum", "aux", "scratch"]
        return lib.smoe_layer_forward(*[bad.get(n, 4096) for n in names], T, H, I, E, K, None, None)

    assert call(I=100) == -1 and call(I=0) == -1 and call(H=100) == -1 and call(E=8) == -1 and call(K=17) == -1
    assert call(T=0) == -1 and call(T=2 ** 30, K=2) == -1
    for name in ("x", "router_w", "w1", "w2", "o", "logits"):
        assert call(**{name: 4096 + 8}) == -2 and call(**{name: None}) == -1, name
    for name in ("expert_count", "prob_colsum", "aux"):
        assert call(**{name: 4096 + 2}) == -2 and call(**{name: None}) == -1, name
    assert call(scratch=4096 + 16) == -2 and call(scratch=None) == -7


def test_layer_training_calls_refuse_before_the_first_launch(built_library):
    """Sizes that do not fit the activation (the scratch is laid out for N1 rows) or that only a later kernel of the call would
    refuse, missing and misaligned pointers (the addresses here belong to nothing)."""
    from sonicmoe._lib import lib

    swiglu, gelu = 0, 5
    sizes = dict(T=4, H=128, I=64, N1=128, E=32, K=2)

    def forward(fused=True, activation=swiglu, dtype=1, **bad):
        s = {**sizes, **{k: bad.pop(k) for k in sizes if k in bad}}
        p = {n: 4096 for n in ("x", "router_w", "logits", "w1", "b1", "w2", "b2", "o", "z", "meta", "expert_count",
                               "prob_colsum", "aux", "scratch")}
        p.update(router_w=4096 if fused else None, b1=None, b2=None, **{} if fused else dict(prob_colsum=None, aux=None))
        p.update(bad)
        return lib.smoe_layer_train_forward(
            p["x"], p["router_w"], p["logits"], dtype, p["w1"], p["b1"], p["w2"], p["b2"], p["o"], p["z"], p["meta"],
            p["expert_count"], p["prob_colsum"], p["aux"], p["scratch"], *s.values(), activation, None, None)

    def act(fused=1, activation=swiglu, dtype=1, **bad):
        s = {**sizes, **{k: bad.pop(k) for k in sizes if k in bad}}
        p = {n: 4096 for n in ("dout", "w2", "z", "meta", "logits", "dlogits", "scratch")}
        p.update(dict.fromkeys(("b2", "g_logits", "g_colsum", "g_aux", "db1", "db2")))
        p.update(bad)
        return lib.smoe_layer_backward_act(
            p["dout"], p["w2"], p["b2"], p["z"], p["meta"], p["logits"], dtype, fused, p["g_logits"], p["g_colsum"],
            p["g_aux"], p["dlogits"], p["db1"], p["db2"], p["scratch"], *s.values(), activation, None, None)

    def dx(**bad):
        s = {**sizes, **{k: bad.pop(k) for k in sizes if k in bad}}
        p = {n: 4096 for n in ("w1", "meta", "scratch", "dx_expanded", "dx")} | bad
        return lib.smoe_layer_backward_dx(p["w1"], p["meta"], p["scratch"], p["dx_expanded"], p["dx"], 0, *s.values(), None,
                                          None)

    def weights(**bad):
        s = {**sizes, **{k: bad.pop(k) for k in sizes if k in bad}}
        p = {n: 4096 for n in ("x", "dout", "meta", "scratch", "dw1", "dw2")} | bad
        return lib.smoe_layer_backward_weights(p["x"], p["dout"], p["meta"], p["scratch"], p["dw1"], p["dw2"], *s.values(),
                                               None, None)

    def unfused(**bad):
        return forward(fused=False, **bad)

    for call in (forward, unfused, act, dx, weights):
        for bad in (dict(T=0), dict(T=2 ** 30), dict(H=100), dict(I=100, N1=200), dict(I=0, N1=0), dict(I=192, N1=192),
                    dict(N1=192), dict(E=0), dict(E=1025), dict(K=0), dict(K=33)):
            assert call(**bad) == -1, (call.__name__, bad)
    for call in (forward, unfused, act):
        assert call(activation=swiglu, I=128, N1=128) == -1 and call(activation=gelu, I=128, N1=256) == -1
        assert call(activation=7) == -1 and call(activation=-1) == -1
    assert forward(E=8) == -1 and forward(K=17) == -1              # not the fused router's
    assert unfused(dtype=2) == -6 and act(fused=0, dtype=2) == -6
    for call, names in ((forward, ("x", "router_w", "logits", "w1", "w2", "o")), (unfused, ("x", "w1", "w2", "o")),
                        (act, ("dout", "w2", "z")), (dx, ("w1", "dx")), (weights, ("x", "dout", "dw1", "dw2"))):
        for name in names:
            assert call(**{name: 4096 + 8}) == -2, (call.__name__, name)
            if name not in ("router_w", "dout") or call is weights:  # (None there selects another form)
                assert call(**{name: None}) == -1, (call.__name__, name)
        assert call(meta=None) == -7 and call(meta=4096 + 2) == -2
        assert call(scratch=None) == -7 and call(scratch=4096 + 16) == -2
    assert unfused(logits=4096 + 1) == -2 and unfused(logits=4096 + 2, dtype=0) == -2 and unfused(logits=None) == -1
    for name in ("b1", "b2", "z"):
        assert forward(**{name: 4096 + 8}) == -2, name
    for name in ("expert_count", "prob_colsum", "aux"):
        assert forward(**{name: 4096 + 2}) == -2, name
    assert forward(expert_count=None) == -1 and forward(aux=None) == -1
    assert act(b2=4096) == -1 and act(b2=4096, db1=4096) == -1 and act(b2=4096, db1=4096, db2=4096 + 8) == -2
    assert act(b2=4096 + 8, db1=4096, db2=4096) == -2
    for given in ("g_colsum", "g_aux"):
        assert act(**{given: 4096}, logits=None) == -1 and act(**{given: 4096 + 2}) == -2
    assert act(dlogits=4096 + 1) == -2 and act(g_logits=4096 + 1) == -2 and act(fused=0, dtype=0, dlogits=4096 + 2) == -2
    assert act(E=512) == -1                                        # more experts than the router's backward pass takes
    assert act(fused=0, dout=None) == -1                           # nothing to derive the logits' gradient from
    assert dx(dx_expanded=None) == -7 and dx(dx_expanded=4096 + 8) == -2


def test_training_forward_scratch_without_rows_that_nothing_writes(built_library):
    """SwiGLU without biases writes the down projection's rows of top-1 routing straight to the output."""
    from sonicmoe._lib import lib

    T, H, I, E = 1000, 192, 64, 8
    for K in (1, 2):
        every = lib.smoe_layer_train_forward_scratch_bytes(T, H, I, E, K)
        plain = lib.smoe_layer_train_forward_plain_scratch_bytes(T, H, I, E, K)
        rows = -(-T * K * H * 2 // 256) * 256
        assert every - plain == (rows if K == 1 else 0) and plain >= T * K * I * 2
    assert lib.smoe_layer_train_forward_plain_scratch_bytes(0, H, I, E, 1) == 0


def test_biases_read_in_16_byte_pieces(built_library):
    """Biases that are a view at another offset of a larger buffer are refused before anything is launched (the addresses here
    belong to nothing)."""
    from sonicmoe._lib import lib

    at, off = 4096, 4096 + 8
    gelu = 5
    assert lib.smoe_up_projection_forward_act(at, at, off, at, at, at, at, 4, 128, 128, 8, 8, gelu, None, None) == -2
    assert lib.smoe_down_projection_forward_bias(at, at, off, at, at, 128, 64, 8, 8, None, None) == -2
    assert lib.smoe_ds_add_bias_term(at, off, at, at, at, at, 0, 8, 128, 8, None) == -2
    assert lib.smoe_ds_add_bias_term(off, at, at, at, at, at, 0, 8, 128, 8, None) == -2
    assert lib.smoe_expert_column_sum(off, 128, None, None, 0, None, at, at, 8, 128, None) == -2
    assert lib.smoe_up_projection_forward_act(at, at, off, at, at, at, at, 4, 128, 128, 8, 0, gelu, None, None) == 0


def test_rule_of_the_dual_tiles(built_library):
    """The lines of the rule: reductions of the up projection above 2048, weight gradients of 480 rows per expert on average, and
    no last unit that is half empty."""
    from sonicmoe._lib import lib

    up, dw1, dw2 = 0, 1, 2
    assert [lib.smoe_dual_tiles(up, H, 960, 8, 4000) for H in (1024, 2048, 2112, 4096)] == [0, 0, 1, 1]
    for gemm in (dw1, dw2):
        assert [lib.smoe_dual_tiles(gemm, 2112, 960, 8, rows) for rows in (256, 3839, 3840, 2 ** 31 - 1)] == [0, 0, 1, 1]
    assert lib.smoe_dual_tiles(up, 4096, 384, 8, 4000) == 0 and lib.smoe_dual_tiles(up, 4096, 768, 8, 4000) == 1
    assert lib.smoe_dual_tiles(dw2, 4096, 768, 8, 8000) == 0 and lib.smoe_dual_tiles(dw1, 4096, 768, 8, 8000) == 1
    assert lib.smoe_dual_tiles(3, 4096, 1024, 8, 8000) == 0
