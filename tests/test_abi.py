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
