"""The C ABI: the library loads, exports every symbol include/b2q.h declares, and rejects bad
arguments with error codes before touching a device (no GPU needed)."""
import ctypes as C
import os
import re

import pytest


@pytest.fixture(scope="module")
def lib(lib_built):
    return C.CDLL(lib_built)


def _declared():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    text = open(os.path.join(root, "include", "b2q.h")).read()
    return sorted(set(re.findall(r"B2Q_API[^;(]*?\b(b2q_[a-z0-9_]+)\s*\(", text)))


def test_header_declares_entry_points():
    names = _declared()
    assert len(names) >= 20
    for must in ("b2q_linear_int4", "b2q_linear_fp8", "b2q_moe_gemm_int4", "b2q_moe_route", "b2q_strerror"):
        assert must in names


def test_every_declared_symbol_is_exported(lib):
    for name in _declared():
        assert hasattr(lib, name), name


def test_python_binding_covers_the_header(lib_built):
    from custom_esimd_kernels_vllm import _lib
    assert sorted(_lib.EXPORTED) == _declared()


def test_strerror_and_version(lib):
    lib.b2q_strerror.restype = C.c_char_p
    assert lib.b2q_strerror(0) == b"ok"
    for code in range(-10, 0):
        assert lib.b2q_strerror(code).startswith(b"b2q:")
    assert lib.b2q_version() >= 100


def test_null_and_shape_errors_need_no_device(lib_built):
    from custom_esimd_kernels_vllm import _lib as L
    lib = L.lib
    assert lib.b2q_linear_int4(None, 0, 128, None, 0, None, 0, 1, 1, None, 16, 1, 16, 128, 128, None, 0, None) == -1
    buf = (C.c_uint8 * 4096)()
    p = C.addressof(buf)
    p = (p + 255) // 256 * 256
    # group != 128
    assert lib.b2q_linear_int4(p, 0, 128, p, 0, p, 0, 1, 1, p, 16, 1, 16, 128, 64, None, 0, None) == -2
    # unknown activation dtype
    assert lib.b2q_linear_int4(p, 7, 128, p, 0, p, 0, 1, 1, p, 16, 1, 16, 128, 128, None, 0, None) == -3
    # unknown layout
    assert lib.b2q_linear_int4(p, 0, 128, p, 9, p, 0, 1, 1, p, 16, 1, 16, 128, 128, None, 0, None) == -5
    # misaligned activation pointer
    assert lib.b2q_linear_int4(p + 2, 0, 128, p, 0, p, 0, 1, 1, p, 16, 1, 16, 128, 128, None, 0, None) == -4
    # fp8: K not a multiple of 16, block mode needs fp32 scales
    assert lib.b2q_linear_fp8(p, 0, 40, p, 0, p, 2, 0, p, 16, 1, 16, 40, None, 0, None) == -2
    assert lib.b2q_linear_fp8(p, 0, 128, p, 0, p, 0, 2, p, 16, 1, 16, 128, None, 0, None) == -3
    # M == 0 is a successful no-op
    assert lib.b2q_linear_int4(p, 0, 128, p, 0, p, 0, 1, 1, p, 16, 0, 16, 128, 128, None, 0, None) == 0
    # route: workspace too small
    assert lib.b2q_moe_route(p, 1024, 8, p, p, p, p, p, 16, None) == -8
    assert lib.b2q_moe_topk(p, 0, 4, 2048, 8, 1, p, 0, p, None) == -10


def test_workspace_size_queries(lib_built):
    from custom_esimd_kernels_vllm import _lib as L
    assert L.lib.b2q_moe_route_workspace_bytes(32768, 128) == 128 * 128 * 4
    small = L.lib.b2q_moe_gemm_workspace_bytes(1024, 8, 256, 512, 0, 0)
    big = L.lib.b2q_moe_gemm_workspace_bytes(1024, 8, 256, 512, 1, 0)
    assert big >= small + 1024 * 256 * 2
    assert small >= 1024 * 512 * 2 + 1024 * 4          # staged activations + per-row scales are always there
    assert L.lib.b2q_linear_workspace_bytes(64, 1024, 8192) >= 64 * 8192 * 2 + 64 * 4 + 64 * 1024 * 4


def test_ops_refuse_cpu_tensors(lib_built):
    import torch
    import custom_esimd_kernels_vllm as e
    x = torch.zeros(1, 128, dtype=torch.bfloat16)
    w = torch.zeros(16, 64, dtype=torch.uint8)
    s = torch.zeros(16, 1, dtype=torch.bfloat16)
    o = torch.zeros(1, 16, dtype=torch.bfloat16)
    with pytest.raises((RuntimeError, NotImplementedError)):
        e.esimd_gemv_int4(x, w, s, o)
    with pytest.raises(RuntimeError):
        e._impl.linear_int4(x, w, s, o)


def test_reference_schemas_are_registered(lib_built):
    import torch
    import custom_esimd_kernels_vllm  # noqa: F401
    for ns, names in {
        "custom_esimd_kernels_vllm": ["esimd_gemv_int4", "esimd_gemv_int4_fused2", "esimd_gemm_int4_pgrp",
                                      "esimd_gemv_fp8_pern", "esimd_gemv_fp8_pert", "esimd_gemm_fp8_pert",
                                      "esimd_gemm_fp8_blockscale", "esimd_moe_topk", "esimd_moe_scatter_fused",
                                      "esimd_moe_silu_mul", "esimd_moe_gather", "esimd_moe_gemm_fp8",
                                      "esimd_moe_gemm_fp8_pert", "esimd_moe_gemm_fp8_blockscale"],
        "moe_int4_prefill_ops": ["moe_prefill_full_int4", "moe_prefill_gather_forward_v2", "moe_prefill_up_forward_v2",
                                 "moe_prefill_down_forward_v2", "moe_prefill_accumulate_forward_v2",
                                 "moe_prefill_accumulate_permuted_forward_v2", "moe_prefill_silu_mul_forward",
                                 "moe_prefill_scatter_x_forward", "moe_topk_softmax"],
        "moe_int4_ops": ["moe_topk_int4", "moe_route_precompute_int4", "moe_silu_mul_int4", "moe_route_gather_int4",
                         "moe_gemm_int4_nmajor"],
        "esimd_topk_v2": ["topk_v2"],
    }.items():
        for n in names:
            assert hasattr(getattr(torch.ops, ns), n), (ns, n)
    s = torch.ops.custom_esimd_kernels_vllm.esimd_gemv_int4.default._schema
    assert str(s) == ("custom_esimd_kernels_vllm::esimd_gemv_int4(Tensor input, Tensor weight, "
                      "Tensor weight_scale, Tensor output) -> Tensor")


def test_whole_reference_op_surface_is_registered(lib_built):
    """Every op name the reference package registers (93 over six namespaces) resolves here; the ones without an
    implementation fail with a clear message instead of being absent (callers probe with getattr(..., None))."""
    import torch
    import custom_esimd_kernels_vllm as pkg
    from custom_esimd_kernels_vllm._surface import UNIMPLEMENTED
    for ns in ("custom_esimd_kernels_vllm", "moe_ops", "moe_int4_ops", "moe_int4_prefill_ops", "esimd_topk_v2", "eagle_ops"):
        assert ns in pkg._register.REGISTERED, ns
    implemented = {(ns, n) for ns, names in pkg._register.IMPLEMENTED.items() for n in names}
    stubs = {(ns, s.split("(", 1)[0]) for ns, l in UNIMPLEMENTED.items() for s in l}
    assert not (implemented & stubs)
    assert len(implemented) + len(stubs) == 93, (len(implemented), len(stubs))
    for ns, n in implemented | stubs:
        assert getattr(getattr(torch.ops, ns), n, None) is not None, (ns, n)
    x = torch.zeros(2, 8, dtype=torch.float16)
    with pytest.raises(RuntimeError, match="b2q: custom_esimd_kernels_vllm::esimd_rms_norm not implemented"):
        torch.ops.custom_esimd_kernels_vllm.esimd_rms_norm(x, x, x[0], 1e-6)
    assert getattr(pkg.moe_ops, "moe_forward_full_v2", None) is not None


def test_cpp_op_library_loads_and_registers_the_dense_linears(lib_built):
    """libb2q_torch.so (csrc/torch_ops.cpp) carries the CUDA-key implementations of the dense linears; the Python
    registration leaves exactly those names to it.  No compute call here."""
    import torch
    import custom_esimd_kernels_vllm as pkg
    from custom_esimd_kernels_vllm import _register as R
    assert os.path.exists(R._CPP_PATH)
    assert R.CPP_OPS == {"esimd_gemv_int4", "esimd_gemm_int4_pgrp", "esimd_gemv_fp8_pern", "esimd_gemv_fp8_pert",
                         "esimd_gemv_fp8_pert_bmg", "esimd_gemm_fp8_pert", "esimd_gemm_fp8_blockscale"}
    for name in R.CPP_OPS:
        assert name in R.IMPLEMENTED["custom_esimd_kernels_vllm"]
        assert torch._C._dispatch_has_kernel_for_dispatch_key("custom_esimd_kernels_vllm::" + name, "CUDA")
    # a CPU tensor is refused by the dispatcher or by the op itself, never computed
    import pytest
    x = torch.zeros(1, 128, dtype=torch.bfloat16)
    with pytest.raises((RuntimeError, NotImplementedError)):
        torch.ops.custom_esimd_kernels_vllm.esimd_gemv_int4(x, torch.zeros(8, 64, dtype=torch.uint8), torch.zeros(8, 1, dtype=torch.bfloat16),
                                                            torch.zeros(1, 8, dtype=torch.bfloat16))


def _expert_layer(L, kind):
    """Arguments of a whole expert layer at addresses that nothing reads: every call below is refused, and refused before a launch."""
    at = iter(range(1 << 20, 1 << 30, 1 << 12))
    if kind == "fp8":
        a = L.MoeFp8(T=1, E=8, top_k=2, H=128, I=128)
        names = ("x", "logits", "w13", "s13", "w2", "s2", "out")
    else:
        a = L.MoeInt4(T=1, E=8, top_k=2, H=128, I=128, shared_I=128)
        names = ("x", "logits", "w13", "s13", "w2", "s2", "shared_w13", "shared_s13", "shared_w2", "shared_s2", "gate_w", "out")
    for n in names:
        setattr(a, n, next(at))
    call = getattr(L.lib, "b2q_moe_forward_" + kind)
    return a, lambda: call(a, 1 << 30, 1 << 30, None)


@pytest.mark.parametrize("kind,pointer", [("int4", n) for n in ("x", "out", "w13", "w2", "shared_w13", "shared_w2", "gate_w")]
                         + [("fp8", n) for n in ("x", "out", "w13", "w2")])
@pytest.mark.parametrize("off", [2, 8])
def test_expert_layers_refuse_what_is_not_aligned(lib_built, kind, pointer, off):
    from custom_esimd_kernels_vllm import _lib as L
    a, call = _expert_layer(L, kind)
    setattr(a, pointer, getattr(a, pointer) + off)
    before = L.launch_count()
    assert call() == -4 and L.launch_count() == before


@pytest.mark.parametrize("kind,field,value,code", [("int4", "s13_dtype", 3, -3), ("int4", "s2_dtype", -1, -3), ("int4", "shared_s13_dtype", 3, -3),
                                                   ("int4", "shared_s2_dtype", 7, -3), ("int4", "layout", 4, -5), ("int4", "shared_layout", -1, -5),
                                                   ("fp8", "fp8_format", 2, -3)])
def test_expert_layers_refuse_types_and_layouts_they_do_not_know(lib_built, kind, field, value, code):
    from custom_esimd_kernels_vllm import _lib as L
    a, call = _expert_layer(L, kind)
    setattr(a, field, value)
    before = L.launch_count()
    assert call() == code and L.launch_count() == before
