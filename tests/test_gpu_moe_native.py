"""The native expert pipelines (b2q_moe_forward_int4 / _fp8) against the same steps taken one by one through the package's own functions,
which the other tests compare with the oracle: the routing launch for a few pairs at the edges of its range, both weight
orders, FP8 in both activation types, logits that leave no maximum.  The steps are the same arithmetic in the same order: results
agree bit for bit."""
import pytest
import torch

from gpu_util import DEV

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def e():
    import custom_esimd_kernels_vllm as pkg
    return pkg


def _int4(g, *lead, N, K, dtype):
    w = torch.randint(-2 ** 31, 2 ** 31, (*lead, N, K // 8), generator=g, device=DEV, dtype=torch.int64).to(torch.int32)
    s = ((0.5 + torch.rand(*lead, N, K // 128, generator=g, device=DEV)) / (4.6 * K ** 0.5)).to(dtype)
    return w, s


def _int4_steps(e, x, logits, w13, s13, w2, s2, k, E, layout):
    I, L, T = e._impl, e._lib, x.shape[0]
    wts, ids = I.moe_topk(logits, k, True, weight_dtype=x.dtype)
    off, tok, perm, _ = I.moe_route(ids, E)
    mid = I.moe_gemm_int4(x, w13, s13, off, T * k, row_map=tok, row_div=k, layout=layout)
    y = I.moe_gemm_int4(mid, w2, s2, off, T * k, act=L.ACT_SILU_MUL_IN, layout=layout)
    return I.moe_combine(y, wts, perm, T, k)


# pairs: one, a few, as many as the single launch sorts (1024) and one token more; experts: its most (255) and one more
@pytest.mark.parametrize("T,E,k", [(1, 8, 1), (3, 32, 8), (128, 64, 8), (129, 64, 8), (16, 255, 4), (16, 256, 4), (341, 33, 3), (40, 8, 8)])
@pytest.mark.parametrize("marlin", [False, True])
def test_int4(e, T, E, k, marlin):
    g = torch.Generator(device=DEV).manual_seed(T + E)
    H, Ii, dtype = 256, 128, torch.bfloat16
    x = torch.randn(T, H, generator=g, device=DEV).to(dtype)
    logits = torch.randn(T, E, generator=g, device=DEV).to(dtype)
    (w13, s13), (w2, s2) = _int4(g, E, N=2 * Ii, K=H, dtype=dtype), _int4(g, E, N=H, K=Ii, dtype=dtype)
    if marlin:
        w13, s13, w2, s2 = (t.transpose(1, 2).contiguous() for t in (w13, s13, w2, s2))
    before = e.launch_count()
    out = e.moe_prefill_full_int4(x, logits, w13, s13, w2, s2, k, E)
    launches = e.launch_count() - before
    ref = _int4_steps(e, x, logits, w13, s13, w2, s2, k, E, None)
    assert torch.equal(out, ref)
    fused = T * k <= 1024 and E < 256
    assert launches <= (7 if fused else 10)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,E,k", [(2, 64, 8), (257, 64, 4), (300, 8, 4)])
def test_fp8(e, dtype, T, E, k):
    g = torch.Generator(device=DEV).manual_seed(T)
    H, Ii, I = 256, 128, e._impl
    x = torch.randn(T, H, generator=g, device=DEV).to(dtype)
    logits = torch.randn(T, E, generator=g, device=DEV).to(dtype)
    w13 = (torch.randn(E, 2 * Ii, H, generator=g, device=DEV) * 64).clamp(-448, 448).to(torch.float8_e4m3fn)
    w2 = (torch.randn(E, H, Ii, generator=g, device=DEV) * 64).clamp(-448, 448).to(torch.float8_e4m3fn)
    s13, s2 = torch.rand(E, generator=g, device=DEV) * 1e-3, torch.rand(E, generator=g, device=DEV) * 1e-3
    out = e.moe_forward_full_gelu_tanh(x, logits, w13, s13, w2, s2, k, E)
    wts, ids = I.moe_topk(logits, k, True, weight_dtype=dtype)
    ref = e.moe_forward_full_gelu_tanh_routed(x, wts, ids, w13, s13, w2, s2, k, E)
    assert torch.equal(out, ref)


def test_logits_without_a_maximum_route_nowhere(e):
    g = torch.Generator(device=DEV).manual_seed(9)
    T, E, k, H, Ii, dtype = 5, 16, 2, 256, 128, torch.float16
    x = torch.randn(T, H, generator=g, device=DEV).to(dtype)
    logits = torch.randn(T, E, generator=g, device=DEV).to(dtype)
    logits[2] = float("nan")
    (w13, s13), (w2, s2) = _int4(g, E, N=2 * Ii, K=H, dtype=dtype), _int4(g, E, N=H, K=Ii, dtype=dtype)
    out = e.moe_prefill_full_int4(x, logits, w13, s13, w2, s2, k, E)
    assert torch.equal(out, _int4_steps(e, x, logits, w13, s13, w2, s2, k, E, None))
    assert (out[2] == 0).all()
