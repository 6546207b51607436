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
    fused = T * k <= 1024 and E < 256
    e.set_force_kernel(2)                      # not the streaming kernel, whose gate_up rows are never rounded
    try:
        before = e.launch_count()
        out = e.moe_prefill_full_int4(x, logits, w13, s13, w2, s2, k, E)
        launches = e.launch_count() - before
        assert torch.equal(out, _int4_steps(e, x, logits, w13, s13, w2, s2, k, E, None))
    finally:
        e.set_force_kernel(0)
    assert launches == (6 if fused else 10)


def _dequant(w, s):
    q = torch.stack([(w >> (4 * i)) & 15 for i in range(8)], -1).reshape(*w.shape[:-1], -1).double() - 8
    return q * s.double().repeat_interleave(128, -1)


# Every stage rounds to 16 bits once (the gate_up product behind the activation, each expert's row, the sum): at most 2^-9 (bf16) or
# 2^-12 (fp16) of its value each, of which a few meet in an output; the 2-norm over a row sees their mean, about 1.5 of them.
@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 2.0 ** -8), (torch.float16, 2.0 ** -11)])
@pytest.mark.parametrize("T,E,k", [(1, 8, 2), (5, 32, 8), (16, 128, 8), (17, 4, 1), (64, 32, 4), (128, 64, 8)])
@pytest.mark.parametrize("shared", [0, 1])
def test_int4_streaming_kernel(e, dtype, tol, T, E, k, shared):
    """Tiles of eight tokens: fewer, exactly as many, one more per expert; experts without rows; the shared expert's tiles behind them, with its
    scales stored the other way round; an odd number of scale groups; strips of the gated form that overhang (I = 384: six halves)."""
    g = torch.Generator(device=DEV).manual_seed(T * E + k)
    H, Ii = 640, 384
    x = torch.randn(T, H, generator=g, device=DEV).to(dtype)
    logits = torch.randn(T, E, generator=g, device=DEV).to(dtype)
    (w13, s13), (w2, s2) = _int4(g, E, N=2 * Ii, K=H, dtype=dtype), _int4(g, E, N=H, K=Ii, dtype=dtype)
    (gu, gus), (dn, dns) = _int4(g, N=2 * Ii, K=H, dtype=dtype), _int4(g, N=H, K=Ii, dtype=dtype)
    gate = (torch.randn(1, H, generator=g, device=DEV) / H ** 0.5).to(dtype)
    e.set_force_kernel(7)
    try:
        before = e.launch_count()
        out = e.moe_forward_full_int4(x, logits, w13, s13, gu, gus.t().contiguous(), w2, s2, dn, dns.t().contiguous(), gate, k, shared, E, True)
        assert e.launch_count() - before == 4
    finally:
        e.set_force_kernel(0)
    wts, ids = e._impl.moe_topk(logits, k, True, weight_dtype=dtype)

    def mlp(rows, a, b):
        h = rows @ a.t()
        return (torch.nn.functional.silu(h[:, :Ii]) * h[:, Ii:]) @ b.t()

    xd, ref = x.double(), torch.zeros(T, H, dtype=torch.float64, device=DEV)
    for ex in range(E):
        t, s = (ids == ex).nonzero(as_tuple=True)
        if t.numel():
            ref.index_add_(0, t, wts[t, s].double().unsqueeze(1) * mlp(xd[t], _dequant(w13[ex], s13[ex]), _dequant(w2[ex], s2[ex])))
    if shared:
        ref += torch.sigmoid(xd @ gate.double().t()) * mlp(xd, _dequant(gu, gus), _dequant(dn, dns))
    err = (out.double() - ref).norm(dim=1) / ref.norm(dim=1)
    assert float(err.max()) < tol, float(err.max())
    assert e._lib.device_status() == 0


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
    for kernel in (2, 7):
        e.set_force_kernel(kernel)
        try:
            out = e.moe_prefill_full_int4(x, logits, w13, s13, w2, s2, k, E)
            ref = _int4_steps(e, x, logits, w13, s13, w2, s2, k, E, None)
        finally:
            e.set_force_kernel(0)
        assert torch.equal(out, ref) if kernel == 2 else torch.allclose(out, ref, rtol=1e-2, atol=1e-2)
        assert (out[2] == 0).all()


@pytest.mark.parametrize("native", [True, False])
def test_silu_mul_refuses_outputs_it_would_write_beyond(e, native):
    """The C++ op and the Python one behind it: the same outputs are taken and refused, with nothing launched for the latter."""
    from custom_esimd_kernels_vllm import _register as R
    from test_host_logic import _outputs
    op = torch.ops.custom_esimd_kernels_vllm.esimd_moe_silu_mul if native else R._moe_silu_mul
    x = torch.randn(6, 64, device=DEV).to(torch.bfloat16)
    ref = None
    for out, fits in _outputs(torch.bfloat16, DEV):
        before = e._lib.launch_count()
        if fits:
            got = op(x, out, 64, 32, 4).reshape(-1)[:128]
            ref = got if ref is None else ref
            assert torch.equal(got, ref) and e._lib.launch_count() == before + 1
        else:
            with pytest.raises((RuntimeError, NotImplementedError)):
                op(x, out, 64, 32, 4)
            assert e._lib.launch_count() == before
    for args in ((x, x[:, :32].contiguous(), 64, 32, -1), (x, x, 128, 64, 4)):
        with pytest.raises(RuntimeError):
            op(*args)
    assert op(x, torch.zeros(6, 32, dtype=torch.bfloat16, device=DEV), 64, 32, 100).shape == (6, 32)


@pytest.mark.parametrize("H", [640, 768, 1024])
def test_expert_decode_repeats_bit_for_bit(e, H):
    """Many launches of several short segments per CTA: stages that are handed back to the producer too early show as a row of one tile
    that differs now and then."""
    g = torch.Generator(device=DEV).manual_seed(H)
    T, E, k, Ii, dtype = 128, 64, 8, 384, torch.float16
    x, logits = torch.randn(T, H, generator=g, device=DEV).to(dtype), torch.randn(T, E, generator=g, device=DEV).to(dtype)
    (w13, s13), (w2, s2) = _int4(g, E, N=2 * Ii, K=H, dtype=dtype), _int4(g, E, N=H, K=Ii, dtype=dtype)
    (gu, gus), (dn, dns) = _int4(g, N=2 * Ii, K=H, dtype=dtype), _int4(g, N=H, K=Ii, dtype=dtype)
    gate = (torch.randn(1, H, generator=g, device=DEV) / H ** 0.5).to(dtype)
    gus, dns = gus.t().contiguous(), dns.t().contiguous()
    e.set_force_kernel(7)
    try:
        outs = [e.moe_forward_full_int4(x, logits, w13, s13, gu, gus, w2, s2, dn, dns, gate, k, 1, E, True) for _ in range(400)]
    finally:
        e.set_force_kernel(0)
    assert len({o.cpu().numpy().tobytes() for o in outs}) == 1
