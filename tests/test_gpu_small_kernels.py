"""The small kernels between the linears at the edges of what a thread fetches at once: rows of a norm beyond what one pass of a CTA holds, many
rows, experts that leave a lane's last logits empty.  Against fp64; the output is rounded once, 2^-9 of an element in bf16, 2^-12 in
fp16, and the fp32 sums in front of it are exact to some 2^-18: twice the rounding in all."""
import pytest
import torch

from gpu_util import DEV

pytestmark = pytest.mark.gpu
TOL = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


@pytest.fixture(scope="module")
def impl():
    from custom_esimd_kernels_vllm import _impl
    return _impl


def _close(out, ref, dtype):
    err = (out.double() - ref).abs() - TOL[dtype] * ref.abs() - (2.0 ** -24 if dtype == torch.float16 else 0.0)
    assert float(err.max()) <= 0, float(err.max())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K", [(1, 8), (3, 1032), (700, 4096), (2, 8192), (5, 8200), (300, 16392), (16, 8192), (17, 8192), (16, 4104)])
def test_residual_norm(impl, dtype, M, K):
    g = torch.Generator(device=DEV).manual_seed(M + K)
    h, r, w, w2 = (torch.randn(*s, generator=g, device=DEV).to(dtype) for s in ((M, K), (M, K), (K,), (K,)))
    v = h.float() + r.float()
    n = v.double() * (v.double().pow(2).mean(1, keepdim=True) + 1e-6).rsqrt()
    res, out, out2 = r.clone(), torch.empty_like(r), torch.empty_like(r)
    impl.resadd_rmsnorm(h, res, w, out, 1e-6)
    assert torch.equal(res, v.to(dtype))
    _close(out, n * w.double(), dtype)
    v = r.double()
    n = v * (v.pow(2).mean(1, keepdim=True) + 1e-6).rsqrt()
    impl.rmsnorm_fused(None, r, 1.0, w, out, w2, out2, 1e-6)
    _close(out, n * w.double(), dtype)
    _close(out2, n * w2.double(), dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,V", [(1, 8), (3, 128), (5, 250), (700, 256), (2, 264), (9, 520)])
def test_gated_norm(impl, dtype, rows, V):
    g = torch.Generator(device=DEV).manual_seed(rows + V)
    x, z, w = (torch.randn(*s, generator=g, device=DEV).to(dtype) for s in ((rows, V), (rows, V), (V,)))
    xd, zd = x.double(), z.double()
    ref = xd * (xd.pow(2).mean(1, keepdim=True) + 1e-6).rsqrt() * w.double() * zd / (1 + (-zd).exp())
    _close(impl.gated_rmsnorm(x, z, w, 1e-6).view(rows, V), ref, dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("T,E,k", [(1, 1, 1), (3, 33, 5), (9, 100, 8), (300, 255, 6), (2, 512, 10), (5, 1000, 32)])
def test_topk_of_distinct_logits(impl, dtype, T, E, k):
    """Logits a sixteenth apart (in bf16 some are equal: the lowest index first), in any order: the same experts in the same order, weights as their softmax."""
    g = torch.Generator(device=DEV).manual_seed(T + E)
    order = torch.stack([torch.randperm(E, generator=g, device=DEV) for _ in range(T)])
    logits = ((order - E // 2) / 16.0).to(dtype)
    wts, ids = impl.moe_topk(logits, k, True, weight_dtype=torch.float32)
    ref = torch.sort(logits.double(), dim=1, descending=True, stable=True)
    assert torch.equal(ids.long(), ref.indices[:, :k])
    p = ref.values[:, :k].softmax(1)
    assert float(((wts.double() - p).abs() / p).max()) < 2.0 ** -16


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,H", [(1, 8), (149, 2048), (3, 8200), (256, 16384)])
def test_shared_gate(impl, dtype, T, H):
    """Fewer rows than SMs and more, behind kernels that write its inputs, several in a row on one stream."""
    g = torch.Generator(device=DEV).manual_seed(T + H)
    x, gate, sh, ro = (torch.randn(*s, generator=g, device=DEV).to(dtype) for s in ((T, H), (1, H), (T, H), (T, H)))
    gate /= H ** 0.5
    ref = ro.double() + torch.sigmoid(x.double() @ gate.double().T) * sh.double()
    for _ in range(3):
        buf = torch.empty_like(sh)
        impl.silu_mul(torch.cat([torch.full_like(sh, 30.0), sh / 30.0], 1), buf)      # silu(30) = 30 in either type
        a = (sh / 30.0).double() * 30.0
        out = impl.moe_shared_gate_add(x, gate, buf, ro)
        lim = TOL[dtype] * (ro.double().abs() + 2 * a.abs()) + 2.0 ** -20
        assert bool(((out.double() - (ref + torch.sigmoid(x.double() @ gate.double().T) * (a - sh.double()))).abs() <= lim).all())
