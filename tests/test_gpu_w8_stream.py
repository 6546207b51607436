"""The FP8 streaming kernel of up to sixteen tokens (csrc/w8_stream.cu) at the edges of its range: every height of a pass and two passes,
k beyond the last window, both token tiles, formats and scales, infinities and NaN, and the line of its dispatch."""
import pytest
import torch

from gpu_util import DEV

pytestmark = pytest.mark.gpu
# The weights and activations are exact and every sum is fp32: only the output's rounding remains, of each element at most
TOL = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}
SMS = 148


@pytest.fixture()
def e():
    import custom_esimd_kernels_vllm as pkg
    pkg.set_force_kernel(8)
    yield pkg
    pkg.set_force_kernel(0)
    pkg.set_overlap_mode(1)


def _inputs(M, N, K, dtype, mode, fmt=torch.float8_e4m3fn):
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    w = (torch.randn(N, K, generator=g, device=DEV) * 96).clamp_(-448, 448).to(fmt)
    shape = {"block": ((N + 127) // 128, K // 128), "channel": (N,), "tensor": (1,)}[mode]
    s = (0.5 + torch.rand(*shape, generator=g, device=DEV)) / 4096
    return torch.randn(M, K, generator=g, device=DEV).to(dtype), w, s


def _linear(e, x, w, s, mode, ws=None):
    L = e._lib
    (M, K), N = x.shape, w.shape[0]
    out = torch.full((M, N), float("nan"), dtype=x.dtype, device=DEV)
    sm = {"block": L.SCALE_BLOCK128, "channel": L.SCALE_CHANNEL, "tensor": L.SCALE_TENSOR}[mode]
    L.check(L.lib.b2q_linear_fp8(x.data_ptr(), L.BF16 if x.dtype == torch.bfloat16 else L.F16, x.stride(0), w.data_ptr(),
                                 L.E4M3 if w.dtype == torch.float8_e4m3fn else L.E5M2, s.data_ptr(), L.F32, sm, out.data_ptr(), N, M, N, K,
                                 ws.data_ptr() if ws is not None else None, ws.numel() if ws is not None else 0,
                                 torch.cuda.current_stream().cuda_stream))
    return out


def _exact(x, w, s, mode):
    full = s.double().repeat_interleave(128, 0)[:w.shape[0]].repeat_interleave(128, 1) if mode == "block" else s.double().reshape(-1, 1)
    return x.double() @ (w.double() * full).T


def _close(out, ref):
    err = float((out.double() - ref).abs().max() / ref.abs().max())
    assert err <= TOL[out.dtype] + 2e-6, err


# rows per CTA: 1 to 16 on one CTA per SM, 17 to 64 on two, then two passes; ragged in every one
@pytest.mark.parametrize("N", [1, 9, SMS * 13 + 5, SMS * 2 * 20 + 7, SMS * 2 * 30 + 1, SMS * 2 * 37 + 3, SMS * 2 * 46 + 9, SMS * 2 * 52, SMS * 2 * 64 + 1])
@pytest.mark.parametrize("K", [128, 640, 1152])
@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("dtype,mode", [(torch.bfloat16, "block"), (torch.bfloat16, "tensor"), (torch.float16, "block"), (torch.float16, "channel")])
def test_shapes(e, M, N, K, dtype, mode):
    x, w, s = _inputs(M, N, K, dtype, mode)
    out = _linear(e, x, w, s, mode)
    assert e.last_kernel() == "w8_stream"
    _close(out, _exact(x, w, s, mode))
    assert e._lib.device_status() == 0


@pytest.mark.parametrize("K", [16, 48, 528, 1040])                # any multiple of 16, odd numbers of lanes' sixteen k
@pytest.mark.parametrize("fmt", [torch.float8_e4m3fn, torch.float8_e5m2])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_k_tails_formats_and_row_strides(e, K, fmt, dtype):
    x, w, s = _inputs(5, 2050, K, dtype, "channel", fmt)
    wide = torch.full((5, K + 24), float("inf"), dtype=dtype, device=DEV)        # what lies behind a row must not be read into the sum
    wide[:, :K] = x
    out = _linear(e, wide[:, :K], w, s, "channel")
    assert e.last_kernel() == "w8_stream"
    _close(out, _exact(x, w, s, "channel"))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_extremes_infinities_and_nan_come_out_as_their_products(e, dtype):
    x, w, s = _inputs(12, 300, 640, dtype, "channel")
    x[0, 5], x[1, 300], x[9, 639] = float("inf"), float("nan"), float("-inf")
    x[2] *= 2.0 ** -14                                             # small next to its neighbours, subnormal in part in fp16
    w.view(torch.uint8)[7, 130], w.view(torch.uint8)[299, 639] = 0x7F, 0xFF       # NaN codes
    out, ref = _linear(e, x, w, s, "channel").double(), _exact(x, w, s, "channel")
    assert torch.equal(out.isnan(), ref.isnan())
    fin = ref.isfinite()
    assert torch.equal(torch.sign(out[~fin].nan_to_num(0)), torch.sign(ref[~fin].nan_to_num(0)))
    for m in (2, 3, 11):
        f = fin[m]
        assert float((out[m][f] - ref[m][f]).abs().max() / ref[m][f].abs().max()) <= TOL[dtype] + (2.0 ** -12 if m == 2 else 2e-6)


@pytest.mark.parametrize("mode", ["block", "tensor"])
def test_overlap_and_repeats_give_the_same_bits(e, mode):
    x, w, s = _inputs(8, 5120, 1152, torch.bfloat16, mode)
    outs = []
    for m in (0, 1, 2):
        e.set_overlap_mode(m)
        outs += [_linear(e, x, w, s, mode) for _ in range(20)]
    torch.cuda.synchronize()
    assert all(torch.equal(outs[0], o) for o in outs[1:])


@pytest.mark.parametrize("M,N,K,dtype,mode,stream", [
    (1, 4096, 1024, torch.bfloat16, "tensor", True), (1, 4096, 1008, torch.bfloat16, "tensor", False),
    (16, 9472, 512, torch.bfloat16, "channel", True), (16, 9473, 512, torch.bfloat16, "channel", False), (9, 4735, 2064, torch.bfloat16, "tensor", True), (9, 4736, 2064, torch.bfloat16, "tensor", False),
    (8, 3072, 8208, torch.bfloat16, "tensor", False), (4, 3072, 8208, torch.bfloat16, "tensor", True), (8, 9473, 512, torch.bfloat16, "channel", True),
    (8, 18945, 512, torch.bfloat16, "channel", False), (8, 9473, 6160, torch.bfloat16, "channel", False), (16, 9473, 512, torch.float16, "channel", True),
    (8, 18945, 3552, torch.float16, "tensor", True), (8, 18945, 3536, torch.float16, "tensor", False),
    (16, 18944, 512, torch.float16, "tensor", True), (16, 18945, 512, torch.float16, "tensor", False), (17, 4096, 1024, torch.float16, "tensor", False),
    (1, 5120, 8192, torch.bfloat16, "block", True), (1, 5120, 8320, torch.bfloat16, "block", False), (8, 9473, 4096, torch.bfloat16, "block", True),
    (8, 9473, 4224, torch.bfloat16, "block", False), (8, 9473, 6144, torch.float16, "block", True), (9, 9472, 4096, torch.bfloat16, "block", True),
    (9, 4736, 1024, torch.float16, "block", False), (9, 4735, 1024, torch.float16, "block", True), (16, 22528, 512, torch.bfloat16, "block", False)])
def test_both_sides_of_the_dispatch_agree(e, M, N, K, dtype, mode, stream):
    """Which calls it takes by itself; those and their neighbours give the product on either kernel, with scratch or without."""
    e.set_force_kernel(0)
    x, w, s = _inputs(M, N, K, dtype, mode)
    ref = _exact(x, w, s, mode)
    ws = torch.empty(e._lib.lib.b2q_linear_fp8_workspace_bytes(M, N, K), dtype=torch.uint8, device=DEV)
    out = _linear(e, x, w, s, mode, ws)
    assert (e.last_kernel() == "w8_stream") == stream
    # the other kernels round weights times their block scale to fp16 or bf16, at most 2^-11 or 2^-9 of each product
    slack = 1.0 if stream else 2.0
    assert float((out.double() - ref).norm() / ref.norm()) <= slack * TOL[dtype]
    out = _linear(e, x, w, s, mode)
    assert float((out.double() - ref).norm() / ref.norm()) <= slack * TOL[dtype]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K", [(1, 4096), (3, 5120), (16, 13824), (2, 264)])
def test_norm_in_front(e, M, K, dtype):
    """Residual add and RMSNorm in front of it: rows that fit a thread's registers and longer ones, against the formulas in fp64."""
    x, w, s = _inputs(M, 1040, K - K % 16, dtype, "tensor")
    K = x.shape[1]
    g = torch.Generator(device=DEV).manual_seed(K)
    res, nw = torch.randn(M, K, generator=g, device=DEV).to(dtype), (1 + 0.1 * torch.randn(K, generator=g, device=DEV)).to(dtype)
    res0, out, normed = res.clone(), torch.empty(M, 1040, dtype=dtype, device=DEV), torch.empty_like(x)
    e.esimd_resadd_norm_gemv_fp8_pert(x, res, nw, w, s, out, normed, 1e-6)
    assert e.last_kernel() == "w8_stream"
    v = x.double() + res0.double()
    assert torch.equal(res, (x.float() + res0.float()).to(dtype))
    n = v * torch.rsqrt(v.pow(2).mean(1, keepdim=True) + 1e-6) * nw.double()
    assert float(((normed.double() - n) / n.abs().clamp_min(1e-3)).abs().max()) <= 1.1 * TOL[dtype]
    _close(out, _exact(normed, w, s, "tensor"))
