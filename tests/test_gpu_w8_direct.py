"""Strips of the FP8 decode GEMM (csrc/umma_w8_direct.cu), whole and cut along k."""
import pytest
import torch

from gpu_util import DEV

pytestmark = pytest.mark.gpu


@pytest.fixture()
def e():
    import custom_esimd_kernels_vllm as pkg
    return pkg


@pytest.mark.parametrize("M,N,K", [(17, 640, 7616), (33, 2048, 7680), (64, 9472, 7680), (24, 9473, 7680), (17, 4736, 7552), (40, 130, 16448), (64, 3000, 256)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_fp8_decode_path_whole_and_cut_strips(e, M, N, K, dtype):
    """The FP8 decode GEMM around the line where strips are cut along k (60 stages of 128, the last one ragged), with two, four and no
    pieces per strip and one or two CTAs per SM; without scratch for partial sums strips stay whole.  The terms are exact down to 2^-14 of a
    row's largest value and the sums fp32: the output's rounding remains, at most 2^-8 or 2^-11 of an element."""
    L = e._lib
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    w = (torch.randn(N, K, generator=g, device=DEV) * 96).clamp_(-448, 448).to(torch.float8_e4m3fn)
    s = (0.5 + torch.rand(N, generator=g, device=DEV)) / 4096
    x = torch.randn(M, K, generator=g, device=DEV).to(dtype)
    ref = x.double() @ (w.double() * s.double()[:, None]).T
    ws = torch.empty(L.lib.b2q_linear_fp8_workspace_bytes(M, N, K), dtype=torch.uint8, device=DEV)
    for _ in range(3):
        out = torch.full((M, N), float("nan"), dtype=dtype, device=DEV)
        L.check(L.lib.b2q_linear_fp8(x.data_ptr(), L.BF16 if dtype == torch.bfloat16 else L.F16, K, w.data_ptr(), L.E4M3, s.data_ptr(), L.F32,
                                     L.SCALE_CHANNEL, out.data_ptr(), N, M, N, K, ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream))
        assert e.last_kernel() == "umma_w8_direct"
        assert float((out.double() - ref).norm() / ref.norm()) <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11)
    assert L.device_status() == 0
