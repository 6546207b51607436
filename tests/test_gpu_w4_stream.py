"""The INT4 decode streaming kernel (csrc/w4_stream.cu) at the edges of its range: ragged strips, odd numbers of scale groups, stages beyond
K, cut and whole strips, scale types and strides, both nibble encodings, infinities and NaN."""
import pytest
import torch

from gpu_util import DEV

pytestmark = pytest.mark.gpu
TOL = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}      # one rounding of the result, over its largest value; fp32 sums add 1e-6


@pytest.fixture()
def e():
    import custom_esimd_kernels_vllm as pkg
    pkg.set_force_kernel(7)
    yield pkg
    pkg.set_force_kernel(0)
    pkg.set_overlap_mode(1)


def _inputs(M, N, K, dtype, sdtype, seed=0):
    g = torch.Generator().manual_seed(seed)
    q = torch.randint(0, 16, (N, K), generator=g, dtype=torch.uint8)
    w = sum(q[:, j::8].to(torch.int64) << (4 * j) for j in range(8))
    w = torch.where(w >= 2 ** 31, w - 2 ** 32, w).to(torch.int32)
    s = ((0.5 + torch.rand(N, K // 128, generator=g)) / (4.6 * K ** 0.5)).to(sdtype)
    x = torch.randn(M, K, generator=g).to(dtype)
    return x, q, w, s


def _exact(x, q, s):
    return x.double() @ ((q.double() - 8) * s.double().repeat_interleave(128, 1)).t()


def _close(out, ref, dtype):
    err = (out.cpu().double() - ref).abs().max() / ref.abs().max()
    assert err <= TOL[dtype] + 2e-6, float(err)


@pytest.mark.parametrize("M", [1, 3, 8])
@pytest.mark.parametrize("N,K", [(1, 128), (100, 256), (127, 384), (129, 1024), (4104, 1152), (300, 4096), (40000, 256)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_shapes(e, M, N, K, dtype):
    """N below, at and above a strip of 128; K of one group, of odd groups (half a stage beyond K), of several scale slots; cut and whole."""
    x, q, w, s = _inputs(M, N, K, dtype, dtype)
    out = torch.empty(M, N, dtype=dtype, device=DEV)
    e.esimd_gemm_int4_pgrp(x.to(DEV), w.to(DEV), s.to(DEV), out)
    assert e.last_kernel() == "w4_stream"
    _close(out, _exact(x, q, s), dtype)
    assert e._lib.device_status() == 0


@pytest.mark.parametrize("sdtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("K", [128 * 3, 128 * 6, 128 * 16])       # element, 4-byte and 16-byte fetches of the scales
def test_scales(e, sdtype, transposed, K):
    x, q, w, s = _inputs(5, 260, K, torch.float16, sdtype)
    sd = s.t().contiguous().to(DEV).t() if transposed else s.to(DEV)
    out = torch.empty(5, 260, dtype=torch.float16, device=DEV)
    e.esimd_gemm_int4_pgrp(x.to(DEV), w.to(DEV), sd, out)
    assert e.last_kernel() == "w4_stream"
    _close(out, _exact(x, q, s), torch.float16)


@pytest.mark.parametrize("M,N,K", [(8, 2048, 2048), (1, 57344, 512)])
def test_overlap_and_repeats_give_the_same_bits(e, M, N, K):
    """Cut strips are summed in CTA order whoever comes last; no mode of overlap changes a bit."""
    x, q, w, s = _inputs(M, N, K, torch.bfloat16, torch.bfloat16)
    xd, wd, sd = x.to(DEV), w.to(DEV), s.to(DEV)
    outs = []
    for mode in (0, 1, 2):
        e.set_overlap_mode(mode)
        for _ in range(20):
            out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
            e.esimd_gemm_int4_pgrp(xd, wd, sd, out)
            outs.append(out)
    torch.cuda.synchronize()
    assert all(torch.equal(outs[0], o) for o in outs[1:])
    _close(outs[0], _exact(x, q, s), torch.bfloat16)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_infinities_and_nan_come_out_as_their_products(e, dtype):
    x, q, w, s = _inputs(4, 256, 512, dtype, dtype)
    x[0, 5], x[1, 300], x[2, 511] = float("inf"), float("nan"), float("-inf")
    out = torch.empty(4, 256, dtype=dtype, device=DEV)
    e.esimd_gemm_int4_pgrp(x.to(DEV), w.to(DEV), s.to(DEV), out)
    o = out.cpu().double()
    ref = _exact(x, q, s)
    assert torch.equal(o.isnan(), ref.isnan())
    assert torch.equal(torch.sign(o[:3].nan_to_num(0)), torch.sign(ref[:3].nan_to_num(0)))
    _close(out[3:], ref[3:], dtype)


def test_dispatch_takes_it_where_the_other_kernel_needs_more_rounds(e):
    e.set_force_kernel(0)
    for M, N, K, name in ((8, 8192, 4096, "w4_stream"), (8, 4096, 4096, "smallm"), (1, 5888, 5888, "smallm"), (1, 7168, 5888, "w4_stream"), (1, 2048, 12288, "w4_stream"),
                          (9, 8192, 8192, "umma_w4")):
        x, q, w, s = _inputs(M, N, K, torch.bfloat16, torch.bfloat16)
        out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
        e.esimd_gemm_int4_pgrp(x.to(DEV), w.to(DEV), s.to(DEV), out)
        assert e.last_kernel() == name


def test_dispatch_counts_the_sums_of_strips_cut_into_many_pieces(e):
    """Few rows and long k: some thirty contributors to a strip cost more than the other kernel's one round takes."""
    e.set_force_kernel(0)
    for M, N, K, name in ((1, 1024, 8192, "smallm"), (8, 512, 8192, "smallm"), (1, 256, 16384, "smallm"), (7, 2128, 8832, "smallm"), (1, 1024, 16384, "w4_stream"), (4, 512, 28672, "w4_stream")):
        x, q, w, s = _inputs(M, N, K, torch.bfloat16, torch.bfloat16)
        out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
        e.esimd_gemm_int4_pgrp(x.to(DEV), w.to(DEV), s.to(DEV), out)
        assert e.last_kernel() == name, (M, N, K)
        _close(out, _exact(x, q, s), torch.bfloat16)


def test_without_room_for_partial_sums_the_other_kernel_takes_strips_that_should_be_cut(e):
    """Scratch is the caller's choice in the C ABI: none, less than asked for, unaligned.  37888 x 1024 is whole strips in any case, and so
    many strips as 24576 x 4096 has are better off whole than there."""
    L = e._lib
    for M, N, K, without in ((1, 2048, 16384, "smallm"), (8, 8192, 8192, "smallm"), (1, 37888, 1024, "w4_stream"), (1, 24576, 4096, "w4_stream")):
        x, q, w, s = _inputs(M, N, K, torch.bfloat16, torch.bfloat16)
        x, wd, sd = x.to(DEV), w.to(DEV), s.to(DEV)
        need = L.lib.b2q_linear_workspace_bytes(M, N, K)
        ws = torch.empty(need + 16, dtype=torch.uint8, device=DEV)
        outs = []
        e.set_force_kernel(0)
        for ptr, size, room in ((ws.data_ptr(), need, True), (None, 0, False), (ws.data_ptr(), 4096, False), (ws.data_ptr() + 8, need, False)):
            out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
            rc = L.lib.b2q_linear_int4(x.data_ptr(), L.BF16, K, wd.data_ptr(), L.W4_NMAJOR, sd.data_ptr(), L.BF16, K // 128, 1, out.data_ptr(), N, M, N, K, 128,
                                       ptr, size, torch.cuda.current_stream().cuda_stream)
            assert rc == 0 and e.last_kernel() == ("w4_stream" if room else without), (N, K, size)
            outs.append(out)
        for out in outs:
            _close(out, _exact(x.cpu(), q, s), torch.bfloat16)


@pytest.mark.parametrize("K", [1024, 512, 768])
def test_a_stage_is_read_before_it_is_overwritten(e, K):
    """Three strips per CTA, a nibble of its own for each, and tokens that each see one group: what a stage loses to the copy that follows it,
    in whichever of many launches, is another strip's value.  (Whole strips: no scratch.)"""
    L = e._lib
    per = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    N, G = per * 3 * 128, K // 128
    nib = (torch.arange(per * 3, device=DEV) // per * 4 + 3).repeat_interleave(128)
    word = sum(nib << (4 * j) for j in range(8))
    w = torch.where(word >= 2 ** 31, word - 2 ** 32, word).to(torch.int32)[:, None].expand(N, K // 8).contiguous()
    s, x = torch.ones(N, G, device=DEV, dtype=torch.float16), torch.zeros(G, K, device=DEV, dtype=torch.float16)
    for m in range(G):
        x[m, m * 128:(m + 1) * 128] = 1
    ref = ((nib - 8) * 128).to(torch.float16).expand(G, N)
    out = torch.empty(G, N, device=DEV, dtype=torch.float16)
    wrong = 0
    for _ in range(500):
        assert L.lib.b2q_linear_int4(x.data_ptr(), L.F16, K, w.data_ptr(), L.W4_NMAJOR, s.data_ptr(), L.F16, G, 1, out.data_ptr(), N, G, N, K, 128, None, 0,
                                     torch.cuda.current_stream().cuda_stream) == 0
        wrong += not torch.equal(out, ref)
    assert e.last_kernel() == "w4_stream" and wrong == 0
