"""The persistent INT4 tcgen05 GEMM at the sizes where its division of work can go wrong: token-tile edges, ragged strips,
a scale-group count that fills no whole raw stage, strips cut between CTAs (several segments per CTA), tall strips, and
the three scale types through both ways of fetching them.

Tolerance, column by column in the 2-norm: the output is rounded to bf16 once (at most 2^-8 of an element: 8 significant
bits), and every weight (q - 8) * s to fp16 once (at most 2^-11, spread evenly: a standard deviation of 2^-11 / sqrt(3)
of a typical column, of which 2^-9 is seven).  One lost or repeated group of 128 k is an error of 1 / sqrt(K / 128) of a
typical column."""
import pytest
import torch

from gpu_util import DEV

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def e():
    import custom_esimd_kernels_vllm as pkg
    pkg.set_force_kernel(2)
    yield pkg
    pkg.set_force_kernel(0)


def _case(M, N, K, scale_dtype, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    w = torch.randint(-2 ** 31, 2 ** 31 - 1, (N, K // 8), generator=g, device=DEV, dtype=torch.int64).to(torch.int32)
    s = ((0.5 + torch.rand(N, K // 128, generator=g, device=DEV)) * 0.01).to(scale_dtype)
    x = torch.randn(M, K, generator=g, device=DEV).to(torch.bfloat16)
    shifts = torch.arange(0, 32, 4, device=DEV, dtype=torch.int32)
    q = ((w.unsqueeze(-1) >> shifts) & 15).reshape(N, K // 128, 128).double() - 8
    ref = x.double() @ (q * s.double().unsqueeze(-1)).view(N, K).T
    return x, w, s, ref


def _check(out, ref, what, rounding=2.0 ** -8):
    norms = ref.norm(dim=0)
    err = (out.double() - ref).norm(dim=0) / (rounding * norms + 2.0 ** -9 * norms.pow(2).mean().sqrt())
    assert float(err.max()) < 1.0, (what, float(err.max()), int(err.argmax()))       # also false for NaN


@pytest.mark.parametrize("scale_dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("M,N,K", [
    (1, 128, 128), (16, 136, 384), (17, 1000, 1024),     # one tile; ragged strip; odd group count; aligned scale fetch
    (33, 520, 2560), (64, 2048, 4096),                   # 64-token tile, cut strips
    (65, 300, 1280), (128, 1032, 2048),                  # 128-token tile, one of them
    (129, 384, 640), (400, 2184, 1152),                  # several token tiles, odd group counts
])
def test_tile_and_group_edges(e, M, N, K, scale_dtype):
    x, w, s, ref = _case(M, N, K, scale_dtype, M + N + K)
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
    e.esimd_gemm_int4_pgrp(x, w, s, out)
    assert e.last_kernel() == "umma_w4"
    _check(out, ref, (M, N, K))
    kmaj = torch.full_like(out, float("nan"))
    if N % 4 == 0:
        e.esimd_gemm_int4_pgrp(x, w.t().contiguous(), s.t().contiguous(), kmaj)
        assert e.last_kernel() == "umma_w4"
        _check(kmaj, ref, ("k-major", M, N, K))
    assert e._lib.device_status() == 0


@pytest.mark.parametrize("scale_dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("M,N,K", [(33, 520, 14336), (64, 2048, 14336)])
def test_cut_tile_edges(e, M, N, K, scale_dtype):
    """Long k, where cuts pay: the last strip ragged; without rest."""
    test_tile_and_group_edges(e, M, N, K, scale_dtype)


def test_the_strips_called_cut_are_cut(e):
    """Scratch beyond the pre-pass's part is asked for where strips are cut."""
    up = lambda n: (n + 255) // 256 * 256
    for M, N, K in ((33, 520, 14336), (64, 2048, 14336), (64, 8192, 14336), (64, 38016, 8192), (100, 4096, 14336), (128, 12288, 14336), (96, 520, 8192)):
        assert e._lib.lib.b2q_linear_workspace_bytes(M, N, K) > up(2 * M * K) + up(4 * M), (M, N, K)
    for M, N, K in ((17, 1032, 8192), (60, 1000, 14336)):
        tok = 32 if M <= 32 else 64
        assert e._lib.lib.b2q_linear_fp8_workspace_bytes(M, N, K) >= up(2 * M * K) + up(4 * M) + 2 * ((N + 127) // 128) * 128 * tok * 4, (M, N, K)


@pytest.mark.parametrize("M,N,K", [(16, 8192, 14336), (64, 8192, 14336), (64, 38016, 2048), (100, 10240, 8192), (700, 8192, 2048),
                                   (100, 4096, 14336), (128, 12288, 14336), (96, 520, 8192)])    # 128-token tiles cut into equal pieces, over the whole grid, ragged
def test_many_segments_repeat_bit_for_bit(e, M, N, K):
    x, w, s, ref = _case(M, N, K, torch.bfloat16, 7)
    first = None
    for _ in range(8):
        out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
        e.esimd_gemm_int4_pgrp(x, w, s, out)
        assert e.last_kernel() == "umma_w4"
        if first is None:
            first = out
            _check(out, ref, (M, N, K))
        assert torch.equal(out, first)
    assert e._lib.device_status() == 0


def test_many_cut_segments_of_256_rows_repeat_bit_for_bit(e):
    """Ragged strips of 256 rows, cut."""
    test_many_segments_repeat_bit_for_bit(e, 64, 38016, 8192)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(1, 128, 128), (16, 200, 384), (17, 1032, 640), (33, 2048, 1152), (64, 8192, 5120), (27, 17408, 5120)])
def test_block_scaled_fp8_strips(e, M, N, K, dtype):
    """The e4m3 form of the kernel: a weight times its fp32 block scale is rounded to fp16 once, as above; with fp16
    output the tolerance is 2^-11 for the output's rounding and the same 2^-9 of a typical column for the weights'."""
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    w = (torch.randn(N, K, generator=g, device=DEV) * 96).clamp_(-448, 448).to(torch.float8_e4m3fn)
    s = (0.5 + torch.rand((N + 127) // 128, K // 128, generator=g, device=DEV)) / 4096
    x = torch.randn(M, K, generator=g, device=DEV).to(dtype)
    full = s.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)
    ref = x.double() @ (w.double() * full).T
    first = None
    for _ in range(3):
        out = torch.full((M, N), float("nan"), dtype=dtype, device=DEV)
        e.esimd_gemm_fp8_blockscale(x, w, s, out)
        assert e.last_kernel() == "umma_w4"
        if first is None:
            first = out
            _check(out, ref, (M, N, K), 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11)
        assert torch.equal(out, first)
    assert e._lib.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(17, 1032, 8192), (60, 1000, 14336)])
def test_block_scaled_fp8_cut_strips(e, M, N, K, dtype):
    """The last of the cut strips ragged."""
    test_block_scaled_fp8_strips(e, M, N, K, dtype)


@pytest.mark.parametrize("rows", [(1, 0, 3, 16, 2), (40, 17, 0, 31, 33), (64, 65, 130, 1, 40)])
@pytest.mark.parametrize("N,K", [(256, 128), (1032, 1152)])
@pytest.mark.parametrize("channel", [False, True])
def test_grouped_fp8_scale_per_expert_or_channel(e, rows, N, K, channel):
    """Grouped e4m3 with one scale per expert or per output channel on fp16 activations: the weights are exact, so only the
    output's rounding (2^-11) and the fp32 sums remain; experts without rows, ragged strips, 16- / 32- / 64-token tiles."""
    E, M = len(rows), sum(rows)
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    w = (torch.randn(E, N, K, generator=g, device=DEV) * 96).clamp_(-448, 448).to(torch.float8_e4m3fn)
    s = (0.5 + torch.rand(*((E, N) if channel else (E,)), generator=g, device=DEV)) / 4096
    x = torch.randn(M, K, generator=g, device=DEV).to(torch.float16)
    off = torch.tensor([0] + list(rows), device=DEV).cumsum(0).to(torch.int32)
    ref = torch.cat([x[off[i]:off[i + 1]].double() @ (w[i].double() * s[i].double().reshape(-1, 1)).T for i in range(E)])
    out = torch.full((M, N), float("nan"), dtype=torch.float16, device=DEV)
    (e.esimd_moe_gemm_fp8 if channel else e.esimd_moe_gemm_fp8_pert)(x, w, s, out, off, N, K, E, M)
    assert e.last_kernel() == "umma_w4"
    err = (out.double() - ref).norm() / ref.norm()
    assert float(err) < 2.0 ** -11, float(err)
    assert e._lib.device_status() == 0


@pytest.mark.parametrize("E,avg,N,kernel", [(8, 40, 1024, "umma_w4"), (8, 80, 2048, "umma_wo"), (12, 40, 2000, "umma_wo"), (8, 60, 4096, "umma_w4"),
                                            (16, 24, 2048, "umma_w4")])
def test_grouped_fp8_route_by_rounds(e, E, avg, N, kernel):
    """64-token tiles in one round over the SMs, in two, in more, and 32-token tiles: which kernel serves them, and that both of
    them give the same product (tolerance as above)."""
    K = 512
    rows = [avg + (avg // 3 if i % 2 else -(avg // 3)) for i in range(E)]
    M = sum(rows)
    g = torch.Generator(device=DEV).manual_seed(M + N)
    w = (torch.randn(E, N, K, generator=g, device=DEV) * 96).clamp_(-448, 448).to(torch.float8_e4m3fn)
    s = (0.5 + torch.rand(E, generator=g, device=DEV)) / 4096
    x = torch.randn(M, K, generator=g, device=DEV).to(torch.float16)
    off = torch.tensor([0] + rows, device=DEV).cumsum(0).to(torch.int32)
    ref = torch.cat([x[off[i]:off[i + 1]].double() @ (w[i].double() * float(s[i])).T for i in range(E)])
    out = torch.full((M, N), float("nan"), dtype=torch.float16, device=DEV)
    e.esimd_moe_gemm_fp8_pert(x, w, s, out, off, N, K, E, M)
    assert e.last_kernel() == kernel
    err = (out.double() - ref).norm() / ref.norm()
    assert float(err) < 2.0 ** -11, float(err)
    assert e._lib.device_status() == 0


@pytest.mark.parametrize("M,N,K", [(100, 2048, 2048), (64, 2048, 4096), (100, 5120, 8192)])
def test_scratch_without_room_for_partial_sums_keeps_the_pre_pass(e, M, N, K):
    """Scratch that a caller sized for another M: the activations are rewritten as ever (two launches), strips stay whole.
    The sums differ from those of cut strips in their order alone, so both stay within the tolerance."""
    L = e._lib
    x, w, s, ref = _case(M, N, K, torch.bfloat16, 11)
    up = lambda n: (n + 255) // 256 * 256
    for size in (up(2 * M * K) + up(4 * M), 2 * (up(2 * M * K) + up(4 * M))):
        ws = torch.empty(size, dtype=torch.uint8, device=DEV)
        out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
        before = e.launch_count()
        L.check(L.lib.b2q_linear_int4(x.data_ptr(), L.BF16, K, w.data_ptr(), L.W4_NMAJOR, s.data_ptr(), L.BF16, K // 128, 1,
                                      out.data_ptr(), N, M, N, K, 128, ws.data_ptr(), size, torch.cuda.current_stream().cuda_stream))
        assert e.launch_count() - before == 2 and e.last_kernel() == "umma_w4"
        _check(out, ref, (M, N, K, size))
    assert e._lib.device_status() == 0


@pytest.mark.parametrize("M,kernel", [(33, "umma_w4"), (100, "umma_wo")])
def test_fp8_scratch_for_the_pre_pass_alone(e, M, kernel):
    """Block-scaled FP8, the same: bf16 activations are rewritten with scratch that holds nothing else."""
    N, K = 2048, 2048
    L = e._lib
    g = torch.Generator(device=DEV).manual_seed(M)
    w = (torch.randn(N, K, generator=g, device=DEV) * 96).clamp_(-448, 448).to(torch.float8_e4m3fn)
    s = (0.5 + torch.rand(N // 128, K // 128, generator=g, device=DEV)) / 4096
    x = torch.randn(M, K, generator=g, device=DEV).to(torch.bfloat16)
    ref = x.double() @ (w.double() * s.double().repeat_interleave(128, 0).repeat_interleave(128, 1)).T
    size = (2 * M * K + 255) // 256 * 256 + (4 * M + 255) // 256 * 256
    ws = torch.empty(size, dtype=torch.uint8, device=DEV)
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
    before = e.launch_count()
    L.check(L.lib.b2q_linear_fp8(x.data_ptr(), L.BF16, K, w.data_ptr(), L.E4M3, s.data_ptr(), L.F32, L.SCALE_BLOCK128, out.data_ptr(), N, M, N, K,
                                 ws.data_ptr(), size, torch.cuda.current_stream().cuda_stream))
    assert e.launch_count() - before == 2 and e.last_kernel() == kernel
    _check(out, ref, M)
    assert e._lib.device_status() == 0


@pytest.mark.parametrize("M,N,K", [(65, 16392, 384), (128, 4104, 1152), (129, 1096, 2048), (300, 1000, 1152), (385, 4680, 640)])
@pytest.mark.parametrize("mode", ["block", "channel", "tensor"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_fp8_dense_above_64_tokens_strips(e, M, N, K, mode, dtype):
    """Dense e4m3 in 128-token tiles: ragged last tiles of tokens and strips, odd counts of 128-wide chunks of k, every scale mode, both activation
    types (bf16 ones are rewritten first).  The output is rounded once, at most 2^-8 (bf16) or 2^-11 (fp16) of each element, and
    spread evenly below 0.58 of that in the 2-norm; so are weights times their block scale, at most 2^-11: together below 2^-8 and 2^-10."""
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    w = (torch.randn(N, K, generator=g, device=DEV) * 96).clamp_(-448, 448).to(torch.float8_e4m3fn)
    x = torch.randn(M, K, generator=g, device=DEV).to(dtype)
    shape = {"block": ((N + 127) // 128, K // 128), "channel": (N,), "tensor": (1,)}[mode]
    s = (0.5 + torch.rand(*shape, generator=g, device=DEV)) / 4096
    full = s.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1) if mode == "block" else s.double().reshape(-1, 1)
    ref = x.double() @ (w.double() * full).T
    sm = {"block": e._lib.SCALE_BLOCK128, "channel": e._lib.SCALE_CHANNEL, "tensor": e._lib.SCALE_TENSOR}[mode]
    L = e._lib
    need = L.lib.b2q_linear_fp8_workspace_bytes(M, N, K)
    ws = torch.empty(max(need, 1), dtype=torch.uint8, device=DEV)
    out = torch.full((M, N), float("nan"), dtype=dtype, device=DEV)
    code = L.BF16 if dtype == torch.bfloat16 else L.F16
    L.check(L.lib.b2q_linear_fp8(x.data_ptr(), code, K, w.data_ptr(), L.E4M3, s.data_ptr(), L.F32, sm, out.data_ptr(), N, M, N, K,
                                 ws.data_ptr(), need, torch.cuda.current_stream().cuda_stream))
    assert e.last_kernel() == "umma_w4"
    assert float((out.double() - ref).norm() / ref.norm()) < (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -10)
    assert e._lib.device_status() == 0


@pytest.mark.parametrize("M,N,K,mode,kernel", [(217, 16422, 640, "block", "umma_wo"), (217, 16424, 640, "block", "umma_w4"), (1611, 1890, 768, "tensor", "umma_wo"),
                                               (1611, 1896, 768, "tensor", "umma_w4"), (151, 12072, 256, "tensor", "umma_wo")])
def test_fp8_dense_above_64_tokens_short_k_route_by_alignment(e, M, N, K, mode, kernel):
    """Rows of output that are not 16-byte aligned, and their aligned neighbours (tolerance as above)."""
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    w = (torch.randn(N, K, generator=g, device=DEV) * 96).clamp_(-448, 448).to(torch.float8_e4m3fn)
    x = torch.randn(M, K, generator=g, device=DEV).to(torch.bfloat16)
    s = (0.5 + torch.rand(*(((N + 127) // 128, K // 128) if mode == "block" else (1,)), generator=g, device=DEV)) / 4096
    full = s.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1) if mode == "block" else s.double()
    ref = x.double() @ (w.double() * full).T
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
    if mode == "block":
        e.esimd_gemm_fp8_blockscale(x, w, s, out)
    else:
        e.esimd_gemm_fp8_pert(x, w, s, out)
    assert e.last_kernel() == kernel
    assert float((out.double() - ref).norm() / ref.norm()) < 2.0 ** -8
    assert e._lib.device_status() == 0


@pytest.mark.parametrize("E,rows,N,K", [
    (3, (60, 0, 33), 1096, 640),                       # 64-token tiles, short strips: few pieces
    (2, (129, 200), 520, 1152),                        # 128-token tiles, short strips
    (64, (1, 40, 65, 54), 2048, 256),                  # 64-token tiles, tall strips: many rounds
    (16, (97, 128, 1, 160), 3072, 4096),               # 128-token tiles, tall strips: long k
    (80, (1, 16, 7, 3), 8192, 128),                    # more pieces per CTA than the table of tiles holds
])
def test_grouped_int4_strip_heights(e, E, rows, N, K):
    """Grouped INT4 over the strip heights and tile sizes it chooses between.  fp16 throughout: the output is rounded once (at
    most 2^-11 of it) and every weight once (at most 2^-11, spread evenly), together below 2^-10 in the 2-norm; one lost tile
    of n is 1 / sqrt(n)."""
    from custom_esimd_kernels_vllm import _impl
    rows = [rows[i % len(rows)] for i in range(E)]
    M = sum(rows)
    g = torch.Generator(device=DEV).manual_seed(E + N + K)
    w = torch.randint(-2 ** 31, 2 ** 31 - 1, (E, N, K // 8), generator=g, device=DEV, dtype=torch.int64).to(torch.int32)
    s = ((0.5 + torch.rand(E, N, K // 128, generator=g, device=DEV)) * 0.01).to(torch.float16)
    x = torch.randn(M, K, generator=g, device=DEV).to(torch.float16)
    off = torch.tensor([0] + rows, device=DEV).cumsum(0).to(torch.int32)
    shifts = torch.arange(0, 32, 4, device=DEV, dtype=torch.int32)
    parts = []
    for i in range(E):
        q = ((w[i].unsqueeze(-1) >> shifts) & 15).reshape(N, K // 128, 128).double() - 8
        parts.append(x[off[i]:off[i + 1]].double() @ (q * s[i].double().unsqueeze(-1)).view(N, K).T)
    ref = torch.cat(parts)
    out = _impl.moe_gemm_int4(x, w, s, off, M)
    assert e.last_kernel() == "umma_w4"
    err = (out.double() - ref).norm() / ref.norm()
    assert float(err) < 2.0 ** -10, float(err)
    assert e._lib.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M", [16, 64, 300])
@pytest.mark.parametrize("unit,spread", [(1e3, 0), (1e-6, 0), (1e-8, 0), (1e-3, 24), (300.0, 24)])
def test_block_scales_outside_fp16_range(e, dtype, M, unit, spread):
    """Block scales whose product with an e4m3 value overflows fp16 or falls among its subnormals, and scales up to 2^24 apart in one
    row, an all but vanishing one first: weights are rounded to fp16 once, relative to the largest block of their strip.
    The activations keep the output within fp16's range; the tolerance is that of the other block-scaled cases."""
    N, K = 520, 1152
    g = torch.Generator(device=DEV).manual_seed(M + spread)
    w = (torch.randn(N, K, generator=g, device=DEV) * 96).clamp_(-448, 448).to(torch.float8_e4m3fn)
    s = (0.5 + torch.rand((N + 127) // 128, K // 128, generator=g, device=DEV)) * unit
    if spread:
        s = s * torch.exp2(-torch.randint(0, spread + 1, s.shape, generator=g, device=DEV).float())
        s[:, 0] = 1e-20
        s[:, 3] = unit
    x = (torch.randn(M, K, generator=g, device=DEV) * min(2.0 ** 11, 2.0 ** -11 / unit)).to(dtype)
    full = s.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)
    ref = x.double() @ (w.double() * full).T
    out = torch.full((M, N), float("nan"), dtype=dtype, device=DEV)
    e.esimd_gemm_fp8_blockscale(x, w, s, out)
    _check(out, ref, (M, unit, spread), 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11)
    assert e._lib.device_status() == 0


@pytest.mark.parametrize("unit", [1e3, 1e-8])
def test_grouped_block_scales_outside_fp16_range(e, unit):
    E, rows, N, K = 2, (40, 90), 256, 512
    g = torch.Generator(device=DEV).manual_seed(3)
    w = (torch.randn(E, N, K, generator=g, device=DEV) * 96).clamp_(-448, 448).to(torch.float8_e4m3fn)
    s = (0.5 + torch.rand(E, N // 128, K // 128, generator=g, device=DEV)) * unit
    x = (torch.randn(sum(rows), K, generator=g, device=DEV) * min(2.0 ** 11, 2.0 ** -11 / unit)).to(torch.float16)
    off = torch.tensor([0, rows[0], sum(rows)], dtype=torch.int32, device=DEV)
    full = s.double().repeat_interleave(128, 1).repeat_interleave(128, 2)
    ref = torch.cat([x[off[i]:off[i + 1]].double() @ (w[i].double() * full[i]).T for i in range(E)])
    out = torch.full((sum(rows), N), float("nan"), dtype=torch.float16, device=DEV)
    e.esimd_moe_gemm_fp8_blockscale(x, w, s, out, off, N, K, E)
    _check(out, ref, unit, 2.0 ** -11)
    assert e._lib.device_status() == 0
