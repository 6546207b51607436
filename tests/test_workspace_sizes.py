"""What the dense linears ask for as scratch, and that less of it than that costs no more than the partial sums.  Sizes need
no device: the library assumes 148 SMs where it sees none."""
import pytest

SMS = 148


def _up(n):
    return (n + 255) // 256 * 256


def _prep(M, K):
    return _up(2 * M * K) + _up(4 * M)


@pytest.fixture(scope="module")
def lib(lib_built):
    from custom_esimd_kernels_vllm import _lib
    return _lib.lib


@pytest.mark.parametrize("M", [65, 100, 128, 129, 256, 4096])
@pytest.mark.parametrize("N,K", [(2048, 2048), (17408, 5120), (57344, 8192)])
def test_fp8_keeps_no_partial_sums_above_64_rows(lib, M, N, K):
    assert lib.b2q_linear_fp8_workspace_bytes(M, N, K) == _prep(M, K)


@pytest.mark.parametrize("M", [17, 33, 64, 65, 100, 128])
@pytest.mark.parametrize("N,K", [(128, 256), (1000, 1024), (2048, 2048), (2048, 28672), (8192, 14336), (57344, 8192)])
def test_int4_partial_sums_are_what_the_cut_can_use(lib, M, N, K):
    """At most two slots for every CTA that gets a raw stage of 256 k, each of the strip's rows x the token tile in fp32;
    256-row strips only where there is one for every SM."""
    tok = 32 if M <= 32 else (64 if M <= 64 else 128)
    rows = 256 if tok >= 64 and (N + 255) // 256 >= SMS else 128
    stages = (N + rows - 1) // rows * (K // 256)
    extra = lib.b2q_linear_workspace_bytes(M, N, K) - _prep(M, K)
    assert 0 <= extra <= 2 * min(SMS, stages) * rows * tok * 4


def test_int4_no_partial_sums_where_nothing_is_cut(lib):
    for M, N, K in ((64, 2048, 128 * 5),           # an odd number of scale groups
                    (64, 128 * SMS, 4096),         # a whole strip for every SM
                    (129, 2048, 2048)):            # two token tiles
        assert lib.b2q_linear_workspace_bytes(M, N, K) == _prep(M, K)


def test_int4_short_k_is_not_cut_for_128_token_tiles(lib):
    """Cutting costs a 128-token tile 4 us and 2 us per contributor, a stage of 256 k 0.8 us: up to K = 4096 no cut of less
    than one round of strips pays, and none ever has more pieces than stages or SMs."""
    for M in (65, 128):
        for N in (512, 2048, 4096, 12288):
            for K in (1024, 2048, 4096):
                assert lib.b2q_linear_workspace_bytes(M, N, K) == _prep(M, K)
        assert lib.b2q_linear_workspace_bytes(M, 4096, 14336) - _prep(M, 14336) == 2 * 4 * 32 * 128 * 128 * 4      # four equal pieces
        assert lib.b2q_linear_workspace_bytes(M, 8192, 28672) - _prep(M, 28672) == 2 * SMS * 128 * 128 * 4         # the whole grid


@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(4096, 4096), (8192, 28672), (57344, 8192)])
def test_int4_few_rows_ask_for_what_can_be_used(lib, M, N, K):
    """The pre-pass with two slots of 128 rows per SM behind it (K-major weights), or two slots of eight tokens for each of two CTAs per SM
    and four counts per strip; the int8 path's term rows only while that path is asked for."""
    most = max(_prep(M, K) + 2 * SMS * 128 * 16 * 4, 2 * 2 * SMS * 128 * 8 * 4 + (N + 127) // 128 * 4 * 8)
    assert _prep(M, K) <= lib.b2q_linear_workspace_bytes(M, N, K) <= most
    lib.b2q_set_force_kernel(5)
    try:
        assert lib.b2q_linear_workspace_bytes(M, N, K) > 4 << 20
    finally:
        lib.b2q_set_force_kernel(0)


@pytest.mark.parametrize("M", [1, 20, 64])
def test_fp8_partial_sums_of_cut_strips_are_one_slot_per_sm(lib, M):
    """Term rows in e4m3 (three per fp16 token, in the MMA's steps), scales, and [SMs][M in eights][128] fp32 with a count per strip."""
    rows = next(r for r in (16, 32, 64, 128, 256) if r >= 3 * ((M + 7) // 8 * 8))
    K = 13824
    assert lib.b2q_linear_fp8_workspace_bytes(M, 5120, K) <= max(_up(rows * K) + _up(4 * M) + SMS * ((M + 7) // 8 * 8) * 128 * 4 + SMS * 8,
                                                                 _prep(M, K) + 2 * SMS * 128 * 64 * 4)
