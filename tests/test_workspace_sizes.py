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
