"""Host-side rules of the batched GEMMs that need no GPU: how many kernels a call launches and the workspace that it is given."""
import pytest

from crownest_b200 import CN_BF16, CN_F32, lib, ops


@pytest.mark.parametrize("rows,k,m,bf16,f32,relaid_bf16,relaid_f32", [
    (17408, 5120, 64, 2, 2, 2, 2),    # 68 row tiles fill the 74 pairs: rows into f16 (or the cascade) and the GEMM
    (5120, 17408, 64, 3, 3, 3, 3),    # 20 row tiles: K is split and a third kernel adds the parts
    (17408, 5120, 512, 1, 2, 1, 2),   # bf16 rows as they are
    (40000, 512, 20, 2, 2, 2, 2),
    (1024, 10240, 512, 2, 3, 2, 3),
    (1024, 10240, 513, 1, 2, 1, 3),   # the pair kernel does not split K beyond 512 rows
    (1024, 100, 64, 0, 0, 0, 0),      # refused: k is no multiple of 256
])
def test_kernels_of_a_call(rows, k, m, bf16, f32, relaid_bf16, relaid_f32):
    L = lib()
    assert [L.cn_nvfp4_gemm_launches(rows, k, m, d) for d in (CN_BF16, CN_F32)] == [bf16, f32]
    assert [L.cn_nvfp4_bs_launches(rows, k, m, d) for d in (CN_BF16, CN_F32)] == [relaid_bf16, relaid_f32]


@pytest.mark.parametrize("m", [1, 9, 128, 129, 512, 513, 4000])
@pytest.mark.parametrize("rows,k", [(64, 256), (1024, 10240), (5120, 17408), (17408, 5120), (32768, 512), (40000, 512)])
def test_workspace_of_a_matrix(rows, k, m):
    """The rows' own figure lies between the activations alone and the figure for any matrix, and has room for sums just where K is split."""
    rows_alone = m * k * 2 + (m * 4 + 255) // 256 * 256 + 256
    own, whole = ops.gemm_workspace_bytes(k, m, rows), ops.gemm_workspace_bytes(k, m)
    sums, left = divmod(own - rows_alone, m * rows * 4)
    assert left == 0 and own <= whole
    split = max(lib().cn_nvfp4_gemm_launches(rows, k, m, CN_BF16) - (m <= 128), lib().cn_nvfp4_gemm_launches(rows, k, m, CN_F32) - 1) > 1
    assert (sums >= 2) == split and (sums != 1)
    if m > 512:
        assert own == whole == rows_alone
