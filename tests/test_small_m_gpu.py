"""The kernel for few rows (M <= 64) against the CPU checker: every number of rows, tile edges in N, K cut over 1..8 CTAs.

Tolerance: |got - ref| <= 1e-3 + 2e-2 * |ref| on the bf16 outputs, zero mismatches (the operator's parity tolerance)."""
import numpy as np
import pytest

import fp8_quant_matmul_b200 as f
import helpers as h
from fp8_quant_matmul_b200.shard import shard_columns_of_B
from test_gemm_gpu import assert_parity, run_gemm

pytestmark = pytest.mark.gpu

# (M, N, K, splits): 0 = the library's choice
CASES = [(16, 16, 128, 0), (16, 128, 128, 1), (32, 144, 256, 2), (48, 80, 640, 5), (64, 512, 512, 1), (64, 272, 1152, 8),
         (16, 400, 1024, 7), (32, 1024, 1664, 4), (64, 576, 7168, 0), (16, 7168, 2304, 0), (48, 2064, 384, 3)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c)))
def test_few_rows_match_the_oracle(case):
    M, N, K, splits = case
    A, B, a_s, b_s = h.make_inputs(M, N, K, seed=500 + M + N + K)
    ref = h.oracle_gemm(A, B, a_s, b_s, M, N, K)
    got = run_gemm(A, B, a_s, b_s, M, N, K, splits=splits, tile_n=f.SMALL_M)
    assert_parity(ref, got, str(case))
    assert np.array_equal(got, run_gemm(A, B, a_s, b_s, M, N, K, splits=splits, tile_n=f.SMALL_M))   # summed in split order


def test_few_rows_column_shard_inside_a_scale_block():
    M, N, K, n0, nl = 32, 1024, 768, 192, 448
    A, B, a_s, b_s = h.make_inputs(M, N, K, seed=78)
    full = h.oracle_gemm(A, B, a_s, b_s, M, N, K)
    got = run_gemm(A, shard_columns_of_B(B, N, K, n0, nl), a_s, b_s, M, nl, K, n0=n0, n_total=N)
    assert f.select_path(M, nl, K)[2] == 128 | f.SMALL_M
    assert_parity(np.ascontiguousarray(full[:, n0:n0 + nl]), got, "few rows, shard")


def test_few_rows_on_the_path_that_does_not_cut_k():
    M, N, K = 32, 1024, 1664
    assert f.select_path(M, N, K)[1] > 1                                # left to itself the library cuts K
    A, B, a_s, b_s = h.make_inputs(M, N, K, seed=79)
    whole = run_gemm(A, B, a_s, b_s, M, N, K, splits=1, tile_n=f.SMALL_M)
    cut = run_gemm(A, B, a_s, b_s, M, N, K, splits=4, tile_n=f.SMALL_M)
    assert not np.array_equal(whole, cut)                               # another order of the sums: these inputs tell the two apart
    assert np.array_equal(whole, run_gemm(A, B, a_s, b_s, M, N, K, path=f.PATH_MN_LARGE, tile_n=f.SMALL_M))
