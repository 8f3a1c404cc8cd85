"""With the number of splits left open, a call that asks for the split-K family takes whatever cut of K its workspace holds, so
that no call is refused because the cost model now prefers a configuration with more partial sums.  Host logic only: without a
GPU a call that passes the workspace check comes back as "no device" (-6), one that does not as -4."""
import ctypes

import pytest

import fp8_quant_matmul_b200 as f

FAKE = ctypes.c_void_p(0x1000)


def small(M, N, K, splits, ws_bytes, static=False):
    lib = f.lib()
    if static:
        return lib.fp8bs_gemm_mn_small_static(FAKE, FAKE, FAKE, FAKE, FAKE, M, N, K, splits, None)
    return lib.fp8bs_gemm_mn_small(FAKE, FAKE, FAKE, FAKE, FAKE, M, N, K, splits, FAKE if ws_bytes else None, ws_bytes, None)


@pytest.fixture(autouse=True)
def no_device():
    torch = pytest.importorskip("torch")
    if torch.cuda.is_available():
        pytest.skip("fake pointers: only where no device can be reached")


@pytest.mark.parametrize("shape", [(384, 96, 1792), (832, 64, 1536), (96, 7680, 1920), (1568, 96, 1792), (64, 15552, 8320)])
def test_open_splits_need_no_workspace_where_a_cluster_can_cut_k(shape):
    assert small(*shape, 0, 0) == -6


@pytest.mark.parametrize("shape", [(12176, 16, 5760), (15088, 304, 256), (3744, 4960, 128)])
def test_open_splits_take_what_fits(shape):
    need = f.workspace_bytes(*shape, f.PATH_MN_SMALL)
    least = min(f.workspace_bytes(*shape, f.PATH_MN_SMALL, 1, t | f.SPLIT_WORKSPACE) for t in (128, 256))
    assert small(*shape, 0, max(need, least)) == -6
    assert small(*shape, 0, least) == -6
    assert small(*shape, 1, 65536) == -4 and small(*shape, 1, 0) == -4      # splits given: what it needs, or refused


@pytest.mark.parametrize("shape", [(1072, 6672, 896), (1136, 6480, 384), (11584, 592, 128)])
def test_built_in_scratch_holds_some_cut_of_k(shape):
    assert small(*shape, 0, 0, static=True) == -6
