"""The rule that chooses a GEMM kernel (``choose_gemm_plan`` in ``csrc/gemm_tcgen05.cu``) against measured times; no GPU needed."""
import ctypes

import pytest

from fairscale_b200 import _native

PAIR, ONE_CTA, CLUSTER_K = 0, 1, 2


@pytest.fixture(scope="module")
def plan_of():
    if not _native.available():
        pytest.skip("the native library has not been built")
    f = _native.lib().fsb_gemm_plan_of
    f.argtypes = [ctypes.c_longlong] + [ctypes.c_int] * 6
    return lambda M, N, K, lda, ldb, problems=1: f(problems, M, N, K, lda, ldb, 148)


# M, N, K, MN-major operands?, us one CTA per tile, us CTA pairs (B200, back to back)
MEASURED = [
    (952, 12048, 704, 0, 20.5, 30.8), (8192, 4096, 1024, 0, 61.5, 80.8), (4096, 4096, 1024, 1, 35.7, 45.7), (5968, 2048, 2048, 0, 42.5, 53.3),
    (5968, 8192, 2048, 0, 174.0, 180.8), (2864, 4800, 6528, 0, 139.6, 161.7), (3872, 4688, 14208, 0, 389.5, 466.7), (2048, 6144, 16384, 1, 393.4, 346.7),
    (4096, 22016, 4096, 0, 553.9, 502.2), (4096, 11008, 4096, 1, 336.6, 302.6), (552, 6912, 3808, 1, 31.5, 60.1), (1984, 5688, 4704, 1, 124.9, 110.6),
    (1936, 5872, 4360, 0, 138.8, 110.1), (2992, 1976, 13208, 1, 238.1, 168.8), (12952, 328, 11496, 0, 242.2, 168.4), (496, 6184, 10920, 1, 107.5, 79.2),
    (928, 12728, 6736, 1, 204.2, 153.6), (6552, 7776, 4440, 0, 541.6, 415.9), (2208, 2640, 2240, 0, 30.4, 37.0), (13640, 13184, 616, 0, 312.6, 331.8),
    (16384, 8192, 2048, 0, 470.8, 459.6), (16384, 2048, 2048, 0, 121.5, 124.8), (16384, 16384, 768, 0, 418.2, 452.2), (16384, 50304, 2048, 0, 2911.8, 2783.5),
]


@pytest.mark.parametrize("M,N,K,mn,one,pair", MEASURED)
def test_rule_takes_the_faster_persistent_kernel(plan_of, M, N, K, mn, one, pair):
    plan = plan_of(M, N, K, *((M, N) if mn else (K, K)))
    assert plan in (PAIR, ONE_CTA)
    assert (pair if plan == PAIR else one) <= 1.05 * min(one, pair)


def test_small_and_short_products_never_take_pairs(plan_of):
    assert plan_of(77, 1024, 4096, 4096, 4096) == CLUSTER_K
    assert plan_of(1024, 1024, 8192, 8192, 8192) == CLUSTER_K
    assert plan_of(2048, 2048, 2048, 2048, 2048) == ONE_CTA
    assert plan_of(255, 60000, 8192, 8192, 8192) == ONE_CTA  # the pairs take M and N from 256 on
    assert plan_of(60000, 255, 8192, 8192, 8192) == ONE_CTA
    assert plan_of(16384, 16384, 1400, 1400, 1400) == ONE_CTA


def test_stacked_products(plan_of):
    assert plan_of(2048, 8192, 1024, 1024, 1024, problems=16) == ONE_CTA  # 510 against 547 us
    assert plan_of(2048, 2048, 8192, 8192, 8192, problems=16) == PAIR  # 972 against 937 us
