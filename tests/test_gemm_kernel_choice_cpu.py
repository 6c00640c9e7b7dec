"""The kernel that ``fsb_gemm_bf16`` and ``fsb_gemm_bf16_batched`` launch (``plan_product`` in ``csrc/gemm_tcgen05.cu``) against measured times; no GPU needed.

``test_gemm_dispatch_cpu.py`` has the part of the rule that decides where results do not go out as bf16 in 16-byte pieces.
"""
import ctypes

import pytest

from fairscale_b200 import _native

PAIR, ONE_CTA, CLUSTER_K, WIDE = 0, 1, 2, 3
NONE, BIAS, RESIDUAL = 0, 1, 5


@pytest.fixture(scope="module")
def kernel_of():
    if not _native.available():
        pytest.skip("the native library has not been built")
    f = _native.lib().fsb_gemm_kernel_of
    f.argtypes = [ctypes.c_int] * 11

    def run(M, N, K, lda=None, ldb=None, problems=1, epilogue=NONE, out_f32=0, ldc=None, ld_aux=0):
        return f(problems, M, N, K, lda or K, ldb or K, ldc or N, ld_aux, epilogue, out_f32, 148)

    return run


# problems, M, N, K, MN-major operands?, us tiles of 512 rows, us CTA pairs, us one CTA (B200, back to back)
PLAIN = [
    (1, 952, 12048, 704, 0, 26.6, 24.6, 20.5), (1, 8192, 4096, 1024, 0, 65.6, 70.3, 66.1), (1, 4096, 4096, 1024, 1, 34.8, 38.3, 35.3),
    (1, 5968, 2048, 2048, 0, 51.3, 48.7, 45.6), (1, 5968, 8192, 2048, 0, 170.1, 178.9, 176.7),
    (1, 2864, 4800, 6528, 0, 162.3, 168.9, 152.6), (1, 3872, 4688, 14208, 0, 479.2, 463.0, 434.1),
    (1, 2048, 6144, 16384, 1, 367.7, 345.2, 357.4), (1, 4096, 22016, 4096, 0, 547.5, 566.7, 596.5),
    (1, 4096, 11008, 4096, 1, 279.0, 304.1, 311.0), (1, 1984, 5688, 4704, 1, 109.6, 104.4, 129.9),
    (1, 1936, 5872, 4360, 0, 105.4, 108.7, 136.0), (1, 2992, 1976, 13208, 1, 155.6, 172.0, 225.8),
    (1, 12952, 328, 11496, 0, 143.0, 173.7, 222.1), (1, 928, 12728, 6736, 1, 163.7, 160.2, 203.9),
    (1, 6552, 7776, 4440, 0, 379.0, 437.7, 558.0), (1, 2208, 2640, 2240, 0, 32.7, 32.8, 30.0),
    (1, 13640, 13184, 616, 0, 245.2, 292.5, 321.8), (1, 16384, 8192, 2048, 0, 417.3, 467.1, 466.3),
    (1, 16384, 2048, 2048, 0, 118.7, 122.0, 120.9), (1, 16384, 16384, 768, 0, 367.5, 410.0, 414.8),
    (1, 16384, 50304, 2048, 0, 2527.0, 2783.8, 2852.5), (1, 16384, 6144, 2048, 0, 322.6, 351.8, 345.3),
    (1, 8192, 2048, 16384, 1, 435.2, 475.7, 481.8), (1, 50304, 2048, 16384, 1, 2551.8, 2837.0, 2798.3),
    (1, 4096, 12288, 4096, 0, 322.2, 322.7, 344.9), (1, 8192, 3072, 1024, 0, 50.8, 55.2, 52.0),
    (1, 2792, 3968, 256, 0, 16.5, 16.4, 14.3), (1, 16384, 16384, 1400, 0, 641.4, 791.3, 894.9),
    (1, 22016, 4096, 4096, 1, 565.7, 606.3, 606.5), (1, 8192, 8192, 2048, 0, 212.5, 235.9, 235.3),
    (8, 2048, 1024, 4096, 0, 122.8, 127.0, 132.7), (16, 2048, 8192, 1024, 0, 463.7, 545.6, 508.6),
    (16, 2048, 2048, 8192, 0, 827.5, 883.1, 924.5), (4, 2048, 4360, 4360, 0, 265.9, 306.7, 394.7),
]


def test_plain_products_take_the_fastest_kernel(kernel_of):
    """Within 10 % each (two kernels that are this close change places with the clock) and 1 % on average."""
    loss = []
    for problems, M, N, K, mn, *us in PLAIN:
        kernel = kernel_of(M, N, K, *((M, N) if mn else (K, K)), problems=problems)
        assert kernel in (WIDE, PAIR, ONE_CTA)
        loss.append({WIDE: us[0], PAIR: us[1], ONE_CTA: us[2]}[kernel] / min(t for t in us if t is not None) - 1)
        assert loss[-1] < 0.10, (problems, M, N, K, kernel)
        assert kernel_of(M, N, K, *((M, N) if mn else (K, K)), problems=problems, epilogue=BIAS) == kernel
    assert sum(loss) / len(loss) < 0.01


def test_where_the_estimates_do_not_decide(kernel_of):
    plan_of = _native.lib().fsb_gemm_plan_of
    plan_of.argtypes = [ctypes.c_longlong] + [ctypes.c_int] * 6
    for M, N, K in ((77, 1024, 4096), (1024, 1024, 8192), (2048, 2048, 2048), (16384, 50304, 2048), (4096, 12288, 4096), (16384, 16384, 200)):
        for problems in (1, 4):
            old = plan_of(problems, M, N, K, K, K, 148)
            assert kernel_of(M, N, K, problems=problems, out_f32=1) == old  # fp32 results
            assert kernel_of(M, N - 1, K, problems=problems, ldc=N) == plan_of(problems, M, N - 1, K, K, K, 148)  # rows in no 16-byte pieces
            assert kernel_of(M, N, K, problems=problems, ldc=N + 4) == old
            assert kernel_of(M, N, K, problems=problems, ld_aux=N + 4, epilogue=RESIDUAL) == old
            if K < 256 or problems * (-(-M // 128)) * (-(-N // 256)) <= 148:
                assert kernel_of(M, N, K, problems=problems) == old
    assert kernel_of(77, 1024, 4096) == CLUSTER_K and kernel_of(2048, 2048, 2048) == ONE_CTA
    assert kernel_of(255, 60000, 8192) == kernel_of(60000, 255, 8192) == ONE_CTA
    assert kernel_of(511, 60000, 8192) in (PAIR, ONE_CTA)  # the tiles of 512 rows take M from 512 on
