"""Which tiles the bfloat16 product takes, without a GPU: the choice against times measured on one."""
from ctypes import c_int

import pytest

PAIRS = 74
# tokens, features, K, epilogue (0 plain, 1 a gate, 2 heads, 4 an activation): us with tiles of 256 tokens, us with the best
# tiles of 256 features
MEASURED = [
    (2048, 8192, 1024, 1, 46.8, 56.9), (2079, 16384, 2048, 1, 120.9, 139.2), (2048, 3072, 2048, 2, 34.4, 37.8),
    (1000, 4608, 3584, 2, 32.0, 41.6), (1537, 4608, 3584, 2, 48.5, 52.3), (700, 4096, 14336, 0, 67.9, 78.9),
    (543, 16384, 2048, 1, 53.6, 44.4), (2079, 4608, 3584, 2, 77.8, 66.0), (257, 37888, 3584, 1, 102.6, 83.9),
    (543, 27648, 5120, 1, 175.7, 153.0), (543, 7168, 5120, 2, 65.3, 50.4), (543, 5120, 13824, 0, 85.1, 73.4),
    (2079, 5120, 5120, 0, 100.5, 86.7), (300, 55296, 5120, 1, 234.6, 182.5), (2079, 27648, 5120, 4, 535.3, 456.9),
    (2079, 2048, 8192, 0, 54.7, 51.6),
]


def pair_form(M, N, K, epilogue):
    from mini_hisparse_b200.kernels import build

    return build.load("gemm_tc").mhb_gemm_tc_pair_form(c_int(M), c_int(N), c_int(K), c_int(PAIRS), c_int(epilogue))


@pytest.mark.parametrize("M,N,K,epilogue,tokens_us,features_us", MEASURED)
def test_the_form_that_measured_faster_is_taken(M, N, K, epilogue, tokens_us, features_us):
    assert (pair_form(M, N, K, epilogue) > 0) == (features_us < tokens_us)


@pytest.mark.parametrize("epilogue", [0, 1, 2, 4])
def test_tiles_are_ones_that_the_kernel_has(epilogue):
    """Widths in steps of 16 (32 behind a gate, whole heads behind the heads' epilogue) up to 256; up to 256 tokens one tile's rows."""
    seen = set()
    for M in (129, 256, 257, 400, 543, 1000, 2079, 5000):
        for N in (64, 192, 256, 1024, 4608, 14016, 37888):
            for K in (8, 200, 1024, 5120, 27648):
                form = pair_form(M, N, K, epilogue)
                seen.add(form > 0)
                if form > 0:
                    assert M > 256 and 96 <= form <= 256 and form % 16 == 0
                else:
                    step = 32 if epilogue == 1 or N < 256 else 128 if epilogue == 2 else 16
                    assert -256 <= form and form % step == 0 and (N < 256 or form <= -128)
    assert seen == {False, True}
