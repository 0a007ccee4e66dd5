"""Which products of 9 to 16 rows go to the kernel for few rows (ops.gemm.rows_pays): shapes whose times on
both sides lie apart, in a chain of launches with cold weights."""
import pytest

from easy_to_hard_b200.ops import gemm

# features, K, rows, bits; us on the kernel for few rows, us on the tcgen05 kernels
MEASURED = [(4096, 4096, 16, 16, 10.3, 12.4), (12288, 4096, 9, 16, 21.8, 25.8),
            (8192, 8192, 16, 16, 27.0, 29.4), (2048, 2048, 16, 16, 6.2, 7.4),
            (5120, 13824, 9, 16, 34.6, 29.7), (5120, 13824, 16, 16, 36.1, 29.6),
            (10240, 8192, 16, 16, 38.9, 35.2), (10240, 22016, 9, 16, 97.9, 80.3),
            (4096, 22016, 16, 16, 39.2, 35.7), (12288, 13824, 12, 16, 65.4, 60.0),
            (4096, 11008, 16, 8, 18.8, 21.0), (8192, 22016, 16, 8, 49.0, 61.1),
            (1536, 13824, 16, 8, 18.3, 15.6), (12288, 4096, 16, 8, 20.3, 27.1),
            (1536, 8192, 16, 4, 16.4, 12.1), (1536, 2048, 16, 4, 5.2, 6.3),
            (4096, 4096, 16, 4, 10.6, 12.1), (4096, 13824, 16, 4, 28.6, 24.7),
            (5120, 13824, 16, 4, 34.8, 42.6), (8192, 8192, 16, 4, 22.9, 28.4),
            (20480, 22016, 16, 4, 123.7, 236.5)]


@pytest.mark.parametrize("F,K,T,bits,rows,wide", MEASURED)
def test_the_faster_side_is_taken(F, K, T, bits, rows, wide):
    assert gemm.rows_pays(F, K, T, bits) == (rows < wide)
