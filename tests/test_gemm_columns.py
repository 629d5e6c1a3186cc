"""Which width the column tiles of the dense GEMM get on a B200 (CPU)."""

import pytest


@pytest.mark.parametrize("rows,n_out,k_bytes,columns", [
    # rounds of tiles over 74 pairs of SMs
    (64, 3072, 12288, 64), (1000, 3072, 12288, 192), (1000, 12288, 3072, 224), (33272, 3072, 12288, 256), (33272, 3072, 6144, 256),
    (2304, 3072, 6144, 192), (2816, 3072, 6144, 256), (1, 8, 128, 64), (1, 264, 6144, 64),
    # less than 128 KB of A: no more than 24 tiles
    (1, 3072, 12288, 128), (10, 3072, 12288, 128), (11, 3072, 12288, 64), (1, 3072, 6144, 128), (21, 3072, 6144, 128), (22, 3072, 6144, 64),
    (1, 4096, 2048, 192), (63, 4096, 2048, 192), (64, 4096, 2048, 64), (1, 2048, 4096, 96), (1, 1536, 4096, 64), (1, 6144, 2048, 256),
    (1, 12288, 3072, 256), (300, 9216, 128, 256)])
def test_columns(native_lib, rows, n_out, k_bytes, columns):
    assert native_lib.h3s_dense_gemm_columns(rows, n_out, k_bytes, 148) == columns


def test_every_width_is_one_that_the_kernel_takes(native_lib):
    for sms in (0, 1, 2, 80, 148):
        for rows in (1, 20, 130, 1000, 4000, 70000):
            for n_out in (8, 64, 200, 1000, 3072, 50000):
                for k_bytes in (128, 3072, 16384):
                    columns = native_lib.h3s_dense_gemm_columns(rows, n_out, k_bytes, sms)
                    assert columns % 32 == 0 and 64 <= columns <= 256
