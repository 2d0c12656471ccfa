"""The rows that k-means takes at a time (csrc/erq_capi.cu, km_rows), over every
size it accepts: a product of them fits one grid, and their buffers fit what the
distances of that many rows took when they were stored."""
import itertools


def test_a_product_fits_a_grid_and_the_memory():
    from erq_b200 import load_library

    lib = load_library()
    most = 0x7fffffff
    for n, dim, k in itertools.product((1, 127, 5000, 10**6, 17 * 10**6, most), (1, 64, 100, 1536, 16384),
                                       (1, 100, 4096, 10**6, 9 * 10**6, 17 * 10**6, most)):
        rows = lib.erq_debug_kmeans_rows(n, dim, k)
        assert 1 <= rows <= n
        tiles = -(-rows // 128) * -(-k // 256)
        assert tiles <= most, (n, dim, k)  # gemm_tc refuses more
        cp = -(-dim // 64) * 64
        stored = min(n, max(1024, (256 << 20) // k))  # rows whose distances were stored
        assert rows * (6 * cp + 12) <= max(stored * (4 * k + 6 * cp + 4), stored * (6 * cp + 12)), (n, dim, k)
        assert rows >= min(stored, most // -(-k // 256) * 128) or rows == n, (n, dim, k)
