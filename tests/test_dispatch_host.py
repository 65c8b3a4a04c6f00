"""Rules by which the host chooses a kernel's shape, for GPUs of a given number of SMs (CPU, no compute)."""
from conftest import pkg


def test_ranks_by_1024_threads_from_a_number_of_pairs_that_depends_on_the_waves():
    f = pkg("_lib").load().b200_moe_rank_threads
    assert [f(n, e, 148) for e in (1, 128, 148) for n in (0, 8191, 8192)] == [256, 256, 1024] * 3
    assert [f(n, e, 148) for e in (149, 256, 1024) for n in (8192, 16383, 16384)] == [256, 256, 1024] * 3
    assert f(8192, 149, 160) == 1024 and f(1, 0, 148) < 0


def test_row_tiles_of_dense_products():
    """Fewest waves of CTAs, then least data; a narrower tile that would need one wave more has to win by more than the estimate errs."""
    f = pkg("_lib").load().b200_dense_gemm_row_tile
    assert [f(m, 2048, 148) for m in (1300, 1500, 1777, 2048)] == [160, 192, 224, 256]
    assert f(4096, 5120, 148) == 256 and f(2246, 9216, 148) == 256 and f(1648, 12288, 148) == 256
    assert all(f(m, n, 148) % 32 == 0 and 32 <= f(m, n, 148) <= 256 for m in range(257, 4097, 37) for n in (100, 512, 5120, 10240))
    assert f(0, 2048, 148) < 0
