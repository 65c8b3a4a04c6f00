"""Rules by which the host chooses a kernel's shape, for GPUs of a given number of SMs (CPU, no compute)."""
from conftest import pkg


def test_ranks_by_1024_threads_from_a_number_of_pairs_that_depends_on_the_waves():
    f = pkg("_lib").load().b200_moe_rank_threads
    assert [f(n, e, 148) for e in (1, 128, 148) for n in (0, 8191, 8192)] == [256, 256, 1024] * 3
    assert [f(n, e, 148) for e in (149, 256, 1024) for n in (8192, 16383, 16384)] == [256, 256, 1024] * 3
    assert f(8192, 149, 160) == 1024 and f(1, 0, 148) < 0
