"""K-slices of the EXL3 GEMV: a legal count for every length that has one, chunks that do not depend on the number of pairs."""
import pytest

from spark_engine_b200.ops import cuda as cu


def _legal(K, s):
    return 1 <= s <= 8 and K // 128 % s == 0 and K // s <= 2048              # what the kernel takes


@pytest.mark.parametrize("pairs", [False, True])
def test_every_length_with_a_legal_count_gets_one(pairs):
    for K in range(128, 8 * 2048 + 1, 128):
        if not any(_legal(K, s) for s in range(1, 9)):
            continue
        for N in (128, 2048, 12288):
            for items in (1, 2, 40, 256):
                assert _legal(K, cu._pick_slices(K, items, N, pairs)), (K, N, items)


def test_chunks_of_a_pair_do_not_depend_on_the_number_of_pairs():
    for K in range(128, 8 * 2048 + 1, 128):
        if any(_legal(K, s) for s in range(1, 9)):
            lengths = [K // cu._pick_slices(K, items, N, True) for N in (128, 1024, 4096) for items in (1, 3, 16, 40, 160, 256, 1000)]
            assert len({256 if k % 256 == 0 else 128 for k in lengths}) == 1, K


def test_chains_of_rows_are_no_longer_than_those_of_slices_of_256():
    """Four warps share a slice of one matrix, every fourth tile of 16 k each: the chain's length is what its rounding grows with."""
    for K in range(128, 8 * 2048 + 1, 128):
        legal = [s for s in range(1, 9) if _legal(K, s)]
        if legal:
            short = next((s for s in legal if K // s <= 256), legal[-1])
            for N in (128, 2048, 12288, 65536, 151936):
                assert K // cu._pick_slices(K, 1, N) // 64 <= K // short // 16, (K, N)
