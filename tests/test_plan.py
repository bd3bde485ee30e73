"""How the tensor-core product of a shape would run is decided on the host, from the shape and the number of SMs
alone (`citlali_gemm_tc_plan`): checked here without a GPU.  The library is compiled if it is not there yet."""
import ctypes

import pytest

from citlali_b200 import ops


def library():
    try:
        return ops.lib()
    except Exception as e:                       # no compiler on this machine
        pytest.skip(f"the kernel library cannot be built here: {e}")


def plan(M, N, K, sms=148, force=0):
    lib = library()
    swapped, bn, splits = ctypes.c_int(), ctypes.c_int(), ctypes.c_int()
    lib.citlali_gemm_tc_plan(M, N, K, sms, force, ctypes.byref(swapped), ctypes.byref(bn), ctypes.byref(splits))
    return bool(swapped.value), bn.value, splits.value


@pytest.mark.parametrize("M,bn", [(1, 16), (8, 16), (16, 16), (17, 32), (33, 64), (64, 64), (65, 128), (128, 128)])
def test_few_rows_put_the_weights_on_the_wide_side(M, bn):
    swapped, width, splits = plan(M, 4096, 4096)
    assert swapped and width == bn
    assert splits in (1, 2, 4, 8)


@pytest.mark.parametrize("N, K, form", [(12288, 2048, (False, 192, 1)), (2048, 2048, (True, 256, 4)), (5632, 1024, (False, 192, 1)),
                                        (2048, 6144, (True, 256, 4)), (4096, 4096, (True, 256, 4)), (1024, 4096, (True, 256, 8)),
                                        (4096, 12288, (True, 256, 4))])
def test_more_than_128_rows_take_the_weights_wide_side_only_where_k_is_long(N, K, form):
    assert plan(129, N, K) == plan(256, N, K) == form
    assert plan(128, N, K)[:2] == (True, 128) and not plan(257, N, K)[0]
    assert plan(200, N, K, force=2)[0]                   # a forced split is one of the few-row form


@pytest.mark.parametrize("K", [2048, 3072, 4096, 12288])
def test_more_than_128_rows_split_k_by_eight_up_to_fifteen_tiles(K):
    """N of 8, 9, 12 and 15 tiles of 128 weight rows; with 16 of them clusters of eight blocks do not fit the device at once."""
    for M in (129, 256):
        assert [plan(M, N, K) for N in (1024, 1025, 1152, 1536, 1920)] == [(True, 256, 8)] * 5
        assert plan(M, 1921, K) == plan(M, 2048, K) == (True, 256, 4)


@pytest.mark.parametrize("N, K, sums", [(2048, 2048, 8), (1152, 12288, 8), (4096, 2624, 4), (4096, 2688, 4), (5632, 5312, 2), (5632, 5376, 2),
                                        (12288, 2048, 1), (256, 256, 1)])
def test_more_than_128_rows_add_k_up_in_as_many_sums_whatever_the_form(monkeypatch, N, K, sums):
    """One sum over all of K is off by as much as K is long: the form for many rows, and a split by four where one by eight does not fit,
    keep as many sums as K would be split over blocks.  A norm's work in the epilogue takes the form that can do it."""
    library()
    monkeypatch.setattr(ops, "sm_count", lambda device: 148)
    for M in (129, 256):
        plain, normed = ops.gemm_tc_plan(M, N, K, None), ops.gemm_tc_plan(M, N, K, None, normed=True)
        assert plain["sums"] == ops.gemm_tc_plan(M, N, K, None, gated=True)["sums"] == normed["sums"] == sums
        assert normed["swapped"] and ops.gemm_tc_is_small_form(M, N, K, None)
        many = K in (2624, 5312) or sums == 1
        assert plain["swapped"] != many and plain["bn"] == (256 if not many else 128 if sums == 4 else 192)
    assert ops.gemm_tc_plan(257, N, K, None)["sums"] == 1 and not ops.gemm_tc_is_small_form(257, N, K, None)


def test_k_is_split_by_shape_alone():
    # 148 SMs, two blocks each: 296 places for (tile, split) pairs; a split keeps four K blocks of 64 at least
    assert plan(8, 6144, 4096) == (True, 16, 4)          # 48 tiles: 6 would fit, powers of two only
    assert plan(8, 4096, 4096) == (True, 16, 8)          # 32 tiles
    assert plan(8, 24576, 4096) == (True, 16, 1)         # 192 tiles: no room for a second split
    assert plan(8, 4096, 12288) == (True, 16, 8)
    assert plan(8, 4096, 256) == (True, 16, 1)           # four K blocks: nothing to split
    assert plan(8, 4096, 512) == (True, 16, 2)
    # the same rows in another batch: the split does not depend on M within a width
    assert plan(1, 6144, 4096)[2] == plan(16, 6144, 4096)[2] == 4
    # a forced split replaces the plan's, up to 8 and the number of K blocks
    assert plan(8, 6144, 4096, force=3)[2] == 3
    assert plan(8, 6144, 4096, force=20)[2] == 8
    assert plan(8, 6144, 128, force=8)[2] == 2


def test_many_rows_put_x_on_the_wide_side():
    for M in (512, 2048, 3000):
        swapped, width, splits = plan(M, 6144, 4096)
        assert not swapped and splits == 1 and width in (256, 240, 224, 208, 192)
    # 16 row tiles x 4,096 outputs: 256 columns give 256 tiles (two waves of 148), 240 give 288 (two waves, cheaper tiles)
    assert plan(2048, 4096, 4096) == (False, 240, 1)
    # up to 256 rows one tile of 256 rows of x against narrow weights, K split, when whole tiles would leave SMs idle
    assert plan(200, 4096, 4096)[0] and plan(200, 4096, 4096)[1] == 256
    assert not plan(300, 4096, 4096)[0]
    # a narrow output has one width only
    assert plan(1000, 96, 72) == (False, 128, 1)


def test_the_plan_depends_on_the_number_of_sms():
    assert plan(8, 6144, 4096, sms=148)[2] == 4
    assert plan(8, 6144, 4096, sms=64)[2] == 2           # 128 places for 48 tiles
    assert plan(8, 6144, 4096, sms=20)[2] == 1


@pytest.mark.parametrize("rows, H, KH, D, V, taps, channel, runs", [case[:6] + (0,) + case[6:] for case in [
    (1, 16, 8, 128, 128, 4, True), (2, 2, 1, 32, 32, 4, True), (3, 16, 8, 128, 128, 4, False), (64, 32, 16, 128, 128, 4, False),
    (319, 16, 8, 128, 128, 4, False), (320, 16, 8, 128, 128, 4, True), (1279, 4, 2, 64, 64, 2, False), (1280, 4, 2, 64, 64, 2, True),
    (4096, 16, 8, 128, 128, 5, False), (4096, 16, 8, 128, 257, 4, False), (4096, 16, 8, 128, 128, 1, False)]] + [
    (1, 4, 4, 64, 64, 4, 1, True), (2, 4, 4, 64, 64, 4, 1, False), (682, 16, 16, 128, 128, 4, 1, False), (683, 16, 16, 128, 128, 4, 1, True)])
def test_the_delta_rules_preparation_takes_runs_of_rows_where_there_are_many(rows, H, KH, D, V, taps, channel, runs):
    assert bool(library().citlali_delta_prepare_in_runs(rows, H, KH, D, V, taps, channel)) == runs


@pytest.mark.parametrize("nq, nkv, d, keys, heads", [
    (8, 8, 128, 1, 0), (8, 8, 128, 7, 0), (8, 8, 128, 8, 1), (6, 2, 64, 7, 0), (6, 2, 64, 8, 1), (8, 2, 128, 1, 4), (16, 8, 128, 1, 2), (12, 1, 128, 1, 4),
    (8, 2, 128, 2867, 4), (8, 2, 128, 2868, 0), (16, 8, 128, 4778, 2), (16, 8, 128, 4779, 0), (8, 8, 128, 7168, 1), (8, 8, 128, 7169, 0), (8, 2, 257, 100, 0)])
def test_heads_that_32_bit_attention_takes_together(nq, nkv, d, keys, heads):
    assert library().citlali_attention_rows_heads(nq, nkv, d, keys) == heads


@pytest.mark.parametrize("lengths, H, D, V, chunks", [
    # the longest sequence's chain
    ([1], 16, 128, 128, False), ([24], 32, 128, 128, False), ([33], 16, 128, 128, False), ([48], 16, 128, 128, True), ([65], 16, 128, 128, True),
    ([2048], 2, 16, 4, True), ([56], 4, 16, 16, True), ([64] * 16, 2, 64, 64, True),
    # the work, where there is more of it than SMs
    ([33] * 16, 32, 128, 128, False), ([64] * 64, 16, 128, 128, True), ([65] * 64, 16, 128, 128, False), ([80] * 64, 16, 128, 128, True),
    ([48] * 64, 16, 96, 96, False), ([256] * 64, 16, 96, 96, True), ([48] * 64, 16, 128, 32, False), ([64] * 300, 16, 128, 64, True),
    # smaller heads: a chunk's blocks are full-sized all the same
    ([64] * 64, 4, 64, 64, False), ([128] * 64, 4, 64, 64, False), ([512] * 300, 4, 16, 16, False), ([96] * 16, 4, 64, 64, True),
    ([128] * 64, 16, 100, 36, False),
    # unequal lengths: neither the mean nor the longest alone
    ([540, 155, 300, 420, 200], 16, 128, 128, True), ([1] * 47 + [3000], 32, 128, 128, True), ([1] * 47 + [800], 16, 128, 128, True),
    ([1] * 300 + [64], 16, 128, 128, False)])
def test_the_delta_rule_runs_in_chunks_where_that_is_quicker(lengths, H, D, V, chunks):
    assert ops.delta_chunks_pay(lengths, H, D, V, 4 * H, 148) == chunks
    for no_pieces in ((D + 2, V, 4 * H), (D, V + 2, 4 * H), (D, V, 4 * H + 2), (132, V, 4 * H)):
        assert not ops.delta_chunks_pay([2048], H, *no_pieces, 148)


@pytest.mark.parametrize("units, tiles, runs", [(1, 1, 1), (1, 63, 32), (8, 33, 17), (8, 32, 32), (24, 8, 8), (16, 12, 12), (32, 5, 5), (64, 3, 3), (16, 63, 16),
                                                (17, 32, 16), (126, 63, 2), (300, 63, 1)])
def test_runs_of_the_latent_walk(units, tiles, runs):
    assert ops.latent_runs(units, tiles, 148) == runs


@pytest.mark.parametrize("tiles", [1, 2, 5, 12, 33, 64, 100])
def test_every_run_of_the_latent_walk_has_a_tile(tiles):
    for units in range(1, 400):
        runs = ops.latent_runs(units, tiles, 148)
        assert 1 <= runs <= 32 and (runs - 1) * -(-tiles // runs) < tiles


F32, BF16 = 0, 1


@pytest.mark.parametrize("entry", ["citlali_gemm_tc_act", "citlali_gemm_tc_pair_act"])
@pytest.mark.parametrize("mode, y_dtype, bias, code", [
    (8, F32, 0, -2), (1 | 8, F32, 0, -2), (1 | 8, BF16, 0, -2), (2 | 4, BF16, 0, -2), (2 | 8, BF16, 0, -2), (1 | 4, F32, 0, -2), (16, F32, 0, -2),
    (0, F32, 4100, -4), (8, BF16, 4104, -4), (4, BF16, 4108, -4)])
def test_epilogues_that_are_none_are_refused_before_any_launch(entry, mode, y_dtype, bias, code):
    """Addresses nobody reads: the answer comes from the arguments alone."""
    lib = library()
    args = [4096, 4096, 4096, y_dtype, 600, 64, 64, mode, bias, None]
    args += [148, None] if entry == "citlali_gemm_tc_act" else [None]
    assert getattr(lib, entry)(*args) == code
