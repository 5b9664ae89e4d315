"""Which kernel a call takes: host functions of sizes, each with the sizes that were measured on either side
of its line (148 SMs, no GPU)."""
import ctypes

import pytest

from minfer_b200.kernels import api as K

SMS = 148
EIGHT = [601, 700, 800, 900, 1000, 1100, 1200, 1300]


@pytest.mark.parametrize("lens,heads,P,N,columns", [
    (EIGHT, 64, 64, 128, 2),
    (EIGHT, 32, 128, 128, 2),
    ([17] * 16, 64, 64, 128, 2),
    ([15] * 16, 64, 64, 128, 1),            # few tokens a row
    ([1] * 64, 64, 64, 128, 1),
    ([3] * 7 + [400], 64, 64, 128, 1),      # one long row: its chain is what counts
    ([3] * 7 + [400], 128, 64, 128, 1),
    (EIGHT, 24, 64, 64, 1),                 # small states want more blocks
    (EIGHT, 64, 64, 64, 2),
    (EIGHT, 64, 80, 200, 1),                # half a block of padding
    (EIGHT, 64, 96, 128, 2),                # the same where two columns gain more
    ([500] * 3, 35, 96, 128, 1),            # fewer blocks than that takes
    (EIGHT, 64, 96, 64, 1),
    (EIGHT, 64, 33, 128, 2),
    (EIGHT, 64, 32, 128, 1),
    ([5000], 64, 64, 128, 1),
])
def test_columns_of_a_thread_of_the_state_space_scan(lens, heads, P, N, columns):
    choose = K._lib("recurrent").mf_ssm_scan_columns
    assert choose(sum(lens), len(lens), max(lens), heads, P, N, SMS) == columns
    # without the longest row's length it is taken to be as long as it can be
    assert choose(sum(lens), len(lens), 0, heads, P, N, SMS) <= columns


@pytest.mark.parametrize("lens,heads,D,Dv,columns", [
    (EIGHT, 8, 128, 256, 4),
    ([100] * 40, 8, 100, 250, 4),
    ([300] * 5, 8, 128, 256, 4),
    ([300] * 3, 8, 128, 256, 2),            # fewer blocks than one and a half an SM
    ([3] * 7 + [400], 8, 128, 256, 2),      # one long row: its chain is what counts
    ([63] * 8, 32, 128, 128, 2),            # few tokens a row
    (EIGHT, 60, 36, 40, 2),                 # half a block of padding, short keys
    (EIGHT, 60, 128, 33, 4),
    (EIGHT, 19, 128, 33, 2),
    (EIGHT, 40, 32, 64, 2),
    (EIGHT, 40, 129, 64, 2),
])
def test_columns_of_a_lane_of_gated_linear_attention(lens, heads, D, Dv, columns):
    choose = K._lib("outer_scan").mf_gla_scan_columns
    assert choose(sum(lens), max(lens), heads, D, Dv, SMS) == columns
    assert choose(sum(lens), 0, heads, D, Dv, SMS) == 2


@pytest.mark.parametrize("lens,tiled", [
    ([16], False), ([31], False), ([32], True), ([200], True),
    ([1] * 64, False),                      # many short sequences: a CTA would walk 32 of them in turn
    ([2] * 32, False), ([16] * 16, False), ([48] * 3, False),
    ([56] * 3, True), ([130, 255], True), ([64] * 8, True),
    ([1] * 31 + [200], False),
    ([1] * 63 + [1000], True),              # one that is worth it
    ([40] * 2, False), ([5, 60], False), ([5, 64], True),
    ([400] * 64, True),
])
def test_which_float32_prompts_walk_their_keys_by_tiles(lens, tiled):
    choose = K._lib("attention").mf_attention_packed_tiled
    assert bool(choose(sum(lens), len(lens), max(lens))) == tiled
    assert choose(sum(lens), len(lens), 0) <= tiled


@pytest.mark.parametrize("m,n,tile", [
    # (rows and columns of the products whose bits and whose wait are tested, among others)
    (17, 31, 2), (129, 1157, 2), (385, 1152, 2), (200, 4096, 2), (385, 896, 2), (1500, 1152, 2),
    (260, 9001, 1), (333, 9031, 1), (385, 9728, 1), (2500, 1152, 1),
    (700, 9001, 0), (2170, 2175, 0), (4096, 1152, 0), (1600, 8448, 0), (385, 151936, 0),
    (20, 4_000_000, 2), (20, 5_000_000, 0),         # 65,535 tiles of 64 columns end at 4,194,240
    (20, 9_000_000, -1),
])
def test_tile_of_a_float32_product(m, n, tile):
    """0: 128 x 128, 1: 64 x 64, 2: 32 x 64, -1: the general kernel."""
    assert K._lib("gemm_simt").mf_gemm_f32_tile(m, n, SMS) == tile


@pytest.mark.parametrize("m,n,k,tile,form", [
    (17, 31, 896, 2, 0), (129, 1157, 896, 2, 0), (385, 1152, 896, 2, 0), (385, 896, 896, 2, 0), (1500, 1152, 896, 2, 0),
    (200, 4096, 2044, 2, 0),
    (260, 9001, 896, 1, 0), (333, 9031, 896, 1, 0), (385, 9728, 896, 1, 0), (2500, 1152, 896, 1, 0),
    (700, 9001, 896, 0, 0), (2170, 2175, 896, 0, 0), (4096, 1152, 896, 0, 0), (1600, 8448, 896, 0, 0),
    (385, 151936, 896, 0, 0),
    (20, 4_000_000, 64, 2, 0), (20, 5_000_000, 64, 0, 0),         # 65,535 tiles of 64 columns end at 4,194,240
    (20, 9_000_000, 64, -1, 0), (20, 9_000_000, 4096, -1, 0),
    # four stretches: a cluster a tile ...
    (17, 896, 4864, 2, 1), (64, 896, 4864, 2, 1), (385, 896, 4864, 2, 1), (700, 896, 4864, 1, 1), (40, 9001, 2048, 1, 1),
    (512, 3584, 18944, 1, 1), (200, 4096, 2048, 0, 1), (1600, 2048, 8448, 0, 1), (485, 2173, 2180, 0, 1),
    # ... or, where one CTA a tile fills the GPU, one after the other
    (400, 9001, 2048, 0, 2), (390, 9001, 2052, 0, 2), (1600, 8448, 2048, 0, 2), (512, 18944, 3584, 0, 2),
    (634, 6420, 2080, 0, 2), (1600, 1157, 2052, 1, 2), (700, 5000, 2180, 1, 2), (41, 12001, 2052, 2, 2),
])
def test_cut_of_a_float32_product(m, n, k, tile, form):
    """0: 128 x 128, 1: 64 x 64, 2: 32 x 64, -1: the general kernel; 0: one stretch of k, 1: a cluster a tile,
    2: one CTA a tile."""
    got = K.gemm_f32_cut(m, n, k, SMS)
    assert got[0] == tile and (tile < 0 or got[1] == form)


@pytest.mark.parametrize("rows,kv,reach,tiles,splits", [
    # (tiles a CTA, CTAs that share a row's keys); four tiles: a tile a warp
    (8, 4, 1300, 4, 11), (8, 4, 1536, 4, 13),      # all CTAs on the GPU at once, merged in one trip
    (3, 2, 1900, 4, 16), (3, 2, 2000, 4, 16),
    (3, 2, 8000, 8, 32), (3, 2, 8192, 8, 33), (26, 1, 3000, 8, 12),    # more splits than one trip takes
    (8, 8, 3000, 20, 5), (64, 4, 1300, 24, 2), (64, 8, 100, 8, 1),     # the rows alone fill the GPU
    (1, 8, 100, 4, 2), (1, 1, 1, 4, 1),
])
def test_cut_of_single_queries(rows, kv, reach, tiles, splits):
    out = (ctypes.c_int * 2)()
    K._lib("attention_sink").mf_sink_decode_plan_on(rows, kv, reach, SMS, ctypes.addressof(out),
                                                    ctypes.addressof(out) + 4)
    assert tuple(out) == (tiles, splits)
    assert tiles * splits * 32 >= reach + 31                 # the reach need not start on a tile


@pytest.mark.parametrize("m,n,k,groups,cluster", [
    # 512 KB to 64 MB of weights, 16 MB beyond 8 tokens
    (1, 256, 1016, 0, 0), (1, 256, 1024, 32, 1), (8, 16384, 2048, 147, 1), (8, 16896, 2048, 0, 0),
    (8, 9728, 896, 136, 1), (9, 9728, 896, 0, 0), (9, 9360, 896, 147, 1), (8, 3584, 3584, 112, 1), (9, 3584, 3584, 0, 0),
    (16, 1152, 896, 144, 1), (17, 1152, 896, 0, 0),
    # many rows and a short K: heads of small models
    (1, 8192, 64, 147, 1), (1, 16000, 64, 0, 0), (8, 16000, 192, 0, 0), (8, 16000, 256, 143, 1), (1, 32000, 768, 0, 0),
    (1, 32000, 1024, 143, 1), (1, 152064, 128, 0, 0), (9, 8192, 192, 0, 0), (9, 8192, 256, 147, 1), (9, 16000, 512, 0, 0),
    # K cut between CTAs: the tokens of one do not fit, or few rows and a long K (the largest cluster where none
    # fills the GPU)
    (8, 896, 4864, 112, 1), (16, 896, 4864, 56, 2), (8, 2048, 8448, 128, 1), (1, 88, 4496, 11, 2), (8, 144, 8840, 18, 4),
    (1, 72, 17632, 9, 4), (3, 40, 20000, 5, 4),
])
def test_products_for_a_handful_of_tokens(m, n, k, groups, cluster):
    assert K.gemm_few_plan(m, n, k, SMS) == (groups, cluster)


def test_nothing_is_kept_for_the_lengths_of_prompts():
    before = dict(K._FEW)
    for m in range(17, 300):
        assert K.gemm_few_groups(m, 1152, 896) == 0 and K.gemm_few_plan(m, 1152, 896, SMS) == (0, 0)
    assert K._FEW == before


@pytest.mark.parametrize("sms", [1, 2, 3, 15, 16, 17, 19, 20, 148, 300])
def test_the_cut_for_a_handful_of_tokens_on_any_number_of_sms(sms):
    for m, n, k in ((1, 1152, 896), (16, 896, 4864), (3, 40, 20000), (8, 2048, 8448)):
        groups, cluster = K.gemm_few_plan(m, n, k, sms)
        assert (groups == 0) == (cluster == 0) and groups <= (n + 7) // 8


@pytest.mark.parametrize("m,n,k,tile,dual", [
    # the largest tile that leaves no pair idle in the last round ...
    (2048, 37888, 3584, 256, False), (20011, 3584, 18944, 256, False), (1024, 11264, 2048, 208, False),
    (515, 27648, 5120, 176, False), (515, 5120, 13824, 176, False),
    # ... but no larger one that makes fewer tiles of a single round
    (515, 3584, 3584, 160, False), (700, 3072, 2048, 160, False), (1000, 2048, 5632, 160, False),
    (515, 7168, 5120, 160, False),
    # two token tiles a pair: long K, one or two rounds
    (2048, 3584, 18944, 208, True), (2048, 3584, 3584, 208, True), (1024, 5120, 13824, 176, True),
    (3000, 2048, 5632, 176, True), (1300, 4608, 3584, 192, False),
])
def test_tile_of_a_product_of_a_prompt(m, n, k, tile, dual):
    assert K.gemm_pair_plan(m, n, k, SMS) == (tile, dual)
