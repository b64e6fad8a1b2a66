"""Which product takes few rows, and in which units (no GPU): what the kernels refuse must never be planned."""
import itertools

from dryft_challenge_htn_2026_b200.csrc import api


def test_plans_of_few_rows_are_ones_the_kernels_take():
    sms = api.sm_count()
    for M, N, K in itertools.product((1, 2, 7, 8), (72, 2560, 6144, 9728, 151936), (304, 2560, 4096, 5120, 9728, 20000)):
        for mode, partial in ((api.MODE_STORE, False), (api.MODE_STORE, True), (api.MODE_STORE_F32, False), (api.MODE_STORE_F32, True),
                              (api.MODE_SILU, False), (api.MODE_XIELU, False)):
            plan = api.few_rows_stream_plan(M, N, K, mode, partial)
            if plan is None:
                continue
            sk, blocks, warps = plan
            assert sk == 1 or (partial and mode not in (api.MODE_SILU, api.MODE_XIELU))
            assert blocks >= sk and warps in (4, 8) and api._stream_smem(M, K, sk, warps) <= 227 * 1024
    for N, K in ((72, 304), (2560, 2560)):            # small matrices: as ever
        assert api.few_rows_stream_plan(4, N, K, api.MODE_STORE, True) == api.stream_plan(4, N, K, api.MODE_STORE, True)
    assert api.few_rows_stream_plan(8, 2560, 4096, api.MODE_STORE, True) == (1, sms, 8)
    assert api.few_rows_stream_plan(8, 2560, 9728, api.MODE_STORE, True) is None
    for N, K, mode in ((6144, 2560, api.MODE_STORE), (9728, 2560, api.MODE_SILU)):
        assert api.few_rows_stream_plan(8, N, K, mode, True) == api.stream_plan(8, N, K, mode, True)


def test_units_of_up_to_32_rows_leave_sms_to_the_kernels_around_them():
    sms = api.sm_count()
    for M, N, K in itertools.product((1, 9, 32), (8, 304, 2560, 6144, 7168, 33000), (64, 520, 2560, 4096, 17408)):
        bn, sk = api.skinny_tc_plan(M, N, K, api.MODE_STORE, True)
        kb, tiles = (K + 63) // 64, (N + bn - 1) // bn
        assert bn in api.TC_TILE_HEIGHTS and sk >= 1 and (sk == 1 or (sk - 1) * ((kb + sk - 1) // sk) < kb)
        assert tiles * sk < 0.9 * sms or N == 33000
        if (N + 255) // 256 <= sms // 4 and K >= 2560:
            assert sk > 1                                 # float32 parts, as many rows as few
    if sms == 148:
        assert api.skinny_tc_plan(16, 2560, 4096, api.MODE_STORE, True) == (160, 8)
        assert api.skinny_tc_plan(16, 4096, 12288, api.MODE_STORE, True) == (256, 8)
