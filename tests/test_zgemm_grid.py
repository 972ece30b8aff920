"""Host arithmetic of the FP64 GEMM: which SMs its tiles land on, and how long its sums are."""
import ctypes

import pytest

import internals


@pytest.mark.parametrize("items", [1, 2, 69, 138, 147, 148, 149, 295, 296, 297, 1000, 100000])
def test_paired_ctas_use_every_sm_before_a_second_team(items):
    sms = 148
    ctas = internals.load().zgemm_ctas(items, sms, 2, 1)
    assert ctas == min(items, sms)
    # item i goes to team i / ctas (mod 2) of CTA i % ctas: per CTA at most one more than the mean
    per = [len(range(c, items, ctas)) for c in range(ctas)]
    assert max(per) == -(-items // sms)


@pytest.mark.parametrize("resident", [2, 3, 4])
def test_unpaired_ctas(resident):
    sms, f = 148, internals.load().zgemm_ctas
    for items in (1, 147, 149, sms * resident, 4 * sms * resident):
        assert f(items, sms, resident, 0) == items
    assert f(4 * sms * resident + 1, sms, resident, 0) == sms * resident


@pytest.mark.parametrize("M,N,K,KB,batch,tri", [
    (120, 120, 676, 8, 12, 1), (120, 120, 676, 8, 12, 0), (160, 160, 400, 8, 12, 1), (250, 250, 1296, 8, 12, 1),
    (400, 400, 2704, 4, 12, 1), (1872, 26, 26, 120, 1, 0), (1440, 20, 20, 160, 1, 0), (36, 36, 36, 7776, 1, 0),
    (403, 611, 2707, 1, 1, 0), (52, 52, 52, 1, 1, 0), (7, 5, 100000, 1, 1, 0), (3744, 52, 52, 400, 1, 0)])
def test_long_sums_are_cut(M, N, K, KB, batch, tri):
    # at most 128 groups of 4 per accumulator, unless the parts would have fewer than 8 groups each, exceed 256 or the
    # room for them, or leave more than four 64 x 64 tiles per SM
    sms, room = 148, 1 << 22
    f = internals.load().zgemm_splits
    f.argtypes = [ctypes.c_int] * 7 + [ctypes.c_int64, ctypes.c_int]
    groups = KB * -(-K // 4)
    tiles64 = -(-M // 64) * -(-N // 64) * batch
    least = max(1, min(-(-groups // 128), -(-4 * sms // tiles64), 256, groups // 8, room // (M * N * batch)))
    splits = f(M, N, K, KB, batch, tri, 0, room, sms)
    assert splits >= least and splits * M * N * batch <= room and (splits == 1 or groups // splits >= 8)
    assert f(M, N, K, KB, batch, tri, 0, 0, sms) == 1          # no room: whole sums
    assert f(M, N, K, KB, batch, tri, 1, room, sms) >= 1       # three products: by time alone
