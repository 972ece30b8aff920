"""Grid of the FP64 GEMM: which SMs its tiles land on (host arithmetic only)."""
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
