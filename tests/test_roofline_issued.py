"""What the multiply's kernels issue per pair (kunpbfv_b200.roofline), counted by hand
from csrc/: pipeline.cuh (TensorRow, KeyIPRow, ModDownKeyRow, OutKeyRow), key_ip.cuh,
limb_mma.cuh (mma_value), k5_kernels.cuh (lift_word) and mul.cu (CPU only)."""
import pytest

from kunpbfv_b200 import roofline as rl


@pytest.mark.parametrize("nq,np_,dnum,prod,mac,b128,shoup,shoup4,outputs,words", [
    # one digit: K4 2 x 15 prod, 30 mac, 15 shoup; the lift's 7 shoup; key 2 x 8 prod; mod down 14 and P^-1 14
    # shoup4; outputs K2 32, K5 24 + 21, lift 1; words 8 a sum over Q and its quotient, 9 over R
    (7, 1, 1, 30 + 16, 30, 0, 15 + 7, 14 + 14, 32 + 24 + 21 + 1, 32 * 8 + 24 * 8 + 21 * 9 + 8),
    # digits of 5, 5 and 4 of 14 primes, two special primes
    (14, 2, 3, 58, 58 + 2 * 16 * 3, 2 * 16, 29 + 14, 2 * 14 * 2 + 2 * 14, 60 + 45 + 42 + 11 + 11 + 12,
     60 * 15 + 45 * 15 + 42 * 16 + 6 * 11 + 6 * 11 + 5 * 12),
    # a digit per prime: no lift; the key products apart, scaled by a full product
    (7, 1, 7, 30, 30 + 2 * 8 * 7, 2 * 8, 15 + 14, 14, 77, 32 * 8 + 24 * 8 + 21 * 9),
])
def test_issued_counts(nq, np_, dnum, prod, mac, b128, shoup, shoup4, outputs, words):
    n, log_n = 16384, 14
    pc = rl.pipeline_counts(n, log_n, nq, np_, dnum)
    got = pc["issued"]
    assert got["bfly"] == pc["ntt_rows"] * (n // 2) * log_n
    want = {"prod": prod, "mac": mac, "b128": b128, "shoup": shoup, "shoup4": shoup4, "hi32": outputs,
            "wide32": outputs, "lo32": outputs}
    assert {k: got[k] / n for k in want} == want
    assert pc["byte_macs"] == 64 * words * n
    assert pc["issued_products"] == got["bfly"] + n * (prod + mac + shoup + shoup4)


def test_floor_takes_the_slower_unit():
    pc = rl.pipeline_counts(16384, 14, 7, 1, 1)
    rates = {k: 1e12 for k in rl.PROBE_KIND}
    assert rl.step_floor_s(pc, rates) == pytest.approx(sum(pc["issued"].values()) / 1e12)
    fast = {k: 1e30 for k in rl.PROBE_KIND}
    assert rl.step_floor_s(pc, fast) == pc["byte_macs"] / rl.IMMA_MACS


def test_an_empty_digit_is_not_negative():
    per, _ = rl.issued_per_coefficient(5, 1, 4)  # digits of 2, 2, 1 and 0 primes
    assert per["shoup"] == 11 + 5 + 10  # K4, the lift, the scaled key products
