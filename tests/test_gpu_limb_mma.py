"""The byte matrix products of the base conversions (csrc/limb_mma.cuh) at the
edges of their shapes: prime counts on both sides of every step count, digit
sizes on both sides of the lift's, one-prime and empty digits, prime sizes from
24 to 60 bits, and residues that are 0 or q - 1 everywhere (the largest digit
sums). Exact integers: equal to the oracle bit for bit."""
import numpy as np
import pytest

from tests.gpu_util import dev, host, make_pair, rand_rows

pytestmark = pytest.mark.gpu

LOG_N = 10


def _pair(nq, np_, bits, dnum):
    import oracle
    ps = oracle.primes_bits(1 << LOG_N, bits, nq + np_)
    return make_pair(LOG_N, ps[np_:], ps[:np_], dnum)


def _rows(orc, idxs, n, seed):
    """per row: random residues, with zeros and q - 1 in whole runs of coefficients"""
    x = rand_rows(orc, idxs, n, seed)
    for r, i in enumerate(idxs):
        x[r, : n // 8] = 0
        x[r, n // 8: n // 4] = orc.primes[i] - 1
    return x


@pytest.mark.parametrize("nq,np_,bits,dnum", [
    (1, 1, 60, 1), (3, 1, 24, 3), (4, 1, 60, 4), (7, 1, 60, 1), (8, 2, 45, 2),
    (5, 1, 50, 4),    # alpha 2: the fourth digit is empty
    (15, 2, 60, 3), (16, 1, 60, 1), (17, 3, 55, 1), (23, 1, 60, 12), (24, 8, 60, 3), (32, 8, 60, 1), (32, 1, 60, 32),
])
def test_multiply_and_conversions(nq, np_, bits, dnum):
    import kunpbfv_b200 as kb
    ctx, orc = _pair(nq, np_, bits, dnum)
    n, q = ctx.N, list(range(nq))
    r = list(range(ctx.idx_r, ctx.idx_r + ctx.r_count))
    x, z = _rows(orc, q, n, 1), _rows(orc, r, n, 2)
    for cpt in (2, 1):
        ctx.tune_set("bconv_cpt", cpt)
        assert np.array_equal(host(ctx.bconv_q_to_r(dev(x))).reshape(-1, n), orc.bconv_q_to_r(x))
        assert np.array_equal(host(ctx.bconv_r_to_q(dev(z))).reshape(-1, n), orc.bconv_r_to_q(z))
    pairs = 3
    a = np.stack([_rows(orc, q + q, n, 10 + i) for i in range(pairs)])
    b = np.stack([_rows(orc, q + q, n, 20 + i) for i in range(pairs)])
    key = rand_rows(orc, (q + list(range(nq, nq + np_))) * 2 * ctx.dnum, n, 30)
    sch = kb.BFVScheme(ctx)
    sch.rlk = dev(key)
    rlk = key.reshape(ctx.dnum, 2, nq + np_, n)
    want = [orc.mul_relin(a[i].reshape(2, nq, n), b[i].reshape(2, nq, n), rlk) for i in range(pairs)]
    ca, cb = kb.Ciphertext(ctx, dev(a)), kb.Ciphertext(ctx, dev(b))
    got = host(sch.mult_relin(ca, cb).cipher_device).reshape(pairs, 2, nq, n)
    two = host(sch.relinearize(sch.mult(ca, cb)).cipher_device).reshape(pairs, 2, nq, n)
    for i in range(pairs):
        assert np.array_equal(got[i], want[i]), i
        assert np.array_equal(two[i], want[i]), i


def test_conversions_of_unaligned_rows():
    """pointers that are only 8-byte aligned"""
    import torch

    from kunpbfv_b200.api import _check, lib
    ctx, orc = _pair(5, 1, 60, 1)
    x = _rows(orc, range(5), ctx.N, 3)
    src = torch.zeros(5 * ctx.N + 1, dtype=torch.int64, device="cuda")
    src[1:] = dev(x).view(-1)
    out = torch.zeros(6 * ctx.N + 1, dtype=torch.int64, device="cuda")
    sp = torch.cuda.current_stream().cuda_stream
    _check(lib().kbfv_bconv_q_to_r(ctx.handle, src.data_ptr() + 8, out.data_ptr() + 8, 1, sp))
    assert np.array_equal(host(out[1:]).reshape(6, -1), orc.bconv_q_to_r(x))
