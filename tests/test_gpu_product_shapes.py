"""The multiply and the tensor alone against the oracle, word for word, where the
transforms of the base extension take their different shapes: whole 2^14-point rows,
few rows, every transform split, several digits on 2^13 points, and the column passes
of 2^15 and 2^16 points with 10 and 18 primes."""
import numpy as np
import pytest

import oracle
from tests.gpu_util import dev, host, make_pair, rand_rows
from tests.params import plain_modulus_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n,nq,np_,bits,dnum,pairs,split_rows", [
    (14, 7, 1, 60, 1, 5, 48),
    (14, 7, 1, 60, 1, 1, 48),
    (14, 7, 1, 60, 1, 3, 1 << 20),
    (13, 3, 1, 50, 3, 4, 48),
    (15, 10, 2, 55, 5, 2, 48),
    (16, 18, 2, 58, 3, 1, 48),
])
def test_product_and_tensor(log_n, nq, np_, bits, dnum, pairs, split_rows):
    import kunpbfv_b200 as kb
    ps = oracle.primes_bits(1 << log_n, bits, nq + np_)
    ctx, orc = make_pair(log_n, ps[np_:], ps[:np_], dnum, plain_modulus_for(log_n))
    n, q, qp = ctx.N, list(range(nq)), list(range(nq + np_))
    a, b = (np.stack([rand_rows(orc, q * 2, n, s + i) for i in range(pairs)]) for s in (10, 20))
    rlk = rand_rows(orc, qp * 2 * dnum, n, 30).reshape(dnum, 2, nq + np_, n)
    sch = kb.BFVScheme(ctx)
    sch.rlk = dev(rlk)
    ctx.tune_set("split_rows", split_rows)
    ca, cb = kb.Ciphertext(ctx, dev(a)), kb.Ciphertext(ctx, dev(b))
    got = host(sch.mult_relin(ca, cb).cipher_device).reshape(pairs, 2, nq, n)
    ten = host(sch.mult(ca, cb).data).reshape(pairs, 3, nq, n)
    for i in range(pairs):
        x, y = a[i].reshape(2, nq, n), b[i].reshape(2, nq, n)
        assert np.array_equal(got[i], orc.mul_relin(x, y, rlk)), i
        assert np.array_equal(ten[i], np.asarray(orc.mul_tensor(x, y)).reshape(3, nq, n)), i
