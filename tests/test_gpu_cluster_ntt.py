"""Transforms of few rows run with one row over a cluster of CTAs: every ring
degree that has the form, at one row and on both sides of each limit of the rule
(the rows of a short last wave too, on a GPU of 148 SMs), forward against the oracle and back, with no synchronisation between
the launches (they start while the one before still runs); and a chain of calls
whose outputs the next call reads and overwrites at once."""
import numpy as np
import pytest

from tests.gpu_util import dev, host, make_pair, rand_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n,rows", [(12, 1), (12, 128), (12, 129), (13, 1), (13, 128), (13, 129),
                                        (14, 1), (14, 18), (14, 19), (14, 38), (14, 112), (14, 113), (14, 149), (14, 166), (14, 167),
                                        (14, 314), (14, 508), (14, 509), (15, 1), (15, 8), (15, 9)])
def test_few_rows(log_n, rows):
    import oracle
    ps = oracle.primes_bits(1 << log_n, 60, 4)
    ctx, orc = make_pair(log_n, ps[1:], ps[:1], 1)
    idx = [r % 3 for r in range(rows)]
    x = rand_rows(orc, idx, ctx.N, rows)
    x[0, :] = orc.primes[0] - 1
    d = dev(x)
    ctx.ntt_fwd(d, 0, 3)
    y = d.clone()
    ctx.ntt_inv(d, 0, 3)
    back, got = host(d).reshape(x.shape), host(y).reshape(x.shape)
    assert np.array_equal(back, x)
    for r in sorted({0, 1 % rows, rows // 2, rows - 1}):
        assert np.array_equal(got[r], orc.ntt_fwd(idx[r], x[r])), r


@pytest.mark.parametrize("log_n", [12, 13, 14, 15])
def test_chain_without_synchronisation(log_n):
    """square in place, decrypt, decode, 20 times over the same buffers: m^2 each time"""
    import kunpbfv_b200 as kb
    import oracle
    ps = oracle.primes_bits(1 << log_n, 60, 5)
    ctx = kb.BFVContext(log_n=log_n, plain_modulus=65537, q_count=4, q=ps[1:], p_count=1, p=ps[:1], dnum=4)
    sk = kb.SecretKey(ctx, bytes(32))
    sch = kb.BFVScheme(ctx, bytes(32))
    sch.addEncKey(sk)
    sch.addMultKey_23(sk)
    rng = np.random.default_rng(log_n)
    outs, want = [], []
    buf = kb.Ciphertext(ctx, count=1)
    for i in range(20):
        v = rng.integers(0, 65537, size=ctx.N, dtype=np.uint64)
        ct = sch.encryptMsg(kb.Plaintext(ctx, ctx.encode(dev(v))), enc_id=i)
        buf.cipher_device.view(-1).copy_(ct.cipher_device.view(-1))
        sch.squareAndEqual(buf)
        outs.append(ctx.decode(sch.decryptMsg(sk, buf).mx_device))
        want.append(v * v % 65537)
    for o, w in zip(outs, want):
        assert np.array_equal(host(o).reshape(-1), w)
