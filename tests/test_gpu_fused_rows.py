"""Encryption, plaintext addition, the modulus switch and the limb-wise operations
on every ring degree their fused transforms take (whole blocks of 2^10..2^14 and
the column passes of 2^15 and 2^16), across the 128-item chunk, in place and out
of place, and on pointers that are only 8-byte aligned: equal to the oracle, or
to the same items alone, bit for bit."""
import numpy as np
import pytest

from tests.gpu_util import dev, host, make_pair, rand_rows

pytestmark = pytest.mark.gpu

SEED = bytes(range(3, 35))


def _scheme(log_n, nq=2, bits=50):
    import kunpbfv_b200 as kb
    import oracle
    ps = oracle.primes_bits(1 << log_n, bits, nq + 1)
    ctx, orc = make_pair(log_n, ps[1:], ps[:1], 1)
    sk = kb.SecretKey(ctx, SEED)
    sch = kb.BFVScheme(ctx, SEED)
    sch.addEncKey(sk)
    return ctx, orc, sk, sch


@pytest.mark.parametrize("log_n", [10, 11, 12, 13, 14, 15, 16])
def test_encrypt_add_plain_mod_switch(log_n):
    import kunpbfv_b200 as kb
    ctx, orc, sk, sch = _scheme(log_n)
    n, nq, t = ctx.N, ctx.q_count, ctx.plain_modulus
    rng = np.random.default_rng(log_n)
    m = rng.integers(0, t, size=(2, n), dtype=np.uint64)
    m[0, :8] = [0, 1, t - 1, t // 2, t // 2 + 1, 2, t - 2, 0]
    osk = orc.keygen_secret(SEED)
    opk = orc.keygen_public(SEED, osk)
    ct = sch.encryptMsg(kb.Plaintext(ctx, dev(m)), enc_id=9)
    got = host(ct.cipher_device).reshape(2, 2, nq, n)
    want = np.stack([np.asarray(orc.encrypt(SEED, 9 + i, opk, m[i])).reshape(2, nq, n) for i in range(2)])
    assert np.array_equal(got, want)
    # b += NTT(delta m), in place and into another ciphertext
    from kunpbfv_b200.api import _check, _ptr, lib
    sp = 0
    out = kb.Ciphertext(ctx, count=2)
    _check(lib().kbfv_add_plain(ctx.handle, _ptr(ct.cipher_device), _ptr(dev(m)), _ptr(out.cipher_device), 2, sp))
    dm = host(ctx.delta_m(dev(m))).reshape(2, nq, n)
    x = dev(dm.reshape(2 * nq, n))
    ctx.ntt_fwd(x, 0, nq)
    q = np.array(ctx.q, dtype=np.uint64)[:, None]
    plus = want.copy()
    plus[:, 1] = (plus[:, 1] + host(x).reshape(2, nq, n)) % q
    assert np.array_equal(host(out.cipher_device).reshape(2, 2, nq, n), plus)
    sch.addConstAndEqual(ct, kb.Plaintext(ctx, dev(m)))
    assert np.array_equal(host(ct.cipher_device).reshape(2, 2, nq, n), plus)
    low = sch.mod_switch(ct)
    sw = np.stack([np.asarray(orc.mod_switch(plus[i])).reshape(2, nq - 1, n) for i in range(2)])
    assert np.array_equal(host(low.cipher_device).reshape(2, 2, nq - 1, n), sw)


def test_more_items_than_one_chunk():
    """131 items: the second chunk's ids, plaintexts and outputs; item 130 alone is the same"""
    import kunpbfv_b200 as kb
    ctx, orc, sk, sch = _scheme(10)
    rng = np.random.default_rng(5)
    m = rng.integers(0, ctx.plain_modulus, size=(131, ctx.N), dtype=np.uint64)
    ct = sch.encryptMsg(kb.Plaintext(ctx, dev(m)), enc_id=2 ** 33 - 3)
    all_ = host(ct.cipher_device).reshape(131, -1)
    for i in (0, 127, 128, 130):
        one = sch.encryptMsg(kb.Plaintext(ctx, dev(m[i:i + 1])), enc_id=2 ** 33 - 3 + i)
        assert np.array_equal(host(one.cipher_device).reshape(-1), all_[i]), i
    assert np.array_equal(host(sch.decryptMsg(sk, ct).mx_device).reshape(131, -1), m)


@pytest.mark.parametrize("shift", [0, 1])
def test_linear_ops_alignment(shift):
    """add, sub, negate, scalar products and plaintext products on 16- and 8-byte aligned buffers"""
    import torch

    from kunpbfv_b200.api import _check, lib
    ctx, orc, sk, sch = _scheme(10, nq=3)
    n, nq, count = ctx.N, ctx.q_count, 3
    rows = list(range(nq)) * 2 * count
    x, y = rand_rows(orc, rows, n, 1), rand_rows(orc, rows, n, 2)
    p = rand_rows(orc, list(range(nq)) * count, n, 3)

    def put(a):
        buf = torch.zeros(a.size + 1, dtype=torch.int64, device="cuda")
        buf[shift:shift + a.size] = dev(a).view(-1)
        return buf, buf.data_ptr() + 8 * shift

    (bx, px), (by, py), (bp, pp), (bo, po) = put(x), put(y), put(p), put(np.zeros_like(x))
    q = [ctx.primes[i] for i in rows]
    big = lambda f: np.array([[f(int(a), int(b), m) for a, b in zip(r, s)] for r, s, m in zip(x, y, q)], dtype=np.uint64)
    L, h, k = lib(), ctx.handle, 0x123456789abcdef

    def check(want):
        assert np.array_equal(host(bo[shift:shift + x.size]).reshape(x.shape), want)

    _check(L.kbfv_add(h, px, py, po, count, 0)); check(big(lambda a, b, m: (a + b) % m))
    _check(L.kbfv_sub(h, px, py, po, count, 0)); check(big(lambda a, b, m: (a - b) % m))
    _check(L.kbfv_negate(h, px, po, count, 0)); check(big(lambda a, b, m: -a % m))
    _check(L.kbfv_mul_scalar(h, px, k, po, count, 0)); check(big(lambda a, b, m: a * k % m))
    bo.copy_(by)
    _check(L.kbfv_mul_scalar_add(h, px, k, po, count, 0)); check(big(lambda a, b, m: (b + a * k) % m))
    _check(L.kbfv_mul_plain(h, px, pp, po, count, 0))
    pr = p.reshape(count, 1, nq, n).repeat(2, axis=1).reshape(x.shape)
    check(np.array([[int(a) * int(b) % m for a, b in zip(r, s)] for r, s, m in zip(x, pr, q)], dtype=np.uint64))
