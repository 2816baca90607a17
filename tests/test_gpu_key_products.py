"""Key switches of four digits and more, whose products with the key are summed
by a kernel of their own: every number of items that a thread takes (1..4, and
groups with a short last one), the smallest ring and split ones, the added term on
both halves (relinearisation) and on one (rotation), and a level's live primes of
the top level's key, against the oracle, bit for bit."""
import numpy as np
import pytest

from tests.gpu_util import dev, host, make_pair, rand_rows

pytestmark = pytest.mark.gpu

SEED = bytes(range(5, 37))


def _relinearize(ctx, rlk, tensors):
    import torch
    from kunpbfv_b200.api import _check, _ptr, _stream_ptr, lib
    out = torch.full((len(tensors), 2, ctx.q_count, ctx.N), -1, dtype=torch.int64, device="cuda")
    d, k = dev(tensors), dev(rlk)
    _check(lib().kbfv_relinearize(ctx.handle, _ptr(k), _ptr(d), _ptr(out), len(tensors), _stream_ptr(None)))
    return host(out).reshape(len(tensors), 2, ctx.q_count, ctx.N)


@pytest.mark.parametrize("log_n,nq,np_,dnum,items", [(10, 4, 1, 4, 1), (12, 5, 1, 5, 2), (13, 8, 2, 4, 3), (14, 7, 1, 7, 4),
                                                     (12, 7, 1, 7, 5), (15, 4, 1, 4, 9), (12, 3, 1, 3, 5)])
def test_relinearize_digits(log_n, nq, np_, dnum, items):
    import oracle
    ps = oracle.primes_bits(1 << log_n, 60, nq + np_)
    ctx, orc = make_pair(log_n, ps[np_:], ps[:np_], dnum)
    n, npq = ctx.N, nq + np_
    rlk = rand_rows(orc, list(range(npq)) * 2 * dnum, n, 1).reshape(dnum, 2, npq, n)
    d = rand_rows(orc, list(range(nq)) * 3 * items, n, 2).reshape(items, 3, nq, n)
    top = np.array(orc.primes[:npq], dtype=np.uint64) - 1
    rlk[:, :, :, 0] = top          # the largest residues throughout
    d[:, :, :, 0] = top[:nq]
    got = _relinearize(ctx, rlk, d)
    for i in sorted({0, items // 2, items - 1}):
        assert np.array_equal(got[i], orc.relinearize(d[i], rlk)), i


def test_rotation_and_level():
    import kunpbfv_b200 as kb
    import oracle
    T = 65537
    ps = oracle.primes_bits(1 << 12, 50, 10)
    q, p = ps[2:], ps[:2]
    ctx, top = make_pair(12, q, p, 4)
    sk = kb.SecretKey(ctx, SEED)
    sch = kb.BFVScheme(ctx, SEED)
    sch.addEncKey(sk)
    sch.addMultKey_23(sk)
    sch.addLeftRotKey_23(sk, 1)
    osk = top.keygen_secret(SEED)
    g = sch.galois_element(1)
    ogk = top.keygen_galois(SEED, osk, g)
    orlk = top.keygen_relin(SEED, osk)
    v = np.random.default_rng(4).integers(0, T, size=(5, ctx.N), dtype=np.uint64)
    ct = sch.encryptMsg(kb.Plaintext(ctx, ctx.encode(dev(v))), enc_id=3)
    h = host(ct.cipher_device).reshape(5, 2, 8, ctx.N)
    got = host(sch.apply_galois(ct, g).cipher_device).reshape(h.shape)
    for i in (0, 4):
        assert np.array_equal(got[i], top.apply_galois(ogk, g, h[i])), i
    c7 = sch.mod_switch(ct)  # 7 live primes: digits 2, 2, 2, 1
    o7 = oracle.Oracle(12, T, q[:7], p, alpha=2)
    rl = np.stack([np.stack([np.concatenate([orlk[d][k][:7], orlk[d][k][8:]]) for k in range(2)]) for d in range(o7.dnum)])
    assert o7.dnum == 4
    h7 = host(c7.cipher_device).reshape(5, 2, 7, ctx.N)
    sq = host(sch.mult_relin(c7, c7).cipher_device).reshape(5, 2, 7, ctx.N)
    for i in (0, 4):
        assert np.array_equal(sq[i], o7.mul_relin(h7[i], h7[i], rl)), i


@pytest.mark.parametrize("log_n,q_bits,p_bits", [(10, [50], 52), (12, [60, 60, 60], 60), (13, [60, 36, 60, 36], 60),
                                                 (14, [36, 60], 36), (15, [30, 59, 45], 60)])
def test_one_prime_digits_near_the_modulus(log_n, q_bits, p_bits):
    """Digits of one prime whose coefficients lie where the single-precision
    quotient x / q rounds to 1 or just does not, over primes of unequal sizes."""
    import oracle
    pool = {b: oracle.primes_bits(1 << log_n, b, 5) for b in set(q_bits) | {p_bits}}
    qs = [pool[b].pop() for b in q_bits]
    p = [pool[p_bits].pop()]
    nq = len(qs)
    ctx, orc = make_pair(log_n, qs, p, nq)
    n, npq = ctx.N, nq + 1
    rlk = rand_rows(orc, list(range(npq)) * 2 * nq, n, 1).reshape(nq, 2, npq, n)
    d = rand_rows(orc, list(range(nq)) * 3 * 2, n, 2).reshape(2, 3, nq, n)
    for l, q in enumerate(qs):
        near = [q - 1 - i for i in range(8)]
        for s in (22, 23, 24, 25, 26):
            near += [q - 1 - (q >> s) + i for i in range(-2, 3)]
        # every midpoint between singles near q, and its neighbours
        f = np.float32(q)
        for _ in range(3):
            g = np.nextafter(f, np.float32(0))
            mid = (int(f) + int(g)) // 2
            near += [mid + i for i in (-1, 0, 1)]
            f = g
        near = np.array([v for v in near if 0 <= v < q], dtype=np.uint64)
        x = d[0, 0, l].copy()
        x[:len(near)] = near
        d[0, 0, l] = orc.ntt_fwd(l, x)
    got = _relinearize(ctx, rlk, d)
    for i in range(2):
        assert np.array_equal(got[i], orc.relinearize(d[i], rlk)), i


def test_t_base_blocks_of_one_prime_near_the_modulus():
    """The T-base key switch whose blocks are one prime each (lifted by the
    transform's loads) equals its pieces called one by one (lifted by the block
    kernel), on coefficients where the quotient estimate is 1 or just not."""
    import torch
    import kunpbfv_b200 as kb
    from kunpbfv_b200.api import _check, _ptr, _stream_ptr, lib
    ctx = kb.reference_context(15)
    assert ctx.p_count == 1
    n, nq, nt = ctx.N, ctx.q_count, ctx.t_count
    nri, nqj, words = ctx.klss_info()
    rng = np.random.default_rng(8)
    count = 2
    x = np.stack([np.stack([rng.integers(0, q, size=n, dtype=np.uint64) for q in ctx.q]) for _ in range(count)])
    for l, q in enumerate(ctx.q):
        near = [q - 1 - i for i in range(8)] + [q - 1 - (q >> s) + i for s in (22, 23, 24, 25, 26) for i in range(-2, 3)]
        f = np.float32(q)
        for _ in range(3):
            g = np.nextafter(f, np.float32(0))
            near += [v for v in ((int(f) + int(g)) // 2 + i for i in (-1, 0, 1)) if v < q]
            f = g
        x[0, l, :len(near)] = np.array(near, dtype=np.uint64)
    key = torch.stack([dev(rng.integers(0, int(ctx.tk[r % nt]), size=n, dtype=np.uint64)) for r in range(words // n)])
    dig = ctx.klss_modup_qj_to_t(dev(x))
    ctx.ntt_fwd(dig, ctx.idx_t, nt)
    z = host(ctx.klss_t_to_pq(ctx.klss_external_product(dig, key))).reshape(count, 2, nq + 1, n)
    want = np.empty((count, 2, nq, n), dtype=np.uint64)
    p = int(ctx.p[0])
    for l, q in enumerate(ctx.q):
        inv = pow(p, -1, int(q))
        diff = (z[:, :, l].astype(object) - z[:, :, nq].astype(object)) * inv % int(q)
        want[:, :, l] = diff.astype(np.uint64)
    wd = dev(want)
    ctx.ntt_fwd(wd, 0, nq)
    d = np.zeros((count, 3, nq, n), dtype=np.uint64)
    d[:, 0] = x
    dd = dev(d)
    ctx.ntt_fwd(dd, 0, nq)
    out = torch.full((count, 2, nq, n), -1, dtype=torch.int64, device="cuda")
    _check(lib().kbfv_relinearize_klss(ctx.handle, _ptr(key), _ptr(dd), _ptr(out), count, _stream_ptr(None)))
    assert np.array_equal(host(out).reshape(want.shape), host(wd).reshape(want.shape))
