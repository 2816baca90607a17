"""The external product over the T base of more items than one launch of the key
products takes (65535 groups of four): the items at both ends and around the launches'
border are the same as in small calls."""
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def test_more_items_than_one_launch():
    import kunpbfv_b200 as kb
    ps = sorted(oracle.primes_bits(1 << 10, 50, 3))  # the R primes lie below q
    ctx = kb.BFVContext(log_n=10, plain_modulus=65537, q_count=1, q=ps[:1], p_count=1, p=ps[1:2], dnum=1,
                        t_primes=ps[2:], gamma=2)
    nri, nqj, _ = ctx.klss_info()
    items, n = 65535 * 4 + 5, ctx.N
    g = torch.Generator(device="cuda").manual_seed(1)
    rand = lambda *s: torch.randint(0, ps[2], s, dtype=torch.int64, device="cuda", generator=g)
    dig, key = rand(items, nqj, 1, n), rand(2, nqj, nri, 1, n)
    got = ctx.klss_external_product(dig, key)
    for at in (0, 65535 * 4 - 3, items - 5):
        assert torch.equal(got[at:at + 5], ctx.klss_external_product(dig[at:at + 5].contiguous(), key)), at
