"""kbfv_add_plain where its buffers share memory: plaintexts that lie inside the output,
and an output shifted by one ciphertext against its input: the words of the call on
separate buffers."""
import pytest
import torch

from tests.gpu_util import small_pair

pytestmark = pytest.mark.gpu


def _words(shape, below, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(0, below, shape, dtype=torch.int64, device="cuda", generator=g)


# few rows on clusters, more rows than are resident at once, a split ring
@pytest.mark.parametrize("log_n,count", [(12, 3), (12, 128), (14, 9), (15, 3), (15, 70)])
def test_shared_buffers(log_n, count):
    from kunpbfv_b200.api import _check, lib
    ctx, _ = small_pair(log_n=log_n, nq=2, np_=1, bits=50)
    n, nq = ctx.N, ctx.q_count
    item = 2 * nq * n
    ct = _words((count * item,), min(ctx.q), 1)
    m = _words((count * n,), ctx.plain_modulus, 2)
    want = torch.empty_like(ct)

    def add(c, p, o):
        _check(lib().kbfv_add_plain(ctx.handle, c, p, o, count, 0))

    add(ct.data_ptr(), m.data_ptr(), want.data_ptr())
    for at in (0, nq * n, (count - 1) * item // 2):  # the plaintexts inside the output
        out = torch.zeros_like(ct)
        out[at:at + m.numel()] = m
        add(ct.data_ptr(), out.data_ptr() + 8 * at, out.data_ptr())
        assert torch.equal(out, want), at
    buf = torch.zeros((count + 1) * item, dtype=torch.int64, device="cuda")
    buf[item:] = ct  # the output one ciphertext before the input
    add(buf.data_ptr() + 8 * item, m.data_ptr(), buf.data_ptr())
    assert torch.equal(buf[:count * item], want)
    inplace = ct.clone()
    add(inplace.data_ptr(), m.data_ptr(), inplace.data_ptr())
    assert torch.equal(inplace, want)
