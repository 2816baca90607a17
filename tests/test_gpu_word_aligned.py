"""Buffers that are aligned to a word and not to 16 bytes, in launches of more rows
than the GPU holds at once (the transforms' kernels then ask L2 for later rows with
bulk prefetches): the results of the same call on aligned buffers, word for word."""
import pytest
import torch

from tests.gpu_util import small_pair

pytestmark = pytest.mark.gpu


def _put(x, shift):
    """a copy of x that starts `shift` words into a buffer; the buffer and the copy's address"""
    buf = torch.zeros(x.numel() + 2, dtype=torch.int64, device="cuda")
    buf[shift:shift + x.numel()] = x.view(-1)
    return buf, buf.data_ptr() + 8 * shift


def _words(shape, below, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(0, below, shape, dtype=torch.int64, device="cuda", generator=g)


# more whole rows or 2^12-point blocks than are resident at once
ROWS = [(10, 5200), (11, 2700), (12, 1300), (13, 620), (14, 310), (15, 170), (16, 90)]


@pytest.mark.parametrize("log_n,rows", ROWS)
def test_transforms(log_n, rows):
    from kunpbfv_b200.api import _check, lib
    ctx, _ = small_pair(log_n=log_n, nq=2, np_=1, bits=50)
    L, h = lib(), ctx.handle
    x = _words((rows, ctx.N), min(ctx.q), 1)
    want = x.clone()
    ctx.ntt_fwd(want, 0, 2)
    buf, p = _put(x, 1)
    _check(L.kbfv_ntt_fwd(h, p, rows, 0, 2, 0))
    assert torch.equal(buf[1:-1], want.view(-1))
    _check(L.kbfv_ntt_inv(h, p, rows, 0, 2, 0))
    assert torch.equal(buf[1:-1], x.view(-1))


@pytest.mark.parametrize("log_n,rows", ROWS)
@pytest.mark.parametrize("src,dst", [(1, 0), (0, 1), (1, 1)])
def test_encode_decode(log_n, rows, src, dst):
    from kunpbfv_b200.api import _check, lib
    ctx, _ = small_pair(log_n=log_n, nq=2, np_=1, bits=50)
    L, h = lib(), ctx.handle
    x = _words((rows, ctx.N), ctx.plain_modulus, 2)
    for call, aligned in ((L.kbfv_encode, ctx.encode), (L.kbfv_decode, ctx.decode)):
        want = aligned(x).view(-1)
        bx, px = _put(x, src)
        bo, po = _put(torch.zeros_like(x), dst)
        _check(call(h, px, po, rows, 0))
        assert torch.equal(bo[dst:dst + x.numel()], want)
        assert torch.equal(bx[src:src + x.numel()], x.view(-1)), "the input is not written"


# few rows (clusters, split and whole rows) and more than are resident at once
@pytest.mark.parametrize("log_n,pairs", [(10, 1), (12, 1), (12, 130), (13, 4), (14, 1), (14, 60), (15, 1), (15, 30),
                                         (16, 1)])
def test_tensor(log_n, pairs):
    """kbfv_mul with its inputs and its tensor word-aligned, each alone and both"""
    from kunpbfv_b200.api import _check, lib
    ctx, _ = small_pair(log_n=log_n, nq=2, np_=1, bits=50)
    L, h = lib(), ctx.handle
    a, b = (_words((pairs, 2, 2, ctx.N), min(ctx.q), s) for s in (3, 4))
    want = torch.empty(pairs * 3 * 2 * ctx.N, dtype=torch.int64, device="cuda")
    _check(L.kbfv_mul(h, a.data_ptr(), b.data_ptr(), want.data_ptr(), pairs, 0))
    for src, dst in ((0, 1), (1, 0), (1, 1)):
        (ba, pa), (bb, pb) = _put(a, src), _put(b, src)
        bo, po = _put(torch.zeros_like(want), dst)
        _check(L.kbfv_mul(h, pa, pb, po, pairs, 0))
        assert torch.equal(bo[dst:dst + want.numel()], want), (src, dst)
        assert not bo[:dst].any() and not bo[dst + want.numel():].any(), "nothing is written beside the tensor"
