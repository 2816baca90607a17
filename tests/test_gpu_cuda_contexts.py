"""The multiply and the transforms in a second CUDA context of the process: kernels
whose shared memory exceeds 48 KB have to be allowed it in each context (another
GPU's, or as here another one on the same GPU), not once per process. The products
are those of the first context."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes as C
import sys

import numpy as np

import kunpbfv_b200 as kb
from kunpbfv_b200.api import _check

log_n, nq, pairs, rows = (int(x) for x in sys.argv[1:5])
cu = C.CDLL("libcuda.so.1")


def ck(rc):
    assert rc == 0, f"driver error {rc}"


ck(cu.cuInit(0))
dev = C.c_int()
ck(cu.cuDeviceGet(C.byref(dev), 0))
L = kb.lib()


def put(x):
    p = C.c_void_p()
    ck(cu.cuMemAlloc_v2(C.byref(p), C.c_size_t(x.nbytes)))
    ck(cu.cuMemcpyHtoD_v2(p, x.ctypes.data_as(C.c_void_p), C.c_size_t(x.nbytes)))
    return p


def get(p, words):
    x = np.empty(words, dtype=np.uint64)
    ck(cu.cuCtxSynchronize())
    ck(cu.cuMemcpyDtoH_v2(x.ctypes.data_as(C.c_void_p), p, C.c_size_t(x.nbytes)))
    return x


def run():
    ctx = kb.BFVContext.from_bits(log_n, [60] * nq, [60], 65537, dnum=1)
    n, rng = ctx.N, np.random.default_rng(1)
    low = min(ctx.primes[:-1])
    draw = lambda *shape: rng.integers(0, low, size=shape, dtype=np.uint64)
    key, a, b = draw(2 * (nq + 1) * n), draw(pairs * 2 * nq * n), draw(pairs * 2 * nq * n)
    out = put(np.zeros_like(a))
    _check(L.kbfv_mul_relin(ctx.handle, put(key), put(a), put(b), out, pairs, None))
    res = [get(out, a.size)]
    x = put(draw(rows * n))
    _check(L.kbfv_ntt_fwd(ctx.handle, x, rows, 0, nq, None))
    res.append(get(x, rows * n))
    _check(L.kbfv_ntt_inv(ctx.handle, x, rows, 0, nq, None))
    res.append(get(x, rows * n))
    return ctx, res


done = []
for i in range(2):
    c = C.c_void_p()
    ck(cu.cuCtxCreate_v2(C.byref(c), 0, dev))  # made current
    done.append(run())
assert all(np.array_equal(x, y) for x, y in zip(done[0][1], done[1][1]))
print("same products in both contexts")
"""


@pytest.mark.parametrize("log_n,nq,pairs,rows", [
    (12, 14, 2, 4),      # base extension, scale-and-round: more than 48 KB from 8 primes on
    (12, 32, 1, 4),
    (13, 3, 2, 400),     # blocks of 2^13 points
    (14, 3, 2, 310),     # and of 2^14
])
def test_second_context(log_n, nq, pairs, rows):
    r = subprocess.run([sys.executable, "-c", CHILD, *map(str, (log_n, nq, pairs, rows))], cwd=ROOT,
                       env=dict(os.environ, PYTHONPATH=ROOT), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same products" in r.stdout, r.stdout + r.stderr
