"""Host-buffer decoding around the size up to which a call goes through one
pinned buffer (256 KB in and out): 187 codewords of 802.11ad 1/2 with all
outputs are below it, 188 and 189 above."""
import ctypes as C

import numpy as np
import pytest

from conftest import make_llr_int8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 149, 187, 188, 189, 400])
@pytest.mark.parametrize("outputs", ["phi", "h", "i", "p", ""])
def test_small_and_large_host_calls(capi, oracle, n, outputs):
    from ldpc_b200 import codes
    code = codes.make_code("11ad 1/2")
    llr, _, _ = make_llr_int8(code, n, -0.75, seed=n, oracle=oracle)
    ctx = capi.Context(capi.Code.from_tables(code))
    post = np.zeros_like(llr) if "p" in outputs else None
    hard = np.zeros((n, 11), np.uint32) if "h" in outputs else None
    iters = np.zeros(n, np.uint8) if "i" in outputs else None
    tot = C.c_uint64()
    for _ in range(2):
        capi.check(capi.lib.ldpc_decode_int8_host(ctx.h, llr.ctypes.data, n, capi._ptr(post), capi._ptr(hard),
                                                  capi._ptr(iters), C.byref(tot)))
        post_o, it_o = oracle.decode_int8(code, llr, 10, 31.0, 1.0)
        assert tot.value == it_o.sum()
        assert post is None or np.array_equal(post, post_o)
        assert iters is None or np.array_equal(iters, it_o)
        if hard is not None:
            bits = np.unpackbits(hard.view(np.uint8), axis=1, bitorder="little")[:, :336]
            assert np.array_equal(bits, (post_o[:, :336] < 0).astype(np.uint8))
