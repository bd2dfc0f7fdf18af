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


@pytest.mark.parametrize("kind", ["int16", "int32", "f32", "f64"])
@pytest.mark.parametrize("outputs", ["phi", "i", ""])
def test_small_host_calls_of_wider_types(capi, kind, outputs):
    """Either side of 256 KB for each element type, against the same LLRs
    decoded from device memory."""
    import torch
    from ldpc_b200 import codes
    code = codes.make_code("11ad 1/2")
    variant, dt, clamp, beta = {"int16": (capi.LDPC_INT16_OMS, torch.int16, 31.0, 1.0),
                                "int32": (capi.LDPC_INT32_OMS, torch.int32, 31.0, 1.0),
                                "f32": (capi.LDPC_F32_SP, torch.float32, 6e-8, 0.0),
                                "f64": (capi.LDPC_F64_OMS, torch.float64, 31.0, 0.5)}[kind]
    ctx = capi.Context(capi.Code.from_tables(code), variant=variant, max_iter=10, max_row_metric=clamp, beta=beta,
                       llr_scale=2.0, max_abs_llr=24.0)
    es = torch.empty(0, dtype=dt).element_size()
    limit = (262144 - 1024) // (code.n * es * (2 if "p" in outputs else 1) + (44 if "h" in outputs else 0) + 1)
    for n in (1, 17, limit - 1, limit, limit + 1):
        llr = torch.empty((1, n, code.n), dtype=dt, device="cuda")
        ctx.generate(n, 0, [-0.75], n, **({"llr_f32": llr} if kind == "f32" else {"llr_int": llr}))
        p, it = torch.empty_like(llr), torch.empty(n, dtype=torch.uint8, device="cuda")
        h = torch.empty((n, 11), dtype=torch.int32, device="cuda")
        getattr(ctx, "decode_" + kind)(llr, n, post=p, hard=h, iters=it)
        host = llr.cpu().numpy()
        post = np.zeros_like(host) if "p" in outputs else None
        hard = np.zeros((n, 11), np.int32) if "h" in outputs else None
        iters = np.zeros(n, np.uint8) if "i" in outputs else None
        tot = C.c_uint64()
        capi.check(getattr(capi.lib, "ldpc_decode_%s_host" % kind)(ctx.h, host.ctypes.data, n, capi._ptr(post),
                                                                   capi._ptr(hard), capi._ptr(iters), C.byref(tot)))
        assert tot.value == int(it.sum(dtype=torch.int64))
        assert post is None or np.array_equal(post.view(np.uint8), p.cpu().numpy().view(np.uint8))
        assert hard is None or np.array_equal(hard, h.cpu().numpy())
        assert iters is None or np.array_equal(iters, it.cpu().numpy())


@pytest.mark.parametrize("where", ["pinned", "pinned in", "pinned out", "device", "device in", "device out"])
@pytest.mark.parametrize("n", [1, 40, 60, 187])
def test_small_host_calls_from_other_memory(capi, n, where):
    """Page-locked buffers on either side of the size up to which they are moved
    by memcpy (32 KB: 48 codewords' LLRs), and device memory given as a host buffer, which is
    an error or decodes as from the host, but is not touched by it."""
    import torch
    from ldpc_b200 import codes
    code = codes.make_code("11ad 1/2")
    ctx = capi.Context(capi.Code.from_tables(code))
    llr = torch.empty((1, n, code.n), dtype=torch.int8, device="cuda")
    ctx.generate(n, 0, [-0.75], n, llr_int=llr)
    want = (torch.empty_like(llr), torch.empty((n, 11), dtype=torch.int32, device="cuda"),
            torch.empty(n, dtype=torch.uint8, device="cuda"))
    ctx.decode_int8(llr, n, post=want[0], hard=want[1], iters=want[2])
    torch.cuda.synchronize()
    kind, _, part = where.partition(" ")
    other = (lambda t: t.pin_memory()) if kind == "pinned" else (lambda t: t.cuda())
    src = llr.cpu() if part == "out" else other(llr.cpu())
    outs = [torch.zeros_like(t, device="cpu") if part == "in" else other(torch.zeros_like(t, device="cpu")) for t in want]
    torch.cuda.synchronize()
    for some in ((0, 1, 2), (1, 2), (0,), ()):
        for t in outs:
            t.zero_()
        torch.cuda.synchronize()
        tot = C.c_uint64()
        ptr = [outs[i].data_ptr() if i in some else None for i in range(3)]
        rc = capi.lib.ldpc_decode_int8_host(ctx.h, src.data_ptr(), n, *ptr, C.byref(tot))
        if kind == "device" and rc == capi.LDPC_ERR_CUDA:
            # the context stays usable
            got = ctx.decode_host(llr[0].cpu().numpy())
            assert np.array_equal(got[0], want[0][0].cpu().numpy())
            continue
        capi.check(rc)
        assert tot.value == int(want[2].sum(dtype=torch.int64))
        for i in some:
            assert torch.equal(outs[i].cpu(), want[i].cpu())
