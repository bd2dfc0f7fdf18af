"""Decodes of one context that overlap on the device: the chunks of a host call
with page-locked buffers, calls on two streams, and a captured call replayed
beside a direct one.  The codes keep their check messages in global memory;
every output is compared with that of one launch on one stream."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# name, variant, max_row_metric, beta, SNR, codewords in 64 MiB of LLRs
CASES = {
    "int8": ("5GNR_n25344_k8448", "LDPC_INT8_OMS", 31.0, 1.0, -4.6, 2570),
    "int16": ("5GNR_n6400_k1280", "LDPC_INT16_OMS", 31.0, 1.0, -6.9, 5041),
    "int32": ("5GNR_n6400_k1280", "LDPC_INT32_OMS", 31.0, 1.0, -6.9, 2520),
    "f32_min_sum": ("11ay 1/2", "LDPC_F32_OMS", 31.0, 0.5, -1.5, 12483),
    "f64_min_sum": ("11ad 1/2", "LDPC_F64_OMS", 31.0, 0.5, -1.5, 12483),
    "f32_sum_product": ("5GNR_n6400_k1280", "LDPC_F32_SP", 6e-8, 0.0, -6.9, 2520),
}


def _setup(capi, kind, n, max_iter, seed=3):
    """Context, LLRs on the device."""
    import torch
    from ldpc_b200 import codes
    name, variant, clamp, beta, snr, _ = CASES[kind]
    code = codes.code_by_name(name)
    ctx = capi.Context(capi.Code.from_tables(code), variant=getattr(capi, variant), max_iter=max_iter,
                       max_row_metric=clamp, beta=beta, llr_scale=2.0, max_abs_llr=24.0)
    dt = {"int8": torch.int8, "int16": torch.int16, "int32": torch.int32, "f32": torch.float32,
          "f64": torch.float64}[kind.split("_")[0]]
    llr = torch.empty((1, n, code.n), dtype=dt, device="cuda")
    ctx.generate(seed, 0, [snr], n, **({"llr_f32": llr} if dt == torch.float32 else {"llr_int": llr}))
    torch.cuda.synchronize()
    return ctx, llr[0]


def _decode(ctx, kind, llr, stream):
    import torch
    n = len(llr)
    post = torch.empty_like(llr)
    hard = torch.empty((n, ctx.info.hard_words), dtype=torch.int32, device="cuda")
    iters = torch.empty(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    fn = getattr(ctx, "decode_" + kind.split("_")[0])
    launch = lambda s: fn(llr, n, post=post, hard=hard, iters=iters, stream=s)
    launch(stream)
    return post, hard, iters, launch


def _alone(ctx, kind, llr):
    import torch
    out = _decode(ctx, kind, llr, torch.cuda.current_stream().cuda_stream)[:3]
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("kind", list(CASES))
def test_chunks_of_a_host_call(capi, kind):
    """Page-locked buffers, so that no copy holds the next chunk's decode back."""
    import torch
    n = 3 * CASES[kind][5] - 17
    ctx, llr = _setup(capi, kind, n, 12)
    want = _alone(ctx, kind, llr)
    host = llr.cpu().pin_memory()
    post, hard, iters = torch.empty_like(host).pin_memory(), torch.empty((n, ctx.info.hard_words), dtype=torch.int32,
                                                                         pin_memory=True), torch.empty(n, dtype=torch.uint8,
                                                                                                       pin_memory=True)
    tot = C.c_uint64()
    fn = getattr(capi.lib, "ldpc_decode_%s_host" % kind.split("_")[0])
    for outputs in (True, False):
        capi.check(fn(ctx.h, host.data_ptr(), n, post.data_ptr() if outputs else None,
                      hard.data_ptr() if outputs else None, iters.data_ptr(), C.byref(tot)))
        assert torch.equal(post, want[0].cpu()) and torch.equal(hard, want[1].cpu()) and torch.equal(iters, want[2].cpu())
        assert tot.value == int(iters.sum(dtype=torch.int64))
        iters.zero_()


@pytest.mark.parametrize("n", [40, 3001])
@pytest.mark.parametrize("kind", list(CASES))
def test_two_streams(capi, kind, n):
    """Few codewords: both launches are resident whole; many: the second one's
    first CTAs run beside the first one's last."""
    import torch
    ctx, llr = _setup(capi, kind, 2 * n + 9, 40)
    a, b = llr[:n], llr[n:]
    want_a, want_b = _alone(ctx, kind, a), _alone(ctx, kind, b)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    *got_a, launch_a = _decode(ctx, kind, a, s1.cuda_stream)
    *got_b, launch_b = _decode(ctx, kind, b, s2.cuda_stream)
    for _ in range(4):
        torch.cuda.synchronize()
        for t in got_a + got_b:
            t.zero_()
        torch.cuda.synchronize()
        for _ in range(3):
            launch_a(s1.cuda_stream)
            launch_b(s2.cuda_stream)
        torch.cuda.synchronize()
        assert all(torch.equal(x, y) for x, y in zip(got_a, want_a))
        assert all(torch.equal(x, y) for x, y in zip(got_b, want_b))


@pytest.mark.parametrize("kind", ["int8", "int16", "f64_min_sum"])
def test_captured_beside_direct(capi, kind):
    import torch
    n = 700
    ctx, llr = _setup(capi, kind, 2 * n, 40)
    a, b = llr[:n], llr[n:]
    want_a, want_b = _alone(ctx, kind, a), _alone(ctx, kind, b)
    *got_a, launch_a = _decode(ctx, kind, a, torch.cuda.current_stream().cuda_stream)
    *got_b, launch_b = _decode(ctx, kind, b, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        launch_a(torch.cuda.current_stream().cuda_stream)
    for t in got_a + got_b:
        t.zero_()
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    g.replay()
    launch_b(s.cuda_stream)
    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(got_a, want_a))
    assert all(torch.equal(x, y) for x, y in zip(got_b, want_b))
