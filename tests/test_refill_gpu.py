"""Slots that are refilled: calls with several times as many codewords as a
launch holds, every codeword's outputs against the oracle.  Codewords repeat in
a random order, so that few are decoded by the oracle, and lie at SNRs where
they finish at different iterations, some at none."""
import numpy as np
import pytest

from conftest import make_llr_int8, pack_bits

pytestmark = pytest.mark.gpu


def _codewords(oracle, code, snrs, per_snr, n, seed):
    """LLRs [n][N] drawn from few codewords, which of them each is, and their sent data bits."""
    parts = [make_llr_int8(code, per_snr, s, seed + i, oracle=oracle) for i, s in enumerate(snrs)]
    few, info = (np.concatenate([p[k] for p in parts]) for k in (0, 1))
    return few, np.random.default_rng(seed).integers(0, len(few), n), pack_bits(info)


def _int8_want(oracle, code, few, max_iter):
    post, its = oracle.decode_int8(code, few, max_iter, 31.0, 1.0)
    assert len(np.unique(its)) > 3
    hard = pack_bits((post[:, :code.z * (code.mcol - code.mrow)] < 0).astype(np.uint8))
    return post, hard, its.astype(np.uint8)


# the first has no room for staging buffers and more warps than slots (12 warps, 4 codewords per
# CTA, 148 CTAs); the second stages and has as many
@pytest.mark.parametrize("name,snrs,n", [("5GNR_n25344_k8448", (-4.6, -4.0, -3.4), 1500),
                                         ("5GNR_n12800_k2560", (-6.9, -6.3, -5.7), 4000)])
@pytest.mark.parametrize("graph", [False, True], ids=["context", "graph"])
def test_long_codes_refill(capi, oracle, name, snrs, n, graph):
    import torch
    from ldpc_b200 import codes
    code = codes.code_by_name(name)
    few, pick, data = _codewords(oracle, code, snrs, 25, n, 5)
    post_o, hard_o, its_o = _int8_want(oracle, code, few, 12)
    llr = torch.from_numpy(few[pick]).cuda()
    post = torch.empty_like(llr)
    hard = torch.empty((n, data.shape[1]), dtype=torch.int32, device="cuda")
    iters = torch.empty(n, dtype=torch.uint8, device="cuda")
    sent = torch.from_numpy(data[pick].view(np.int32)).cuda()
    cnt = torch.zeros((1, 4), dtype=torch.int64, device="cuda")
    handle = capi.Code.from_tables(code)
    kw = dict(max_iter=12, max_row_metric=31.0, beta=1.0)
    stream = torch.cuda.current_stream().cuda_stream
    if graph:
        job = dict(code=0, llr=llr, n=n, post=post, hard=hard, iters=iters, data_bits=sent, ref_period=n, bucket_size=n,
                   counters=cnt, n_buckets=1)
        plan = capi.Batch([handle], [kw]).plan([job])
        plan.graph_launch(stream)
    else:
        ctx = capi.Context(handle, **kw)
        ctx.decode_int8(llr, n, post=post, hard=hard, iters=iters, stream=stream)
    torch.cuda.synchronize()
    assert np.array_equal(iters.cpu().numpy(), its_o[pick])
    assert np.array_equal(hard.cpu().numpy().view(np.uint32), hard_o[pick])
    assert np.array_equal(post.cpu().numpy(), post_o[pick])
    if not graph:
        ctx.decode_count(llr, n, hard=hard, iters=iters, data_bits=sent, ref_period=n, bucket_size=n, counters=cnt,
                         n_buckets=1, stream=stream)
        torch.cuda.synchronize()
        assert np.array_equal(hard.cpu().numpy().view(np.uint32), hard_o[pick])
    wrong = np.unpackbits((hard_o ^ data).view(np.uint8), axis=1).sum(1)
    got = cnt.cpu().numpy()[0]
    assert got[0] == n and got[1] == its_o[pick].sum(dtype=np.int64) and got[2] == wrong[pick].sum()
