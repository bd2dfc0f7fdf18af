"""Every slot of a CTA: launches held to one or two CTAs (LDPC_MAX_CTAS), so that
a few codewords fill all groups and all bytes of a word and refill them.  All
outputs against the oracle."""
import numpy as np
import pytest

from conftest import make_llr_int8, pack_bits
from test_row_widths_gpu import WEIGHTS, _code, _int_decode

pytestmark = pytest.mark.gpu


def _same(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))


# 37 codewords: slots filled, then refilled; 3: on the int8 tables two codewords per word
@pytest.mark.parametrize("n", [37, 3])
@pytest.mark.parametrize("z", [5, 33, 64])
@pytest.mark.parametrize("rows", list(WEIGHTS))
@pytest.mark.parametrize("variant", ["i8", "i16", "i32", "f32sp", "f32ms", "f64sp", "f64ms"])
def test_every_row_weight_in_one_cta(capi, oracle, monkeypatch, variant, rows, z, n):
    monkeypatch.setenv("LDPC_MAX_CTAS", "1")
    code = _code(WEIGHTS[rows], z)
    h = capi.Code.from_bytes(code.dec_dat_bytes())
    rng = np.random.default_rng(z + n)
    if variant[0] == "i":
        kind = dict(i8=capi.LDPC_INT8_OMS, i16=capi.LDPC_INT16_OMS, i32=capi.LDPC_INT32_OMS)[variant]
        dt = dict(i8=np.int8, i16=np.int16, i32=np.int32)[variant]
        lim = np.iinfo(dt)
        llr = np.clip(np.rint(rng.normal(3, 6, (n, code.n))), -24, 24).astype(dt)
        llr[1] = rng.integers(lim.min, lim.max, code.n, endpoint=True)
        llr[2] = lim.min
        ctx = capi.Context(h, variant=kind, max_iter=4, max_row_metric=31.0, beta=1.0)
        want, its = _int_decode(code, llr, int(variant[1:]), 4, 31, 1)
    else:
        single, prod = variant.startswith("f32"), variant.endswith("sp")
        kind = dict(f32sp=capi.LDPC_F32_SP, f32ms=capi.LDPC_F32_OMS, f64sp=capi.LDPC_F64_SP,
                    f64ms=capi.LDPC_F64_OMS)[variant]
        clamp, beta = (6e-8 if single else 1e-16, 0.0) if prod else (31.0, 0.5)
        llr = rng.normal(2, 4, (n, code.n)).astype(np.float32 if single else np.float64)
        ctx = capi.Context(h, variant=kind, max_iter=4, max_row_metric=clamp, beta=beta, llr_scale=1.0, max_abs_llr=1e9)
        want, its = (oracle.decode_f32 if single else oracle.decode_f64)(code, llr, int(prod), 4, clamp, beta)
    post, _, iters, _ = ctx.decode_host(llr)
    assert np.array_equal(iters, its.astype(np.uint8))
    assert _same(post, want)


CODES = [("11ad 1/2", -0.5, {}), ("11ad 1/2", -0.5, {"LDPC_OMS_RT": "1"}),
         ("11ad 1/2", -0.5, {"LDPC_OMS_RT": "1", "LDPC_OMS_RT_GLOBAL": "1"}), ("11n 2/3 z81", 0.9, {}),
         ("ITU G.hn 1/2 z14", 1.0, {}), ("5GNR_n1000_k500", -1.0, {}), ("5GNR_n12800_k2560", -6.3, {})]


@pytest.mark.parametrize("offsets", ["beta", "zero", "layers", "table"])
@pytest.mark.parametrize("name,snr,env", CODES, ids=["%s-%s" % (c[0], "-".join(c[2])) for c in CODES])
def test_int8_offsets_in_two_ctas(capi, oracle, monkeypatch, name, snr, env, offsets):
    """Ordinary LLRs with every seventh codeword at the type's limits; one
    offset, the abs8(-128) quirk, offsets per layer, and per iteration (each
    byte of a word in an iteration of its own)."""
    import torch
    from ldpc_b200 import codes
    monkeypatch.setenv("LDPC_MAX_CTAS", "2")
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    code = codes.code_by_name(name)
    n = 60 if code.n > 5000 else 200
    llr, info, _ = make_llr_int8(code, n, snr, seed=6, oracle=oracle)
    rng = np.random.default_rng(2)
    llr[::7] = np.where(rng.random(llr[::7].shape) < 0.5, -128, 127)
    beta = 0.0 if offsets == "zero" else 1.0
    ctx = capi.Context(capi.Code.from_tables(code), max_iter=12, max_row_metric=31.0, beta=beta)
    kw = dict(beta=beta)
    if offsets == "layers":
        b = rng.integers(0, 4, code.mrow)
        ctx.set_layer_offsets(b.astype(np.float32))
        kw = dict(beta_layers=b.astype(np.int8))
    if offsets == "table":
        b = rng.integers(0, 4, (9, code.mrow))
        ctx.set_offset_table(b.astype(np.float32))
        kw = dict(beta_table=b.astype(np.int8))
    want, its = oracle.decode_int8(code, llr, 12, 31.0, **kw)
    assert offsets != "beta" or len(np.unique(its)) > 2
    hard = pack_bits((want[:, :code.z * (code.mcol - code.mrow)] < 0).astype(np.uint8))
    d = torch.from_numpy(llr).cuda()
    post, it = torch.empty_like(d), torch.empty(n, dtype=torch.uint8, device="cuda")
    h = torch.empty(hard.shape, dtype=torch.int32, device="cuda")
    ctx.decode_int8(d, n, post=post, hard=h, iters=it)
    assert np.array_equal(it.cpu().numpy(), its.astype(np.uint8))
    assert np.array_equal(post.cpu().numpy(), want)
    assert np.array_equal(h.cpu().numpy().view(np.uint32), hard)
    data = pack_bits(info)
    cnt = torch.zeros((3, 4), dtype=torch.int64, device="cuda")
    ctx.decode_count(d, n, hard=h, iters=it, data_bits=torch.from_numpy(data.view(np.int32)).cuda(), ref_period=n,
                     bucket_size=(n + 2) // 3, counters=cnt, n_buckets=3)
    wrong = np.unpackbits((hard ^ data).view(np.uint8), axis=1).sum(1, dtype=np.int64)
    for b, sl in enumerate(np.array_split(np.arange(3 * ((n + 2) // 3)), 3)):
        sl = sl[sl < n]
        assert cnt[b].tolist() == [len(sl), its[sl].sum(), wrong[sl].sum(), (wrong[sl] > 0).sum()]


@pytest.mark.parametrize("ctas", ["1", "3"])
@pytest.mark.parametrize("scale", [1, 20])
def test_batch_in_few_ctas(capi, oracle, monkeypatch, scale, ctas):
    """Batch plans of a few CTAs: the smaller one gives two codewords a word, the
    larger one four, both refill."""
    import torch
    from ldpc_b200 import codes
    monkeypatch.setenv("LDPC_MAX_CTAS", ctas)
    parts = [("11ad 1/2", -0.5, 9), ("16e 1/2", 1.2, 5), ("5GNR_n3136_k576", -6.0, 4), ("11ay 1/2", -0.25, 13)]
    objs = [codes.code_by_name(p[0]) for p in parts]
    batch = capi.Batch([capi.Code.from_tables(c) for c in objs], [dict(max_iter=12, max_row_metric=31.0, beta=1.0)] * 4)
    jobs, want = [], []
    for i, (c, (_, snr, n)) in enumerate(zip(objs, parts)):
        n *= scale
        llr, _, _ = make_llr_int8(c, n, snr, seed=i, oracle=oracle)
        d = torch.from_numpy(llr).cuda()
        jobs.append(dict(code=i, llr=d, n=n, post=torch.empty_like(d), iters=torch.empty(n, dtype=torch.uint8, device="cuda")))
        want.append(oracle.decode_int8(c, llr, 12, 31.0, 1.0))
    plan = batch.plan(jobs)
    for _ in range(2):
        plan.graph_launch(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    for job, (post, its) in zip(jobs, want):
        assert np.array_equal(job["iters"].cpu().numpy(), its.astype(np.uint8))
        assert np.array_equal(job["post"].cpu().numpy(), post)
