"""Work that programs using the library have it do, at fixed and at drawn sizes.

Every case is one pass through a public entry point of ``ldpc_b200``:

====== ==========================================================================
kind   entry point
====== ==========================================================================
count  ``Context.decode_count``: a simulator's decode of resident LLRs at one or
       more SNR points, hard decisions, iteration counts and error counters out
post   ``Context.decode_<type>``: decoding of resident LLRs with posteriors,
       hard decisions and iteration counts out
host   ``Context.decode_host``: decoding of LLRs in host memory, as
       LDPCdecode_set is called
batch  ``Batch.plan`` + ``BatchPlan.graph_launch``: several codes in one graph
gen    ``Context.generate``: data bits, encoding, noise, LLRs at every SNR point
encode ``Context.encode``: packed data bits to code bits
train  ``learned.LearnedOMSLoss``: one training step's loss and offset gradient
sim    ``Context.simulate``: a whole simulation loop, counters out
====== ==========================================================================

Codes, decoder parameters, SNR points and iteration limits are those of
``bench.py`` and ``ldpc_b200/workloads.py``: 802.11ad 1/2 over -1..0 dB, the
802.11n/ay/ad mix at a codeword error rate near 1e-3, 802.16e 1/2 at Eb/N0
0.5..2 dB, 5G NR at Eb/N0 0.5..1.5 dB.  LLRs come from the library's generator
(whose output depends on the seed alone).
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("simd-fecfun_b200"))
from ldpc_b200 import capi, codes, learned  # noqa: E402

# variant: (library constant, torch type of LLRs and posteriors, max_row_metric, beta, LLR scale, max |LLR|)
VARIANTS = {
    "i8": (capi.LDPC_INT8_OMS, torch.int8, 31.0, 1.0, 2.0, 24.0),
    "i16": (capi.LDPC_INT16_OMS, torch.int16, 31.0, 1.0, 2.0, 24.0),
    "i32": (capi.LDPC_INT32_OMS, torch.int32, 31.0, 1.0, 2.0, 24.0),
    "f32sp": (capi.LDPC_F32_SP, torch.float32, 6e-8, 0.0, 1.0, 1e9),
    "f32ms": (capi.LDPC_F32_OMS, torch.float32, 31.0, 0.5, 1.0, 1e9),
    "f64sp": (capi.LDPC_F64_SP, torch.float64, 1e-16, 0.0, 1.0, 1e9),
    "f64ms": (capi.LDPC_F64_OMS, torch.float64, 31.0, 0.5, 1.0, 1e9),
}

AD12 = "11ad 1/2"
NR1 = "5GNR_n25344_k8448"
NR2 = ("5GNR_n3136_k576", "5GNR_n6400_k1280", "5GNR_n12800_k2560")
# Es/N0 (dB) at which the int8 decoder's codeword error rate is near 1e-3
WIFI = {
    "11n 1/2 z27": -0.52, "11n 2/3 z27": 1.44, "11n 3/4 z27": 2.40, "11n 5/6 z27": 3.57,
    "11n 1/2 z54": -0.82, "11n 2/3 z54": 1.01, "11n 3/4 z54": 2.05, "11n 5/6 z54": 3.21,
    "11n 1/2 z81": -0.96, "11n 2/3 z81": 0.85, "11n 3/4 z81": 1.87, "11n 5/6 z81": 3.10,
    "11ay 1/2": -0.79, "11ay 5/8": 0.66, "11ay 3/4": 2.04, "11ay 13/16": 3.04, "11ay 7/8": 3.93,
    "11ad 13/16": 3.39,
}
OTHER = {"11ad 5/8": 1.03, "11ad 3/4": 2.42, "16e 2/3A": 1.44, "16e 3/4A": 2.57, "16e 5/6": 4.29}
ITERS_TRAIN = 10


def listed():
    return [
        # the simulator's step: 802.11ad 1/2, 1e6 codewords at each of five SNR points, errors counted
        dict(name="int8_11ad_sim_step", kind="count", variant="i8", code=AD12, z=0, n=1000000, points=5, snr=-1.0,
             step=0.25, iters=10),
        # a receiver decoding a ragged block of 802.11n codewords, soft outputs wanted
        dict(name="int8_11n_soft_out", kind="post", variant="i8", code="11n 2/3 z81", z=0, n=33333, points=1, snr=0.85,
             step=0.0, iters=10),
        # 5G NR base graph 1 at its largest lifting size
        dict(name="int8_nr_bg1", kind="count", variant="i8", code=NR1, z=0, n=6001, points=1, snr=-3.77, step=0.0,
             iters=20),
        # an access point's mix of codes in one graph
        dict(name="int8_wifi_mix", kind="batch", variant="i8", mix="wifi", n=50000, iters=10),
        # the smallest call: a handful of codewords in host memory, decoded as LDPCdecode_set does
        dict(name="int8_host_few", kind="host", variant="i8", code=AD12, z=0, n=50, snr=-0.5, iters=10),
        # sum-product reference curves, 802.16e 1/2 at its largest lifting size
        dict(name="f32_sum_product_16e", kind="post", variant="f32sp", code="16e 1/2", z=96, n=20011, points=1, snr=-1.51,
             step=0.0, iters=10),
        # the same in double
        dict(name="f64_sum_product_11ad", kind="post", variant="f64sp", code=AD12, z=0, n=30000, points=1, snr=-0.5,
             step=0.0, iters=10),
        # wide-integer min-sum
        dict(name="int16_11ad", kind="count", variant="i16", code=AD12, z=0, n=20001, points=5, snr=-1.0, step=0.25,
             iters=10),
        # channel generation for the simulator's step
        dict(name="generate_11ad", kind="gen", variant="i8", code=AD12, z=0, n=400000, points=5, snr=-1.0, step=0.25),
        # code bits of a training batch
        dict(name="encode_16e", kind="encode", code="16e 1/2", z=96, n=65536),
        # a training step of the learned offsets: 802.16e 1/2 Z=96, 10 iterations x 12 layers
        dict(name="learned_step_16e", kind="train", code="16e 1/2", z=96, n=65536),
        # one loop of the simulation program
        dict(name="simulate_11ad", kind="sim", variant="i8", code=AD12, z=0, n=100000, points=5, snr=-1.0, step=0.25,
             iters=10),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_code(rng):
    """(code, z, snr, iterations) of one of the families above."""
    fam = rng.choice(("ad", "wifi", "16e", "other", "nr"))
    if fam == "ad":
        return AD12, 0, round(rng.uniform(-1.0, 0.0), 2), 10
    if fam == "16e":
        return "16e 1/2", 4 * rng.randint(6, 24), round(rng.uniform(0.5, 2.0) - 3.01, 2), 10
    if fam == "nr":
        return rng.choice(NR2 + (NR1,)), 0, None, 20
    name = rng.choice(sorted(WIFI if fam == "wifi" else OTHER))
    return name, 0, (WIFI if fam == "wifi" else OTHER)[name], 10


# most codewords x edges of one drawn pass, per variant
MOST_EDGES = {"i8": 2e9, "i16": 1e9, "i32": 1e9, "f32sp": 2e8, "f32ms": 1e9, "f64sp": 1e8, "f64ms": 5e8}


def draw(rng):
    kind = rng.choice(("count", "post", "count", "post", "host", "batch", "gen", "encode", "train", "sim"))
    if kind == "batch":
        mix = rng.choice(("wifi", "wifi", "nr", "16e"))
        most = {"wifi": 100000, "nr": 1000, "16e": 2000}[mix]
        return dict(kind=kind, variant="f32sp" if mix == "16e" else "i8", mix=mix, n=_log(rng, 100, most),
                    iters=20 if mix == "nr" else 10)
    if kind == "train":
        return dict(kind=kind, code="16e 1/2", z=4 * rng.randint(6, 24), n=_log(rng, 256, 32768))
    code, z, snr, iters = _draw_code(rng)
    c = tables(code, z)
    if snr is None:
        snr = round(rng.uniform(0.5, 1.5) + 10.0 * math.log10(_rate(c)), 2)
    if kind == "encode":
        return dict(kind=kind, code=code, z=z, n=_log(rng, 500, 2e8 / c.n))
    points = rng.choice((1, 1, 3, 5))
    if kind == "gen":
        variant = rng.choice(("i8", "i8", "f32sp", "i16"))
        most = 1.2e9 / (points * c.n * _bytes(variant))
        return dict(kind=kind, variant=variant, code=code, z=z, n=_log(rng, 500, most), points=points, snr=snr, step=0.25)
    if kind == "sim":
        most = MOST_EDGES["i8"] / 4 / (points * c.edges)
        return dict(kind=kind, variant="i8", code=code, z=z, n=_log(rng, 200, max(400, most)), points=points, snr=snr,
                    step=0.25, iters=iters)
    variant = rng.choice(("i8", "i8", "i8", "i16", "i32", "f32sp", "f32ms", "f64sp", "f64ms"))
    if kind == "host":
        return dict(kind=kind, variant=variant, code=code, z=z, n=_log(rng, 16, MOST_EDGES[variant] / 20 / c.edges),
                    snr=snr, iters=iters)
    if kind == "post":
        points = 1
    most = MOST_EDGES[variant] / (points * c.edges)
    return dict(kind=kind, variant=variant, code=code, z=z, n=_log(rng, 64, max(128, most)), points=points, snr=snr,
                step=0.25, iters=iters)


@functools.lru_cache(maxsize=None)
def tables(code, z):
    return codes.code_by_name(code, z_over=z) if z else codes.code_by_name(code)


@functools.lru_cache(maxsize=None)
def _handle(code, z):
    return capi.Code.from_tables(tables(code, z))


def _rate(c):
    return c.k / (c.n - c.punc_cnt_bits - c.fill_cnt)


def _bytes(variant):
    return torch.empty(0, dtype=VARIANTS[variant][1]).element_size()


def _context(variant, code, z, iters):
    v, _, clamp, beta, scale, most = VARIANTS[variant]
    return capi.Context(_handle(code, z), variant=v, max_iter=iters, max_row_metric=clamp, beta=beta, llr_scale=scale,
                        max_abs_llr=most)


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _snrs(case):
    return [case["snr"] + case["step"] * i for i in range(case["points"])]


def _draw_llr(ctx, variant, seed, snrs, n):
    """LLRs [points][n][N] and the sent data bits."""
    dt = VARIANTS[variant][1]
    llr = torch.empty((len(snrs), n, ctx.info.n), dtype=dt, device="cuda")
    data = torch.empty((n, ctx.info.hard_words), dtype=torch.int32, device="cuda")
    out = dict(llr_f32=llr) if dt == torch.float32 else dict(llr_int=llr)
    ctx.generate(seed, 0, snrs, n, data_bits=data, stream=_stream(), **out)
    return llr, data


def _mix(mix):
    """[(code, z, snr)] of a batch."""
    if mix == "wifi":
        return [(name, 0, snr) for name, snr in WIFI.items()]
    if mix == "16e":
        return [("16e 1/2", z, 1.25 - 3.01) for z in range(24, 97, 4)]
    return [(name, 0, 1.0 + 10.0 * math.log10(_rate(tables(name, 0)))) for name in (NR1,) + NR2]


def prepare(case, seed):
    kind, st = case["kind"], dict(case=case)
    dev = "cuda"
    if kind == "batch":
        parts = _mix(case["mix"])
        v, _, clamp, beta, _, _ = VARIANTS[case["variant"]]
        batch = capi.Batch([_handle(c, z) for c, z, _ in parts],
                           [dict(variant=v, max_iter=case["iters"], max_row_metric=clamp, beta=beta)] * len(parts))
        counters = torch.zeros((len(parts), 4), dtype=torch.int64, device=dev)
        jobs = []
        for i, (c, z, snr) in enumerate(parts):
            ctx = _context(case["variant"], c, z, case["iters"])
            n = case["n"] + i % 3   # the codes' blocks are not all alike
            llr, data = _draw_llr(ctx, case["variant"], seed + 1000 * i, [snr], n)
            jobs.append(dict(code=i, llr=llr, n=n, data_bits=data, ref_period=n, bucket_size=n, counters=counters[i],
                             n_buckets=1, hard=torch.empty_like(data),
                             iters=torch.empty(n, dtype=torch.uint8, device=dev)))
        st.update(batch=batch, jobs=jobs, plan=batch.plan(jobs), counters=counters)
        return st
    if kind == "train":
        ctx = _context("f32ms", case["code"], case["z"], ITERS_TRAIN)
        c = tables(case["code"], case["z"])
        g = torch.Generator(device=dev).manual_seed(seed)
        ebn0 = 1.0 + 1.5 * torch.rand(16, generator=g, device=dev)
        llr, bits = learned.draw(ctx, c, case["n"], [e + 10.0 * math.log10(_rate(c)) for e in ebn0.tolist()], seed, 0)
        beta = 0.5 + 0.05 * torch.randn((ITERS_TRAIN, c.mrow), generator=g, device=dev)
        st.update(ctx=ctx, llr=llr, bits=bits, beta=beta.requires_grad_(True), w=torch.ones(ITERS_TRAIN, device=dev))
        return st
    if kind == "encode":
        ctx = _context("i8", case["code"], case["z"], 10)
        g = torch.Generator(device=dev).manual_seed(seed)
        data = torch.randint(-2 ** 31, 2 ** 31, (case["n"], ctx.info.hard_words), dtype=torch.int32, generator=g, device=dev)
        st.update(ctx=ctx, data=data, bits=torch.empty((case["n"], ctx.info.n), dtype=torch.uint8, device=dev))
        return st
    ctx = _context(case["variant"], case["code"], case["z"], case.get("iters", 10))
    st.update(ctx=ctx, seed=seed)
    n = case["n"]
    if kind == "gen":
        dt = VARIANTS[case["variant"]][1]
        llr = torch.empty((case["points"], n, ctx.info.n), dtype=dt, device=dev)
        st.update(llr=llr, out=dict(llr_f32=llr) if dt == torch.float32 else dict(llr_int=llr), snrs=_snrs(case),
                  data=torch.empty((n, ctx.info.hard_words), dtype=torch.int32, device=dev),
                  uncoded=torch.zeros(case["points"], dtype=torch.int64, device=dev))
    elif kind == "host":
        llr, _ = _draw_llr(ctx, case["variant"], seed, [case["snr"]], n)
        st.update(llr=llr[0].cpu().numpy())
    elif kind in ("count", "post"):
        llr, data = _draw_llr(ctx, case["variant"], seed, _snrs(case), n)
        total = n * case["points"]
        st.update(llr=llr, data=data, total=total, iters=torch.empty(total, dtype=torch.uint8, device=dev),
                  hard=torch.empty((total, ctx.info.hard_words), dtype=torch.int32, device=dev))
        if kind == "post":
            st.update(post=torch.empty_like(llr))
        else:
            st.update(counters=torch.zeros((case["points"], 4), dtype=torch.int64, device=dev))
    return st


_DECODE = {"i8": "decode_int8", "i16": "decode_int16", "i32": "decode_int32", "f32sp": "decode_f32",
           "f32ms": "decode_f32", "f64sp": "decode_f64", "f64ms": "decode_f64"}


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "count":
        st["counters"].zero_()
        st["ctx"].decode_count(st["llr"], st["total"], hard=st["hard"], iters=st["iters"], data_bits=st["data"],
                               ref_period=case["n"], bucket_size=case["n"], counters=st["counters"],
                               n_buckets=case["points"], stream=_stream())
        return dict(hard=st["hard"], iters=st["iters"], counters=st["counters"])
    if kind == "post":
        getattr(st["ctx"], _DECODE[case["variant"]])(st["llr"], st["total"], post=st["post"], hard=st["hard"],
                                                     iters=st["iters"], stream=_stream())
        return dict(hard=st["hard"], iters=st["iters"], post=st["post"])
    if kind == "host":
        post, hard, iters, total = st["ctx"].decode_host(st["llr"])
        return dict(hard=hard.view(np.int32), iters=iters, post=post, total=total)
    if kind == "batch":
        st["counters"].zero_()
        st["plan"].graph_launch(_stream())
        return dict(counters=st["counters"], hard=[j["hard"] for j in st["jobs"]], iters=[j["iters"] for j in st["jobs"]])
    if kind == "gen":
        st["uncoded"].zero_()
        st["ctx"].generate(st["seed"], 0, st["snrs"], case["n"], data_bits=st["data"], uncoded=st["uncoded"],
                           stream=_stream(), **st["out"])
        return dict(data=st["data"], llr=st["llr"], uncoded=st["uncoded"])
    if kind == "encode":
        st["ctx"].encode(st["data"], case["n"], st["bits"], stream=_stream())
        return st["bits"]
    if kind == "train":
        st["beta"].grad = None
        loss = learned.LearnedOMSLoss.apply(st["beta"], st["llr"], st["bits"], st["w"], st["ctx"])
        loss.backward()
        return dict(grad=st["beta"].grad, loss=loss.detach())
    stats = st["ctx"].simulate(st["seed"], 0, _snrs(case), case["n"])
    return [[s["codewords"], s["iterations"], s["bit_errors"], s["cw_errors"], s["uncoded_errors"]] for s in stats]


def work(case):
    """Inputs read once, outputs written once; operations of one decoder
    iteration on every codeword (each codeword runs at least one)."""
    kind = case["kind"]
    if kind == "batch":
        parts = [(tables(c, z), case["n"] + i % 3) for i, (c, z, _) in enumerate(_mix(case["mix"]))]
        es, ops = _bytes(case["variant"]), _ops(case["variant"])
        return dict(bytes=sum(n * (c.n * es + 8 * _words(c) + 1) for c, n in parts),
                    flops=sum(n * c.edges * ops for c, n in parts))
    c = tables(case["code"], case["z"])
    n = case["n"]
    if kind == "encode":
        return dict(bytes=n * (4 * _words(c) + c.n), flops=0)
    if kind == "train":
        # every iteration runs, forward and adjoint
        return dict(bytes=n * c.n * 5, flops=n * c.edges * ITERS_TRAIN * 30)
    es, p = _bytes(case["variant"]), case.get("points", 1)
    if kind == "gen":
        return dict(bytes=n * (p * c.n * es + 4 * _words(c)), flops=n * c.n * (20 + 4 * p))
    ops = n * p * c.edges * _ops(case["variant"])
    if kind == "count":
        return dict(bytes=n * p * (c.n * es + 4 * _words(c) + 1) + n * 4 * _words(c), flops=ops)
    if kind == "sim":
        return dict(bytes=40 * p, flops=ops + n * c.n * (20 + 4 * p))
    return dict(bytes=n * p * (2 * c.n * es + 4 * _words(c) + 1), flops=ops)


def _words(c):
    return (c.z * (c.mcol - c.mrow) + 31) // 32


def _ops(variant):
    """Operations of one edge update: ten for min-sum, 58 for sum-product (tanh 23, atanh 27, the rest 8)."""
    return 58 if variant.endswith("sp") else 10


# ---- the same results in 64 bits, as plain torch gives them ----

def _layers(c):
    """Per layer, the posterior index of check t's edge j: [Z][weight]."""
    out, e = [], 0
    t = torch.arange(c.z, device="cuda")
    for w in c.dec["row_weights"]:
        col = torch.tensor(c.dec["row_cols"][e:e + w], device="cuda")
        shift = torch.tensor(c.dec["row_shifts"][e:e + w], device="cuda")
        out.append(col * c.z + (t[:, None] + shift) % c.z)
        e += w
    return out


def _others(x, op):
    """op over all elements of the last axis but each one."""
    d = x.shape[-1]
    left, right = [None] * d, [None] * d
    for j in range(1, d):
        left[j] = x[..., j - 1] if j == 1 else op(left[j - 1], x[..., j - 1])
        right[d - 1 - j] = x[..., d - j] if j == 1 else op(right[d - j], x[..., d - j])
    return torch.stack([right[j] if left[j] is None else left[j] if right[j] is None else op(left[j], right[j])
                        for j in range(d)], -1)


def _exact_posteriors(llr, c, product, clamp, beta, iters):
    idx = _layers(c)
    P = llr.double().clone()
    n = P.shape[0]
    R = [torch.zeros((n,) + tuple(v.shape), dtype=torch.float64, device="cuda") for v in idx]
    live = torch.ones(n, dtype=torch.bool, device="cuda")
    for _ in range(iters):
        at = live.nonzero()[:, 0]
        if not at.numel():
            break
        p = P[at]
        for l, v in enumerate(idx):
            q = p[:, v] - R[l][at]
            a = (q.abs() - beta).clamp_min(0.0)
            if product:
                f = 2.0 * torch.atanh(_others(torch.tanh(0.5 * a), torch.mul).clamp_max(clamp))
            else:
                f = _others(a, torch.minimum).clamp_max(clamp)
            neg = q < 0
            f = torch.where((neg.sum(-1, keepdim=True) - neg.long()) % 2 == 1, -f, f)
            R[l][at] = f
            p[:, v.reshape(-1)] = (q + f).reshape(len(at), -1)
        P[at] = p
        bad = torch.zeros(len(at), dtype=torch.bool, device="cuda")
        for v in idx:
            bad |= ((p[:, v] < 0).sum(-1) % 2 == 1).any(-1)
        live[at] = bad
    return P


def _exact_loss(llr, bits, beta, c, clamp, inv_norm):
    """Loss of some codewords, each iteration weighted 1, with its gradient left in beta."""
    s = 1.0 - 2.0 * bits.double()
    P = llr.double()
    idx = _layers(c)
    R = [0.0] * len(idx)
    loss = 0.0
    for it in range(beta.shape[0]):
        for l, v in enumerate(idx):
            q = P[:, v] - R[l]
            a = torch.relu(q.abs() - beta[it, l])
            m1, i1 = a.min(-1, keepdim=True)
            m2 = a.scatter(-1, i1, float("inf")).min(-1, keepdim=True).values
            first = torch.arange(a.shape[-1], device="cuda") == i1
            f = torch.where(first, m2, m1).clamp_max(clamp)
            neg = q < 0
            R[l] = torch.where((neg.sum(-1, keepdim=True) - neg.long()) % 2 == 1, -f, f)
            P = P.index_copy(1, v.reshape(-1), (q + R[l]).reshape(len(P), -1))
        loss = loss + torch.nn.functional.softplus(-s * P).sum() * inv_norm
    loss.backward()
    return loss.detach()


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        c = tables(case["code"], case["z"])
        st = prepare(case, seed)
        beta = st["beta"].detach().double().requires_grad_(True)
        loss = torch.zeros((), dtype=torch.float64, device="cuda")
        for i in range(0, case["n"], 2048):
            loss += _exact_loss(st["llr"][i:i + 2048], st["bits"][i:i + 2048], beta, c, 31.0, 1.0 / (case["n"] * c.n))
        return dict(grad=beta.grad, loss=loss)
    if kind in ("post", "host") and case["variant"][0] == "f":
        v, dt, clamp, beta, _, _ = VARIANTS[case["variant"]]
        c = tables(case["code"], case["z"])
        llr = torch.as_tensor(prepare(case, seed)["llr"]).cuda().reshape(-1, c.n)
        f = np.float32 if dt == torch.float32 else np.float64
        clamp = float(np.float32(clamp))
        clamp = float(f(1.0 - clamp)) if clamp < 1e-6 else clamp
        some = max(1, int(4e8 / 8 / c.edges))
        post = torch.cat([_exact_posteriors(llr[i:i + some], c, v in (capi.LDPC_F32_SP, capi.LDPC_F64_SP), clamp, beta,
                                            case["iters"]) for i in range(0, len(llr), some)])
        return dict(hard=None, iters=None, post=post if kind == "host" else post[None],
                    **(dict(total=None) if kind == "host" else {}))
    return None
