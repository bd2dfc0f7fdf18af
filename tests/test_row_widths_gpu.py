"""Row updates at every row weight: each decoder unrolls a row's edges to a
width chosen from its weight, so a synthetic code with rows of weights
2..32 passes through each width with and without spare edge slots.  Integer
and min-sum results are exact; sum-product is bit-identical because both
sides evaluate the same functions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _code(weights, z, seed=1):
    """A decoder-only code: row r has weights[r] random columns and shifts."""
    from ldpc_b200 import codes
    rng = np.random.default_rng(seed)
    mcol = max(len(weights) + 1, max(weights) + 1)
    hc = np.full((len(weights), mcol), -1)
    for r, w in enumerate(weights):
        hc[r, np.sort(rng.choice(mcol, w, replace=False))] = rng.integers(0, z, w)
    dec = codes._gen_decode(hc, z, 64)
    return codes.Code(name="rows", z=z, mrow=len(weights), mcol=mcol, num_par=1, hc=hc, hc_dec=hc, dec=dec, par_cnts=[],
                      par_colnum=[], par_offset=[])


def _int_decode(code, llr, bits, max_iter, maxv, beta):
    """Layered offset min-sum on bits-wide saturating lanes (decode_functions.cpp:11-103), in int64:
    posteriors and iteration counts."""
    lo, hi = -(1 << (bits - 1)), (1 << (bits - 1)) - 1
    wrap = lambda v: (v - lo) % (1 << bits) + lo
    t = np.arange(code.z)
    rows, e = [], 0
    for w in code.dec["row_weights"]:
        cols, sh = (np.array(code.dec[k][e:e + w]) for k in ("row_cols", "row_shifts"))
        rows.append(cols * code.z + (t[:, None] + sh) % code.z)
        e += w
    P = llr.astype(np.int64)
    R = [np.zeros((len(P),) + v.shape, np.int64) for v in rows]
    its = np.zeros(len(P), np.int64)
    live = np.ones(len(P), bool)
    for _ in range(max_iter):
        at = np.nonzero(live)[0]
        if not len(at):
            break
        its[at] += 1
        p = P[at]
        for l, v in enumerate(rows):
            q = np.clip(p[:, v] - R[l][at], lo, hi)
            m = np.maximum(wrap(wrap(np.abs(q)) - beta), 0)
            others = np.stack([np.delete(m, j, -1).min(-1) for j in range(v.shape[1])], -1)
            neg = (np.sum(q < 0, -1, keepdims=True) - (q < 0)) % 2 == 1
            r = np.where(neg, -1, 1) * np.minimum(others, maxv)
            R[l][at] = r
            p[:, v.reshape(-1)] = np.clip(q + r, lo, hi).reshape(len(at), -1)
        P[at] = p
        bad = np.zeros(len(at), bool)
        for v in rows:
            bad |= (np.sum(p[:, v] < 0, -1) % 2 == 1).any(-1)
        live[at] = bad
    return P.astype(llr.dtype), its


WEIGHTS = {"2..8": list(range(2, 9)), "2..12": list(range(12, 1, -1)), "3..16": list(range(3, 17)),
           "2..24": list(range(24, 1, -2)) + [23, 21, 19, 17, 5], "2..32": list(range(32, 1, -2)) + [31, 29, 27, 25, 3]}


@pytest.mark.parametrize("z", [5, 33, 64])
@pytest.mark.parametrize("rows", list(WEIGHTS))
@pytest.mark.parametrize("variant", ["i8", "i16", "i32", "f32sp", "f32ms", "f64sp", "f64ms"])
def test_every_row_weight(capi, oracle, variant, rows, z):
    code = _code(WEIGHTS[rows], z)
    rng = np.random.default_rng(z)
    n = 37
    h = capi.Code.from_bytes(code.dec_dat_bytes())
    if variant[0] == "i":
        kind = dict(i8=capi.LDPC_INT8_OMS, i16=capi.LDPC_INT16_OMS, i32=capi.LDPC_INT32_OMS)[variant]
        dt = dict(i8=np.int8, i16=np.int16, i32=np.int32)[variant]
        llr = np.clip(np.rint(rng.normal(3, 6, (n, code.n))), -24, 24).astype(dt)
        lim = np.iinfo(dt)
        llr[0] = lim.max          # saturation on every edge
        llr[1] = lim.min
        llr[2] = rng.integers(lim.min, lim.max, code.n, endpoint=True)
        llr[3] = 0
        ctx = capi.Context(h, variant=kind, max_iter=4, max_row_metric=31.0, beta=1.0)
        post, _, iters, _ = ctx.decode_host(llr)
        post_o, it_o = _int_decode(code, llr, int(variant[1:]), 4, 31, 1)
        if variant == "i8":       # the restatement above against the oracle
            post_c, it_c = oracle.decode_int8(code, llr, 4, 31.0, 1.0)
            assert np.array_equal(post_o, post_c) and np.array_equal(it_o, it_c)
        assert np.array_equal(post, post_o)
    else:
        single = variant.startswith("f32")
        prod = variant.endswith("sp")
        kind = dict(f32sp=capi.LDPC_F32_SP, f32ms=capi.LDPC_F32_OMS, f64sp=capi.LDPC_F64_SP,
                    f64ms=capi.LDPC_F64_OMS)[variant]
        llr = rng.normal(2, 4, (n, code.n)).astype(np.float32 if single else np.float64)
        llr[0] = 0
        llr[1] *= 100             # the clamp
        llr[2] *= 1e-6            # the series next to 0
        clamp, beta = (6e-8 if single else 1e-16, 0.0) if prod else (31.0, 0.5)
        ctx = capi.Context(h, variant=kind, max_iter=4, max_row_metric=clamp, beta=beta, llr_scale=1.0, max_abs_llr=1e9)
        post, _, iters, _ = ctx.decode_host(llr)
        post_o, it_o = (oracle.decode_f32 if single else oracle.decode_f64)(code, llr, int(prod), 4, clamp, beta)
        assert np.array_equal(post.view(np.uint32), post_o.view(np.uint32))
    assert np.array_equal(iters, it_o.astype(np.uint8))


def test_branch_free_tanh_atanh(capi):
    """Every float, and 3e8 doubles of each function: no bit differs."""
    assert capi.probe_sp_math(samples=1000) == 0
