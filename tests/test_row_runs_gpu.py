"""int8 run-time tables: codes whose layers come in runs of a weight use a row
instance per weight, others one for several neighbouring weights.  Both, at every
weight up to 12, with runs of odd and even length, and together in a batch plan
(which then uses the second kind for all of its codes)."""
import numpy as np
import pytest

from test_row_widths_gpu import _code, _int_decode

pytestmark = pytest.mark.gpu

ROWS = {
    "runs 2..8": [w for w in range(2, 9) for _ in range(3 + w % 2)],
    "runs 2..12": [w for w in range(12, 1, -1) for _ in range(3 + w % 2)],
    "one run": [11] * 7,
    "neighbours": [7, 8, 7, 7, 8, 5, 6, 6, 5, 4, 2, 3],
    "neighbours, wide": [14, 15, 16, 13, 13, 16],
    "neighbours, wider": [21, 21, 22, 21, 24, 17],
}


def _llr(code, n, seed):
    rng = np.random.default_rng(seed)
    llr = np.clip(np.rint(rng.normal(3, 6, (n, code.n))), -24, 24).astype(np.int8)
    llr[1] = rng.integers(-128, 127, code.n, endpoint=True)
    return llr


# 37: four codewords per word, refilled; 3: two per word
@pytest.mark.parametrize("n", [37, 3])
@pytest.mark.parametrize("beta", [1, 0])
@pytest.mark.parametrize("z", [7, 42])
@pytest.mark.parametrize("rows", list(ROWS))
def test_runs_of_a_weight(capi, oracle, monkeypatch, rows, z, beta, n):
    monkeypatch.setenv("LDPC_MAX_CTAS", "1")
    code = _code(ROWS[rows], z)
    llr = _llr(code, n, z + n)
    ctx = capi.Context(capi.Code.from_bytes(code.dec_dat_bytes()), max_iter=4, max_row_metric=31.0, beta=float(beta))
    want, its = oracle.decode_int8(code, llr, 4, 31.0, float(beta))
    post, _, iters, _ = ctx.decode_host(llr)
    assert np.array_equal(iters, its.astype(np.uint8))
    assert np.array_equal(post, want)


def test_both_kinds_in_one_plan(capi):
    import torch
    objs = [_code(ROWS[r], 42) for r in ("runs 2..8", "neighbours", "one run")]
    batch = capi.Batch([capi.Code.from_bytes(c.dec_dat_bytes()) for c in objs],
                       [dict(max_iter=5, max_row_metric=31.0, beta=1.0)] * 3)
    for used in ((0, 1, 2), (0, 2), (1,)):
        jobs, want = [], []
        for i in used:
            llr = _llr(objs[i], 50, i)
            d = torch.from_numpy(llr).cuda()
            jobs.append(dict(code=i, llr=d, n=len(llr), post=torch.empty_like(d),
                             iters=torch.empty(len(llr), dtype=torch.uint8, device="cuda")))
            want.append(_int_decode(objs[i], llr, 8, 5, 31, 1))
        plan = batch.plan(jobs)
        plan.graph_launch(torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        for job, (post, its) in zip(jobs, want):
            assert np.array_equal(job["iters"].cpu().numpy(), its.astype(np.uint8))
            assert np.array_equal(job["post"].cpu().numpy(), post)
