"""Whole batches against the CPU oracle: every row of the batched configuration and of the benchmark workload, and rows built
to sit on the edge of the candidate kernel's FP32 decision band. Bit-exact tokens and thresholds."""
import os

import numpy as np
import pytest
import torch

import bench
import lithos_metal_b200 as lm
import oracle
from tests import inputs, routes
from tests.test_gpu_sampling import bf16_tensor

pytestmark = pytest.mark.gpu
THREADS = max(1, len(os.sched_getaffinity(0)))


def gpu_and_oracle(cfg, **extra):
    x = bf16_tensor(cfg["logits"])
    knobs = {k: torch.from_numpy(np.ascontiguousarray(cfg[k])).cuda() for k in ("temperature", "top_k", "top_p")}
    hist = torch.from_numpy(cfg["history"]).cuda() if cfg.get("history") is not None else None
    pen = dict(repetition_penalty=1.1, presence_penalty=0.5) if hist is not None else {}
    r = lm.sample(x, lm.SamplingParams(draw="inverse_cdf", **pen, **knobs, **extra), history=hist, uniforms=torch.from_numpy(cfg["uniforms"]).cuda(),
                  return_tau=True, return_status=True)
    tok, tau, _ = oracle.sample_batch(cfg["logits"], temperature=cfg["temperature"], top_k=cfg["top_k"], top_p=cfg["top_p"], history=cfg.get("history"),
                                      draw="inverse_cdf", uniforms=cfg["uniforms"], n_threads=THREADS, **pen, **extra)
    return r, tok, tau


def test_every_row_of_the_batched_configuration():
    """Benchmark configuration 3: 256 penalised rows with per-row knobs."""
    r, tok, tau = gpu_and_oracle(inputs.config3())
    status = r.status.cpu().numpy()
    np.testing.assert_array_equal(r.tau.cpu().numpy(), tau)
    np.testing.assert_array_equal(r.tokens.cpu().numpy(), tok)
    assert not np.any(status & 1) and np.count_nonzero(status & 64) > 100    # nothing on the generic path; most rows with a top_k on the candidate path


def test_every_row_of_the_benchmark_workload():
    """The 4096 rows bench.py times (generated the same way), all of them."""
    inp = bench.make_inputs(torch, bench.TOTAL_ROWS, 0, torch.device("cuda", 0))
    params = lm.SamplingParams(temperature=inp["temperature"], top_k=inp["top_k"], top_p=inp["top_p"], repetition_penalty=bench.RHO,
                               presence_penalty=bench.PI, draw="inverse_cdf")
    r = lm.sample(inp["logits"], params, history=inp["history"], uniforms=inp["uniforms"], return_tau=True, return_status=True)
    hc = bench.host_copy(torch, inp, bench.TOTAL_ROWS)
    tok, tau, _ = oracle.sample_batch(hc["logits"], temperature=hc["temperature"], top_k=hc["top_k"], top_p=hc["top_p"], history=hc["history"],
                                      repetition_penalty=bench.RHO, presence_penalty=bench.PI, draw="inverse_cdf", uniforms=hc["uniforms"], n_threads=THREADS)
    np.testing.assert_array_equal(r.tau.cpu().numpy(), tau)
    np.testing.assert_array_equal(r.tokens.cpu().numpy(), tok)
    status = r.status.cpu().numpy()
    n_topk = int((hc["top_k"] > 0).sum())
    assert np.count_nonzero(status & 1) <= 2 and np.count_nonzero(status & 64) >= 0.97 * n_topk   # the candidate kernel keeps nearly all of its rows


def test_rows_on_the_edge_of_the_fp32_decision_band():
    """The candidate kernel knows the row's mass only in FP32 and forms it again in FP64 when a cumulative-mass boundary lies inside its
    error band around top_p * Z. Here top_p is placed at relative distances 0 .. 1e-4 on both sides of an exact boundary inside the
    top-k set: however the row is decided, the threshold must be the oracle's (FP64). Far from the boundary the FP32 mass must do
    (the band is narrow)."""
    base = inputs.config3(rows=8, seed=77)
    deltas = np.array([0.0, 3e-7, -3e-7, 1e-6, -1e-6, 3e-6, -3e-6, 1e-5, -1e-5, 3e-5, -3e-5, 1e-4, -1e-4])
    rows = []
    for r in range(8):
        T = np.float32(0.45 + 0.05 * r)
        z = oracle.bf16_to_f32(base["logits"][r]).astype(np.float64)
        vals, counts = np.unique(z, return_counts=True)
        vals, counts = vals[::-1], counts[::-1]
        cum = np.cumsum(counts * np.exp((vals - vals[0]) / np.float64(T)))
        n_top = np.cumsum(counts)
        i = int(np.searchsorted(n_top, 300))                               # a boundary well inside the top 1000
        for d in deltas:
            rows.append((r, T, np.float32(cum[i] / cum[-1] * (1.0 + d)), d))
    cfg = dict(logits=np.stack([base["logits"][r] for r, _, _, _ in rows]), temperature=np.array([t for _, t, _, _ in rows], np.float32),
               top_k=np.full(len(rows), 1000, np.int32), top_p=np.array([p for _, _, p, _ in rows], np.float32), history=None,
               uniforms=np.linspace(0.05, 0.95, len(rows)).astype(np.float32))
    assert np.all((cfg["top_p"] > 0.3) & (cfg["top_p"] < 1.0))
    r, tok, tau = gpu_and_oracle(cfg)
    np.testing.assert_array_equal(r.tau.cpu().numpy(), tau)
    np.testing.assert_array_equal(r.tokens.cpu().numpy(), tok)
    on_candidate_path = (r.status.cpu().numpy() & 64) != 0
    far = np.abs(np.array([d for _, _, _, d in rows])) >= 1e-4
    assert on_candidate_path[far].all()                                    # the band does not reach 1e-4
    assert not on_candidate_path[np.array([d for _, _, _, d in rows]) == 0.0].any()   # dead on the boundary: never decided in FP32


@pytest.mark.parametrize("exact_only", [False, True])
def test_draw_over_runs_of_equal_logits_from_both_sources(exact_only):
    """The inverse-CDF draw walks equal logits in index order. With repetition 2.0 and presence 0.5 a penalised logit lands exactly
    on BF16 codes that unpenalised logits of the row carry too (z / 2 - 0.5), so runs of equal values mix penalised and unpenalised
    positions; coarse logits (multiples of 1/4) make the runs long. Uniforms spread over [0, 1) land inside such runs in every
    kernel: rows with a top_k (candidate kernel), without one (histogram kernel), and with exact_only (histogram kernel for all)."""
    rows, vocab = 96, 65536
    rng = np.random.default_rng(123)
    z = np.round(rng.standard_normal((rows, vocab)) * 8.0) / 4.0                                  # values k / 4, |z| up to ~10
    codes = oracle.f32_to_bf16(z.astype(np.float32))
    hist = rng.integers(0, vocab, (rows, 1500)).astype(np.int32)
    top = np.argsort(-z, axis=1)[:, :200]
    hist[:, :200] = top                                                                            # the penalties reach the top of the row
    cfg = dict(logits=codes, temperature=rng.uniform(0.8, 2.5, rows).astype(np.float32),
               top_k=np.where(np.arange(rows) % 3 == 0, 0, np.where(np.arange(rows) % 3 == 1, 40, 700)).astype(np.int32),
               top_p=rng.uniform(0.85, 0.999, rows).astype(np.float32), history=hist, uniforms=np.linspace(0.001, 0.999, rows).astype(np.float32))
    x = bf16_tensor(cfg["logits"])
    knobs = {k: torch.from_numpy(cfg[k]).cuda() for k in ("temperature", "top_k", "top_p")}
    pen = dict(repetition_penalty=2.0, presence_penalty=0.5)
    r = lm.sample(x, lm.SamplingParams(draw="inverse_cdf", exact_only=exact_only, **pen, **knobs), history=torch.from_numpy(hist).cuda(),
                  uniforms=torch.from_numpy(cfg["uniforms"]).cuda(), return_tau=True, return_status=True)
    tok, tau, _ = oracle.sample_batch(codes, temperature=cfg["temperature"], top_k=cfg["top_k"], top_p=cfg["top_p"], history=hist, draw="inverse_cdf",
                                      uniforms=cfg["uniforms"], n_threads=THREADS, **pen)
    np.testing.assert_array_equal(r.tau.cpu().numpy(), tau)
    np.testing.assert_array_equal(r.tokens.cpu().numpy(), tok)
    status = r.status.cpu().numpy()
    assert np.count_nonzero(status & 1) <= rows // 8, status                                       # the streaming kernels keep (nearly) all of these rows
    # the drawn tokens do sit in mixed runs: for some rows the token's value is carried by penalised and unpenalised positions alike
    zf = oracle.bf16_to_f32(codes)
    mixed = 0
    for i in range(rows):
        zi = oracle.apply_penalties(zf[i], hist[i], 2.0, 0.5)
        same = np.nonzero(zi == zi[tok[i]])[0]
        pen_ids = np.unique(hist[i])
        mixed += int(np.isin(same, pen_ids).any() and (~np.isin(same, pen_ids)).any())
    assert mixed >= 3, mixed


@pytest.mark.parametrize("copies,one_k,kernel", [(1, False, "sample_cluster_kernel"), (2, False, "sample_topk_kernel"), (2, True, "sample_topk_kernel")])
def test_penalised_rows_inside_the_fp32_decision_band_are_decided_in_fp64(copies, one_k, kernel):
    """As above with penalties: the mass is formed again in FP64, penalised positions at their penalised values; by the cluster kernel (48 rows)
    and by the candidate kernel (96), beside the histogram kernel's rows or, with one top_k for all, ahead of them."""
    rng = np.random.default_rng(31)
    vocab, T, rho, pi = 40008, np.float32(0.7), 1.2, 0.4
    codes = oracle.f32_to_bf16((rng.standard_normal(vocab) * 2.0).astype(np.float32))
    hist = np.concatenate([np.argsort(-oracle.bf16_to_f32(codes))[:400:2], rng.integers(0, vocab, 500)]).astype(np.int32)
    z = np.asarray(oracle.apply_penalties(oracle.bf16_to_f32(codes), hist, rho, pi), dtype=np.float64)
    vals, counts = np.unique(z, return_counts=True)
    vals, counts = vals[::-1], counts[::-1]
    cum = np.cumsum(counts * np.exp((vals - vals[0]) / np.float64(T)))
    top_p = np.array([cum[int(np.searchsorted(np.cumsum(counts), n))] / cum[-1] * (1.0 + d) for n in (60, 150, 250, 333, 390, 450)
                      for d in (0.0, 1e-7, -1e-7, 4e-7, -4e-7, 1e-6, -1e-6, 1e-4)] * copies, dtype=np.float32)
    n = len(top_p)
    cfg = dict(logits=np.tile(codes, (n, 1)), temperature=np.full(n, T, np.float32), top_k=np.full(n, 600, np.int32), top_p=top_p)
    u = np.linspace(0.02, 0.98, n).astype(np.float32)
    x, h, ut = bf16_tensor(cfg["logits"]), torch.from_numpy(np.tile(hist, (n, 1))).cuda(), torch.from_numpy(u).cuda()
    knobs = {k: torch.from_numpy(cfg[k]).cuda() for k in ("temperature", "top_k", "top_p")}
    if one_k:
        knobs["top_k"] = 600
    p = lm.SamplingParams(draw="inverse_cdf", repetition_penalty=rho, presence_penalty=pi, **knobs)
    launched = routes.names(lambda: lm.sample(x, p, history=h, uniforms=ut))
    assert kernel in launched and (len(launched) == 1) == (copies == 1), launched
    r = lm.sample(x, p, history=h, uniforms=ut, return_tau=True, return_status=True)
    tok, tau, _ = oracle.sample_batch(cfg["logits"], temperature=cfg["temperature"], top_k=cfg["top_k"], top_p=top_p, history=np.tile(hist, (n, 1)), repetition_penalty=rho,
                                      presence_penalty=pi, draw="inverse_cdf", uniforms=u, n_threads=THREADS)
    np.testing.assert_array_equal(r.tau.cpu().numpy(), tau)
    np.testing.assert_array_equal(r.tokens.cpu().numpy(), tok)
    on_candidate_path = (r.status.cpu().numpy() & 64) != 0
    assert on_candidate_path[7::8].all() and not on_candidate_path[::8].any()


@pytest.mark.parametrize("top_k", [850, 1000])
def test_large_top_ks_at_the_largest_vocabularies_stay_on_the_candidate_path(top_k):
    """The cutoff accepts no more sampled logits than its list of candidates has room for (one stands for 32 here): of 256 rows of N(0, 2^2)
    about 1.5 % meet an unlucky sample and are handed on, where an eighth of them was when half as many samples again were accepted."""
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    x = torch.cat([(torch.randn(64, 262144, generator=g, device="cuda") * 2).to(torch.bfloat16) for _ in range(4)])
    r = lm.sample(x, lm.SamplingParams(temperature=0.8, top_k=top_k, top_p=0.9, seed=2), return_status=True)
    assert int((r.status & 64 == 0).sum()) <= 12                             # binomial(256, 0.015): beyond 12 in 1e-4 of all seeds


@pytest.mark.parametrize("vocab,grid,top_k", [(151936, 1.0, 450), (151936, 1.0, 1000), (151936, 0.5, 700), (151936, 0.25, 1000), (262144, 1.0, 100), (262144, 1.0, 300),
                                              (262144, 0.5, 450), (32768, 1.0, 100)])
def test_coarse_logits_stay_on_the_candidate_path(vocab, grid, top_k):
    """N(0, 2^2) rounded to a multiple of `grid`: neighbouring values are many BF16 codes and hundreds to thousands of candidates apart, and some value has
    between top_k and 2048 logits at or above it. A cutoff is taken from samples where they put it three standard deviations inside, one row
    in 700 wrongly (of 256 more than 4 in 1e-4 of all seeds), else the row is counted."""
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    x = torch.cat([(torch.round(torch.randn(64, vocab, generator=g, device="cuda") * (2.0 / grid)) * grid).to(torch.bfloat16) for _ in range(4)])
    p = dict(temperature=0.8, top_k=top_k, top_p=0.9, seed=2)
    assert "sample_topk_kernel" in routes.names(lambda: lm.sample(x, lm.SamplingParams(**p)))
    r = lm.sample(x, lm.SamplingParams(**p), return_status=True, return_tau=True)
    assert int((r.status & 64 == 0).sum()) <= 4
    exact = lm.sample(x, lm.SamplingParams(exact_only=True, **p), return_tau=True, return_status=True)
    near = ((r.status | exact.status) & 4) != 0
    assert torch.equal(r.tau, exact.tau) and bool(torch.all((r.tokens == exact.tokens) | near))


@pytest.mark.parametrize("rows,grid_limit", [(295, 0), (296, 0), (297, 0), (407, 0), (408, 0), (20, 16), (22, 16), (23, 16)])
def test_every_row_is_taken_where_half_the_blocks_leave_after_one(rows, grid_limit):
    """Rows up to, and just beyond, eleven eighths of the candidate kernel's blocks (two to each of 148 SMs, or a grid limit): each one is sampled, once and as
    by the exact kernels."""
    g = torch.Generator(device="cuda")
    g.manual_seed(rows)
    x = (torch.randn(rows, 40960, generator=g, device="cuda") * 2).to(torch.bfloat16)
    p, e = (lm.SamplingParams(temperature=0.8, top_k=30, top_p=0.9, seed=5, exact_only=exact, grid_limit=grid_limit) for exact in (False, True))
    assert "sample_topk_kernel" in routes.names(lambda: lm.sample(x, p)) or rows < 75
    out = torch.full((rows,), -7, dtype=torch.int32, device="cuda")
    r, q = lm.sample(x, p, return_tau=True, return_status=True, out=out), lm.sample(x, e, return_tau=True, return_status=True)
    assert torch.equal(r.tau, q.tau) and bool(torch.all((r.tokens == q.tokens) | (((r.status | q.status) & 4) != 0)))


def test_the_fp32_mass_of_rows_far_from_zero():
    """Logits around 100: the candidate kernel's mass must not carry the rounding of the slope log2(e) / T times the maximum (2e-5 at T 0.3), which
    its band does not hold. top_p a few 1e-6 on either side of a boundary of the cumulative mass inside the top-k set."""
    rng = np.random.default_rng(67)
    rows = []
    for r in range(16):
        T = np.float32(rng.uniform(0.25, 0.5))
        codes = oracle.f32_to_bf16((100.0 + 2.0 * rng.standard_normal(40000)).astype(np.float32))
        vals, counts = np.unique(oracle.bf16_to_f32(codes).astype(np.float64), return_counts=True)
        vals, counts = vals[::-1], counts[::-1]
        cum = np.cumsum(counts * np.exp((vals - vals[0]) / np.float64(T)))
        i = int(np.searchsorted(np.cumsum(counts), 100))
        for d in (0.0, 3e-6, -3e-6, 6e-6, -6e-6, 1.2e-5, -1.2e-5, 1e-4):
            rows.append((codes, T, np.float32(cum[i] / cum[-1] * (1.0 + d))))
    n = len(rows)
    cfg = dict(logits=np.stack([c for c, _, _ in rows]), temperature=np.array([t for _, t, _ in rows], np.float32), top_k=np.full(n, 500, np.int32),
               top_p=np.array([p for _, _, p in rows], np.float32), uniforms=np.linspace(0.02, 0.98, n).astype(np.float32))
    r, tok, tau = gpu_and_oracle(cfg)
    np.testing.assert_array_equal(r.tau.cpu().numpy(), tau)
    np.testing.assert_array_equal(r.tokens.cpu().numpy(), tok)


@pytest.mark.parametrize("vocab", [8, 264, 256 * 160, 256 * 160 + 8, 2 * 256 * 160 + 264, 262144])
@pytest.mark.parametrize("penalised", [False, True])
def test_the_histogram_draw_at_the_edges_of_its_batches(vocab, penalised):
    """The inverse-CDF draw counts equal logits in batches of 160 segments of 256, from the nearer end of the row. Runs of thousands of equal logits
    (multiples of 1/2) put the drawn one into any batch and segment; vocabularies of one batch, a chunk more, two batches and a ragged segment."""
    rows = 48
    rng = np.random.default_rng(vocab)
    codes = oracle.f32_to_bf16((np.round(rng.standard_normal((rows, vocab)) * 4.0) / 2.0).astype(np.float32))
    u = np.concatenate([[0.0, 1.0 - 2.0 ** -24], np.linspace(0.01, 0.99, rows - 2)]).astype(np.float32)
    hist = rng.integers(0, vocab, (rows, min(vocab, 1500))).astype(np.int32) if penalised else None
    pen = dict(repetition_penalty=2.0, presence_penalty=0.5) if penalised else {}
    T = rng.uniform(0.5, 3.0, rows).astype(np.float32)
    p = lm.SamplingParams(draw="inverse_cdf", exact_only=True, temperature=torch.from_numpy(T).cuda(), top_p=0.97, **pen)
    x, ut, h = bf16_tensor(codes), torch.from_numpy(u).cuda(), torch.from_numpy(hist).cuda() if penalised else None
    assert "sample_hist_kernel" in routes.names(lambda: lm.sample(x, p, history=h, uniforms=ut))
    r = lm.sample(x, p, history=h, uniforms=ut, return_tau=True, return_status=True)
    tok, tau, _ = oracle.sample_batch(codes, temperature=T, top_p=0.97, history=hist, draw="inverse_cdf", uniforms=u, n_threads=THREADS, **pen)
    np.testing.assert_array_equal(r.tau.cpu().numpy(), tau)
    np.testing.assert_array_equal(r.tokens.cpu().numpy(), tok)
    assert not np.any(r.status.cpu().numpy() & 1)                            # none handed on to the generic algorithm


@pytest.mark.parametrize("rows,vocab,top_k", [(80, 32768, 1), (80, 40008, 63), (80, 40008, 64), (80, 40008, 65), (400, 32768, 20), (400, 32768, 450), (80, 262144, 1024)])
@pytest.mark.parametrize("draw", ["inverse_cdf", "gumbel"])
def test_the_candidate_kernel_around_its_one_warp_finish_and_its_cutoff(rows, vocab, top_k, draw):
    """Up to 64 candidates down to the top-k crossing one warp finishes the row, beyond that the block; the cutoff of a block's first row comes from the
    threads' maxima, a later one's from the row before (400 rows: more than there are blocks), a large top_k's is corrected by a second sample.
    Ties at the crossing (half the rows are coarse) and penalised logits at the top of the row put 63 .. 66 candidates there."""
    rng = np.random.default_rng(vocab + top_k)
    z = rng.standard_normal((rows, vocab)).astype(np.float32) * 2.0
    z[::2] = np.round(z[::2] * 16.0) / 16.0
    codes = oracle.f32_to_bf16(z)
    hist = rng.integers(0, vocab, (rows, 200)).astype(np.int32)
    hist[:, :60] = np.argsort(-z, axis=1)[:, :120:2]
    T, top_p = rng.uniform(0.3, 1.5, rows).astype(np.float32), rng.uniform(0.5, 1.0, rows).astype(np.float32)
    u = rng.random(rows).astype(np.float32)
    x, h, ut = bf16_tensor(codes), torch.from_numpy(hist).cuda(), torch.from_numpy(u).cuda()
    for extra in (dict(), dict(min_p=0.02, topp_in_topk=True)):
        p = lm.SamplingParams(draw=draw, seed=7, temperature=torch.from_numpy(T).cuda(), top_k=top_k, top_p=torch.from_numpy(top_p).cuda(), repetition_penalty=1.2,
                              presence_penalty=0.3, **extra)
        assert vocab == 32768 and rows == 80 or "sample_topk_kernel" in routes.names(lambda: lm.sample(x, p, history=h, uniforms=ut))
        r = lm.sample(x, p, history=h, uniforms=ut, return_tau=True, return_status=True, return_vmax=True)
        tok, tau, _ = oracle.sample_batch(codes, temperature=T, top_k=top_k, top_p=top_p, history=hist, draw=draw, uniforms=u, seed=7, repetition_penalty=1.2,
                                          presence_penalty=0.3, n_threads=THREADS, **extra)
        status = r.status.cpu().numpy()
        np.testing.assert_array_equal(r.tau.cpu().numpy(), tau)
        assert np.all((r.tokens.cpu().numpy() == tok) | ((status & 4) != 0))
        if rows == 80:
            zf = oracle.bf16_to_f32(codes)
            for i in range(0, rows, 9):
                assert int(r.mass[i]) == oracle.kept_mass(oracle.apply_penalties(zf[i], hist[i], 1.2, 0.3), tau[i], T[i]), i
