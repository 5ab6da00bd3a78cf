"""The cluster row sampler (one row per thread-block cluster): what the streaming kernels do not take -- binary32 rows, ragged
vocabularies and misaligned rows, statistics and probabilities -- and batches too small to fill the GPU with a block per row.
Tokens and thresholds are the oracle's, bit for bit; probabilities and masses are binary32 roundings of FP64 sums (1e-6)."""
import numpy as np
import pytest
import torch

import oracle
import lithos_metal_b200 as lm
from tests import routes

pytestmark = pytest.mark.gpu


def _tensor(host):
    return torch.from_numpy(host.view(np.int16)).cuda().view(torch.bfloat16) if host.dtype == np.uint16 else torch.from_numpy(host).cuda()


def _check(x, host, knobs, *, draw, history=None, rho=1.0, pi=0.0, seed=3, step=5, row_offset=0, exact_only=False, topp_in_topk=False, stats=False):
    rows = x.shape[0]
    u = np.random.default_rng(seed + 7).random(rows).astype(np.float32)
    dev = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() if isinstance(v, np.ndarray) else v for k, v in knobs.items()}
    p = lm.SamplingParams(seed=seed, draw=draw, repetition_penalty=rho, presence_penalty=pi, exact_only=exact_only, topp_in_topk=topp_in_topk, **dev)
    r = lm.sample(x, p, history=None if history is None else torch.from_numpy(history).cuda(), uniforms=torch.from_numpy(u).cuda(), step=step,
                  row_offset=row_offset, return_tau=True, return_status=True, return_stats=stats, return_probs=stats, return_vmax=True)
    tok, tau, st = oracle.sample_batch(host, history=history, repetition_penalty=rho, presence_penalty=pi, draw=draw, uniforms=u, seed=seed, step=step,
                                       row_offset=row_offset, topp_in_topk=topp_in_topk, n_threads=8, **knobs)
    status = r.status.cpu().numpy()
    np.testing.assert_array_equal(r.tau.cpu().numpy(), tau)
    vmax, mass = r.vmax.cpu().numpy(), r.mass.cpu().numpy()
    z = oracle.bf16_to_f32(host) if host.dtype == np.uint16 else host
    for i in range(rows):                                                   # what the verification takes over: the maximum and the kept integer mass
        zi = z[i] if history is None else oracle.apply_penalties(z[i], history[i], rho, pi)
        t = knobs["temperature"][i] if isinstance(knobs["temperature"], np.ndarray) else knobs["temperature"]
        assert vmax[i] == zi.max(), i
        assert t == 0 or int(mass[i]) == oracle.kept_mass(zi, tau[i], t), i
    assert np.all((r.tokens.cpu().numpy() == tok) | ((status & 4) != 0)), np.nonzero(r.tokens.cpu().numpy() != tok)
    if stats:
        np.testing.assert_allclose(r.stats.cpu().numpy(), st, rtol=1e-6)
        pr = r.probs.cpu().numpy().astype(np.float64)
        np.testing.assert_allclose(pr.sum(-1), 1.0, rtol=1e-5)
        for i in range(rows):
            zi = z[i] if history is None else oracle.apply_penalties(z[i], history[i], rho, pi)
            t = knobs["temperature"][i] if isinstance(knobs["temperature"], np.ndarray) else knobs["temperature"]
            e = np.where(zi >= tau[i], np.exp((zi.astype(np.float64) - float(zi.max())) / np.float64(np.float32(t))), 0.0)
            np.testing.assert_allclose(pr[i], e / e.sum(), rtol=1e-6, atol=1e-40)
    return r, status


def _mixed(rng, rows, top_ks=(0, 1, 20, 50, 1000)):
    return dict(temperature=rng.uniform(0.3, 1.5, rows).astype(np.float32), top_k=rng.choice(np.array(top_ks, np.int32), rows),
                top_p=rng.uniform(0.7, 1.02, rows).astype(np.float32), min_p=rng.choice(np.array([0.0, 0.0, 0.03], np.float32), rows))


# rows choose the blocks per row (16 / 8 / 4 / 2 / 1), vocabularies the edges of chunks (8), of the smallest slices (2048) and of the
# blocks' sweeps (8192 logits), views the alignment of the rows
@pytest.mark.parametrize("rows,vocab", [(1, 151936), (8, 40001), (9, 16385), (19, 8191), (38, 50257), (75, 4099), (150, 2049), (3, 1), (5, 9), (2, 262139)])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("draw", ["inverse_cdf", "gumbel"])
def test_rows_and_sizes(rows, vocab, dtype, draw):
    rng = np.random.default_rng(rows * 7 + vocab)
    z = (rng.standard_normal((rows, vocab)) * 2).astype(np.float32)
    host = oracle.f32_to_bf16(z) if dtype == "bf16" else z
    hist = rng.integers(-3, vocab + 3, (rows, 300)).astype(np.int32)
    _check(_tensor(host), host, _mixed(rng, rows), draw=draw, history=hist, rho=1.2, pi=0.3, row_offset=11)
    wide = np.zeros((rows, vocab + 5), host.dtype)                          # a view with an offset: another alignment for every row
    wide[:, 3:3 + vocab] = host
    _check(_tensor(wide)[:, 3:3 + vocab], host, _mixed(rng, rows, (0,)), draw=draw)


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("rows", [2, 40])
def test_statistics_and_probabilities(dtype, rows):
    rng = np.random.default_rng(rows)
    z = (rng.standard_normal((rows, 30011)) * 2).astype(np.float32)
    host = oracle.f32_to_bf16(z) if dtype == "bf16" else z
    hist = rng.integers(0, 30011, (rows, 100)).astype(np.int32)
    knobs = _mixed(rng, rows)
    _, status = _check(_tensor(host), host, knobs, draw="gumbel", history=hist, rho=1.1, pi=0.5, stats=True)
    assert np.all(status & 1)                                              # reported for such calls, whoever serves them
    _check(_tensor(host), host, dict(temperature=0.9, top_k=0, top_p=0.0, min_p=0.0), draw="inverse_cdf", stats=True)


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_without_lists_of_the_top_k(dtype):
    """Crossing bins for everything: a top_k beyond the list, and exact_only; top-p inside the top-k set."""
    rng = np.random.default_rng(5)
    z = (rng.standard_normal((6, 65543)) * 2).astype(np.float32)
    host = oracle.f32_to_bf16(z) if dtype == "bf16" else z
    for kw in (dict(), dict(exact_only=True), dict(topp_in_topk=True), dict(exact_only=True, topp_in_topk=True)):
        for draw in ("inverse_cdf", "gumbel"):
            _, status = _check(_tensor(host), host, _mixed(rng, 6, (3, 700, 1500, 5000)), draw=draw, **kw)
            assert np.count_nonzero(status & 1) <= 1


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_rows_that_are_handed_on_and_degenerate_rows(dtype):
    V = 40000
    rng = np.random.default_rng(9)
    z = (rng.standard_normal((8, V)) * 2).astype(np.float32)
    z[0] = 1.5                                                              # every logit equal: no list holds the bin
    z[1, 100:] = -np.inf                                                    # a masked row
    z[2, ::2] = -1e9                                                        # masked by a large negative number
    z[3, 5:4000] = 9.0                                                      # more ties at the top than a list holds
    z[4] *= 300.0                                                           # nearly greedy
    z[5] *= 1e-3                                                            # nearly uniform
    z[6, 17] = 80.0                                                         # one logit far above the rest
    host = oracle.f32_to_bf16(z) if dtype == "bf16" else z
    for draw in ("inverse_cdf", "gumbel"):
        for k in (0, 30, 2000):
            knobs = dict(temperature=np.full(8, 0.8, np.float32), top_k=np.full(8, k, np.int32), top_p=np.full(8, 0.9, np.float32), min_p=np.zeros(8, np.float32))
            knobs["temperature"][7] = 0.0
            _check(_tensor(host), host, knobs, draw=draw)
    x = _tensor(host).clone()
    x[2, 77] = float("nan"); x[3, 9] = float("inf")
    r = lm.sample(x, lm.SamplingParams(temperature=0.8, top_p=0.9, seed=1), return_status=True)
    st = r.status.cpu().numpy()
    assert st[2] & 2 and st[2] & 1 and st[3] & 1 and not np.any(st[[1, 4, 5, 6, 7]] & 3)


def test_a_top_p_boundary_inside_the_error_bound_is_decided_in_fp64():
    """top_p placed on (and a hair beside) an exact boundary of the cumulative mass: the coarse sums hand the decision to the fine ones."""
    rng = np.random.default_rng(21)
    rows = []
    z0 = oracle.bf16_to_f32(oracle.f32_to_bf16((rng.standard_normal(60000) * 2).astype(np.float32)))
    vals, counts = np.unique(z0.astype(np.float64), return_counts=True)
    vals, counts = vals[::-1], counts[::-1]
    cum = np.cumsum(counts * np.exp(vals - vals[0]))
    for i in (40, 200, 600):
        for d in (0.0, 1e-8, -1e-8, 1e-7, -1e-7, 1e-6, -1e-6, 1e-5, -1e-5):
            rows.append(np.float32(cum[i] / cum[-1] * (1.0 + d)))
    n = len(rows)
    for host in (np.tile(oracle.f32_to_bf16(z0), (n, 1)), np.tile(z0, (n, 1))):
        for k in (0, 1000):
            knobs = dict(temperature=1.0, top_k=np.full(n, k, np.int32), top_p=np.array(rows, np.float32), min_p=0.0)
            _check(_tensor(host), host, knobs, draw="inverse_cdf")


# the edges of the rule for the blocks per row on 148 SMs (16 / 8 / 4 / 2 / 1 of them), by rows and by the length of a row
@pytest.mark.parametrize("rows,vocab", [(7, 33001), (15, 33001), (16, 33001), (32, 20011), (33, 49153), (49, 49153), (50, 98305), (75, 98305), (98, 20011), (99, 40001), (297, 40001)])
@pytest.mark.parametrize("draw", ["inverse_cdf", "gumbel"])
def test_every_split_of_a_batch(rows, vocab, draw):
    rng = np.random.default_rng(rows + vocab)
    host = (rng.standard_normal((rows, vocab)) * 2).astype(np.float32)
    _check(_tensor(host), host, _mixed(rng, rows), draw=draw)
    _check(_tensor(host), host, dict(temperature=0.8, top_k=30, top_p=0.9, min_p=0.0), draw=draw)   # one top_k for every row


# BF16 rows that the streaming kernels take: a row per SM, two, more, and enough for one kernel behind the other
@pytest.mark.parametrize("rows", [38, 148, 149, 296, 297, 741])
@pytest.mark.parametrize("draw", ["inverse_cdf", "gumbel"])
@pytest.mark.parametrize("penalised", [False, True])
def test_streaming_batches_of_every_geometry(rows, draw, penalised):
    vocab = 32776                                                           # the last chunk of a step is alone
    rng = np.random.default_rng(rows)
    host = oracle.f32_to_bf16((rng.standard_normal((rows, vocab)) * 2).astype(np.float32))
    kw = dict(history=rng.integers(0, vocab, (rows, 700)).astype(np.int32), rho=1.1, pi=0.5) if penalised else {}
    _check(_tensor(host), host, _mixed(rng, rows, (0, 0, 20, 50, 1000)), draw=draw, **kw)
    _check(_tensor(host), host, dict(temperature=0.9, top_k=0, top_p=0.9, min_p=0.0), draw=draw, **kw)


# BF16 batches on both sides of the lines between clusters and streaming kernels (rows per SM, length of a row)
@pytest.mark.parametrize("rows,vocab", [(74, 40000), (74, 40008), (74, 65536), (74, 65544), (75, 40000), (148, 40000), (148, 40008), (149, 40000)])
@pytest.mark.parametrize("top_k", ["per row", 30, 0])
def test_batches_at_the_lines_between_the_kernels(rows, vocab, top_k):
    rng = np.random.default_rng(rows + vocab)
    host = oracle.f32_to_bf16((rng.standard_normal((rows, vocab)) * 2).astype(np.float32))
    knobs = _mixed(rng, rows) if top_k == "per row" else dict(temperature=0.8, top_k=top_k, top_p=0.9, min_p=0.0)
    hist = rng.integers(0, vocab, (rows, 400)).astype(np.int32) if top_k != 0 else None
    _check(_tensor(host), host, knobs, draw="inverse_cdf" if top_k != 0 else "gumbel", history=hist, rho=1.1, pi=0.5)


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_thresholds_at_very_small_temperatures(dtype):
    """top-p next to a top_k where the exponent of the maximum, vmax log2(e) / T, is far beyond what binary32 resolves: the kept set is the
    maximum (and its ties) alone. Up to 64 candidates and more, the clusters and the streaming kernels; and a maximum of 1e10."""
    rng = np.random.default_rng(13)
    for rows in (40, 80):
        z = (rng.standard_normal((rows, 40008)) * 2).astype(np.float32)
        z[1, 500], z[1, 7000] = 13.0, 13.0
        z[2, 123] = 1e10
        host = oracle.f32_to_bf16(z) if dtype == "bf16" else z
        for t in (1e-6, 1e-8, 3e-9, 1e-9, 1e-12):
            for k in (50, 200):
                knobs = dict(temperature=np.full(rows, t, np.float32), top_k=np.full(rows, k, np.int32), top_p=np.full(rows, 0.9, np.float32), min_p=0.0)
                _check(_tensor(host), host, knobs, draw="gumbel" if k == 50 else "inverse_cdf")


def _masked(rng, rows, vocab, mask, dtype):
    """Logits of which a third and the first eighth carry a mask's value."""
    z = (rng.standard_normal((rows, vocab)) * 2).astype(np.float32)
    z[rng.random((rows, vocab)) < 1 / 3] = mask
    z[:, : vocab // 8] = mask
    return oracle.f32_to_bf16(z) if dtype == "bf16" else z


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("mask", [-1e4, -1e9, -3.3e38])
def test_a_large_negative_mask_is_no_reason_for_the_generic_algorithm(dtype, mask):
    rng = np.random.default_rng(41)
    host = _masked(rng, 8, 40008, mask, dtype)
    for k, p in ((0, 0.9), (50, 0.9), (1000, 0.9)):
        for draw in ("inverse_cdf", "gumbel"):
            knobs = dict(temperature=np.full(8, 0.8, np.float32), top_k=np.full(8, k, np.int32), top_p=np.full(8, p, np.float32), min_p=0.0)
            _, status = _check(_tensor(host), host, knobs, draw=draw)
            assert not np.any(status & 1), (k, draw, status)


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("mask", [-1e3, -1e4, -1e9, -3.3e38])
@pytest.mark.parametrize("rows,vocab", [(1, 2048), (8, 40008), (50, 30011), (100, 16395)])
def test_a_masked_row_keeps_the_list_of_its_top_k(dtype, mask, rows, vocab):
    """Groups of nothing but masked logits do not spoil the bound of the top_k-th logit: the row stays on the list (status 64)."""
    rng = np.random.default_rng(rows + vocab)
    host = _masked(rng, rows, vocab, mask, dtype)
    for k in (1, 50, 200):
        knobs = dict(temperature=np.full(rows, 0.8, np.float32), top_k=np.full(rows, k, np.int32), top_p=np.full(rows, 0.9, np.float32), min_p=0.0)
        _, status = _check(_tensor(host), host, knobs, draw="gumbel")
        assert np.count_nonzero(status & 64) >= rows - 1, (k, status)       # (a top-p boundary inside the FP32 mass's band leaves it)


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("mask", [0.0, -1e4, -1e9, -3.3e38])
def test_a_count_is_found_wherever_it_crosses(dtype, mask):
    """A top_k beyond the list, and exact_only: the k-th logit next to a mask's value that stretches the bins, and deeper than the weights
    reach (a low temperature). More equal logits at the crossing than a list holds are left to the generic algorithm."""
    rng = np.random.default_rng(43)
    host = _masked(rng, 6, 65543, mask, dtype) if mask else _masked(rng, 6, 65543, 0.5, dtype)
    for k, exact in ((2000, False), (9000, False), (50, True)):
        for t, p in ((0.8, 0.0), (0.8, 0.9), (0.05, 0.9), (1e-9, 0.0)):
            for draw in ("inverse_cdf", "gumbel"):
                knobs = dict(temperature=np.full(6, t, np.float32), top_k=np.full(6, k, np.int32), top_p=np.full(6, p, np.float32), min_p=0.0)
                _, status = _check(_tensor(host), host, knobs, draw=draw, exact_only=exact)
                assert not np.any(status & 1) or (not mask and k == 9000), (k, t, p, draw, status)
    knobs = dict(temperature=np.full(6, 0.8, np.float32), top_k=np.full(6, 60000, np.int32), top_p=np.full(6, 0.9, np.float32), min_p=0.0)
    _check(_tensor(host), host, knobs, draw="inverse_cdf", exact_only=True)  # the k-th is one of the masked


def test_every_warp_looks_the_thresholds_bin_up_in_the_same_window():
    """A bin that holds more than a list, met by the threshold's own step (no barrier of a list in between): hundreds of rows whose logits lie
    within a few units in the last place of one another, a third of them far below, thresholds from a top_k and a top_p close to 1."""
    rng = np.random.default_rng(47)
    z = (rng.standard_normal((148, 4096)) * 1e-4 + 100.0).astype(np.float32)
    z[:, ::3] -= 40.0
    for top_p in (0.9999999, 0.95, 0.5):
        for draw in ("gumbel", "inverse_cdf"):
            knobs = dict(temperature=np.full(148, 50.0, np.float32), top_k=np.full(148, 1000, np.int32), top_p=np.full(148, top_p, np.float32), min_p=0.0)
            for _ in range(5):
                _check(_tensor(z), z, knobs, draw=draw)


@pytest.mark.parametrize("rows,vocab", [(48, 49157), (300, 1003), (2048, 515), (2049, 515)])
def test_more_clusters_than_run_at_once_take_every_row_once(rows, vocab):
    """Batches of more clusters than the device holds take their rows by kind (no top_k, a large one, the rest, greedy), up to 2048 rows of them: every
    row's token and threshold are its own, whatever the mixture and the number of rows."""
    rng = np.random.default_rng(rows)
    z = (rng.standard_normal((rows, vocab)) * 2.0).astype(np.float32)
    top_k = rng.choice(np.array([0, 0, 20, 64, 65, 1000, 1025, 2000], np.int32), rows)
    T = np.where(rng.random(rows) < 0.1, 0.0, rng.uniform(0.3, 1.5, rows)).astype(np.float32)
    u = rng.random(rows).astype(np.float32)
    p = lm.SamplingParams(draw="inverse_cdf", temperature=torch.from_numpy(T).cuda(), top_k=torch.from_numpy(top_k).cuda(), top_p=0.9)
    x, ut = torch.from_numpy(z).cuda(), torch.from_numpy(u).cuda()
    tok, tau, _ = oracle.sample_batch(z, temperature=T, top_k=top_k, top_p=0.9, draw="inverse_cdf", uniforms=u, n_threads=8)
    runs = [lm.sample(x, p, uniforms=ut, return_tau=True, out=torch.full((rows,), -7, dtype=torch.int32, device="cuda")) for _ in range(30)]   # (in a row)
    for r in runs:
        np.testing.assert_array_equal(r.tokens.cpu().numpy(), tok)
        np.testing.assert_array_equal(r.tau.cpu().numpy(), tau)


@pytest.mark.parametrize("rows", [1, 4, 100, 760])
def test_calls_in_a_row_see_what_the_one_before_them_left(rows):
    """Kernels are made ready beside the one in front of them in the stream and wait for it. Chains of this library's calls with no other kernel in between
    (few rows; streaming kernels with one top_k, none, or the rows' own): each reads what the one right before it wrote -- its tokens as a history, its
    logits -- or writes over what that one read, and all share one workspace. The same as with the device idle between any two."""
    vocab, H = 40960, 512
    g = torch.Generator(device="cuda")
    g.manual_seed(rows)
    x = (torch.randn(rows, vocab, generator=g, device="cuda") * 2).to(torch.bfloat16)
    pen = dict(repetition_penalty=1.3, presence_penalty=4.0)
    p = lm.SamplingParams(temperature=0.8, top_p=0.9, seed=3, **pen)
    q = lm.SamplingParams(temperature=0.8, top_k=20, top_p=0.9, seed=3, **pen)
    own = lm.SamplingParams(temperature=0.8, top_k=torch.tensor([0, 20, 700], dtype=torch.int32, device="cuda").repeat(rows // 3 + 1)[:rows].contiguous(), top_p=0.9, seed=3, **pen)
    few = min(rows, 8)
    hidden = [(torch.randn(few, H, generator=g, device="cuda") * (i + 1)).to(torch.bfloat16) for i in range(3)]
    weight = (torch.randn(vocab, H, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    first = torch.zeros(rows, dtype=torch.int32, device="cuda")
    steps = 12
    tokens = [[torch.empty(rows, dtype=torch.int32, device="cuda") for _ in range(7 * steps)] for _ in range(2)]
    drawn = [[torch.empty(few, dtype=torch.int32, device="cuda") for _ in range(6 * steps)] for _ in range(2)]
    logits = torch.empty(few, vocab, dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()

    def run(arm, wait):
        def then(_):
            if wait:
                torch.cuda.synchronize()
        last, t, d = first, iter(tokens[arm]), iter(drawn[arm])
        for step in range(steps):
            for params in (p, q, own, q, p, own):                           # the last call's tokens are this one's history
                now = next(t)
                then(lm.sample(x, params, history=last[:, None], step=step, out=now))
                last = now
            then(lm.argmax(x, out=next(t)))
            for h in hidden:                                                # logits written over as soon as they have been drawn from
                then(lm.lm_head(h, weight, out=logits))
                then(lm.sample(logits, q if step % 2 else p, history=last[:few, None], step=step, out=next(d)))
                then(lm.argmax(logits, out=next(d)))

    run(0, False)
    torch.cuda.synchronize()
    run(1, True)
    for a, b in zip(tokens[0] + drawn[0], tokens[1] + drawn[1]):
        assert torch.equal(a, b)
    assert len({tuple(v.tolist()) for v in tokens[1][::7]}) > 1             # (the chain moves)


@pytest.mark.parametrize("rows,vocab,top_k", [(38, 66001, 50), (64, 262144, 50), (65, 262144, 1000), (74, 151936, 1)])
def test_one_top_k_for_all_rows_of_half_the_gpu(rows, vocab, top_k):
    """BF16 batches of up to half a row per SM with one top_k: two or four blocks to a row, whatever its length."""
    rng = np.random.default_rng(vocab)
    host = oracle.f32_to_bf16((rng.standard_normal((rows, vocab)) * 2).astype(np.float32))
    knobs = dict(temperature=np.float32(0.8), top_k=top_k, top_p=np.float32(0.9), min_p=np.float32(0.0))
    u = rng.random(rows).astype(np.float32)
    for draw in ("inverse_cdf", "gumbel"):
        p = lm.SamplingParams(draw=draw, seed=5, **{k: v if k == "top_k" else float(v) for k, v in knobs.items()})
        r = lm.sample(_tensor(host), p, uniforms=torch.from_numpy(u).cuda(), return_tau=True, return_status=True)
        tok, tau, _ = oracle.sample_batch(host, draw=draw, seed=5, uniforms=u, n_threads=8, **knobs)
        near = r.status.cpu().numpy() & 4
        np.testing.assert_array_equal(r.tau.cpu().numpy(), tau)
        assert np.all((r.tokens.cpu().numpy() == tok) | (near != 0))


@pytest.mark.parametrize("rows,vocab,top_k,dtype,blocks", [(64, 196608, 50, "bf16", 2), (64, 196608, 1000, "bf16", 4), (48, 229376, 50, "bf16", 2), (56, 229376, 50, "bf16", 4),
                                                           (40, 262144, 50, "bf16", 2), (65, 262144, 50, "bf16", 2), (40, 196608, 20, "f32", 4), (64, 196608, 20, "f32", 2)])
def test_blocks_to_a_row_with_one_top_k(rows, vocab, top_k, dtype, blocks):
    """33 to 64 long rows with one top_k: two blocks to a row, or four where those measured faster (the line is made for 148 SMs); the same results."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines depend on the number of SMs")
    g = torch.Generator(device="cuda")
    g.manual_seed(rows)
    x = torch.randn(rows, vocab, generator=g, device="cuda") * 2
    x = x.to(torch.bfloat16) if dtype == "bf16" else x
    p, e = (lm.SamplingParams(temperature=0.8, top_k=top_k, top_p=0.9, seed=5, exact_only=exact) for exact in (False, True))
    assert [k[:2] for k in routes.kernels(lambda: lm.sample(x, p))[0]] == [("sample_cluster_kernel", rows * blocks)]
    r, q = (lm.sample(x, params, return_tau=True, return_status=True) for params in (p, e))
    assert torch.equal(r.tau, q.tau) and bool(torch.all((r.tokens == q.tokens) | (((r.status | q.status) & 4) != 0)))


@pytest.mark.parametrize("vocab", [16384, 40964, 151936])
@pytest.mark.parametrize("top_k", [0, 20, 700])
def test_probabilities_of_aligned_and_ragged_rows(vocab, top_k):
    """The kept mass comes from the ordered top-k set where there is one, and probabilities are written 16 bytes at a time where a row's slice of the output
    is aligned (a vocabulary of 40,964: its last chunk is not whole, and BF16 rows begin at odd offsets)."""
    rng = np.random.default_rng(vocab + top_k)
    z = (rng.standard_normal((3, vocab)) * 2).astype(np.float32)
    hist = rng.integers(0, vocab, (3, 100)).astype(np.int32)
    knobs = dict(temperature=np.float32([0.7, 1.0, 1.4]), top_k=np.full(3, top_k, np.int32), top_p=np.float32([0.95, 0.0, 0.8]), min_p=np.float32([0.0, 0.01, 0.0]))
    for host in (z, oracle.f32_to_bf16(z)):
        _check(_tensor(host), host, knobs, draw="inverse_cdf", history=hist, rho=1.1, pi=0.5, stats=True)
