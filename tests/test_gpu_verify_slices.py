"""The verification's slices: every way a row can lie in memory and be cut, every draw, against the CPU oracle (exact)."""
import numpy as np
import pytest
import torch

import lithos_metal_b200 as lm
import oracle
from tests.test_gpu_sampling import bf16_tensor

pytestmark = pytest.mark.gpu


def step(vocab, n, dtype, seed):
    rng = np.random.default_rng(seed)
    z = (rng.standard_normal((n + 1, vocab)) * 2.0).astype(np.float32)
    codes = oracle.f32_to_bf16(z)
    target = codes if dtype == "bf16" else z
    noisy = oracle.bf16_to_f32(codes)[:n] + (rng.standard_normal((n, vocab)) * 0.5).astype(np.float32)
    e = np.exp((noisy - noisy.max(-1, keepdims=True)).astype(np.float64))
    q = (e / e.sum(-1, keepdims=True)).astype(np.float32)
    return rng, target, noisy, q


LAST = np.float32(1.0 - 2.0**-24)                                            # the largest uniform


def rejecting(z, q, at, T=1.0, tau=None):
    """Drafts and accept uniforms of which the one at `at` is the first to be rejected: likely tokens before it, from it on the one where q exceeds p by most."""
    n = len(q)
    drafts, ua = z[:n].argmax(-1).astype(np.int32), np.zeros(n, np.float32)
    for r in range(at, n):
        p = np.exp((z[r].astype(np.float64) - z[r].max()) / T) * (True if tau is None else z[r] >= tau[r])
        drafts[r], ua[r] = np.argmax(q[r] - p / p.sum()), LAST
    return drafts, ua


def on_gpu(target):
    return bf16_tensor(target) if target.dtype == np.uint16 else torch.from_numpy(target).cuda()


def check(target, drafts, q, ua, uf, gpu_q=None, **kw):
    """Stochastic, then with the row maxima and the masses handed over: the oracle's accept length, token and p(draft)."""
    tau, T = kw.get("tau"), kw.get("temperature", 1.0)
    acc, fin, pd = oracle.verify_stochastic(target, drafts, q, ua, uf, temperature=T, tau=tau)
    x = on_gpu(target)
    z = oracle.bf16_to_f32(target) if target.dtype == np.uint16 else target
    vmax = z.max(-1)
    mass = np.array([oracle.kept_mass(z[r], -np.inf if tau is None else tau[r], T) for r in range(len(z))], dtype=np.uint64)
    given = dict(target_vmax=torch.from_numpy(vmax).cuda())
    for more in ({}, given, dict(given, target_mass=torch.from_numpy(mass.view(np.int64)).cuda())):
        out = lm.verify(x, torch.from_numpy(drafts).cuda(), None if gpu_q else torch.from_numpy(q).cuda(), torch.from_numpy(ua).cuda(), torch.tensor([uf]), "stochastic",
                        temperature=T, tau=None if tau is None else torch.from_numpy(tau).cuda(), return_p_draft=True, **(gpu_q or {}), **more)
        assert (int(out[0]), int(out[1])) == (acc, fin), more.keys()
        assert out[2].tolist() == drafts[:acc].tolist() + [fin] + [-1] * (len(drafts) - acc)
        np.testing.assert_array_equal(out[3].cpu().numpy(), pd)
        # the reference's form of the draw (a token only where its two logarithms leave no doubt: they are library functions)
        acc_g, fin_g, gap = oracle.verify_gumbel(target, drafts, q, seed=17, step=5, temperature=T, tau=tau, u_accept=ua)
        out = lm.verify(x, torch.from_numpy(drafts).cuda(), None if gpu_q else torch.from_numpy(q).cuda(), torch.from_numpy(ua).cuda(), None, "stochastic",
                        temperature=T, tau=None if tau is None else torch.from_numpy(tau).cuda(), residual_draw="gumbel", seed=17, step=5, **(gpu_q or {}), **more)
        assert int(out[0]) == acc_g and (int(out[1]) == fin_g or gap < 1e-5), more.keys()


# one block a row, a few, sixteen; vocabularies that are no multiple of 8 (rows at every alignment); one draft, and so many that a row gets eight blocks; slices that
# fit shared memory without the drafter's ((151936, 15), (262144, 7), (262143, 7)) and that do not fit at all ((262144, 14), (700001, 2))
@pytest.mark.parametrize("vocab,n,dtype", [(1, 1, "bf16"), (9, 2, "fp32"), (2049, 3, "bf16"), (4095, 15, "fp32"), (32769, 1, "bf16"), (50257, 7, "bf16"), (50257, 7, "fp32"),
                                           (151936, 15, "bf16"), (151937, 13, "fp32"), (262144, 7, "bf16"), (262143, 7, "fp32"), (262144, 14, "fp32"), (700001, 2, "bf16")])
def test_slices_of_every_shape(vocab, n, dtype):
    rng, target, noisy, q = step(vocab, n, dtype, vocab + n)
    ua, uf = rng.random(n).astype(np.float32), np.float32(rng.random())
    z = oracle.bf16_to_f32(target) if target.dtype == np.uint16 else target
    random, likely = rng.integers(0, vocab, n).astype(np.int32), z[:n].argmax(-1).astype(np.int32)
    for d, u in ((random, ua), (likely, np.zeros(n, np.float32)), (np.where(np.arange(n) < n // 2, likely, random).astype(np.int32), ua)):
        check(target, d, q, u, uf)
    for at in {0, n // 2, n - 1}:                                            # and with a rejected draft for certain
        d, u = rejecting(z, q, at)
        assert vocab == 1 or oracle.verify_stochastic(target, d, q, u, uf)[0] == at
        check(target, d, q, u, uf)
    acc, fin, toks = oracle.verify_greedy(target, likely)
    out = lm.verify(on_gpu(target), torch.from_numpy(likely).cuda(), mode="greedy")
    assert (int(out[0]), int(out[1])) == (acc, fin)
    # the drafter's BF16 logits in the place of its probabilities
    lb = oracle.f32_to_bf16(noisy)
    stats = lm.draft_q(bf16_tensor(lb), temperature=0.7, seed=3)
    q2 = np.stack([oracle.draft_probs(lb[k], temperature=0.7, vmax=float(stats.vmax[k]), mass=int(stats.mass[k])) for k in range(n)])
    for d, u in ((random, ua), rejecting(z, q2, n // 2, 0.7)):
        check(target, d, q2, u, uf, gpu_q=dict(draft_logits=bf16_tensor(lb), draft_stats=stats), temperature=0.7)


@pytest.mark.parametrize("dtype", ["bf16", "fp32"])
def test_draws_where_little_is_left(dtype):
    """Thresholds that keep a few logits, a residual that is empty (the row's own kept softmax is drawn from), masked rows, rows of one value, temperatures at which
    all but a few weights vanish, uniforms at both ends."""
    vocab, n = 40001, 4
    rng, target, _, q = step(vocab, n, dtype, 5)
    z = oracle.bf16_to_f32(target) if target.dtype == np.uint16 else target
    masked = z.copy()
    masked[:, ::3] = -np.inf
    masked[1, :] = -np.inf
    masked[1, 777] = -3.0
    masked[2, :] = 1.5
    masked = oracle.f32_to_bf16(masked) if dtype == "bf16" else masked
    ends = np.float32(1.0 - 2.0**-24)
    likely = z[:n].argmax(-1).astype(np.int32)
    for t in (target, masked):
        zt = oracle.bf16_to_f32(t) if t.dtype == np.uint16 else t
        some = rng.integers(0, vocab, n).astype(np.int32)
        for T in (0.05, 1.0, 7.0):
            tau = np.sort(zt, axis=-1)[:, -20].astype(np.float32)
            for uf in (np.float32(0.0), ends):
                for kept in (None, tau):
                    check(t, some, q, np.full(n, 0.5, np.float32), uf, temperature=T, tau=kept)
                    check(t, likely, np.ones_like(q), np.full(n, ends), uf, temperature=T, tau=kept)   # q = 1 everywhere: nothing of p - q is left
                check(t, np.array([-1, vocab, 2**30, -2**31], dtype=np.int32), q, np.zeros(n, np.float32), uf, temperature=T)   # ids outside the vocabulary: p = 0
    nothing = np.full((n + 1, vocab), -np.inf, np.float32)
    check(oracle.f32_to_bf16(nothing) if dtype == "bf16" else nothing, likely, q, np.full(n, 0.5, np.float32), np.float32(0.3))
