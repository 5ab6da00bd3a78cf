"""Replacement tokens of rejected drafts (the draw over max(p - q, 0)) in every layout of the verification's slices: the drafter's row beside the target's in shared
memory, the target's alone, neither. Every case asserts that a draft was rejected and that something of p - q is left. Against the CPU oracle (exact)."""
import numpy as np
import pytest
import torch

import lithos_metal_b200 as lm
import oracle
from lithos_metal_b200 import _lib
from tests.test_gpu_sampling import bf16_tensor
from tests.test_gpu_verify_slices import LAST, check, on_gpu, rejecting, step

pytestmark = pytest.mark.gpu


# 16 blocks a row up to 13 drafts, 8 beyond: (50257, 7) holds both rows, (700001, 2) neither (two launches), the others the target's alone
@pytest.mark.parametrize("vocab,n", [(248320, 1), (248320, 7), (262144, 7), (262143, 13), (151936, 14), (151936, 15), (50257, 7), (700001, 2)])
@pytest.mark.parametrize("dtype", ["bf16", "fp32"])
def test_first_rejected_draft_is_replaced(vocab, n, dtype):
    rng, target, noisy, q = step(vocab, n, dtype, vocab + 3 * n)
    z = oracle.bf16_to_f32(target) if dtype == "bf16" else target
    lb = oracle.f32_to_bf16(noisy)
    stats = lm.draft_q(bf16_tensor(lb), temperature=0.7, seed=3)
    q2 = np.stack([oracle.draft_probs(lb[k], temperature=0.7, vmax=float(stats.vmax[k]), mass=int(stats.mass[k])) for k in range(n)])
    tau = np.partition(z, vocab - min(300, vocab), axis=-1)[:, vocab - min(300, vocab)].astype(np.float32)
    for at in sorted({0, n // 2, n - 1}):
        for kept in (None, tau):
            d, ua = rejecting(z, q, at, tau=kept)
            acc, fin, _ = oracle.verify_stochastic(target, d, q, ua, 0.5, tau=kept)
            assert acc == at and fin >= 0
            for uf in (rng.random(), 0.0, LAST):
                check(target, d, q, ua, np.float32(uf), tau=kept)
        d, ua = rejecting(z, q2, at, 0.7)
        assert oracle.verify_stochastic(target, d, q2, ua, 0.5, temperature=0.7)[0] == at
        check(target, d, q2, ua, np.float32(rng.random()), gpu_q=dict(draft_logits=bf16_tensor(lb), draft_stats=stats), temperature=0.7)


@pytest.mark.parametrize("vocab,n", [(248320, 7), (400001, 7), (262144, 15)])   # (the last two in two launches)
@pytest.mark.parametrize("draft_form", ["probabilities", "logits"])
def test_replaced_in_a_round_that_closes_itself(draft_form, vocab, n):
    """With a StepState that the launch reads and moves on: the state's token is the oracle's."""
    at, T = 3, 0.7
    layout = lm.StepStateLayout(n + 1, n)
    rng, target, noisy, q = step(vocab, n, "bf16", 11)
    z = oracle.bf16_to_f32(target)
    lb = oracle.f32_to_bf16(noisy)
    stats = lm.draft_q(bf16_tensor(lb), temperature=T, seed=3)
    if draft_form == "logits":
        q = np.stack([oracle.draft_probs(lb[k], temperature=T, vmax=float(stats.vmax[k]), mass=int(stats.mass[k])) for k in range(n)])
    d, ua = rejecting(z, q, at, T)
    uf = np.float32(rng.random())
    acc, fin, _ = oracle.verify_stochastic(target, d, q, ua, uf, temperature=T)
    assert acc == at
    st = layout.to_device(dict(step=2, verify_len=n, t_this_step=n + 1, pending_tokens=[5] + d.tolist(), position=40, kv_len=40))
    ring = torch.zeros(64, dtype=torch.int64, device="cuda")
    out = lm.verify(on_gpu(target), None, torch.from_numpy(q).cuda() if draft_form == "probabilities" else None, torch.from_numpy(ua).cuda(), torch.tensor([uf]), "stochastic",
                    temperature=T, step_state=(layout, st), commit=dict(layout=layout, state=st, ring=ring),
                    **(dict(draft_logits=bf16_tensor(lb), draft_stats=stats) if draft_form == "logits" else {}))
    assert (int(out[0]), int(out[1])) == (acc, fin)
    after = layout.from_device(st)
    assert [int(t) & 0xFFFFFFFF for t in ring[:acc + 1].tolist()] == d[:acc].tolist() + [fin]
    assert after["anchor"] == fin and after["accepted"] == at and after["step"] == 3


# every layout again (both rows in shared memory, the target's alone, neither), a threshold that cuts nothing, statistics given or not (check)
@pytest.mark.parametrize("vocab,n", [(151936, 7), (262144, 7), (151936, 15), (700001, 2)])
@pytest.mark.parametrize("dtype", ["bf16", "fp32"])
def test_residuals_below_the_fixed_point_have_their_keys(vocab, n, dtype):
    """A flat row, and a drafter an ulp below it: p - q is less than 2^-40 everywhere. The reference's draw takes the best ln(p - q) + noise all the same (the
    inverse CDF, on floors of 2^-40, draws from the row itself). Then with a few residuals above 2^-40 in one place, and with one positive one at the very end."""
    host = np.zeros((n + 1, vocab), np.float32)
    target = oracle.f32_to_bf16(host) if dtype == "bf16" else host
    p = np.float32(1.0) / np.float32(vocab)
    q = np.full((n, vocab), np.nextafter(p, np.float32(0.0)), np.float32)
    d, ua = np.full(n, 77, np.int32), np.zeros(n, np.float32)
    at = n // 2
    q[:, 77], ua[at] = 2 * p, LAST
    some, last = q.copy(), np.full_like(q, 1.0)
    some[:, 5000:5003] = p - np.float32(2.0**-38)
    last[:, vocab - 1] = np.nextafter(p, np.float32(0.0))
    for x in (q, some, last):
        acc, fin, _ = oracle.verify_gumbel(target, d, x, seed=17, step=5, u_accept=ua)
        assert acc == at and 0 < p - x[at, vocab - 1] < 2.0**-40
        for kept in (None, np.full(n + 1, -1.0, np.float32)):
            check(target, d, x, ua, np.float32(0.3), tau=kept)
    assert fin == vocab - 1


# (a flat row of 700,001: sums of residuals pass 2^64, so that the draw's point lies in two slices or in none)
@pytest.mark.parametrize("residual_draw", ["inverse_cdf", "gumbel"])
@pytest.mark.parametrize("vocab,flat", [(50257, False), (700001, True)])
def test_masses_of_no_row_end_in_outputs(vocab, flat, residual_draw):
    """Masses that are not the rows' give unspecified tokens, but outputs are written, the round is closed once and the launches behind it are right."""
    n = 3
    layout = lm.StepStateLayout(n + 1, n)
    rng, target, _, q = step(vocab, n, "bf16", 23)
    if flat:
        target = np.zeros_like(target)
    z = oracle.bf16_to_f32(target)
    x, gq = on_gpu(target), torch.from_numpy(q).cuda()
    vmax = torch.from_numpy(z.max(-1)).cuda()
    right = torch.tensor([oracle.kept_mass(z[r], -np.inf, 1.0) for r in range(n + 1)], dtype=torch.int64, device="cuda")
    drafts = torch.full((n,), -1, dtype=torch.int32, device="cuda")          # no id of the vocabulary: rejected whatever the masses
    for mass in (1, 3, 1 << 12, 1 << 24, 1 << 36, -1):
        for uf in (0.0, 0.01, 0.3, 0.9, LAST):
            wrong = torch.full((n + 1,), mass, dtype=torch.int64, device="cuda")
            kw = dict(uniforms=torch.full((n,), 0.5).cuda(), u_resample=torch.tensor([uf], dtype=torch.float32), residual_draw=residual_draw, seed=4)
            out = torch.full((n + 3,), -7, dtype=torch.int32, device="cuda")
            lm.verify(x, drafts, gq, mode="stochastic", out=out, target_vmax=vmax, target_mass=wrong, **kw)
            assert int(out[0]) == 0 and -1 <= int(out[1]) < vocab, (mass, uf)
            st = layout.to_device(dict(step=2, verify_len=n, t_this_step=n + 1, pending_tokens=[5, -1, -1, -1]))
            ring = torch.zeros(8, dtype=torch.int64, device="cuda")
            close = lambda **more: lm.verify(x, None, gq, mode="stochastic", out=out, target_vmax=vmax, step_state=(layout, st),   # noqa: E731
                                             commit=dict(layout=layout, state=st, ring=ring), **kw, **more)
            close(target_mass=wrong)
            assert layout.from_device(st)["step"] == 3, (mass, uf)
            out.fill_(-7)
            close(target_mass=right)                                         # no drafts: the row's own draw
            after = layout.from_device(st)
            assert after["step"] == 4 and after["anchor"] == int(out[1]) and int(out[0]) == 0
            if residual_draw == "inverse_cdf":
                assert int(out[1]) == oracle.sample_invcdf_index_order(z[0], uf)


@pytest.mark.parametrize("vocab,n", [(50257, 7), (262144, 7), (700001, 2)])
@pytest.mark.parametrize("dtype", ["bf16", "fp32"])
def test_draft_values_below_zero(vocab, n, dtype):
    """What a drafter gives need not be a distribution: where q < 0 the residual may exceed 1, and the draw is still the definition's."""
    rng, target, _, q = step(vocab, n, dtype, 7)
    z = oracle.bf16_to_f32(target) if dtype == "bf16" else target
    sharp = np.full_like(z, -40.0)                                           # p = 1 at one token
    sharp[:, 1234] = 3.0
    for t, zt in ((target, z), (oracle.f32_to_bf16(sharp) if dtype == "bf16" else sharp, sharp)):
        d, ua = rejecting(zt, q, n // 2)
        tau = np.partition(zt, vocab - 300, axis=-1)[:, vocab - 300].astype(np.float32)
        for least in (-1e-7, -0.3, -3.0, -1000.0):
            x = q.copy()
            x[:, rng.integers(0, vocab, 40)] = np.float32(least) * rng.random(40).astype(np.float32)
            x[:, 1234], x[:, 4321] = np.float32(least), np.float32(least)
            x[np.arange(n), d] = q[np.arange(n), d]
            assert oracle.verify_stochastic(t, d, x, ua, 0.5)[0] == n // 2
            for uf in (0.0, rng.random(), rng.random(), LAST):
                check(t, d, x, ua, np.float32(uf))
            check(t, d, x, ua, np.float32(rng.random()), tau=tau)


@pytest.mark.parametrize("residual_draw", ["inverse_cdf", "gumbel"])
def test_withheld_shares_are_reported_where_masses_are_given(residual_draw):
    """The decisive row's shares: the first block's does not come, the launch reports an error through outputs and state, and the next one is right."""
    vocab, n = 151936, 7
    layout = lm.StepStateLayout(n + 1, n)
    rng, target, _, q = step(vocab, n, "bf16", 3)
    z = oracle.bf16_to_f32(target)
    d, ua = rejecting(z, q, 2)
    given = dict(target_vmax=torch.from_numpy(z.max(-1)).cuda(),
                 target_mass=torch.tensor([oracle.kept_mass(z[r], -np.inf, 1.0) for r in range(n + 1)], dtype=torch.int64, device="cuda"))
    st = layout.to_device(dict(step=2, verify_len=n, t_this_step=n + 1, pending_tokens=[5] + d.tolist(), position=40))
    ring = torch.zeros(16, dtype=torch.int64, device="cuda")
    call = lambda **kw: lm.verify(on_gpu(target), torch.from_numpy(d).cuda(), torch.from_numpy(q).cuda(), torch.from_numpy(ua).cuda(), torch.tensor([0.4]),   # noqa: E731
                                  "stochastic", residual_draw=residual_draw, seed=9, step=4, **given, **kw)
    out = call(commit=dict(layout=layout, state=st, ring=ring), wait_limit=300, selftest=_lib.VERIFY_SELFTEST_WITHHOLD)
    assert int(out[0]) == -1 and out[2].tolist() == [-1] * (n + 1)
    after = layout.from_device(st)
    assert after["error"] == 3 and after["done"] == 1 and int(ring.abs().sum()) == 0
    acc, fin, gap = oracle.verify_gumbel(target, d, q, seed=9, step=4, u_accept=ua) if residual_draw == "gumbel" else (*oracle.verify_stochastic(target, d, q, ua, 0.4)[:2], 1.0)
    out = call()
    assert int(out[0]) == acc == 2 and (int(out[1]) == fin or gap < 1e-5)


# one block, two, as many as there are chunks of 64 for, the line of 120, several turns a block; slices whose last halves lie outside the row
@pytest.mark.parametrize("vocab", [1, 7, 511, 513, 1027, 61439, 61448, 245761, 303105, 700003])
@pytest.mark.parametrize("dtype", ["bf16", "fp32"])
def test_decisive_row_over_all_blocks(vocab, dtype):
    n = 2
    rng, target, _, q = step(vocab, n, dtype, vocab)
    z = oracle.bf16_to_f32(target) if dtype == "bf16" else target
    tau = np.sort(z, axis=-1)[:, -max(1, vocab // 3)].astype(np.float32)
    for at in (0, n - 1):
        for kept in (None, tau):
            d, ua = rejecting(z, q, at, tau=kept)
            for uf in (0.0, rng.random(), LAST):
                check(target, d, q, ua, np.float32(uf), tau=kept)
    check(target, z[:n].argmax(-1).astype(np.int32), q, np.zeros(n, np.float32), np.float32(rng.random()))


@pytest.mark.parametrize("vocab,n", [(16385, 2), (50257, 7), (151936, 15)])
@pytest.mark.parametrize("dtype", ["bf16", "fp32"])
def test_best_keys_of_rows_and_residuals(vocab, n, dtype):
    """The reference's draw where the best key lies far above or below what a slice's weight lets expect: one token with all the weight, a flat row, a row of two
    values, temperatures at both ends, a residual of one element; accepted and rejected rounds, many noises."""
    rng, target, _, q = step(vocab, n, "fp32", 29)
    rows = {"random": target, "flat": np.zeros_like(target), "one": np.where(np.arange(vocab) == vocab // 3, 9.0, -9.0) + np.zeros_like(target),
            "two": np.where(np.arange(vocab) % 2 == 0, 1.0, -30.0) + np.zeros_like(target)}
    for name, zf in rows.items():
        t = oracle.f32_to_bf16(zf.astype(np.float32)) if dtype == "bf16" else zf.astype(np.float32)
        z = oracle.bf16_to_f32(t) if dtype == "bf16" else t
        lone = np.ones_like(q)
        lone[:, vocab - 2] = 0.0
        for T in (0.05, 1.0, 30.0):
            for x, d, u in ((q, z[:n].argmax(-1), np.zeros(n)), (q, np.full(n, -1), np.full(n, LAST)), (lone, np.full(n, 5), np.full(n, LAST))):
                d, u = d.astype(np.int32), u.astype(np.float32)
                for seed in (0, 1, 2):
                    acc, fin, gap = oracle.verify_gumbel(t, d, x, seed=seed, step=seed, temperature=T, u_accept=u)
                    out = lm.verify(on_gpu(t), torch.from_numpy(d).cuda(), torch.from_numpy(x).cuda(), torch.from_numpy(u).cuda(), None, "stochastic", temperature=T,
                                    residual_draw="gumbel", seed=seed, step=seed)
                    assert int(out[0]) == acc and (int(out[1]) == fin or gap < 1e-5 * max(1.0, abs(z).max() / T)), (name, T, seed)


@pytest.mark.parametrize("vocab", [50257, 400001])                           # in one launch, in two
def test_states_without_a_round_are_closed_once(vocab):
    """A prefill chunk is closed once, a finished state left alone, a state whose rows do not fit reported, also where the step takes two launches."""
    n = 2
    layout = lm.StepStateLayout(4, 3)
    x, q = torch.randn(4, vocab, device="cuda").to(torch.bfloat16), torch.full((3, vocab), 1.0 / vocab, device="cuda")
    ring = torch.zeros(8, dtype=torch.int64, device="cuda")

    def after(**fields):
        st = layout.to_device(fields)
        out = torch.full((6,), -7, dtype=torch.int32, device="cuda")
        lm.verify(x, None, q, torch.zeros(3).cuda(), torch.tensor([0.5]), "stochastic", step_state=(layout, st), out=out, commit=dict(layout=layout, state=st, ring=ring))
        return layout.from_device(st), out.tolist()

    got, out = after(step=5, position=40, t_this_step=4, prefill_left=9)
    assert (got["step"], got["position"], got["n_inject"], got["done"]) == (6, 44, 4, 0) and out == [-7] * 6
    got, out = after(step=5, position=40, t_this_step=3, verify_len=n, done=1)
    assert (got["step"], got["position"]) == (5, 40) and out == [-7] * 6
    got, out = after(step=5, position=40, t_this_step=1, verify_len=3)
    assert (got["error"], got["done"], got["step"]) == (4, 1, 5) and out[:2] == [-1, -1]
    assert int(ring.abs().sum()) == 0
    got, out = after(step=5, position=40, t_this_step=3, verify_len=n, pending_tokens=[1, 2, 3])
    assert got["step"] == 6 and got["ring_head"] == got["accepted"] + 1 and got["anchor"] == out[1]
