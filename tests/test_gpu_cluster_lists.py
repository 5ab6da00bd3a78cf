"""The ordered list of a crossing bin in the cluster kernel: lists on both sides of the length from which bins order them, of few and of many distinct values, near
zero (where neighbouring BF16 values share a bin of the list) and far from it, with and without what forbids the short cut (penalties, the draw by inverse CDF)."""
import numpy as np
import pytest
import torch

import oracle
from tests.test_gpu_cluster import _check, _tensor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("centre", [0.0, 0.03, 2.5, -2.5, -0.02, 30.0, -300.0])
@pytest.mark.parametrize("dtype,draw,penalised", [("bf16", "gumbel", False), ("bf16", "gumbel", True), ("bf16", "inverse_cdf", False), ("f32", "gumbel", False)])
def test_lists_of_every_kind(centre, dtype, draw, penalised):
    rng = np.random.default_rng(int(abs(centre) * 100) + 7)
    vocab = 40013
    # a few hundred to two thousand logits around the centre, so near one another that they share a bin; the rest below, a few above
    z = (centre - 4.0 - np.abs(rng.standard_normal((8, vocab)))).astype(np.float32)
    for r, n in enumerate((60, 109, 110, 111, 160, 512, 1200, 2000)):
        at = rng.permutation(vocab)[:n + 4]
        z[r, at[:n]] = centre + rng.uniform(-1e-3, 1e-3, n) * (1.0 if r % 2 else abs(centre) + 1.0)
        z[r, at[n:]] = centre + rng.uniform(0.5, 6.0, 4)
    host = oracle.f32_to_bf16(z) if dtype == "bf16" else z
    hist = rng.integers(0, vocab, (8, 400)).astype(np.int32) if penalised else None
    for top_p in (0.2, 0.6, 0.9):
        _check(_tensor(host), host, dict(temperature=0.9, top_k=0, top_p=top_p, min_p=0.0), draw=draw, history=hist, rho=1.05, pi=0.01)


@pytest.mark.parametrize("draw,near_zero,penalised", [("inverse_cdf", False, False), ("gumbel", True, False), ("gumbel", False, True), ("inverse_cdf", False, True)])
def test_lists_of_few_values_on_both_sides_of_their_line(draw, near_zero, penalised):
    """BF16 lists that bins alone do not put in order: of a few distinct values for the inverse CDF, around zero, and with penalties."""
    rng = np.random.default_rng(17)
    vocab, centre = 30011, 0.0 if near_zero else 1.75
    z = (centre - 4.0 - np.abs(rng.standard_normal((8, vocab)))).astype(np.float32)
    for r, n in enumerate((111, 254, 255, 256, 257, 300, 321, 700)):
        at = rng.permutation(vocab)[:n + 3]
        z[r, at[:n]] = rng.choice([-4e-3, -1e-5, 0.0, 2e-5, 3e-3] if near_zero else [1.75, 1.7578125, 1.765625], n)
        z[r, at[n:]] = centre + rng.uniform(0.5, 4.0, 3)
    host = oracle.f32_to_bf16(z)
    hist = rng.integers(0, vocab, (8, 600)).astype(np.int32) if penalised else None
    for top_p in (0.3, 0.7, 0.95):
        _check(_tensor(host), host, dict(temperature=0.9, top_k=0, top_p=top_p, min_p=0.0), draw=draw, history=hist, rho=1.05, pi=0.01)
