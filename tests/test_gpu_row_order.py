"""The order in which the candidate kernel's blocks take the rows of a batch with a top_k per row: every row is taken once, whatever the top_k are."""
import numpy as np
import pytest
import torch

import lithos_metal_b200 as lm
from tests import routes

pytestmark = pytest.mark.gpu

PATTERNS = {"short": [20], "long": [500], "mixed": [0, 64, 65, 1000], "one long": [20] * 60 + [1000], "few of this kernel's": [0] * 30 + [50]}


# rows on both sides of the batches that go to clusters, of one and of two rows a block, and of the batches whose rows come unordered
@pytest.mark.parametrize("rows", [75, 148, 149, 297, 500, 740, 741])
@pytest.mark.parametrize("pattern", PATTERNS)
def test_every_row_is_taken_once(rows, pattern):
    vocab = 40960
    g = torch.Generator(device="cuda"); g.manual_seed(rows)
    x = (torch.randn(rows, vocab, generator=g, device="cuda") * 2).to(torch.bfloat16)
    k = torch.tensor(np.resize(np.array(PATTERNS[pattern], np.int32), rows), device="cuda")
    knobs = dict(temperature=torch.rand(rows, generator=g, device="cuda") + 0.4, top_k=k, top_p=0.9, draw="inverse_cdf")
    u = torch.rand(rows, generator=g, device="cuda")
    call = lambda **kw: lm.sample(x, lm.SamplingParams(**knobs, **kw), uniforms=u, return_tau=True, return_status=True)   # noqa: E731
    r, exact = call(), call(exact_only=True)
    assert "sample_topk_kernel" in routes.names(call)
    assert torch.equal(r.tokens, exact.tokens) and torch.equal(r.tau, exact.tau)
    assert int(((r.status & 64) != 0).sum()) >= 0.9 * int((k > 0).sum())     # (by the candidate kernel, but for the rows that it hands on)


@pytest.mark.parametrize("rows,ordered", [(75, False), (148, False), (1, True), (0, False)])
def test_rows_are_ordered_where_some_wait_for_a_block(rows, ordered):
    """Up to 1.6 rows per SM every row of the candidate kernel has a block at once, and the kernel that looks the order up is not launched."""
    line = 8 * torch.cuda.get_device_properties(0).multi_processor_count // 5
    rows = rows if rows > 1 else line + rows
    x = torch.randn(rows, 40960, device="cuda").to(torch.bfloat16)
    k = torch.tensor([0, 20, 50, 1000] * rows, dtype=torch.int32, device="cuda")[:rows]
    found = [name for name, _, _ in routes.kernels(lambda: lm.sample(x, lm.SamplingParams(temperature=0.8, top_k=k, top_p=0.9)), full=True)[0] if "sample_topk_kernel" in name]
    assert found and all(("Lb1" in name) == ordered for name in found), found
