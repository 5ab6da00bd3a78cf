"""The native call path of the Python layer (csrc/host_ext.cpp): what it does beside filling argument structures."""
import ctypes as C
import os
import subprocess
import tempfile
import threading

import pytest
import torch

import lithos_metal_b200 as lm
from lithos_metal_b200 import _lib, sampler
from lithos_metal_b200.verify import DraftQ

pytestmark = pytest.mark.gpu
NAMES = ("lm_sample", "lm_argmax", "lm_argmax_i64", "lm_verify", "lm_draft_q", "lm_head", "lm_workspace_bytes", "lm_verify_workspace_bytes")

# stands in for every entry point: waits (two seconds at most) until another thread has set the flag
FAKE = "#include <unistd.h>\nvolatile int flag, calls;\nint entry(void){calls++;for(int i=0;i<2000&&!flag;i++)usleep(1000);return flag?0:-1;}\n"


def _init(addresses):
    _lib.host().init(addresses, sampler.SamplingParams, sampler.SampleOutput, DraftQ, _lib.check, sampler._workspace)


def _calls():
    x = torch.zeros(2, 64, dtype=torch.bfloat16, device="cuda")
    w = torch.zeros(64, 128, dtype=torch.bfloat16, device="cuda")
    ids = torch.zeros(1, dtype=torch.int32, device="cuda")
    return [lambda: lm.sample(x, temperature=0.8), lambda: lm.argmax(x), lambda: lm.GreedySampler().forward(x), lambda: lm.StochasticSampler().forward(x),
            lambda: lm.draft_q(x, temperature=0.8), lambda: lm.verify(x, ids), lambda: lm.lm_head(torch.zeros(1, 128, dtype=torch.bfloat16, device="cuda"), w)]


def test_other_python_threads_run_while_a_call_waits():
    """A launch can wait for the GPU; ctypes calls let other threads run meanwhile, and so do these."""
    L, real = _lib.lib(), {}
    for n in NAMES:
        real[n] = C.cast(getattr(L, n), C.c_void_p).value
    calls = _calls()
    with tempfile.TemporaryDirectory() as d:
        open(os.path.join(d, "f.c"), "w").write(FAKE)
        subprocess.run(["gcc", "-shared", "-fPIC", "-o", os.path.join(d, "f.so"), os.path.join(d, "f.c")], check=True)
        fake = C.CDLL(os.path.join(d, "f.so"))
        flag, entered = C.c_int.in_dll(fake, "flag"), C.c_int.in_dll(fake, "calls")
        entry = C.cast(fake.entry, C.c_void_p).value
        for f in calls:
            f()                                                             # (workspaces are there)
        try:
            _init({n: real[n] if n.endswith("bytes") else entry for n in NAMES})
            for f in calls:
                flag.value = entered.value = 0

                def release():
                    while not entered.value:
                        pass
                    flag.value = 1

                t = threading.Thread(target=release, daemon=True)
                t.start()
                f()                                                         # raises if the flag was never set
                t.join()
        finally:
            _init(real)


def test_threads_that_share_a_stream_take_turns_with_its_workspace():
    """A batch is several launches that pass rows on in the stream's workspace: calls of two threads on one stream must not interleave."""
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    work = []
    for rows in (160, 800):
        x = (torch.randn(rows, 32768, generator=g, device="cuda") * 2).to(torch.bfloat16)
        k = torch.tensor([0, 20, 50, 1000], dtype=torch.int32, device="cuda")[torch.arange(rows, device="cuda") % 4]
        p = lm.SamplingParams(temperature=0.8, top_k=k, top_p=0.9, seed=6)
        work.append((x, p, lm.sample(x, p).tokens))
    torch.cuda.synchronize()
    wrong = []

    def run(x, p, want):
        got = [lm.sample(x, p).tokens for _ in range(200)]
        torch.cuda.synchronize()
        wrong.extend(int((t != want).sum()) for t in got if not torch.equal(t, want))

    threads = [threading.Thread(target=run, args=w) for w in work for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_calls_give_the_same_with_and_without_the_native_path(monkeypatch):
    """What host_ext.cpp takes, what it leaves to Python (other types, layouts and knobs) and what both refuse."""
    g = torch.Generator(device="cuda")
    g.manual_seed(8)
    x = (torch.randn(8, 40000, generator=g, device="cuda") * 2).to(torch.bfloat16)
    hist = torch.randint(0, 40000, (8, 100), generator=g, device="cuda")
    u = torch.rand(8, generator=g, device="cuda")
    w = torch.randn(1000, 128, generator=g, device="cuda").to(torch.bfloat16)
    h = torch.randn(8, 128, generator=g, device="cuda").to(torch.bfloat16)
    ids = torch.randint(0, 40000, (7,), generator=g, device="cuda")
    q = torch.softmax(x[:7].float(), -1)
    K = torch.arange(8, device="cuda")

    def flat(r):
        r = list(vars(r).values()) if isinstance(r, lm.SampleOutput) else list(r) if isinstance(r, tuple) else [r]
        return [t for t in r if isinstance(t, torch.Tensor)]

    def out_of(call):
        try:
            return [t.clone() for t in flat(call())]
        except (ValueError, TypeError, RuntimeError) as e:
            return type(e), str(e)

    everything = dict(return_tau=True, return_stats=True, return_probs=True, return_status=True, return_vmax=True)
    draft = lm.draft_q(x[:7], temperature=0.9, seed=4)
    calls = [
        lambda: lm.sample(x, temperature=0.8, top_k=20, top_p=0.9, seed=2, step=3, row_offset=5, **everything),
        lambda: lm.sample(x, temperature=1, top_k=20.0, seed=-1, step=-1, **everything),                            # knobs of other types, masked to 64 and 32 bits
        lambda: lm.sample(x, temperature=u + 0.3, top_k=K, top_p=u.double(), min_p=0.01, seed=1 << 70, **everything),   # per-row knobs that need a conversion
        lambda: lm.sample(x, temperature=u + 0.3, top_k=K.int(), top_p=u, history=hist, repetition_penalty=1.2, draw="inverse_cdf", uniforms=u, **everything),
        lambda: lm.sample(x, temperature=0.8, history=hist.int(), presence_penalty=0.5, draw="inverse_cdf", uniforms=u.cpu(), **everything),
        lambda: lm.sample(x[:, ::2], temperature=0.8, top_p=0.9, **everything),                                     # a stride along the vocabulary
        lambda: lm.sample(x[2:3].expand(4, -1), temperature=0.8),                                                   # refused: rows on top of one another
        lambda: lm.sample(x[3:4, 5:999], temperature=0.8, top_p=0.9, **everything),
        lambda: lm.sample(x[:0], temperature=0.8, **everything),
        lambda: lm.sample(x, temperature=0.8, out=torch.empty(8, dtype=torch.int32, device="cuda")),
        lambda: lm.sample(x, temperature=0.8, out=torch.empty(7, dtype=torch.int32, device="cuda")),
        lambda: lm.sample(x, temperature=float("nan")), lambda: lm.sample(x, temperature=-0.5), lambda: lm.sample(x.half(), temperature=1.0), lambda: lm.sample(x.cpu(), temperature=1.0),
        lambda: lm.sample(x, temperature=0.8, draw="other"), lambda: lm.sample(x, temperature=0.8, draw="inverse_cdf"), lambda: lm.sample(x, temperature=0.8, top_k=K[:3]),
        lambda: lm.sample(x, temperature=0.8, repetition_penalty=0.0), lambda: lm.sample(x, temperature=0.8, history=hist[:3]), lambda: lm.sample(x[0], temperature=0.8),
        lambda: lm.argmax(x), lambda: lm.argmax(x.float()), lambda: lm.argmax(x.t()), lambda: lm.argmax(x, out=torch.empty(8, dtype=torch.int32, device="cuda")), lambda: lm.argmax(x[0]),
        lambda: lm.GreedySampler().forward(x), lambda: lm.StochasticSampler(0.7, 20, 0.9, seed=3).forward(x, 4), lambda: lm.StochasticSampler(0.7, 20, 0.9).forward(x.float()[:, ::2]),
        lambda: lm.draft_q(x[:7], temperature=0.9, seed=4, step=2, first_position=3), lambda: lm.draft_q(x[:7], temperature=0.9, copy_logits=True), lambda: lm.draft_q(x, temperature=0.0),
        lambda: lm.draft_q(torch.cat([x] * 3), temperature=0.5),
        lambda: lm.verify(x, ids), lambda: lm.verify(x, ids.int(), q, u[:7], u[:1], "stochastic", temperature=0.9, return_p_draft=True),
        lambda: lm.verify(x, ids, None, u[:7].cpu(), 0.3 * u[:1], "stochastic", temperature=0.9, draft_logits=x[:7], draft_stats=draft, seed=3, step=1, residual_draw="gumbel"),
        lambda: lm.verify(x, ids, None, None, None, "stochastic"), lambda: lm.verify(x, ids[:3]), lambda: lm.verify(x, ids, q[:3], mode="stochastic"), lambda: lm.verify(x, ids, mode="other"),
        lambda: lm.lm_head(h, w), lambda: lm.lm_head(h, w, h[0], eps=1, one_plus=False), lambda: lm.lm_head(h, w[:, :64]), lambda: lm.lm_head(torch.cat([h, h]), w), lambda: lm.lm_head(h.float(), w),
    ]
    native = [out_of(c) for c in calls]
    monkeypatch.setattr(_lib, "_host", _lib._NoHost())
    for i, (a, c) in enumerate(zip(native, calls)):
        b = out_of(c)
        if isinstance(a, tuple):
            assert a == b, i
        else:
            assert isinstance(b, list) and len(a) == len(b), (i, b)
            assert all(s.dtype == t.dtype and s.shape == t.shape and torch.equal(s, t) for s, t in zip(a, b)), i


def test_a_subclass_of_the_stochastic_sampler_forms_its_own_knobs():
    class Annealed(lm.StochasticSampler):
        def params(self):
            p = super().params()
            p.top_k = 1
            return p

    g = torch.Generator(device="cuda").manual_seed(3)                        # (rows whose largest logit is one: a top_k of 1 keeps equal ones)
    x = (torch.randn(4, 4096, generator=g, device="cuda") * 2).to(torch.bfloat16)
    top = x.float().topk(2).values
    assert bool((top[:, 0] > top[:, 1]).all())
    assert torch.equal(Annealed(temperature=2.0, seed=5).forward(x), x.float().argmax(-1))
