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
