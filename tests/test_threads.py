"""Host threads that share a stream (torch's default stream, unless they choose another) share its workspace."""
from __future__ import annotations

import threading

import pytest
import torch

from conftest import make_inputs


def _in_threads(jobs, rounds):
    """Runs every job `rounds` times in a thread of its own; the threads start together.  Returns the results."""
    gate, got, errors = threading.Barrier(len(jobs)), [[] for _ in jobs], []

    def work(i):
        try:
            gate.wait(30)
            for _ in range(rounds):
                got[i].append(jobs[i]())
        except Exception as e:   # shown by the assert below
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors and not any(t.is_alive() for t in threads)
    return got


@pytest.mark.gpu
@pytest.mark.parametrize("caller", ("native", "ctypes"))
@pytest.mark.parametrize("dtype,d", [(torch.bfloat16, 64), (torch.float32, 64), (torch.float32, 96)])
def test_threads_on_one_stream_get_their_own_results(dtype, d, caller):
    import fhob
    jobs, ref = [], []
    for seed, n in ((1, 200), (2, 330), (3, 200)):
        x = make_inputs(2, n, n, d, seed=seed, dtype=dtype, device="cuda")
        o, lse = fhob.attention_forward(x["q"], x["k"], x["v"], 0.1, is_causal=True)

        def job(x=x, o=o, lse=lse):
            q, k, v, do = x["q"], x["k"], x["v"], x["do"]
            out = tuple(torch.empty_like(t) for t in (q, k, v, do)) if caller == "ctypes" else None
            first = fhob.attention_backward(q, k, v, o, do, lse, 0.1, is_causal=True)
            second = fhob.flash_bwdbwd(q, k, v, o, do, x["ddq"], x["ddk"], x["ddv"], lse, 0.1, is_causal=True, out=out)
            return (*fhob.attention_forward(q, k, v, 0.1, is_causal=True), *first, *second)

        jobs.append(job)
        ref.append(job())
    torch.cuda.synchronize()
    got = _in_threads(jobs, 60)
    torch.cuda.synchronize()
    for r, results in zip(ref, got):
        for g in results:
            assert all(torch.equal(a, b) for a, b in zip(g, r))


@pytest.mark.gpu
def test_threads_with_host_tensors_get_their_own_results():
    """Calls of one shape stage through the same device buffers."""
    import fhob
    jobs, ref = [], []
    for seed in (1, 2, 3):
        x = make_inputs(8, 256, 256, 64, seed=seed, dtype=torch.bfloat16, device="cuda")
        o, lse = fhob.attention_forward(x["q"], x["k"], x["v"], 0.1)
        args = [t.cpu().pin_memory() for t in (x["q"], x["k"], x["v"], o, x["do"], x["ddq"], x["ddk"], x["ddv"], lse)]
        jobs.append(lambda args=args: fhob.flash_bwdbwd(*args, 0.1))
        ref.append(jobs[-1]())
    for r, results in zip(ref, _in_threads(jobs, 20)):
        for g in results:
            assert all(torch.equal(a, b) for a, b in zip(g, r))
