"""A kernel starts while the one in front drains: what it reads must still be what that one wrote."""
from __future__ import annotations

import pytest
import torch

from conftest import make_inputs


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,d", [(torch.bfloat16, 64), (torch.bfloat16, 128), (torch.float32, 64), (torch.float32, 128)])
def test_backward_reads_the_forward_in_front_of_it(dtype, d):
    """O and L are written over on every turn, directly before the first backward's pre-pass reads them."""
    import ctypes as C
    import fhob
    from fhob import _lib
    lib = _lib.load()
    bh, n = 3, 700
    x = make_inputs(bh, n, n, d, seed=5, dtype=dtype, device="cuda")
    o, lse = torch.empty_like(x["q"]), torch.empty(bh, n, device="cuda")
    grads = [torch.empty_like(x["q"]) for _ in range(3)]
    p = _lib.FhobProblem()
    p.bh, p.n_q, p.n_k, p.d, p.dtype, p.scale = bh, n, n, d, _lib.DTYPES[str(dtype)], 0.1
    p.k, p.v, p.o, p.d_o, p.lse = (t.data_ptr() for t in (x["k"], x["v"], o, x["do"], lse))
    ws = torch.zeros(lib.fhob_workspace_bytes_problem(C.byref(p)), dtype=torch.uint8, device="cuda")
    p.workspace, p.workspace_bytes = ws.data_ptr(), ws.numel()
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    queries = [x["q"], x["ddq"], x["do"]]   # three sets of queries in turn

    def turn(q, wait):
        p.q = q.data_ptr()
        assert lib.fhob_forward(C.byref(p), C.c_void_p(o.data_ptr()), C.c_void_p(lse.data_ptr()), s) == 0
        if wait:
            torch.cuda.synchronize()
        assert lib.fhob_backward(C.byref(p), *(C.c_void_p(g.data_ptr()) for g in grads), s) == 0
        return [g.clone() for g in grads]

    ref = [turn(q, True) for q in queries]
    got = [[turn(q, False) for q in queries] for _ in range(20)]
    for results in got:
        for r, g in zip(ref, results):
            assert all(torch.equal(a, b) for a, b in zip(r, g))
