"""CUDA-core operator and first backward at the edges of their 64 x 32 tiles and 64-column halves."""
from __future__ import annotations

import math

import pytest
import torch

from oracle import attn_oracle as O

# n_q, n_k, d, d_v, causal, window
EDGES = [(1, 1, 4, 4, False, None), (64, 32, 64, 68, False, None), (65, 33, 68, 64, False, None), (63, 31, 128, 4, False, None),
         (64, 128, 60, 128, True, None), (97, 161, 124, 128, True, None), (130, 130, 128, 128, True, 33), (96, 200, 72, 80, True, 64),
         (64, 1500, 128, 128, False, None), (700, 40, 96, 96, False, None)]


@pytest.mark.gpu
@pytest.mark.parametrize("bh", (1, 3))
@pytest.mark.parametrize("nq,nk,d,dv,causal,window", EDGES)
def test_edges_match_oracle(bh, nq, nk, d, dv, causal, window):
    import fhob
    g = torch.Generator().manual_seed(nq * 7 + nk)
    mk = lambda n, e: torch.randn(bh, n, e, generator=g)
    x = dict(q=mk(nq, d), k=mk(nk, d), v=mk(nk, dv), do=mk(nq, dv), ddq=mk(nq, d), ddk=mk(nk, d), ddv=mk(nk, dv))
    x64 = {n: t.double() for n, t in x.items()}
    w = math.inf if window is None else window
    scale = d ** -0.5
    ref2 = O.bwdbwd_closed_form(*x64.values(), scale, causal, sliding_window_length=w)
    ref1 = O.attn_bwd(x64["q"], x64["k"], x64["v"], x64["do"], scale, causal, sliding_window_length=w)
    dev = {n: t.cuda() for n, t in x.items()}
    kw = dict(is_causal=causal, sliding_window=window, impl="simt")
    o, lse = fhob.attention_forward(dev["q"], dev["k"], dev["v"], scale, **kw)
    args = (dev["q"], dev["k"], dev["v"], o, dev["do"], dev["ddq"], dev["ddk"], dev["ddv"], lse, scale)
    got2 = fhob.flash_bwdbwd(*args, **kw)
    got1 = fhob.attention_backward(*args[:5], lse, scale, **kw)
    # chains of n + 2 d fp32 multiply-adds, 2^-24 each, as a random walk: sqrt(1756) * 2^-24 = 2.5e-6 of a
    # typical entry; the differences dP - D and X + k23 lose at most three bits of that (1 key: exact zeros)
    for n, a, r in zip(("dq", "dk", "dv", "dq2", "dk2", "dv2", "ddo"), got1 + got2, tuple(ref1) + tuple(ref2)):
        err = float((a.double().cpu() - r).abs().max()) / max(float(r.abs().max()), 0.1)
        assert err < 2e-5, (n, err)
    again = fhob.flash_bwdbwd(*args, **kw)
    assert all(torch.equal(a, b) for a, b in zip(got2, again))   # one order of sums


@pytest.mark.gpu
def test_single_passes_give_the_operator():
    """The four passes one by one, over the same workspace, leave the results of the whole operator."""
    import ctypes as C
    import fhob
    from fhob import _lib
    lib = _lib.load()
    bh, nq, nk, d = 2, 70, 100, 96
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v, do, ddq, ddk, ddv = (torch.randn(bh, n, d, generator=g, device="cuda") for n in (nq, nk, nk, nq, nq, nk, nk))
    o, lse = fhob.attention_forward(q, k, v, 0.1)
    ref = fhob.flash_bwdbwd(q, k, v, o, do, ddq, ddk, ddv, lse, 0.1)
    out = [torch.full_like(t, float("nan")) for t in (q, k, v, do)]
    p = _lib.FhobProblem()
    p.bh, p.n_q, p.n_k, p.d, p.dtype, p.scale = bh, nq, nk, d, _lib.FHOB_F32, 0.1
    for n, t in zip(("q", "k", "v", "o", "d_o", "lse", "ddq", "ddk", "ddv", "dq2", "dk2", "dv2", "ddo"),
                    (q, k, v, o, do, lse, ddq, ddk, ddv, *out)):
        setattr(p, n, t.data_ptr())
    ws = torch.zeros(lib.fhob_workspace_bytes(bh, nq), dtype=torch.uint8, device="cuda")
    p.workspace, p.workspace_bytes = ws.data_ptr(), ws.numel()
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for f in (lib.fhob_prepass, lib.fhob_pass1, lib.fhob_pass2, lib.fhob_pass3, lib.fhob_pass4):
        assert f(C.byref(p), s) == 0
    for a, b in zip(out, ref):   # the same partial sums, whatever shares a launch
        assert torch.equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("bh,nq,nk,d,dv,causal,window",
                         [(1, 1, 1, 4, 128, False, None), (2, 64, 128, 128, 64, False, None), (3, 65, 129, 96, 4, True, None),
                          (1, 200, 127, 128, 128, True, None), (2, 130, 300, 68, 72, True, 40), (1, 64, 4000, 128, 128, False, None),
                          (5, 70, 3000, 128, 96, True, 900), (1, 33, 70, 5, 7, False, None), (2, 100, 600, 127, 2, True, None)])
def test_forward_matches_oracle(bh, nq, nk, d, dv, causal, window):
    """The forward at the edges of its 64 x 128 tiles, split keys, dead rows, and rows that are not whole 16-byte pieces (C ABI)."""
    import ctypes as C
    from fhob import _lib
    lib = _lib.load()
    g = torch.Generator().manual_seed(nq + nk)
    q, k, v = torch.randn(bh, nq, d, generator=g), torch.randn(bh, nk, d, generator=g), torch.randn(bh, nk, dv, generator=g)
    w = math.inf if window is None else window
    scale = d ** -0.5
    dead = max(0, nq - nk) if causal else 0
    dev = [t.cuda() for t in (q, k, v)]
    p = _lib.FhobProblem()
    p.bh, p.n_q, p.n_k, p.d, p.d_v, p.dtype, p.scale = bh, nq, nk, d, dv, _lib.FHOB_F32, scale
    p.causal, p.window, p.impl = int(causal), window or 0, _lib.IMPL["simt"]
    p.q, p.k, p.v = (t.data_ptr() for t in dev)
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for need_o in (True, False):
        o = torch.full((bh, nq, dv), float("nan"), device="cuda")
        lse = torch.full((bh, nq), float("nan"), device="cuda")
        assert lib.fhob_forward(C.byref(p), C.c_void_p(o.data_ptr() if need_o else None), C.c_void_p(lse.data_ptr()), stream) == 0
        ql = q[:, dead:].double()
        ref_l = O.attn_lse(ql, k.double(), scale, causal, w)
        # sums of up to 4000 + 128 terms with 2^-24 each as a random walk (4e-6), doubled for the exponent of 2
        assert float((lse[:, dead:].double().cpu() - ref_l).abs().max()) < 1e-5
        assert (lse[:, :dead] == -math.inf).all()
        if need_o:
            assert O.rel_err(o[:, dead:], O.attn_fwd(ql, k.double(), v.double(), scale, causal, w)) < 1e-5
            assert (o[:, :dead] == 0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("impl,dtype,d", [("auto", "fp32", 128), ("simt", "bf16", 64), ("auto", "bf16", 64), ("auto", "fp32", 64)])
def test_forward_clears_the_status_word(impl, dtype, d):
    """Whatever the workspace held before the call; both families of kernels."""
    import ctypes as C
    from fhob import _lib
    lib = _lib.load()
    t = {"fp32": torch.float32, "bf16": torch.bfloat16}[dtype]
    q, k, v, o = (torch.randn(2, n, d, device="cuda").to(t) for n in (70, 90, 90, 70))
    lse = torch.empty(2, 70, device="cuda")
    p = _lib.FhobProblem()
    p.bh, p.n_q, p.n_k, p.d, p.scale, p.impl = 2, 70, 90, d, 0.1, _lib.IMPL[impl]
    p.dtype = {"fp32": _lib.FHOB_F32, "bf16": _lib.FHOB_BF16}[dtype]
    p.q, p.k, p.v = q.data_ptr(), k.data_ptr(), v.data_ptr()
    ws = torch.full((lib.fhob_workspace_bytes_problem(C.byref(p)),), 255, dtype=torch.uint8, device="cuda")
    p.workspace, p.workspace_bytes = ws.data_ptr(), ws.numel()
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.fhob_forward(C.byref(p), C.c_void_p(o.data_ptr()), C.c_void_p(lse.data_ptr()), s) == 0
    assert lib.fhob_read_status(C.byref(p), s) == 0
    ws.fill_(255)   # the CUDA-core kernels never needed a workspace that would do for the others
    if impl == "simt":
        p.workspace = ws.data_ptr() + 8
        assert lib.fhob_forward(C.byref(p), C.c_void_p(o.data_ptr()), C.c_void_p(lse.data_ptr()), s) == 0
        assert (ws == 255).all()
