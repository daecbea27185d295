"""The native host path of the Python package against the Python path it stands in front of."""
from __future__ import annotations

import pytest
import torch

from conftest import make_inputs


def _args(dtype, view, batch=2, heads=3, nq=70, nk=129, d=64):
    """Operator arguments as (B, H, N, D) tensors, contiguous or views of (B, N, H, D) projections."""
    import fhob
    x = make_inputs(batch * heads, nq, nk, d, seed=5, dtype=dtype, device="cuda")
    if view:
        x = {n: t.view(batch, heads, t.shape[1], d).transpose(1, 2).contiguous().transpose(1, 2) for n, t in x.items()}
    else:
        x = {n: t.view(batch, heads, t.shape[1], d) for n, t in x.items()}
    o, lse = fhob.attention_forward(x["q"], x["k"], x["v"], d ** -0.5)
    return [x["q"], x["k"], x["v"], o, x["do"], x["ddq"], x["ddk"], x["ddv"], lse, d ** -0.5]


@pytest.mark.gpu
@pytest.mark.parametrize("view", (False, True))
@pytest.mark.parametrize("dtype", (torch.bfloat16, torch.float32))
def test_native_call_matches_python_call(dtype, view):
    import fhob
    args = _args(dtype, view)
    native = fhob.ops._native()
    got = native.bwdbwd(*args, False, None, "auto")
    assert got is not None
    # caller-given results and workspace take the Python path: the same kernels, so the same bits
    out = tuple(torch.empty(t.shape, dtype=dtype, device="cuda") for t in (args[0], args[1], args[2], args[4]))
    fhob.flash_bwdbwd(*args, out=out, check=True)
    for g, r, like in zip(got, out, (args[0], args[1], args[2], args[4])):
        assert g.shape == like.shape and g.is_contiguous() and torch.equal(g, r)
    assert native.backward(*args[:5], *args[8:], False, None, "auto") is not None


@pytest.mark.gpu
def test_calls_the_native_path_leaves_to_python():
    import fhob
    args = _args(torch.bfloat16, False)
    native = fhob.ops._native()
    ref = fhob.flash_bwdbwd(*args, check=True)
    odd = {
        "16-bit logsumexp": args[:8] + [args[8].bfloat16(), args[9]],
        "expanded rows": args[:4] + [args[4][:, :, :1].expand_as(args[4])] + args[5:],
        "host tensors": [t.cpu() if isinstance(t, torch.Tensor) else t for t in args],
    }
    for name, a in odd.items():
        assert native.bwdbwd(*a, False, None, "auto") is None, name
        assert all(torch.isfinite(t.float()).all() for t in fhob.flash_bwdbwd(*a)), name
    for g, r in zip(fhob.flash_bwdbwd(*odd["host tensors"]), ref):
        assert torch.equal(g.cuda(), r)
    assert native.bwdbwd(*args, False, 4, "auto") is None            # a window without a causal mask
    with pytest.raises(ValueError):
        fhob.flash_bwdbwd(*args, sliding_window=4)
    with pytest.raises(TypeError):
        fhob.flash_bwdbwd(*([args[0].float()] + args[1:]))
