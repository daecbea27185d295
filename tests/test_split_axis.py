"""Problems with few 128-row tiles: the streamed axis is split over the CTAs of a cluster."""
from __future__ import annotations

import pytest
import torch

from conftest import make_inputs
from oracle import attn_oracle as O


# one item of one tile to many items; parts of unequal length; more parts than one pass has tiles for
SHAPES = [(1, 1, 64), (1, 100, 130), (1, 129, 700), (3, 100, 1000), (1, 1, 4096), (5, 300, 64), (3, 640, 3000), (16, 100, 6000)]
# Passes 3 and 4 in one launch of clusters, one of them split and the other not, with a number of items of
# the other that leaves a cluster with CTAs that have no item (47 key tiles a head in clusters of 8, ...)
PADDED = [(3, 100, 6000), (4, 100, 6000), (2, 640, 6000), (5, 100, 4000), (3, 6000, 100), (4, 4000, 100)]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,d,tol", [(torch.bfloat16, 64, 2e-2), (torch.bfloat16, 128, 2e-2), (torch.float32, 64, 1e-4)])
@pytest.mark.parametrize("bh,nq,nk", SHAPES + PADDED)
def test_split_matches_oracle(bh, nq, nk, dtype, d, tol):
    import fhob
    scale = d ** -0.5
    x = make_inputs(bh, nq, nk, d, seed=nq + nk, dtype=dtype, device="cuda")
    for causal in ((False, True) if nk >= nq else (False,)):
        ref = [t.double().cpu() for t in x.values()]
        o, lse = fhob.attention_forward(x["q"], x["k"], x["v"], scale, is_causal=causal, check=True)
        # the bounds of the other parity tests, relative to each tensor's largest entry
        assert O.rel_err(o.cpu(), O.attn_fwd(*ref[:3], scale, causal)) < tol
        got = fhob.flash_bwdbwd(x["q"], x["k"], x["v"], o, x["do"], x["ddq"], x["ddk"], x["ddv"], lse, scale,
                                is_causal=causal, check=True)
        for n, g, r in zip(("dq2", "dk2", "dv2", "ddo"), got, O.bwdbwd_closed_form(*ref, scale, causal)):
            assert O.rel_err(g.cpu(), r) < tol, (n, causal)
        again = fhob.flash_bwdbwd(x["q"], x["k"], x["v"], o, x["do"], x["ddq"], x["ddk"], x["ddv"], lse, scale,
                                  is_causal=causal)
        assert all(torch.equal(a, b) for a, b in zip(got, again))     # parts are added in a fixed order
        grads = fhob.attention_backward(x["q"], x["k"], x["v"], o, x["do"], lse, scale, is_causal=causal)
        for n, g, r in zip(("dq", "dk", "dv"), grads, O.attn_bwd(ref[0], ref[1], ref[2], ref[3], scale, causal)):
            assert O.rel_err(g.cpu(), r) < tol, (n, causal)
