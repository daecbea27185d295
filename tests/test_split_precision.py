"""fp32 operands as bf16 pairs: the small terms of a product do not wear away the large one's accumulator."""
from __future__ import annotations

import pytest
import torch

from conftest import make_inputs
from oracle import attn_oracle as O


@pytest.mark.gpu
@pytest.mark.parametrize("causal", (False, True))
def test_long_sums_keep_their_precision(causal):
    """2-norm errors of O, dQ, dK and dV over 4096 rows against those of 256: what a split leaves out (lo.lo, and the
    rounding of lo) does not grow with the length.  What grows is the low bits that the tensor core cuts off with
    each addition to an accumulator, 2^-24 of it on average.  There are n / 16 of them a row for hi.hi, and a sum of
    random signs has on average 2/3 of its final size: 2/3 * 256 * 2^-24 = 1.0e-5 at most, if all errors point the
    same way.  Three terms in one accumulator make it up to three times as much (measured: 1.1e-5 to 1.9e-5)."""
    import fhob

    def errors(n):
        x = make_inputs(2, n, n, 64, seed=n, dtype=torch.float32, device="cuda")
        # fp32 values that bf16 does not hold
        g = torch.Generator(device="cuda").manual_seed(n)
        q, k, v, do = (x[m] + 1e-3 * torch.randn(x[m].shape, generator=g, device="cuda") for m in ("q", "k", "v", "do"))
        o, lse = fhob.attention_forward(q, k, v, 0.125, is_causal=causal)
        got = (o, *fhob.attention_backward(q, k, v, o, do, lse, 0.125, is_causal=causal))
        r = [t.double() for t in (q, k, v, do)]
        ref = (O.attn_fwd(*r[:3], 0.125, causal), *O.attn_bwd(*r, 0.125, causal))
        return [float((a.double() - b.cuda()).norm() / b.cuda().norm()) for a, b in zip(got, ref)]

    for name, long, short in zip(("o", "dq", "dk", "dv"), errors(4096), errors(256)):
        assert long < short + 1.0e-5, (name, long, short)
