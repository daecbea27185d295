"""A NaN among the inputs reaches every result that depends on it, and no other."""
from __future__ import annotations

import pytest
import torch

# (dtype, head dim): tensor cores with 64- and 128-key tiles, fp32 operands as pairs, CUDA cores
KINDS = [(torch.bfloat16, 64), (torch.bfloat16, 128), (torch.float16, 96), (torch.float32, 64), (torch.float32, 128)]


@pytest.mark.gpu
@pytest.mark.parametrize("need_o", (False, True))
@pytest.mark.parametrize("causal", (False, True))
@pytest.mark.parametrize("nq,nk", [(130, 200), (40, 6000)])   # the second: keys split over a cluster
@pytest.mark.parametrize("dtype,d", KINDS)
def test_nan_key_reaches_the_logsumexp(dtype, d, nq, nk, causal, need_o):
    import fhob
    heads, first = 17, nk - 100   # head h has its NaN in key first + h: every column of a 16-column group
    g = torch.Generator().manual_seed(7)
    q, k, v = (torch.randn(heads, n, d, generator=g).to("cuda", dtype) for n in (nq, nk, nk))
    clean = fhob.attention_forward(q, k, v, 0.1, is_causal=causal, need_o=need_o)
    bad = k.clone()
    for h in range(heads):
        bad[h, first + h, 3] = float("nan")
    o, lse = fhob.attention_forward(q, bad, v, 0.1, is_causal=causal, need_o=need_o)
    key = torch.arange(heads, device="cuda") + first
    row = torch.arange(nq, device="cuda")
    sees = key[:, None] <= row[None, :] + nk - nq if causal else torch.ones(heads, nq, dtype=torch.bool, device="cuda")
    assert torch.isnan(lse[sees]).all()
    assert torch.equal(lse[~sees], clean[1][~sees])
    if need_o:
        assert torch.isnan(o[sees]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("need_o", (False, True))
@pytest.mark.parametrize("nq,nk", [(130, 200), (40, 6000)])
@pytest.mark.parametrize("dtype,d", KINDS)
def test_nan_query_has_no_logsumexp(dtype, d, nq, nk, need_o):
    """A row whose scores are all NaN has L = NaN, not the -inf of a row without visible keys."""
    import fhob
    g = torch.Generator().manual_seed(8)
    q, k, v = (torch.randn(3, n, d, generator=g).to("cuda", dtype) for n in (nq, nk, nk))
    clean = fhob.attention_forward(q, k, v, 0.1, need_o=need_o)
    q = q.clone()
    q[:, 5] = float("nan")
    o, lse = fhob.attention_forward(q, k, v, 0.1, need_o=need_o)
    keep = torch.arange(nq, device="cuda") != 5
    assert torch.isnan(lse[:, 5]).all() and torch.equal(lse[:, keep], clean[1][:, keep])
    if need_o:
        assert torch.isnan(o[:, 5]).all() and torch.equal(o[:, keep], clean[0][:, keep])
