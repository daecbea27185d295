"""Problems with few 128-row tiles: the streamed axis is split over the CTAs of a cluster."""
from __future__ import annotations

import ctypes as C

import pytest
import torch

from conftest import make_inputs
from oracle import attn_oracle as O


# one item of one tile to many items; parts of unequal length; more parts than one pass has tiles for
SHAPES = [(1, 1, 64), (1, 100, 130), (1, 129, 700), (3, 100, 1000), (1, 1, 4096), (5, 300, 64), (3, 640, 3000), (16, 100, 6000)]
# Passes 3 and 4 in one launch of clusters, one of them split and the other not, with a number of items of
# the other that leaves a cluster with CTAs that have no item (3 x 47 key tiles in clusters of 4, 3 x 17 in clusters of 2, ...)
PADDED = [(3, 100, 6000), (3, 100, 2100), (1, 200, 11000), (3, 6000, 100), (3, 2100, 100), (1, 11000, 200)]


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
        for n, a, b in zip(("dq2", "dk2", "dv2", "ddo"), got, again):     # parts are added in a fixed order
            where = (a != b).nonzero()
            assert len(where) == 0, (n, causal, len(where), where[0].tolist(), where[-1].tolist(), float((a - b).abs().max()))
        grads = fhob.attention_backward(x["q"], x["k"], x["v"], o, x["do"], lse, scale, is_causal=causal)
        for n, g, r in zip(("dq", "dk", "dv"), grads, O.attn_bwd(ref[0], ref[1], ref[2], ref[3], scale, causal)):
            assert O.rel_err(g.cpu(), r) < tol, (n, causal)


# one head and two; a window of a few tiles of a long sequence (not split), one of half of it (two parts)
@pytest.mark.gpu
@pytest.mark.parametrize("dtype,d,tol", [(torch.bfloat16, 64, 2e-2), (torch.bfloat16, 128, 2e-2), (torch.float32, 64, 1e-4), (torch.float32, 96, 1e-4)])
@pytest.mark.parametrize("bh,nq,nk,window", [(1, 100, 6000, 64), (2, 100, 8000, 4000), (1, 3000, 3000, 64)])
def test_split_with_a_window_matches_oracle(bh, nq, nk, window, dtype, d, tol):
    import fhob
    x = make_inputs(bh, nq, nk, d, seed=nq + nk, dtype=dtype, device="cuda")
    ref = [t.double().cpu() for t in x.values()]
    kw = dict(is_causal=True, sliding_window=window)
    o, lse = fhob.attention_forward(x["q"], x["k"], x["v"], 0.1, **kw, check=True)
    assert O.rel_err(o.cpu(), O.attn_fwd(*ref[:3], 0.1, True, window)) < tol
    got = fhob.flash_bwdbwd(x["q"], x["k"], x["v"], o, x["do"], x["ddq"], x["ddk"], x["ddv"], lse, 0.1, **kw, check=True)
    for n, g, r in zip(("dq2", "dk2", "dv2", "ddo"), got, O.bwdbwd_closed_form(*ref, 0.1, True, sliding_window_length=window)):
        assert O.rel_err(g.cpu(), r) < tol, n
    grads = fhob.attention_backward(x["q"], x["k"], x["v"], o, x["do"], lse, 0.1, **kw)
    for n, g, r in zip(("dq", "dk", "dv"), grads, O.attn_bwd(*ref[:4], 0.1, True, window)):
        assert O.rel_err(g.cpu(), r) < tol, n


# one to many tiles a head on either side, with and without parts; windows; both families of kernels
INVARIANT = [(9, 100, 3000, False, None), (9, 2048, 2048, True, None), (8, 1024, 1024, False, None), (7, 300, 300, True, 64),
             (16, 100, 6000, True, 700), (6, 640, 3000, False, None), (12, 64, 1500, True, None), (5, 3000, 100, False, None)]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,d", [(torch.bfloat16, 64), (torch.bfloat16, 128), (torch.float32, 64), (torch.float32, 96)])
@pytest.mark.parametrize("bh,nq,nk,causal,window", INVARIANT)
def test_bits_of_a_head_do_not_depend_on_the_heads_it_is_launched_with(bh, nq, nk, causal, window, dtype, d):
    import fhob
    x = make_inputs(bh, nq, nk, d, seed=nq + nk, dtype=dtype, device="cuda")
    kw = dict(is_causal=causal, sliding_window=window)

    def calls(lo, hi):
        t = {n: v[lo:hi].contiguous() for n, v in x.items()}
        o, lse = fhob.attention_forward(t["q"], t["k"], t["v"], 0.1, **kw)
        alone = fhob.produce_L(t["q"], t["k"], causal, 0.1, window)
        first = fhob.attention_backward(t["q"], t["k"], t["v"], o, t["do"], lse, 0.1, **kw)
        second = fhob.flash_bwdbwd(t["q"], t["k"], t["v"], o, t["do"], t["ddq"], t["ddk"], t["ddv"], lse, 0.1, **kw)
        return (o, lse, alone, *first, *second)

    whole = calls(0, bh)
    for lo, hi in ((0, 1), (bh - 2, bh)):
        for n, a, b in zip(("o", "lse", "L", "dq", "dk", "dv", "dq2", "dk2", "dv2", "ddo"), whole, calls(lo, hi)):
            assert torch.equal(a[lo:hi], b), (n, lo)


def _ctas(family, bh, nq, nk, window=0):
    """What the CTAs of the launch of passes 3 and 4 do: [(pass, item, part, parts)] in grid order."""
    from fhob import _lib
    lib = _lib.load()
    p = _lib.FhobProblem()
    p.bh, p.n_q, p.n_k, p.d, p.causal, p.window = bh, nq, nk, 64, int(window > 0), window
    p.dtype, p.impl = _lib.FHOB_BF16, _lib.IMPL[family]
    out = [C.c_int32() for _ in range(4)]
    ctas = []
    while lib.fhob_cta_work(C.byref(p), len(ctas), *(C.byref(x) for x in out)) == 0:
        ctas.append(tuple(x.value for x in out))
    return ctas


WALK = [(bh, nq, nk) for bh in (1, 2, 3, 5, 7) for nq, nk in
        [(1, 1), (64, 64), (100, 6000), (6000, 100), (640, 6000), (129, 700), (300, 3000), (500, 2000), (3000, 513), (256, 256), (513, 8192)]]


@pytest.mark.parametrize("family,rows", [("tcgen05", 128), ("simt", 64)])
@pytest.mark.parametrize("bh,nq,nk", WALK)
def test_every_part_of_every_tile_has_one_cta(family, rows, bh, nq, nk):
    ctas = _ctas(family, bh, nq, nk)
    parts = {}
    for kind, n in ((3, nq), (4, nk)):
        mine = [c for c in ctas if c[0] == kind]
        split = {c[3] for c in mine}
        assert len(split) == 1
        parts[kind] = split.pop()
        assert sorted((c[1], c[2]) for c in mine) == [(i, s) for i in range(bh * -(-n // rows)) for s in range(parts[kind])]
    cluster = max(parts.values())
    assert cluster <= 8 and len(ctas) % cluster == 0
    for i, c in enumerate(ctas):   # the parts of an item are neighbours in one cluster, in order
        if c[0] and c[2]:
            assert i % cluster and ctas[i - 1][:3] == (c[0], c[1], c[2] - 1)
    alone = _ctas(family, 1, nq, nk)
    assert {c[0]: c[3] for c in alone if c[0]} == parts   # a head's own


def test_some_walked_shapes_have_idle_ctas_beside_an_unsplit_pass():
    hit = 0
    for bh, nq, nk in WALK:
        ctas = _ctas("tcgen05", bh, nq, nk)
        hit += any(c[0] == 0 and c[3] == 1 for c in ctas)
    assert hit >= 3


@pytest.mark.parametrize("family", ("tcgen05", "simt"))
def test_a_window_bounds_the_number_of_parts(family):
    """Parts are of the tiles an item sees: a window of a few tiles leaves nothing to split."""
    def parts(window):
        return {c[0]: c[3] for c in _ctas(family, 1, 100, 8000, window)}[3]
    assert parts(0) > 1 and parts(64) == 1
    assert 1 < parts(4000) <= parts(0) and parts(8000) == parts(0)
