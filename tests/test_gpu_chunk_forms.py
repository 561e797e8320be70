"""Chunk attention where the launch form changes with the size: straight from the cache for few pairs,
key slices folded in a cluster (2 to 8 of them) where a launch has few query tiles, the plain form
beyond. CPU definition: attention.rs:56-102 per query row."""
import numpy as np
import pytest
import torch

import oracle as O
from tests import cases

pytestmark = pytest.mark.gpu


def _sampled(tokens):
    return sorted({0, tokens // 3, tokens // 2, max(0, tokens - 2), tokens - 1})


# (tokens, pos0): small form at its edges; 8, 7, .. 2 slices; odd tile counts; slices without keys; none
SIZES = [(1, 0), (3, 4), (1, 383), (1, 384), (9, 375), (9, 376), (5, 127), (37, 29), (90, 45), (91, 46), (37, 700), (21, 1900), (43, 1111), (64, 2500),
         (130, 1500), (170, 1024), (301, 3001), (230, 90), (337, 120)]


@pytest.mark.parametrize("dtype", [0, 1, 2], ids=["f32", "q8_0", "q4_0"])
@pytest.mark.parametrize("tokens,pos0", SIZES)
def test_chunk_form_follows_the_size(tokens, pos0, dtype):
    from hipml_b200 import api
    heads, n_kv, hd = 24, 4, 256
    seq, stride = pos0 + tokens, pos0 + tokens + 5
    gen = torch.Generator(device="cuda").manual_seed(seq)
    kf, vf = (torch.randn(seq, n_kv * hd, device="cuda", generator=gen) for _ in range(2))
    q = torch.randn(tokens, heads * hd, device="cuda", generator=gen)
    if dtype == 0:
        k, v = (torch.full((stride, n_kv * hd), float("nan"), device="cuda") for _ in range(2))
        k[:seq], v[:seq] = kf, vf
        kq, vq = kf.cpu().numpy(), vf.cpu().numpy()
    else:
        row = (272, 144)[dtype - 1]
        k, v = (torch.full((n_kv * stride * row,), 0x7E, dtype=torch.uint8, device="cuda") for _ in range(2))
        api.kv_encode_bulk(kf, vf, k, v, n_kv, hd, stride, 0, 0, seq, dtype - 1)
        deq = (O.dequantize_q8, O.dequantize_q4)[dtype - 1]
        kq, vq = (cases.unpack_head_major(deq(np.ascontiguousarray(c.cpu().numpy().reshape(n_kv, stride, row)[:, :seq])),
                                          n_kv, seq, hd) for c in (k, v))
    ws = torch.full((api.attn_chunk_workspace_bytes(n_kv, hd, pos0, tokens),), 0x7E, dtype=torch.uint8, device="cuda")
    out = torch.full((tokens, heads * hd), float("nan"), device="cuda")
    api.attn_chunk(q, k, v, out, heads, n_kv, hd, pos0, tokens, dtype, stride, workspace=ws)
    assert api.check_device_status() == 0
    got, qn = out.cpu().numpy(), q.cpu().numpy()
    assert np.all(np.isfinite(got))
    for t in _sampled(tokens):
        n = pos0 + t + 1
        want = O.attn_causal_f32(qn[t], kq[:n], vq[:n], heads, n_kv, hd, n, 0.0625)
        ok, ma, rl = cases.attention_within_bar(want, got[t])
        assert ok and rl <= 5e-5, (t, ma, rl)
    # the staged entry (never the small form), with the output gate
    cap = (seq + 127) // 128 * 128
    api.attn_chunk_stage(k, v, n_kv, hd, dtype, stride, 0, seq, cap, ws)
    gate = torch.randn(tokens, heads * hd, device="cuda", generator=gen)
    gated = torch.full_like(out, float("nan"))
    api.attn_chunk_staged_gated(q, gated, gate, heads, n_kv, hd, pos0, tokens, cap, ws)
    assert api.check_device_status() == 0
    ma = O.max_abs(got * torch.sigmoid(gate).cpu().numpy(), gated.cpu().numpy())
    assert ma <= 2e-5, ma


# one slice written by bulk copies; read back through the gate; 2, 4 and 8 slices folded in a cluster
@pytest.mark.parametrize("tokens,pos0", [(2048, 0), (301, 3001), (130, 1500), (37, 700)])
def test_a_row_without_a_finite_score_is_not_a_number(tokens, pos0):
    """Keys past the largest f16 overflow in the single-pass form. A row that sees one finite score has its value; one
    whose scores are all -infinity has no softmax, and says so."""
    from hipml_b200 import api
    heads, n_kv, hd = 24, 4, 256
    seq, cap = pos0 + tokens, (pos0 + tokens + 127) // 128 * 128
    gen = torch.Generator(device="cuda").manual_seed(seq)
    k = torch.full((seq, n_kv * hd), 1e5, device="cuda")
    k[0, 2 * hd:] = 0.0   # (KV heads 2 and 3: the first key is finite)
    v = torch.randn(seq, n_kv * hd, device="cuda", generator=gen)
    q = -1.0 - torch.rand(tokens, heads * hd, device="cuda", generator=gen)
    gate = torch.randn(tokens, heads * hd, device="cuda", generator=gen)
    ws = torch.full((api.attn_chunk_workspace_bytes(n_kv, hd, 0, cap),), 0x7E, dtype=torch.uint8, device="cuda")
    api.attn_chunk_stage(k, v, n_kv, hd, 0, seq, 0, seq, cap, ws)
    out, gated = (torch.full((tokens, heads * hd), 3.0, device="cuda") for _ in range(2))
    api.attn_chunk_staged(q, out, heads, n_kv, hd, pos0, tokens, cap, ws, mode=1)
    api.attn_chunk_staged_gated(q, gated, gate, heads, n_kv, hd, pos0, tokens, cap, ws, mode=1)
    assert api.check_device_status() == 0
    want = v[0].view(n_kv, 1, hd)[2:].expand(2, heads // n_kv, hd).reshape(-1)   # (f16 values: half a unit in 2^-11)
    half = heads * hd // 2
    for got, scale in ((out, torch.ones_like(gate)), (gated, torch.sigmoid(gate))):
        assert torch.isnan(got[:, :half]).all()
        assert ((got[:, half:] - want * scale[:, half:]).abs() <= 5e-4 * want.abs() + 1e-6).all()


# rows_live is 126 and 6 (21 queries of six heads, one left over) or 128 and 96: rows in fours, and a remainder
@pytest.mark.parametrize("heads,n_kv,tokens", [(24, 4, 1996), (32, 4, 2044)], ids=["group6", "group8"])
def test_gated_rows_that_were_also_moved_to_memory(heads, n_kv, tokens):
    """More than 64 key tiles in one slice: part of a row is in memory when it is read out, and the gate with it."""
    from hipml_b200 import api
    hd, pos0 = 256, 9000
    seq, cap = pos0 + tokens, (pos0 + tokens + 127) // 128 * 128
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    kc, vc = (torch.zeros(n_kv * seq * 272, dtype=torch.uint8, device="cuda") for _ in range(2))
    k, v = (torch.randn(seq, n_kv * hd, device="cuda", generator=gen) for _ in range(2))
    api.kv_encode_bulk(k, v, kc, vc, n_kv, hd, seq, 0, 0, seq)
    q, gate = (torch.randn(tokens, heads * hd, device="cuda", generator=gen) for _ in range(2))
    ws = torch.full((api.attn_chunk_workspace_bytes(n_kv, hd, 0, cap),), 0x7E, dtype=torch.uint8, device="cuda")
    api.attn_chunk_stage(kc, vc, n_kv, hd, 1, seq, 0, seq, cap, ws)
    plain, gated = (torch.full((tokens, heads * hd), float("nan"), device="cuda") for _ in range(2))
    api.attn_chunk_staged(q, plain, heads, n_kv, hd, pos0, tokens, cap, ws)
    api.attn_chunk_staged_gated(q, gated, 2.0 * gate, heads, n_kv, hd, pos0, tokens, cap, ws)
    assert api.check_device_status() == 0
    assert torch.isfinite(plain).all()
    want = plain.double() * torch.sigmoid(2.0 * gate.double())
    # (the attention's bits are the ungated call's; expf, a sum, a division and a product: four roundings and expf's two)
    assert ((gated.double() - want).abs() <= 4e-7 * want.abs() + 1e-30).all()
    for t in (0, 20, 21, tokens - 2, tokens - 1):   # and against the definition
        n = pos0 + t + 1
        kq, vq = (cases.unpack_head_major(O.dequantize_q8(np.ascontiguousarray(
            c.cpu().numpy().reshape(n_kv, seq, 272)[:, :n])), n_kv, n, hd) for c in (kc, vc))
        ok, ma, rl = cases.attention_within_bar(
            O.attn_causal_f32(q[t].cpu().numpy(), kq, vq, heads, n_kv, hd, n, 0.0625), plain[t].cpu().numpy())
        assert ok and rl <= 5e-5, (t, ma, rl)
