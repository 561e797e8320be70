"""Decode at the edges of the default body's work units: a warp takes 16 rows, or 32 once a step has
more 16-row units than warps; 8 warps per CTA, two CTAs per run. CPU definition: ops.rs:449-518."""
import numpy as np
import pytest
import torch

import oracle as O
from tests import cases

pytestmark = pytest.mark.gpu

# 288 warps per head at 4 KV heads: the unit becomes 32 rows past 4,608; 9,217 is a second unit
LENGTHS = [1, 15, 16, 17, 31, 33, 127, 129, 255, 257, 4608, 4609, 4640, 9217]


@pytest.mark.parametrize("dtype", [0, 1], ids=["q8_0", "q4_0"])
@pytest.mark.parametrize("seq", LENGTHS)
def test_step_with_append_at_the_edges_of_a_unit(seq, dtype):
    from hipml_b200 import api
    heads, n_kv, hd, scale, row = 24, 4, 256, 0.0625, (272, 144)[dtype]
    stride = seq + 3
    gen = torch.Generator(device="cuda").manual_seed(seq)
    k, v = (torch.randn(seq, n_kv * hd, device="cuda", generator=gen) for _ in range(2))
    q = torch.randn(heads * hd, device="cuda", generator=gen)
    # rows past the live ones have scales that would poison any output they reach (f16 NaN)
    kc, vc = (torch.full((n_kv * stride * row,), 0x7E, dtype=torch.uint8, device="cuda") for _ in range(2))
    api.kv_encode_bulk(k, v, kc, vc, n_kv, hd, stride, 0, 0, seq, dtype)
    want_k, want_v = kc.cpu().numpy(), vc.cpu().numpy()
    for c in (kc, vc):    # the row to append arrives with the step
        c.view(n_kv, stride, row)[:, seq - 1] = 0x7E
    splits = api.decode_splits(seq)
    acc, ml = torch.empty(heads * splits * hd, device="cuda"), torch.empty(heads * splits * 2, device="cuda")
    out = torch.full((heads * hd,), float("nan"), device="cuda")
    step = torch.tensor([seq - 1, seq] + [0] * 6, dtype=torch.int32, device="cuda")
    api.attn_decode_kv_append(step, k[seq - 1], v[seq - 1], q, kc, vc, acc, ml, out, heads, n_kv, hd, stride, scale,
                              splits, selector=dtype)
    assert api.check_device_status() == 0
    assert np.array_equal(kc.cpu().numpy(), want_k) and np.array_equal(vc.cpu().numpy(), want_v)
    want = O.attn_decode_kv(q.cpu().numpy(), want_k.reshape(n_kv, stride, row), want_v.reshape(n_kv, stride, row),
                            dtype, heads, n_kv, hd, seq, scale, stride=stride)
    ok, ma, rl = cases.attention_within_bar(want, out.cpu().numpy())
    assert ok and ma <= 2e-5 and rl <= 2e-5, (ma, rl)


# clusters of four, eight and two; slices of the outputs that lie within, begin or cross a head
@pytest.mark.parametrize("seq", [40, 700, 1500])
@pytest.mark.parametrize("group", [1, 3, 5, 7, 8])
def test_partials_sent_within_a_cluster_for_any_group(group, seq):
    from hipml_b200 import api
    n_kv, hd, scale = 4, 256, 0.0625
    heads = n_kv * group
    gen = torch.Generator(device="cuda").manual_seed(seq + group)
    k, v = (torch.randn(seq, n_kv * hd, device="cuda", generator=gen) for _ in range(2))
    q = torch.randn(heads * hd, device="cuda", generator=gen)
    kc, vc = (torch.zeros(n_kv * seq * 272, dtype=torch.uint8, device="cuda") for _ in range(2))
    api.kv_encode_bulk(k, v, kc, vc, n_kv, hd, seq, 0, 0, seq)
    splits = api.decode_splits(seq)
    acc, ml = torch.empty(heads * splits * hd, device="cuda"), torch.empty(heads * splits * 2, device="cuda")
    out = torch.full((heads * hd,), float("nan"), device="cuda")
    step = torch.tensor([seq - 1, seq] + [0] * 6, dtype=torch.int32, device="cuda")
    api.attn_decode_kv(step, q, kc, vc, acc, ml, out, heads, n_kv, hd, seq, scale, splits)
    assert api.check_device_status() == 0
    want = O.attn_decode_kv(q.cpu().numpy(), kc.cpu().numpy().reshape(n_kv, seq, 272), vc.cpu().numpy().reshape(n_kv, seq, 272),
                            0, heads, n_kv, hd, seq, scale, stride=seq)
    ok, ma, rl = cases.attention_within_bar(want, out.cpu().numpy())
    assert ok and ma <= 2e-5 and rl <= 2e-5, (ma, rl)


def test_lengths_that_change_between_launches_are_seen():
    """The kernel plans from the length as it stands before the grids ahead are done; a length written by
    the kernel right before it must win."""
    from hipml_b200 import api
    heads, n_kv, hd, scale, stride = 24, 4, 256, 0.0625, 6000
    gen = torch.Generator(device="cuda").manual_seed(5)
    kc, vc = (torch.zeros(n_kv * stride * 272, dtype=torch.uint8, device="cuda") for _ in range(2))
    k, v = (torch.randn(stride, n_kv * hd, device="cuda", generator=gen) for _ in range(2))
    api.kv_encode_bulk(k, v, kc, vc, n_kv, hd, stride, 0, 0, stride)
    q = torch.randn(heads * hd, device="cuda", generator=gen)
    lengths = [1, 5000, 700, 4700, 16, 5999, 33]
    steps = [torch.tensor([n - 1, n] + [0] * 6, dtype=torch.int32, device="cuda") for n in lengths]
    splits = api.decode_splits(stride)
    acc, ml = torch.empty(heads * splits * hd, device="cuda"), torch.empty(heads * splits * 2, device="cuda")
    moving, outs, want = steps[0].clone(), [], []
    for s in steps:
        o = torch.empty(heads * hd, device="cuda")
        api.attn_decode_kv(s, q, kc, vc, acc, ml, o, heads, n_kv, hd, stride, scale, splits)
        want.append(o)
    for s in steps:
        moving.copy_(s)
        o = torch.empty(heads * hd, device="cuda")
        api.attn_decode_kv(moving, q, kc, vc, acc, ml, o, heads, n_kv, hd, stride, scale, splits)
        outs.append(o)
    assert api.check_device_status() == 0
    for a, b in zip(outs, want):
        assert torch.equal(a, b)


# columns whose lengths cross a 16- or 32-row unit, the change of the unit (4,608) or nothing
@pytest.mark.parametrize("cols", [2, 4, 5, 8])
@pytest.mark.parametrize("pos0", [0, 13, 29, 125, 200, 1278, 4604, 9214])
def test_columns_side_by_side_give_each_columns_own_bits(pos0, cols):
    from hipml_b200 import api
    heads, n_kv, hd, scale, stride = 24, 4, 256, 0.0625, pos0 + cols + 2
    gen = torch.Generator(device="cuda").manual_seed(pos0 + cols)
    kc, vc = (torch.full((n_kv * stride * 272,), 0x7E, dtype=torch.uint8, device="cuda") for _ in range(2))
    k, v = (torch.randn(pos0 + cols, n_kv * hd, device="cuda", generator=gen) for _ in range(2))
    api.kv_encode_bulk(k, v, kc, vc, n_kv, hd, stride, 0, 0, pos0 + cols)
    q = torch.randn(cols, heads * hd, device="cuda", generator=gen)
    splits = api.decode_splits(pos0 + cols)
    acc, ml = (torch.empty(cols * heads * splits * n, device="cuda") for n in (hd, 2))
    out = torch.full((cols, heads * hd), float("nan"), device="cuda")
    pos = torch.tensor([[pos0 + c, pos0 + c + 1] for c in range(cols)], dtype=torch.int32, device="cuda")
    for _ in range(2):   # the second launch finds the first one's counters
        api.attn_decode_cols(pos, q, kc, vc, acc, ml, out, heads, n_kv, hd, stride, scale, splits, cols,
                             heads * splits * hd, heads * splits * 2, heads * hd)
    for c in range(cols):
        one = torch.empty(heads * hd, device="cuda")
        step = torch.tensor([pos0 + c, pos0 + c + 1] + [0] * 6, dtype=torch.int32, device="cuda")
        api.attn_decode_kv(step, q[c], kc, vc, acc, ml, one, heads, n_kv, hd, stride, scale, splits)
        assert torch.equal(one, out[c]), f"column {c}"
    assert api.check_device_status() == 0


@pytest.mark.parametrize("heads,n_kv", [(24, 4), (8, 1), (2, 2)])
@pytest.mark.parametrize("n_ctx,pos0,rows", [(1, 0, 1), (33, 31, 2), (260, 250, 3), (2100, 2090, 8), (8200, 8199, 1),
                                             (8200, 3, 2)])
def test_f32_cache_decode_at_the_edges_of_runs(heads, n_kv, n_ctx, pos0, rows):
    """head_dim 256: runs of ceil(n_ctx / splits) rows, eight warps per run, eight runs per cluster."""
    from hipml_b200 import api
    hd = 256
    gen = torch.Generator(device="cuda").manual_seed(n_ctx + rows)
    k, v = (torch.full((n_ctx, n_kv * hd), float("nan"), device="cuda") for _ in range(2))
    live = pos0 + rows
    k[:live] = torch.randn(live, n_kv * hd, device="cuda", generator=gen)
    v[:live] = torch.randn(live, n_kv * hd, device="cuda", generator=gen)
    q = torch.randn(rows, heads * hd, device="cuda", generator=gen)
    splits = api.cols_splits(n_ctx)
    acc, ml = (torch.full((rows * heads * splits * n,), float("nan"), device="cuda") for n in (hd, 2))
    out = torch.full((rows, heads * hd), float("nan"), device="cuda")
    for _ in range(2):
        api.attn_decode_cols_f32(q, k, v, acc, ml, out, heads, n_kv, hd, n_ctx, pos0, rows)
    kn, vn, qn = k.cpu().numpy(), v.cpu().numpy(), q.cpu().numpy()
    for c in range(rows):
        seq = pos0 + c + 1
        want = O.attn_causal_f32(qn[c], kn[:seq], vn[:seq], heads, n_kv, hd, seq, 0.0625)
        assert O.max_abs(want, out[c].cpu().numpy()) <= 5e-6 and O.rel_l2(want, out[c].cpu().numpy()) <= 5e-6
