"""Decode at the edges of the default body's work units: a warp takes 16 rows, or 32 once a step has
more 16-row units than warps; 8 warps per CTA, two CTAs per run. CPU definition: ops.rs:449-518."""
import math
import re

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


@pytest.mark.parametrize("append", [False, True], ids=["rows", "rows and append"])
@pytest.mark.parametrize("dtype", [0, 1], ids=["q8_0", "q4_0"])
@pytest.mark.parametrize("seq,stride", [(1, 40), (700, 704), (700, 9000), (8999, 9000)])
def test_one_slot_is_a_stream(seq, stride, dtype, append):
    from hipml_b200 import api
    heads, n_kv, hd, scale, row = 24, 4, 256, 0.0625, (272, 144)[dtype]
    gen = torch.Generator(device="cuda").manual_seed(seq + dtype)
    k, v = (torch.randn(seq, n_kv * hd, device="cuda", generator=gen) for _ in range(2))
    q = torch.randn(heads * hd, device="cuda", generator=gen)
    kc, vc = (torch.full((n_kv * stride * row,), 0x7E, dtype=torch.uint8, device="cuda") for _ in range(2))
    api.kv_encode_bulk(k, v, kc, vc, n_kv, hd, stride, 0, 0, seq, dtype)
    want_k, want_v = kc.clone(), vc.clone()
    deq = (O.dequantize_q8, O.dequantize_q4)[dtype]
    kq, vq = (torch.from_numpy(cases.unpack_head_major(deq(np.ascontiguousarray(
        c.cpu().numpy().reshape(n_kv, stride, row)[:, :seq])), n_kv, seq, hd)).cuda() for c in (kc, vc))
    splits = api.batch_splits(stride, 1)
    acc, ml = (torch.full((heads * splits * n,), float("nan"), device="cuda") for n in (hd, 2))
    out = torch.full((heads * hd,), float("nan"), device="cuda")
    pos = torch.tensor([[seq - 1, seq]], dtype=torch.int32, device="cuda")
    tail = (heads, n_kv, hd, stride, scale, splits, n_kv * stride * row, heads * splits * hd, heads * splits * 2, heads * hd, 1)
    if append:
        for c in (kc, vc):   # the row to append arrives with the step
            c.view(n_kv, stride, row)[:, seq - 1] = 0x7E
        api.attn_decode_batch_append(pos, k[seq - 1:], v[seq - 1:], q, kc, vc, acc, ml, out, *tail, dtype=dtype)
    else:
        api.attn_decode_rows(pos, q, kc, vc, acc, ml, out, *tail, dtype=dtype)
    assert api.check_device_status() == 0
    assert torch.equal(kc, want_k) and torch.equal(vc, want_v)
    assert _close(out, _attend(q, kq, vq, n_kv, hd, scale))


# more KV heads than the device holds clusters of eight for two launches, and a tensor-parallel rank's one
@pytest.mark.parametrize("n_kv,group", [(8, 4), (7, 3), (6, 4), (1, 6)])
@pytest.mark.parametrize("seq", [300, 600, 1000, 1300])
def test_step_with_other_numbers_of_heads(seq, n_kv, group):
    from hipml_b200 import api
    heads, hd, scale = n_kv * group, 256, 0.0625
    gen = torch.Generator(device="cuda").manual_seed(seq + n_kv)
    k, v = (torch.randn(seq, n_kv * hd, device="cuda", generator=gen) for _ in range(2))
    q = torch.randn(heads * hd, device="cuda", generator=gen)
    kc, vc = (torch.zeros(n_kv * seq * 272, dtype=torch.uint8, device="cuda") for _ in range(2))
    api.kv_encode_bulk(k, v, kc, vc, n_kv, hd, seq, 0, 0, seq)
    kq, vq = (torch.from_numpy(cases.unpack_head_major(O.dequantize_q8(c.cpu().numpy().reshape(n_kv, seq, 272)), n_kv,
                                                       seq, hd)).cuda() for c in (kc, vc))
    splits = api.decode_splits(seq)
    acc, ml = (torch.full((heads * splits * n,), float("nan"), device="cuda") for n in (hd, 2))
    out = torch.full((heads * hd,), float("nan"), device="cuda")
    step = torch.tensor([seq - 1, seq] + [0] * 6, dtype=torch.int32, device="cuda")
    api.attn_decode_kv(step, q, kc, vc, acc, ml, out, heads, n_kv, hd, seq, scale, splits)
    assert api.check_device_status() == 0
    assert _close(out, _attend(q, kq, vq, n_kv, hd, scale))


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


@pytest.mark.parametrize("cols", [2, 5, 8])
def test_column_lengths_that_change_between_launches_are_seen(cols):
    """The columns are grouped and planned from the lengths as they stand before the grids ahead are done; lengths written
    by the kernel right before must win: other units, runs, groups and tiles of heads."""
    from hipml_b200 import api
    heads, n_kv, hd, scale, stride = 24, 4, 256, 0.0625, 6000
    gen = torch.Generator(device="cuda").manual_seed(6)
    kc, vc = (torch.zeros(n_kv * stride * 272, dtype=torch.uint8, device="cuda") for _ in range(2))
    k, v = (torch.randn(stride, n_kv * hd, device="cuda", generator=gen) for _ in range(2))
    api.kv_encode_bulk(k, v, kc, vc, n_kv, hd, stride, 0, 0, stride)
    q = torch.randn(cols, heads * hd, device="cuda", generator=gen)
    splits = api.decode_splits(stride)
    acc, ml = (torch.empty(cols * heads * splits * n, device="cuda") for n in (hd, 2))
    args = (heads, n_kv, hd, stride, scale, splits, cols, heads * splits * hd, heads * splits * 2, heads * hd)
    # neighbours of one plan; across the change of the unit (4,608); every column its own plan; empty ones among them
    sets = [[1 + c for c in range(cols)], [5000 + c for c in range(cols)], [700 + c for c in range(cols)],
            [4607 + c for c in range(cols)], [100 + 733 * c for c in range(cols)], [(c % 2) * 5990 + c for c in range(cols)],
            [300 + c // 2 for c in range(cols)]]
    tables = [torch.tensor([[n - 1, n] for n in s], dtype=torch.int32, device="cuda") for s in sets]

    def attend(pos):
        out = torch.full((cols, heads * hd), float("nan"), device="cuda")
        api.attn_decode_cols(pos, q, kc, vc, acc, ml, out, *args)
        return out

    want = []
    for t in tables:
        attend(t)
        want.append(attend(t))
        torch.cuda.synchronize()
    moving, outs = tables[-1].clone(), []
    for t in tables:
        moving.copy_(t)
        outs.append(attend(moving))
    assert api.check_device_status() == 0
    for s, a, b in zip(sets, outs, want):
        assert torch.isfinite(a).all() and torch.equal(a, b), s
    kq, vq = (torch.from_numpy(cases.unpack_head_major(O.dequantize_q8(c.cpu().numpy().reshape(n_kv, stride, 272)), n_kv,
                                                       stride, hd)).cuda() for c in (kc, vc))
    for s, a in zip(sets, outs):
        for c, n in enumerate(s):
            if n:
                assert _close(a[c], _attend(q[c], kq[:n], vq[:n], n_kv, hd, scale)), (s, c)


def _device_status():
    from hipml_b200 import _lib, api
    try:
        return api.check_device_status()
    except _lib.HipmlError as e:
        return int(re.search(r"code (\d+)", e.text).group(1))


@pytest.mark.parametrize("fold_mode", [0, 1], ids=["fold_inside", "fold_launch"])
@pytest.mark.parametrize("entry", ["step", "step append", "columns", "slots", "slots append"])
def test_a_length_past_the_cache_counts_as_the_cache_s(entry, fold_mode):
    """No form reads or writes past the `stride` rows of a head; an append past them is reported (status 22)."""
    from hipml_b200 import api
    heads, n_kv, hd, scale, stride, beyond = 24, 4, 256, 0.0625, 300, 40
    gen = torch.Generator(device="cuda").manual_seed(8)
    # (rows follow the last head, so that a kernel that went on would be seen and not fault)
    room = n_kv * stride * 272 + 4096 * 272
    kc, vc = (torch.full((2, room), 0x7E, dtype=torch.uint8, device="cuda") for _ in range(2))
    k, v = (torch.randn(stride, n_kv * hd, device="cuda", generator=gen) for _ in range(2))
    for s in range(2):
        api.kv_encode_bulk(k, v, kc[s], vc[s], n_kv, hd, stride, 0, 0, stride)
    want_k, want_v = kc.clone(), vc.clone()
    live = n_kv * stride * 272
    kq, vq = (torch.from_numpy(cases.unpack_head_major(O.dequantize_q8(c[0, :live].cpu().numpy().reshape(n_kv, stride, 272)),
                                                       n_kv, stride, hd)).cuda() for c in (kc, vc))
    q = torch.randn(2, heads * hd, device="cuda", generator=gen)
    new = torch.randn(2, n_kv * hd, device="cuda", generator=gen)
    splits = 8
    acc, ml = (torch.empty(2 * heads * splits * n, device="cuda") for n in (hd, 2))
    out = torch.full((2, heads * hd), float("nan"), device="cuda")
    lens = [stride + beyond, 7] if entry.startswith("slots") else [stride + beyond, stride + 1]
    pos = torch.tensor([[n - 1, n] for n in lens], dtype=torch.int32, device="cuda")
    args = (heads, n_kv, hd, stride, scale, splits)
    slots = (heads * splits * hd, heads * splits * 2, heads * hd, 2)
    api.set_decode_fold_mode(fold_mode)
    try:
        if entry == "step":
            api.attn_decode_kv(pos[0], q[0], kc[0], vc[0], acc, ml, out[0], *args)
        elif entry == "step append":
            api.attn_decode_kv_append(pos[0], new[0], new[0], q[0], kc[0], vc[0], acc, ml, out[0], *args)
        elif entry == "columns":
            api.attn_decode_cols(pos, q, kc, vc, acc, ml, out, *args, 2, *slots[:3])
        elif entry == "slots":
            api.attn_decode_rows(pos, q, kc, vc, acc, ml, out, *args, room, *slots)
        else:
            new_rows = torch.stack([new[0], k[6]])   # (slot 1 appends what it holds already)
            new_v = torch.stack([new[1], v[6]])
            api.attn_decode_batch_append(pos, new_rows, new_v, q, kc, vc, acc, ml, out, *args, room, *slots)
    finally:
        api.set_decode_fold_mode(0)
    assert _device_status() == (22 if "append" in entry else 0)
    assert torch.equal(kc, want_k) and torch.equal(vc, want_v)
    for s, n in enumerate(lens):
        if s == 0 or not entry.startswith("step"):
            n = min(n, stride)
            assert _close(out[s], _attend(q[s], kq[:n], vq[:n], n_kv, hd, scale)), f"row {s}"


@pytest.mark.parametrize("entry,selector,hd", [("step", 6, 256), ("step", 6, 64), ("step", 0, 64), ("step", 1, 64),
                                               ("step", 8, 256), ("append", 8, 256), ("slots", 0, 64), ("slots", 1, 64),
                                               ("shared slots", 8, 256)])
def test_a_length_past_the_cache_counts_as_the_cache_s_in_every_body(entry, selector, hd):
    """The scalar body (any head size) and the tcgen05 one: as the default one in the test above."""
    from hipml_b200 import api
    heads, n_kv, scale, stride, beyond, slots = 12, 2, 0.0625, 300, 200, 2
    dtype = int(selector == 1)
    row = (34, 18)[dtype] * hd // 32
    gen = torch.Generator(device="cuda").manual_seed(hd)
    room = n_kv * stride * row + 1024 * 272   # (rows follow the last head: a kernel that went on would be seen and not fault)
    kc, vc = (torch.full((slots, room), 0x7E, dtype=torch.uint8, device="cuda") for _ in range(2))
    k, v = (torch.randn(stride, n_kv * hd, device="cuda", generator=gen) for _ in range(2))
    for s in range(slots):
        api.kv_encode_bulk(k, v, kc[s], vc[s], n_kv, hd, stride, 0, 0, stride, dtype)
    before = kc.clone(), vc.clone()
    live, deq = n_kv * stride * row, (O.dequantize_q8, O.dequantize_q4)[dtype]
    kq, vq = (torch.from_numpy(cases.unpack_head_major(deq(c[0, :live].cpu().numpy().reshape(n_kv, stride, row)), n_kv, stride,
                                                       hd)).cuda() for c in (kc, vc))
    q = torch.randn(slots, heads * hd, device="cuda", generator=gen)
    new = torch.randn(n_kv * hd, device="cuda", generator=gen)
    splits = 8
    acc, ml = (torch.full((slots * heads * splits * n,), float("nan"), device="cuda") for n in (hd, 2))
    out = torch.full((slots, heads * hd), float("nan"), device="cuda")
    pos = torch.tensor([[stride + beyond - 1, stride + beyond], [6, 7]], dtype=torch.int32, device="cuda")
    args = (heads, n_kv, hd, stride, scale, splits)
    try:
        if entry == "step":
            api.attn_decode_kv(pos[0], q[0], kc[0], vc[0], acc, ml, out[0], *args, selector=selector)
        elif entry == "append":
            api.attn_decode_kv_append(pos[0], new, new, q[0], kc[0], vc[0], acc, ml, out[0], *args, selector=selector)
        else:
            api.set_decode_body(2 if selector == 8 else 1)
            api.attn_decode_rows(pos, q, kc, vc, acc, ml, out, *args, room, heads * splits * hd, heads * splits * 2,
                                 heads * hd, slots, dtype=dtype)
    finally:
        api.set_decode_body(1)
    assert _device_status() == (22 if entry == "append" else 0)
    assert torch.equal(kc, before[0]) and torch.equal(vc, before[1])
    for s, n in enumerate([stride, 7] if "slots" in entry else [stride]):
        assert _close(out[s], _attend(q[s], kq[:n], vq[:n], n_kv, hd, scale)), f"row {s}"


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
    for _ in range(2):   # the second launch finds the first one's counters, and scratch that was never written
        acc.fill_(float("nan"))
        ml.fill_(float("nan"))
        out.fill_(float("nan"))
        api.attn_decode_cols(pos, q, kc, vc, acc, ml, out, heads, n_kv, hd, stride, scale, splits, cols,
                             heads * splits * hd, heads * splits * 2, heads * hd)
    for c in range(cols):
        one = torch.empty(heads * hd, device="cuda")
        step = torch.tensor([pos0 + c, pos0 + c + 1] + [0] * 6, dtype=torch.int32, device="cuda")
        api.attn_decode_kv(step, q[c], kc, vc, acc, ml, one, heads, n_kv, hd, stride, scale, splits)
        assert torch.equal(one, out[c]), f"column {c}"
    assert api.check_device_status() == 0


# groups of columns in turn and side by side, columns of two launches, few splits over a long stream
@pytest.mark.parametrize("fold_mode", [0, 1], ids=["fold_inside", "fold_launch"])
@pytest.mark.parametrize("pos0,cols,splits", [(0, 3, 1), (10, 33, 5), (100, 16, 13), (700, 40, 90), (1278, 40, 128),
                                              (3000, 3, 64), (5000, 9, 24), (5000, 12, 128)])
def test_columns_of_every_form_give_each_columns_own_bits(pos0, cols, splits, fold_mode):
    from hipml_b200 import api
    heads, n_kv, hd, scale, stride = 24, 4, 256, 0.0625, pos0 + cols + 2
    gen = torch.Generator(device="cuda").manual_seed(pos0 + cols)
    kc, vc = (torch.full((n_kv * stride * 272,), 0x7E, dtype=torch.uint8, device="cuda") for _ in range(2))
    k, v = (torch.randn(pos0 + cols, n_kv * hd, device="cuda", generator=gen) for _ in range(2))
    api.kv_encode_bulk(k, v, kc, vc, n_kv, hd, stride, 0, 0, pos0 + cols)
    q = torch.randn(cols, heads * hd, device="cuda", generator=gen)
    acc, ml = (torch.empty(cols * heads * splits * n, device="cuda") for n in (hd, 2))
    out = torch.empty(cols, heads * hd, device="cuda")
    pos = torch.tensor([[pos0 + c, pos0 + c + 1] for c in range(cols)], dtype=torch.int32, device="cuda")
    api.set_decode_fold_mode(fold_mode)
    try:
        for _ in range(2):
            for x in (acc, ml, out):
                x.fill_(float("nan"))
            api.attn_decode_cols(pos, q, kc, vc, acc, ml, out, heads, n_kv, hd, stride, scale, splits, cols,
                                 heads * splits * hd, heads * splits * 2, heads * hd)
    finally:
        api.set_decode_fold_mode(0)
    for c in range(cols):
        one = torch.empty(heads * hd, device="cuda")
        step = torch.tensor([pos0 + c, pos0 + c + 1] + [0] * 6, dtype=torch.int32, device="cuda")
        api.attn_decode_kv(step, q[c], kc, vc, acc, ml, one, heads, n_kv, hd, stride, scale, splits)
        assert torch.equal(one, out[c]), f"column {c}"
    assert api.check_device_status() == 0


def _quantised_cache(gen, rows, stride, n_kv, dtype, room=0):
    """K and V bytes of `rows` random rows per head (NaN scales past them), and the rows as f64 [rows][n_kv * 256]."""
    from hipml_b200 import api
    row = (272, 144)[dtype]
    kc, vc = (torch.full((n_kv * stride * row + room,), 0x7E, dtype=torch.uint8, device="cuda") for _ in range(2))
    if rows:
        k, v = (torch.randn(rows, n_kv * 256, device="cuda", generator=gen) for _ in range(2))
        api.kv_encode_bulk(k, v, kc, vc, n_kv, 256, stride, 0, 0, rows, dtype)
    deq = (O.dequantize_q8, O.dequantize_q4)[dtype]
    return kc, vc, [torch.from_numpy(cases.unpack_head_major(
        deq(np.ascontiguousarray(c[:n_kv * stride * row].cpu().numpy().reshape(n_kv, stride, row)[:, :rows])), n_kv, rows,
        256)).double().cuda() for c in (kc, vc)]


def _triple(q, k, v, n_kv, scale):
    """log2 of the sum of 2^score per head, and the attention output [heads][256], in f64."""
    group = q.numel() // 256 // n_kv
    s = torch.einsum("hgd,nhd->hgn", q.double().view(n_kv, group, 256), k.view(-1, n_kv, 256)) * scale
    out = torch.einsum("hgn,nhd->hgd", s.softmax(-1), v.view(-1, n_kv, 256))
    return s.logsumexp(-1).flatten() / math.log(2.0), out.reshape(n_kv * group, 256)


# every body of the head_dim-256 kernel: one run, several, a head in one cluster
@pytest.mark.parametrize("fold_mode", [0, 1], ids=["fold_inside", "fold_launch"])
@pytest.mark.parametrize("selector", [0, 1, 6, 7, 8])
@pytest.mark.parametrize("seq", [1, 40, 700, 5000])
def test_a_shard_s_triple_is_its_sum_of_weights(seq, selector, fold_mode):
    """acc * 2^max and sum * 2^max are the sums over the rows, whichever body made them: a caller folds them with others."""
    from hipml_b200 import api
    heads, n_kv, hd, scale = 24, 4, 256, 0.0625
    gen = torch.Generator(device="cuda").manual_seed(seq)
    kc, vc, (k, v) = _quantised_cache(gen, seq, seq + 3, n_kv, int(selector == 1))
    q = torch.randn(heads * hd, device="cuda", generator=gen)
    splits = api.decode_splits(seq)
    acc, ml = (torch.full((heads * splits * n,), float("nan"), device="cuda") for n in (hd, 2))
    got = torch.full((heads, hd + 2), float("nan"), device="cuda")
    step = torch.tensor([seq - 1, seq] + [0] * 6, dtype=torch.int32, device="cuda")
    api.set_decode_fold_mode(fold_mode)
    try:
        api.attn_decode_kv_shard(step, q, kc, vc, acc, ml, got, heads, n_kv, hd, seq + 3, scale, splits, selector=selector)
    finally:
        api.set_decode_fold_mode(0)
    assert api.check_device_status() == 0
    total, out = _triple(q, k, v, n_kv, scale)
    got = got.double()
    # (a sum is good to 1e-5, the bar of decode: 1.5e-5 of its logarithm; f32 holds a maximum of up to 32 to 4e-6)
    assert (got[:, hd] + got[:, hd + 1].log2() - total).abs().max() <= 2e-5
    assert _close(got[:, :hd] / got[:, hd + 1:], out)


def test_shards_of_different_bodies_fold_to_the_whole_cache():
    from hipml_b200 import api
    heads, n_kv, hd, scale = 24, 4, 256, 0.0625
    gen = torch.Generator(device="cuda").manual_seed(3)
    q = torch.randn(heads * hd, device="cuda", generator=gen)
    parts = [(0, 0, 700), (6, 0, 300), (8, 0, 900), (1, 1, 500), (7, 0, 20)]
    gathered = torch.full((len(parts), heads, hd + 2), float("nan"), device="cuda")
    keys, values = [], []
    for i, (selector, dtype, n) in enumerate(parts):
        kc, vc, (k, v) = _quantised_cache(gen, n, n, n_kv, dtype)
        keys.append(k)
        values.append(v)
        splits = api.decode_splits(n)
        acc, ml = (torch.full((heads * splits * m,), float("nan"), device="cuda") for m in (hd, 2))
        step = torch.tensor([n - 1, n] + [0] * 6, dtype=torch.int32, device="cuda")
        api.attn_decode_kv_shard(step, q, kc, vc, acc, ml, gathered[i], heads, n_kv, hd, n, scale, splits, selector=selector)
    out = torch.full((heads, hd), float("nan"), device="cuda")
    api.attn_decode_combine(gathered, out, heads, hd, len(parts))
    assert api.check_device_status() == 0
    assert _close(out, _triple(q, torch.cat(keys), torch.cat(values), n_kv, scale)[1])


@pytest.mark.parametrize("fold_mode", [0, 1], ids=["fold_inside", "fold_launch"])
def test_ranks_of_different_bodies_exchange_the_same_sums(fold_mode):
    """Each rank's workspace on this device, all publish, then all collect."""
    from hipml_b200 import api
    heads, n_kv, hd, scale, lens, selectors = 24, 4, 256, 0.0625, (700, 300), (0, 8)
    gen = torch.Generator(device="cuda").manual_seed(4)
    q = torch.randn(heads * hd, device="cuda", generator=gen)
    ws = [torch.zeros(api.decode_exchange_bytes(heads, hd, 2), dtype=torch.uint8, device="cuda") for _ in lens]
    ranks = [_quantised_cache(gen, n, n, n_kv, 0) for n in lens]
    outs = torch.full((2, heads, hd), float("nan"), device="cuda")
    api.set_decode_fold_mode(fold_mode)
    try:
        for phase in (1, 2):
            for r, (n, (kc, vc, _)) in enumerate(zip(lens, ranks)):
                splits = api.decode_splits(n)
                acc, ml = (torch.full((heads * splits * m,), float("nan"), device="cuda") for m in (hd, 2))
                step = torch.tensor([n - 1, n] + [0] * 6, dtype=torch.int32, device="cuda")
                api.attn_decode_kv_shard_exchange(step, q, kc, vc, acc, ml, outs[r], heads, n_kv, hd, n, scale, splits,
                                                  [w.data_ptr() for w in ws], r, phases=phase, wait_limit_us=1000,
                                                  selector=selectors[r])
    finally:
        api.set_decode_fold_mode(0)
    assert api.check_device_status() == 0
    want = _triple(q, *(torch.cat([c[2][i] for c in ranks]) for i in range(2)), n_kv, scale)[1]
    for out in outs:
        assert _close(out, want)


# an empty shard, one row, one run, several; a length past the cache, whose rows are followed by others that would be seen
@pytest.mark.parametrize("selector", [0, 1, 7, 8])
@pytest.mark.parametrize("seq,stride", [(0, 5), (1, 1), (300, 300), (4700, 4710), (340, 300)])
def test_a_shard_with_scratch_on_8_bytes_keeps_its_body(seq, stride, selector):
    from hipml_b200 import _lib, api
    heads, n_kv, hd, scale = 24, 4, 256, 0.0625
    gen = torch.Generator(device="cuda").manual_seed(seq)
    live = min(seq, stride)
    kc, vc, (k, v) = _quantised_cache(gen, live, stride, n_kv, int(selector == 1), room=512 * 272)
    q = torch.randn(heads * hd, device="cuda", generator=gen)
    splits = api.decode_splits(max(seq, 1))
    ml = torch.full((heads * splits * 2,), float("nan"), device="cuda")
    got = torch.full((heads, hd + 2), float("nan"), device="cuda")
    step = torch.tensor([seq - 1, seq] + [0] * 6, dtype=torch.int32, device="cuda")

    def shard(off, q):
        acc = torch.full((heads * splits * hd + 4,), float("nan"), device="cuda")[off:]
        api.attn_decode_kv_shard(step, q, kc, vc, acc, ml, got, heads, n_kv, hd, stride, scale, splits, selector=selector)

    shard(2, q)
    assert api.check_device_status() == 0
    if live:
        total, out = _triple(q, k, v, n_kv, scale)
        mine = got.double()
        assert (mine[:, hd] + mine[:, hd + 1].log2() - total).abs().max() <= 2e-5
        assert _close(mine[:, :hd] / mine[:, hd + 1:], out)
    else:
        assert (got[:, hd] == -math.inf).all() and (got[:, hd + 1] == 0).all() and (got[:, :hd] == 0).all()
    for off, query in ((1, q), (2, torch.randn(heads * hd + 1, device="cuda", generator=gen)[1:])):
        with pytest.raises(_lib.HipmlError, match="aligned"):
            shard(off, query)


# heads packed into one to four tiles of eight, full and not, columns across a tile's end; five and more columns a group
@pytest.mark.parametrize("group,n_kv,cols", [(1, 4, 8), (2, 4, 7), (3, 2, 8), (4, 4, 8), (5, 2, 6), (6, 4, 5), (7, 2, 4), (8, 4, 5)])
@pytest.mark.parametrize("pos0,bad", [(300, False), (4601, True), (9300, False)], ids=["short", "infinite_scales", "two_units"])
def test_columns_packed_into_tiles_give_each_columns_own_bits(group, n_kv, cols, pos0, bad):
    from hipml_b200 import api
    heads, hd, scale, stride = group * n_kv, 256, 0.0625, pos0 + cols + 2
    gen = torch.Generator(device="cuda").manual_seed(pos0 + 10 * group + cols)
    kc, vc = (torch.zeros(n_kv * stride * 272, dtype=torch.uint8, device="cuda") for _ in range(2))
    k, v = (torch.randn(pos0 + cols, n_kv * hd, device="cuda", generator=gen) for _ in range(2))
    if bad:
        v[pos0 + cols - 2:] = 1e9   # rows that only the last two columns see have an infinite scale
    api.kv_encode_bulk(k, v, kc, vc, n_kv, hd, stride, 0, 0, pos0 + cols)
    q = torch.randn(cols, heads * hd, device="cuda", generator=gen)
    splits = api.decode_splits(pos0 + cols)
    acc, ml = (torch.empty(cols * heads * splits * n, device="cuda") for n in (hd, 2))
    out = torch.full((cols, heads * hd), float("nan"), device="cuda")
    pos = torch.tensor([[pos0 + c, pos0 + c + 1] for c in range(cols)], dtype=torch.int32, device="cuda")
    api.attn_decode_cols(pos, q, kc, vc, acc, ml, out, heads, n_kv, hd, stride, scale, splits, cols,
                         heads * splits * hd, heads * splits * 2, heads * hd)
    assert torch.isfinite(out[:cols - 2] if bad else out).all()
    for c in range(cols):
        one = torch.empty(heads * hd, device="cuda")
        step = torch.tensor([pos0 + c, pos0 + c + 1] + [0] * 6, dtype=torch.int32, device="cuda")
        api.attn_decode_kv(step, q[c], kc, vc, acc, ml, one, heads, n_kv, hd, stride, scale, splits)
        assert torch.equal(one.nan_to_num(7.0), out[c].nan_to_num(7.0)), f"column {c}"
    assert api.check_device_status() == 0


# the last columns' rows in the first one's last unit, or in one of their own
@pytest.mark.parametrize("cols", [2, 4, 7])
@pytest.mark.parametrize("pos0", [0, 13, 29, 200, 1278, 4604, 9214])
@pytest.mark.parametrize("which", ["k", "v"])
def test_a_column_does_not_see_the_next_one_s_infinite_scale(pos0, cols, which):
    """A row whose values overflow f16 has infinite scales: what an earlier column does not see has no weight there,
    whatever it holds."""
    from hipml_b200 import api
    heads, n_kv, hd, scale, stride = 24, 4, 256, 0.0625, pos0 + cols + 2
    gen = torch.Generator(device="cuda").manual_seed(pos0 + cols)
    kc, vc = (torch.zeros(n_kv * stride * 272, dtype=torch.uint8, device="cuda") for _ in range(2))
    k, v = (torch.randn(pos0 + cols, n_kv * hd, device="cuda", generator=gen) for _ in range(2))
    (k if which == "k" else v)[pos0 + 1:] = 1e9   # f16 scale: infinity
    api.kv_encode_bulk(k, v, kc, vc, n_kv, hd, stride, 0, 0, pos0 + cols)
    q = torch.randn(cols, heads * hd, device="cuda", generator=gen)
    splits = api.decode_splits(pos0 + cols)
    acc, ml = (torch.empty(cols * heads * splits * n, device="cuda") for n in (hd, 2))
    out = torch.empty(cols, heads * hd, device="cuda")
    pos = torch.tensor([[pos0 + c, pos0 + c + 1] for c in range(cols)], dtype=torch.int32, device="cuda")
    api.attn_decode_cols(pos, q, kc, vc, acc, ml, out, heads, n_kv, hd, stride, scale, splits, cols,
                         heads * splits * hd, heads * splits * 2, heads * hd)
    assert torch.isfinite(out[0]).all()
    for c in range(cols):
        one = torch.empty(heads * hd, device="cuda")
        step = torch.tensor([pos0 + c, pos0 + c + 1] + [0] * 6, dtype=torch.int32, device="cuda")
        api.attn_decode_kv(step, q[c], kc, vc, acc, ml, one, heads, n_kv, hd, stride, scale, splits)
        assert torch.equal(one.nan_to_num(7.0), out[c].nan_to_num(7.0)), f"column {c}"
    assert api.check_device_status() == 0


def _attend(q, k, v, n_kv, hd, scale):
    """softmax(q k^T) v of one query row per head, 64 bits: q [heads * hd], k and v [rows, n_kv * hd]."""
    heads = q.numel() // hd
    q = q.double().view(n_kv, heads // n_kv, hd)
    k, v = (x.double().view(-1, n_kv, hd).transpose(0, 1) for x in (k, v))
    return (torch.softmax(q @ k.transpose(1, 2) * scale, dim=-1) @ v).reshape(-1)


def _close(got, want):
    """The bar of the decode tests: largest difference and relative 2-norm."""
    d = got.double() - want
    return bool(torch.isfinite(got).all()) and d.abs().max() <= 2e-5 and d.norm() <= 2e-5 * want.norm()


LAUNCHES = 24   # with scratch that would poison an output that read any of it too early, and a query each


# few splits keep their clusters of four or eight when the stream is longer than one cluster holds; at 128 pairs
@pytest.mark.parametrize("splits,seq", [(8, 600), (32, 2000), (64, 519), (64, 2500), (100, 2000), (128, 3000)])
@pytest.mark.parametrize("group", [1, 5, 6, 7, 8])
def test_no_launch_reads_partials_that_are_not_written_yet(group, splits, seq):
    """A head's runs meet in memory, slice by slice of its outputs: slices begin inside a head here."""
    from hipml_b200 import api
    n_kv, hd, scale = 4, 256, 0.0625
    heads = n_kv * group
    gen = torch.Generator(device="cuda").manual_seed(seq + group)
    k, v = (torch.randn(seq, n_kv * hd, device="cuda", generator=gen) for _ in range(2))
    kc, vc = (torch.zeros(n_kv * seq * 272, dtype=torch.uint8, device="cuda") for _ in range(2))
    api.kv_encode_bulk(k, v, kc, vc, n_kv, hd, seq, 0, 0, seq)
    kq, vq = (torch.from_numpy(cases.unpack_head_major(O.dequantize_q8(c.cpu().numpy().reshape(n_kv, seq, 272)), n_kv,
                                                       seq, hd)).cuda() for c in (kc, vc))
    acc, ml = (torch.empty(heads * splits * n, device="cuda") for n in (hd, 2))
    q = torch.randn(LAUNCHES, heads * hd, device="cuda", generator=gen)
    out = torch.full((LAUNCHES, heads * hd), float("nan"), device="cuda")
    step = torch.tensor([seq - 1, seq] + [0] * 6, dtype=torch.int32, device="cuda")
    for i in range(LAUNCHES):
        acc.fill_(float("nan"))
        ml.fill_(float("nan"))
        api.attn_decode_kv(step, q[i], kc, vc, acc, ml, out[i], heads, n_kv, hd, seq, scale, splits)
    assert api.check_device_status() == 0
    for i in range(LAUNCHES):
        assert _close(out[i], _attend(q[i], kq, vq, n_kv, hd, scale)), f"launch {i}"


@pytest.mark.parametrize("splits,pos0", [(32, 2000), (64, 2500), (100, 2000), (128, 3000)])
@pytest.mark.parametrize("group", [5, 6, 7])
def test_no_launch_of_columns_reads_partials_that_are_not_written_yet(group, splits, pos0):
    from hipml_b200 import api
    n_kv, hd, scale, cols = 4, 256, 0.0625, 4
    heads, seq = n_kv * group, pos0 + cols
    gen = torch.Generator(device="cuda").manual_seed(pos0 + group)
    k, v = (torch.randn(seq, n_kv * hd, device="cuda", generator=gen) for _ in range(2))
    kc, vc = (torch.zeros(n_kv * seq * 272, dtype=torch.uint8, device="cuda") for _ in range(2))
    api.kv_encode_bulk(k, v, kc, vc, n_kv, hd, seq, 0, 0, seq)
    kq, vq = (torch.from_numpy(cases.unpack_head_major(O.dequantize_q8(c.cpu().numpy().reshape(n_kv, seq, 272)), n_kv,
                                                       seq, hd)).cuda() for c in (kc, vc))
    acc, ml = (torch.empty(cols * heads * splits * n, device="cuda") for n in (hd, 2))
    q = torch.randn(LAUNCHES, cols, heads * hd, device="cuda", generator=gen)
    out = torch.full((LAUNCHES, cols, heads * hd), float("nan"), device="cuda")
    pos = torch.tensor([[pos0 + c, pos0 + c + 1] for c in range(cols)], dtype=torch.int32, device="cuda")
    for i in range(LAUNCHES):
        acc.fill_(float("nan"))
        ml.fill_(float("nan"))
        api.attn_decode_cols(pos, q[i], kc, vc, acc, ml, out[i], heads, n_kv, hd, seq, scale, splits, cols,
                             heads * splits * hd, heads * splits * 2, heads * hd)
    assert api.check_device_status() == 0
    for i in range(LAUNCHES):
        for c in range(cols):
            n = pos0 + c + 1
            assert _close(out[i, c], _attend(q[i, c], kq[:n], vq[:n], n_kv, hd, scale)), f"launch {i}, column {c}"


@pytest.mark.parametrize("group", [1, 3, 5, 6, 7, 8])
@pytest.mark.parametrize("n_ctx,pos0,rows", [(300, 298, 1), (600, 590, 2), (2100, 2047, 1), (2100, 2092, 8)])
def test_no_launch_over_the_f32_cache_reads_partials_that_are_not_written_yet(group, n_ctx, pos0, rows):
    from hipml_b200 import api
    n_kv, hd = 4, 256
    heads, seq = n_kv * group, pos0 + rows
    gen = torch.Generator(device="cuda").manual_seed(n_ctx + group)
    k, v = (torch.randn(n_ctx, n_kv * hd, device="cuda", generator=gen) for _ in range(2))
    splits = api.cols_splits(n_ctx)
    acc, ml = (torch.empty(rows * heads * splits * n, device="cuda") for n in (hd, 2))
    q = torch.randn(LAUNCHES, rows, heads * hd, device="cuda", generator=gen)
    out = torch.full((LAUNCHES, rows, heads * hd), float("nan"), device="cuda")
    for i in range(LAUNCHES):
        acc.fill_(float("nan"))
        ml.fill_(float("nan"))
        api.attn_decode_cols_f32(q[i], k, v, acc, ml, out[i], heads, n_kv, hd, n_ctx, pos0, rows)
    assert api.check_device_status() == 0
    for i in range(LAUNCHES):
        for c in range(rows):
            n = pos0 + c + 1
            assert _close(out[i, c], _attend(q[i, c], k[:n], v[:n], n_kv, hd, 0.0625)), f"launch {i}, column {c}"


# floats by which part_acc, part_ml and their slots are off the alignment that the fold inside the kernel wants
@pytest.mark.parametrize("acc_off,ml_off,acc_odd,ml_odd", [(0, 1, 0, 0), (0, 0, 0, 1), (0, 1, 0, 1), (1, 0, 3, 0), (3, 1, 1, 1)])
@pytest.mark.parametrize("entry", ["rows q8_0", "rows q4_0", "batch append q8_0", "one slot", "columns"])
def test_scratch_of_several_slots_may_lie_on_any_float(entry, acc_off, ml_off, acc_odd, ml_odd):
    from hipml_b200 import api
    heads, n_kv, hd, scale = 24, 4, 256, 0.0625
    dtype = 1 if "q4" in entry else 0
    row, deq = ((272, O.dequantize_q8), (144, O.dequantize_q4))[dtype]
    lens = [700] if entry == "one slot" else [300, 301, 302] if entry == "columns" else [1, 700, 333]
    slots, stride = len(lens), 704
    caches = 1 if entry == "columns" else slots
    gen = torch.Generator(device="cuda").manual_seed(acc_off + 8 * ml_off + 64 * acc_odd)
    k, v = (torch.randn(caches, max(lens), n_kv * hd, device="cuda", generator=gen) for _ in range(2))
    kc, vc = (torch.zeros(caches, n_kv * stride * row, dtype=torch.uint8, device="cuda") for _ in range(2))
    for s in range(caches):
        api.kv_encode_bulk(k[s], v[s], kc[s], vc[s], n_kv, hd, stride, 0, 0, max(lens), dtype)
    kq, vq = (torch.from_numpy(np.stack([cases.unpack_head_major(deq(c[s].cpu().numpy().reshape(n_kv, stride, row)), n_kv,
                                                                 stride, hd) for s in range(caches)])).cuda() for c in (kc, vc))
    splits = 6
    acc_slot, ml_slot = heads * splits * hd + acc_odd, heads * splits * 2 + ml_odd
    acc = torch.full((slots * acc_slot + 4,), float("nan"), device="cuda")[acc_off:]
    ml = torch.full((slots * ml_slot + 4,), float("nan"), device="cuda")[ml_off:]
    q = torch.randn(slots, heads * hd, device="cuda", generator=gen)
    out = torch.full((slots, heads * hd), float("nan"), device="cuda")
    pos = torch.tensor([[n - 1, n] for n in lens], dtype=torch.int32, device="cuda")
    tail = (splits, n_kv * stride * row, acc_slot, ml_slot, heads * hd, slots)
    if entry == "columns":
        api.attn_decode_cols(pos, q, kc, vc, acc, ml, out, heads, n_kv, hd, stride, scale, splits, slots, acc_slot, ml_slot,
                             heads * hd)
    elif entry == "one slot":
        api.attn_decode_batch(pos, q, kc, vc, acc, ml, out, heads, n_kv, hd, stride, scale, *tail, lens[0])
    elif entry == "batch append q8_0":
        new = [torch.stack([x[s, n - 1] for s, n in enumerate(lens)]).contiguous() for x in (k, v)]
        api.attn_decode_batch_append(pos, new[0], new[1], q, kc, vc, acc, ml, out, heads, n_kv, hd, stride, scale, *tail)
    else:
        api.attn_decode_rows(pos, q, kc, vc, acc, ml, out, heads, n_kv, hd, stride, scale, *tail, dtype=dtype)
    assert api.check_device_status() == 0
    for s, n in enumerate(lens):
        c = 0 if entry == "columns" else s
        assert _close(out[s], _attend(q[s], kq[c, :n], vq[c, :n], n_kv, hd, scale)), f"slot {s}"


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
    for _ in range(2):   # (the second finds the first one's counters, and scratch that was never written)
        acc.fill_(float("nan"))
        ml.fill_(float("nan"))
        out.fill_(float("nan"))
        api.attn_decode_cols_f32(q, k, v, acc, ml, out, heads, n_kv, hd, n_ctx, pos0, rows)
    kn, vn, qn = k.cpu().numpy(), v.cpu().numpy(), q.cpu().numpy()
    for c in range(rows):
        seq = pos0 + c + 1
        want = O.attn_causal_f32(qn[c], kn[:seq], vn[:seq], heads, n_kv, hd, seq, 0.0625)
        assert O.max_abs(want, out[c].cpu().numpy()) <= 5e-6 and O.rel_l2(want, out[c].cpu().numpy()) <= 5e-6
