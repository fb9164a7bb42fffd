"""Prompt attention on the tensor cores (csrc/seq/seq_attn_tc.cu) against float64 at the sizes where it can go wrong: head sizes that are not a
power of two and differ between keys and values, row tiles that end inside a token's heads, several entries behind their own pasts, key tiles
that end inside a page, windows, chunks, kept first positions, soft caps, sinks, negative head scales, gates, key splits.

Bound: operands enter as 24-bit splits, products are summed by the tensor core in f32 over at most 128 terms (its truncation: 2^-23 of the sum
a step, 8 steps) and the value tiles by f32 adds; the f32 tiles it stands beside are tested at 2e-5 of the largest value, this one at 4e-6."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from blazr_b200 import seqops
    seqops.lib()
    return seqops


CASES = [
    # (tokens, past) per entry, H, G, D, V, options
    ([(17, 0)], 4, 4, 16, 16, {}),                                  # few tokens with few keys: the f32 tiles
    ([(64, 64)], 4, 2, 32, 32, {}),                                 # the last such step, and the first ones beside it
    ([(64, 65)], 4, 2, 32, 32, {}),
    ([(65, 0)], 4, 4, 16, 16, {}),
    ([(66, 0)], 300, 2, 32, 32, {}),
    ([(64, 0), (33, 100)], 8, 2, 64, 64, dict(chunk=48)),
    ([(130, 5)], 6, 2, 48, 80, dict(window=37)),
    ([(40, 300), (1, 64), (20, 0)], 8, 1, 128, 128, dict(window=64, keep_first=3)),
    ([(200, 0)], 3, 3, 96, 32, dict(softcap=5.0)),
    ([(70, 10)], 10, 2, 64, 48, dict(sink=True, head_scale=True)),
    ([(129, 63)], 4, 2, 112, 64, dict(gated=True, gate_elem=True)),
    ([(300, 0)], 64, 8, 64, 64, dict(gated=True, chunk=128)),       # two row tiles per CTA
    ([(1300, 0)], 32, 8, 64, 64, dict(window=200)),
    ([(20, 1500)], 2, 1, 64, 64, dict(split=True)),
    ([(18, 2000)], 4, 1, 128, 128, dict(split=True, sink=True, gated=True)),
    ([(50, 0)], 300, 2, 32, 32, {}),                                # more heads of one key head than a tile has rows
    ([(100, 0)], 300, 2, 32, 32, {}),
    # the same forms with enough keys for this kernel to be the one chosen (tc_is_faster)
    ([(130, 5)], 6, 2, 48, 80, dict(window=100)),
    ([(40, 300), (1, 64), (20, 0), (50, 7)], 8, 1, 128, 128, dict(window=128, keep_first=3)),
    ([(20, 1500)], 16, 4, 64, 64, dict(split=True)),
    ([(18, 2000)], 32, 4, 128, 128, dict(split=True, sink=True, gated=True)),
]


def attend(ops, entries, H, G, D, V, o, odt, plant=None):
    """(outputs, float64 reference): a query row meets the keys it sees and no others.  plant(rows, kp, vp, slot) changes the inputs first; slot(entry,
    position) is a position's row in the pools"""
    from blazr_b200.batch import StepEntry, build_step
    bs, gen = 16, torch.Generator().manual_seed(H * D + V)
    rnd = lambda *s: torch.randn(*s, generator=gen)
    need = [-(-(n + p) // bs) for n, p in entries]
    perm = torch.randperm(sum(need), generator=gen).tolist()
    tables, at = [], 0
    for n in need:
        tables.append(perm[at:at + n])
        at += n
    sa = build_step([StepEntry([0] * n, p, i, tables[i]) for i, (n, p) in enumerate(entries)], bs)
    t = {k: torch.from_numpy(np.ascontiguousarray(getattr(sa, k))).to(DEV) for k in ("tok_ent", "tok_pos", "ent_start", "ent_slot", "ent_pos0", "block_table")}
    st = ops.StepDesc(t["tok_ent"].data_ptr(), t["tok_pos"].data_ptr(), t["ent_start"].data_ptr(), t["ent_slot"].data_ptr(), t["ent_pos0"].data_ptr(),
                      t["block_table"].data_ptr(), sa.T, sa.B, sa.block_table.shape[1], bs)
    gated, elem = o.get("gated", False), o.get("gate_elem", False)
    sink = rnd(H) if o.get("sink") else None
    hs = rnd(H) if o.get("head_scale") else None
    desc = ops.attn_desc(H, G, D, V, 2.0 * D ** -0.5, gated=gated, chunk=o.get("chunk", 0), window=o.get("window", 0), keep_first=o.get("keep_first", 0),
                         softcap=o.get("softcap", 0.0), sink=sink.to(DEV) if sink is not None else None, head_scale=hs.to(DEV) if hs is not None else None, gate_elem=elem)
    keep = (desc, sink, hs)
    sink_d, hs_d = (x.to(DEV) if x is not None else None for x in (sink, hs))
    desc.sink, desc.head_scale = (x.data_ptr() if x is not None else None for x in (sink_d, hs_d))
    width = -(-desc.width // 4) * 4
    rows = rnd(sa.T, width)
    kp, vp = rnd(sum(need) * bs, G, D), rnd(sum(need) * bs, G, V)
    kp[tables[0][-1] * bs + bs - 1] = float("nan") if (entries[0][0] + entries[0][1]) % bs else kp[tables[0][-1] * bs + bs - 1]   # a slot no position uses
    if plant is not None:
        plant(rows, kp, vp, lambda e, pos: tables[e][pos // bs] * bs + pos % bs)
    ref = torch.zeros(sa.T, H, V, dtype=torch.float64)
    r0 = 0
    for (n, past), tab in zip(entries, tables):
        slots = (torch.tensor(tab)[:, None] * bs + torch.arange(bs)).reshape(-1)[:n + past]
        q, k, v = rows[r0:r0 + n, :H * D].double().reshape(n, H, D), kp[slots].double(), vp[slots].double()
        qp, kpos = torch.arange(past, past + n)[:, None], torch.arange(n + past)[None]
        see = kpos <= qp
        if o.get("chunk"):
            see = see & (kpos // o["chunk"] == qp // o["chunk"])
        if o.get("window"):
            see = see & ((qp - kpos < o["window"]) | (kpos < o.get("keep_first", 0)))
        for h in range(H):
            s = (q[:, h] @ k[:, h // (H // G)].T) * 2.0 * D ** -0.5 * (hs[h].double() if hs is not None else 1.0)
            if o.get("softcap"):
                s = o["softcap"] * torch.tanh(s / o["softcap"])
            s = s.masked_fill(~see, float("-inf"))
            if sink is not None:
                s = torch.cat([s, sink[h].double().expand(n, 1)], 1)
            p = torch.softmax(s, 1)[:, :n + past]
            if plant is None:
                ref[r0:r0 + n, h] = p @ v[:, h // (H // G)]
            else:                                                   # (0 x inf: keys that are not seen stay out of the sum)
                ref[r0:r0 + n, h] = (p[:, :, None] * v[None, :, h // (H // G)]).masked_fill(~see[:, :, None] | (s[:, :n + past, None] == float("-inf")), 0.0).sum(1)
        if gated:
            gl = rows[r0:r0 + n, desc.gate_col:].double()
            ref[r0:r0 + n] *= torch.sigmoid(gl[:, :H * V].reshape(n, H, V) if elem else gl[:, :H, None])
        r0 += n
    out = torch.full((sa.T + 1, H * V), 3.0, device=DEV, dtype=odt)
    scratch = torch.empty(1 << 22, device=DEV) if o.get("split") else None
    ops.attn_ex(rows.to(DEV), st, desc, kp.to(DEV), vp.to(DEV), out[:sa.T], scratch)
    assert bool((out[sa.T] == 3.0).all()) and ops.error_flags() == 0 and keep is not None
    return out[:sa.T].double().cpu(), ref.reshape(sa.T, -1)


@pytest.mark.parametrize("entries,H,G,D,V,o", CASES)
@pytest.mark.parametrize("odt", [torch.float32, torch.bfloat16])
def test_against_float64(ops, entries, H, G, D, V, o, odt):
    out, ref = attend(ops, entries, H, G, D, V, o, odt)
    err = (out - ref).abs().max().item() / ref.abs().max().item()
    assert err < (4e-6 if odt == torch.float32 else 2 ** -8), err


@pytest.mark.parametrize("H,G,D", [(16, 4, 64), (8, 1, 128)])
@pytest.mark.parametrize("B,extra", [(17, 0), (40, 0), (65, 0), (24, 70)])
@pytest.mark.parametrize("split", [False, True])
def test_many_entries_of_one_token(ops, H, G, D, B, extra, split):
    """Batched decoding: every entry has a tile of its own, some beside a longer portion of another sequence."""
    entries = [(1, (37 * i) % 300) for i in range(B)] + ([(extra, 11)] if extra else [])
    out, ref = attend(ops, entries, H, G, D, D, dict(split=split), torch.float32)
    assert (out - ref).abs().max().item() / ref.abs().max().item() < 4e-6


INF, NAN = float("inf"), float("nan")
PLANTS = {
    # what is planted at position 70 of the first entry (key head 1, column 3): values, keys, the query of that position
    "value inf": lambda rows, kp, vp, at, w: vp.__setitem__((at, 1, 3), INF),
    "value -inf": lambda rows, kp, vp, at, w: vp.__setitem__((at, 1, 3), -INF),
    "value nan": lambda rows, kp, vp, at, w: vp.__setitem__((at, 1, 3), NAN),
    "value 3.4e38": lambda rows, kp, vp, at, w: vp.__setitem__((at, 1, 3), 3.4e38),
    "key -inf": lambda rows, kp, vp, at, w: kp.__setitem__((at, 1, 3), -INF),
    "key 3.4e38": lambda rows, kp, vp, at, w: (kp.__setitem__((at, 1, 3), 3.4e38), rows[:, 3::16].mul_(1e-37)),
    "key nan": lambda rows, kp, vp, at, w: kp.__setitem__((at, 1, 3), NAN),
    "query inf": lambda rows, kp, vp, at, w: rows.__setitem__((70, w), INF),
}


@pytest.mark.parametrize("what", sorted(PLANTS))
@pytest.mark.parametrize("H,G,D,V,o", [(8, 2, 64, 64, {}), (4, 2, 128, 128, dict(window=100)), (64, 2, 32, 48, dict(softcap=5.0)), (64, 8, 16, 16, dict(tokens=600)), (6, 2, 64, 64, dict(split=True, sink=True, gated=True))])
def test_values_that_are_not_finite(ops, what, H, G, D, V, o):
    """They reach the rows that see them, as infinities or NaN where plain f32 sums give those, and no other row."""
    R = H // G
    out, ref = attend(ops, [(150, 700)] if o.get("split") else [(o.get("tokens", 150), 0), (90, 20)], H, G, D, V, o, torch.float32,
                      lambda rows, kp, vp, slot: PLANTS[what](rows, kp, vp, slot(0, 70), R * D + 3))
    ref32 = ref.float().double()                                    # a sum beyond the f32 range is infinite
    fine = torch.isfinite(ref32)
    assert fine.any() and ("key -inf" in what or "3.4e38" in what or (what == "query inf" and o.get("softcap")) or not fine.all())
    seen_big = (out - ref).abs() > 1e30                             # (near the range's end a sum may overflow on the way)
    assert bool(((torch.isnan(out) == torch.isnan(ref32)) | seen_big).all()) and bool(((torch.isposinf(out) == torch.isposinf(ref32)) | seen_big).all())
    ok = fine & (ref32.abs() < 1e30)
    assert ((out - ref)[ok].abs().max() / ref[ok].abs().max()).item() < 4e-6


def test_more_tokens_than_a_grid_has_rows(ops):
    """128 query heads of one key head: a tile holds one token, and a step has more tiles than the second dimension of a grid."""
    T, H, D, bs = 65600, 128, 16, 16
    g = torch.Generator(device=DEV)
    g.manual_seed(5)
    rows = torch.randn(T, H * D + 2 * D, device=DEV, generator=g)
    kp, vp = (torch.randn(T, 1, D, device=DEV, generator=g) for _ in range(2))
    i32 = dict(dtype=torch.int32, device=DEV)
    t = [torch.zeros(T, **i32), torch.arange(T, **i32), torch.tensor([0, T], **i32), torch.zeros(1, **i32), torch.zeros(1, **i32), torch.arange(T // bs, **i32)[None].contiguous()]
    st = ops.StepDesc(*(x.data_ptr() for x in t), T, 1, T // bs, bs)
    desc = ops.attn_desc(H, 1, D, D, D ** -0.5, gated=False, window=8)
    out = torch.empty(T, H * D, device=DEV)
    ops.attn_ex(rows, st, desc, kp, vp, out, None)
    for p in (0, 7, 40000, 65535, 65599):
        lo = max(0, p - 7)
        s = rows[p, :H * D].double().reshape(H, D) @ kp[lo:p + 1, 0].double().T * D ** -0.5
        want = torch.softmax(s, 1) @ vp[lo:p + 1, 0].double()
        assert ((out[p].double() - want.reshape(-1)).abs().max() / want.abs().max()).item() < 4e-6
    assert ops.error_flags() == 0
