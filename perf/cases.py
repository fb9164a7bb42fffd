"""The work that users of this framework have it do, as cases that can be timed and checked one by one.

Two libraries do the work: libb200q (quantized linear layers and the llama / mistral decoder around them) and libb200seq (the operators of
layer-list models).  A case is one call, or one short sequence of calls, of the public Python entry points over them, at sizes taken from the
repository's presets (blazr_b200/decode.py), its layered sizes (blazr_b200/layered_bench.py) and its benchmark.  `listed` names twelve,
`draw` gives others of the same ranges, `exact` restates each in 64 bits in plain torch.
"""
import math

import numpy as np
import torch

from blazr_b200 import decode, ops, seqops

DEV = "cuda:0"
GGML = {"Q4_K": 12, "Q6_K": 14, "Q8_0": 8}
BLOCK = {"Q4_K": (256, 144), "Q6_K": (256, 210), "Q8_0": (32, 34)}          # weights, bytes of one block
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
# (N, K) of the projections of the presets: q|k|v, o, gate or up, gate|up, down
SHAPES = {"llama-3.2-1b": (2048, 8192, 512), "mistral-7b": (4096, 14336, 1024), "llama-3-70b": (8192, 28672, 1024)}


def listed():
    return [
        # one token through an attention output projection: the smallest call of a decode step
        dict(name="o_q4k_1_token", kind="qmm", fmt="Q4_K", N=4096, K=4096, M=1, dtype="f32"),
        # one token through the widest projection of an 8B model, AWQ weights and 16-bit activations
        dict(name="gate_up_awq_1_token", kind="qmm", fmt="AWQ", N=28672, K=4096, M=1, dtype="f16"),
        # batched decode: 32 sequences, one token each
        dict(name="gate_q6k_32_tokens", kind="qmm", fmt="Q6_K", N=14336, K=4096, M=32, dtype="f32"),
        # a 2048-token prompt through an up projection
        dict(name="gate_q6k_2048_tokens", kind="qmm", fmt="Q6_K", N=14336, K=4096, M=2048, dtype="f32"),
        # a prompt of odd length through the fused q|k|v projection
        dict(name="qkv_awq_1531_tokens", kind="qmm", fmt="AWQ", N=6144, K=4096, M=1531, dtype="f16"),
        # mixture-of-experts MLP of a decode step: 2 tokens, 6 of 64 experts each and two shared halves, as in the benchmark
        dict(name="experts_q4k_2_tokens", kind="qmoe", T=2, E=66, top=8, hidden=2048, ffn=1408, fmt="Q4_K", fmt_down="Q8_0"),
        # greedy generation as a program calls it: 48 positions, one by one, replayed from the captured step
        dict(name="generate_48_positions", kind="generate", S=48),
        # a 2048-token prompt through a whole decoder: last logits and the keys and values it leaves in the cache
        dict(name="prompt_2048_tokens", kind="prompt", S=2048),
        # dense feed-forward of a layer-list model over a 4096-token prompt (gate|up with the activation, then down)
        dict(name="feed_forward_4096_tokens", kind="ff", T=4096, W=2048, F=8192),
        # attention of a layer-list model over a 4096-token prompt, keys of the token's own chunk
        dict(name="attention_4096_tokens", kind="attn", T=4096, B=1, past=0, H=32, G=8, D=64, chunk=2048, window=0),
        # routed experts of a layer-list model over a 4096-token prompt
        dict(name="experts_4096_tokens", kind="moe", T=4096, W=1024, F=1024, E=32, top=4),
        # state-space recurrence of a layer-list model over a 4096-token prompt
        dict(name="state_space_4096_tokens", kind="ssm", T=4096, H=64, V=64, N=128, G=8),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["qmm", "qmm", "qmm", "qmm", "qmoe", "prompt", "generate", "ff", "ff", "attn", "attn", "moe", "ssm"])
    if kind == "qmm":
        h, f, kv = SHAPES[rng.choice(["llama-3.2-1b", "mistral-7b", "mistral-7b", "llama-3-70b"])]
        N, K = rng.choice([(h + 2 * kv, h), (h, h), (f, h), (2 * f, h), (h, f)])
        most = max(8, min(2048, int(2.4e11 / (2.0 * N * K))))               # no more than the largest listed one
        M = rng.choice([1, _log(rng, 1, 4), _log(rng, 5, min(128, most)), _log(rng, min(129, most), most)])
        return dict(kind=kind, fmt=rng.choice(["Q4_K", "Q6_K", "Q8_0", "AWQ", "GPTQ"]), N=N, K=K, M=M, dtype=rng.choice(["f32", "f16", "bf16"]))
    if kind == "qmoe":
        return dict(kind=kind, T=rng.randint(1, 8), E=66, top=rng.choice([2, 4, 6, 8]), hidden=2048, ffn=rng.choice([768, 1024, 1408]), fmt=rng.choice(["Q4_K", "Q6_K"]),
                    fmt_down="Q8_0")
    if kind == "generate":
        return dict(kind=kind, S=_log(rng, 4, 48))
    if kind == "prompt":
        return dict(kind=kind, S=_log(rng, 8, 2048))
    W, F = rng.choice([(1024, 4096), (2048, 8192)])
    if kind == "ff":
        return dict(kind=kind, T=_log(rng, 1, 4096), W=W, F=F)
    if kind == "attn":
        H, G, D = rng.choice([(16, 4, 64), (32, 8, 64), (32, 8, 128)])
        chunk, window = rng.choice([(1024, 0), (2048, 0), (0, 1024), (0, 2048), (0, 0)])
        if rng.random() < 0.4:                                               # a decode step: one token of each sequence behind its own past
            return dict(kind=kind, T=1, B=rng.randint(1, 4), past=_log(rng, 64, 4000), H=H, G=G, D=D, chunk=chunk, window=window)
        return dict(kind=kind, T=_log(rng, 64, 4096 if D == 64 and chunk + window > 0 else 2048), B=1, past=0, H=H, G=G, D=D, chunk=chunk, window=window)
    if kind == "moe":
        return dict(kind=kind, T=_log(rng, 1, 4096), W=1024, F=rng.choice([512, 1024]), E=32, top=rng.choice([2, 4]))
    H, N, G = rng.choice([(32, 64, 2), (64, 128, 8)])
    return dict(kind=kind, T=_log(rng, 1, 4096), H=H, V=64, N=N, G=G)


# ---- inputs -----------------------------------------------------------------------------------------------------------------------
def _gen(seed, more=0):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + more) & 0x7FFFFFFF)
    return g


def _rand_blocks(fmt, N, K, g):
    """raw ggml blocks of an [N, K] weight of unit-gain rows: uniform payload, scales spread by a factor of three"""
    be, bb = BLOCK[fmt]
    nb = N * (K // be)
    blk = torch.randint(0, 256, (nb, bb), dtype=torch.uint8, device=DEV, generator=g)
    std = {"Q4_K": 259.2, "Q6_K": 1363.9, "Q8_0": 74.0}[fmt]                # of a weight at scale 1 with such a payload
    d = ((torch.rand(nb, device=DEV, generator=g) + 0.5) / (std * math.sqrt(K))).half()
    at = 208 if fmt == "Q6_K" else 0
    blk[:, at:at + 2] = d.view(torch.uint8).reshape(nb, 2)
    if fmt == "Q4_K":
        blk[:, 2:4] = (d.float() * 7.5).half().view(torch.uint8).reshape(nb, 2)
    return blk.reshape(N, K // be * bb)


def _rand_int4(fmt, N, K, g):
    """AWQ / GPTQ tensors of group size 128, as the loaders hand them over"""
    u32 = lambda *s: torch.randint(-2 ** 31, 2 ** 31, s, dtype=torch.int32, device=DEV, generator=g)
    sc = ((torch.rand((K // 128, N), device=DEV, generator=g) + 0.5) / (4.6 * math.sqrt(K))).half().float()
    if fmt == "AWQ":
        return u32(K, N // 8), sc, torch.randint(0, 16, (K // 128, N), device=DEV, generator=g).float()
    return u32(K // 8, N), sc, u32(K // 128, N // 8)


def _packed(fmt, N, K, g):
    return (_rand_blocks(fmt, N, K, g),) if fmt in GGML else _rand_int4(fmt, N, K, g)


def _upload(client, fmt, N, K, packed):
    if fmt in GGML:
        return client.weight_from_ggml(GGML[fmt], packed[0], N, K)
    return client.weight_from_decomposed(ops.DecomposedQuantTensor(*packed, None, ops.DecomposedQuantMethod(fmt.lower(), 128), (N, K)))


SMALL = decode.ModelConfig("small-1b", 2048, 4, 32, 8, 64, 8192, 16384, 500000.0)   # decode.PRESETS["small-1b"]


def _model_parts(seed):
    """packed weights of the small decoder, Q4_K with the Q6_K parts of the Q4_K_M mix, and its f16 embedding and f32 norms"""
    c, g = SMALL, _gen(seed, 1)
    qd, kvd = c.n_heads * c.head_dim, c.n_kv_heads * c.head_dim
    shapes = dict(q=(qd, c.hidden), k=(kvd, c.hidden), v=(kvd, c.hidden), o=(c.hidden, qd), gate=(c.ffn, c.hidden), up=(c.ffn, c.hidden), down=(c.hidden, c.ffn))
    layers = []
    for i in range(c.n_layers):
        more = "Q6_K" if i % 2 == 0 else "Q4_K"
        lay = {p: (more if p in ("v", "down") else "Q4_K", N, K) for p, (N, K) in shapes.items()}
        lay = {p: (f, N, K, _rand_blocks(f, N, K, g)) for p, (f, N, K) in lay.items()}
        for n in ("attn_norm", "mlp_norm"):
            lay[n] = 1.0 + 0.1 * torch.randn(c.hidden, device=DEV, generator=g)
        layers.append(lay)
    return dict(layers=layers, embed=torch.randn((c.vocab, c.hidden), device=DEV, generator=g).half(), final=1.0 + 0.1 * torch.randn(c.hidden, device=DEV, generator=g),
                head=("Q6_K", c.vocab, c.hidden, _rand_blocks("Q6_K", c.vocab, c.hidden, g)))


def _decoder(seed, max_ctx):
    parts = _model_parts(seed)
    lin = lambda t: decode.HostLinear(t[0], t[1], t[2], t[3].cpu().numpy())
    hm = decode.HostModel(SMALL, "Q4_K_M", embed=parts["embed"].cpu().numpy())
    for lay in parts["layers"]:
        hm.layers.append({p: (v.cpu().numpy() if p.endswith("norm") else lin(v)) for p, v in lay.items()})
    hm.final_norm, hm.lm_head = parts["final"].cpu().numpy(), lin(parts["head"])
    return decode.Decoder(ops.B200Client(0), SMALL, "Q4_K_M", batch=1, max_ctx=max_ctx, host=hm)


def _prompt(case, seed):
    return torch.randint(0, SMALL.vocab, (case["S"],), device=DEV, generator=_gen(seed, 2)).cpu().numpy().astype(np.int64)


def _ff_inputs(c, seed):
    g = _gen(seed)
    x = torch.randn((c["T"], c["W"]), device=DEV, generator=g).bfloat16()
    gu = (torch.randn((2 * c["F"], c["W"]), device=DEV, generator=g) / math.sqrt(c["W"])).bfloat16()     # rows alternate gate, up
    dn = (torch.randn((c["W"], c["F"]), device=DEV, generator=g) / math.sqrt(c["F"])).bfloat16()
    return x, gu, dn


def _attn_inputs(c, seed):
    """projection rows q | k | v | gate of the step's tokens, and the pools with every sequence's past in scattered pages of 16"""
    g = _gen(seed)
    H, G, D, B, T, past = c["H"], c["G"], c["D"], c["B"], c["T"], c["past"]
    width = H * D + 2 * G * D + H
    rows = torch.randn((B * T, width), device=DEV, generator=g)
    pages = -(-(past + T) // 16)
    table = torch.randperm(B * pages, device=DEV, generator=g).to(torch.int32).reshape(B, pages)
    unit = lambda t: t / torch.sqrt((t * t).mean(-1, keepdim=True) + 1e-5)
    kpool = unit(torch.randn((B * pages * 16, G, D), device=DEV, generator=g))
    vpool = torch.randn((B * pages * 16, G, D), device=DEV, generator=g)
    return rows, table, kpool, vpool


def _moe_inputs(c, seed):
    g = _gen(seed)
    E, W, F = c["E"], c["W"], c["F"]
    x = torch.randn((c["T"], W), device=DEV, generator=g).bfloat16()
    gu = (torch.randn((E, 2 * F, W), device=DEV, generator=g) / math.sqrt(W)).bfloat16()                 # rows alternate gate, up
    dn = (torch.randn((E, W, F), device=DEV, generator=g) / math.sqrt(F)).bfloat16()
    z = torch.randn((c["T"], E), device=DEV, generator=g)
    return x, gu, dn, z


def _ssm_inputs(c, seed):
    """the in-projection's rows z | x | B | C | dt and, after convolution and silu, x | B | C; decays from slow to fast"""
    g = _gen(seed)
    H, V, N, G, T = c["H"], c["V"], c["N"], c["G"], c["T"]
    proj = torch.randn((T, 2 * H * V + 2 * G * N + H), device=DEV, generator=g)
    xbc = torch.nn.functional.silu(torch.randn((T, H * V + 2 * G * N), device=DEV, generator=g))
    A_log = 0.7 * torch.randn(H, device=DEV, generator=g)
    Dp = torch.randn(H, device=DEV, generator=g)
    dtb = torch.randn(H, device=DEV, generator=g) - 2.0
    return proj, xbc, A_log, Dp, dtb


def _step(T, B, past, table):
    """int32 arrays of a step of B sequences that bring T tokens each behind `past` earlier ones"""
    i32 = dict(dtype=torch.int32, device=DEV)
    t = dict(ent=torch.arange(B, **i32).repeat_interleave(T), pos=torch.arange(past, past + T, **i32).repeat(B), start=torch.arange(0, B * T + 1, T, **i32),
             slot=torch.arange(B, **i32), pos0=torch.full((B,), past, **i32), bt=table)
    d = seqops.StepDesc(t["ent"].data_ptr(), t["pos"].data_ptr(), t["start"].data_ptr(), t["slot"].data_ptr(), t["pos0"].data_ptr(), table.data_ptr(), B * T, B, table.shape[1], 16)
    return d, t


def prepare(case, seed):
    c = case
    k = c["kind"]
    f32 = dict(dtype=torch.float32, device=DEV)
    i32 = dict(dtype=torch.int32, device=DEV)
    if k == "qmm":
        client, g = ops.B200Client(0), _gen(seed)
        w = _upload(client, c["fmt"], c["N"], c["K"], _packed(c["fmt"], c["N"], c["K"], g))
        x = torch.randn((c["M"], c["K"]), device=DEV, generator=g).to(DTYPES[c["dtype"]])
        return dict(c=c, client=client, w=w, x=x, out=torch.empty((c["M"], c["N"]), dtype=x.dtype, device=DEV), ws=w.workspace(c["M"]))
    if k == "qmoe":
        client, g = ops.B200Client(0), _gen(seed)
        H, F = c["hidden"], c["ffn"]
        order = torch.from_numpy(ops.gate_up_row_order(F)).to(DEV)
        experts = []
        for _ in range(c["E"]):
            gu, dn = _rand_blocks(c["fmt"], 2 * F, H, g), _rand_blocks(c["fmt_down"], H, F, g)
            experts.append(ops.ExpertWeights(client.weight_from_ggml(GGML[c["fmt"]], gu[order].contiguous(), 2 * F, H), client.weight_from_ggml(GGML[c["fmt_down"]], dn, H, F),
                                             interleaved=F % 64 == 0))
        x, sel, gw = _qmoe_step(c, g)
        return dict(c=c, moe=ops.MoeMlp(client, experts, F, H), x=x, sel=sel, gw=gw)
    if k == "generate":
        dec = _decoder(seed, 64)
        dec.capture()
        return dict(c=c, dec=dec, prompt=_prompt(c, seed)[None])
    if k == "prompt":
        return dict(c=c, dec=_decoder(seed, 2048), prompt=_prompt(c, seed))
    if k == "ff":
        x, gu, dn = _ff_inputs(c, seed)
        mid, z = torch.empty((c["T"], c["F"]), dtype=torch.bfloat16, device=DEV), torch.empty((c["T"], 2 * c["F"]), **f32)
        return dict(c=c, x=x, gu=gu, dn=dn, mid=mid, z=z, y=torch.empty((c["T"], c["W"]), **f32))
    if k == "attn":
        rows, table, kpool, vpool = _attn_inputs(c, seed)
        H, G, D = c["H"], c["G"], c["D"]
        d, keep = _step(c["T"], c["B"], c["past"], table)
        desc = seqops.attn_desc(H, G, D, D, D ** -0.5, chunk=c["chunk"], window=c["window"], qk_eps=1e-5)
        keys = min([c["past"] + c["T"]] + [n for n in (c["chunk"], c["window"]) if n > 0])
        need = seqops.attn_scratch_floats(c["T"] * c["B"], c["B"], H, G, D, keys)
        return dict(c=c, rows=rows, work=torch.empty_like(rows), kpool=kpool, vpool=vpool, step=d, keep=keep, desc=desc, scratch=torch.empty(max(1, need), **f32),
                    out=torch.empty((c["T"] * c["B"], H * D), **f32))
    if k == "moe":
        x, gu, dn, z = _moe_inputs(c, seed)
        n, E = c["T"] * c["top"], c["E"]
        return dict(c=c, x=x, gu=gu, dn=dn, z=z, ids=torch.empty(n, **i32), wts=torch.empty(n, **f32), cnt=torch.zeros(E, **i32), off=torch.zeros(E + 1, **i32),
                    order=torch.empty(n, **i32), slot=torch.empty(n, **i32), xs=torch.empty((n, c["W"]), dtype=torch.bfloat16, device=DEV),
                    mid=torch.empty((n, c["F"]), dtype=torch.bfloat16, device=DEV), ys=torch.empty((n, c["W"]), **f32), y=torch.empty((c["T"], c["W"]), **f32))
    proj, xbc, A_log, Dp, dtb = _ssm_inputs(c, seed)
    H, V, N = c["H"], c["V"], c["N"]
    d, keep = _step(c["T"], 1, 0, torch.arange(-(-c["T"] // 16), **i32)[None].contiguous())
    need = seqops.ssm_scratch_floats(c["T"], 1, H, V, N)
    return dict(c=c, proj=proj, xbc=xbc, A_log=A_log, Dp=Dp, dtb=dtb, step=d, keep=keep, state=torch.zeros((1, H, N, V), **f32), scratch=torch.empty(max(1, need), **f32),
                out=torch.empty((c["T"], H * V), **f32))


def _qmoe_step(c, g):
    """activations, chosen experts (the last two of the bank are the shared halves of every token) and their weights"""
    T, E, top = c["T"], c["E"], c["top"]
    x = torch.randn((T, c["hidden"]), device=DEV, generator=g)
    z = torch.randn((T, E - 2), device=DEV, generator=g)
    best = torch.topk(z, top - 2, dim=1) if top > 2 else None
    sel = torch.tensor([[E - 2, E - 1]], device=DEV).expand(T, 2)
    gw = torch.ones((T, 2), device=DEV)
    if best is not None:
        sel, gw = torch.cat([best.indices, sel], 1), torch.cat([torch.softmax(best.values, 1), gw], 1)
    return x, sel.to(torch.int32).contiguous(), gw.float().contiguous()


# ---- one pass ---------------------------------------------------------------------------------------------------------------------
def run(s):
    c = s["c"]
    k = c["kind"]
    if k == "qmm":
        return s["client"].quant_matmul(s["x"], s["w"], out=s["out"], workspace=s["ws"])
    if k == "qmoe":
        return s["moe"].forward_decode(s["x"], s["sel"], s["gw"])
    if k == "generate":
        ids = s["dec"].generate(s["prompt"], 1)
        kv = s["dec"].kv_rows(s["dec"].layers[-1], 0, c["S"])
        return dict(ids=ids, logits=s["dec"].full_logits(), k=kv[0], v=kv[1])
    if k == "prompt":
        logits = s["dec"].prefill(s["prompt"])
        kv = [s["dec"].kv_rows(lay, 0, c["S"]) for lay in s["dec"].layers]
        return dict(logits=logits, k=[t[0] for t in kv], v=[t[1] for t in kv])
    if k == "ff":                                     # as LayeredModel runs a dense feed-forward
        x = s["x"]
        if c["T"] <= 8 or (c["T"] >= seqops.TC_MIN_ROWS and seqops.tc_usable(x, c["W"])):
            seqops.linear_act(x, s["gu"], seqops.ACT_SWISH_CLAMP, s["mid"], 7.0, 1.702, 1.0)
        else:
            seqops.linear(x, s["gu"], s["z"])
            seqops.act(s["z"], seqops.ACT_SWISH_CLAMP, s["mid"], 7.0, 1.702, 1.0)
        seqops.linear(s["mid"], s["dn"], s["y"])
        return s["mid"], s["y"]
    if k == "attn":                                   # the rows are prepared in place: a fresh copy, as the projection would write it
        s["work"].copy_(s["rows"])
        seqops.attn_prep_ex(s["work"], s["step"], s["desc"], s["kpool"], s["vpool"])
        seqops.attn_ex(s["work"], s["step"], s["desc"], s["kpool"], s["vpool"], s["out"], s["scratch"])
        return s["out"]
    if k == "moe":                                    # as LayeredModel runs routed experts behind a router's logits
        n = c["T"] * c["top"]
        few = n <= 64                                 # the weights are streamed per pair
        seqops.moe_route_ex(s["z"], c["E"], 1, 1, c["top"], seqops.ROUTE_TOP_SOFTMAX, None, s["ids"], s["wts"], None if few else s["cnt"])
        if few:
            seqops.moe_linear(s["x"], c["top"], s["gu"], s["ids"], None, None, n, seqops.ACT_SWISH_CLAMP, s["mid"], 7.0, 1.702, 1.0)
            seqops.moe_linear(s["mid"], 0, s["dn"], s["ids"], None, None, n, seqops.ACT_NONE, s["ys"])
        else:
            seqops.moe_sort(s["ids"], n, c["E"], s["cnt"], s["off"], s["order"], s["slot"])
            seqops.moe_gather(s["x"], c["top"], s["order"], n, s["xs"])
            seqops.moe_linear(s["xs"], 0, s["gu"], s["ids"], s["order"], s["off"], n, seqops.ACT_SWISH_CLAMP, s["mid"], 7.0, 1.702, 1.0)
            seqops.moe_linear(s["mid"], 0, s["dn"], s["ids"], s["order"], s["off"], n, seqops.ACT_NONE, s["ys"])
        seqops.moe_combine(s["ys"], s["wts"], None if few else s["slot"], c["T"], c["top"], None, None, s["y"])
        return s["y"]
    H, V, N, G = c["H"], c["V"], c["N"], c["G"]
    seqops.ssm_scan(s["proj"], 0, 2 * H * V + 2 * G * N, s["xbc"], s["A_log"], s["Dp"], s["dtb"], s["state"], s["step"], H, V, N, G, s["out"], s["scratch"])
    return s["out"], s["state"]


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------------
def _weight_bytes(fmt, N, K):
    if fmt in BLOCK:
        return N * K // BLOCK[fmt][0] * BLOCK[fmt][1]
    return N * K // 2 + N * (K // 128) * 5 // 2                       # a 16-bit scale and a 4-bit zero per group of 128


def _visible(c):
    """(query, key) pairs that a query head sees over the whole step, and the keys that are read at all"""
    pairs = 0
    for p in range(c["past"], c["past"] + c["T"]):
        lo = p // c["chunk"] * c["chunk"] if c["chunk"] else 0
        pairs += p + 1 - max(lo, p - c["window"] + 1 if c["window"] else 0)
    first = c["past"] // c["chunk"] * c["chunk"] if c["chunk"] else 0
    first = max(first, c["past"] - c["window"] + 1 if c["window"] else 0)
    return pairs * c["B"], (c["past"] + c["T"] - first) * c["B"]


def _model_work(S, one_by_one):
    m = SMALL
    qd, kvd = m.n_heads * m.head_dim, m.n_kv_heads * m.head_dim
    wb, per = 0, 0
    for i in range(m.n_layers):
        more = "Q6_K" if i % 2 == 0 else "Q4_K"
        for f, N, K in (("Q4_K", qd + kvd, m.hidden), (more, kvd, m.hidden), ("Q4_K", m.hidden, qd), ("Q4_K", 2 * m.ffn, m.hidden), (more, m.hidden, m.ffn)):
            wb, per = wb + _weight_bytes(f, N, K), per + 2 * N * K
    head, hf = _weight_bytes("Q6_K", m.vocab, m.hidden), 2 * m.vocab * m.hidden
    times = S if one_by_one else 1
    kv = 4 * 2 * kvd * m.n_layers
    attn = 4 * qd * m.n_layers * S * (S + 1) // 2
    moved = (wb + head) * times + kv * S + (kv * S * (S + 1) // 2 if one_by_one else 0) + S * m.hidden * 2 + 4 * m.vocab
    return dict(bytes=moved, flops=per * S + hf * times + attn)


def work(case):
    c = case
    k = c["kind"]
    if k == "qmm":
        es = 4 if c["dtype"] == "f32" else 2
        return dict(bytes=_weight_bytes(c["fmt"], c["N"], c["K"]) + es * c["M"] * (c["N"] + c["K"]), flops=2 * c["M"] * c["N"] * c["K"])
    if k == "qmoe":
        T, top, E, H, F = c["T"], c["top"], c["E"], c["hidden"], c["ffn"]
        used = min(2, top) + (E - 2) * (1 - (1 - (top - 2) / (E - 2)) ** T)      # experts that T tokens touch, on average
        one = _weight_bytes(c["fmt"], 2 * F, H) + _weight_bytes(c["fmt_down"], H, F)
        return dict(bytes=used * one + 8 * T * H, flops=T * top * 6 * F * H)
    if k in ("generate", "prompt"):
        return _model_work(c["S"], k == "generate")
    if k == "ff":
        T, W, F = c["T"], c["W"], c["F"]
        return dict(bytes=6 * W * F + 2 * T * W + 2 * T * F + 4 * T * W, flops=6 * T * W * F)
    if k == "attn":
        pairs, keys = _visible(c)
        T, H, G, D = c["T"] * c["B"], c["H"], c["G"], c["D"]
        return dict(bytes=4 * (T * (H * D + 2 * G * D + H) + T * H * D + 2 * keys * G * D), flops=4 * pairs * H * D)
    if k == "moe":
        T, W, F, E, top = c["T"], c["W"], c["F"], c["E"], c["top"]
        used = E * (1 - (1 - top / E) ** T)
        return dict(bytes=used * 6 * W * F + 2 * T * W + 4 * T * E + 4 * T * W, flops=6 * T * top * W * F)
    T, H, V, N, G = c["T"], c["H"], c["V"], c["N"], c["G"]
    return dict(bytes=4 * (T * (3 * H * V + 2 * G * N + H) + 2 * H * N * V), flops=4 * T * H * V * N)


def tolerance(case):
    k = case["kind"]
    if k == "qmm":
        if case["M"] <= 4:       # whole-number partial sums in 64 bits: the same to the rounding of the output
            return {"rel": 1e-6, "max": 1e-5} if case["dtype"] == "f32" else {"rel": 1e-3, "max": 1e-2}
        return {"rel": 2e-5, "max": 1e-3} if case["dtype"] == "f32" else {"rel": 5e-3, "max": 4e-2}
    return {
        "qmoe": {"rel": 1e-5, "max": 1e-4},
        "generate": {"rel": 1e-2, "max": 0.2, "differ": 0.0},
        "prompt": {"rel": 1e-2, "max": 0.2},
        "ff": {"rel": 1e-2, "max": 0.1},
        "attn": {"rel": 2e-5, "max": 1e-3},
        "moe": {"rel": 1e-2, "max": 0.1},
        "ssm": {"rel": 2e-5, "max": 1e-3},
    }[k]


# ---- the same in 64 bits -----------------------------------------------------------------------------------------------------------
def _nibbles(b):
    return torch.cat([b & 15, b >> 4], -1)


def _dequant(fmt, N, K, packed):
    """f64 [N, K] of packed weights, from the public layouts"""
    f16 = lambda t: t.contiguous().view(torch.float16).double()
    if fmt == "Q8_0":
        b = packed[0].reshape(-1, 34)
        return (f16(b[:, :2]) * b[:, 2:].contiguous().view(torch.int8).double()).reshape(N, K)
    if fmt == "Q4_K":
        b = packed[0].reshape(-1, 144)
        s = b[:, 4:16].int()
        sc = torch.cat([s[:, 0:4] & 63, (s[:, 8:12] & 15) | ((s[:, 0:4] >> 6) << 4)], 1).double()
        mn = torch.cat([s[:, 4:8] & 63, (s[:, 8:12] >> 4) | ((s[:, 4:8] >> 6) << 4)], 1).double()
        q = _nibbles(b[:, 16:].reshape(-1, 4, 32)).reshape(-1, 8, 32).double()
        return ((f16(b[:, :2]) * sc)[:, :, None] * q - (f16(b[:, 2:4]) * mn)[:, :, None]).reshape(N, K)
    if fmt == "Q6_K":
        b = packed[0].reshape(-1, 210)
        ql, qh = b[:, :128].reshape(-1, 2, 64).int(), b[:, 128:192].reshape(-1, 2, 32).int()
        sc, d = b[:, 192:208].contiguous().view(torch.int8).double(), f16(b[:, 208:210])
        lo = [ql[..., :32] & 15, ql[..., 32:] & 15, ql[..., :32] >> 4, ql[..., 32:] >> 4]
        q = torch.stack([lo[j] | (((qh >> (2 * j)) & 3) << 4) for j in range(4)], 2) - 32      # [blocks, half, quarter, 32]
        return ((d * sc)[:, :, None] * q.reshape(-1, 16, 16).double()).reshape(N, K)
    qw, sc, z = packed
    if fmt == "AWQ":                                                # word i of row k: columns 8 i .. in the order 0 2 4 6 1 3 5 7
        sh = torch.tensor([0, 16, 4, 20, 8, 24, 12, 28], device=DEV)
        q = ((qw[:, :, None] >> sh) & 15).reshape(K, N).double()
        zero = z.double()
    else:
        sh = torch.arange(0, 32, 4, device=DEV)
        q = ((qw[:, None, :] >> sh[None, :, None]) & 15).reshape(K, N).double()
        zero = ((z[:, :, None] >> sh) & 15).reshape(K // 128, N).double() + 1.0
    grp = torch.arange(K, device=DEV) // 128
    return ((q - zero[grp]) * sc.double()[grp]).T


def _swish(z, limit=7.0):
    g, u = z[:, 0::2].clamp(max=limit), z[:, 1::2].clamp(-limit, limit)
    return g * torch.sigmoid(1.702 * g) * (u + 1.0)


def _unit(t, eps=1e-5):
    return t / torch.sqrt((t * t).mean(-1, keepdim=True) + eps)


def _model_exact(c, seed):
    m, parts = SMALL, _model_parts(seed)
    ids = torch.from_numpy(_prompt(c, seed)).to(DEV)
    S, hd = c["S"], m.head_dim
    W = lambda t: _dequant(*t[:3], (t[3],))
    ang = torch.arange(S, device=DEV).double()[:, None] * (m.rope_theta ** (-2.0 * torch.arange(hd // 2, device=DEV).double() / hd))[None]
    cs, sn = ang.cos()[:, None], ang.sin()[:, None]

    def rot(x):
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * cs - b * sn, a * sn + b * cs], -1).flatten(-2)

    h = parts["embed"][ids].double()
    mask = torch.ones((S, S), dtype=torch.bool, device=DEV).tril()
    ks, vs = [], []
    for lay in parts["layers"]:
        x = _unit(h, m.eps) * lay["attn_norm"].double()
        q, kk, v = (x @ W(lay[p]).T for p in ("q", "k", "v"))
        q, kk, v = rot(q.reshape(S, -1, hd)), rot(kk.reshape(S, -1, hd)), v.reshape(S, -1, hd)
        ks.append(kk), vs.append(v)
        per = m.n_heads // m.n_kv_heads
        o = torch.empty_like(q)
        for i in range(m.n_heads):
            p = (q[:, i] @ kk[:, i // per].T) / math.sqrt(hd)
            o[:, i] = torch.softmax(p.masked_fill(~mask, float("-inf")), 1) @ v[:, i // per]
        h = h + o.reshape(S, -1) @ W(lay["o"]).T
        x = _unit(h, m.eps) * lay["mlp_norm"].double()
        g = x @ W(lay["gate"]).T
        h = h + (g * torch.sigmoid(g) * (x @ W(lay["up"]).T)) @ W(lay["down"]).T
    x = _unit(h[-1:], m.eps) * parts["final"].double()
    return (x @ W(parts["head"]).T), ks, vs


def exact(case, seed):
    c = case
    k = c["kind"]
    if k == "qmm":
        g = _gen(seed)
        w = _dequant(c["fmt"], c["N"], c["K"], _packed(c["fmt"], c["N"], c["K"], g))
        return torch.randn((c["M"], c["K"]), device=DEV, generator=g).to(DTYPES[c["dtype"]]).double() @ w.T
    if k == "qmoe":
        g = _gen(seed)
        H, F = c["hidden"], c["ffn"]
        ws = [(_rand_blocks(c["fmt"], 2 * F, H, g), _rand_blocks(c["fmt_down"], H, F, g)) for _ in range(c["E"])]
        x, sel, gw = _qmoe_step(c, g)
        y = torch.zeros((c["T"], H), dtype=torch.float64, device=DEV)
        for t in range(c["T"]):
            for j in range(c["top"]):
                a, b = ws[int(sel[t, j])]
                z = _dequant(c["fmt"], 2 * F, H, (a,)) @ x[t].double()
                y[t] += gw[t, j].double() * (_dequant(c["fmt_down"], H, F, (b,)) @ (z[:F] * torch.sigmoid(z[:F]) * z[F:]))
        return y
    if k == "generate":
        logits, ks, vs = _model_exact(c, seed)
        return dict(ids=None, logits=logits, k=ks[-1], v=vs[-1])
    if k == "prompt":
        logits, ks, vs = _model_exact(c, seed)
        return dict(logits=logits[0], k=ks, v=vs)
    if k == "ff":
        x, gu, dn = _ff_inputs(c, seed)
        mid = _swish(x.double() @ gu.double().T)
        return mid, mid @ dn.double().T
    if k == "attn":
        rows, table, kpool, vpool = _attn_inputs(c, seed)
        H, G, D, B, T, past = c["H"], c["G"], c["D"], c["B"], c["T"], c["past"]
        out = torch.empty((B, T, H, D), dtype=torch.float64, device=DEV)
        r = rows.double().reshape(B, T, -1)
        qpos, kpos = torch.arange(past, past + T, device=DEV)[:, None], torch.arange(past + T, device=DEV)[None]
        see = kpos <= qpos
        if c["chunk"]:
            see = see & (kpos // c["chunk"] == qpos // c["chunk"])
        if c["window"]:
            see = see & (qpos - kpos < c["window"])
        for b in range(B):
            slots = (table[b].long()[:, None] * 16 + torch.arange(16, device=DEV)[None]).reshape(-1)[:past]
            q = _unit(r[b, :, :H * D].reshape(T, H, D))
            kk = torch.cat([kpool[slots].double(), _unit(r[b, :, H * D:(H + G) * D].reshape(T, G, D))])
            v = torch.cat([vpool[slots].double(), r[b, :, (H + G) * D:(H + 2 * G) * D].reshape(T, G, D)])
            for h in range(H):
                p = (q[:, h] @ kk[:, h // (H // G)].T) * D ** -0.5
                out[b, :, h] = torch.softmax(p.masked_fill(~see, float("-inf")), 1) @ v[:, h // (H // G)]
            out[b] *= torch.sigmoid(r[b, :, (H + 2 * G) * D:])[:, :, None]
        return out.reshape(B * T, H * D)
    if k == "moe":
        x, gu, dn, z = _moe_inputs(c, seed)
        best = torch.topk(torch.softmax(z.double(), 1), c["top"], dim=1)
        wts = best.values / best.values.sum(1, keepdim=True)
        y = torch.zeros((c["T"], c["W"]), dtype=torch.float64, device=DEV)
        for e in range(c["E"]):
            t, j = (best.indices == e).nonzero(as_tuple=True)
            if t.numel():
                y.index_add_(0, t, wts[t, j][:, None] * (_swish(x[t].double() @ gu[e].double().T) @ dn[e].double().T))
        return y
    proj, xbc, A_log, Dp, dtb = (t.double() for t in _ssm_inputs(c, seed))
    H, V, N, G, T = c["H"], c["V"], c["N"], c["G"], c["T"]
    x = xbc[:, :H * V].reshape(T, H, V)
    Bm, Cm = (xbc[:, H * V + i * G * N:H * V + (i + 1) * G * N].reshape(T, G, N).repeat_interleave(H // G, 1) for i in (0, 1))
    dt = torch.nn.functional.softplus(proj[:, -H:] + dtb)
    decay = torch.exp(-torch.exp(A_log) * dt)
    S = torch.zeros((H, N, V), dtype=torch.float64, device=DEV)
    y = torch.empty((T, H, V), dtype=torch.float64, device=DEV)
    dx = dt[:, :, None] * x
    for t in range(T):
        S.mul_(decay[t][:, None, None]).baddbmm_(Bm[t][:, :, None], dx[t][:, None, :])
        torch.bmm(Cm[t][:, None, :], S, out=y[t][:, None, :])
    y += Dp[:, None] * x
    z = proj[:, :H * V]
    return (y.reshape(T, H * V) * z * torch.sigmoid(z)), S[None]
