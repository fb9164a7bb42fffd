"""The row operators of a prompt (norm, SwiGLU, RoPE with the cache rows) against the same formulas in torch: f16 results equal the rounded f32
ones, sizes that leave threads without a column, paged caches, extreme values."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def L():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from blazr_b200 import ops
    return ops.lib()


P = lambda t: C.c_void_p(t.data_ptr()) if t is not None else None
St = lambda: C.c_void_p(torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("M,H", [(1, 256), (130, 768), (200, 2048), (129, 4352), (128, 8192)])
@pytest.mark.parametrize("with_delta", [False, True])
def test_norm(L, M, H, with_delta):
    h, d, w = torch.randn(M, H, device=DEV), torch.randn(M, H, device=DEV) if with_delta else None, torch.randn(H, device=DEV)
    h[0, 0] = 3e5
    w[0] = 1e4                                        # the largest value leaves the f16 range: clamped
    s = h + d if with_delta else h
    ref = s.double() / torch.sqrt((s.double() ** 2).mean(1, keepdim=True) + 1e-5) * w.double()
    out, x16, x32 = torch.empty_like(h), torch.empty(M, H, device=DEV, dtype=torch.float16), torch.empty_like(h)
    assert L.b200q_add_rmsnorm_f16(P(h), P(d), P(out), P(w), C.c_float(1e-5), C.c_int64(H), C.c_int64(M), P(x16), St()) == 0
    assert torch.equal(out, s)
    assert ((x16.double() - ref.clamp(-65504, 65504)).abs() / (ref.abs() + 1e-3)).max().item() < 2 ** -10
    assert L.b200q_add_rmsnorm_quant(P(h), P(d), P(out), P(w), C.c_float(1e-5), C.c_int64(H), C.c_int64(M), None, P(x32), St()) == 0
    assert torch.equal(x32.clamp(-65504, 65504).half(), x16) and torch.equal(out, s)


@pytest.mark.parametrize("M,F", [(1, 64), (7, 192), (300, 1408), (2, 8256)])
@pytest.mark.parametrize("il", [0, 1])
def test_swiglu(L, M, F, il):
    from blazr_b200 import ops
    gu = torch.randn(M, 2 * F, device=DEV) * 4
    gu[0, 0], gu[0, F] = 100.0, 5000.0
    x = gu[:, torch.from_numpy(ops.gate_up_row_order(F)).to(DEV)].contiguous() if il else gu
    a16, a32 = torch.empty(M, F, device=DEV, dtype=torch.float16), torch.empty(M, F, device=DEV)
    assert L.b200q_swiglu_f16(P(x), C.c_int64(F), C.c_int64(M), C.c_int32(il), P(a16), St()) == 0
    assert (L.b200q_swiglu_f32_interleaved if il else L.b200q_swiglu_f32)(P(x), C.c_int64(F), C.c_int64(M), P(a32), St()) == 0
    g, u = gu[:, :F].double(), gu[:, F:].double()
    ref = g * torch.sigmoid(g) * u
    assert ((a32.double() - ref).abs() / (ref.abs() + 1e-3)).max().item() < 2e-6
    assert torch.equal(a32.clamp(-65504, 65504).half(), a16)


@pytest.mark.parametrize("S,nh,nkv,hd,bs", [(1, 2, 1, 64, 0), (37, 8, 2, 128, 0), (50, 6, 3, 64, 16), (5, 40, 8, 128, 4)])
def test_rope_and_cache_rows(L, S, nh, nkv, hd, bs):
    from blazr_b200.decode import rope_table
    qkv = torch.randn(S, (nh + 2 * nkv) * hd, device=DEV)
    rope = torch.from_numpy(rope_table(64, hd, 10000.0)).to(DEV)
    nb = 64 // bs if bs else 1
    bt = torch.randperm(nb, device=DEV).to(torch.int32) if bs else None
    ck, cv = (torch.full((64, nkv, hd), 9.0, device=DEV) for _ in range(2))
    q16, k16, v16 = (torch.empty(S, n, hd, device=DEV, dtype=torch.float16) for n in (nh, nkv, nkv))
    assert L.b200q_rope_kv_prefill(P(qkv), P(rope), nh, nkv, hd, C.c_int64(S), P(q16), P(k16), P(v16), P(ck), P(cv), P(bt), bs, St()) == 0
    cos, sin = rope[:S, None, :, 0], rope[:S, None, :, 1]

    def rot(x):
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack((a * cos - b * sin, a * sin + b * cos), -1).flatten(-2)

    q, k, v = rot(qkv[:, :nh * hd].reshape(S, nh, hd)), rot(qkv[:, nh * hd:(nh + nkv) * hd].reshape(S, nkv, hd)), qkv[:, (nh + nkv) * hd:].reshape(S, nkv, hd)
    j = torch.arange(S, device=DEV)
    at = bt[j // bs].long() * bs + j % bs if bs else j
    assert torch.equal(ck[at], k) and torch.equal(cv[at], v)                   # the products and sums torch rounds, one by one
    assert torch.equal(q16, q.half()) and torch.equal(k16, k.half()) and torch.equal(v16, v.half())
    rest = torch.ones(64, dtype=torch.bool, device=DEV)
    rest[at] = False
    assert bool((ck[rest] == 9.0).all()) and bool((cv[rest] == 9.0).all())


def _decoders(cfg, scheme, change=None):
    from blazr_b200 import decode, ops
    hm = decode.build_host_model(cfg, scheme, seed=4)
    for lay in hm.layers:
        if change is not None:
            change(lay)
    client = ops.B200Client(0)
    return [decode.Decoder(client, cfg, scheme, batch=1, max_ctx=16, host=hm) for _ in range(2)]


def _token_by_token(dec, prompt):
    dec.reset([int(prompt[0])])
    for t in prompt:
        dec.ids.fill_(int(t))
        dec.step()
    torch.cuda.synchronize()
    return dec.full_logits().reshape(-1)


@pytest.mark.parametrize("scheme", ["Q4_K_M", "Q6_K", "Q8_0"])
@pytest.mark.parametrize("S", [1, 2, 3, 4])
def test_prompts_of_up_to_four_tokens_quantize_their_f32_rows(scheme, S):
    """Up to four rows take the integer matvec, as a decode step does: the first layer's keys and values are those of token-by-token decoding, bit for
    bit, and rows beyond the f16 range are not clamped (norm weights of 1e5: the activations reach 1e10, and clamped at 65504 little but their signs
    would be left).  Bound of that part: the attention of a prompt is rounded to f16, which moves int8 roundings (half a unit of 1 / 127 of a block of 32's
    largest value, 0.3 % of the block's size each) in four products of each of the two layers and the head: below 3e-2."""
    from blazr_b200 import decode
    cfg = decode.PRESETS["tiny"]
    prompt = torch.arange(7, 7 + S).numpy() * 31
    a, b = _decoders(cfg, scheme)
    a.prefill(prompt)
    _token_by_token(b, prompt)
    for name in ("ck", "cv"):
        assert torch.equal(a.layers[0][name][0, :S], b.layers[0][name][0, :S])

    def loud(lay):
        lay["mlp_norm"] = (lay["mlp_norm"] * 1e5).astype("float32")

    a, b = _decoders(cfg, scheme, loud)
    got, want = a.prefill(prompt).double(), _token_by_token(b, prompt).double()
    assert ((got - want).norm() / want.norm()).item() < 3e-2


def test_prompts_of_heads_that_are_not_a_multiple_of_four():
    from blazr_b200 import decode
    from oracle.model import OracleModel
    cfg = decode.ModelConfig("odd", 512, 2, 16, 4, 66, 1024, 512)
    a, _ = _decoders(cfg, "Q8_0")
    prompt = torch.arange(3, 12).numpy() * 17
    got = a.prefill(prompt).double().cpu()
    oracle = OracleModel(decode.build_host_model(cfg, "Q8_0", seed=4), flavour="A")
    for t in prompt:
        want = oracle.step(int(t))
    want = torch.as_tensor(want).double().reshape(-1)
    assert ((got - want).norm() / want.norm()).item() < 1e-2


def test_prompt_buffers_are_those_that_the_pass_uses(monkeypatch):
    """Gate|up products that leave as activations keep no rows of their own, and each of the two expansion buffers has the size of the projections that use
    it; without that epilogue the rows are there, and the logits are the same, bit for bit."""
    import dataclasses
    from blazr_b200 import decode, ops
    cfg = dataclasses.replace(decode.PRESETS["small-1b"], n_layers=2)
    hm = decode.build_host_model(cfg, "Q4_K", seed=9)
    client = ops.B200Client(0)
    prompt = (torch.arange(2048) * 37 % cfg.vocab).numpy()
    got = []
    for epi in ("1", "0"):
        monkeypatch.setenv("B200Q_SWIGLU_EPI", epi)
        dec = decode.Decoder(client, cfg, "Q4_K", batch=1, max_ctx=2048, host=hm)
        got.append(dec.prefill(prompt).clone())
        b = dec._pf
        assert (b["gu"] is None) == (epi == "1") == all(b["gated"])
        for p in range(2):
            assert b["panels"][p].numel() == max([256] + [sum(n for _, n in g) for g in b["groups"][p::2]])
        assert b["panels"][0].numel() > 256
    assert torch.equal(got[0], got[1])
