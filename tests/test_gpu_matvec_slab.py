"""Matvec of weights whose rows, dealt over the SMs, fit their shared memory (csrc/matvec_slab.cuh).  A row's result does not depend on the rows beside it,
so the results are those of the same rows inside a weight that is too large for this kernel, bit for bit: row counts that fill one slab, end inside one,
cross a tile, or need the widest slabs; one to four rows of activations; every format that has planes; and the fused forms on whole tiles."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
BIG = 20480      # rows: more than 148 slabs of 128


@pytest.fixture(scope="module")
def client():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from blazr_b200 import ops
    return ops.B200Client(0)


def pair(client, fmt, N, K, seed=5):
    """the first N rows of a weight, and the whole of it"""
    from blazr_b200 import ops, synth
    if fmt in synth.GGML:
        t = synth.GGML[fmt]
        blk = synth.random_ggml(t, BIG, K, seed=seed)
        return client.weight_from_ggml(t, np.ascontiguousarray(blk[:N]), N, K), client.weight_from_ggml(t, blk, BIG, K)
    gs = int(fmt[3:])
    qw, sc, zr = synth.random_awq(BIG, K, gs, seed=seed)
    dq = ops.DecomposedQuantTensor(qw, sc, zr, None, ops.DecomposedQuantMethod("awq", gs), (BIG, K))
    return client.weight_from_decomposed(dq, rows=(0, N)), client.weight_from_decomposed(dq)


@pytest.mark.parametrize("fmt,K", [("Q4_K", 512), ("Q6_K", 1024), ("Q8_0", 1056), ("AWQ128", 512), ("AWQ256", 512), ("AWQ32", 768)])
@pytest.mark.parametrize("N", [8, 128, 1192, 2960, 3072, 9000, 18944])
def test_rows_of_a_larger_weight(client, fmt, K, N):
    small, large = pair(client, fmt, N, K)
    x = torch.randn((4, K), device="cuda", generator=torch.Generator(device="cuda").manual_seed(N))
    for M in (1, 2, 3, 4):
        xq = client.quantize_act(x[:M].contiguous())
        a, b = client.matmul_q8(xq, M, small), client.matmul_q8(xq, M, large)[:, :N]
        assert torch.equal(a.view(torch.int32), b.contiguous().view(torch.int32)), (fmt, N, M)
        assert torch.equal(client.quant_matmul(x[:M], small).view(torch.int32), a.view(torch.int32))


@pytest.mark.parametrize("fmt,K", [("Q4_K", 8192), ("Q6_K", 4096), ("Q8_0", 2048)])
def test_norm_prologue(client, fmt, K):
    from blazr_b200 import ops
    small, large = pair(client, fmt, 2056, K)
    L, P = ops.lib(), lambda t: C.c_void_p(t.data_ptr())
    for M in (1, 3):
        h, d, nw = torch.randn((M, K), device="cuda"), torch.randn((M, K), device="cuda"), torch.randn(K, device="cuda")
        res = []
        for w in (small, large):
            ho, y, ws = torch.zeros((M, K), device="cuda"), torch.zeros((M, w.N), device="cuda"), w.workspace(M)
            ops._check(L.b200q_matmul_norm(w.handle, P(h), P(d), P(ho), P(nw), C.c_float(1e-5), C.c_int64(M), P(y), C.c_int32(ops.F32), C.c_int64(w.N), P(ws), C.c_size_t(ws.numel()), None))
            res.append((ho, y[:, :2056].contiguous()))
        assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1].view(torch.int32), res[1][1].view(torch.int32))


def gated_pair(client, fmt, F, K):
    """a gate|up weight with its rows as they lie in a file, and the same in the order of whole tiles; the sizes at which a CTA takes a whole tile"""
    from blazr_b200 import ops, synth
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert 104 * sms < 2 * F <= 128 * sms
    t = synth.GGML[fmt]
    blk = synth.random_ggml(t, 2 * F, K, seed=F)
    return client.weight_from_ggml(t, blk, 2 * F, K), client.weight_from_ggml(t, np.ascontiguousarray(blk[ops.gate_up_row_order(F)]), 2 * F, K)


@pytest.mark.parametrize("fmt,F,M", [("Q4_K", 8192, 1), ("Q6_K", 7744, 2), ("Q6_K", 9472, 3), ("Q8_0", 9472, 4)])
def test_gated_tiles(client, fmt, F, M):
    from blazr_b200 import ops
    K = 512
    plain, mixed = gated_pair(client, fmt, F, K)
    L, P = ops.lib(), lambda t_: C.c_void_p(t_.data_ptr())
    xq = client.quantize_act(torch.randn((M, K), device="cuda"))
    gu = client.matmul_q8(xq, M, plain)
    want, got = (torch.zeros(int(L.b200q_act_bytes(C.c_int64(F), C.c_int64(M))), dtype=torch.uint8, device="cuda") for _ in range(2))
    ops._check(L.b200q_swiglu_quant(P(gu), C.c_int64(F), C.c_int64(M), P(want), None))
    ws = mixed.workspace(M)
    ops._check(L.b200q_matmul_q8_swiglu(mixed.handle, P(xq), C.c_int64(M), P(got), P(ws), C.c_size_t(ws.numel()), None))
    assert torch.equal(got, want)


@pytest.mark.parametrize("fmt,F,K,M", [("Q4_K", 8192, 2048, 1), ("Q6_K", 7744, 1024, 2), ("Q8_0", 9472, 512, 3), ("Q4_K", 9472, 512, 4)])
def test_norm_and_gated_tiles(client, fmt, F, K, M):
    from blazr_b200 import ops
    plain, mixed = gated_pair(client, fmt, F, K)
    L, P = ops.lib(), lambda t_: C.c_void_p(t_.data_ptr())
    h, d, nw = torch.randn((M, K), device="cuda"), torch.randn((M, K), device="cuda"), torch.randn(K, device="cuda")
    gu, xq = torch.zeros((M, 2 * F), device="cuda"), torch.zeros(int(L.b200q_act_bytes(C.c_int64(K), C.c_int64(M))), dtype=torch.uint8, device="cuda")
    h1, h2 = torch.zeros_like(h), torch.zeros_like(h)
    want, got = (torch.zeros(int(L.b200q_act_bytes(C.c_int64(F), C.c_int64(M))), dtype=torch.uint8, device="cuda") for _ in range(2))
    ops._check(L.b200q_add_rmsnorm_quant(P(h), P(d), P(h1), P(nw), C.c_float(1e-5), C.c_int64(K), C.c_int64(M), P(xq), None, None))
    client.matmul_q8(xq, M, plain, out=gu)
    ops._check(L.b200q_swiglu_quant(P(gu), C.c_int64(F), C.c_int64(M), P(want), None))
    ws = mixed.workspace(M)
    ops._check(L.b200q_matmul_norm_swiglu(mixed.handle, P(h), P(d), P(h2), P(nw), C.c_float(1e-5), C.c_int64(M), P(got), P(ws), C.c_size_t(ws.numel()), None))
    assert torch.equal(got, want) and torch.equal(h1, h2)


def test_the_next_weights_hint_changes_no_result(client):
    """b200q_weight_set_next on a weight of this kernel, on a larger one, on the quantising forms and on a chain that ends where it began"""
    from blazr_b200 import synth
    t, K = synth.GGML["Q4_K"], 2048
    ws = [client.weight_from_ggml(t, synth.random_ggml(t, N, K, seed=N), N, K) for N in (2048, 20480, 1000, 8192)]
    x = torch.randn((2, K), device="cuda")
    xq = client.quantize_act(x)
    want = [(client.matmul_q8(xq, 2, w), client.quant_matmul(x, w)) for w in ws]
    for a, b in zip(ws, ws[1:] + ws[:1]):
        a.set_next(b)
    for _ in range(3):
        got = [(client.matmul_q8(xq, 2, w), client.quant_matmul(x, w)) for w in ws]
        assert all(torch.equal(g, v) for gs, vs in zip(got, want) for g, v in zip(gs, vs))
    for w in ws:
        w.set_next(None)
