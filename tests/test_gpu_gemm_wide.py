"""The dequant-GEMM of large steps (csrc/gemm_wide.cu: weights expanded once into f16 rows, paired-SM GEMM) against the dequantized weight in
float64, at sizes where it can go wrong: rows that end inside a 128- and a 256-row tile, K that is not a multiple of a chunk, several panels,
activations of every type, unaligned and with a row stride, act-order, bias -- and against the fused kernel, which a smaller workspace keeps.

Bound: weights and activations are rounded to f16 (2^-11 each), so a product is off by at most 2^-10 of its size and, the roundings being
independent, the sum's relative 2-norm error stays below 2^-11 * sqrt(2) * 1.2 = 8.3e-4; a 16-bit output adds its own half unit."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def client():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from blazr_b200 import ops
    return ops.B200Client(0)


def weight(client, fmt, N, K):
    from blazr_b200 import ops, synth
    if fmt in synth.GGML:
        t = synth.GGML[fmt]
        return client.weight_from_ggml(t, synth.random_ggml(t, N, K, seed=N + K), N, K)
    if fmt == "AWQ":
        return client.weight_from_decomposed(ops.DecomposedQuantTensor(*synth.random_awq(N, K, 128, seed=5), None, ops.DecomposedQuantMethod("awq", 128), (N, K)))
    qw, sc, qz, gi, b = synth.random_gptq(N, K, 128, seed=6, act_order=True, bias=True)
    return client.weight_from_decomposed(ops.DecomposedQuantTensor(qw, sc, qz, gi, ops.DecomposedQuantMethod("gptq", 128), (N, K), bias=b)), b


@pytest.mark.parametrize("fmt,N,K,M", [("Q4_K", 300, 512, 1100), ("Q6_K", 2500, 256, 2100), ("Q8_0", 777, 1056, 1500), ("AWQ", 1536, 1152, 1025), ("Q5_K", 128, 2048, 3000),
                                       ("Q8_0", 33000, 2080, 700), ("Q4_0", 513, 96, 4097), ("IQ4_XS", 640, 768, 1300)])
@pytest.mark.parametrize("dt", [torch.float32, torch.float16, torch.bfloat16])
def test_against_the_dequantized_weight(client, fmt, N, K, M, dt):
    from blazr_b200 import ops
    w = weight(client, fmt, N, K)
    wd = client.dequantize(w).double()
    g = torch.Generator(device="cuda:0")
    g.manual_seed(1)
    x = torch.randn((M, K + 3), device="cuda:0", generator=g).to(dt)[:, 1:K + 1]      # rows that start anywhere
    xa = x.contiguous()
    ref = xa.double() @ wd.T
    y = torch.full((M, N), 7.0, device="cuda:0")
    need = w.workspace_bytes(M)
    ws = torch.zeros(need, dtype=torch.uint8, device="cuda:0")
    for xx in (x, xa):
        client.quant_matmul(xx, w, out=y, workspace=ws)
        assert ((y.double() - ref).norm() / ref.norm()).item() < 8.3e-4
    y16 = client.quant_matmul(xa, w, out_dtype=torch.bfloat16, workspace=ws)
    assert ((y16.double() - ref).norm() / ref.norm()).item() < 8.3e-4 + 2 ** -9
    flags = C.c_int32(0)
    assert ops.lib().b200q_decode_error(C.byref(flags)) == 0 and flags.value == 0
    # the least workspace that is accepted keeps the fused kernel: the same result
    lo, hi = 0, need // 256
    y2 = torch.empty_like(y)
    while lo < hi:
        mid = (lo + hi) // 2
        try:
            client.quant_matmul(xa, w, out=y2, workspace=ws[:mid * 256])
            hi = mid
        except ops.B200QError:
            lo = mid + 1
    client.quant_matmul(xa, w, out=y2, workspace=ws[:hi * 256])
    assert ((y2.double() - y.double()).norm() / ref.norm()).item() < 2e-5


def test_act_order_and_bias(client):
    N, K, M = 1024, 1024, 1200
    w, b = weight(client, "GPTQ", N, K)
    wd = client.dequantize(w).double()
    x = torch.randn((M, K), device="cuda:0")
    ref = x.double() @ wd.T + torch.from_numpy(np.asarray(b)).cuda().double()
    y = client.quant_matmul(x, w)
    assert ((y.double() - ref).norm() / ref.norm()).item() < 8.3e-4


def test_extreme_activations_are_clamped_as_before(client):
    w = weight(client, "Q8_0", 256, 256)
    x = torch.randn((1500, 256), device="cuda:0")
    x[3, 5], x[4, 6], x[5, 7] = float("inf"), -1e9, float("nan")
    y = client.quant_matmul(x, w)
    small = client.quant_matmul(x[:16].contiguous(), w)          # the fused kernel's staging
    assert torch.isfinite(y).all() and ((y[:16] - small).abs().max() / small.abs().max()).item() < 1e-5


@pytest.mark.parametrize("N,K,M", [(512, 2048, 512), (512, 2048, 2048), (1024, 4096, 2048), (4096, 1024, 512)])
def test_products_that_are_cut_along_k_stay_cut(client, N, K, M):
    """Weights of one, 65504 in the first half of K, 1 / 64 in the second.  A single chain of f32 sums loses the small terms (16 of them make 1 / 4, half a
    unit of the large sum is 4 and more); cut along K, they are summed by themselves first and arrive whole."""
    blk = np.zeros((N, K // 32, 34), np.uint8)
    blk[:, :, :2] = np.frombuffer(np.float16(1.0).tobytes(), np.uint8)
    blk[:, :, 2:] = 1
    w = client.weight_from_ggml(8, blk.reshape(N, -1), N, K)
    x = torch.full((M, K), 65504.0, device="cuda:0")
    x[:, K // 2:] = 2.0 ** -6
    y = client.quant_matmul(x, w)
    big, small = K // 2 * 65504.0, K // 2 * 2.0 ** -6
    want = torch.tensor(big + small, dtype=torch.float64).float().item()
    assert want > big and (y == want).all()


def fused_need(w, N, K, M):
    """bytes of scratch that the fused kernel asks for: staged rows, and partial sums where it cuts K (csrc/gemm_tc.cu)"""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    mt, tiles = -(-M // 256), -(-N // 128)
    rows = -(-(-(-M // mt)) // 32) * 32
    cut = max(1, min(sms // (tiles * mt), 8, max(1, w.K_pad // 256 // 2)))
    return -(-(mt * rows * w.K_pad * 2) // 256) * 256 + (cut * M * N * 4 if cut > 1 else 0)


@pytest.mark.parametrize("fmt,N,K,M,launches", [
    ("Q4_K", 512, 2048, 520, 4),            # K in four parts: rows staged, weight expanded, one GEMM, sums of the parts
    ("Q6_K", 1000, 4096, 1500, 4),          # K in three parts that are not equal, rows of a weight that end inside a tile
    ("AWQ", 6144, 4096, 1531, 3),
    ("Q6_K", 14400, 4096, 2048, 5),         # two panels
    ("Q4_K", 24700, 8192, 800, 15),         # seven panels, odd tile counts and a short last one: both buffers are used again
    ("Q8_0", 12300, 4128, 2000, 5),         # K that ends inside a chunk
])
def test_the_expanded_weight_is_used_and_gives_the_fused_kernels_bits(client, fmt, N, K, M, launches):
    """Same operands, same order of k, same cuts of it: equal bits.  Several calls run back to back over one workspace, each on rows of its own."""
    from blazr_b200 import ops
    w = weight(client, fmt, N, K)
    full, least = w.workspace_bytes(M), -(-fused_need(w, N, K, M) // 256) * 256
    assert full > least
    ws = torch.zeros(full, dtype=torch.uint8, device="cuda:0")
    g = torch.Generator(device="cuda:0")
    g.manual_seed(2)
    xs = [torch.randn((M, K), device="cuda:0", generator=g).half() for _ in range(3)]
    ys = [torch.empty((M, N), device="cuda:0") for _ in xs]
    n0 = ops.launch_count()
    for x, y in zip(xs, ys):
        client.quant_matmul(x, w, out=y, workspace=ws)
    assert ops.launch_count() - n0 == 3 * launches
    y2 = torch.empty_like(ys[0])
    for x, y in zip(xs, ys):
        client.quant_matmul(x, w, out=y2, workspace=ws[:least])
        assert torch.equal(y, y2)


def test_large_steps_leave_no_scratch_behind(client):
    """Scratch of a large step is tens of megabytes (the expanded weight): it goes back to the allocator with the call, whatever lengths a program runs."""
    w = weight(client, "Q4_K", 4096, 2048)
    x = torch.randn((1500, 2048), device="cuda:0")
    y = torch.empty((1500, 4096), device="cuda:0")
    client.quant_matmul(x[:1024], w, out=y[:1024])
    torch.cuda.synchronize()
    held = torch.cuda.memory_allocated()
    for M in (1500, 1400, 1300, 1200, 1100, 600):
        client.quant_matmul(x[:M], w, out=y[:M])
    torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() == held


@pytest.mark.parametrize("fmt,N,K,M", [("Q4_K", 2048, 2048, 513), ("Q6_K", 512, 2048, 2048), ("Q6_K", 14336, 4096, 2048), ("Q8_0", 1000, 1024, 2048), ("AWQ", 6144, 4096, 1531)])
def test_rows_with_the_expansion_made_ahead(client, fmt, N, K, M):
    """b200q_expand + b200q_matmul_rows, rows staged or read in place (also with a longer stride), give the bits of b200q_matmul: whole weights, cut K, several panels."""
    from blazr_b200 import ops
    from blazr_b200 import synth
    if fmt in synth.GGML:
        w = client.weight_from_ggml(synth.GGML[fmt], synth.random_ggml(synth.GGML[fmt], N, K, seed=4), N, K)
    else:
        w = client.weight_from_decomposed(ops.DecomposedQuantTensor(*synth.random_awq(N, K, 128, seed=4), None, ops.DecomposedQuantMethod("awq", 128), (N, K)))
    L, P = ops.lib(), lambda t: C.c_void_p(t.data_ptr())
    n = int(L.b200q_expand_bytes(w.handle, C.c_int64(M)))
    assert n > 0
    x = torch.randn((M, K + 8), device="cuda", generator=torch.Generator(device="cuda").manual_seed(M)).half()
    want = client.quant_matmul(x[:, :K].contiguous(), w, out_dtype=torch.float32)
    panel, ws = torch.empty(n, dtype=torch.uint8, device="cuda"), torch.zeros(w.workspace_bytes(M), dtype=torch.uint8, device="cuda")
    for rows in (x[:, :K].contiguous(), x[:, :K]):
        for ready in (0, 1):
            for beside in (0, 1):
                panel.zero_()
                got = torch.zeros((M, N), device="cuda")
                ops._check(L.b200q_expand(w.handle, C.c_int64(M), P(panel), C.c_int32(beside), None))
                ops._check(L.b200q_matmul_rows(w.handle, P(rows), C.c_int32(ready), C.c_int64(M), C.c_int64(rows.stride(0)), P(panel), P(got), None, C.c_int64(N), P(ws), C.c_size_t(ws.numel()), None))
                assert torch.equal(got.view(torch.int32), want.view(torch.int32))


@pytest.mark.parametrize("F,K,M", [(8192, 2048, 1001), (5504, 2048, 777), (7168, 4096, 2047)])
def test_gated_rows(client, F, K, M):
    """The gated epilogue writes what the product and b200q_swiglu_f16 write, a step whose last tokens end inside a group of 16 included."""
    from blazr_b200 import ops, synth
    t, N = synth.GGML["Q4_K"], 2 * F
    w = client.weight_from_ggml(t, synth.random_ggml(t, N, K, seed=F), N, K)
    L, P = ops.lib(), lambda t_: C.c_void_p(t_.data_ptr())
    while L.b200q_expand_bytes(w.handle, C.c_int64(M)) == 0:   # (from where on a step expands is a rule on measured times)
        M += 256
    n = int(L.b200q_expand_bytes(w.handle, C.c_int64(M)))
    assert M < 8192 and L.b200q_gated_rows_ok(w.handle, C.c_int64(M)) == 1
    x = (3.0 * torch.randn((M, K), device="cuda", generator=torch.Generator(device="cuda").manual_seed(F))).half()
    gu = client.quant_matmul(x, w, out_dtype=torch.float32)
    want, got = torch.zeros((M, F), dtype=torch.float16, device="cuda"), torch.zeros((M + 3, F), dtype=torch.float16, device="cuda")
    ops._check(L.b200q_swiglu_f16(P(gu), C.c_int64(F), C.c_int64(M), C.c_int32(1), P(want), None))
    panel, ws = torch.empty(n, dtype=torch.uint8, device="cuda"), torch.zeros(w.workspace_bytes(M), dtype=torch.uint8, device="cuda")
    ops._check(L.b200q_expand(w.handle, C.c_int64(M), P(panel), C.c_int32(0), None))
    ops._check(L.b200q_matmul_rows(w.handle, P(x), C.c_int32(1), C.c_int64(M), C.c_int64(K), P(panel), None, P(got), C.c_int64(F), P(ws), C.c_size_t(ws.numel()), None))
    assert torch.equal(got[:M].view(torch.int16), want.view(torch.int16)) and not bool(got[M:].any())
