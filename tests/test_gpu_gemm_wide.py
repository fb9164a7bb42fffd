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
