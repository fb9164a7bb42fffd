"""The dequant-GEMM on pairs of SMs (csrc/gemm_pair.cuh) where it can go wrong: every format, one chunk of K and several, one tile and several to a pair of
CTAs, token tiles that end inside 16, 32 and 64 columns, f32 / f16 / bf16 rows with any start and stride, results in every type.  It expands weights to the
operands of the other two kernels and sums in their order of k, so its results are theirs, bit for bit (rows of 160 take the fused kernel; 80 and more
weight tiles are not cut along K there).  Bound against 64 bits: weights and activations are rounded to f16 (2^-11 each), see test_gpu_gemm_wide.py."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
FORMATS = ["Q4_K", "Q6_K", "Q8_0", "Q5_K", "Q4_1", "Q5_1", "Q2_K", "Q3_K", "IQ4_XS", "TQ2_0", "IQ2_S", "AWQ", "GPTQ"]


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
        return client.weight_from_ggml(t, synth.random_ggml(t, N, K, seed=N + K), N, K), None
    if fmt == "AWQ":
        return client.weight_from_decomposed(ops.DecomposedQuantTensor(*synth.random_awq(N, K, 128, seed=5), None, ops.DecomposedQuantMethod("awq", 128), (N, K))), None
    qw, sc, qz, gi, b = synth.random_gptq(N, K, 128, seed=6, act_order=True, bias=True)
    return client.weight_from_decomposed(ops.DecomposedQuantTensor(qw, sc, qz, gi, ops.DecomposedQuantMethod("gptq", 128), (N, K), bias=b)), torch.from_numpy(np.asarray(b)).cuda()


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("N,K,M", [(10240, 256, 513), (10240, 1024, 785)])
def test_the_bits_of_the_fused_kernel(client, fmt, N, K, M):
    from blazr_b200 import ops
    w, _ = weight(client, fmt, N, K)
    x = torch.randn((M, K + 3), device="cuda:0", generator=torch.Generator(device="cuda:0").manual_seed(1)).half()[:, 1:K + 1]
    y = torch.full((M + 1, N + 8), 7.0, dtype=torch.float16, device="cuda:0")
    n0 = ops.launch_count()
    client.quant_matmul(x, w, out=y[:M, :N])
    assert ops.launch_count() - n0 == 2                                   # rows staged, one GEMM
    for a in range(0, M, 160):
        assert torch.equal(y[a:min(a + 160, M), :N], client.quant_matmul(x[a:a + 160].contiguous(), w))
    assert bool((y[M] == 7).all()) and bool((y[:, N:] == 7).all())


@pytest.mark.parametrize("fmt", FORMATS)
def test_the_bits_of_the_fused_kernel_in_f32(client, fmt):
    """unrounded: the sums themselves are the same (int4 weights with f32 results are expanded where the workspace has room: they bring staged rows' worth)"""
    from blazr_b200 import ops
    N, K, M = 10240, 1024, 785
    w, _ = weight(client, fmt, N, K)
    x = torch.randn((M, K), device="cuda:0", generator=torch.Generator(device="cuda:0").manual_seed(4))
    ws = torch.zeros(1024 * w.K_pad * 2, dtype=torch.uint8, device="cuda:0")      # what the fused kernel asks for: four tiles of up to 256 rows
    n0 = ops.launch_count()
    y = client.quant_matmul(x, w, workspace=ws)
    assert ops.launch_count() - n0 == 2
    for a in range(0, M, 160):
        assert torch.equal(y[a:a + 160], client.quant_matmul(x[a:a + 160], w))


@pytest.mark.parametrize("fmt,N,K,M", [("Q4_K", 12800, 512, 512), ("Q6_K", 2560, 256, 4099), ("Q8_0", 5120, 1056, 1537), ("GPTQ", 20480, 512, 1300), ("AWQ", 28672, 4096, 250)])
@pytest.mark.parametrize("dt", [torch.float32, torch.float16, torch.bfloat16])
def test_against_the_dequantized_weight(client, fmt, N, K, M, dt):
    w, b = weight(client, fmt, N, K)
    x = torch.randn((M, K), device="cuda:0", generator=torch.Generator(device="cuda:0").manual_seed(2)).to(dt)
    ref = x.double() @ client.dequantize(w).double().T + (b.double() if b is not None else 0.0)
    ws = torch.zeros(w.workspace_bytes(M), dtype=torch.uint8, device="cuda:0")
    for out in (torch.float32, torch.float16, torch.bfloat16):
        y = client.quant_matmul(x, w, out_dtype=out, workspace=ws)
        assert ((y.double() - ref).norm() / ref.norm()).item() < 8.3e-4 + {torch.float32: 0.0, torch.float16: 2 ** -11, torch.bfloat16: 2 ** -9}[out]
    from blazr_b200 import ops
    ops.check_device_errors()


@pytest.mark.parametrize("fmt,N,K,M", [("Q8_0", 14336, 4096, 800), ("Q8_0", 10240, 8192, 800), ("Q6_K", 4096, 14336, 1300), ("AWQ", 8192, 8192, 640)])
def test_a_chunk_is_read_before_its_slot_is_refilled(client, fmt, N, K, M):
    """narrow token tiles over a long K: the expansion is the bound, two to four slots of packed chunks turn over as fast as they can, call behind call"""
    w, _ = weight(client, fmt, N, K)
    x = torch.randn((M, K), device="cuda:0", generator=torch.Generator(device="cuda:0").manual_seed(3)).half()
    ref = x.double() @ client.dequantize(w).double().T
    ws = w.workspace(M)
    outs = [torch.empty((M, N), dtype=torch.float16, device="cuda:0") for _ in range(8)]
    for _ in range(8):
        for y in outs:
            client.quant_matmul(x, w, out=y, workspace=ws)
        for y in outs:
            assert torch.equal(y, outs[0])
    # one unit of 32 k that is another chunk's moves its row by sqrt(64 / K) of the result, 6.7 % and more; the roundings of 2^-11 each stay below 1 % at any element
    assert ((outs[0].double() - ref).abs().max() / ref.square().mean().sqrt()).item() < 2e-2


@pytest.mark.parametrize("fmt,N,K,M,launches", [("IQ4_XS", 2560, 2048, 2048, 3), ("Q3_K", 2560, 2048, 2048, 3), ("IQ4_XS", 14336, 4096, 2048, 5), ("Q4_K", 5120, 1280, 4096, 3),
                                                ("Q6_K", 14336, 4096, 2048, 2), ("AWQ", 6144, 4096, 1531, 2), ("Q8_0", 6144, 4096, 900, 2)])
def test_which_products_are_expanded_ahead(client, fmt, N, K, M, launches):
    """the calls that the expansion takes by 4 to 21 % are its own again, those that the paired kernel takes by 10 % and more stay (csrc/gemm_pair.cu gemm_pair_wins)"""
    from blazr_b200 import ops
    w, _ = weight(client, fmt, N, K)
    x = torch.randn((M, K), device="cuda:0", generator=torch.Generator(device="cuda:0").manual_seed(5)).half()
    n0 = ops.launch_count()
    y = client.quant_matmul(x, w, workspace=w.workspace(M))
    assert ops.launch_count() - n0 == launches
    least = torch.zeros(-(-M // 256) * 256 * w.K_pad * 2, dtype=torch.uint8, device="cuda:0")       # no room for an expansion
    assert torch.equal(y, client.quant_matmul(x, w, workspace=least))
