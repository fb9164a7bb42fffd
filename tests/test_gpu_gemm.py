"""GPU parity tests for the tcgen05/TMEM dequant-GEMM path (M >= 5: batched decode and prefill) against
the CPU oracle's f32 flavour A (dequantized weights x f32 activations, double accumulation).

Tolerance: max-abs error / max-abs reference <= 1e-2.  The kernel rounds weights and
activations to f16 (2^-11 relative each) and accumulates in f32, so the observed error is ~1e-3.
"""
import numpy as np
import pytest
import torch

from blazr_b200 import ops, synth
from qcases import ALL, Case

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(120)]
TOL = 1e-2


def rel_err(y, ref):
    return float(np.abs(y.astype(np.float64) - ref.astype(np.float64)).max() / max(np.abs(ref).max(), 1e-30))


@pytest.mark.parametrize("fmt", ALL)
@pytest.mark.parametrize("NKM", [(128, 256, 32), (256, 1024, 5), (200, 768, 100), (1408, 2048, 32), (384, 4096, 256)])
def test_gemm_vs_oracle(client, fmt, NKM):
    N, K, M = NKM
    c = Case(client, fmt, N, K, seed=N + K + M)
    x = synth.random_act(M, K, seed=M)
    y = client.quant_matmul(torch.from_numpy(x).cuda(), c.w, path=ops.PATH_GEMM).cpu().numpy()
    assert y.shape == (M, N)
    assert np.isfinite(y).all()
    assert rel_err(y, c.oracle_a(x)) < TOL


@pytest.mark.parametrize("fmt", ["Q4_K", "Q6_K", "Q8_0", "AWQ"])
def test_gemm_multiple_m_tiles_and_ragged_m(client, fmt):
    N, K, M = 640, 1024, 300  # two m-tiles of 160 rows (last one ragged) x 5 n-tiles: persistent loop
    c = Case(client, fmt, N, K, seed=4)
    x = synth.random_act(M, K, seed=2)
    y = client.quant_matmul(torch.from_numpy(x).cuda(), c.w).cpu().numpy()  # auto dispatch -> GEMM
    assert rel_err(y, c.oracle_a(x)) < TOL


def test_gemm_many_tiles_persistent(client):
    """more tiles than SMs: each CTA walks several (n-tile, m-tile) pairs and re-uses its TMEM"""
    N, K, M = 128 * 40, 512, 1024  # 40 x 4 = 160 tiles
    c = Case(client, "Q4_K", N, K, seed=6)
    x = synth.random_act(M, K, seed=3)
    y = client.quant_matmul(torch.from_numpy(x).cuda(), c.w).cpu().numpy()
    assert rel_err(y, c.oracle_a(x)) < TOL


def test_gemm_matches_matvec_path(client):
    """M = 4 through both kernels: int8-activation dp4a path and f16 tensor path agree within tolerance"""
    N, K, M = 512, 2048, 4
    c = Case(client, "Q6_K", N, K, seed=8)
    x = torch.from_numpy(synth.random_act(M, K)).cuda()
    y1 = client.quant_matmul(x, c.w, path=ops.PATH_MATVEC).cpu().numpy()
    y2 = client.quant_matmul(x, c.w, path=ops.PATH_GEMM).cpu().numpy()
    assert rel_err(y2, y1) < TOL


def test_gemm_half_io_bias_and_strides(client):
    N, K, M = 256, 1024, 48
    c = Case(client, "GPTQ", N, K, seed=9, bias=True)
    xbig = torch.from_numpy(synth.random_act(M, K + 8)).cuda().half()
    x = xbig[:, :K]
    ybig = torch.zeros((M, N + 16), device="cuda", dtype=torch.float16)
    client.quant_matmul(x, c.w, out=ybig[:, :N])
    ref = c.oracle_a(x.float().cpu().numpy())
    assert rel_err(ybig[:, :N].float().cpu().numpy(), ref) < TOL
    assert float(ybig[:, N:].abs().max()) == 0.0


def test_gemm_act_order_permutation(client):
    N, K, M = 256, 1024, 64
    c = Case(client, "GPTQ_ACT", N, K, seed=10)
    x = synth.random_act(M, K, seed=1)
    y = client.quant_matmul(torch.from_numpy(x).cuda(), c.w).cpu().numpy()
    assert rel_err(y, c.oracle_a(x)) < TOL


def test_gemm_prefill_shape_property(client):
    """A projection's shape (Mistral-7B q_proj, S = 2048): check sampled rows against the oracle and
    linearity in the activations (scaling x by 2 is exact in f16/f32)"""
    N, K, M = 4096, 4096, 2048
    c = Case(client, "Q6_K", N, K, seed=42)
    x = torch.from_numpy(synth.random_act(M, K, seed=4)).cuda()
    y = client.quant_matmul(x, c.w)
    y2 = client.quant_matmul(2.0 * x, c.w)
    assert torch.allclose(y2, 2.0 * y, rtol=1e-3, atol=1e-3)  # f16 staging: subnormal inputs round differently
    rows = [0, 1, 777, 2047]
    ref = c.oracle_a(x[rows].cpu().numpy())
    assert rel_err(y[rows].cpu().numpy(), ref) < TOL


@pytest.mark.parametrize("fmt,bias", [("Q6_K", False), ("Q4_K", False), ("GPTQ", True)])
def test_gemm_tail_split_k_wave_quantisation(client, fmt, bias, monkeypatch):
    """(opt-in path, B200Q_GEMM_TAIL=1 -- the switch is read once per process, so the default suite exercises the plain
    persistent loop on this shape and `B200Q_GEMM_TAIL=1 pytest -k tail_split` the split form; both have run green)
    wide-M launch whose tile count is not a multiple of the SM count: the tiles of the last, partial wave are split along K
    (tail split-K: 19 x 8 = 152 tiles on 148 SMs -> 4 tail tiles x 4 splits), partial accumulators reduced by a second kernel;
    ragged M so the last activation tile is partly empty"""
    N, K, M = 128 * 19, 2048, 2000
    c = Case(client, fmt, N, K, seed=12, bias=bias) if bias else Case(client, fmt, N, K, seed=12)
    x = synth.random_act(M, K, seed=5)
    y = client.quant_matmul(torch.from_numpy(x).cuda(), c.w).cpu().numpy()
    assert rel_err(y, c.oracle_a(x)) < TOL


# One chunk of K per item and three or more items per CTA (148 SMs: more than 37 888 rows): the warps that expand the weight, which also store the CTA's last
# item, reach it up to three items ahead of the products.  A row's result does not depend on the rows beside it, so it is that of the same row in a
# weight whose CTAs have one item each, bit for bit.
@pytest.mark.parametrize("fmt,K", [("Q4_K", 256), ("Q6_K", 256), ("Q8_0", 96), ("Q8_0", 256), ("AWQ", 256), ("Q5_K", 256), ("Q4_1", 96), ("Q3_K", 256), ("IQ4_XS", 256), ("TQ2_0", 256)])
@pytest.mark.parametrize("N", [37904, 57000, 130000])
def test_gemm_many_items_of_one_chunk(client, fmt, K, N):
    if fmt == "AWQ":
        qw, sc, zr = synth.random_awq(N, K, 128, seed=N)
        dq = ops.DecomposedQuantTensor(qw, sc, zr, None, ops.DecomposedQuantMethod("awq", 128), (N, K))
        part = lambda a, b: client.weight_from_decomposed(dq, rows=(a, b))
    else:
        blk = synth.random_ggml(synth.GGML[fmt], N, K, seed=N)
        part = lambda a, b: client.weight_from_ggml(synth.GGML[fmt], np.ascontiguousarray(blk[a:b]), b - a, K)
    w, cuts = part(0, N), list(range(0, N, 18432)) + [N]                 # 144 tiles of 128 rows
    small = [part(a, b) for a, b in zip(cuts, cuts[1:])]
    for M in (5, 32, 64, 128):
        xs = [torch.randn((M, K), device="cuda", generator=torch.Generator(device="cuda").manual_seed(i)) for i in range(4)]
        ys = [client.quant_matmul(x, w) for x in xs]                       # back to back: each is launched beside the end of the one before
        for x, y in zip(xs, ys):
            want = torch.cat([client.quant_matmul(x, s) for s in small], 1)
            assert torch.equal(y.view(torch.int32), want.view(torch.int32)), (fmt, N, M)


@pytest.mark.parametrize("N,K,M,parts", [(14336, 4096, 5, 5), (14336, 4096, 16, 5), (28672, 4096, 16, 3), (10240, 8192, 5, 7), (10240, 8192, 16, 5), (10240, 8192, 128, 3), (4096, 4096, 32, 4)])
def test_skinny_products_are_cut_along_k(client, N, K, M, parts):
    """Weights of one, 65504 in the first chunk of K and 1 / 64 in the others.  Beside the large sum (2^24: its unit is 1) the 16 products that a tensor-core
    step adds (1 / 4) are lost; the parts of K that do not hold the first chunk arrive whole, 4 for each of their chunks."""
    blk = np.zeros((N, K // 32, 34), np.uint8)
    blk[:, :, :2] = np.frombuffer(np.float16(1.0).tobytes(), np.uint8)
    blk[:, :, 2:] = 1
    w = client.weight_from_ggml(8, blk.reshape(N, -1), N, K)
    x = torch.full((M, K), 2.0 ** -6, device="cuda")
    x[:, :256] = 65504.0
    more = client.quant_matmul(x, w).double() - 256 * 65504.0
    chunks = K // 256
    assert more.min().item() >= 4 * (chunks - -(-chunks // parts)) and more.max().item() <= 4 * (chunks - 1)
