"""quant_matmul of one to four rows quantises x inside the matvec launch (csrc/matvec_impl.cuh, quant_prologue_t).  The records it makes are those of
quantize_act, so its results are those of quantize_act + matmul_q8 bit for bit: rows of every type, strides and alignments that rule out 16-byte loads, K
that ends inside a chunk, CTAs with part of the k-chunks, all of them, or a range that starts inside a tile, act-order weights, a bias."""
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


def same(client, w, x, M, K, perm=None):
    want = client.matmul_q8(client.quantize_act(x.contiguous(), perm), M, w)
    got = client.quant_matmul(x, w, out_dtype=torch.float32)
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))


@pytest.mark.parametrize("fmt,N,K", [("Q4_K", 128, 256), ("Q4_K", 4096, 4096), ("Q6_K", 1000, 5120), ("Q8_0", 640, 1056), ("Q8_0", 300, 96), ("Q4_K", 33000, 512), ("Q6_K", 4096, 14336)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_same_bits_as_two_launches(client, fmt, N, K, dtype):
    from blazr_b200 import synth
    t = synth.GGML[fmt]
    w = client.weight_from_ggml(t, synth.random_ggml(t, N, K, seed=1), N, K)
    g = torch.Generator(device="cuda").manual_seed(N + K)
    for M in (1, 2, 3, 4):
        rows = torch.randn((M, K + 24), device="cuda", generator=g).to(dtype)
        rows[:, 5:40] = 0.0          # a block of zeros
        for x in (rows[:, :K].contiguous(), rows[:, :K], rows[:, 3:K + 3]):
            same(client, w, x, M, K)


def test_values_that_are_not_finite(client):
    from blazr_b200 import synth
    t = synth.GGML["Q4_K"]
    w = client.weight_from_ggml(t, synth.random_ggml(t, 256, 1024, seed=2), 256, 1024)
    x = torch.randn((2, 1024), device="cuda")
    x[0, 7], x[1, 300] = float("inf"), float("nan")
    want = client.matmul_q8(client.quantize_act(x), 2, w)
    got = client.quant_matmul(x, w)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.nan_to_num(got), torch.nan_to_num(want))


@pytest.mark.parametrize("fmt", ["GPTQ_ACT", "GPTQ", "AWQ_G64"])
def test_act_order_and_bias(client, fmt):
    from qcases import Case
    c = Case(client, fmt, 384, 1024, seed=3, bias=fmt.startswith("GPTQ"))
    perm = None if c.perm is None else torch.from_numpy(np.ascontiguousarray(c.perm, dtype=np.int32)).cuda()
    for M in (1, 4):
        same(client, c.w, torch.randn((M, 1024), device="cuda"), M, 1024, perm)


@pytest.mark.parametrize("N", [2048, 4096, 20480])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_results_over_the_rows_they_come_from(client, N, dtype):
    """y on x itself, y a row further on in x's buffer, y of a wider type that begins inside x: what the call gives with an output of its own"""
    from blazr_b200 import synth
    K = min(N, 4096)
    t = synth.GGML["Q4_K"]
    w = client.weight_from_ggml(t, synth.random_ggml(t, N, K, seed=6), N, K)
    g = torch.Generator(device="cuda").manual_seed(N)
    for M in (1, 2, 3, 4):
        for rep in range(20):
            buf = torch.randn((M + 2, N), device="cuda", generator=g).to(dtype)
            x = buf[:M, :K]
            want = client.quant_matmul(x.clone(), w, out_dtype=dtype)
            for row in (0, 1):
                b = buf.clone()
                got = client.quant_matmul(b[:M, :K], w, out=b[row:row + M])
                assert torch.equal(got, want), (M, rep, row)
            flat = torch.zeros(2 * M * N + 64, device="cuda")            # f32
            src = flat.view(dtype)[:M * K].view(M, K)
            src.copy_(x)
            wide = client.quant_matmul(x.clone(), w, out_dtype=torch.float32)
            assert torch.equal(client.quant_matmul(src, w, out=flat[32:32 + M * N].view(M, N)), wide)


def test_rows_side_by_side_in_one_buffer(client):
    """x and y as columns of one buffer share no bytes: one launch, as ever, and the same bits"""
    from blazr_b200 import ops, synth
    t = synth.GGML["Q6_K"]
    w = client.weight_from_ggml(t, synth.random_ggml(t, 1024, 2048, seed=7), 1024, 2048)
    for first in (0, 1024):
        buf = torch.randn((4, 3072), device="cuda")
        x, y = buf[:, first:first + 2048], buf[:, 2048 if first == 0 else 0:][:, :1024]
        want = client.quant_matmul(x.clone(), w)
        n0 = ops.launch_count()
        assert torch.equal(client.quant_matmul(x, w, out=y), want) and ops.launch_count() - n0 == 1
