"""Dense products of 9 to 31 rows (csrc/seq/seq_linear.cu streams_rows): the weight-streaming kernel takes whole 16-byte rows of 512 elements and more, the f32 tiles the others.  Every
product of two bf16 numbers is exact in f32, so an output is off by the roundings of its sum alone: below K 2^-24 of the sum of sizes, and, the roundings being
independent, by sqrt(K) 2^-24 of the result in the 2-norm with a factor of four in hand (f32 rows: one more rounding of each product)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [8, 9, 13, 16, 17, 31, 32])
@pytest.mark.parametrize("N,K", [(1, 8), (65, 504), (65, 512), (257, 1000), (2048, 1032), (1025, 2048), (96, 77)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shift", [0, 1])
def test_rows_between_decode_steps_and_tiles(M, N, K, dt, shift):
    from blazr_b200 import seqops
    g = torch.Generator(device="cuda:0").manual_seed(M * N + K)
    w = (torch.randn((N, K), device="cuda:0", generator=g) / K ** 0.5).bfloat16()
    x = torch.randn((M, K + 8), device="cuda:0", generator=g).to(dt)[:, shift:shift + K]        # shift: rows that start beside a 16-byte boundary
    y = torch.full((M + 1, N + 3), 7.0, device="cuda:0")
    seqops.linear(x, w, y[:M, :N])
    ref = x.double() @ w.double().T
    tc = M >= 32 and dt == torch.bfloat16 and K % 8 == 0 and shift == 0          # the tensor cores truncate their sums
    assert ((y[:M, :N].double() - ref).norm() / ref.norm()).item() < 4 * K ** 0.5 * 2.0 ** -24 * (16 if tc else 1) + 2.0 ** -23
    assert bool((y[M] == 7).all()) and bool((y[:, N:] == 7).all())


@pytest.mark.parametrize("M", [8, 9, 16, 17, 31, 32])
@pytest.mark.parametrize("N,K", [(65, 504), (65, 512), (257, 1000), (130, 2040), (130, 2048)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shift", [0, 1])
def test_which_kernel_takes_them(M, N, K, dt, shift):
    """the kernels sum in different orders, so the bits say which one ran: the rule's, and no other"""
    from blazr_b200 import seqops
    g = torch.Generator(device="cuda:0").manual_seed(M + K)
    w = (torch.randn((N, K), device="cuda:0", generator=g) / K ** 0.5).bfloat16()
    x = torch.randn((M, K + 8), device="cuda:0", generator=g).to(dt)[:, shift:shift + K]
    y = {}
    for path in (seqops.PATH_AUTO, seqops.PATH_ROWS, seqops.PATH_TILED):
        y[path] = torch.empty((M, N), device="cuda:0")
        seqops.linear(x, w, y[path], path=path)
    streamed = M <= 8 or (M < 32 and K >= 512 and K % 8 == 0 and shift == 0 and (dt == torch.bfloat16 or M <= 16 or K >= 2048))
    tc = M >= 32 and dt == torch.bfloat16 and K % 8 == 0 and shift == 0
    assert not torch.equal(y[seqops.PATH_ROWS], y[seqops.PATH_TILED])
    assert torch.equal(y[seqops.PATH_AUTO], y[seqops.PATH_ROWS]) == streamed
    assert torch.equal(y[seqops.PATH_AUTO], y[seqops.PATH_TILED]) == (not streamed and not tc)
