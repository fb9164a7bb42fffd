"""The paired-SM GEMM (csrc/seq/tc_pair.cuh) at the sizes where its tiles can go wrong, against float64: one token row past a tile, weight rows
that end inside a pair's second half, k that is not a whole slab, more tiles than pairs (the accumulator buffers alternate), groups without
rows, groups of one row, more groups than lanes in the scan.

Bound: f32 sums of K bf16 products differ from the exact sum by at most K * 2^-24 of the sum of magnitudes, which for these inputs is below
K * 2^-24 * sqrt(K) of the result's rms; 5e-6 covers K <= 1032 with the tensor core's own rounding.  bf16 outputs add half a unit, 2^-9."""
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


def rnd(*shape, seed=0, scale=1.0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale


def close(got, ref, tol):
    err = (got.double().cpu() - ref).abs().max().item() / max(ref.abs().max().item(), 1e-30)
    assert err < tol, f"relative error {err:.3e} >= {tol}"


@pytest.mark.parametrize("M,N,K", [(129, 257, 8), (257, 514, 72), (300, 1000, 1032), (1, 256, 64), (2500, 2300, 136), (4100, 130, 64)])
def test_linear(ops, M, N, K):
    x, w = rnd(M, K + 8, seed=1).bfloat16()[:, :K], rnd(N, K, seed=2, scale=K ** -0.5).bfloat16()
    ref = x.double() @ w.double().T
    y = torch.full((M + 1, N + 3), 7.0, device=DEV)
    ops.linear(x.to(DEV), w.to(DEV), y[:M, :N], ops.PATH_TC, silu=(N // 3, N // 2))
    ref[:, N // 3:N // 2] = torch.nn.functional.silu(ref[:, N // 3:N // 2])
    close(y[:M, :N], ref, 5e-6)
    assert bool((y[:, N:] == 7.0).all()) and bool((y[M] == 7.0).all()) and ops.error_flags() == 0


@pytest.mark.parametrize("M,F,ldo", [(130, 64, 64), (257, 129, 131), (300, 130, 132), (1030, 1100, 1102)])
@pytest.mark.parametrize("kind", ["swish_clamp", "gelu_tanh"])
def test_gated_epilogue_in_bf16(ops, M, F, ldo, kind):
    K = 200
    x = rnd(M, K, seed=3, scale=3.0).bfloat16()
    w = rnd(2 * F, K, seed=4, scale=K ** -0.5).bfloat16()
    x[0, 0], w[0, 0], w[1, 0] = 300.0, 40.0, 2.0        # one gate so large (and, on the next row, so negative) that its sigmoid saturates
    x[1, 0] = -300.0
    z = x.double() @ w.double().T
    g, u = z[:, 0::2], z[:, 1::2]
    if kind == "swish_clamp":
        g, u = g.clamp(max=7.0), u.clamp(-7.0, 7.0)
        ref = g * torch.sigmoid(1.702 * g) * (u + 1.0)
    else:
        ref = torch.nn.functional.gelu(g, approximate="tanh") * u
    out = torch.full((M, ldo), 3.0, device=DEV, dtype=torch.bfloat16)
    ops.linear_act(x.to(DEV), w.to(DEV), ops.ACT_KINDS[kind], out[:, :F], 7.0, 1.702, 1.0)
    err = (out[:, :F].double().cpu() - ref).abs() / (ref.abs() + 1e-3 * z.abs().max())
    assert err.max().item() < 2 ** -8 and bool((out[:, F:] == 3.0).all()) and ops.error_flags() == 0


@pytest.mark.parametrize("sizes", [[0, 1, 300, 0, 129, 0], [5] * 40 + [0] * 30 + [700], [257]])
@pytest.mark.parametrize("act", ["none", "swish_clamp"])
def test_grouped_rows(ops, sizes, act):
    E, N, K = len(sizes), 200, 72
    rows = sum(sizes)
    x, w = rnd(rows, K, seed=5).bfloat16(), rnd(E, N, K, seed=6, scale=K ** -0.5).bfloat16()
    offs = torch.zeros(E + 1, dtype=torch.int32)
    offs[1:] = torch.tensor(sizes).cumsum(0)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(sizes)).to(torch.int32)
    ref = torch.cat([x[offs[e]:offs[e + 1]].double() @ w[e].double().T for e in range(E)])
    kind, No, dt = ops.ACT_NONE, N, torch.float32
    if act != "none":
        kind, No, dt = ops.ACT_SWISH_CLAMP, N // 2, torch.bfloat16
        g, u = ref[:, 0::2].clamp(max=7.0), ref[:, 1::2].clamp(-7.0, 7.0)
        ref = g * torch.sigmoid(1.702 * g) * (u + 1.0)
    out = torch.full((rows + 1, No), 3.0, device=DEV, dtype=dt)
    order = torch.arange(rows, dtype=torch.int32, device=DEV)
    ops.moe_linear(x.to(DEV), 0, w.to(DEV), ids.to(DEV), order, offs.to(DEV), rows, kind, out, 7.0, 1.702, 1.0)
    close(out[:rows].float(), ref, 5e-6 if act == "none" else 2 ** -8)
    assert bool((out[rows] == 3.0).all()) and ops.error_flags() == 0


@pytest.mark.parametrize("kind", ["swish_clamp", "gelu_tanh"])
def test_gates_far_below_zero(ops, kind):
    """The sigmoid of a gate falls to zero, so that nothing is left of a product whose gate is large: gates of -50 to -1e36 and one that is -inf."""
    M, F, K = 300, 64, 64
    x, w = torch.zeros(M, K).bfloat16(), torch.zeros(2 * F, K).bfloat16()
    gates = [-50.0, -80.0, -86.0, -87.5, -90.0, -1e3, -1e9, -1e18, -1e30, -1e36, float("-inf")]
    for i, v in enumerate(gates):
        x[i, 0] = v
    x[:, 1] = 1.0
    w[0::2, 0] = 1.0
    w[1::2, 1] = 2.0
    g, u = x[:, :1].double(), torch.full((M, F), 2.0, dtype=torch.float64)
    if kind == "swish_clamp":
        ref = g * torch.sigmoid(g) * (u + 1.0)
    else:
        ref = g * torch.sigmoid(1.5957691216057308 * (g + 0.044715 * g ** 3)) * u
    out = torch.full((M, F), 3.0, device=DEV, dtype=torch.bfloat16)
    ops.linear_act(x.to(DEV), w.to(DEV), ops.ACT_KINDS[kind], out, 3e38, 1.0, 1.0)
    got = out.double().cpu()
    n = len(gates)
    assert torch.isnan(got[n - 1]).all() and torch.isnan(ref[n - 1]).all()
    assert ((got[:n - 1] - ref[:n - 1]).abs() <= ref[:n - 1].abs() * 2 ** -8 + 1e-36).all() and (got[n:] == 0).all()


def test_more_experts_than_the_pair_kernel_lists(ops):
    """A bank of more than 1024 experts keeps the one-SM kernel, with its grouped and gated epilogues."""
    E, N, K = 1030, 64, 40
    sizes = [(3 * e) % 5 if e % 7 else 0 for e in range(E)]
    rows = sum(sizes)
    x, w = rnd(rows, K, seed=8).bfloat16(), rnd(E, N, K, seed=9, scale=K ** -0.5).bfloat16()
    offs = torch.zeros(E + 1, dtype=torch.int32)
    offs[1:] = torch.tensor(sizes).cumsum(0)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(sizes)).to(torch.int32)
    z = torch.einsum("rk,rnk->rn", x.double(), w.double()[ids.long()])
    g, u = z[:, 0::2].clamp(max=7.0), z[:, 1::2].clamp(-7.0, 7.0)
    order = torch.arange(rows, dtype=torch.int32, device=DEV)
    for kind, ref, dt, tol in ((ops.ACT_NONE, z, torch.float32, 5e-6), (ops.ACT_SWISH_CLAMP, g * torch.sigmoid(1.702 * g) * (u + 1.0), torch.bfloat16, 2 ** -8)):
        out = torch.full((rows + 1, ref.shape[1]), 3.0, device=DEV, dtype=dt)
        ops.moe_linear(x.to(DEV), 0, w.to(DEV), ids.to(DEV), order, offs.to(DEV), rows, kind, out, 7.0, 1.702, 1.0)
        close(out[:rows].float(), ref, tol)
        assert bool((out[rows] == 3.0).all()) and ops.error_flags() == 0
