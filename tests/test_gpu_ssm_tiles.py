"""The state-space scan of long steps as tile products (csrc/seq/seq_ssm_tc.cu) against the recurrence in float64: portions that end inside a segment and
inside a block of 32, state and column counts that end inside a tile, one to many heads per group, carried states, fast and slow decays.

Bound: f32 products and sums in another order than the recurrence's; the recurrence is tested at 2e-5 of the largest value, this at 3e-6."""
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


def scan(ops, lens, H, V, N, G, speed, plant=None, gates=None):
    """(outputs, states) of the kernel and of the recurrence in float64; plant(xbc, A_log, Dp) and gates(proj) change the inputs first"""
    from blazr_b200.batch import StepEntry, build_step
    g = torch.Generator(device=DEV)
    g.manual_seed(H * V + N)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    T, inner, B = sum(lens), H * V, len(lens)
    pos0 = [0 if i % 2 == 0 else 64 for i in range(B)]
    sa = build_step([StepEntry([0] * n, p, B - 1 - i, list(range(-(-(p + n) // 16)))) for i, (n, p) in enumerate(zip(lens, pos0))], 16)
    t = {k: torch.from_numpy(getattr(sa, k)).to(DEV) for k in ("tok_ent", "tok_pos", "ent_start", "ent_slot", "ent_pos0", "block_table")}
    st = ops.StepDesc(*(t[k].data_ptr() for k in ("tok_ent", "tok_pos", "ent_start", "ent_slot", "ent_pos0", "block_table")), sa.T, sa.B, sa.block_table.shape[1], 16)
    ld, ldx = -(-(2 * inner + 2 * G * N + H) // 4) * 4, -(-(inner + 2 * G * N) // 4) * 4
    proj, xbc, A_log, Dp, dtb = rnd(T, ld), rnd(T, ldx), 0.7 * rnd(H) + speed, rnd(H), rnd(H) - 1.0
    dt0 = 2 * inner + 2 * G * N
    if plant is not None:
        plant(xbc, A_log, Dp)
    if gates is not None:
        gates(proj)
    state = rnd(B, H, N, V)
    ref_state, ref = state.double().clone(), torch.empty(T, inner, dtype=torch.float64, device=DEV)
    x = xbc[:, :inner].double().reshape(T, H, V)
    Bm, Cm = (xbc[:, inner + i * G * N:inner + (i + 1) * G * N].double().reshape(T, G, N).repeat_interleave(H // G, 1) for i in (0, 1))
    dt = torch.nn.functional.softplus(proj[:, dt0:dt0 + H].double() + dtb.double())
    dec = torch.exp(-torch.exp(A_log.double()) * dt)
    r = 0
    for i, n in enumerate(lens):
        S = ref_state[B - 1 - i]
        if pos0[i] == 0:
            S.zero_()
        for k in range(r, r + n):
            S.mul_(dec[k][:, None, None]).add_(Bm[k][:, :, None] * (dt[k][:, None] * x[k])[:, None, :])
            y = torch.einsum("hn,hnv->hv", Cm[k], S) + Dp.double()[:, None] * x[k]
            ref[k] = (y.reshape(-1) * torch.nn.functional.silu(proj[k, :inner].double()))
        r += n
    out = torch.empty(T, inner, device=DEV)
    scratch = torch.empty(ops.ssm_scratch_floats(T, B, H, V, N), device=DEV)
    assert (scratch.numel() > 0) == (T > 128)
    ops.ssm_scan(proj, 0, dt0, xbc, A_log, Dp, dtb, state, st, H, V, N, G, out, scratch)
    return (out, ref), (state, ref_state)


@pytest.mark.parametrize("lens,H,V,N,G", [([129], 2, 64, 128, 1), ([300, 31], 6, 68, 36, 2), ([257, 1, 130], 5, 4, 64, 5), ([700], 9, 64, 100, 1), ([128, 128], 4, 132, 48, 4)])
@pytest.mark.parametrize("speed", [-8.0, 0.0, 3.0])
def test_against_the_recurrence(ops, lens, H, V, N, G, speed):
    for got, want in scan(ops, lens, H, V, N, G, speed):
        err = (got.double() - want).abs().max().item() / want.abs().max().item()
        assert err < 3e-6, err


@pytest.mark.parametrize("lens,H,V,N,G", [([32], 2, 64, 128, 1), ([41], 9, 68, 36, 3), ([128], 4, 4, 100, 1), ([90, 1, 33], 3, 64, 64, 3), ([64, 64], 16, 132, 128, 2), ([31], 2, 64, 128, 1)])
@pytest.mark.parametrize("speed", [-8.0, 0.0, 3.0])
def test_entries_of_one_segment(ops, lens, H, V, N, G, speed):
    """Steps of up to 128 tokens: outputs from the slots' states (new and carried), then the states; the last one stays on the recurrence."""
    test_against_the_recurrence(ops, lens, H, V, N, G, speed)


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("token", [0, 17, 31, 32, 200, 255])
def test_a_value_that_is_not_finite_reaches_no_earlier_token(ops, value, token, T=256):
    """Head 1, column 5 of one token: the outputs of the tokens before it, of the other columns and of the other heads stay what they are."""
    def plant(xbc, A_log, Dp):
        xbc[token, 64 + 5] = value
    (out, ref), (state, ref_state) = scan(ops, [T], 4, 64, 64, 2, 0.0, plant)
    top = ref[torch.isfinite(ref)].abs().max().item()
    fine = torch.isfinite(ref)
    assert bool(fine[:token].all()) and not bool(fine[token, 64 + 5]) and torch.equal(torch.isfinite(out), fine)
    assert ((out.double() - ref)[fine].abs().max().item()) / top < 3e-6
    fine = torch.isfinite(ref_state)
    assert torch.equal(torch.isfinite(state), fine) and ((state.double() - ref_state)[fine].abs().max().item()) / ref_state[fine].abs().max().item() < 3e-6


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("token", [0, 17, 63])
def test_a_value_that_is_not_finite_in_one_segment(ops, value, token):
    test_a_value_that_is_not_finite_reaches_no_earlier_token(ops, value, token, 64)


def test_decays_that_forget_at_once(ops):
    """A head whose rate overflows f32 (exp(100)) keeps nothing of the token before, as the recurrence has it; the heads beside it are what they are."""
    def plant(xbc, A_log, Dp):
        A_log[1], A_log[2] = 100.0, 12.0
    for got, want in scan(ops, [300, 40], 4, 64, 64, 2, 0.0, plant):
        assert bool(torch.isfinite(got).all())
        assert (got.double() - want).abs().max().item() / want.abs().max().item() < 3e-6


@pytest.mark.parametrize("lens", [[31], [32], [128], [300]])
def test_gates_of_every_size(ops, lens):
    """Outputs that are x silu(z) alone (no states, D 1, x 1), z over all of f32: the recurrence (31 tokens) and the tiles give the same value for the same gate.
    Bound: z / (1 + exp(-z)) with an exponential, a sum and a quotient in f32, 2 + 1/2 + 1/2 units of 2^-23; what lies below f32's normal numbers may be 0."""
    H, V = 4, 64
    z = torch.cat([torch.linspace(-104, 104, 4001), torch.tensor([0.0, -0.0, 1e-30, -1e-30, 1e30, -1e30, 3e38, -3e38, float("inf"), -float("inf"), float("nan")]), -torch.logspace(0, 38.4, 900),
                   torch.logspace(-38, 38, 900)]).to(DEV)
    seen = torch.empty_like(z)
    per = sum(lens) * H * V
    for at in range(0, z.numel(), per):
        part = torch.zeros(per, device=DEV)
        n = min(per, z.numel() - at)
        part[:n] = z[at:at + n]

        def plant(xbc, A_log, Dp):
            xbc[:, :H * V], xbc[:, H * V:] = 1.0, 0.0
            Dp.fill_(1.0)

        def gates(proj):
            proj[:, :H * V] = part.view(sum(lens), H * V)
        (out, _), _ = scan(ops, lens, H, V, 64, 2, 0.0, plant, gates)
        seen[at:at + n] = out.reshape(-1)[:n]
    want = z.double() / (1 + torch.exp(-z.double()))
    wild = z.isnan() | (z == -float("inf"))                       # -inf / inf, as the quotient has it
    assert torch.equal(seen.isnan(), wild)
    tame = ~wild & want.isfinite()
    assert torch.equal(seen[~wild & ~tame], want[~wild & ~tame].float())
    assert ((seen.double() - want).abs()[tame] <= 3.0 * 2.0 ** -23 * want.abs()[tame] + 2.0 ** -126 * 128).all()


@pytest.mark.parametrize("lens", [[20], [20, 44], [32], [40], [129]])
def test_a_rate_that_is_not_a_number(ops, lens):
    """A head whose rate is NaN has NaN outputs and states from its first token on, as the recurrence has it; the other heads are what they are."""
    def plant(xbc, A_log, Dp):
        A_log[1] = float("nan")
    for got, want in scan(ops, lens, 4, 64, 64, 2, 0.0, plant):
        fine = want.isfinite()
        assert torch.equal(got.isfinite(), fine) and bool((~fine).any())
        assert (got.double() - want).abs()[fine].max().item() / want[fine].abs().max().item() < 3e-6
