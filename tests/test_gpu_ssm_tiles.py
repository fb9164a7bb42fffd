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


def scan(ops, lens, H, V, N, G, speed, plant=None):
    """(outputs, states) of the kernel and of the recurrence in float64; plant(xbc, A_log, Dp) changes the inputs first"""
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
