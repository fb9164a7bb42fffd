"""The choice of experts and the gathering of rows for many tokens: the forms of several tokens to a block equal the block-per-token forms, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from blazr_b200 import seqops
    return seqops


# 1023 tokens: the last block-per-token size; 1024 .. 1031: whole and ragged last blocks of eight; 1024 experts: eight tokens' scores exceed the shared memory
@pytest.mark.parametrize("T", [1023, 1024, 1025, 1031, 4099])
@pytest.mark.parametrize("E,groups,keep,top,kind", [(32, 1, 1, 4, "ROUTE_SOFTMAX"), (5, 5, 3, 3, "ROUTE_SIGMOID"), (512, 8, 4, 8, "ROUTE_SIGMOID"), (1024, 1, 1, 6, "ROUTE_TOP_SOFTMAX")])
def test_choice(ops, T, E, groups, keep, top, kind):
    g = torch.Generator(device=DEV).manual_seed(T + E)
    z = torch.randn(T, E + 3, device=DEV, generator=g)
    z[::7, :] = 0.25                                      # ties
    z[T - 1, 1] = float("inf")
    z = z[:, :E]
    corr = torch.randn(E, device=DEV, generator=g) * 0.1

    def run(zz, counts):
        ids = torch.full((zz.shape[0] * top,), -1, dtype=torch.int32, device=DEV)
        w = torch.full((zz.shape[0] * top,), -1.0, device=DEV)
        ops.moe_route_ex(zz, E, groups, keep, top, getattr(ops, kind), corr, ids, w, counts)
        return ids, w

    cnt = torch.full((E,), 99, dtype=torch.int32, device=DEV)
    ids, w = run(z, cnt)
    parts = [run(z[i:i + 500], None) for i in range(0, T, 500)]
    assert torch.equal(ids, torch.cat([p[0] for p in parts]))
    assert torch.equal(w.view(torch.int32), torch.cat([p[1] for p in parts]).view(torch.int32))
    assert torch.equal(cnt.long(), torch.bincount(ids.long(), minlength=E))
    again = run(z, None)                                  # without the counts
    assert torch.equal(again[0], ids) and torch.equal(again[1].view(torch.int32), w.view(torch.int32))


# K: less than a warp's 32 pieces of eight, a ragged share of its 128, several shares, not a multiple of eight (the element form)
@pytest.mark.parametrize("pairs", [1023, 1024, 1025, 5003])
@pytest.mark.parametrize("K", [8, 200, 1024, 1544, 4096, 1020])
@pytest.mark.parametrize("pad,off", [(8, 0), (4, 0), (8, 4)])
def test_gather(ops, pairs, K, pad, off):
    g = torch.Generator(device=DEV).manual_seed(pairs + K)
    T, top = 701, 3
    store = torch.randint(-2 ** 15, 2 ** 15, (T * (K + pad) + 8,), device=DEV, generator=g, dtype=torch.int16).view(torch.bfloat16)
    x = store[off:off + T * (K + pad)].view(T, K + pad)[:, :K]
    order = torch.randint(0, T * top, (pairs,), device=DEV, generator=g, dtype=torch.int32)
    out = torch.full((pairs + 1, K + pad), 7.0, device=DEV, dtype=torch.bfloat16)
    ops.moe_gather(x, top, order, pairs, out[:pairs, :K])
    want = x[(order // top).long()]
    assert torch.equal(out[:pairs, :K].contiguous().view(torch.int16), want.contiguous().view(torch.int16))
    assert bool((out[pairs:] == 7.0).all()) and bool((out[:, K:] == 7.0).all())
