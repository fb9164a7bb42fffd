"""Captured steps that follow one another in one graph (csrc/decode_ops.cu argmax_next_kernel, Decoder.capture): the prompt's tokens are fed and the choices
kept on the device, and every step but the first of a graph finds its token embedded.  Tokens, logits, keys and values are those of steps launched one by one,
bit for bit, at lengths around the graph's, with one and several sequences, contiguous and paged; afterwards a step takes its own choice again."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def host():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from blazr_b200 import decode
    return decode.build_host_model(decode.PRESETS["tiny"], "Q4_K_M", seed=4)


def _decoder(host, M, paged):
    from blazr_b200 import decode, ops
    return decode.Decoder(ops.B200Client(0), decode.PRESETS["tiny"], "Q4_K_M", batch=M, max_ctx=32, host=host, **(dict(paged=True, block_size=4) if paged else {}))


class _Counted:
    """a captured graph that counts its replays"""
    def __init__(self, graph):
        self.graph, self.n = graph, 0

    def replay(self):
        self.n += 1
        self.graph.replay()


@pytest.mark.parametrize("M,paged", [(1, False), (1, True), (3, False)])
@pytest.mark.parametrize("S,n_new", [(1, 1), (7, 1), (8, 1), (9, 1), (5, 4), (3, 17), (17, 16)])
def test_generate_in_one_graph(host, M, paged, S, n_new):
    from blazr_b200 import decode
    vocab = decode.PRESETS["tiny"].vocab
    a, b = _decoder(host, M, paged), _decoder(host, M, paged)
    prompt = np.random.default_rng(S).integers(0, vocab, (M, S))
    a.capture()
    assert a.chain_steps == decode.CHAIN > 1
    a.graph, a.chain_graph = _Counted(a.graph), _Counted(a.chain_graph)
    got, want = a.generate(prompt, n_new), b.generate(prompt, n_new, use_graph=False)
    assert (a.chain_graph.n, a.graph.n) == divmod(S + n_new - 1, decode.CHAIN) and bool((a.fed == -1).all())
    assert got.dtype == want.dtype and got.shape == (M, n_new) and (got == want).all()
    for _ in range(2):
        assert torch.equal(a.full_logits(), b.full_logits()) and torch.equal(a.ids, b.ids) and torch.equal(a.pos, b.pos)
        n = int(a.pos[0])
        for x, y in zip(a.layers, b.layers):
            for m in range(M):
                assert all(torch.equal(u, v) for u, v in zip(a.kv_rows(x, m, n), b.kv_rows(y, m, n)))
        if n >= 32:
            break
        a.replay()
        b.step()
        torch.cuda.synchronize()


def test_ids_outside_the_table_take_its_first_row():
    """embedded by the launch at the head of a step or by the end of the step before, an id without a row (a choice among logits that are no numbers) is the same one"""
    from blazr_b200 import ops
    L, V, dev = ops.lib(), 40, "cuda:0"
    P, st = (lambda t: t.data_ptr()), None
    for H in (64, 66):
        table = torch.randn((V, H), device=dev).half()
        ids = torch.tensor([3, V - 1, V, -1, 2 ** 31 - 1, -2 ** 40], device=dev)
        want = table[torch.where((ids >= 0) & (ids < V), ids, 0)].float()
        h = torch.empty((len(ids), H), device=dev)
        ops._check(L.b200q_embed_rows(P(table), V, P(ids), H, len(ids), P(h), st))
        assert torch.equal(h, want)
        for i in range(len(ids)):                                            # (one row is a kernel of its own)
            ops._check(L.b200q_embed_rows(P(table), V, P(ids[i:]), H, 1, P(h), st))
            assert torch.equal(h[0], want[i])
        # the end of a step: choices 7, none (not a number), 5 with a token fed behind it, 9 with one that is not in the table
        logits = torch.zeros((4, V), device=dev)
        logits[0, 7] = logits[2, 5] = logits[3, 9] = 1.0
        logits[1] = float("nan")
        pos, nxt = torch.tensor([0, 1, 2, 0], dtype=torch.int32, device=dev), torch.full((4,), -7, device=dev)
        fed, chosen = torch.full((4, 4), -1, device=dev), torch.full((4, 4), -9, device=dev)
        fed[3, 2], fed[1, 3] = 11, V + 2
        want = torch.tensor([7, 2 ** 31 - 1, 11, V + 2], device=dev)
        import ctypes as C
        ops._check(L.b200q_argmax_next(C.c_void_p(P(logits)), C.c_int64(V), C.c_int64(4), C.c_void_p(P(nxt)), C.c_void_p(P(pos)), C.c_void_p(P(fed)), C.c_void_p(P(chosen)),
                                       C.c_int64(4), C.c_void_p(P(table)), C.c_int64(H), C.c_void_p(P(h)), None))
        assert torch.equal(nxt, want) and pos.tolist() == [1, 2, 3, 1]
        assert chosen[0].tolist() == [7, -9, -9, 9] and chosen[1].tolist() == [-9, 2 ** 31 - 1, -9, -9] and chosen[2].tolist() == [-9, -9, 5, -9]
        assert torch.equal(h[:4], table[torch.where(want < V, want, 0)].float())


@pytest.mark.parametrize("use_graph", [True, False])
def test_generate_refuses_ids_without_a_row(host, use_graph):
    from blazr_b200 import decode
    vocab, a = decode.PRESETS["tiny"].vocab, _decoder(host, 1, False)
    for bad in (-1, vocab, 2 ** 31 - 1):
        for at in (0, 2):
            prompt = np.array([[1, 2, 3, 4]])
            prompt[0, at] = bad
            with pytest.raises(ValueError, match="outside"):
                a.generate(prompt, 2, use_graph)
    assert a.generate(np.array([[0, vocab - 1]]), 2, use_graph).shape == (1, 2)


@pytest.mark.parametrize("use_graph", [True, False])
def test_generate_refuses_no_new_tokens(host, use_graph):
    a = _decoder(host, 1, False)
    for n_new in (0, -2):
        with pytest.raises(ValueError, match="at least one"):
            a.generate(np.array([[1, 2, 3, 4]]), n_new, use_graph)
