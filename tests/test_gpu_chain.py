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


@pytest.mark.parametrize("M,paged", [(1, False), (1, True), (3, False)])
@pytest.mark.parametrize("S,n_new", [(1, 1), (7, 1), (8, 1), (9, 1), (5, 4), (3, 17), (17, 16)])
def test_generate_in_one_graph(host, M, paged, S, n_new):
    from blazr_b200 import decode
    vocab = decode.PRESETS["tiny"].vocab
    a, b = _decoder(host, M, paged), _decoder(host, M, paged)
    prompt = np.random.default_rng(S).integers(0, vocab, (M, S))
    got, want = a.generate(prompt, n_new), b.generate(prompt, n_new, use_graph=False)
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
