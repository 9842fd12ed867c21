"""Prompt passes against passes of eight rows at the 27B model's widths (4 layers, reduced vocabulary).

Passes of up to eight rows run the kernels that the oracle tests pin (one attention CTA per head and row, delta rule and gated
norm in one launch, the small-M product); longer ones run the prompt kernels: tiled or grouped attention, by size,
the delta rule spread over the GPU, the tile products.  The chunk size changes no result, so
logits, recurrent state and caches must agree bit for bit.
"""
import numpy as np
import pytest

from tests.util import bits

pytestmark = pytest.mark.gpu

N_VOCAB = 2048


@pytest.fixture(scope="module")
def eng():
    from irontimber_b200.engine import CudaEngine, config_27b
    e = CudaEngine(config_27b(n_layer=4, ctx_len=2304, n_vocab=N_VOCAB), seed=31)
    yield e
    e.close()


def states(eng):
    return [bits(eng.state(il, k)).copy() for il in range(eng.cfg.n_layer) for k in ((0, 1) if eng.cfg.is_recurrent(il) else (2, 3))]


# 9: shortest prompt pass; 17 / 49: one row into the next stage of tokens; 127: grouped attention, as in the two uneven calls of 300; 300, 700:
# tiled attention with ragged tiles of rows, positions and elements behind the diagonal; 2250: several passes, a block of rows at a time
@pytest.mark.parametrize("n", [9, 17, 49, 127, 300, 700, 2250])
def test_prompt_pass_equals_eight_row_passes(eng, n):
    prompt = np.random.default_rng(n).integers(0, N_VOCAB, n).astype(np.uint32)
    eng.reset()
    for s in range(0, n, 8):
        want = eng.eval(prompt[s:s + 8])
    want, want_states, tail = bits(want).copy(), states(eng), bits(eng.eval([5])).copy()
    eng.reset()
    got = eng.eval(prompt)
    assert np.array_equal(bits(got), want)
    assert all(np.array_equal(a, b) for a, b in zip(states(eng), want_states))
    assert np.array_equal(bits(eng.eval([5])), tail)
    # the same prompt in two uneven calls: the second one's rows start at a position of their own
    eng.reset()
    k = n // 3 + 1
    eng.eval(prompt[:k])
    if k < n:
        assert np.array_equal(bits(eng.eval(prompt[k:])), want)
        assert all(np.array_equal(a, b) for a, b in zip(states(eng), want_states))


# rows at a position: on either side of a tile of rows (21 x 6 = 126, 22 x 6 = 132) and of positions, one row, and a few rows far into a context
@pytest.mark.parametrize("at,n", [(0, 9), (0, 21), (0, 22), (0, 127), (0, 129), (0, 257), (100, 28), (1500, 24), (1500, 128)])
def test_both_attention_kernels_take_the_same_pass(eng, monkeypatch, at, n):
    """The rule by sizes gives a pass to one kernel; either one must give the same bits on any pass that it accepts."""
    toks = np.random.default_rng(at + n).integers(0, N_VOCAB, at + n).astype(np.uint32)
    got = {}
    for tiled in ("0", "1"):
        eng.reset()
        if at:
            monkeypatch.delenv("IT_ATTN_TILED", raising=False)
            eng.eval(toks[:at], want_logits=False)
        monkeypatch.setenv("IT_ATTN_TILED", tiled)
        got[tiled] = [bits(eng.eval(toks[at:])).copy()] + states(eng)
    assert all(np.array_equal(a, b) for a, b in zip(got["0"], got["1"]))


@pytest.mark.parametrize("n", [1025, 1034])      # a last pass of one row (recorded) and of ten
def test_speculative_prefill_of_two_passes_equals_forced_steps(n):
    """The head's catch-up across two prompt passes, against a prompt of one pass followed by verification passes of two rows that are fed
    the rest of the prompt: the same caches of trunk and head, the same next draft."""
    from irontimber_b200.engine import CudaEngine, config_27b
    eng = CudaEngine(config_27b(n_layer=4, ctx_len=1056, n_vocab=N_VOCAB), seed=13, with_mtp=True)
    try:
        prompt = [int(t) for t in np.random.default_rng(n).integers(0, N_VOCAB, n)]
        x = eng.mtp_prefill(prompt)
        want = states(eng) + [bits(eng.state(0, k)).copy() for k in (4, 5)] + [eng.mtp_draft([x])]
        at = n - 6
        eng.mtp_prefill(prompt[:at])
        pending = [prompt[at]]
        for i in range(at, n, 2):
            eng.mtp_draft(pending)
            picks = eng.mtp_verify(prompt[i], prompt[i + 1])
            pending = [prompt[i + 1], prompt[i + 2] if i + 2 < n else x]
        assert picks[1] == x
        got = states(eng)
        draft = eng.mtp_draft(pending)              # adds the pairs (h, last token) and (h, x) to the head's cache
        kvd = eng.cfg.n_head_kv * eng.cfg.head_dim
        got += [bits(eng.state(0, k))[:(n - 1) * kvd] for k in (4, 5)] + [draft]
        assert all(np.array_equal(a, b) for a, b in zip(got, want))
    finally:
        eng.close()
