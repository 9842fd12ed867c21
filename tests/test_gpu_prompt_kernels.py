"""Prompt passes against passes of eight rows at the 27B model's widths (4 layers, reduced vocabulary).

Passes of up to eight rows run the kernels that the oracle tests pin (one attention CTA per head and row, delta rule and gated
norm in one launch, the small-M product); longer ones run the prompt kernels: tiled attention once there are enough tiles,
grouped attention before that, the delta rule spread over the GPU, the tile products.  The chunk size changes no result, so
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


# 9: shortest prompt pass; 17 / 49: one row into the next stage of tokens; 127, 300: grouped attention; 700: tiled attention with ragged
# tiles of rows, positions and elements behind the diagonal; 2250: several passes, a block of rows at a time
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
