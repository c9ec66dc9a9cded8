"""GPU: what a batched step returns beside other calls on the same context."""
import ctypes as C

import numpy as np
import pytest

import cabi
import temuvik_util as tu
from temuvik_util import attention, config, latent

pytestmark = pytest.mark.gpu


def decoder(cfg, w, slots, pages, *, max_step_tokens=2048, dtype=cabi.EFM_BF16):
    d = cabi.Decoder(cfg, cache_pages=pages * slots, state_slots=0, max_slots=slots, max_step_tokens=max_step_tokens, dtype=dtype)
    d.load_weights(w)
    d.set_sampling(0.0, 1.0, 0)
    for s in range(slots):
        d.map_slot(s, list(range(s * pages, (s + 1) * pages)), -1)
    return d


def step(d, entries, logits=True, sampled=True):
    """entries: (slot, kv_offset, tokens, want, random counter) -> logits [wanted, vocab], ids [wanted]; None for what is not asked for."""
    batch, keep = (cabi.StepEntry * len(entries))(), []
    for e, (slot, at, tokens, want, counter) in zip(batch, entries):
        keep += [cabi._i32_array(tokens), cabi._i32_array(want)]
        e.slot, e.n_tokens, e.kv_offset, e.n_want, e.rng_step, e.tokens, e.want = slot, len(tokens), at, len(want), counter, keep[-2], keep[-1]
    n = sum(len(e[3]) for e in entries)
    z = np.full((n, d.cfg.vocab), np.nan, np.float32) if logits else None
    ids = np.full(n, -1, np.int32) if sampled else None
    d.check(d.L.efm_b200_decoder_step(d.ctx, batch, len(entries), z.ctypes.data_as(C.POINTER(C.c_float)) if logits else None,
                                      ids.ctypes.data_as(C.POINTER(C.c_int32)) if sampled else None), "decoder_step")
    return z, ids


@pytest.mark.parametrize("temperature", [0.0, 0.8])
@pytest.mark.parametrize("live", [1, 20])
def test_a_step_leaves_the_response_of_a_decoding_slot_alone(built, live, temperature):
    """Tokens decoded on one slot are read after a sampled step (a single row, or 20) of other slots."""
    cfg = config([attention(), latent()], vocab=150)
    d = decoder(cfg, tu.weights(cfg, seed=4), live + 1, 2)
    prompt, n = tu.tokens(cfg, 21), 24

    def response(between):
        d.set_sampling(0.0, 1.0, 0)
        d.prefill(live, prompt, sample=True)
        d.decode_begin(live, len(prompt))
        d.decode_steps(n - 1)
        d.set_sampling(temperature, 1.0, 3)
        between()
        return d.read_tokens(0, n)
    expected = response(lambda: None)
    for s in range(live):
        step(d, [(s, 0, tu.tokens(cfg, 9, seed=s), [], 0)])
    assert response(lambda: step(d, [(s, 9, [s % 150], [0], s) for s in range(live)])) == expected
    d.close()
