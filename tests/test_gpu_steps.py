"""GPU: what a batched step returns beside other calls on the same context."""
import ctypes as C

import numpy as np
import pytest

import cabi
import temuvik_util as tu
from oracle import temuvik
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


# heads and kv heads: a row walked by a cluster of its own costs least with few kv heads, a block for all rows of an entry with many
@pytest.mark.parametrize("dtype", ["fp32", "bf16"])
@pytest.mark.parametrize("dim,vdim", [(24, 40), (128, 72), (200, 144)])
@pytest.mark.parametrize("heads,kv_heads,sizes", [(8, 8, [15]), (8, 8, [15] * 40), (8, 8, [1, 15] * 30), (9, 9, list(range(1, 16)) * 4), (9, 3, [2, 3, 5, 14] * 16),
                                                  (9, 1, [9, 15] * 24), (8, 8, [5] * 64), (8, 8, [1] * 40 + [16, 33, 7])])
def test_short_entries_of_any_size(built, heads, kv_heads, sizes, dim, vdim, dtype):
    """Rows walked one by one, blocks of an entry's rows, and both in one pass, beside entries long enough for the tensor cores; every row
    against the CPU statement."""
    cfg = config([attention(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, scale=0.1, size=70, keep=3), attention(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, scale=0.1, size=None)],
                 width=64, vocab=60)
    w = tu.weights(cfg, seed=8)
    before = [(7 * i + 61) % 130 + 1 for i in range(len(sizes))]
    seq = tu.tokens(cfg, 130 + max(sizes))
    ref = temuvik.forward(cfg, w, seq).logits.numpy()
    d = decoder(cfg, w, len(sizes), 3, dtype=cabi.EFM_F32 if dtype == "fp32" else cabi.EFM_BF16)
    step(d, [(s, 0, seq[:n], [], 0) for s, n in enumerate(before)], logits=False, sampled=False)
    got, _ = step(d, [(s, n, seq[n:n + k], list(range(k)), 0) for s, (n, k) in enumerate(zip(before, sizes))], sampled=False)
    d.close()
    assert tu.error(got, np.concatenate([ref[n:n + k] for n, k in zip(before, sizes)])) < tu.LIMIT[dtype]


@pytest.mark.parametrize("dtype", ["fp32", "bf16"])
@pytest.mark.parametrize("heads", [8, 120])
def test_short_prompt_of_many_heads(built, heads, dtype):
    """The 15 rows in front of a prompt's last token: walked one by one with 8 heads, blocks of all of them with 120."""
    cfg = config([attention(heads=heads, kv_heads=heads, dim=16, vdim=24, scale=0.1, rot=16, size=10, keep=2)] * 2, width=64, vocab=60)
    w = tu.weights(cfg, seed=8)
    seq = tu.tokens(cfg, 16)
    d = decoder(cfg, w, 1, 1, dtype=cabi.EFM_F32 if dtype == "fp32" else cabi.EFM_BF16)
    d.prefill(0, seq, sample=True)
    got = np.array(d.read_logits())
    d.close()
    assert tu.error(got[None], temuvik.forward(cfg, w, seq).logits.numpy()[-1:]) < tu.LIMIT[dtype]


LENGTHS = [200, 130, 9, 1]


def wants(count):
    """`count` of the rows of four entries: an entry's last rows in descending order, then rows with gaps, a repeated one, a single one."""
    lists = [list(range(199, -1, -1)), list(range(1, 130, 2)) + list(range(0, 130, 2)), [8, 8, 0], [0]]
    share = [max(0, min(len(l), n)) for l, n in zip(lists, (count - 6 - (count - 6) // 3, (count - 6) // 3, 3, 1))] if count > 8 else [0, 0, 0, 1] if count == 1 else [0, count - 1, 0, 1]
    share[0] += count - sum(share)
    return [l[:n] for l, n in zip(lists, share)]


@pytest.mark.parametrize("max_step_tokens", [2048, 96])
@pytest.mark.parametrize("dtype", ["fp32", "bf16"])
@pytest.mark.parametrize("vocab", [64, 147])
@pytest.mark.parametrize("count", [1, 2, 40, 256, 257, 300])
def test_wanted_rows_of_a_step(built, count, vocab, dtype, max_step_tokens):
    """Logits and samples of one call, in one pass and in passes that cut entries, up to more rows than the head takes at a time."""
    cfg = config([attention(), latent()], vocab=vocab)
    w = tu.weights(cfg, seed=5)
    seqs = [tu.tokens(cfg, n, seed=n) for n in LENGTHS]
    d = decoder(cfg, w, 4, 4, max_step_tokens=max_step_tokens, dtype=cabi.EFM_F32 if dtype == "fp32" else cabi.EFM_BF16)
    lists = wants(count)
    assert sum(map(len, lists)) == count
    entries = [(s, 0, seq, l, 0) for s, (seq, l) in enumerate(zip(seqs, lists))]
    z, ids = step(d, entries)
    ref = np.concatenate([temuvik.forward(cfg, w, seq).logits.numpy()[l] for seq, l in zip(seqs, lists) if l])
    assert tu.error(z, ref) < tu.LIMIT[dtype]
    assert ids.tolist() == z.argmax(1).tolist()
    assert np.array_equal(step(d, entries, sampled=False)[0], z)
    assert np.array_equal(step(d, entries, logits=False)[1], ids)
    d.close()


def test_sampled_rows_of_a_step_are_those_of_single_rows(built):
    """Nucleus samples of many rows in one call, and of the same rows wanted one at a time, with the same counters (32-bit mode: a row's logits do
    not depend on the others)."""
    cfg = config([attention(), latent()], vocab=147)
    w = tu.weights(cfg, seed=5)
    seqs = [tu.tokens(cfg, n, seed=n) for n in LENGTHS]
    d = decoder(cfg, w, 4, 4, dtype=cabi.EFM_F32)
    d.set_sampling(1.2, 0.9, 11)
    lists = [[199, 4, 77], [0, 1, 2, 129], [8, 8, 3], [0]]

    def entries(lists):
        return [(s, 0, seq, l, 100 + s) for s, (seq, l) in enumerate(zip(seqs, lists))]
    z, ids = step(d, entries(lists))
    alone = [step(d, entries([[p] if t == s else [] for t in range(4)]), logits=False)[1][0] for s, l in enumerate(lists) for p in l]
    d.close()
    assert ids.tolist() == alone
    assert ids.tolist() != z.argmax(1).tolist()
