"""hp_prefill over more than one 8-row pass (the chunked GEMM path) against the CPU oracle's 8-row passes, bit for bit: sizes
around the edges of its row tiles (8), of the GEMV / GEMM rule and of a chunk (512), one and several attention batches per
chunk and several chunks per prompt; the tail rows, the draft block's cache and hidden rows, the recurrent state (through the
pass that follows) and pending accepts. (The GEMM's column ranges: test_gemm_gpu.py.)"""
import numpy as np
import pytest

import hipster_b200 as hb
from oracle import orc

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.mark.parametrize("preset,n,over", [("tiny", 9, {}), ("tiny", 33, {}), ("tiny", 64, {}), ("tiny", 131, {}), ("tiny", 515, dict(max_ctx=640)),
                                           ("tiny", 70, dict(n_head=24, n_head_kv=2)), ("tiny-moe", 33, {}), ("tiny-moe", 75, dict(synth_router_logits=1))])
def test_prefill_chunks_bit_exact_vs_oracle(preset, n, over):
    cfg = hb.ModelCfg.preset(preset, **{"max_ctx": 160, **over})
    eng = hb.Engine(cfg); ref = orc.Model(cfg)
    rng = np.random.default_rng(n)
    prompt = [int(x) for x in rng.integers(0, cfg.n_vocab, size=n)]
    first = prompt[:3]                                           # rows accepted before the prompt: their commit is still pending
    for e in (eng, ref):
        e.forward([(0, first, 0)]); e.accept(0, 2)
    base = 2
    eng.prefill(0, prompt, pos0=base, with_mtp=False)
    for p in range(0, n, 8):
        T = min(8, n - p)
        ref.forward([(0, prompt[p:p + T], base + p)]); ref.accept(0, T)
    assert np.array_equal(bits(eng.logits(1)[0]), bits(ref.logits(T)[T - 1]))
    assert np.array_equal(bits(eng.h_nextn(1)[0]), bits(ref.h_nextn(T)[T - 1]))
    assert np.array_equal(bits(eng.h_nextn(T)[1:]), bits(ref.h_nextn(T)[1:]))
    assert int(eng.topk(0, 1)[0][0]) == int(orc.argmax(ref.logits(T))[0][T - 1])
    toks = [int(x) for x in rng.integers(0, cfg.n_vocab, size=3)]
    for e in (eng, ref):                                         # the state, the conv history and the caches behind the prompt
        e.forward([(0, toks, base + n)])
    assert np.array_equal(bits(eng.logits(3)), bits(ref.logits(3)))
    eng.close()


@pytest.mark.parametrize("n", [32, 40, 48, 49])   # projections in one and two GEMV launches, and beyond the rows that always take it
def test_prefill_on_both_sides_of_the_gemm_line(n):
    test_prefill_chunks_bit_exact_vs_oracle("tiny", n, {})


# experts grouped over a whole chunk: one row beyond a pass, segments that are full and not, two chunks of unequal length, the shared expert behind
# 1024 others (a bucket of its own beyond the threads of the scan), a full chunk of the most slots per row (512 x 16 pairs) and one with a ragged last
# group of rows
@pytest.mark.parametrize("n,over", [(40, dict(n_expert=1024)), (128, {}), (300, dict(synth_router_logits=1)), (515, dict(max_ctx=640, synth_router_logits=1)),
                                    (512, dict(max_ctx=640, n_expert=64, n_expert_used=15)), (507, dict(max_ctx=640, synth_router_logits=1))])
def test_prefill_groups_the_experts_of_a_chunk(n, over):
    test_prefill_chunks_bit_exact_vs_oracle("tiny-moe", n, {"max_ctx": 320, **over})


@pytest.mark.parametrize("n", [56, 57, 88, 104, 160])   # all projections in the GEMV, some of them, all in the GEMM
def test_prefill_around_the_lines_of_its_projections(n):
    test_prefill_chunks_bit_exact_vs_oracle("tiny", n, dict(max_ctx=192))


@pytest.mark.parametrize("n", [17, 42])
def test_prefill_chunks_fill_the_draft_block(n):
    cfg = hb.ModelCfg.preset("tiny", max_ctx=128)
    eng = hb.Engine(cfg); ref = orc.Model(cfg)
    prompt = [int(x) for x in np.random.default_rng(n).integers(0, cfg.n_vocab, size=n)]
    cut = 13                                                     # two calls: the second pairs its first row with the first call's last
    eng.prefill(0, prompt[:cut], with_mtp=True); eng.prefill(0, prompt[cut:], pos0=cut, with_mtp=True)
    prev = np.zeros(cfg.n_embd, dtype=np.float32)
    for a, b in ((0, cut), (cut, n)):
        for p in range(a, b, 8):
            T = min(8, b - p)
            ref.forward([(0, prompt[p:p + T], p)]); ref.accept(0, T)
            h = ref.h_nextn(T)
            ref.mtp_forward(0, prompt[p:p + T], np.vstack([prev[None, :], h[:T - 1]]), p)
            prev = h[T - 1].copy()
    assert np.array_equal(bits(eng.mtp_h(T)), bits(ref.mtp_h(T)))
    tok = int(eng.topk(0, 1)[0][0])
    eng.mtp_forward(0, [tok], eng.h_nextn_ptr(), n)
    ref.mtp_forward(0, [tok], prev[None, :], n)
    assert np.array_equal(bits(eng.mtp_logits(1)), bits(ref.mtp_logits(1)))
    eng.close()


def oracle_prefill(ref, slot, prompt, pos0, prev, with_mtp):
    """hp_prefill as 8-row passes of the oracle; prev: hidden row in front of the prompt -> rows of the last pass, its last row."""
    for p in range(0, len(prompt), 8):
        T = min(8, len(prompt) - p)
        ref.forward([(slot, prompt[p:p + T], pos0 + p)]); ref.accept(slot, T)
        h = ref.h_nextn(T)
        if with_mtp:
            ref.mtp_forward(slot, prompt[p:p + T], np.vstack([prev[None, :], h[:T - 1]]), pos0 + p)
        prev = h[T - 1].copy()
    return T, prev


@pytest.mark.parametrize("over,n0,n,batches", [(dict(n_head=24, n_head_kv=2, max_ctx=1024), 400, 501, 4),    # 4 rows per group: batches of 128, 128, 128, 117
                                               (dict(max_ctx=1024), 500, 512, 2),                            # 8 rows per group
                                               (dict(n_head=24, n_head_kv=2, max_ctx=700), 150, 515, 2)])    # chunks of 264 and 251 rows, two batches each
def test_prefill_attention_in_several_batches(over, n0, n, batches):
    cfg = hb.ModelCfg.preset("tiny", **over)
    gr = min(8, 48 // (cfg.n_head // cfg.n_head_kv))             # rows per attention row group
    size = n if n <= 512 else (-(-n // 2) + 7) & ~7
    rows, end = n - (n > 512) * size, n0 + n                     # the last chunk
    per = max(32, (32 * -(-cfg.max_ctx // 128) // -(-end // 128)) * gr & ~7)
    assert -(-rows // per) == batches
    eng = hb.Engine(cfg); ref = orc.Model(cfg)
    prompt = [int(x) for x in np.random.default_rng(n).integers(0, cfg.n_vocab, size=n0 + n)]
    eng.prefill(0, prompt[:n0], with_mtp=False); eng.prefill(0, prompt[n0:], pos0=n0, with_mtp=False)
    _, prev = oracle_prefill(ref, 0, prompt[:n0], 0, None, False)
    T, prev = oracle_prefill(ref, 0, prompt[n0:], n0, prev, False)
    assert np.array_equal(bits(eng.logits(1)[0]), bits(ref.logits(T)[T - 1]))
    assert np.array_equal(bits(eng.h_nextn(T)[1:]), bits(ref.h_nextn(T)[1:]))
    for e in (eng, ref):
        e.forward([(0, [9, 8, 7], n0 + n)])
    assert np.array_equal(bits(eng.logits(3)), bits(ref.logits(3)))
    eng.close()


def test_prefill_several_chunks_fill_the_draft_block():
    cfg = hb.ModelCfg.preset("tiny", max_ctx=1100)
    eng = hb.Engine(cfg); ref = orc.Model(cfg)
    n = 1030                                                     # chunks of 344, 344 and 342 rows
    prompt = [int(x) for x in np.random.default_rng(n).integers(0, cfg.n_vocab, size=n)]
    eng.prefill(1, prompt, with_mtp=True)
    T, prev = oracle_prefill(ref, 1, prompt, 0, np.zeros(cfg.n_embd, dtype=np.float32), True)
    assert np.array_equal(bits(eng.logits(1)[0]), bits(ref.logits(T)[T - 1]))
    assert np.array_equal(bits(eng.mtp_h(T)), bits(ref.mtp_h(T)))
    tok = int(eng.topk(0, 1)[0][0])
    eng.mtp_forward(1, [tok], eng.h_nextn_ptr(), n)              # attends over the draft block's K/V rows of every chunk
    ref.mtp_forward(1, [tok], prev[None, :], n)
    assert np.array_equal(bits(eng.mtp_logits(1)), bits(ref.mtp_logits(1)))
    eng.close()


@pytest.mark.parametrize("decide", ["before", "after"])
def test_prefill_with_other_slots_rows_pending(decide):
    """Slot 1 has rows of which a prefix is accepted before or after the prompt of slot 0, whose own pending rows make the
    prompt commit every slot's."""
    cfg = hb.ModelCfg.preset("tiny", max_ctx=128)
    eng = hb.Engine(cfg); ref = orc.Model(cfg)
    a, b, c, prompt = [[int(x) for x in np.random.default_rng(i).integers(0, cfg.n_vocab, size=n)] for i, n in enumerate((4, 5, 6, 37))]
    for e in (eng, ref):
        e.forward([(0, a, 0), (1, b, 0)])
        e.accept(0, 3)
        if decide == "before" or e is ref:                       # the oracle keeps one pass' rows only
            e.accept(1, 2)
    eng.prefill(0, prompt, pos0=3, with_mtp=False)
    oracle_prefill(ref, 0, prompt, 3, None, False)
    if decide == "after":
        eng.accept(1, 2)
    for e in (eng, ref):
        e.forward([(1, c, 2), (0, [1, 2], 40)])
    assert np.array_equal(bits(eng.logits(8)), bits(ref.logits(8)))
    eng.close()


def test_chunk_buffers_come_with_the_first_long_prompt_and_only_where_they_fit():
    """A model loads with what its passes need, also where the buffers of the prompt chunks (about 170 MB for this shape)
    would not fit beside it; prompts then run as 8-row passes with the same bits, and as chunks once there is room."""
    import torch
    MB = 1 << 20
    cfg = hb.ModelCfg.preset("tiny", n_ff=17408)
    free = lambda: torch.cuda.mem_get_info()[0]  # noqa: E731
    rng = np.random.default_rng(5)
    prompts = [[int(x) for x in rng.integers(0, cfg.n_vocab, size=n)] for n in (20, 21)]
    ref = orc.Model(cfg)
    warm = hb.Engine(cfg); warm.prefill(0, prompts[0], with_mtp=False); warm.prefill(1, prompts[0][:8]); warm.close()   # kernels loaded
    torch.cuda.empty_cache()
    f0 = free()
    eng = hb.Engine(cfg)
    weights = f0 - free()
    eng.prefill(0, prompts[0][:8], with_mtp=False)
    assert f0 - free() - weights <= 4 * MB                       # short prompts do not take them
    eng.prefill(0, prompts[0], with_mtp=False)
    chunks = f0 - free() - weights
    assert 100 * MB < chunks < 200 * MB
    eng.close()
    assert free() >= f0 - 4 * MB
    hog = torch.empty(free() - weights - chunks // 2, dtype=torch.uint8, device="cuda")
    eng = hb.Engine(cfg)                                         # half of the buffers' size is left
    left = free()
    assert left < chunks

    def check(slot, prompt):
        eng.prefill(slot, prompt, with_mtp=False)
        T, _ = oracle_prefill(ref, slot, prompt, 0, None, False)
        assert np.array_equal(bits(eng.logits(1)[0]), bits(ref.logits(T)[T - 1]))
        assert np.array_equal(bits(eng.h_nextn(T)[1:]), bits(ref.h_nextn(T)[1:]))

    check(0, prompts[0])
    assert free() >= left - 4 * MB                               # (a kernel used for the first time may take its code's page)
    del hog
    torch.cuda.empty_cache()
    check(1, prompts[1])                                         # the other slot, as a chunk
    for e in (eng, ref):                                         # both go on from their prompts
        e.forward([(0, [3, 4], 20), (1, [5], 21)])
    assert np.array_equal(bits(eng.logits(3)), bits(ref.logits(3)))
    eng.close()
