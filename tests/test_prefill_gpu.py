"""hp_prefill over more than one 8-row pass (the chunked GEMM path) against the CPU oracle's 8-row passes, bit for bit: sizes
around the edges of its row tiles (8), of the GEMV / GEMM rule (32), of the column ranges (32, 64, 128) and of a chunk (512);
the tail rows, the draft block's cache and hidden rows, and the recurrent state (through the pass that follows)."""
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
        for p in range(0, len(prompt), 8):
            T = min(8, len(prompt) - p)
            ref.forward([(slot, prompt[p:p + T], p)]); ref.accept(slot, T)
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
