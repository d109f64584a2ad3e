"""Performance cases of the speculative-decode path, through the entry points that a caller uses.

Two levels, as in the library: the kernel-level calls on torch tensors (`hipster_b200.kernels` and, where it has no
wrapper, the C ABI itself) and the engine-level calls (`hipster_b200.Engine`). Sizes are those of the benchmark
configurations and presets of this repository, and ragged ones around them. Weights, prompts and rows are random, made
from the seed with the distributions that the benchmark states: Q4_K quants and 6-bit scales uniform, d and dmin
|N(0, 0.01)|, activations N(0, 1), prompts uniform over the vocabulary.

The library fixes the order of every floating-point sum by the tensor shapes alone and reproduces its oracle bit for
bit, so every case is compared exactly.
"""
import ctypes
import math

import numpy as np
import torch

import hipster_b200 as hb
from hipster_b200 import kernels as K
from hipster_b200._lib import check, lib, ptr

DENSE, MOE = "qwen35-27b", "flash-next"


def listed():
    return [
        # ---- kernel level
        # The smallest call: one row through a small projection (an expert's down projection by itself). Latency of the calls.
        dict(name="gemv_small", kind="gemv", N=2048, K=512, R=1, drafts=0),
        # Verify GEMV of one dense FFN projection over one token and two drafts, arg-max and greedy acceptance on the device.
        dict(name="gemv_verify", kind="gemv", N=17408, K=5120, R=3, drafts=2),
        # A ragged projection over the rows of several slots: N is no multiple of a tile, 13 rows need two column tiles.
        dict(name="gemv_ragged", kind="gemv", N=4999, K=6144, R=13, drafts=0),
        # One Gated-DeltaNet layer of a verify pass: six rows, after the commit of four rows of the pass before.
        dict(name="gdn_verify", kind="gdn", n_qk=16, n_v=48, T=6, replay=4),
        # One attention layer of a verify pass at the context of the benchmark's prompt.
        dict(name="attn_verify", kind="attn", n_head=24, n_kv=4, R=6, pos=4091),
        # One mixture-of-experts FFN over the 24 rows of eight slots.
        dict(name="moe_layer", kind="moe", T=24, E=2048, F=512, experts=512, top=10),
        # ---- engine level, dense 27B-shaped model
        # Plain greedy decode: one row per pass.
        dict(name="decode_dense", kind="forward", preset=DENSE, rows="1", ctx=253),
        # A pass over four sequences that verify different numbers of rows.
        dict(name="batch_dense", kind="forward", preset=DENSE, rows="5,1,8,3", ctx=61),
        # Prompt ingestion, the draft block's K/V rows included. The odd length ends in a short chunk.
        dict(name="prefill_dense", kind="prefill", preset=DENSE, tokens=301),
        # The flagship: one speculative round with five drafts for one sequence, deep in its context.
        dict(name="round_dense", kind="round", preset=DENSE, slots=1, drafts=5, ctx=2043),
        # ---- engine level, mixture-of-experts model
        # One sequence, two drafts: three verify rows, so latency and launches count.
        dict(name="round_moe", kind="round", preset=MOE, slots=1, drafts=2, ctx=1021),
        # Eight sequences in lock step, two drafts each: 24 verify rows.
        dict(name="round_moe_slots", kind="round", preset=MOE, slots=8, drafts=2, ctx=253),
    ]


def _log(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(["gemv", "gdn", "attn", "moe", "forward", "prefill", "round"])
    if kind == "gemv":
        R, nb = _log(rng, 1, 32), _log(rng, 1, 68)
        nb += nb & 1 if nb > 36 else 0                   # longer rows are cut into equal parts of at most 36 blocks
        N = _log(rng, 16, min(34816, 34816 * 20 // nb))
        return dict(kind=kind, N=N, K=256 * nb, R=R, drafts=R - 1 if rng.random() < 0.5 else 0)
    if kind == "gdn":
        n_qk, n_v = rng.choice([(16, 48), (16, 32), (8, 24), (2, 4)])
        T = rng.randint(1, 8)
        return dict(kind=kind, n_qk=n_qk, n_v=n_v, T=T, replay=rng.randint(0, T))
    if kind == "attn":
        n_head, n_kv = rng.choice([(24, 4), (24, 2), (4, 2)])
        return dict(kind=kind, n_head=n_head, n_kv=n_kv, R=rng.randint(1, 8), pos=_log(rng, 1, 8000))
    if kind == "moe":
        return dict(kind=kind, T=_log(rng, 1, 32), E=rng.choice([512, 1024, 2048]), F=rng.choice([256, 512]), experts=_log(rng, 16, 512), top=rng.randint(2, 10))
    preset = rng.choice([DENSE, MOE])
    if kind == "forward":
        S = rng.randint(1, 4 if preset == DENSE else 8)
        rows = [min(_log(rng, 1, 8), 32 // S) for _ in range(S)]
        return dict(kind=kind, preset=preset, rows=",".join(map(str, rows)), ctx=_log(rng, 8, 253))
    if kind == "prefill":
        return dict(kind=kind, preset=preset, tokens=_log(rng, 9, 300))
    drafts = rng.randint(1, 7 if preset == DENSE else 3)
    S = rng.randint(1, min(4 if preset == DENSE else 8, 32 // (drafts + 1)))
    return dict(kind=kind, preset=preset, slots=S, drafts=drafts, ctx=_log(rng, 8, 2043 // S))


def tolerance(case):
    return "exact"


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _q4k(g, rows, k):
    """A Q4_K matrix [rows][k / 256 blocks of 144 bytes]: random bytes, d and dmin = f16(|N(0, 0.01)|)."""
    n = rows * (k // 256)
    blk = torch.randint(0, 256, (n, 144), dtype=torch.uint8, device="cuda", generator=g)
    blk[:, :4] = torch.randn((n, 2), device="cuda", generator=g).mul_(0.01).abs_().half().view(torch.uint8)
    return blk.reshape(rows, -1)


def _normal(g, *shape, std=1.0, mean=0.0):
    return torch.randn(shape, device="cuda", generator=g).mul_(std).add_(mean)


def _bf16(t):
    return t.bfloat16().view(torch.int16)


def _prompt(cfg, seed, slot, n):
    return [int(x) for x in np.random.default_rng([seed, slot]).integers(0, cfg.n_vocab, size=n)]


# ------------------------------------------------------------------ kernel level
def _prepare_gemv(c, seed):
    g = _gen(seed)
    s = dict(w=_q4k(g, c["N"], c["K"]), x=_normal(g, c["R"], c["K"]))
    s["xq"] = K.XQ8(c["R"], c["K"])
    s["y"] = torch.empty((c["R"], c["N"]), dtype=torch.float32, device="cuda")
    if c["drafts"]:
        s["ids"] = torch.randint(0, c["N"], (c["drafts"],), dtype=torch.int32, device="cuda", generator=g)
    return s


def _run_gemv(c, s):
    K.quantize_x_q8(s["x"], s["xq"])
    K.gemv_q4k_q8(s["w"], s["xq"], c["N"], c["K"], s["y"])
    if not c["drafts"]:
        return s["y"]
    ids, vals = K.argmax(s["y"])
    return s["y"], ids, vals, K.accept_greedy(ids, s["ids"])


def _prepare_gdn(c, seed):
    g, n_qk, n_v = _gen(seed), c["n_qk"], c["n_v"]
    ld = (2 * n_qk + 2 * n_v) * 128 + 2 * n_v
    L = lib()
    L.hp_gdn_conv_state_floats.restype = L.hp_gdn_saved_floats.restype = ctypes.c_size_t
    s = dict(rows=_normal(g, c["T"], ld), ld=ld, conv_w=_normal(g, (2 * n_qk + n_v) * 128, 4, std=0.5), dt=_bf16(_normal(g, n_v, std=0.5)),
             a_neg=_bf16(-_normal(g, n_v).abs_()), norm=_bf16(_normal(g, 128, std=0.3, mean=1.0)), state=_normal(g, n_v, 128, 128, std=0.1),
             conv=_normal(g, L.hp_gdn_conv_state_floats(n_v)), saved=torch.zeros(L.hp_gdn_saved_floats(n_v), device="cuda"),
             out=torch.empty((c["T"], n_v * 128), device="cuda"), xq=K.XQ8(c["T"], n_v * 128))
    _gdn(c, s, 0)                                        # the pass before, whose first rows are then committed
    return s


def _gdn(c, s, replay):
    check(lib().hp_gdn_layer(ptr(s["rows"]), s["ld"], c["T"], replay, c["n_qk"], c["n_v"], ptr(s["conv_w"]), ptr(s["dt"]), ptr(s["a_neg"]), ptr(s["norm"]),
                             ptr(s["state"]), ptr(s["conv"]), ptr(s["saved"]), ptr(s["out"]), ptr(s["xq"].q), ptr(s["xq"].sc), None,
                             ctypes.c_float(1e-6), 0, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))


def _run_gdn(c, s):
    _gdn(c, s, c["replay"])
    return s["out"], s["state"], s["conv"], s["saved"], s["xq"].q, s["xq"].sc


def _prepare_attn(c, seed):
    g, R, pos = _gen(seed), c["R"], c["pos"]
    ctx = (pos + R + 127) // 128 * 128
    ang = torch.arange(ctx, dtype=torch.float64)[:, None] * 1e7 ** (-2.0 * torch.arange(32, dtype=torch.float64) / 64)
    return dict(proj=_normal(g, R, c["n_head"] * 512 + 2 * c["n_kv"] * 256), qkv=torch.empty((R, c["n_head"] * 512 + 2 * c["n_kv"] * 256), device="cuda"),
                qn=_bf16(_normal(g, 256, std=0.2, mean=1.0)), kn=_bf16(_normal(g, 256, std=0.2, mean=1.0)), rope=torch.stack([ang.cos(), ang.sin()], -1).float().cuda().contiguous(),
                kc=_normal(g, c["n_kv"], ctx, 256).half(), vc=_normal(g, c["n_kv"], ctx, 256).half(), ctx=ctx)


def _run_attn(c, s):
    s["qkv"].copy_(s["proj"])                            # the call normalises and rotates the projection's rows in place
    out, xq = K.attn_decode(s["qkv"], c["pos"], c["n_head"], c["n_kv"], 64, s["qn"], s["kn"], s["rope"], s["kc"], s["vc"], s["ctx"])
    return out, xq.q, xq.sc, s["kc"], s["vc"]


def _prepare_moe(c, seed):
    g, T, E, F, n, k = _gen(seed), c["T"], c["E"], c["F"], c["experts"], c["top"]
    tiled = lambda rows, cols, half: K.repack_tiled(_q4k(g, rows, cols).reshape(-1), rows, cols, half)  # noqa: E731
    L = lib()
    L.hp_moe_workspace_bytes.restype = ctypes.c_size_t
    return dict(x=_normal(g, T, E), xq=K.XQ8(T, E), router=_normal(g, n + 1, E, std=E ** -0.5), egu=tiled(n * 2 * F, E, F), edn=tiled(n * E, F, 0),
                sgu=tiled(2 * F, E, F), sdn=tiled(E, F, 0), ws=torch.empty(L.hp_moe_workspace_bytes(T, E, F, n, k), dtype=torch.uint8, device="cuda"),
                ids=torch.empty((T, k + 1), dtype=torch.int32, device="cuda"), w=torch.empty((T, k + 1), device="cuda"), y=torch.empty((T, E), device="cuda"))


def _run_moe(c, s):
    K.quantize_x_q8(s["x"], s["xq"])
    check(lib().hp_moe_layer(ptr(s["x"]), ptr(s["xq"].q), ptr(s["xq"].sc), ptr(s["router"]), ptr(s["egu"]), ptr(s["edn"]), ptr(s["sgu"]), ptr(s["sdn"]),
                             c["T"], c["E"], c["F"], c["experts"], c["top"], ptr(s["ids"]), ptr(s["w"]), ptr(s["y"]), ptr(s["ws"]),
                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return s["ids"], s["w"], s["y"]


# ------------------------------------------------------------------ engine level
class _Rows:
    """Rows of one of the engine's own buffers as a tensor that keeps the engine alive."""

    def __init__(self, eng, address, *shape):
        self.eng = eng
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (int(address), False), "version": 2}


def _view(eng, address, rows, width):
    return torch.as_tensor(_Rows(eng, address, rows, width), device="cuda")


def _engine(preset, seed, slots):
    return hb.Engine(hb.ModelCfg.preset(preset, n_slots=slots, seed=seed + 1))


def _prefilled(c, seed, slots, with_mtp):
    """An engine whose slots hold prompts of their own, and per slot the first token and the hidden row behind it."""
    eng = _engine(c["preset"], seed, slots)
    first, h = [], []
    for s in range(slots):
        eng.prefill(s, _prompt(eng.cfg, seed, s, c["ctx"]), with_mtp=with_mtp)
        first.append(int(eng.topk(0, 1)[0][0]))
        h.append(_view(eng, eng.h_nextn_ptr(), 1, eng.cfg.n_embd).clone())
    return eng, first, h


def _prepare_forward(c, seed):
    T = [int(t) for t in c["rows"].split(",")]
    eng, first, _ = _prefilled(c, seed, len(T), False)
    drafts = [_prompt(eng.cfg, seed + 1, s, t - 1) for s, t in enumerate(T)]
    keep = [1 + d % t for d, t in zip(range(2, 2 + len(T)), T)]     # rows of each slot that are then accepted
    return dict(eng=eng, T=T, last=first, pos=[c["ctx"]] * len(T), drafts=drafts, keep=keep)


def _run_forward(c, s):
    eng, T = s["eng"], s["T"]
    for i, t in enumerate(T):
        if s["pos"][i] + t > eng.cfg.max_ctx:
            s["pos"][i] = c["ctx"]
    eng.forward([(i, [s["last"][i]] + s["drafts"][i], s["pos"][i]) for i in range(len(T))])
    ids, vals = eng.topk(0, sum(T))
    r0 = 0
    for i, t in enumerate(T):
        m = s["keep"][i]
        eng.accept(i, m)
        s["last"][i], s["pos"][i] = int(ids[r0 + m - 1]), s["pos"][i] + m
        r0 += t
    return ids, vals, _view(eng, eng.logits_ptr(), r0, eng.cfg.n_vocab), _view(eng, eng.h_nextn_ptr(), r0, eng.cfg.n_embd)


def _prepare_prefill(c, seed):
    eng = _engine(c["preset"], seed, 1)
    return dict(eng=eng, prompt=_prompt(eng.cfg, seed, 0, c["tokens"]))


def _run_prefill(c, s):
    eng = s["eng"]
    eng.reset_slot(0)
    eng.prefill(0, s["prompt"], with_mtp=True)
    ids, vals = eng.topk(0, 1)
    return ids, vals, _view(eng, eng.logits_ptr(), 1, eng.cfg.n_vocab), _view(eng, eng.h_nextn_ptr(), 1, eng.cfg.n_embd)


def _prepare_round(c, seed):
    S = c["slots"]
    eng, first, h = _prefilled(c, seed, S, True)
    s = dict(eng=eng, slots=list(range(S)), first=first, h=h, pos=[0] * S)
    for i in range(S):
        _begin(c, s, i)
    return s


def _begin(c, s, i):
    s["eng"].spec_begin(i, s["first"][i], c["ctx"], s["h"][i].data_ptr())
    s["pos"][i] = c["ctx"]


def _run_round(c, s):
    eng, S, n = s["eng"], c["slots"], c["drafts"]
    for i in range(S):
        if s["pos"][i] + 2 * n + 2 > eng.cfg.max_ctx:    # the context is full: from the end of the prompt again
            _begin(c, s, i)
    out = eng.spec_round_slots(s["slots"], n)
    for i, got in enumerate(out):
        s["pos"][i] += len(got)
    R = S * (n + 1)
    return (out, _view(eng, eng.logits_ptr(), R, eng.cfg.n_vocab), _view(eng, eng.h_nextn_ptr(), R, eng.cfg.n_embd),
            _view(eng, eng.mtp_logits_ptr(), S, eng.cfg.n_vocab), _view(eng, eng.mtp_h_ptr(), S, eng.cfg.n_embd))


_KINDS = {"gemv": (_prepare_gemv, _run_gemv), "gdn": (_prepare_gdn, _run_gdn), "attn": (_prepare_attn, _run_attn), "moe": (_prepare_moe, _run_moe),
          "forward": (_prepare_forward, _run_forward), "prefill": (_prepare_prefill, _run_prefill), "round": (_prepare_round, _run_round)}


def prepare(case, seed):
    make, run_it = _KINDS[case["kind"]]
    return case, run_it, make(case, seed)


def run(state):
    case, run_it, s = state
    return run_it(case, s)


# ------------------------------------------------------------------ bytes and operations of one pass
def _w(n, k):
    return n * (k // 256) * 144


def _experts(n, top, rows):
    """Distinct experts that `rows` rows touch when each takes `top` of `n` evenly."""
    return n * (1.0 - (1.0 - top / n) ** rows)


def _attn_layer(m, rows, seqs, ctx):
    n_in = m.n_head * 512 + 2 * m.n_head_kv * 256
    kv = seqs * ctx * m.n_head_kv * 512 * 2
    return _w(n_in, m.n_embd) + _w(m.n_embd, m.n_head * 256) + kv, 2 * rows * (n_in * m.n_embd + m.n_embd * m.n_head * 256 + 2 * ctx * m.n_head * 256)


def _gdn_layer(m, rows, seqs):
    n_in = (2 * m.gdn_qk_heads + 2 * m.gdn_v_heads) * 128 + 2 * m.gdn_v_heads
    state = m.gdn_v_heads * 128 * 128
    return (_w(n_in, m.n_embd) + _w(m.n_embd, m.gdn_v_heads * 128) + seqs * 2 * state * 4,
            2 * rows * (n_in * m.n_embd + m.n_embd * m.gdn_v_heads * 128 + 3 * state))


def _ffn(m, rows):
    if not m.n_expert:
        return _w(2 * m.n_ff, m.n_embd) + _w(m.n_embd, m.n_ff), 6 * rows * m.n_ff * m.n_embd
    one, F = _w(2 * m.expert_ff, m.n_embd) + _w(m.n_embd, m.expert_ff), m.expert_ff
    return ((_experts(m.n_expert, m.n_expert_used, rows) + 1) * one + (m.n_expert + 1) * m.n_embd * 4,
            2 * rows * (3 * F * m.n_embd * (m.n_expert_used + 1) + (m.n_expert + 1) * m.n_embd))


def _sum(*parts):
    return [sum(p) for p in zip(*parts)]


def _head(m, rows):
    return _w(m.n_vocab, m.n_embd) + rows * m.n_vocab * 4, 2 * rows * m.n_vocab * m.n_embd


def _trunk(m, rows, seqs, ctx, head_rows):
    parts = []
    for il in range(m.n_layer):
        parts += [_attn_layer(m, rows, seqs, ctx) if (il + 1) % m.attn_every == 0 else _gdn_layer(m, rows, seqs), _ffn(m, rows)]
    return _sum(*parts, _head(m, head_rows))


def _draft(m, rows, seqs, ctx):
    eh = (_w(m.n_embd, 2 * m.n_embd), 4 * rows * m.n_embd * m.n_embd)
    return _sum(eh, _attn_layer(m, rows, seqs, ctx), _ffn(m, rows), _head(m, rows))


def _draft_kv(m, rows):
    kv = 2 * m.n_head_kv * 256                           # only the K and V rows of the draft block are wanted
    return _w(m.n_embd, 2 * m.n_embd) + _w(kv, m.n_embd), 2 * rows * (2 * m.n_embd * m.n_embd + kv * m.n_embd)


def work(case):
    c = case
    if c["kind"] == "gemv":
        b, f = _w(c["N"], c["K"]) + 4 * c["R"] * (c["K"] + c["N"]), 2 * c["N"] * c["K"] * c["R"]
    elif c["kind"] == "gdn":
        n_in, Z = (2 * c["n_qk"] + 2 * c["n_v"]) * 128 + 2 * c["n_v"], c["n_v"] * 128
        b = c["n_v"] * 128 * 128 * 4 * (2 if c["replay"] else 1) + 4 * c["T"] * (n_in + 2 * Z) + 4 * c["replay"] * c["n_v"] * 386
        f = 6 * (c["T"] + c["replay"]) * c["n_v"] * 128 * 128
    elif c["kind"] == "attn":
        keys = c["pos"] + c["R"]
        b, f = keys * c["n_kv"] * 512 * 2 + 4 * c["R"] * (c["n_head"] * 768 + c["n_kv"] * 512), 4 * c["R"] * keys * c["n_head"] * 256
    elif c["kind"] == "moe":
        E, F, T = c["E"], c["F"], c["T"]
        b = (_experts(c["experts"], c["top"], T) + 1) * (_w(2 * F, E) + _w(E, F)) + 4 * ((c["experts"] + 1) * E + 2 * T * E)
        f = 2 * T * (3 * E * F * (c["top"] + 1) + (c["experts"] + 1) * E)
    else:
        m = hb.ModelCfg.preset(c["preset"])
        if c["kind"] == "forward":
            T = [int(t) for t in c["rows"].split(",")]
            b, f = _trunk(m, sum(T), len(T), c["ctx"], sum(T))
        elif c["kind"] == "prefill":
            n = c["tokens"]
            b, f = _sum(_trunk(m, n, 1, n / 2, 1), _draft_kv(m, n))
        else:
            S, n = c["slots"], c["drafts"]
            b, f = _sum(_trunk(m, S * (n + 1), S, c["ctx"], S * (n + 1)), [n * v for v in _draft(m, S, S, c["ctx"])], _draft_kv(m, S * n))
    return {"bytes": b, "flops": f}
