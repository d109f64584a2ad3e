"""Benchmark configuration 2: one Gated-DeltaNet layer verify step at full size (hidden 5120 -> 16 key heads, 48 value heads,
dim 128, conv 4), fp32 state ~ N(0, 0.1), 6 bf16-rounded input rows ~ N(0, 1): per-row state snapshots, rollback to
accepted length k in {0..5}, compared with the sequential one-row-at-a-time scan (GPU and CPU oracle).
The stated tolerance is 1e-5 relative; the CUDA kernel and the oracle actually agree bit for bit.
Mirrors engine/bench/test_fnkernels.cpp:28-53 (same generator style: a_neg = -|N(0,1)|, dt ~ N(0,0.5), norm w = 1+N(0,0.3))."""
import ctypes

import numpy as np
import pytest
import torch

import hipster_b200 as hb
from oracle import orc

pytestmark = pytest.mark.gpu

NQK, NV, D = 16, 48, 128
C = (2 * NQK + NV) * D
LD = C + NV * D + 2 * NV


def bf16_round(a):
    u = np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)
    u = ((u + 0x7FFF + ((u >> 16) & 1)) >> 16).astype(np.uint16)
    return u


def bf16_to_f32(u):
    return (u.astype(np.uint32) << 16).view(np.float32)


def private_conv_state(hist):
    """reference layout [3][C] -> this library's per-value-head layout [n_v][3][q | k | v]."""
    out = np.zeros((NV, 3, 384), dtype=np.float32)
    for h in range(NV):
        hk = h % NQK
        out[h, :, 0:128] = hist[:, hk * D:(hk + 1) * D]
        out[h, :, 128:256] = hist[:, NQK * D + hk * D:NQK * D + (hk + 1) * D]
        out[h, :, 256:384] = hist[:, 2 * NQK * D + h * D:2 * NQK * D + (h + 1) * D]
    return out


class Layer:
    def __init__(self, seed, sigmoid_gate=0):
        rng = np.random.default_rng(seed)
        self.rows = bf16_to_f32(bf16_round(rng.normal(0, 1, size=(6, LD)))).astype(np.float32)
        self.conv_w = rng.normal(0, 0.5, size=(C, 4)).astype(np.float32)
        self.dt = bf16_round(rng.normal(0, 0.5, size=NV)); self.an = bf16_round(-np.abs(rng.normal(0, 1, size=NV)))
        self.nw = bf16_round(1 + rng.normal(0, 0.3, size=D))
        self.state0 = rng.normal(0, 0.1, size=(NV, D, D)).astype(np.float32)
        self.hist0 = rng.normal(0, 1, size=(3, C)).astype(np.float32)
        self.gate = sigmoid_gate
        self.eps = 1e-6

    def dev(self):
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
        d = dict(rows=t(self.rows), conv_w=t(self.conv_w), dt=t(self.dt.view(np.int16)), an=t(self.an.view(np.int16)), nw=t(self.nw.view(np.int16)),
                 state=t(self.state0), conv=t(private_conv_state(self.hist0)),
                 saved=torch.zeros(hb.lib().hp_gdn_saved_floats(NV), dtype=torch.float32, device="cuda"))
        return d

    def call(self, d, rows, T, n_replay, out=None, snap=None):
        L = hb.lib()
        hb.check(L.hp_gdn_layer(hb.ptr(rows), LD, T, n_replay, NQK, NV, hb.ptr(d["conv_w"]), hb.ptr(d["dt"]), hb.ptr(d["an"]), hb.ptr(d["nw"]),
                                hb.ptr(d["state"]), hb.ptr(d["conv"]), hb.ptr(d["saved"]), hb.ptr(out), ctypes.c_void_p(0), ctypes.c_void_p(0),
                                hb.ptr(snap), ctypes.c_float(self.eps), self.gate, ctypes.c_void_p(0)))
        torch.cuda.synchronize()


@pytest.fixture(scope="module")
def setup():
    hb.lib().hp_gdn_saved_floats.restype = ctypes.c_size_t
    hb.lib().hp_gdn_conv_state_floats.restype = ctypes.c_size_t
    return Layer(seed=2)


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


def test_six_row_verify_with_snapshots_matches_sequential_scan(setup):
    Ly = setup
    d = Ly.dev()
    out6 = torch.empty((6, NV * D), dtype=torch.float32, device="cuda"); snap = torch.empty((6, NV, D, D), dtype=torch.float32, device="cuda")
    Ly.call(d, d["rows"], 6, 0, out6, snap)
    # CPU oracle, sequential scan (reference layout of the conv history)
    st = Ly.state0.copy(); hist = Ly.hist0.copy()
    oout, osnap = orc.gdn_rows(Ly.rows, NQK, NV, Ly.conv_w, Ly.dt, Ly.an, Ly.nw, st, hist, Ly.eps, Ly.gate, want_snap=True)
    o = out6.cpu().numpy(); s = snap.cpu().numpy()
    rel = np.max(np.abs(o - oout)) / np.max(np.abs(oout)); rels = np.max(np.abs(s - osnap)) / np.max(np.abs(osnap))
    assert rel < 1e-5 and rels < 1e-5
    assert np.array_equal(bits(o), bits(oout)) and np.array_equal(bits(s), bits(osnap))
    # GPU sequential one-row-at-a-time scan: each call accepts the previous row and processes one new row
    d2 = Ly.dev(); o1 = torch.empty((1, NV * D), dtype=torch.float32, device="cuda")
    for t in range(6):
        Ly.call(d2, d2["rows"][t:t + 1].contiguous(), 1, 1 if t > 0 else 0, o1, None)
        assert np.array_equal(bits(o1.cpu().numpy()[0]), bits(o[t]))
    # the verify pass did not advance the committed state
    assert np.array_equal(bits(d["state"].cpu().numpy()), bits(Ly.state0))


@pytest.mark.parametrize("k", [0, 1, 2, 3, 4, 5])
def test_rollback_to_accepted_length(setup, k):
    """k accepted drafts = the first k+1 of the 6 rows are committed; the committed state must equal snapshot k and the
    state of a sequential scan over k+1 rows; a following row must see exactly that state."""
    Ly = setup
    d = Ly.dev()
    snap = torch.empty((6, NV, D, D), dtype=torch.float32, device="cuda")
    Ly.call(d, d["rows"], 6, 0, None, snap)
    nxt = torch.from_numpy(Ly.rows[5:6].copy()).cuda(); out_next = torch.empty((1, NV * D), dtype=torch.float32, device="cuda")
    Ly.call(d, nxt, 1, k + 1, out_next, None)          # accept k+1 rows, then one more row
    committed = d["state"].cpu().numpy()
    assert np.array_equal(bits(committed), bits(snap[k].cpu().numpy()))
    st = Ly.state0.copy(); hist = Ly.hist0.copy()
    orc.gdn_rows(Ly.rows[:k + 1], NQK, NV, Ly.conv_w, Ly.dt, Ly.an, Ly.nw, st, hist, Ly.eps, Ly.gate)
    assert np.max(np.abs(committed - st)) / np.max(np.abs(st)) < 1e-5
    assert np.array_equal(bits(committed), bits(st))
    assert np.array_equal(bits(d["conv"].cpu().numpy()), bits(private_conv_state(hist)))
    o2, _ = orc.gdn_rows(Ly.rows[5:6], NQK, NV, Ly.conv_w, Ly.dt, Ly.an, Ly.nw, st, hist, Ly.eps, Ly.gate)
    assert np.array_equal(bits(out_next.cpu().numpy()), bits(o2))


def test_commit_only_call_and_sigmoid_gate():
    Ly = Layer(seed=5, sigmoid_gate=1)
    d = Ly.dev()
    out = torch.empty((4, NV * D), dtype=torch.float32, device="cuda")
    Ly.call(d, d["rows"][:4].contiguous(), 4, 0, out, None)
    Ly.call(d, None, 0, 3, None, None)                   # T = 0: commit 3 rows, nothing else
    st = Ly.state0.copy(); hist = Ly.hist0.copy()
    oo, _ = orc.gdn_rows(Ly.rows[:3], NQK, NV, Ly.conv_w, Ly.dt, Ly.an, Ly.nw, st, hist, Ly.eps, 1)
    assert np.array_equal(bits(d["state"].cpu().numpy()), bits(st))
    assert np.array_equal(bits(out.cpu().numpy()[:3]), bits(oo))


@pytest.mark.parametrize("gate", [0, 1])
def test_kernel_within_1e5_of_the_double_precision_transcription(gate):
    """The stated tolerance of configuration 2 against a checker that owes nothing to this build's kernels: the reference's
    conv + step source (engine/kernels/ops.hip:188-256) evaluated in double precision. Outputs of the 6 rows, every
    per-row state snapshot and the committed state agree within 1e-5 of the largest magnitude."""
    lay = Layer(seed=5, sigmoid_gate=gate)
    d = lay.dev()
    out = torch.zeros((6, NV * D), dtype=torch.float32, device="cuda")
    snap = torch.zeros((6, NV, D, D), dtype=torch.float32, device="cuda")
    lay.call(d, d["rows"], 6, 0, out=out, snap=snap)
    lay.call(d, None, 0, 6)                                   # commit all six rows
    st64 = lay.state0.astype(np.float64); hist64 = lay.hist0.astype(np.float64)
    snaps64 = []
    outs64 = []
    for r in range(6):
        outs64.append(orc.ref64_gdn_rows(lay.rows[r:r + 1], NQK, NV, lay.conv_w.reshape(-1), bf16_to_f32(lay.dt), bf16_to_f32(lay.an), bf16_to_f32(lay.nw),
                                         st64, hist64, lay.eps, gate)[0])
        snaps64.append(st64.copy())
    out64 = np.stack(outs64); snap64 = np.stack(snaps64)
    o = out.cpu().numpy().astype(np.float64); sn = snap.cpu().numpy().astype(np.float64); st = d["state"].cpu().numpy().astype(np.float64)
    assert np.abs(o - out64).max() <= 1e-5 * np.abs(out64).max()
    assert np.abs(sn - snap64).max() <= 1e-5 * np.abs(snap64).max()
    assert np.abs(st - st64).max() <= 1e-5 * np.abs(st64).max()


def test_weights_written_on_the_stream_right_before(setup):
    """Conv taps and norm weights change between two calls, by kernels on the stream, with and without a quantiser (which
    triggers early launches in its first instruction) in between. No rows are committed, so the state stays."""
    from hipster_b200 import kernels as K_
    T = 6
    a, b = setup, Layer(seed=3)
    d, e = a.dev(), b.dev()
    cw, nw = [d["conv_w"].clone(), e["conv_w"].clone()], [d["nw"].clone(), e["nw"].clone()]
    x = d["rows"][:, :512].contiguous(); xq = K_.XQ8(T, 512); s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def call(out):
        L = hb.lib()
        hb.check(L.hp_gdn_layer(hb.ptr(d["rows"]), LD, T, 0, NQK, NV, hb.ptr(d["conv_w"]), hb.ptr(d["dt"]), hb.ptr(d["an"]), hb.ptr(d["nw"]),
                                hb.ptr(d["state"]), hb.ptr(d["conv"]), hb.ptr(d["saved"]), hb.ptr(out), ctypes.c_void_p(0), ctypes.c_void_p(0),
                                ctypes.c_void_p(0), ctypes.c_float(a.eps), a.gate, s))
        return out
    new = lambda: torch.empty((T, NV * D), device="cuda")
    want = []
    for i in range(2):
        d["conv_w"].copy_(cw[i]); d["nw"].copy_(nw[i]); torch.cuda.synchronize()
        want.append(call(new())); torch.cuda.synchronize()
    assert not torch.equal(want[0], want[1])
    got = []
    for i in range(40):
        torch.mul(cw[i % 2], 1.0, out=d["conv_w"]); torch.bitwise_or(nw[i % 2], 0, out=d["nw"])
        if i % 4 < 2:
            K_.quantize_x_q8(x, xq)
        got.append(call(new()))
    for i, o in enumerate(got):
        assert torch.equal(o.view(torch.int32), want[i % 2].view(torch.int32)), i


class _Gdn(ctypes.Structure):   # struct GdnParams (csrc/kernels.h)
    _fields_ = [(n, t) for t, names in ((ctypes.c_void_p, "rows saved"), (ctypes.c_size_t, "saved_stride"), (ctypes.c_int, "ld off_z off_b off_a n_qk n_v"),
                                        (ctypes.c_void_p, "conv_w dt_bias a_neg norm_w state conv_state"), (ctypes.c_size_t, "state_stride conv_stride"),
                                        (ctypes.c_void_p, "seq replay_n"), (ctypes.c_int, "imm_T imm_replay"), (ctypes.c_void_p, "out q sc snap"),
                                        (ctypes.c_size_t, "snap_row_stride"), (ctypes.c_float, "eps"), (ctypes.c_int, "sigmoid_gate"), (ctypes.c_bool, "late")) for n in names.split()]


@pytest.mark.parametrize("Ts,reps", [((1, 8, 3), (0, 8, 2)), ((8, 8, 8), (8, 1, 0)), ((0, 2, 5), (3, 0, 7)), ((0, 0, 0), (1, 8, 0)), ((4, 1, 2), (1, 2, 4))])
@pytest.mark.parametrize("n_qk,n_v", [(2, 4), (1, 3)])
def test_three_sequences_take_the_wide_kernel_and_match_one_at_a_time(Ts, reps, n_qk, n_v):
    """Passes over three or more sequences run another kernel (csrc/ops.cu, k_gdn_wide) than one sequence by itself: outputs, state,
    history and saved rows have the same bits, for rows and replayed rows at both ends of their range."""
    f = getattr(hb.lib(), "_ZN2hp11gdn_forwardERKNS_9GdnParamsEiP11CUstream_st")
    f.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
    g = torch.Generator(device="cuda").manual_seed(sum(Ts) + n_v)
    rnd = lambda *s, std=1.0, mean=0.0: torch.randn(s, device="cuda", generator=g) * std + mean  # noqa: E731
    bf = lambda t: t.bfloat16().view(torch.int16)  # noqa: E731
    ld, R, K = (2 * n_qk + 2 * n_v) * 128 + 2 * n_v, max(sum(Ts), 1), n_v * 128
    w = dict(rows=rnd(R, ld), conv_w=rnd((2 * n_qk + n_v) * 128, 4, std=0.5), dt_bias=bf(rnd(n_v, std=0.5)), a_neg=bf(-rnd(n_v).abs()), norm_w=bf(rnd(128, std=0.3, mean=1.0)))
    mut = dict(state=rnd(3, n_v, 128, 128, std=0.1), conv_state=rnd(3, n_v, 3, 384), saved=rnd(3, n_v, 8, 388))
    res = []
    for together in (True, False):
        m = {k: v.clone() for k, v in mut.items()}
        out, xq = torch.zeros((R, K), device="cuda"), hb.kernels.XQ8(R, K)
        p = _Gdn(ld=ld, off_z=(2 * n_qk + n_v) * 128, off_b=(2 * n_qk + 2 * n_v) * 128, off_a=(2 * n_qk + 2 * n_v) * 128 + n_v, n_qk=n_qk, n_v=n_v, out=out.data_ptr(), q=xq.q.data_ptr(),
                 sc=xq.sc.data_ptr(), saved_stride=n_v * 8 * 388, state_stride=n_v * 128 * 128, conv_stride=n_v * 3 * 384, eps=1e-6, **{k: v.data_ptr() for k, v in {**w, **m}.items()})
        seq = torch.tensor([[sum(Ts[:i]), Ts[i], i, 0] for i in range(3)], dtype=torch.int32, device="cuda"); rep = torch.tensor(reps, dtype=torch.int32, device="cuda")
        p.replay_n = rep.data_ptr()
        for i in [None] if together else range(3):
            p.seq = seq.data_ptr() + (16 * i if i else 0)
            hb.check(f(ctypes.addressof(p), 3 if together else 1, torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        res.append([out, xq.q, xq.sc, m["state"], m["conv_state"], m["saved"]])
    for a, b in zip(*res):
        assert torch.equal(a.contiguous().view(torch.uint8), b.contiguous().view(torch.uint8))
