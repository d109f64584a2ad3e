"""Parity of the CUDA Q4_K GEMV path (through the C ABI) with the CPU oracle. Bit-exact for the quantised
activations, the dequantised weights, the int8-activation GEMV, the f32-activation GEMV, argmax and acceptance."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

import hipster_b200 as hb
from hipster_b200 import kernels as K_, synth
from oracle import orc

pytestmark = pytest.mark.gpu
ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


def test_dequant_q4k_bit_exact():
    W = synth.q4k_matrix(64, 1024, seed=11)
    got = K_.dequant_q4k(dev(W), 64 * 4).cpu().numpy()
    assert np.array_equal(bits(got), bits(orc.dequant_q4k(W)))


@pytest.mark.parametrize("R,K", [(1, 256), (3, 5120), (6, 17408), (9, 512), (24, 2048)])
def test_quantize_x_q8_bit_exact(R, K):
    x = synth.activations(R, K, seed=R * 7 + 1)
    x[0, 64:96] = 0.0
    xq = K_.quantize_x_q8(dev(x))
    q, d, s = [t.cpu().numpy() for t in xq.unpack()]
    oq, od, os_ = orc.quantize_x_q8(x)
    assert np.array_equal(q, oq) and np.array_equal(bits(d), bits(od)) and np.array_equal(bits(s), bits(os_))


@pytest.mark.parametrize("N,K,R", [(16, 256, 1), (48, 1024, 3), (512, 5120, 6), (100, 768, 2), (40, 2048, 8),
                                     (64, 1024, 9), (128, 2048, 24), (32, 17408, 6), (7, 512, 5),
                                     (256, 6144, 24), (80, 6144, 12), (48, 9216, 32)])   # the last three: activations read from L2 (too large to stage)
def test_gemv_q8_bit_exact_vs_oracle(N, K, R):
    W = synth.q4k_matrix(N, K, seed=N + K); x = synth.activations(R, K, seed=R)
    xq = K_.quantize_x_q8(dev(x))
    y = K_.gemv_q4k_q8(dev(W), xq, N, K).cpu().numpy()
    K_.device_status()
    q, d, s = orc.quantize_x_q8(x)
    want = orc.gemv_q4k_q8(W, q, d, s, N, K)
    assert np.array_equal(bits(y), bits(want))


# up to 4 rows take the form that holds each column twice, 5 the full tile: one tile, a ragged last one, odd and even K parts, a tile shared by all warps
@pytest.mark.parametrize("R", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("N,K", [(16, 256), (50, 768), (100, 5120), (7, 17408)])
def test_gemv_q8_few_rows_bit_exact_vs_oracle(N, K, R):
    W = synth.q4k_matrix(N, K, seed=N); x = synth.activations(R, K, seed=R)
    y = K_.gemv_q4k_q8(dev(W), K_.quantize_x_q8(dev(x)), N, K).cpu().numpy()
    K_.device_status()
    assert np.array_equal(bits(y), bits(orc.gemv_q4k_q8(W, *orc.quantize_x_q8(x), N, K)))


def test_gemv_q8_row_result_independent_of_row_count():
    # the reference's T-invariance contract (README.md:65: T>1 vs T=1 logit difference 0.0000)
    N, K = 256, 5120
    W = dev(synth.q4k_matrix(N, K, seed=3)); x = synth.activations(24, K, seed=4)
    y24 = K_.gemv_q4k_q8(W, K_.quantize_x_q8(dev(x)), N, K).cpu().numpy()
    for r in (0, 5, 8, 23):
        y1 = K_.gemv_q4k_q8(W, K_.quantize_x_q8(dev(x[r:r + 1])), N, K).cpu().numpy()
        assert np.array_equal(bits(y1[0]), bits(y24[r]))
    y6 = K_.gemv_q4k_q8(W, K_.quantize_x_q8(dev(x[:6])), N, K).cpu().numpy()
    assert np.array_equal(bits(y6), bits(y24[:6]))


@pytest.mark.parametrize("N,K,R", [(64, 1024, 1), (200, 5120, 3), (33, 768, 8)])
def test_gemv_f32_bit_exact_vs_oracle(N, K, R):
    W = synth.q4k_matrix(N, K, seed=N); x = synth.activations(R, K, seed=R + 100)
    y = K_.gemv_q4k_f32(dev(W), dev(x), N, K).cpu().numpy()
    assert np.array_equal(bits(y), bits(orc.gemv_q4k_f32(W, x, N, K, tpr=4)))


def test_argmax_and_accept():
    rng = np.random.default_rng(0)
    lg = rng.normal(size=(6, 248320)).astype(np.float32)
    lg[1, 100] = lg[1, 200000] = 50.0      # tie across chunks -> lower index
    lg[2, 248319] = 60.0
    lg[3, 0] = 60.0
    ids, vals = K_.argmax(dev(lg))
    oi, ov = orc.argmax(lg)
    assert np.array_equal(ids.cpu().numpy(), oi) and np.array_equal(bits(vals.cpu().numpy()), bits(ov))
    for drafts in ([int(oi[0]), int(oi[1]), 5, int(oi[3]), 7], [1, 2, 3, 4, 5], [int(v) for v in oi[:5]]):
        out = K_.accept_greedy(ids, dev(np.array(drafts, dtype=np.int32))).cpu().numpy()
        assert tuple(out) == orc.accept(oi, drafts)


# one CTA per row for short rows, clusters for longer ones; pieces that are empty, ragged and unaligned rows (odd ld), ties across pieces
@pytest.mark.parametrize("n,ld", [(1, 1), (7, 9), (4095, 4096), (4096, 4096), (4097, 4097), (4100, 4100), (70001, 70003), (262147, 262148)])
def test_argmax_at_the_edges_of_its_pieces(n, ld):
    rng = np.random.default_rng(n)
    a = rng.normal(size=(5, ld)).astype(np.float32)
    a[:, n:] = 1e9                                                       # beyond the row: not looked at
    a[0, n - 1] = 50.0
    a[1, :n] = a[1, 0]                                                   # all equal: the lowest index
    a[2, n // 2] = a[2, n - 1] = 50.0
    a[3, :n] = -np.inf; a[3, n // 3] = -1.0
    a[4, : n - 1] = np.nan if n > 1 else a[4, : n - 1]; a[4, n - 1] = -3.0   # NaN never wins
    ids, vals = K_.argmax(dev(a), n)
    want = [n - 1, 0, n // 2, n // 3, n - 1]
    assert ids.cpu().tolist() == want and np.array_equal(bits(vals.cpu().numpy()), bits(a[range(5), want]))
    none, v = K_.argmax(dev(np.full((1, n), -np.inf, np.float32)))
    assert none.item() == -1 and v.item() == -np.inf


# both sides of every line between the forms (rows of one CTA, of 8 small ones, of 8, of 16 for up to 12 rows, two launches for up to 5),
# rows that start at every offset from a 16-byte boundary; the maximum in front of the first whole group, behind the last, tied with the middle
@pytest.mark.parametrize("R,n", [(2, 3), (2, 32768), (2, 32769), (3, 65536), (3, 65537), (2, 262144), (12, 262147), (13, 262147), (1, 524288), (5, 524289), (6, 524289), (1, 1 << 21)])
def test_argmax_forms(R, n):
    for off in (0, 1, 3):
        buf = torch.randn((R, n + 4 + (off & 1)), device="cuda"); x = buf[:, off:off + n]
        buf[:, :off] = 1e9; buf[:, off + n:] = 1e9
        want = x.argmax(1).tolist()
        for r, (hi, lo) in enumerate([(n - 1, n - 1), (n // 2, 0), (n - 1, n // 3), (1, 0)][:R]):
            x[r, hi] = x[r, lo] = 50.0
            want[r] = lo
        ids, vals = K_.argmax(x)
        assert ids.tolist() == want and torch.equal(vals, x[torch.arange(R), torch.tensor(want)])


def test_config1_kernel_check_full_size():
    """Benchmark configuration 1: N=17408 x K=5120 Q4_K, 3 f32 activation rows, seed 0 -> GEMV, per-row argmax, greedy
    acceptance against 2 seeded draft ids; CUDA vs the CPU restatement, plus the reference's own tolerance rule."""
    N, K, R = 17408, 5120, 3
    W = synth.q4k_matrix(N, K, seed=0); x = synth.activations(R, K, seed=0)
    Wd = dev(W)
    xq = K_.quantize_x_q8(dev(x))
    y = K_.gemv_q4k_q8(Wd, xq, N, K)
    ids, _ = K_.argmax(y)
    q, d, s = orc.quantize_x_q8(x)
    want = orc.gemv_q4k_q8(W, q, d, s, N, K)
    assert np.array_equal(bits(y.cpu().numpy()), bits(want))
    oi, _ = orc.argmax(want)
    assert np.array_equal(ids.cpu().numpy(), oi)
    rng = np.random.default_rng(0)
    drafts = np.array([oi[0], oi[1] if rng.random() < 0.5 else (oi[1] + 1) % N], dtype=np.int32)
    assert tuple(K_.accept_greedy(ids, dev(drafts)).cpu().numpy()) == orc.accept(oi, drafts)
    # reference acceptance rule (bench_gemv.cpp:111): maxrel < 1e-5 vs dequantised weights . quantised x in double
    xr = (q.astype(np.float32).reshape(R, -1, 32) * d[:, :, None]).reshape(R, K).astype(np.float32)
    ref, mag = orc.gemv_q4k_double(W, xr, N, K)
    assert np.max(np.abs(ref - y.cpu().numpy()) / (mag + 1e-20)) < 1e-5
    # f32-activation kernel on the same inputs, bit-exact vs its restatement, and argmax agreement is reported
    yf = K_.gemv_q4k_f32(Wd, dev(x), N, K).cpu().numpy()
    assert np.array_equal(bits(yf), bits(orc.gemv_q4k_f32(W, x, N, K, tpr=4)))


def test_bad_arguments_are_rejected_not_launched():
    W = torch.zeros(144 * 16, dtype=torch.uint8, device="cuda")
    xq = K_.XQ8(1, 256)
    with pytest.raises(hb.HipsterError):
        K_.gemv_q4k_q8(W, xq, 16, 100)         # K not a multiple of 256
    with pytest.raises(hb.HipsterError):
        K_.gemv_q4k_q8(W[1:], xq, 16, 256)     # misaligned weights


def test_all_zero_and_tiny_activations():
    """A 32-element sub-block of zeros quantises to d = 0, q = 0 (no 0/0), and a whole zero row gives exact zeros."""
    N, K = 48, 512
    W = synth.q4k_matrix(N, K, seed=3)
    x = synth.activations(3, K, seed=4); x[1] = 0.0; x[2, 64:96] = 0.0; x[0, :32] = 1e-30
    xq = K_.quantize_x_q8(dev(x))
    q, d, s = [t.cpu().numpy() for t in xq.unpack()]
    oq, od, os_ = orc.quantize_x_q8(x)
    assert np.array_equal(q, oq) and np.array_equal(bits(d), bits(od)) and np.array_equal(bits(s), bits(os_))
    y = K_.gemv_q4k_q8(dev(W), xq, N, K).cpu().numpy()
    assert np.array_equal(bits(y), bits(orc.gemv_q4k_q8(W, oq, od, os_, N, K)))
    assert not y[1].any() and np.isfinite(y).all()


# Weights written by a kernel right in front of the call: plain (a torch kernel), by a kernel of this library that triggers
# early launches in its first instruction (its output taken as the next weights), and inside a captured graph.
@pytest.mark.parametrize("N,K", [(4096, 5120), (4999, 512), (16, 256)])   # 4, 2 and 1 K parts; a ragged last tile
def test_gemv_q8_weights_written_on_the_stream_right_before(N, K):
    R = 3
    Ws = [synth.q4k_matrix(N, K, seed=s) for s in (1, 2)]; x = synth.activations(R, K, seed=5)
    q, d, s = orc.quantize_x_q8(x)
    want = [bits(orc.gemv_q4k_q8(w, q, d, s, N, K)) for w in Ws]
    key = dev(Ws[0].reshape(-1) ^ Ws[1].reshape(-1)); W = dev(Ws[1].reshape(-1)); xd = dev(x); xq = K_.XQ8(R, K)
    ys = []
    for _ in range(40):
        W.bitwise_xor_(key)                              # the other matrix, written by a kernel
        K_.quantize_x_q8(xd, xq)
        ys.append(K_.gemv_q4k_q8(W, xq, N, K))
    W.bitwise_xor_(key)
    ys.append(K_.gemv_q4k_q8(W, xq, N, K))               # the writer is the kernel directly in front
    for i, y in enumerate(ys):
        assert np.array_equal(bits(y.cpu().numpy()), want[i % 2]), i
    K_.device_status()


def test_gemv_q8_weights_written_by_an_early_triggering_kernel():
    xa, Wa = dev(synth.activations(32, 5120, seed=1)), [dev(synth.q4k_matrix(1152, 5120, seed=s)) for s in (2, 3)]
    xb = K_.quantize_x_q8(dev(synth.activations(2, 256, seed=4))); qa, qb = K_.quantize_x_q8(xa), K_.XQ8(2, 256)
    src = dev(synth.activations(2, 256, seed=4))
    w = torch.empty((32, 1152), device="cuda")           # [1024] rows of one block: any bytes are a matrix
    got = []
    for i in range(20):
        K_.gemv_q4k_q8(Wa[i % 2], qa, 1152, 5120, w)
        K_.quantize_x_q8(src, qb)
        got.append(K_.gemv_q4k_q8(w.view(torch.uint8), qb, 1024, 256))
    for i in range(2):
        K_.gemv_q4k_q8(Wa[i], qa, 1152, 5120, w)
        torch.cuda.synchronize()
        want = K_.gemv_q4k_q8(w.view(torch.uint8), xb, 1024, 256).view(torch.int32)
        for y in got[i::2]:
            assert torch.equal(y.view(torch.int32), want)


@pytest.mark.parametrize("N,K", [(4096, 5120), (4999, 512)])
def test_gemv_chain_captured_behind_copies_kernels_and_joins(N, K):
    R = 3
    Ws = [synth.q4k_matrix(N, K, seed=s) for s in (1, 2)]; x = synth.activations(R, K, seed=5)
    q, d, s = orc.quantize_x_q8(x)
    want = [bits(orc.gemv_q4k_q8(w, q, d, s, N, K)) for w in Ws]
    Wd = [dev(w.reshape(-1)) for w in Ws]; src = Wd[0].clone(); W = torch.zeros_like(src); xd = dev(x); xq = K_.XQ8(R, K)
    zero = torch.zeros_like(src); drafts = torch.zeros(R - 1, dtype=torch.int32, device="cuda")
    K_.accept_greedy(K_.argmax(K_.gemv_q4k_q8(W, K_.quantize_x_q8(xd, xq), N, K))[0], drafts)   # workspaces exist before the capture
    torch.cuda.synchronize()
    for writer in ("kernel", "copy", "join"):
        g, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.graph(g):
            main = torch.cuda.current_stream()
            if writer == "join":
                side.wait_stream(main)
                with torch.cuda.stream(side):
                    torch.bitwise_xor(src, zero, out=W)
            K_.quantize_x_q8(xd, xq)
            if writer == "kernel":
                torch.bitwise_xor(src, zero, out=W)
            elif writer == "copy":
                W.copy_(src)
            else:
                main.wait_stream(side)
            y = K_.gemv_q4k_q8(W, xq, N, K)
            out = K_.accept_greedy(K_.argmax(y)[0], drafts)
        for i in (0, 1, 0):
            src.copy_(Wd[i]); y.zero_(); out.fill_(-1)
            g.replay()
            torch.cuda.synchronize()
            assert np.array_equal(bits(y.cpu().numpy()), want[i]), (writer, i)
            ids = orc.argmax(want[i].view(np.float32))[0]
            mm = next((j for j in range(R - 1) if ids[j] != 0), R - 1)
            assert out.cpu().tolist() == [mm, int(ids[mm])]
    K_.device_status()


# cuGraphGetEdges_v2 by ctypes, into arrays that live until they are read (the cuda.bindings call of the same name hands out edge data
# of an array that it has freed). An edge is two node handles and 8 bytes of data: from port, to port, type (1 = programmatic), reserved.
_EDGES = """
import ctypes
import torch
from hipster_b200 import kernels as K_
w = torch.zeros(4096 * 144 * 2, dtype=torch.uint8, device="cuda"); x = torch.ones((3, 512), device="cuda"); xq = K_.XQ8(3, 512); y = torch.empty((3, 4096), device="cuda")
K_.gemv_q4k_q8(w, K_.quantize_x_q8(x, xq), 4096, 512, y); torch.cuda.synchronize()
g = torch.cuda.CUDAGraph(keep_graph=True)
with torch.cuda.graph(g):
    K_.gemv_q4k_q8(w, K_.quantize_x_q8(x, xq), 4096, 512, y)
get = ctypes.CDLL("libcuda.so.1").cuGraphGetEdges_v2
get.argtypes = [ctypes.c_void_p] * 5
src, dst, data, n = (ctypes.c_void_p * 16)(), (ctypes.c_void_p * 16)(), (ctypes.c_ubyte * 8 * 16)(*[(ctypes.c_ubyte * 8)(*[255] * 8) for _ in range(16)]), ctypes.c_size_t(16)
err = get(g.raw_cuda_graph(), src, dst, data, ctypes.byref(n))
assert err == 0 and n.value >= 1, (err, n.value)
types = [e[2] for e in data[:n.value]]
assert set(types) <= {0, 1}, types      # the arrays were filled with 255
print("edges", sum(types))
"""


@pytest.mark.parametrize("env,want", [({}, 1), ({"HIPSTER_B200_NO_PDL": "1"}, 0), ({"HIPSTER_B200_PDL_OFF": "64"}, 0)])
def test_public_gemv_honours_the_early_launch_switches(env, want):
    """Programmatic edges of a captured quantise + GEMV call (one K part: two nodes, one edge between them)."""
    clean = {k: v for k, v in os.environ.items() if not k.startswith("HIPSTER_B200_NO_PDL") and not k.startswith("HIPSTER_B200_PDL_OFF")}
    r = subprocess.run([sys.executable, "-c", _EDGES], cwd=ROOT, env={**clean, **env}, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split()[-1] == str(want), r.stdout
