"""Kernel-level host API: the Python mirror of the reference's free kernel launchers
(engine/kernels/gemv.h, ops.h). Arguments are torch CUDA tensors; every call goes through the C ABI."""
import ctypes
import functools

import torch

from ._lib import lib, hot, check, ptr

# The calls below are a few microseconds of device work, so what they spend in Python counts: the handle of the current stream
# comes without a Stream object around it, the short calls go through native entry points that take addresses as integers (_lib.hot; to
# a ctypes function an integer would pass as 32 bits, hence the wrapper of _stream), and sizes that depend on shapes alone are computed once (per
# type of the numbers, too: a float or a numpy integer that equals an earlier size is still refused by the library's function).
try:
    _raw_stream, _device = torch._C._cuda_getCurrentRawStream, torch._C._cuda_getDevice
except AttributeError:   # torch without CUDA: the package still imports, and a call raises torch's own error
    _raw_stream, _device = (lambda _: torch.cuda.current_stream().cuda_stream), (lambda: 0)


def _stream():
    return ctypes.c_void_p(_raw_stream(_device()))


@functools.lru_cache(maxsize=256, typed=True)
def _xq8_bytes(R, K):
    return lib().hp_xq8_q_bytes(R, K), lib().hp_xq8_sc_bytes(R, K)


@functools.lru_cache(maxsize=256, typed=True)
def _argmax_scratch_bytes(R, n):
    return lib().hp_argmax_scratch_bytes(R, n)


@functools.lru_cache(maxsize=256, typed=True)
def _attn_workspace_bytes(R, n_head, n_kv, max_ctx):
    return lib().hp_attn_workspace_bytes(R, n_head, n_kv, max_ctx)


class XQ8:
    """Quantised activations (reference: struct XQ8, engine/kernels/gemv.h:8) in the library's private layout."""

    def __init__(self, R, K, device="cuda"):
        self.R, self.K = R, K
        nq, ns = _xq8_bytes(R, K)   # nq is a multiple of 512: the scales stay aligned
        self.q, self.sc = torch.zeros(nq + ns, dtype=torch.uint8, device=device).split((nq, ns))

    def unpack(self):
        """-> (q int8 [R][K], d f32 [R][K/32], s f32 [R][K/32]) in the reference's row layout."""
        q = torch.empty((self.R, self.K), dtype=torch.int8, device=self.q.device)
        d = torch.empty((self.R, self.K // 32), dtype=torch.float32, device=self.q.device)
        s = torch.empty_like(d)
        check(lib().hp_xq8_unpack(ptr(self.q), ptr(self.sc), self.R, self.K, ptr(q), ptr(d), ptr(s), _stream()))
        return q, d, s


def quantize_x_q8(x, xq=None):
    """x f32 [R][K] -> XQ8 (reference quantize_x_q8, gemv.h:9)."""
    stride = x.stride()
    assert x.dtype == torch.float32 and len(stride) == 2 and stride[1] == 1
    R, K = x.shape
    xq = xq or XQ8(R, K, x.device)
    check(hot().hp_quantize_x_q8(x.data_ptr(), stride[0], R, K, xq.q.data_ptr(), xq.sc.data_ptr(), _raw_stream(_device())))
    return xq


def dequant_q4k(w, nblk):
    out = torch.empty(nblk * 256, dtype=torch.float32, device=w.device)
    check(lib().hp_dequant_q4k(ptr(w), ctypes.c_size_t(nblk), ptr(out), _stream()))
    return out


def gemv_q4k_q8(w, xq, N, K, y=None):
    """y [R][N] = W . x for Q4_K W [N][K/256 blocks] (uint8 tensor) and quantised x (reference gemv_wmma, gemv.h:33)."""
    R = xq.R
    if y is None:
        y = torch.empty((R, N), dtype=torch.float32, device=w.device)
    check(hot().hp_gemv_q4k_q8(None if w is None else w.data_ptr(), xq.q.data_ptr(), xq.sc.data_ptr(), y.data_ptr(), N, K, R, y.stride(0), _raw_stream(_device())))
    return y


def gemv_q4k_f32(w, x, N, K):
    """f32-activation baseline (reference gemv_q4_K_f32, gemv.h:57)."""
    R = x.shape[0]
    y = torch.empty((R, N), dtype=torch.float32, device=w.device)
    check(lib().hp_gemv_q4k_f32(ptr(w), ptr(x), ptr(y), N, K, R, _stream()))
    return y


def argmax(logits, n=None):
    """Row-wise argmax (max value, lowest index) -> (ids int32 [R], vals f32 [R]) (reference argmax_topk k=1, ops.h:118)."""
    R, ld = logits.shape[0], logits.stride(0)
    n = n or logits.shape[1]
    dev, nb = logits.device, _argmax_scratch_bytes(R, n)
    ids = torch.empty(R, dtype=torch.int32, device=dev)
    vals = torch.empty(R, dtype=torch.float32, device=dev)
    scratch = torch.empty(nb, dtype=torch.uint8, device=dev) if nb else None
    check(hot().hp_argmax(logits.data_ptr(), R, n, ld, ids.data_ptr(), vals.data_ptr(), scratch.data_ptr() if nb else None, _raw_stream(_device())))
    return ids, vals


def argmax_noalloc(logits, n=None):
    """argmax() through the entry point for callers that cannot allocate device memory: it takes only the input and the two
    output tensors (a C caller creates these beforehand), for at most 32 rows of 524288 entries."""
    R, ld = logits.shape[0], logits.stride(0)
    n = n or logits.shape[1]
    ids = torch.empty(R, dtype=torch.int32, device=logits.device)
    vals = torch.empty(R, dtype=torch.float32, device=logits.device)
    check(lib().hp_argmax_noalloc(ptr(logits), R, n, ld, ptr(ids), ptr(vals), _stream()))
    return ids, vals


def accept_greedy(ids, drafts):
    """-> int32 tensor [mm, bonus] on device (reference host loop, engine/bench/spec27b.cpp:92-97)."""
    out = torch.empty(2, dtype=torch.int32, device=ids.device)
    check(hot().hp_accept_greedy(ids.data_ptr(), drafts.data_ptr(), drafts.numel(), out.data_ptr(), _raw_stream(_device())))
    return out


def device_status():
    check(lib().hp_device_status(_stream()))


def attn_decode(qkv, pos0, n_head, n_kv, n_rot, q_norm, k_norm, rope, kc, vc, max_ctx, eps=1e-6, want_q8=True):
    """GQA decode attention of one sequence: qkv f32 [R][ld] (normalised / rotated in place), rows at positions pos0 + r;
    q_norm / k_norm bf16 [256] (int16 tensors), rope f32 [max_ctx][n_rot/2][2], kc / vc f16 [n_kv][max_ctx][256] (updated).
    -> (out f32 [R][n_head*256], XQ8 of it or None). Reference: qk_norm_rope_kv + attn_decode_mq (ops.h:71-72,96)."""
    R, ld = qkv.shape[0], qkv.stride(0)
    ws = torch.empty(_attn_workspace_bytes(R, n_head, n_kv, max_ctx), dtype=torch.uint8, device=qkv.device)
    out = torch.empty((R, n_head * 256), dtype=torch.float32, device=qkv.device)
    xq = XQ8(R, n_head * 256, qkv.device) if want_q8 else None
    check(hot().hp_attn_decode(qkv.data_ptr(), ld, R, int(pos0), n_head, n_kv, n_rot, None if q_norm is None else q_norm.data_ptr(),
                               None if k_norm is None else k_norm.data_ptr(), None if rope is None else rope.data_ptr(), None if kc is None else kc.data_ptr(),
                               None if vc is None else vc.data_ptr(), int(max_ctx), out.data_ptr(), xq.q.data_ptr() if xq else None, xq.sc.data_ptr() if xq else None,
                               eps, ws.data_ptr(), _raw_stream(_device())))
    return out, xq


def repack_tiled(w, N, K, interleave_half=0):
    """ggml Q4_K [N][K/256 blocks] (uint8 tensor) -> the library's tile-major streaming layout (same bytes, permuted)."""
    L = lib()
    L.hp_q4k_tiled_bytes.restype = ctypes.c_size_t
    L.hp_q4k_tiled_bytes.argtypes = [ctypes.c_size_t, ctypes.c_int]
    out = torch.empty(L.hp_q4k_tiled_bytes(N, K), dtype=torch.uint8, device=w.device)
    check(L.hp_q4k_repack_tiled(ptr(w), ptr(out), ctypes.c_size_t(N), K, interleave_half, _stream()))
    return out


def moe_layer(xn, router, exp_gate_up, exp_down, sh_gate_up, sh_down, F, n_expert, k):
    """One mixture-of-experts FFN over the rows of xn f32 [T][E] -> (ids int32 [T][k+1], weights f32 [T][k+1], y f32 [T][E]).
    The expert tensors are given in ggml order and repacked here (an engine does that once at load).
    Reference: Qwen4Exp::moe_layer (qwen4exp.cpp:345-354)."""
    L = lib()
    L.hp_moe_workspace_bytes.restype = ctypes.c_size_t
    T, E = xn.shape
    xq = quantize_x_q8(xn)
    egu = repack_tiled(exp_gate_up, n_expert * 2 * F, E, F); edn = repack_tiled(exp_down, n_expert * E, F, 0)
    sgu = repack_tiled(sh_gate_up, 2 * F, E, F); sdn = repack_tiled(sh_down, E, F, 0)
    ws = torch.empty(L.hp_moe_workspace_bytes(T, E, F, n_expert, k), dtype=torch.uint8, device=xn.device)
    ids = torch.empty((T, k + 1), dtype=torch.int32, device=xn.device)
    w = torch.empty((T, k + 1), dtype=torch.float32, device=xn.device)
    y = torch.empty((T, E), dtype=torch.float32, device=xn.device)
    check(L.hp_moe_layer(ptr(xn), ptr(xq.q), ptr(xq.sc), ptr(router), ptr(egu), ptr(edn), ptr(sgu), ptr(sdn), T, E, F, n_expert, k,
                         ptr(ids), ptr(w), ptr(y), ptr(ws), _stream()))
    return ids, w, y
