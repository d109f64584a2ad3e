// Per-row argmax over the vocabulary and greedy prefix acceptance, on device.
// Reference: k_topk with k = 1 (engine/kernels/ops.hip:702-716: maximum value, ties -> lowest index) and the
// host acceptance loop of the MTP driver (engine/bench/spec27b.cpp:92-97). The reference copies the ids to the
// host and compares there; here the comparison runs on the device so that no logits or ids round-trip is needed.
#include "hp_common.cuh"
#include "kernels.h"

namespace hp {
namespace {

constexpr int AM_CHUNK = 8192;   // elements per stage-1 block of the top-k

__device__ __forceinline__ void am_better(float& bv, int& bi, float v, int i) {
    if (v > bv || (v == bv && i < bi && i >= 0)) { bv = v; bi = i; }
}
__device__ __forceinline__ void am_block_reduce(float& bv, int& bi, float* sv, int* si) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, off); const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
        am_better(bv, bi, ov, oi);
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) { sv[w] = bv; si[w] = bi; }
    __syncthreads();
    if (w == 0) {
        bv = l < (int)(blockDim.x >> 5) ? sv[l] : -INFINITY; bi = l < (int)(blockDim.x >> 5) ? si[l] : -1;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, off); const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
            am_better(bv, bi, ov, oi);
        }
    }
}
// One cluster of up to 8 CTAs per row, each with a contiguous piece of it; the CTAs' winners meet in the first one's shared memory.
// Bound by latency: one launch instead of a partial and a final one, and no scratch (back to back, 248320 entries: 1 row 3.5 -> 3.9
// us, 6 rows 3.9 and 3.9, 24 rows 5.5 -> 4.7; a caller saves a launch and an allocation).
// -inf (an absent entry, or a real one) and NaN never win; a row of nothing else yields -1.
constexpr int AM_CL = 8, AM_THREADS = 512;
template <int CL>
__global__ void __launch_bounds__(AM_THREADS) k_argmax(const float* __restrict__ x, int n, int ld, int* __restrict__ ids, float* __restrict__ vals) {
    __shared__ float sv[AM_THREADS / 32]; __shared__ int si[AM_THREADS / 32];
    __shared__ float cv[CL]; __shared__ int ci[CL];
    pdl_launch_dependents();
    if constexpr (CL > 1) cluster_arrive_relaxed();   // matched by cluster_wait(): every CTA has started before the first store into another one
    const int r = blockIdx.x / CL, rank = blockIdx.x % CL, tid = threadIdx.x;
    const int per = (n + 4 * CL - 1) / (4 * CL) * 4, c0 = min(n, rank * per), c1 = min(n, c0 + per);
    const float* xr = x + (size_t)r * ld;
    pdl_wait();
    float bv = -INFINITY; int bi = -1;
    const bool vec = (reinterpret_cast<uintptr_t>(xr) & 15) == 0;
    const int v1 = vec ? c0 + ((c1 - c0) & ~3) : c0;   // [c0, v1) by 128-bit loads, 16 of a thread in flight; the rest one by one
    constexpr int NV = 16;
    for (int b = c0 + 4 * tid; b < v1; b += 4 * AM_THREADS * NV) {
        float4 v[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) { const int i = b + 4 * AM_THREADS * k; v[k] = i < v1 ? *reinterpret_cast<const float4*>(xr + i) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY); }
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const int i = b + 4 * AM_THREADS * k;
            if (v[k].x > bv) { bv = v[k].x; bi = i; }
            if (v[k].y > bv) { bv = v[k].y; bi = i + 1; }
            if (v[k].z > bv) { bv = v[k].z; bi = i + 2; }
            if (v[k].w > bv) { bv = v[k].w; bi = i + 3; }
        }
    }
#pragma unroll 4
    for (int i = v1 + tid; i < c1; i += AM_THREADS) am_better(bv, bi, xr[i], i);
    am_block_reduce(bv, bi, sv, si);
    if constexpr (CL > 1) {
        cluster_wait();
        if (tid == 0) { st_cluster_f32(&cv[rank], 0, bv); st_cluster_f32(reinterpret_cast<float*>(&ci[rank]), 0, __int_as_float(bi)); }
        cluster_sync_all();
        if (rank == 0 && tid == 0) {
            bv = cv[0]; bi = ci[0];
#pragma unroll
            for (int k = 1; k < CL; ++k) am_better(bv, bi, cv[k], ci[k]);
        }
    }
    if (rank == 0 && tid == 0) { ids[r] = bi; if (vals) vals[r] = bv; }
}
// ---- top-k per row (k <= TOPK_MAX), values descending, ties -> lower index (reference k_topk, ops.hip:702-716: k rounds
// of a masked arg-max). Stage 1: each block holds a chunk of the row in shared memory and extracts the chunk's own top k by
// k rounds of a block arg-max, masking each winner; stage 2 merges the np * k candidates of a row the same way. The k
// largest of the row are among the k largest of every chunk, so the result equals k rounds over the whole row.
constexpr int TOPK_MAX = 32;
__global__ void __launch_bounds__(256) k_topk_part(const float* __restrict__ x, int n, int ld, int k, float* __restrict__ pv, int* __restrict__ pi) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float buf[AM_CHUNK]; __shared__ float sv[8]; __shared__ int si[8]; __shared__ int s_win;
    const int r = blockIdx.y, c0 = blockIdx.x * AM_CHUNK, cn = min(n - c0, AM_CHUNK);
    const float* xr = x + (size_t)r * ld + c0;
    for (int i = threadIdx.x; i < cn; i += 256) buf[i] = xr[i];
    __syncthreads();
    for (int rd = 0; rd < k; ++rd) {
        float bv = -INFINITY; int bi = -1;
        for (int i = threadIdx.x; i < cn; i += 256) { const float v = buf[i]; if (v > bv) { bv = v; bi = c0 + i; } }
        am_block_reduce(bv, bi, sv, si);
        if (threadIdx.x == 0) { const size_t o = ((size_t)r * gridDim.x + blockIdx.x) * k + rd; pv[o] = bv; pi[o] = bi; s_win = bi; }
        __syncthreads();
        if (threadIdx.x == 0 && s_win >= 0) buf[s_win - c0] = -INFINITY;   // taken (an entry equal to -inf is never selected, as in the reference)
        __syncthreads();
    }
}
__global__ void __launch_bounds__(256) k_topk_final(const float* __restrict__ pv, const int* __restrict__ pi, int nc, int k, int* __restrict__ ids, float* __restrict__ vals) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float cv[64 * TOPK_MAX]; __shared__ int ci[64 * TOPK_MAX]; __shared__ float sv[8]; __shared__ int si[8]; __shared__ int s_win;
    const int r = blockIdx.x;
    for (int i = threadIdx.x; i < nc; i += 256) { cv[i] = pv[(size_t)r * nc + i]; ci[i] = pi[(size_t)r * nc + i]; }
    __syncthreads();
    for (int rd = 0; rd < k; ++rd) {
        float bv = -INFINITY; int bi = -1;
        for (int i = threadIdx.x; i < nc; i += 256) if (ci[i] >= 0) am_better(bv, bi, cv[i], ci[i]);
        am_block_reduce(bv, bi, sv, si);
        if (threadIdx.x == 0) { ids[(size_t)r * k + rd] = bi; if (vals) vals[(size_t)r * k + rd] = bv; s_win = bi; }
        __syncthreads();
        for (int i = threadIdx.x; i < nc; i += 256) if (ci[i] == s_win) ci[i] = -1;   // taken
        __syncthreads();
    }
}
// out[0] = mm (accepted drafts), out[1] = bonus token ids[mm]
__global__ void k_accept(const int* __restrict__ ids, const int* __restrict__ drafts, int n_draft, int* __restrict__ out) {
    pdl_launch_dependents();
    pdl_wait();
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        int mm = 0; while (mm < n_draft && ids[mm] == drafts[mm]) ++mm;
        out[0] = mm; out[1] = ids[mm];
    }
}

// Limits of the allocation-free entry point: part of its interface
constexpr int AM_STATIC_ROWS = 32, AM_STATIC_N = 64 * AM_CHUNK;

// rows of up to 4096 entries take one CTA, longer ones a cluster
int launch_argmax(const float* logits, int R, int n, int ld, int* ids, float* vals, cudaStream_t s) {
    if (n <= 4096) { HP_CUDA(launch_pdl<1>(k_argmax<1>, dim3(R), dim3(AM_THREADS), 0, s, logits, n, ld, ids, vals)); return HP_OK; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(R * AM_CL); cfg.blockDim = dim3(AM_THREADS); cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension; at[0].val.clusterDim.x = AM_CL; at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = (pdl_off_mask(s) & 1) ? 1 : 2;
    HP_CUDA(cudaLaunchKernelEx(&cfg, k_argmax<AM_CL>, logits, n, ld, ids, vals));
    return HP_OK;
}

}  // namespace

size_t argmax_scratch_bytes(int R, int n) { return (size_t)R * ((n + AM_CHUNK - 1) / AM_CHUNK) * 8; }

int argmax_rows(const float* logits, int R, int n, int ld, int* ids, float* vals, void* scratch, cudaStream_t s) {
    HP_REQUIRE(R >= 1 && n >= 1 && ld >= n && scratch, "argmax_rows: bad arguments R=%d n=%d ld=%d", R, n, ld);
    return launch_argmax(logits, R, n, ld, ids, vals, s);
}
size_t topk_scratch_bytes(int R, int n, int k) { return (size_t)R * ((n + AM_CHUNK - 1) / AM_CHUNK) * k * 8; }
int topk_max_k() { return TOPK_MAX; }
int topk_rows(const float* logits, int R, int n, int ld, int k, int* ids, float* vals, void* scratch, cudaStream_t s) {
    HP_REQUIRE(R >= 1 && n >= 1 && ld >= n && scratch && ids, "topk_rows: bad arguments R=%d n=%d ld=%d", R, n, ld);
    const int np = (n + AM_CHUNK - 1) / AM_CHUNK;
    HP_REQUIRE(k >= 1 && k <= TOPK_MAX && k <= n && np <= 64, "topk_rows: k=%d must be in 1..%d (and the row at most %d entries)", k, TOPK_MAX, 64 * AM_CHUNK);
    float* pv = (float*)scratch; int* pi = (int*)(pv + (size_t)R * np * k);
    HP_CUDA(launch_pdl<1>(k_topk_part, dim3(np, R), dim3(256), 0, s, logits, n, ld, k, pv, pi));
    HP_CUDA(launch_pdl<1>(k_topk_final, dim3(R), dim3(256), 0, s, (const float*)pv, (const int*)pi, np * k, k, ids, vals));
    HP_CUDA(cudaGetLastError());
    return HP_OK;
}
int argmax_static_max_rows() { return AM_STATIC_ROWS; }
int argmax_static_max_n() { return AM_STATIC_N; }

// Same kernel as argmax_rows, for callers without any scratch.
int argmax_rows_static(const float* logits, int R, int n, int ld, int* ids, float* vals, cudaStream_t s) {
    HP_REQUIRE(R >= 1 && n >= 1 && ld >= n, "argmax_rows_static: bad arguments R=%d n=%d ld=%d", R, n, ld);
    HP_REQUIRE(R <= AM_STATIC_ROWS && n <= AM_STATIC_N, "argmax_rows_static: R=%d n=%d exceed the limits (at most %d rows of %d entries)", R, n, AM_STATIC_ROWS, AM_STATIC_N);
    // a kernel can only be launched into a stream of the current device
    const int cur = current_device();
    int dev = cur;
    if (s != nullptr && s != cudaStreamLegacy && s != cudaStreamPerThread) HP_CUDA(cudaStreamGetDevice(s, &dev));
    HP_REQUIRE(cur >= 0 && dev == cur, "argmax_rows_static: the stream belongs to device %d but device %d is current", dev, cur);
    return launch_argmax(logits, R, n, ld, ids, vals, s);
}

int accept_greedy(const int* ids, const int* drafts, int n_draft, int* out, cudaStream_t s) {
    HP_REQUIRE(n_draft >= 0 && n_draft <= 31, "accept_greedy: n_draft=%d out of range", n_draft);
    HP_CUDA(launch_pdl<1>(k_accept, dim3(1), dim3(32), 0, s, ids, drafts, n_draft, out));
    return HP_OK;
}

}  // namespace hp
