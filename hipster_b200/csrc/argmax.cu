// Per-row argmax over the vocabulary and greedy prefix acceptance, on device.
// Reference: k_topk with k = 1 (engine/kernels/ops.hip:702-716: maximum value, ties -> lowest index) and the
// host acceptance loop of the MTP driver (engine/bench/spec27b.cpp:92-97). The reference copies the ids to the
// host and compares there; here the comparison runs on the device so that no logits or ids round-trip is needed.
#include "hp_common.cuh"
#include "kernels.h"

namespace hp {
namespace {

constexpr int AM_CHUNK = 8192;   // elements per stage-1 block of the top-k and of the two-launch arg-max

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
// One cluster of CL CTAs of NT threads per row, each with a contiguous piece of the 16-byte groups of the row; the CTAs' winners meet in
// the first one's shared memory. Bound by latency: a thread's 16 loads are in flight before its first comparison (launch bounds of
// one CTA per SM: left alone the compiler takes 32 registers, half the loads and 3.6 us for one row of 248320), the entries in front
// of the first 16-byte boundary and behind the last one are read one by one. -inf (an absent entry, or a real one) and NaN never win; a
// row of nothing else yields -1.
template <int CL, int NT>
__global__ void __launch_bounds__(NT, 1) k_argmax(const float* __restrict__ x, int n, int ld, int* __restrict__ ids, float* __restrict__ vals) {
    __shared__ float sv[NT / 32]; __shared__ int si[NT / 32];
    __shared__ float cv[CL]; __shared__ int ci[CL];
    pdl_launch_dependents();
    if constexpr (CL > 1) cluster_arrive_relaxed();   // matched by cluster_wait(): every CTA has started before the first store into another one
    const int r = blockIdx.x / CL, rank = blockIdx.x % CL, tid = threadIdx.x;
    const float* xr = x + (size_t)r * ld;
    const int head = min(n, (int)((16 - (reinterpret_cast<uintptr_t>(xr) & 15)) & 15) / 4), nq = (n - head) / 4;   // whole 16-byte groups
    const int per = (nq + CL - 1) / CL, q0 = min(nq, rank * per), q1 = min(nq, q0 + per);
    const float4* xa = reinterpret_cast<const float4*>(xr + head);
    pdl_wait();
    float bv = -INFINITY; int bi = -1;
    if (rank == 0 && tid < head) am_better(bv, bi, xr[tid], tid);
    constexpr int NV = 16;
    for (int b = q0 + tid; b < q1; b += NT * NV) {
        float4 v[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) v[k] = b + NT * k < q1 ? xa[b + NT * k] : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const int i = head + 4 * (b + NT * k);
            if (v[k].x > bv) { bv = v[k].x; bi = i; }
            if (v[k].y > bv) { bv = v[k].y; bi = i + 1; }
            if (v[k].z > bv) { bv = v[k].z; bi = i + 2; }
            if (v[k].w > bv) { bv = v[k].w; bi = i + 3; }
        }
    }
    if (rank == CL - 1) { const int i = head + 4 * nq + tid; if (i < n) am_better(bv, bi, xr[i], i); }
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
// The form of a few very long rows: one CTA per 8192 entries, whose winners meet in a second launch. All loads of a thread are in flight
// before the first comparison.
__global__ void __launch_bounds__(256) k_argmax_part(const float* __restrict__ x, int n, int ld, float* __restrict__ pv, int* __restrict__ pi) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float sv[8]; __shared__ int si[8];
    const int r = blockIdx.y, c0 = blockIdx.x * AM_CHUNK, c1 = min(n, c0 + AM_CHUNK);
    const float* xr = x + (size_t)r * ld;
    float bv = -INFINITY; int bi = -1;
    constexpr int NV = AM_CHUNK / 256;
    float v[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) { const int i = c0 + threadIdx.x + 256 * k; v[k] = i < c1 ? xr[i] : -INFINITY; }
#pragma unroll
    for (int k = 0; k < NV; ++k) if (v[k] > bv) { bv = v[k]; bi = c0 + threadIdx.x + 256 * k; }
    am_block_reduce(bv, bi, sv, si);
    if (threadIdx.x == 0) { pv[(size_t)r * gridDim.x + blockIdx.x] = bv; pi[(size_t)r * gridDim.x + blockIdx.x] = bi; }
}
__global__ void __launch_bounds__(256) k_argmax_final(const float* __restrict__ pv, const int* __restrict__ pi, int np, int* __restrict__ ids, float* __restrict__ vals) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float sv[8]; __shared__ int si[8];
    const int r = blockIdx.x;
    float bv = -INFINITY; int bi = -1;
    for (int i = threadIdx.x; i < np; i += 256) am_better(bv, bi, pv[(size_t)r * np + i], pi[(size_t)r * np + i]);
    am_block_reduce(bv, bi, sv, si);
    if (threadIdx.x == 0) { ids[r] = bi; if (vals) vals[r] = bv; }
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

template <int CL, int NT>
int launch_argmax_cl(const float* logits, int R, int n, int ld, int* ids, float* vals, cudaStream_t s) {
    if constexpr (CL > 8) {   // beyond the portable cluster size
        static bool attr[MAX_DEVICES] = {};   // per device: the opt-in belongs to the device's copy of the kernel
        const int dev = current_device(); if (dev < 0) return HP_ECUDA;
        if (!attr[dev]) { HP_CUDA(cudaFuncSetAttribute(k_argmax<CL, NT>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)); attr[dev] = true; }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(R * CL); cfg.blockDim = dim3(NT); cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension; at[0].val.clusterDim.x = CL; at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = (pdl_off_mask(s) & 1) ? 1 : 2;
    HP_CUDA(cudaLaunchKernelEx(&cfg, k_argmax<CL, NT>, logits, n, ld, ids, vals));
    return HP_OK;
}
// One launch, without scratch. us in a captured graph for rows of 1, 6 and 24 (two launches of 8192-entry pieces in brackets): one CTA
// up to 32768 entries, 2.6 2.7 2.8 there (3.5 3.7 4.2); 8 small CTAs, 65536: 2.6 2.8 3.3 (3.5 3.6 4.4); 8 CTAs, 248320: 3.3 3.4 4.8
// (3.9 3.9 5.8); 16 CTAs for up to 12 longer rows, 524288: 3.6 3.7 (4.0 4.9), where 8 take 4.3 4.4, and 24 rows 6.8 (16: 8.0).
int launch_argmax(const float* logits, int R, int n, int ld, int* ids, float* vals, cudaStream_t s) {
    if (n <= 32768) { HP_CUDA(launch_pdl<1>(k_argmax<1, 512>, dim3(R), dim3(512), 0, s, logits, n, ld, ids, vals)); return HP_OK; }
    if (n <= 65536) return launch_argmax_cl<8, 256>(logits, R, n, ld, ids, vals, s);
    if (n <= 262144 || R > 12) return launch_argmax_cl<8, 512>(logits, R, n, ld, ids, vals, s);
    return launch_argmax_cl<16, 512>(logits, R, n, ld, ids, vals, s);
}

}  // namespace

// winners of the pieces of a row; rows of up to 65536 entries take one launch whatever their number
size_t argmax_scratch_bytes(int R, int n) { return n <= 65536 ? 0 : (size_t)R * ((n + AM_CHUNK - 1) / AM_CHUNK) * 8; }

int argmax_rows(const float* logits, int R, int n, int ld, int* ids, float* vals, void* scratch, cudaStream_t s) {
    HP_REQUIRE(R >= 1 && n >= 1 && ld >= n && (scratch || argmax_scratch_bytes(R, n) == 0), "argmax_rows: bad arguments R=%d n=%d ld=%d", R, n, ld);
    // few rows longer than a cluster reads at once take two launches (one row of 1 M entries 4.0 us, 4.5 in one launch; 4 M 5.7 and 10.0;
    // 24 rows of 1 M 16.2 and 11.3)
    if (n <= 524288 || R > 5) return launch_argmax(logits, R, n, ld, ids, vals, s);
    const int np = (n + AM_CHUNK - 1) / AM_CHUNK;
    float* pv = (float*)scratch; int* pi = (int*)(pv + (size_t)R * np);
    HP_CUDA(launch_pdl<1>(k_argmax_part, dim3(np, R), dim3(256), 0, s, logits, n, ld, pv, pi));
    HP_CUDA(launch_pdl<1>(k_argmax_final, dim3(R), dim3(256), 0, s, (const float*)pv, (const int*)pi, np, ids, vals));
    return HP_OK;
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

// For callers without any scratch: always one launch.
int argmax_rows_static(const float* logits, int R, int n, int ld, int* ids, float* vals, cudaStream_t s) {
    HP_REQUIRE(R >= 1 && n >= 1 && ld >= n, "argmax_rows_static: bad arguments R=%d n=%d ld=%d", R, n, ld);
    HP_REQUIRE(R <= AM_STATIC_ROWS && n <= AM_STATIC_N, "argmax_rows_static: R=%d n=%d exceed the limits (at most %d rows of %d entries)", R, n, AM_STATIC_ROWS, AM_STATIC_N);
    // a kernel can only be launched into a stream of the current device. A capturing stream may not be asked for its device (the question
    // would end the capture): there the launch itself refuses
    const int cur = current_device();
    int dev = cur;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (s != nullptr && s != cudaStreamLegacy && s != cudaStreamPerThread) {
        HP_CUDA(cudaStreamIsCapturing(s, &cap));
        if (cap == cudaStreamCaptureStatusNone) HP_CUDA(cudaStreamGetDevice(s, &dev));
    }
    HP_REQUIRE(cur >= 0 && dev == cur, "argmax_rows_static: the stream belongs to device %d but device %d is current", dev, cur);
    return launch_argmax(logits, R, n, ld, ids, vals, s);
}

int accept_greedy(const int* ids, const int* drafts, int n_draft, int* out, cudaStream_t s) {
    HP_REQUIRE(n_draft >= 0 && n_draft <= 31, "accept_greedy: n_draft=%d out of range", n_draft);
    HP_CUDA(launch_pdl<1>(k_accept, dim3(1), dim3(32), 0, s, ids, drafts, n_draft, out));
    return HP_OK;
}

}  // namespace hp
