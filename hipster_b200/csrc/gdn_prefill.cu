// Gated DeltaNet over a prompt chunk of one sequence: the arithmetic of k_gdn (ops.cu) operation by operation for any
// number of rows, every row committed.
//
// k_gdn takes at most 8 new rows per launch and is a chain of loads, cluster barriers and norms around its recurrence
// (15.7 us per launch). Only the recurrence is serial in the rows, so a chunk runs as three launches: convolution, SiLU, l2
// norms and gates of all rows in parallel; the recurrence alone, with the state in registers from the first row to the
// last; the output norm, gate and quantiser of all rows in parallel.
#include "hp_common.cuh"
#include "kernels.h"
#include <type_traits>

namespace hp {
namespace {

constexpr int D = 128, PF_CH = 16, PF_STR = 320;   // rows per staged piece of the scan; floats of a staged q | k row (16-float chunks padded to 20)

__device__ __forceinline__ float warp_sum_xor(float v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = v + __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// grid (heads: q heads, k heads, v heads; rows), 128 threads = channels. qk [row][q heads | k heads][128] normalised,
// v [row][v head][128], gate [row][v head] = (beta, decay). The taps before row 0 come from the conv history, which every v head keeps for itself: a
// q / k head reads that of the v head with its own number.
__global__ void __launch_bounds__(D) k_gdn_pf_conv(GdnPrefillParams a) {
    pdl_launch_dependents();
    __shared__ float sh[4];
    const int hd = blockIdx.x, r = blockIdx.y, c = threadIdx.x, lane = c & 31, warp = c >> 5;
    const int grp = hd < a.n_qk ? 0 : hd < 2 * a.n_qk ? 1 : 2, h = hd - grp * a.n_qk;   // q, k or v head h
    const int col = hd * D + c;
    const float4 w = *reinterpret_cast<const float4*>(a.conv_w + (size_t)col * 4);
    pdl_wait();
    const float* cst = a.conv_state + (size_t)h * 3 * 384 + grp * D + c;
    float x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) { const int rr = r + i - 3; x[i] = rr < 0 ? cst[(rr + 3) * 384] : a.rows[(size_t)rr * a.ld + col]; }
    float t = w.x * x[0]; t = fmaf(w.y, x[1], t); t = fmaf(w.z, x[2], t); t = fmaf(w.w, x[3], t);
    const float v = silu_det(t);
    if (grp == 2) {
        a.v[((size_t)r * a.n_v + h) * D + c] = v;
        if (c == 0) {
            const float* row = a.rows + (size_t)r * a.ld;
            const float beta = sigmoid_det(row[a.off_b + h]);
            const float decay = expf_det(bf2f(((const uint16_t*)a.a_neg)[h]) * softplus_det(row[a.off_a + h] + bf2f(((const uint16_t*)a.dt_bias)[h])));
            reinterpret_cast<float2*>(a.gate)[(size_t)r * a.n_v + h] = make_float2(beta, decay);
        }
        return;
    }
    const float p = warp_sum_xor(v * v);
    if (lane == 0) sh[warp] = p;
    __syncthreads();
    float tot = sh[0]; tot = tot + sh[1]; tot = tot + sh[2]; tot = tot + sh[3];
    a.qk[((size_t)r * 2 * a.n_qk + hd) * D + c] = v / fmaxf(sqrtf(tot), a.eps);
}

// grid (8, v heads), 64 threads: 16 rows of the head's state, thread = 16 columns of two rows (k_gdn's layout), in registers
// for the whole chunk. Bound by the dependent chain of a row (16 fmaf, 3 shuffles) with 1.3 warps per scheduler to hide it: a row's output
// product is issued beside the next row's first product. 301 rows, 48 heads, ncu: 116 us, 183 instructions of a warp per row, issue 39 %
// (products one after the other 120 us; one state row per thread 121, four 145). q and k are read 64 bits at a time (see lds_f2) and serve
// two state rows; q, k, v and gates arrive by asynchronous copies, 16 rows ahead.
constexpr int PF_ST = 64;   // threads of the scan
__global__ void __launch_bounds__(PF_ST) k_gdn_pf_scan(GdnPrefillParams a) {
    __shared__ __align__(16) float sqk[2][PF_CH][PF_STR];
    __shared__ float sv[2][PF_CH][16];
    __shared__ float2 sg[2][PF_CH];
    pdl_launch_dependents();
    const int part = blockIdx.x, h = blockIdx.y, hk = h % a.n_qk, tid = threadIdx.x, jl = tid >> 3, ck = tid & 7, j = 16 * part + jl;
    pdl_wait();
    float* Mrow = a.state + ((size_t)h * D + j) * D + 16 * ck;
    float2 m[2][8];   // rows j and j + 8
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int i = 0; i < 8; i += 2) { const float4 v = *reinterpret_cast<const float4*>(Mrow + q * 8 * D + 2 * i); m[q][i] = make_float2(v.x, v.y); m[q][i + 1] = make_float2(v.z, v.w); }
    auto stage = [&](int r0, int s) {
        const int n = min(PF_CH, a.T - r0);
        for (int e = tid; e < n * 64; e += PF_ST) {   // 16-byte pieces of q (32) and k (32) of every row
            const int r = e >> 6, i = e & 63, g = i >> 5, p = i & 31;
            const float* src = a.qk + ((size_t)(r0 + r) * 2 * a.n_qk + g * a.n_qk + hk) * D + p * 4;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(&sqk[s][r][g * 160 + (p >> 2) * 20 + (p & 3) * 4])), "l"(src) : "memory");
        }
        for (int e = tid; e < n * 16; e += PF_ST) cp_async4(&sv[s][e >> 4][e & 15], a.v + ((size_t)(r0 + (e >> 4)) * a.n_v + h) * D + 16 * part + (e & 15));
        for (int e = tid; e < n * 2; e += PF_ST) cp_async4(reinterpret_cast<float*>(&sg[s][e >> 1]) + (e & 1), a.gate + ((size_t)(r0 + (e >> 1)) * a.n_v + h) * 2 + (e & 1));
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    stage(0, 0);
    for (int r0 = 0, s = 0; r0 < a.T; r0 += PF_CH, s ^= 1) {
        if (r0 + PF_CH < a.T) { stage(r0 + PF_CH, s ^ 1); asm volatile("cp.async.wait_group 1;" ::: "memory"); }
        else cp_async_wait_all();
        __syncthreads();
        const int n = min(PF_CH, a.T - r0);
        // as in k_gdn: the second product of a row runs beside the decay and the first product of the next one, its reduction beside that
        // one's, and the reads of the next row's k are in flight under both
        float2 kr[8];
        float d0 = 0.f, d1 = 0.f, o0 = 0.f, o1 = 0.f;
        auto ld8 = [&](float2 (&r)[8], const float* p) {
#pragma unroll
            for (int i = 0; i < 8; ++i) r[i] = lds_f2(p + 2 * i);
        };
        auto first = [&](float2 dc2, const float2& k, int i) {   // decay and first product of one column pair
            m[0][i] = mul2(m[0][i], dc2); m[1][i] = mul2(m[1][i], dc2);
            d0 = fmaf(m[0][i].x, k.x, d0); d1 = fmaf(m[1][i].x, k.x, d1);
            d0 = fmaf(m[0][i].y, k.y, d0); d1 = fmaf(m[1][i].y, k.y, d1);
        };
        auto put = [&](int it) {
#pragma unroll
            for (int off = 1; off < 8; off <<= 1) { o0 = o0 + __shfl_xor_sync(0xffffffffu, o0, off); o1 = o1 + __shfl_xor_sync(0xffffffffu, o1, off); }
            if (ck == 0) { float* o = a.o + ((size_t)(r0 + it) * a.n_v + h) * D + j; o[0] = o0 * 0.08838834764831845f; o[8] = o1 * 0.08838834764831845f; }
        };
        ld8(kr, &sqk[s][0][160 + 20 * ck]);
#pragma unroll
        for (int i = 0; i < 8; ++i) first(make_float2(sg[s][0].y, sg[s][0].y), kr[i], i);
        auto row = [&](int it, auto last_) {
            constexpr bool last = decltype(last_)::value;   // of the piece: the state stays as it is behind it
            float2 qr[8], kn[8];
            ld8(qr, &sqk[s][it][20 * ck]);
            if constexpr (!last) ld8(kn, &sqk[s][it + 1][160 + 20 * ck]);
            const float beta = sg[s][it].x, decay = last ? 1.f : sg[s][it + 1].y, v0 = sv[s][it][jl], v1 = sv[s][it][jl + 8];
#pragma unroll
            for (int off = 1; off < 8; off <<= 1) { d0 = d0 + __shfl_xor_sync(0xffffffffu, d0, off); d1 = d1 + __shfl_xor_sync(0xffffffffu, d1, off); }
            if (it > 0) put(it - 1);
            const float e0 = (v0 - d0) * beta, e1 = (v1 - d1) * beta;
            const float2 dl0 = make_float2(e0, e0), dl1 = make_float2(e1, e1), dc2 = make_float2(decay, decay);
#pragma unroll
            for (int i = 0; i < 8; ++i) { fma2(m[0][i], dl0, kr[i]); fma2(m[1][i], dl1, kr[i]); }
            o0 = o1 = d0 = d1 = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                o0 = fmaf(m[0][i].x, qr[i].x, o0); o1 = fmaf(m[1][i].x, qr[i].x, o1);
                o0 = fmaf(m[0][i].y, qr[i].y, o0); o1 = fmaf(m[1][i].y, qr[i].y, o1);
                if constexpr (!last) { first(dc2, kn[i], i); kr[i] = kn[i]; }
            }
        };
        for (int it = 0; it + 1 < n; ++it) row(it, std::false_type());
        row(n - 1, std::true_type());
        put(n - 1);
        __syncthreads();   // the stage is free again
    }
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int i = 0; i < 8; i += 2) *reinterpret_cast<float4*>(Mrow + q * 8 * D + 2 * i) = make_float4(m[q][i].x, m[q][i].y, m[q][i + 1].x, m[q][i + 1].y);
    if (part == 0)   // conv history after the chunk: ascending taps, so that a chunk of fewer than 3 rows shifts the old ones in place
        for (int c = tid; c < 384; c += PF_ST) {
            const int g = c >> 7, col = g == 0 ? hk * D + c : g == 1 ? a.n_qk * D + hk * D + (c - D) : 2 * a.n_qk * D + h * D + (c - 2 * D);
            float* cst = a.conv_state + (size_t)h * 3 * 384 + c;
            for (int tap = 0; tap < 3; ++tap) { const int rr = a.T - 3 + tap; cst[tap * 384] = rr < 0 ? cst[(rr + 3) * 384] : a.rows[(size_t)rr * a.ld + col]; }
        }
}

// grid (v heads, rows), 128 threads: per-head RMSNorm * w * gate(z), quantised
__global__ void __launch_bounds__(D) k_gdn_pf_out(GdnPrefillParams a) {
    pdl_launch_dependents();
    __shared__ float sh[4];
    const int h = blockIdx.x, r = blockIdx.y, c = threadIdx.x, lane = c & 31, warp = c >> 5;
    const float nw = bf2f(((const uint16_t*)a.norm_w)[c]);
    pdl_wait();
    const float o = a.o[((size_t)r * a.n_v + h) * D + c], z = a.rows[(size_t)r * a.ld + a.off_z + h * D + c];
    const float p = warp_sum_xor(o * o);
    if (lane == 0) sh[warp] = p;
    const float gate = a.sigmoid_gate ? sigmoid_det(z) : silu_det(z);
    __syncthreads();
    float ss = sh[0]; ss = ss + sh[1]; ss = ss + sh[2]; ss = ss + sh[3];
    const float v = ((o * (1.0f / sqrtf(ss / (float)D + a.eps))) * nw) * gate;
    warp_quant32_store(v, r, (h * D + c) >> 5, a.n_v * D, (int8_t*)a.xq.q, (float*)a.xq.sc, lane);
}

}  // namespace

size_t gdn_prefill_floats(int rows, int n_qk, int n_v) { return (size_t)rows * ((size_t)(2 * n_qk + 2 * n_v) * D + 2 * n_v); }

int gdn_prefill(GdnPrefillParams p, float* scratch, cudaStream_t s) {
    HP_REQUIRE(p.T >= 1 && p.n_qk >= 1 && p.n_v >= p.n_qk && scratch && ((uintptr_t)scratch & 15) == 0, "gdn_prefill: bad arguments");
    p.qk = scratch; p.v = p.qk + (size_t)p.T * 2 * p.n_qk * D; p.o = p.v + (size_t)p.T * p.n_v * D; p.gate = p.o + (size_t)p.T * p.n_v * D;
    HP_CUDA(launch_pdl<128>(k_gdn_pf_conv, dim3(2 * p.n_qk + p.n_v, p.T), dim3(D), 0, s, p));
    HP_CUDA(launch_pdl<128>(k_gdn_pf_scan, dim3(8, p.n_v), dim3(PF_ST), 0, s, p));
    HP_CUDA(launch_pdl<128>(k_gdn_pf_out, dim3(p.n_v, p.T), dim3(D), 0, s, p));
    HP_CUDA(cudaGetLastError()); return HP_OK;
}

}  // namespace hp
