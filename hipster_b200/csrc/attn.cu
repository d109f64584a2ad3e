// GQA decode attention over the f16 KV cache for the rows of a verify pass.
//
// Reference: k_qk_norm_rope_kv (engine/kernels/ops.hip:363-411), the scalar decode attention k_attn (:413-465, the
// semantic reference) and the production split-KV structure k_attn_mq + k_attn_mq_merge (:831-948): fixed absolute
// key splits merged in split order, so that a row's result does not depend on the number of rows in the pass.
//
// Here: head_dim 256, NeoX RoPE on the first n_rot = 64 dims from a host-built cos/sin table (double precision,
// rounded to fp32), K and V stored row-major f16 [slot][kv head][position][256]. One CTA per (split of 128 keys,
// kv head, row group <= 8 rows): the K and V tiles are read once for all rows x q-heads of the group. All arithmetic
// is fp32 FMA in a fixed order (scores: fmaf chain over d = 0..255; P.V: fmaf chain over keys in position order;
// merge: splits in order), so the CPU oracle reproduces it bit for bit. KV traffic is ~2 % of a pass's bytes, so SIMT
// fp32 is affordable, and it avoids the tensor-core rounding hazard the reference documents (docs/decode-27b.md:117-126).
#include "hp_common.cuh"
#include "kernels.h"
#include <algorithm>

namespace hp {
namespace {

constexpr int HD = 256, SPL = ATTN_SPLIT, MAXP = ATTN_MAX_PAIRS;   // pairs = rows of the group x q-heads per kv head
constexpr int KSTR = HD + 8;                                        // f16 elements per K tile row (528 B): 8 lanes = 8 keys read 16 B each from distinct banks

template <int NW>
__device__ __forceinline__ float block_sum_det(float v, float* sh) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = v + __shfl_xor_sync(0xffffffffu, v, off);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sh[w] = v;
    __syncthreads();
    float tot = sh[0];
#pragma unroll
    for (int i = 1; i < NW; ++i) tot = tot + sh[i];
    return tot;
}

// grid: rows * (n_head + n_kv) blocks of 256 threads; row layout: [q_full: n_head x (256 q | 256 gate) | k: n_kv x 256 | v: n_kv x 256]
// planes != nullptr: the projection arrives as P K-part planes ([rows][ld] each, part_stride apart); they are added in
// part order here (q, gate, k and v slices of this block) and q / gate are written to qkv for the attention kernels.
__global__ void __launch_bounds__(256) k_qk_norm_rope_kv(float* __restrict__ qkv, const float* __restrict__ planes, int P, size_t part_stride,
                                                          int ld, int n_head, int n_kv, const uint16_t* __restrict__ qw, const uint16_t* __restrict__ kw,
                                                          const float2* __restrict__ rope, int n_rot, const int* __restrict__ row_pos, const int* __restrict__ row_slot, int imm_pos0,
                                                          uint16_t* __restrict__ kc, uint16_t* __restrict__ vc, size_t kv_stride, int max_ctx, float eps) {
    pdl_wait();
    pdl_launch_dependents();   // behind the wait: all that was enqueued in front of this kernel is complete when k_attn_split starts
    __shared__ float sh[8]; __shared__ float buf[HD];
    const int t = threadIdx.x, hb = blockIdx.x % (n_head + n_kv), r = blockIdx.x / (n_head + n_kv);
    const int pos = row_pos ? row_pos[r] : imm_pos0 + r, slot = row_slot ? row_slot[r] : 0;
    const bool isq = hb < n_head;
    const size_t xoff = (isq ? (size_t)r * ld + hb * 512 : (size_t)r * ld + n_head * 512 + (hb - n_head) * HD) + t;
    // second slice of this block: the gate of a q head, the v of a kv head
    const size_t yoff = isq ? xoff + HD : (size_t)r * ld + n_head * 512 + n_kv * HD + (hb - n_head) * HD + t;
    float* x = qkv + (xoff - t);
    float xv, yv;
    if (planes) {
        float xa[4], ya[4];   // P <= 4: every plane's load in flight at once
#pragma unroll
        for (int p = 0; p < 4; ++p) if (p < P) { xa[p] = planes[(size_t)p * part_stride + xoff]; ya[p] = planes[(size_t)p * part_stride + yoff]; }
        xv = xa[0]; yv = ya[0];
#pragma unroll
        for (int p = 1; p < 4; ++p) if (p < P) { xv = xv + xa[p]; yv = yv + ya[p]; }
        if (isq) qkv[yoff] = yv;
    } else { xv = x[t]; yv = qkv[yoff]; }
    const int half = n_rot / 2, i = t < half ? t : t - half;
    const float nw = bf2f((isq ? qw : kw)[t]);
    const float2 cs = t < n_rot ? rope[(size_t)pos * half + i] : make_float2(0.f, 0.f);   // (cos, sin) of pos * base^(-2i/n_rot)
    const float ss = block_sum_det<8>(xv * xv, sh);
    float n = (xv * (1.0f / sqrtf(ss / (float)HD + eps))) * nw;
    buf[t] = n;
    __syncthreads();
    if (t < n_rot) {
        const float x0 = buf[i], x1 = buf[i + half];
        n = t < half ? fmaf(-x1, cs.y, x0 * cs.x) : fmaf(x1, cs.x, x0 * cs.y);
    }
    x[t] = n;
    if (!isq) {
        const int kh = hb - n_head;
        const float vv = yv;
        const size_t o = (size_t)slot * kv_stride + ((size_t)kh * max_ctx + pos) * HD + t;
        kc[o] = f2h(n); vc[o] = f2h(vv);
    }
}

__device__ __forceinline__ float2 attn_fma2(float2 a, float2 b, float2 c) {   // a * b + c per lane
    float2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(reinterpret_cast<unsigned long long&>(r))
        : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)), "l"(reinterpret_cast<unsigned long long&>(c)));
    return r;
}
struct AttnArgs {
    const float* qkv; int ld, n_head, n_kv;
    const uint16_t* kc; const uint16_t* vc; size_t kv_stride; int max_ctx;
    const int* groups;        // device: per group {r0, T, slot, pos0}; nullptr: rows 0 .. imm_rows - 1 of slot 0 at imm_pos0 .., imm_gr rows per group
    int imm_pos0, imm_rows, imm_gr, rows;   // rows: of the launch
    float* pO; float* pm; float* pl; int nsplit_max;   // partials [group][kv head][split][MAXP] (x 256 for pO)
};
__device__ __forceinline__ int4 attn_group(const int* groups, int gi, int pos0, int rows, int gr) {   // {r0, T, slot, pos0}
    if (groups) return make_int4(groups[gi * 4], groups[gi * 4 + 1], groups[gi * 4 + 2], groups[gi * 4 + 3]);
    return make_int4(gi * gr, min(gr, rows - gi * gr), 0, pos0 + gi * gr);
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory"); }
// Tile geometry. Score phase: a lane takes KPL = 2 keys against PPT (row, head) pairs, a warp 64 keys, so two warps share a
// group of PPT pairs. P.V phase: thread = (two dims, part of the pairs). NP = pairs a CTA holds.
template <int PPT, int NT> struct AttnGeom {
    static constexpr int NW = NT / 32, KPL = 2, KG = SPL / (32 * KPL), NP = NW / KG * PPT, PARTS = NT / (HD / 2), PP = NP / PARTS;
    static constexpr int ESTR = ((NP / 4) | 1) * 4;   // floats per key row of the score tile: an odd multiple of 4, lanes = keys hit 8 bank groups
    static constexpr int SMEM = NP * HD * 4 + SPL * ESTR * 4 + SPL * KSTR * 2 + SPL * HD * 2;
    static_assert(PPT % 2 == 0 && NT % (HD / 2) == 0 && PP % 4 == 0 && NP <= MAXP, "attention tile geometry");
};
// grid (nsplit_max, n_kv, ngroups), NT threads, dynamic smem. Bound by the fp32 FMA pipe of one SM per split and kv head (36 pairs:
// 2 x 36 x 128 x 256 fmaf = 9.6 us at 128 a clock); every score and every output element is one fmaf chain (over d, over
// the keys), two chains per packed instruction. Hence tiles that fit the pairs (12 per 128 threads: idle pairs cost as much as live ones),
// 6 pairs x 2 keys per thread in the score phase (16 f16 -> f32 conversions and 8 broadcasts, which share the pipe and the issue slots
// with the math, per 96 fmaf; 3 pairs x 4 keys needed 16 per 48), and the V tile in flight under the scores. 36 pairs, thousand clocks
// of a CTA: staging 4.5 (6.0 with the scalar stores of q), scores 16.4, softmax 3.5 (4.3 a pair at a time), P.V 14.9 (16.7 with four dims x
// half the pairs per thread: more duplicated operands).
template <int PPT, int NT>
__global__ void __launch_bounds__(NT, 1) k_attn_split(AttnArgs a) {
    using Geo = AttnGeom<PPT, NT>;
    constexpr int NW = Geo::NW, KPL = Geo::KPL, KG = Geo::KG, PP = Geo::PP, ESTR = Geo::ESTR;
    extern __shared__ __align__(16) uint8_t sm_raw[];
    float* sQ = reinterpret_cast<float*>(sm_raw);                                   // [NP / 2][256][2]: two pairs side by side
    float* sE = sQ + Geo::NP * HD;                                                  // [SPL][ESTR] scores, then weights
    uint16_t* sK = reinterpret_cast<uint16_t*>(sE + SPL * ESTR);                    // [SPL][KSTR]
    uint16_t* sV = sK + SPL * KSTR;                                                 // [SPL][256]
    const int split = blockIdx.x, kh = blockIdx.y, gi = blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int4 gd = attn_group(a.groups, gi, a.imm_pos0, a.imm_rows, a.imm_gr);
    const int r0 = gd.x, T = gd.y, slot = gd.z, pos0 = gd.w;
    const int G = a.n_head / a.n_kv, npairs = T * G;
    const int k_lo = split * SPL;
    const int nkeys = min(SPL, pos0 + T - k_lo);          // keys of this split visible to the last row of the group
    if (nkeys <= 0 || T <= 0) return;
    // Keys in front of every row of this launch were written by earlier passes: they are fetched in front of the dependency wait, under the
    // kernel that writes the new ones (it releases this one once its own predecessors are complete).
    const int nold = max(0, min(nkeys, pos0 - a.rows - k_lo));
    const size_t pbase = (((size_t)gi * a.n_kv + kh) * a.nsplit_max + split) * MAXP;
    const uint16_t* Kg = a.kc + (size_t)slot * a.kv_stride + ((size_t)kh * a.max_ctx + k_lo) * HD;
    const uint16_t* Vg = a.vc + (size_t)slot * a.kv_stride + ((size_t)kh * a.max_ctx + k_lo) * HD;
    auto fetch_k = [&](int k0, int k1) { for (int i = k0 * (HD / 8) + tid; i < k1 * (HD / 8); i += NT) { const int k = i / (HD / 8), c = i % (HD / 8); cp_async16(sK + k * KSTR + c * 8, Kg + (size_t)k * HD + c * 8); } };
    auto fetch_v = [&](int k0, int k1) { for (int i = k0 * (HD / 8) + tid; i < k1 * (HD / 8); i += NT) cp_async16(sV + i * 8, Vg + (size_t)i * 8); };
    fetch_k(0, nold); fetch_v(0, nold);
    pdl_wait();
    pdl_launch_dependents();   // behind the wait, for the splits of a further launch over the same rows (see nold)
    fetch_k(nold, nkeys);
    asm volatile("cp.async.commit_group;" ::: "memory");
    fetch_v(nold, nkeys);
    asm volatile("cp.async.commit_group;" ::: "memory");
    // pair = t*G + hh -> row r0+t, head kh*G + hh
    // two neighbouring pairs at once: 128-bit stores of interleaved dims (scalar ones of a single pair hit every bank eight times)
#pragma unroll 3
    for (int i = tid; i < (npairs + 1) / 2 * (HD / 4); i += NT) {
        const int p = i / (HD / 4) * 2, d4 = i % (HD / 4), t0 = p / G, p1 = min(p + 1, npairs - 1), t1 = p1 / G;
        const float4 q0 = reinterpret_cast<const float4*>(a.qkv + (size_t)(r0 + t0) * a.ld + (kh * G + p - t0 * G) * 512)[d4], q1 = reinterpret_cast<const float4*>(a.qkv + (size_t)(r0 + t1) * a.ld + (kh * G + p1 - t1 * G) * 512)[d4];
        float4* dst = reinterpret_cast<float4*>(sQ + (size_t)p * HD + 8 * d4);
        dst[0] = make_float4(q0.x, q1.x, q0.y, q1.y); dst[1] = make_float4(q0.z, q1.z, q0.w, q1.w);
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    {   // scores: warp = (64 keys, group of PPT pairs); fmaf chain over d
        const int k0 = (warp % KG) * 32 * KPL + lane, p0 = warp / KG * PPT;
        if (p0 < npairs && k0 - lane < nkeys) {
            float2 s[KPL][PPT / 2];
#pragma unroll
            for (int i = 0; i < KPL; ++i)
#pragma unroll
                for (int j = 0; j < PPT / 2; ++j) s[i][j] = make_float2(0.f, 0.f);
            const float* qb = sQ + (size_t)p0 * HD;
#pragma unroll 2
            for (int d = 0; d < HD; d += 8) {
                float2 kf[KPL][4];
#pragma unroll
                for (int i = 0; i < KPL; ++i) {
                    const uint4 kk = *reinterpret_cast<const uint4*>(sK + (k0 + 32 * i) * KSTR + d);
                    kf[i][0] = __half22float2(*reinterpret_cast<const __half2*>(&kk.x)); kf[i][1] = __half22float2(*reinterpret_cast<const __half2*>(&kk.y));
                    kf[i][2] = __half22float2(*reinterpret_cast<const __half2*>(&kk.z)); kf[i][3] = __half22float2(*reinterpret_cast<const __half2*>(&kk.w));
                }
#pragma unroll
                for (int e = 0; e < 4; ++e)   // dims d + 2 e, d + 2 e + 1
#pragma unroll
                    for (int j = 0; j < PPT / 2; ++j) {
                        const float4 q = *reinterpret_cast<const float4*>(qb + (size_t)j * 2 * HD + 2 * (d + 2 * e));
#pragma unroll
                        for (int i = 0; i < KPL; ++i) {
                            s[i][j] = attn_fma2(make_float2(q.x, q.y), make_float2(kf[i][e].x, kf[i][e].x), s[i][j]);
                            s[i][j] = attn_fma2(make_float2(q.z, q.w), make_float2(kf[i][e].y, kf[i][e].y), s[i][j]);
                        }
                    }
            }
#pragma unroll
            for (int i = 0; i < KPL; ++i)
#pragma unroll
                for (int j = 0; j < PPT / 2; ++j) *reinterpret_cast<float2*>(sE + (k0 + 32 * i) * ESTR + p0 + 2 * j) = make_float2(s[i][j].x * 0.0625f, s[i][j].y * 0.0625f);
        }
    }
    __syncthreads();
    // softmax pieces: a warp takes QP neighbouring pairs, lane l keys l, l+32, l+64, l+96. Row t of the group sees keys <= pos0 + t.
    // Maximum: exact in any order. Sum: the lane's keys in ascending order, then the xor tree (16..1). Four pairs at once (one where there
    // are as many warps as pairs): a 128-bit access per key, and their chains of reductions run side by side.
    constexpr int QP = PPT == 2 ? 1 : 4;
    static_assert(Geo::NP / QP <= NW, "one group of pairs per warp");
    if (warp * QP < npairs) {
        const int pq = warp * QP;
        float sc[QP][4], mx[QP], l[QP]; int nk[QP];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = lane + 32 * i;
            if constexpr (QP == 4) { const float4 v = *reinterpret_cast<const float4*>(sE + k * ESTR + pq); sc[0][i] = v.x; sc[1][i] = v.y; sc[2][i] = v.z; sc[3][i] = v.w; }
            else sc[0][i] = sE[k * ESTR + pq];
        }
#pragma unroll
        for (int c = 0; c < QP; ++c) {
            nk[c] = min(nkeys, pos0 + (pq + c) / G + 1 - k_lo); mx[c] = -INFINITY;
#pragma unroll
            for (int i = 0; i < 4; ++i) { if (lane + 32 * i >= nk[c]) sc[c][i] = -INFINITY; mx[c] = fmaxf(mx[c], sc[c][i]); }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
#pragma unroll
            for (int c = 0; c < QP; ++c) mx[c] = fmaxf(mx[c], __shfl_xor_sync(0xffffffffu, mx[c], off));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = lane + 32 * i;
#pragma unroll
            for (int c = 0; c < QP; ++c) {
                const float e = k < nk[c] ? expf_det(sc[c][i] - mx[c]) : 0.f;
                sc[c][i] = e;
                l[c] = i == 0 ? e : l[c] + e;
            }
            if (k < nkeys) {
                if constexpr (QP == 4) *reinterpret_cast<float4*>(sE + k * ESTR + pq) = make_float4(sc[0][i], sc[1][i], sc[2][i], sc[3][i]);
                else sE[k * ESTR + pq] = sc[0][i];
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
#pragma unroll
            for (int c = 0; c < QP; ++c) l[c] = l[c] + __shfl_xor_sync(0xffffffffu, l[c], off);
        if (lane == 0) {   // nk <= 0: mx = -inf, l = 0 (the merge skips it)
#pragma unroll
            for (int c = 0; c < QP; ++c) if (pq + c < npairs) { a.pm[pbase + pq + c] = mx[c]; a.pl[pbase + pq + c] = l[c]; }
        }
    }
    cp_async_wait_all();
    __syncthreads();
    // o[pair][d] = sum_k e[k][pair] * v[k][d], keys in position order; thread = (dims 2 dq and 2 dq + 1, part of the pairs):
    // a warp's read of four weights serves 64 dims
    {
        const int dq = tid % (HD / 2), p_lo = (tid / (HD / 2)) * PP;
        if (p_lo < npairs) {
            float2 o[PP / 2][2];   // [pairs 2 p, 2 p + 1][dim]: two fp32 fmaf per instruction, each rounded once
#pragma unroll
            for (int p = 0; p < PP / 2; ++p) { o[p][0] = make_float2(0.f, 0.f); o[p][1] = make_float2(0.f, 0.f); }
            auto step = [&](int k) {
                const float2 v = __half22float2(*reinterpret_cast<const __half2*>(sV + k * HD + 2 * dq));
                const float2 v0 = make_float2(v.x, v.x), v1 = make_float2(v.y, v.y);
#pragma unroll
                for (int p4 = 0; p4 < PP / 4; ++p4) {
                    const float4 e = *reinterpret_cast<const float4*>(sE + k * ESTR + p_lo + p4 * 4);
                    o[p4 * 2][0] = attn_fma2(make_float2(e.x, e.y), v0, o[p4 * 2][0]);
                    o[p4 * 2][1] = attn_fma2(make_float2(e.x, e.y), v1, o[p4 * 2][1]);
                    o[p4 * 2 + 1][0] = attn_fma2(make_float2(e.z, e.w), v0, o[p4 * 2 + 1][0]);
                    o[p4 * 2 + 1][1] = attn_fma2(make_float2(e.z, e.w), v1, o[p4 * 2 + 1][1]);
                }
            };
            int k = 0;
            for (; k + 4 <= nkeys; k += 4) { step(k); step(k + 1); step(k + 2); step(k + 3); }
            for (; k < nkeys; ++k) step(k);
#pragma unroll
            for (int p = 0; p < PP / 2; ++p) {
                if (p_lo + 2 * p < npairs) *reinterpret_cast<float2*>(a.pO + (pbase + p_lo + 2 * p) * HD + 2 * dq) = make_float2(o[p][0].x, o[p][1].x);
                if (p_lo + 2 * p + 1 < npairs) *reinterpret_cast<float2*>(a.pO + (pbase + p_lo + 2 * p + 1) * HD + 2 * dq) = make_float2(o[p][0].y, o[p][1].y);
            }
        }
    }
}

// merge the splits of one (row, q-head) in split order, gate, write f32 + q8. grid rows * n_head, 256 threads. Bound by latency: the
// maxima, weights and sums of up to 256 splits are fetched by as many threads at once, 16 partial outputs are in flight, the first under the weights.
__global__ void __launch_bounds__(256) k_attn_merge(const float* __restrict__ qkv, int ld, int n_head, int n_kv, const int* __restrict__ groups, const int* __restrict__ row_group,
                                                     int imm_pos0, int imm_rows, int imm_gr, const float* __restrict__ pO, const float* __restrict__ pm, const float* __restrict__ pl, int nsplit_max,
                                                     float* __restrict__ out, int8_t* __restrict__ oq, float* __restrict__ osc) {
    __shared__ float sw[256], sl[256], smx[8];
    pdl_launch_dependents();
    pdl_wait();
    const int r = blockIdx.x / n_head, head = blockIdx.x % n_head, d = threadIdx.x, lane = d & 31;
    const float gate = qkv[(size_t)r * ld + head * 512 + HD + d];
    const int gi = row_group ? row_group[r] : r / imm_gr;
    const int4 gd = attn_group(groups, gi, imm_pos0, imm_rows, imm_gr);
    const int G = n_head / n_kv, kh = head / G, hh = head % G, tr = r - gd.x, pair = tr * G + hh;
    const int nsplit = (gd.w + tr + 1 + SPL - 1) / SPL;
    const size_t pb = (((size_t)gi * n_kv + kh) * nsplit_max) * MAXP + pair;
    const float* po = pO + pb * HD + d;
    float m0 = d < nsplit ? pm[pb + (size_t)d * MAXP] : -INFINITY, mx = m0;
    for (int s = d + 256; s < nsplit; s += 256) mx = fmaxf(mx, pm[pb + (size_t)s * MAXP]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    float o = 0.f, l = 0.f;
    constexpr int PF = 16;   // partial outputs in flight; the first ones under the weights
    float pv[PF];
#pragma unroll
    for (int i = 0; i < PF; ++i) pv[i] = i < nsplit ? po[(size_t)i * MAXP * HD] : 0.f;
    if (lane == 0) smx[d >> 5] = mx;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w) mx = fmaxf(mx, smx[w]);
    for (int s0 = 0; s0 < nsplit; s0 += 256) {
        const int n = min(256, nsplit - s0);
        if (s0) { __syncthreads(); if (d < n) m0 = pm[pb + (size_t)(s0 + d) * MAXP]; }
        if (d < n) { sw[d] = expf_det(m0 - mx); sl[d] = pl[pb + (size_t)(s0 + d) * MAXP]; }
        __syncthreads();
        for (int s = 0; s < n; s += PF) {
#pragma unroll
            for (int i = 0; i < PF; ++i) {
                if (i % 4 == 0 && s + i >= n) break;   // nothing left to read ahead either (6 rows at position 500: a layer 31.2 -> 30.0 us)
                if (s + i < n) { o = fmaf(sw[s + i], pv[i], o); l = fmaf(sw[s + i], sl[s + i], l); }
                pv[i] = s0 + s + PF + i < nsplit ? po[(size_t)(s0 + s + PF + i) * MAXP * HD] : 0.f;
            }
        }
    }
    const float v = (o / l) * sigmoid_det(gate);
    const size_t oi = (size_t)r * n_head * HD + head * HD + d;
    if (out) out[oi] = v;
    if (oq) warp_quant32_store(v, r, (head * HD + d) >> 5, n_head * HD, oq, osc, lane);
}

template <int PPT, int NT>
int launch_split(const AttnArgs& a, dim3 grid, cudaStream_t s) {
    static bool attr[MAX_DEVICES] = {};   // per device: the opt-in belongs to the device's copy of the kernel
    const int dev = current_device(); if (dev < 0) return HP_ECUDA;
    constexpr int smem = AttnGeom<PPT, NT>::SMEM;
    if (!attr[dev]) { HP_CUDA(cudaFuncSetAttribute(k_attn_split<PPT, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)); attr[dev] = true; }
    HP_CUDA(launch_pdl<4>(k_attn_split<PPT, NT>, grid, dim3(NT), smem, s, a));
    return HP_OK;
}

}  // namespace

size_t attn_partial_floats(int ngroups, int n_kv, int nsplit_max) { return (size_t)ngroups * n_kv * nsplit_max * MAXP; }

int attn_rope_kv(const AttnParams& p, int rows, cudaStream_t s) {
    HP_REQUIRE(rows >= 1 && p.n_head % p.n_kv == 0 && p.n_rot % 2 == 0 && p.n_rot <= HD, "attn_rope_kv: bad shape");
    HP_CUDA(launch_pdl<4>(k_qk_norm_rope_kv, dim3(rows * (p.n_head + p.n_kv)), dim3(256), 0, s, p.qkv, p.planes, p.P, p.part_stride, p.ld, p.n_head, p.n_kv, (const uint16_t*)p.q_norm, (const uint16_t*)p.k_norm, (const float2*)p.rope, p.n_rot,
                       p.row_pos, p.row_slot, p.imm_pos0, (uint16_t*)p.kc, (uint16_t*)p.vc, p.kv_stride, p.max_ctx, p.eps));
    HP_CUDA(cudaGetLastError()); return HP_OK;
}
int attn_decode(const AttnParams& p, int rows, int ngroups, cudaStream_t s) {
    HP_REQUIRE(rows >= 1 && ngroups >= 1 && p.n_head % p.n_kv == 0 && (p.n_head / p.n_kv) <= MAXP, "attn_decode: at most %d (row, head) pairs per kv head and group", MAXP);
    AttnArgs a; a.qkv = p.qkv; a.ld = p.ld; a.n_head = p.n_head; a.n_kv = p.n_kv; a.kc = (const uint16_t*)p.kc; a.vc = (const uint16_t*)p.vc;
    a.kv_stride = p.kv_stride; a.max_ctx = p.max_ctx; a.groups = p.groups; a.imm_pos0 = p.imm_pos0; a.imm_rows = a.rows = rows; a.imm_gr = p.imm_gr; a.pO = p.pO; a.pm = p.pm; a.pl = p.pl; a.nsplit_max = p.nsplit_max;
    // group sizes live on the device; group_rows bounds them. Up to 8 pairs (the rows of a draft or decode step) take 2 pairs per thread
    const int pairs = (p.group_rows > 0 && p.group_rows < rows ? p.group_rows : rows) * (p.n_head / p.n_kv);
    const dim3 grid(p.nsplit_max, p.n_kv, ngroups);
    const int rc = pairs <= 8 ? launch_split<2, 256>(a, grid, s) : pairs <= 12 ? launch_split<6, 128>(a, grid, s) : pairs <= 24 ? launch_split<6, 256>(a, grid, s)
                 : pairs <= 36 ? launch_split<6, 384>(a, grid, s) : launch_split<6, 512>(a, grid, s);
    if (rc != HP_OK) return rc;
    HP_CUDA(launch_pdl<4>(k_attn_merge, dim3(rows * p.n_head), dim3(256), 0, s, p.qkv, p.ld, p.n_head, p.n_kv, p.groups, p.row_group, p.imm_pos0, rows, p.imm_gr, p.pO, p.pm, p.pl, p.nsplit_max, p.out, (int8_t*)p.xq.q, (float*)p.xq.sc));
    HP_CUDA(cudaGetLastError()); return HP_OK;
}

}  // namespace hp

namespace hp {
// Kernel-level form for one sequence: rows r = 0..R-1 at positions pos0 + r, described by value. The workspace holds the split partials.
static int attn_seq_groups(int R, int n_head, int n_kv) { const int gr = std::max(1, std::min(8, ATTN_MAX_PAIRS / (n_head / n_kv))); return (R + gr - 1) / gr; }
size_t attn_seq_workspace_bytes(int R, int n_head, int n_kv, int max_ctx) {
    const size_t np = attn_partial_floats(attn_seq_groups(R, n_head, n_kv), n_kv, (max_ctx + ATTN_SPLIT - 1) / ATTN_SPLIT);
    return np * (HD + 2) * sizeof(float);
}
int attn_decode_seq(float* qkv, int ld, int R, int pos0, int n_head, int n_kv, int n_rot, const void* q_norm, const void* k_norm, const void* rope, void* kc, void* vc, int max_ctx,
                    float* out, XQ8F xq, float eps, void* workspace, cudaStream_t s) {
    HP_REQUIRE(R >= 1 && R <= 8 && pos0 >= 0 && pos0 + R <= max_ctx, "attn_decode_seq: 1 <= R <= 8 rows inside the context");
    HP_REQUIRE(n_kv >= 1 && n_head % n_kv == 0 && n_head / n_kv <= ATTN_MAX_PAIRS && ld >= n_head * 512 + 2 * n_kv * HD, "attn_decode_seq: bad head geometry");
    const int gr = std::max(1, std::min(8, ATTN_MAX_PAIRS / (n_head / n_kv))), ng = attn_seq_groups(R, n_head, n_kv);
    AttnParams p; p.qkv = qkv; p.ld = ld; p.n_head = n_head; p.n_kv = n_kv; p.n_rot = n_rot; p.q_norm = q_norm; p.k_norm = k_norm; p.rope = rope;
    p.row_pos = p.row_slot = p.row_group = p.groups = nullptr; p.imm_pos0 = pos0; p.imm_gr = gr; p.group_rows = std::min(gr, R);
    p.kc = kc; p.vc = vc; p.kv_stride = 0; p.max_ctx = max_ctx; p.nsplit_max = (max_ctx + ATTN_SPLIT - 1) / ATTN_SPLIT;
    const size_t np = attn_partial_floats(ng, n_kv, p.nsplit_max);
    p.pO = (float*)workspace; p.pm = p.pO + np * HD; p.pl = p.pm + np;
    p.out = out; p.xq = xq; p.eps = eps;
    const int rc = attn_rope_kv(p, R, s);
    return rc != HP_OK ? rc : attn_decode(p, R, ng, s);
}
}  // namespace hp
