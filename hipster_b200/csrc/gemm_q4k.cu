// Q4_K x int8 GEMM for prompt chunks (many rows) on the 5th-generation tensor cores: tcgen05.mma kind::f8f6f4 with the
// accumulator in TMEM.
//
// The arithmetic is that of the verify GEMV (gemv_q4k.cu) operation by operation: the exact integer dot of every 32-element
// sub-block, then acc = fmaf((d*sc) * xd, (float)idot, acc); acc = fmaf(-(dmin*mn), xs, acc) in block order, with the
// sums of a 16-row tile cut where the GEMV's partition cuts them (K parts, warp boundaries of the tile's CTA) and added
// in the same order. A row therefore has the same bits whichever of the two kernels computed it.
//
// The dots come as fp32: a nibble q, read as e4m3, is q / 512 (subnormal up to 7), an int8 activation is 16 a + b with |a|, |b| <= 8, both
// exact in e4m3, and the two products accumulate exactly (at most 16 significant bits). The accumulator holds idot / 512 and the row scales
// carry the 512 (see tc_plain). (kind::i8 took one MMA instead of two, but each dot cost a conversion in the update: 34816 x 5120 at 512 rows 692 us,
// now 610.)
//
// What bounds it: the fp32 update, three packed instructions per two outputs and sub-block (12 clocks of an SM sub-partition per 16x8x32
// tile), which hardly overlaps with what brings its operands into registers: TMEM loads (16x256b fills 64 bytes a clock) and column
// scales. The loop by itself, two warps per sub-partition, takes 16 clocks per tile; in place, at 1965 MHz, 32 at 512 rows of 34816 x 5120 and 35 to 41 for
// the other projections. Left out one at a time (611 us): waits of the TMEM slots 17, closing of partial sums 24, MMAs 56, TMEM loads
// 73, column scales 128.
// Hence:
//   * one CTA per SM, M = 128 weight rows (8 tiles of 16), N = 32..128 pass rows, two tcgen05.mma (K = 32) per sub-block: TMEM
//     only hands the dots over to the update, in slots of 2 or 4 sub-blocks (slots of one, or of half the columns, cost more waits than they
//     hide: 797 and 619 us);
//   * 8 update warps (4 TMEM lane quadrants x 2 column halves) read the dots with 16x256b loads, which leave a lane two
//     rows x two adjacent columns per 16 lanes: one 16-byte read of the scales of the activations serves 4 rows. A step of a
//     warp is 5 to 8 (column tile, sub-block) pairs whatever N is, all loads in front. (16 warps with steps of half the size
//     hide more latency but execute the loads and addresses of a step twice, and these compete with the update for the
//     register ports; half a step ahead of the arithmetic: 809 us.)
//   * 4 conversion warps split the nibbles into bytes in the K-major, 64-byte-swizzled layout of the tensor core. Rows 2, 3, 6, 7 of a
//     group store their high nibbles first, so that the 16 lanes of a store phase hit distinct banks;
//   * the activations are brought into that layout, as two planes of e4m3, once per call by k_tc_pack (a few microseconds), so that a
//     half-block of a column range is one bulk copy (8-byte asynchronous copies by two warps took 2800 clocks per half-block);
//   * one warp streams the weights (2304-byte tile chunks, ring of 3 blocks, primed before the dependency wait), one the
//     activations, one thread issues the MMAs.
// Registers: 512 threads x 128 at launch; the update warps take 184 (8 x 32 threads) from the conversion warps (72) and the
// last four warps (56): 63488 in all.
// Every wait is bounded and reports through the device status word.
#include "hp_common.cuh"
#include "kernels.h"
#include <cuda_fp8.h>

namespace hp {
namespace {

constexpr int TC_EPI = 8, TC_CNV = 4, TC_THREADS = (TC_EPI + TC_CNV + 4) * 32, TC_RAWS = 3, TC_CNVS = 3;
constexpr int TC_W_CNV = TC_EPI, TC_W_LD = TC_W_CNV + TC_CNV, TC_W_TMA = TC_W_LD + 1, TC_W_MMA = TC_W_TMA + 1;   // first warp of each role
constexpr int TC_RAW_BYTES = 8 * 2304, TC_A_BYTES = 2 * 128 * 64;   // weights of one block; converted weights of half a block
template <int NTC> struct TcGeom {
    static constexpr int N = NTC * 8, GS = NTC <= 8 ? 4 : 2, SLOT = GS * N <= 128 ? 128 : 256, SLOTS = 512 / SLOT;   // GS sub-blocks per TMEM slot
    static constexpr int BST = NTC <= 8 ? 4 : NTC <= 12 ? 3 : 2, SCS = NTC <= 8 ? 4 : 3, B_BYTES = 4 * N * 64;   // rings: half-blocks of activations (two planes), blocks of scales
    static constexpr int PACK = 2 * B_BYTES + NTC * 512;                                         // packed activations of a block: two half-blocks, scales
    static constexpr int SC_BYTES = 8 * 128 * 8 + NTC * 512;
    static constexpr int OFF_A = TC_RAWS * TC_RAW_BYTES, OFF_B = OFF_A + TC_CNVS * TC_A_BYTES, OFF_SC = OFF_B + BST * B_BYTES, OFF_BAR = OFF_SC + SCS * SC_BYTES;
    static constexpr int SMEM = OFF_BAR + 512 + 1024;   // + slack to align the ring to 1024 bytes
};
static_assert(TcGeom<16>::SMEM <= GEMV_SMEM_LIMIT && TcGeom<12>::SMEM <= GEMV_SMEM_LIMIT && TcGeom<8>::SMEM <= GEMV_SMEM_LIMIT, "shared memory of the widest tiles");

// Bounded wait that lets the hardware park the warp: up to 2^20 attempts of up to a microsecond
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity, int* err) {
    for (uint32_t it = 0; it < (1u << 20); ++it) {
        uint32_t ok;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(bar), "r"(parity), "r"(1000u) : "memory");
        if (ok) return true;
    }
    if (err) atomicExch(err, HP_ETIMEOUT);
    return false;
}
// one lane of a converged warp; unlike lane == 0 the compiler knows that a single thread issues what follows
__device__ __forceinline__ bool tc_elect() {
    uint32_t p;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr) {   // K-major operand, 64-byte swizzle: 8-row groups 512 bytes apart
    return (uint64_t)((addr >> 4) & 0x3FFF) | (1ull << 16) | (32ull << 32) | (1ull << 46) | (4ull << 61);
}
__device__ __forceinline__ void tc_mma_f8(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, int add) {   // D = A * B (+ D)
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(add) : "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
template <int N> __device__ __forceinline__ void tc_reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void tc_reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;"); }
__device__ __forceinline__ void tc_after_wait(uint32_t& v) { asm volatile("" : "+r"(v)); }   // orders the use of a loaded register behind tc_wait_ld
// W column tiles of 8 for 16 TMEM lanes: v[4 i ..] = {row g: cols 2t, 2t+1; row g + 8: cols 2t, 2t+1} of tile i
template <int W, int OFF = 0> __device__ __forceinline__ void tc_ld(uint32_t (&v)[W * 4], uint32_t addr) {
    constexpr int o = OFF * 4;
    if constexpr (W - OFF >= 4) {
        asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                     : "=r"(v[o]), "=r"(v[o + 1]), "=r"(v[o + 2]), "=r"(v[o + 3]), "=r"(v[o + 4]), "=r"(v[o + 5]), "=r"(v[o + 6]), "=r"(v[o + 7]), "=r"(v[o + 8]),
                       "=r"(v[o + 9]), "=r"(v[o + 10]), "=r"(v[o + 11]), "=r"(v[o + 12]), "=r"(v[o + 13]), "=r"(v[o + 14]), "=r"(v[o + 15]) : "r"(addr + OFF * 8));
        if constexpr (W - OFF > 4) tc_ld<W, OFF + 4>(v, addr);
    } else if constexpr (W - OFF >= 2) {
        asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(v[o]), "=r"(v[o + 1]), "=r"(v[o + 2]), "=r"(v[o + 3]), "=r"(v[o + 4]), "=r"(v[o + 5]), "=r"(v[o + 6]), "=r"(v[o + 7]) : "r"(addr + OFF * 8));
        if constexpr (W - OFF > 2) tc_ld<W, OFF + 2>(v, addr);
    } else
        asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[o]), "=r"(v[o + 1]), "=r"(v[o + 2]), "=r"(v[o + 3]) : "r"(addr + OFF * 8));
}

struct TcArgs {
    const uint8_t* W; const uint8_t* xp; float* y;   // xp: packed activations
    int N, nb, P, R, ldy; size_t part_stride;
    int G, ngrp, ncg;        // tiles of 16 rows per work item (8, or 4 with every second tile position empty), items along M, along the pass rows
    int nlong, heavy, light; // ranges of NTC column tiles (the others have two less); CTAs with one item more, items of the other CTAs
    int* err;
};
// Item `it` of the launch: column range, its first column tile, and part * ngrp + group. Wide ranges go to the CTAs with fewer items first
// (34816 x 5120 at 304 rows, 38 tiles as 14 + 12 + 12 instead of 3 x 14: 433 -> 410 us, 5120 x 17408 269 -> 248).
struct TcItem { int cg, c0, rest; bool narrow; };
__device__ __forceinline__ TcItem tc_item(const TcArgs& a, int it, int ntc) {
    const int n = gridDim.x, k = it / n, i = it % n, nl = a.nlong * a.ngrp * a.P;
    int j = i >= a.heavy ? k * (n - a.heavy) + i - a.heavy : a.light + k * a.heavy + i;
    TcItem v;
    v.narrow = j >= nl;
    if (!v.narrow) { v.cg = j % a.nlong; v.rest = j / a.nlong; v.c0 = v.cg * ntc; }
    else { j -= nl; const int ns = a.ncg - a.nlong; v.cg = a.nlong + j % ns; v.rest = j / ns; v.c0 = a.nlong * ntc + (j % ns) * (ntc - 2); }
    return v;
}
// Units of tile `tile` after which the GEMV's partition closes a partial sum: bit c of the result = after unit c (CB blocks) of the K part
__device__ __forceinline__ uint64_t tc_cuts(int N, int nb, int P, int tile, int lane) {
    const int tiles = (N + 15) / 16, gc = GEMV_NCTA / P, nbp = nb / P, C = nbp % 2 == 0 ? nbp / 2 : nbp;
    const int cg = (int)(((long long)(tile + 1) * gc - 1) / tiles);
    const int t0 = (int)((long long)cg * tiles / gc), t1 = (int)((long long)(cg + 1) * tiles / gc);
    const int cu = (t1 - t0) * C, weff = cu < GEMV_WARPS ? cu : GEMV_WARPS;
    uint64_t m = 0;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int c = lane + 32 * half, u = (tile - t0) * C + c + 1;
        bool cut = false;
        if (c < C) { const int w = (u * weff + cu - 1) / cu; cut = c == C - 1 || (w < weff && gemv_warp_start(cu, weff, w) == u); }
        m |= (uint64_t)__ballot_sync(0xffffffffu, cut) << (32 * half);
    }
    return m;
}

// The one rounding in front of the fmaf is that of the product (d * sc) * xd, of d / 16 where the GEMV leaves the high nibbles shifted. With xd of this
// range it is no subnormal number (f16 d: d / 16 is 2^-28 at least) and 512 times (d * sc) * xd no infinity (d * sc is less than 2^22), so the row
// scales may carry the 512. A launch with other scales (heads whose gates underflow have them; NaN) takes the GEMV's own product, one packed
// multiplication more per two outputs: in a prompt of the 27B shape two launches of 192. Prompts against a kernel without these loops (which also shift
// the registers of the common ones): 27B shape 52 tokens 19.7 -> 19.5 ms, 130 tokens 42.7 -> 42.2, 301 tokens 75.1 -> 75.3, 2048-wide experts 200 tokens
// 24.4 -> 24.6. (Left to the tensor core, which then repeats its products up to the GEMV's dot, such a launch takes three to eight times as long.)
__device__ __forceinline__ bool tc_plain(float xd) { return xd == 0.f || (xd >= 0x1p-98f && xd <= 0x1p96f); }

// One step of an update warp: its W column tiles over GB sub-blocks (row scales 128 float2 apart, one 64-byte group of
// activation scales per sub-block). H1: the quadrant's second tile exists. EXACT: the scale and the dot of the GEMV, d * sc and idot, or (odd
// sub-block) d / 16 * sc and 16 idot, GB = 1.
template <int W, int GB, bool H1, bool EXACT>
__device__ __forceinline__ void tc_update(float2 (&acc)[4][W], uint32_t ta, uint32_t sb_cols, const float4* xs, const float2* rs, bool odd) {
    uint32_t v0[GB][W * 4], v1[H1 ? GB : 1][W * 4];
#pragma unroll
    for (int b = 0; b < GB; ++b) {
        tc_ld<W>(v0[b], ta + b * sb_cols);
        if constexpr (H1) tc_ld<W>(v1[b], ta + b * sb_cols + (16u << 16));
    }
    float2 r[GB][H1 ? 4 : 2];
#pragma unroll
    for (int b = 0; b < GB; ++b)
#pragma unroll
        for (int i = 0; i < (H1 ? 4 : 2); ++i) r[b][i] = rs[b * 128 + 8 * i];
    // column scales of up to 8 column tiles four (tile, sub-block) pairs ahead: the first under the accumulator loads, the others under
    // the arithmetic (34816 x 5120: 32 rows 73 -> 67 us, 64 rows 113 -> 104; wider tiles have no registers for it: 512 rows 693 -> 752)
    constexpr int NX = GB * W, XA = W > 4 ? 1 : 4;
    auto xat = [&](int j) { return xs[(j % W) * 32 + (j / W) * 4]; };
    float4 xb[XA];
#pragma unroll
    for (int j = 0; j < XA; ++j) if (W <= 4 && j < NX) xb[j] = xat(j);
    tc_wait_ld();
#pragma unroll
    for (int b = 0; b < GB; ++b)
#pragma unroll
        for (int i = 0; i < W * 4; ++i) { tc_after_wait(v0[b][i]); if constexpr (H1) tc_after_wait(v1[b][i]); }
    const float f = odd ? 8192.f : 512.f;
    if constexpr (EXACT) {
        static_assert(GB == 1, "one parity");
#pragma unroll
        for (int i = 0; i < (H1 ? 4 : 2); ++i) r[0][i].x *= odd ? 1.f / 8192.f : 1.f / 512.f;
    }
    auto upd = [&](float2& a, float2 sc, float4 xv, uint32_t i0, uint32_t i1) {
        float2 dot = make_float2(__uint_as_float(i0), __uint_as_float(i1));
        if constexpr (EXACT) dot = mul2(dot, make_float2(f, f));
        fma2(a, mul2(make_float2(sc.x, sc.x), make_float2(xv.x, xv.y)), dot);
        fma2(a, make_float2(sc.y, sc.y), make_float2(xv.z, xv.w));
    };
#pragma unroll
    for (int b = 0; b < GB; ++b)
#pragma unroll
        for (int i = 0; i < W; ++i) {
            const int j = b * W + i;
            const float4 x = W <= 4 ? xb[j % XA] : xat(j);
            if (W <= 4 && j + XA < NX) xb[j % XA] = xat(j + XA);
            upd(acc[0][i], r[b][0], x, v0[b][4 * i], v0[b][4 * i + 1]);
            upd(acc[1][i], r[b][1], x, v0[b][4 * i + 2], v0[b][4 * i + 3]);
            if constexpr (H1) {
                upd(acc[2][i], r[b][2], x, v1[b][4 * i], v1[b][4 * i + 1]);
                upd(acc[3][i], r[b][3], x, v1[b][4 * i + 2], v1[b][4 * i + 3]);
            }
        }
}

template <int NTC>
__global__ void __launch_bounds__(TC_THREADS, 1) k_gemm_q4k_tc(const TcArgs a) {
    using Geo = TcGeom<NTC>;
    constexpr int GS = Geo::GS, SLOTS = Geo::SLOTS, BST = Geo::BST;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint32_t tmem_ptr;
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const uint32_t bars = smem_u32(smem + Geo::OFF_BAR);
    const uint32_t raw_full = bars, raw_empty = bars + 64, a_full = bars + 128, a_empty = bars + 160, sc_full = bars + 192, sc_empty = bars + 224,
                   tm_full = bars + 256, tm_empty = bars + 288, b_full = bars + 320, b_empty = bars + 384, fin = bars + 448;
    pdl_launch_dependents();
    if (tid == 0) {
        for (int i = 0; i < TC_RAWS; ++i) { mbar_init(raw_full + 8 * i, 1); mbar_init(raw_empty + 8 * i, TC_CNV); }
        for (int i = 0; i < TC_CNVS; ++i) { mbar_init(a_full + 8 * i, TC_CNV); mbar_init(a_empty + 8 * i, 1); }
        for (int i = 0; i < Geo::SCS; ++i) { mbar_init(sc_full + 8 * i, TC_CNV + 1); mbar_init(sc_empty + 8 * i, TC_EPI); }
        for (int i = 0; i < 4; ++i) { mbar_init(tm_full + 8 * i, 1); mbar_init(tm_empty + 8 * i, TC_EPI); }
        for (int i = 0; i < BST; ++i) { mbar_init(b_full + 8 * i, 1); mbar_init(b_empty + 8 * i, 1); }
        mbar_init(fin, 1);
        fence_barrier_init();
    }
    if (warp == TC_W_MMA) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_ptr)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_ptr;
    const int nb = a.nb, nbp = nb / a.P, tiles = (a.N + 15) / 16, G = a.G, items = a.ncg * a.ngrp * a.P;
    // 8 bytes of lane (g, t) in a swizzled group of 8 rows x 64 bytes: first store (low half of the 64 elements, high half
    // for odd row pairs); the other half is at sw ^ 32
    const bool sel = (g >> 1) & 1;
    const uint32_t sw = (uint32_t)(((((sel ? 2 : 0) + (t >> 1)) ^ ((g >> 1) & 3)) << 4) + (t & 1) * 8 + g * 64);

    if (warp >= TC_W_LD) {
        tc_reg_dec<56>();
        if (warp == TC_W_TMA) {   // ---- weight stream: one 2304-byte chunk per tile and block
            int k = 0; bool ok = true;
            for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
                const int rest = tc_item(a, it, NTC).rest, grp = rest % a.ngrp, part = rest / a.ngrp, nt = min(G, tiles - grp * G);
                const uint8_t* src = a.W + ((size_t)(grp * G) * nb + (size_t)part * nbp) * 2304;
                for (int b = 0; b < nbp; ++b, ++k) {
                    const int s = k % TC_RAWS;
                    ok = tc_wait(raw_empty + 8 * s, ((k / TC_RAWS) & 1) ^ 1, a.err);
                    if (!ok) break;
                    if (tc_elect()) {
                        mbar_expect_tx(raw_full + 8 * s, (uint32_t)nt * 2304u);
                        const uint32_t d = smem_u32(smem + s * TC_RAW_BYTES);
                        for (int i = 0; i < nt; ++i) bulk_g2s(d + i * 2304, src + ((size_t)i * nb + b) * 2304, 2304u, raw_full + 8 * s);
                    }
                    __syncwarp();
                }
            }
            for (int i = k > TC_RAWS ? k - TC_RAWS : 0; i < k; ++i) tc_wait(raw_full + 8 * (i % TC_RAWS), (i / TC_RAWS) & 1, a.err);   // no copy outlives the CTA
        } else if (warp == TC_W_MMA) {   // ---- MMA issue
            int hb = 0, gr = 0; bool ok = true;
            for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
                const uint32_t idesc = (1u << 4) | ((uint32_t)(tc_item(a, it, NTC).narrow ? NTC - 2 : NTC) << 17) | (8u << 24);   // f32 = e4m3 x e4m3, M = 128
                for (int h = 0; h < 2 * nbp && ok; ++h, ++hb) {
                    const int as = hb % TC_CNVS, bs = hb % BST;
                    ok = tc_wait(b_full + 8 * bs, (hb / BST) & 1, a.err) && tc_wait(a_full + 8 * as, (hb / TC_CNVS) & 1, a.err);
                    const uint32_t abase = smem_u32(smem + Geo::OFF_A + as * TC_A_BYTES), bbase = smem_u32(smem + Geo::OFF_B + bs * Geo::B_BYTES);
#pragma unroll
                    for (int q = 0; q < 4 && ok; q += GS, ++gr) {
                        const int slot = gr % SLOTS;
                        ok = tc_wait(tm_empty + 8 * slot, ((gr / SLOTS) & 1) ^ 1, a.err);
                        if (!ok) break;
                        tc_fence_after();
                        if (tc_elect()) {
#pragma unroll
                            for (int v = q; v < q + GS; ++v)
#pragma unroll
                                for (int pl = 0; pl < 2; ++pl)
                                    tc_mma_f8(tmem + slot * Geo::SLOT + (v - q) * Geo::N, tc_desc(abase + (v >> 1) * 8192 + (v & 1) * 32),
                                              tc_desc(bbase + ((v >> 1) * 2 + pl) * (Geo::N * 64) + (v & 1) * 32), idesc, pl);
                            tc_commit(tm_full + 8 * slot);
                            if (q + GS == 4) { tc_commit(a_empty + 8 * as); tc_commit(b_empty + 8 * bs); }
                        }
                        __syncwarp();
                    }
                }
            }
            if (tc_elect()) tc_commit(fin);
            __syncwarp();
            tc_wait(fin, 0, a.err);   // nothing in flight when the accumulator memory is given back
        } else if (warp == TC_W_LD) {   // ---- activations and their scales
            pdl_wait();
            int hb = 0, k = 0; bool ok = true;
            for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
                const TcItem im = tc_item(a, it, NTC); const int cg = im.cg, part = im.rest / a.ngrp;
                const uint8_t* src = a.xp + ((size_t)cg * nb + (size_t)part * nbp) * Geo::PACK;
                for (int b = 0; b < nbp && ok; ++b, ++k, src += Geo::PACK) {
                    const int ss = k % Geo::SCS;
                    ok = tc_wait(sc_empty + 8 * ss, ((k / Geo::SCS) & 1) ^ 1, a.err);
                    if (!ok) break;
                    if (tc_elect()) {
                        mbar_expect_tx(sc_full + 8 * ss, NTC * 512);
                        bulk_g2s(smem_u32(smem + Geo::OFF_SC + ss * Geo::SC_BYTES + 8192), src + 2 * Geo::B_BYTES, NTC * 512, sc_full + 8 * ss);
                    }
                    __syncwarp();
                    for (int h = 0; h < 2 && ok; ++h, ++hb) {
                        const int bs = hb % BST;
                        ok = tc_wait(b_empty + 8 * bs, ((hb / BST) & 1) ^ 1, a.err);
                        if (ok && tc_elect()) {
                            mbar_expect_tx(b_full + 8 * bs, Geo::B_BYTES);
                            bulk_g2s(smem_u32(smem + Geo::OFF_B + bs * Geo::B_BYTES), src + h * Geo::B_BYTES, Geo::B_BYTES, b_full + 8 * bs);
                        }
                        __syncwarp();
                    }
                }
            }
            // no copy outlives the CTA (the scales of a block are issued before its activations)
            const int nh = ok ? hb : hb ? hb - 1 : 0;
            for (int i = nh > BST ? nh - BST : 0; i < nh; ++i) tc_wait(b_full + 8 * (i % BST), (i / BST) & 1, a.err);
            if (k) { const int i = k - 1; tc_wait(sc_full + 8 * (i % Geo::SCS), (i / Geo::SCS) & 1, a.err); }
        }
    } else if (warp >= TC_W_CNV) {   // ---- weights: row scales, nibbles -> bytes
        tc_reg_dec<72>();
        const int cw = warp - TC_W_CNV, ct = cw * 32 + lane;
        const int sh_a = sel ? 4 : 0, sh_b = 4 - sh_a;   // nibbles of the first store; the second takes the others
        auto nib = [](uint32_t v, int sh) { return (v >> sh) & 0x0F0F0F0Fu; };
        int k = 0, hb = 0; bool ok = true;
        for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
            const int grp = tc_item(a, it, NTC).rest % a.ngrp, nt = min(G, tiles - grp * G);
            for (int b = 0; b < nbp && ok; ++b, ++k) {
                const int s = k % TC_RAWS, ss = k % Geo::SCS;
                const uint8_t* raw = smem + s * TC_RAW_BYTES;
                ok = tc_wait(raw_full + 8 * s, (k / TC_RAWS) & 1, a.err);
#pragma unroll 1
                for (int h = 0; h < 2 && ok; ++h, ++hb) {
                    const int as = hb % TC_CNVS;
                    ok = tc_wait(a_empty + 8 * as, ((hb / TC_CNVS) & 1) ^ 1, a.err);
                    if (!ok) break;
                    uint8_t* A = smem + Geo::OFF_A + as * TC_A_BYTES;
                    const uint8_t* rp = raw + 256 + 2 * h * 512 + lane * 16;
                    uint4 w[4];   // unit u = cw + 4 i: tile u / 2, 64-element group u % 2 of the half-block
#pragma unroll
                    for (int i = 0; i < 4; ++i) { const int u = cw + 4 * i; if ((u >> 1) < nt) w[i] = *reinterpret_cast<const uint4*>(rp + (u >> 1) * 2304 + (u & 1) * 512); }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int u = cw + 4 * i;
                        if ((u >> 1) < nt) {
                            uint8_t* d = A + (u & 1) * 8192 + (G == 8 ? (u >> 1) : (u & ~1)) * 1024;
                            *reinterpret_cast<uint2*>(d + sw) = make_uint2(nib(w[i].x, sh_a), nib(w[i].y, sh_a));
                            *reinterpret_cast<uint2*>(d + (sw ^ 32)) = make_uint2(nib(w[i].x, sh_b), nib(w[i].y, sh_b));
                            *reinterpret_cast<uint2*>(d + 512 + sw) = make_uint2(nib(w[i].z, sh_a), nib(w[i].w, sh_a));
                            *reinterpret_cast<uint2*>(d + 512 + (sw ^ 32)) = make_uint2(nib(w[i].z, sh_b), nib(w[i].w, sh_b));
                        }
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(a_full + 8 * as);
                    if (h == 0) {   // scales of tile position ct / 16, row ct % 16: (d * sc, -(dmin * mn)) of the 8 sub-blocks
                        ok = tc_wait(sc_empty + 8 * ss, ((k / Geo::SCS) & 1) ^ 1, a.err);
                        if (!ok) break;
                        const int pos = ct >> 4, ti = G == 8 ? pos : pos >> 1;
                        if (ti < nt && (G == 8 || !(pos & 1))) {
                            RowScales rs = decode_scales(*reinterpret_cast<const uint4*>(raw + ti * 2304 + (ct & 15) * 16));
                            rs.dq = rs.d = rs.d * 512.f; rs.cdq = rs.cd = -(rs.d * 8388608.f);   // the accumulators hold idot / 512
                            float2* sp = reinterpret_cast<float2*>(smem + Geo::OFF_SC + ss * Geo::SC_BYTES) + ct;
#pragma unroll
                            for (int q = 0; q < 8; ++q) { const float4 v = rs.get(q); sp[q * 128] = make_float2(v.x, v.z); }
                        }
                        __syncwarp();
                        if (lane == 0) mbar_arrive(sc_full + 8 * ss);
                    }
                }
                if (ok && lane == 0) mbar_arrive(raw_empty + 8 * s);
            }
        }
    } else {   // ---- fp32 update: warp = (lane quadrant q, column half); half h of the quadrant holds one tile of 16 rows
        tc_reg_inc<184>();
        const int q = warp & 3;
        pdl_wait();
        int k = 0, gr = 0; bool ok = true;
        const int cb1 = nbp % 2 == 0 ? 1 : 0;   // blocks per unit of the GEMV's partition, less 1
        auto item = [&](const TcItem im, auto wt, auto exact) {
            constexpr bool EXACT = decltype(exact)::value;
            constexpr int W = decltype(wt)::value, GB = EXACT ? 1 : W <= 2 ? 4 : W <= 4 ? 2 : 1;   // column tiles of this warp, sub-blocks per step
            const int grp = im.rest % a.ngrp, part = im.rest / a.ngrp, tile0 = grp * G, tend = min(tiles, tile0 + G), n0 = (warp >> 2) * W;
            const int tl[2] = {tile0 + (G == 8 ? 2 * q : q), G == 8 ? tile0 + 2 * q + 1 : tiles};
            const bool has0 = tl[0] < tend, has1 = tl[1] < tend;
            const uint64_t cut[2] = {has0 ? tc_cuts(a.N, nb, a.P, tl[0], lane) : 0, has1 ? tc_cuts(a.N, nb, a.P, tl[1], lane) : 0};
            float* y = a.y + (size_t)part * a.part_stride;
            constexpr bool VREG = W <= 4;   // running sum of the closed pieces in registers, else in the output plane
            float2 acc[4][W], sum[VREG ? 4 : 1][VREG ? W : 1];
            bool first[2] = {true, true};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int w = 0; w < W; ++w) acc[i][w] = make_float2(0.f, 0.f);
            for (int b = 0; b < nbp && ok; ++b, ++k) {
                const int ss = k % Geo::SCS;
                const uint8_t* scp = smem + Geo::OFF_SC + ss * Geo::SC_BYTES;
                ok = tc_wait(sc_full + 8 * ss, (k / Geo::SCS) & 1, a.err);
                if (!ok) break;
                const float2* rsp = reinterpret_cast<const float2*>(scp) + q * 32 + g;
                const float4* xsp = reinterpret_cast<const float4*>(scp + 8192) + n0 * 32 + t;
#pragma unroll 1
                for (int u = 0; u < 8 / GS && ok; ++u, ++gr) {
                    const int slot = gr % SLOTS;
                    ok = tc_wait(tm_full + 8 * slot, (gr / SLOTS) & 1, a.err);
                    if (!ok) break;
                    tc_fence_after();
                    if (has0) {
#pragma unroll 1
                        for (int v = 0; v < GS; v += GB) {
                            const int sb = u * GS + v;
                            const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + slot * Geo::SLOT + v * Geo::N + n0 * 8;
                            if (has1) tc_update<W, GB, true, EXACT>(acc, ta, Geo::N, xsp + sb * 4, rsp + sb * 128, sb & 1);
                            else tc_update<W, GB, false, EXACT>(acc, ta, Geo::N, xsp + sb * 4, rsp + sb * 128, sb & 1);
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(tm_empty + 8 * slot);
                }
                if (!ok) break;
                __syncwarp();
                if (lane == 0) mbar_arrive(sc_empty + 8 * ss);
                // partial sums that end with this block
                if ((b & cb1) == cb1) {
                    const int c = b >> cb1;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (!((cut[h] >> c) & 1)) continue;
                        const bool last = b + 1 == nbp;
                        int ldy = a.ldy;
                        asm volatile("" : "+r"(ldy));   // keeps the addresses of this rare path out of the registers of the loop
                        if constexpr (VREG) {
#pragma unroll
                            for (int i = 0; i < 2; ++i)
#pragma unroll
                                for (int w = 0; w < W; ++w) {
                                    float2 v = acc[2 * h + i][w]; acc[2 * h + i][w] = make_float2(0.f, 0.f);
                                    if (!first[h]) v = make_float2(sum[2 * h + i][w].x + v.x, sum[2 * h + i][w].y + v.y);
                                    sum[2 * h + i][w] = v;
                                }
                            if (!last) { first[h] = false; continue; }
                        }
                        // element {i, w, e}: row + 8 i, column 2 t + 8 w + e. Other warps wait at the next slot for the one that closes a
                        // tile: whole tiles and ranges without predicates, one pointer per column pair, all loads in front
                        const int row = tl[h] * 16 + g, col = (im.c0 + n0) * 8 + 2 * t;
                        float* yt = y + (size_t)col * ldy + row;
                        const size_t step = (size_t)8 * ldy;
                        auto close = [&](auto live) {
                            if constexpr (!VREG) {
                                if (!first[h]) {
                                    float p[W][4];
                                    const float* yp = yt;
#pragma unroll
                                    for (int w = 0; w < W; ++w, yp += step) {
                                        const float* yq = yp + ldy;
                                        p[w][0] = live(0, w, 0) ? yp[0] : 0.f; p[w][1] = live(0, w, 1) ? yq[0] : 0.f; p[w][2] = live(1, w, 0) ? yp[8] : 0.f; p[w][3] = live(1, w, 1) ? yq[8] : 0.f;
                                    }
#pragma unroll
                                    for (int w = 0; w < W; ++w)
#pragma unroll
                                        for (int i = 0; i < 2; ++i) { float2& v = acc[2 * h + i][w]; v.x = p[w][2 * i] + v.x; v.y = p[w][2 * i + 1] + v.y; }
                                }
                            }
                            float* yp = yt;
#pragma unroll
                            for (int w = 0; w < W; ++w, yp += step) {
                                float* yq = yp + ldy;
#pragma unroll
                                for (int i = 0; i < 2; ++i) {
                                    const float2 v = VREG ? sum[VREG ? 2 * h + i : 0][VREG ? w : 0] : acc[2 * h + i][w];
                                    if (live(i, w, 0)) yp[8 * i] = v.x;
                                    if (live(i, w, 1)) yq[8 * i] = v.y;
                                    if constexpr (!VREG) acc[2 * h + i][w] = make_float2(0.f, 0.f);
                                }
                            }
                        };
                        if (tl[h] * 16 + 16 <= a.N && (im.c0 + n0 + W) * 8 <= a.R) close([](int, int, int) { return true; });
                        else close([&](int i, int w, int e) { return row + 8 * i < a.N && col + 8 * w + e < a.R; });
                        first[h] = false;
                    }
                }
            }
        };
        auto all_items = [&](auto exact) {
            for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
                const TcItem im = tc_item(a, it, NTC);
                if (im.narrow) item(im, std::integral_constant<int, NTC / 2 - 1>(), exact); else item(im, std::integral_constant<int, NTC / 2>(), exact);
            }
        };
        const int* flags = reinterpret_cast<const int*>(a.xp + (size_t)a.ncg * nb * Geo::PACK);   // of k_tc_pack; read at once, while the first slots fill
        int other = 0;
        for (int i0 = lane; i0 < a.ncg * nb; i0 += 256) {
#pragma unroll
            for (int i = 0; i < 256; i += 32) other |= i0 + i < a.ncg * nb ? __ldcg(flags + i0 + i) : 0;
        }
        if (__any_sync(0xffffffffu, other)) all_items(std::true_type()); else all_items(std::false_type());
    }
    tc_fence_before();
    __syncthreads();
    if (warp == TC_W_MMA)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// four int8 as e4m3: x = 16 a + b with |a|, |b| <= 8; hi = 16 a, lo = b, both exact
__device__ __forceinline__ void tc_split(uint32_t x, uint32_t& hi, uint32_t& lo) {
    hi = lo = 0u;
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
        const int v0 = (int)(int8_t)(x >> (8 * i)), v1 = (int)(int8_t)(x >> (8 * i + 8)), a0 = (v0 + 8) & ~15, a1 = (v1 + 8) & ~15;
        hi |= (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2((float)a0, (float)a1), __NV_SATFINITE, __NV_E4M3) << (8 * i);
        lo |= (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2((float)(v0 - a0), (float)(v1 - a1)), __NV_SATFINITE, __NV_E4M3) << (8 * i);
    }
}
// Activations in the order the GEMM copies them: per column range of NTC tiles and block two half-blocks (per 64-element
// group the swizzled K-major tile of all columns), then the scales. Tiles beyond the range and the rows are zero. Behind all of them an int per
// range and block: whether one of its scales is beyond tc_plain.
template <int NTC>
__global__ void __launch_bounds__(256) k_tc_pack(const uint4* __restrict__ xq, const float4* __restrict__ xsc, uint8_t* __restrict__ xp, int nb, int tiles8, int nlong) {
    pdl_launch_dependents();
    pdl_wait();
    const int blk = blockIdx.x, cg = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int c0 = cg * NTC - 2 * max(cg - nlong, 0), cend = min(tiles8, c0 + (cg < nlong ? NTC : NTC - 2));
    uint8_t* d = xp + ((size_t)cg * nb + blk) * TcGeom<NTC>::PACK;
    const uint32_t lo = (uint32_t)((((t >> 1) ^ ((g >> 1) & 3)) << 4) + (t & 1) * 8 + g * 64);   // the low sub-block's 8 bytes; the high one's: lo ^ 32
#pragma unroll
    for (int u = warp; u < NTC * 4; u += 8) {
        const int n = u >> 2, jj = u & 3, nt = c0 + n;
        const uint4 v = nt < cend ? xq[((size_t)nt * nb * 4 + (size_t)blk * 4 + jj) * 32 + lane] : make_uint4(0, 0, 0, 0);
        uint8_t* p = d + (jj >> 1) * TcGeom<NTC>::B_BYTES + (jj & 1) * (2 * NTC * 512) + n * 512;
        uint2 h, l;
        tc_split(v.x, h.x, l.x); tc_split(v.y, h.y, l.y);
        *reinterpret_cast<uint2*>(p + lo) = h; *reinterpret_cast<uint2*>(p + NTC * 512 + lo) = l;
        tc_split(v.z, h.x, l.x); tc_split(v.w, h.y, l.y);
        *reinterpret_cast<uint2*>(p + (lo ^ 32)) = h; *reinterpret_cast<uint2*>(p + NTC * 512 + (lo ^ 32)) = l;
    }
    bool other = false;
    for (int n = warp; n < NTC; n += 8) {
        const int nt = c0 + n;
        const float4 v = nt < cend ? xsc[((size_t)nt * nb + blk) * 32 + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
        other |= !tc_plain(v.x) || !tc_plain(v.y);
        reinterpret_cast<float4*>(d + 2 * TcGeom<NTC>::B_BYTES)[n * 32 + lane] = v;
    }
    other = __syncthreads_or(other);
    if (threadIdx.x == 0) reinterpret_cast<int*>(xp + (size_t)gridDim.y * nb * TcGeom<NTC>::PACK)[cg * nb + blk] = other;
}

template <int NTC>
int launch_tc(const TcArgs& a, const XQ8F& x, int grid, cudaStream_t s, bool pdl) {
    constexpr int smem = TcGeom<NTC>::SMEM;
    static bool attr[MAX_DEVICES] = {};   // per device: the opt-in belongs to the device's copy of the kernel
    const int dev = current_device(); if (dev < 0) return HP_ECUDA;
    if (!attr[dev]) { HP_CUDA(cudaFuncSetAttribute(k_gemm_q4k_tc<NTC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)); attr[dev] = true; }
    k_tc_pack<NTC><<<dim3(a.nb, a.ncg), 256, 0, s>>>((const uint4*)x.q, (const float4*)x.sc, (uint8_t*)a.xp, a.nb, (a.R + 7) / 8, a.nlong);
    HP_CUDA(cudaGetLastError());
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid); cfg.blockDim = dim3(TC_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = s;
    cudaLaunchAttribute at[1]; at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = pdl && !(pdl_off_mask(s) & 64) ? 1 : 0;
    HP_CUDA(cudaLaunchKernelEx(&cfg, k_gemm_q4k_tc<NTC>, a));
    return HP_OK;
}

}  // namespace

size_t gemm_pack_bytes(int R, int K) { return (size_t)((R + 7) / 8 + 15) * (size_t)(K / 256) * (4608 + 4); }
// A cut into ranges of ntc column tiles leaves up to ntc - 1 empty: the number of ranges, not the first, that get two tiles less instead.
static int tc_narrow(int R, int ntc) {
    const int t8 = (R + 7) / 8, ncg = (t8 + ntc - 1) / ntc, k = (ncg * ntc - t8) / 2;
    return k < ncg - 1 ? k : ncg - 1;
}
// The cut of the rows into column ranges of ntc tiles of 8, and of the weight tiles into items of G = 8 or 4 (the latter leaves every second
// tile position empty): the one whose fullest CTA takes the least time. Of an item of 20 blocks that is, at ntc = 4, 8, 10, 14 and 16, 34, 47, 63, 76
// and 83 us (ntc + 8, from 10 on ntc + 11: half as many sub-blocks per TMEM slot), 1.25 of these units less for a narrow range, four fifths
// with G = 4. Over eight projections and 18 row counts from 56 to 512 that is 0.4 % slower than the best cut on average, 6 % at most (with ntc + 6,
// narrow ranges 2 less, 1.0 and 15 %).
struct TcCost { long items, cost; };   // of the fullest CTA: items, and quarters of the units above x (5 or 4)
static TcCost tc_cost(int N, int K, int R, int c, int g) {
    const int t8 = (R + 7) / 8, tiles = (N + 15) / 16, P = gemv_num_parts(N, K / 256);
    // CTAs with one item more and the others: their items, and at most how many wide ones among these (see tc_item)
    const long ncg = (t8 + c - 1) / c, per = (long)P * ((tiles + g - 1) / g), nl = (ncg - tc_narrow(R, c)) * per, items = ncg * per;
    const long n = items < GEMV_NCTA ? items : GEMV_NCTA, full = items / n, heavy = items % n, light = n - heavy, over = nl - full * light;
    const long wl = (nl + light - 1) / light, wh = heavy && over > 0 ? (over + heavy - 1) / heavy : 0;
    const long u = 4 * (c + (c > 8 ? 11 : 8)) - 5, cl = full * u + 5 * (wl < full ? wl : full), ch = heavy ? (full + 1) * u + 5 * wh : 0;
    return {full + (heavy ? 1 : 0), (cl > ch ? cl : ch) * (g == 8 ? 5 : 4)};
}
void gemm_cut(int N, int K, int R, int* ntc, int* G) {
    long best = 0; *ntc = 0;
    for (int c = 4; c <= 16; c += 2)
        for (int g = 8; g >= 4; g -= 4) {
            const long cost = tc_cost(N, K, R, c, g).cost;
            if (!*ntc || cost < best) { best = cost; *ntc = c; *G = g; }
        }
}
// The GEMM against the GEMV in launches of 32 rows, in us. A GEMV launch: 1.2, 0.24 per block of a K part (staging) and 0.52 per block and column
// tile of its fullest warp; the GEMM: 5.2, 1.9 per item of the fullest CTA and the cost above, and 2 for its second launch, which nothing
// hides in a prompt (up to 48 rows that decides it: 44 rows of the 27B shape 17.3 and 17.7 ms). Over ten projections and 21 row counts from 33
// to 192, one by one, the choice is 1.2 % slower than the faster of the two on average, 22 % at most (one line at 48 rows for all projections: 7 and
// 97 %). 56 rows, 5120 x 17408: 55 us instead of 86; 64 rows, 14336 x 2048: 23 instead of 32. Prompts (ms), one line and this rule: 27B shape, 52 tokens
// 22.1 and 19.9, 84 tokens 30.7 and 28.0, 130 tokens 44.3 and 42.8; 2048-wide mixture of experts, 60 tokens 13.9 and 13.2.
bool gemm_pays(int N, int K, int R) {
    const int tiles = (N + 15) / 16, P = gemv_num_parts(N, K / 256);
    if (R <= 48 || P <= 0) return false;
    const int nbp = K / 256 / P, cb = nbp % 2 == 0 ? 2 : 1, gc = GEMV_NCTA / P, cu = (tiles + gc - 1) / gc * (nbp / cb), per_warp = (cu + GEMV_WARPS - 1) / GEMV_WARPS * cb;
    double gemv = 0;
    for (int r0 = 0; r0 < R; r0 += 32) gemv += 1.2 + 0.242 * nbp + 0.5165 * per_warp * (((R - r0 < 32 ? R - r0 : 32) + 7) / 8);
    int c, g; gemm_cut(N, K, R, &c, &g);
    const TcCost t = tc_cost(N, K, R, c, g);
    return 0.96 * (7.2 + 1.91 * t.items + 0.00712 * t.cost * nbp) < gemv;
}
int gemm_q4k_q8_cut(const void* Wt, const XQ8F& x, float* yparts, int N, int K, int R, int ldy, size_t part_stride, void* pack, int* err, cudaStream_t s, bool pdl, int ntc, int G) {
    HP_REQUIRE(K > 0 && K % 256 == 0, "gemm_q4k_q8: K=%d must be a positive multiple of 256", K);
    HP_REQUIRE(N > 0 && R >= 1 && ldy >= N, "gemm_q4k_q8: bad shape N=%d R=%d ldy=%d", N, R, ldy);
    HP_REQUIRE(pack && ((uintptr_t)pack & 15) == 0 && ((uintptr_t)Wt & 15) == 0, "gemm_q4k_q8: the pack buffer and the weights must be 16-byte aligned");
    HP_REQUIRE((G == 8 || G == 4) && ntc >= 4 && ntc <= 16 && ntc % 2 == 0, "gemm_q4k_q8: no cut of %d column tiles and %d weight tiles", ntc, G);
    TcArgs a; a.W = (const uint8_t*)Wt; a.xp = (const uint8_t*)pack; a.y = yparts;
    a.N = N; a.nb = K / 256; a.P = gemv_num_parts(N, a.nb); a.R = R; a.ldy = ldy; a.part_stride = part_stride; a.err = err;
    HP_REQUIRE(a.P > 0, "gemm_q4k_q8: K=%d is too large for the K-part partition", K);
    a.G = G; a.ngrp = ((N + 15) / 16 + G - 1) / G; a.ncg = ((R + 7) / 8 + ntc - 1) / ntc;
    const int items = a.ncg * a.ngrp * a.P, grid = items < GEMV_NCTA ? items : GEMV_NCTA;
    a.nlong = a.ncg - tc_narrow(R, ntc);
    a.heavy = a.nlong < a.ncg ? items % grid : 0; a.light = items / grid * (grid - a.heavy);
    switch (ntc) {
        case 4: return launch_tc<4>(a, x, grid, s, pdl);   case 6: return launch_tc<6>(a, x, grid, s, pdl);
        case 8: return launch_tc<8>(a, x, grid, s, pdl);   case 10: return launch_tc<10>(a, x, grid, s, pdl);
        case 12: return launch_tc<12>(a, x, grid, s, pdl); case 14: return launch_tc<14>(a, x, grid, s, pdl);
        default: return launch_tc<16>(a, x, grid, s, pdl);
    }
}
int gemm_q4k_q8_parts(const void* Wt, const XQ8F& x, float* yparts, int N, int K, int R, int ldy, size_t part_stride, void* pack, int* err, cudaStream_t s, bool pdl) {
    HP_REQUIRE(K > 0 && K % 256 == 0 && N > 0 && R >= 1 && gemv_num_parts(N, K / 256) > 0, "gemm_q4k_q8: bad shape N=%d K=%d R=%d", N, K, R);
    int ntc, G; gemm_cut(N, K, R, &ntc, &G);
    return gemm_q4k_q8_cut(Wt, x, yparts, N, K, R, ldy, part_stride, pack, err, s, pdl, ntc, G);
}

}  // namespace hp
