// Quantised matrix product on the 5th-generation tensor cores for any number of rows: Y[M, N] = T(X[M, K] . dequant(W)^T + residual)
// or the gated activation of gate/up pairs, 4-bit weights in the streaming layout (units of 16 rows x 8 groups, fk_stream.cuh).
//
// Arithmetic: one pass of kind::f16 (fp16 operands, fp32 accumulation in tensor memory), with operands that are exact within these limits.
//   * A weight is (q - 8) s + e, e = b + 8 s, after a power of two per weight row (k_row_factors: the larger of 1024 |s| and |e| lands in
//     [2^14, 2^15)).  A nibble in the low bits of 0x6400 is 1024 + q (published: arXiv
//     2211.10017; the upper nibble of a byte comes by 1/16), so one fused multiply-add gives (1024 + q) s + c; with c = -1032 s
//     rounded towards zero to fp16, c = -1032 s + d, the result (q - 8) s + d is a multiple of s's last place below 2^11 of them, hence exact,
//     and d (the same for all nibbles of a group: c + 960 s, the constant of nibbles 4 bits up, is exact too) is taken off e.
//     Scales down to 2^-18 of the row's largest are exact, smaller ones carry an error of 2^-23 of the row's largest weight.
//   * An activation is bf16: 8 bits, exact in fp16 after a power of two per row (k_stage_rows: the row's largest lands in [2^8, 2^9))
//     for everything down to 2^-25 of the row's largest, rounded to 2^-33 of it below.
//   * e enters as three extra k slots per group, (e_hi, e_hi, e_lo) . (X_hi, X_lo, X_hi), X the sum of the group's activations: 22 bits
//     of both, a fourth slot is zero.  A super-block of 8 groups is 8 k-blocks of 64 slots and one of 32.
// Scales inside the operand leave nothing to do per group after the product: accumulators stay in tensor memory until a tile is done.
//
// A block owns 256 weight rows (two M = 128 accumulators) x BN rows of X.  16 warps turn one unit each (16 weight rows) into fp16
// and write it straight into tensor memory as the A operand (tcgen05.st .16x256b: the lane layout of the units is its lane layout; a ring
// of four to seven k-blocks); through shared memory the expanded operand costs two more crossings of it than the packed weights.  One warp
// fetches X by TMA (128-byte swizzle), one warp per accumulator issues its MMAs, 8 warps store finished tiles.  Weight rings are filled before
// griddepcontrol.wait.  Waits: fk_tc.cuh; a storing warp gives up by itself, the four that store a tile by whole lines do together.
//
// Bound by the dequantising warps (a k-block and the latencies around it, 3.1 us a super-block, against 2.9 of MMAs) and by the store between tiles, under
// which the MMAs wait.  256 x 128 tiles therefore cross shared memory 16 rows of X at a time: a warp stores whole lines of one row, factors are per
// lane and not shuffled, eight activations are worked on side by side (one after the other they took 6.5 of 11.6 us a tile; a tile's columns are 3.5 us per 512).
// 1000 rows, 3584 -> 2 x 18944: 290 -> 243 us = 1.12 PFLOP/s, 3584 -> 4608 34.8 -> 33.0; 16 rows, 5120 -> 2 x 27648, 64.6 -> 62.4 us = 2.55 TB/s of
// weights (k_qmm4 98 us; 20 -> 22 us at 5120 -> 5120, where start-up counts).
//
// Sums are kept in tensor memory over at most 5120 columns (fkq_stretch); longer ones are added up in the scratch area by the warp that
// stores them.
//
// Work split: `whole` = tiles dealt whole in turn, else all (tile, super-block) steps dealt in equal runs; a run that covers part of a
// tile leaves fp32 sums in the scratch area, and of the warps that hold the same rows the last to arrive adds the parts in K order.  Or a cluster
// splits a tile, and its blocks add the parts up through distributed shared memory (fkq_cluster_plan).
#pragma once
#include "fk_stream.cuh"
#include "fk_layers.h"
#include "fk_qplan.h"
#include "fk_tc.cuh"
#include <cuda_fp16.h>

#define FKQ_SB 576                      // staged halves per super-block: 512 activations, 32 slots for the sums, 32 unused
#define FKQ_DEQ 16                      // dequantising warps: one unit each
#define FKQ_THREADS ((FKQ_DEQ + FKQ_EPI + 3) * 32)      // .. a warp for X, two for the MMAs
#define FKQ_MAX_K 32768                 // a row is staged from registers: 1024 threads x 4 vectors of 8
#define FKQ_ERR_WAIT 0x400000u
template <int BN> struct QgTile {
    static constexpr int XG = BN >= 128 ? 1 : 3, XS = BN == 64 ? 3 : 4, XBYTES = BN * 128;        // k-blocks per stage of X, stages, bytes of a k-block
    static constexpr int NBUF = BN <= 64 ? 2 : 1, DCOLS = NBUF * 2 * BN, AS = (512 - DCOLS) / 64;                 // accumulators of a tile and the next, columns, k-blocks of A operand
    static constexpr int BOX = BN >= 128 ? 2 * 16 * 128 * 4 : 0;                                                   // of a stored tile: 16 rows of X of each accumulator
    static constexpr size_t SMEM = 1024 + (size_t)XS * XG * XBYTES + (size_t)FKQ_DEQ * FK_STAGES * FK_UNIT_BYTES + BOX;
};

struct QGemmArgs { TiledW W; const float *xscale; const uint16_t *residual; uint16_t *y; float *scratch; unsigned int *counters; const float *rowmul; int m, n, ldr, act, whole, mtiles, tiles; uint32_t limit; uint16_t *tail; int from; };      // tail: plain rows of y from `from` on once more

// D += A B^T: A (128 rows, 16 halves) in tensor memory, B (the descriptor's rows) in shared memory; more = 0 overwrites D
__device__ __forceinline__ void qg_mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t more) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(more) : "memory");
}
__device__ __forceinline__ uint32_t h2_fma(uint32_t a, uint32_t b, uint32_t c) {
    __half2 r = __hfma2(*reinterpret_cast<__half2 *>(&a), *reinterpret_cast<__half2 *>(&b), *reinterpret_cast<__half2 *>(&c)); return *reinterpret_cast<uint32_t *>(&r);
}
// (w & MASK) | 0x64006400 in one instruction
template <uint32_t MASK> __device__ __forceinline__ uint32_t qg_nibbles(uint32_t w) {
    uint32_t r; asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(w), "n"(MASK), "r"(0x64006400u)); return r;
}
__device__ __forceinline__ uint32_t h2_mul(uint32_t a, uint32_t b) { __half2 r = __hmul2(*reinterpret_cast<__half2 *>(&a), *reinterpret_cast<__half2 *>(&b)); return *reinterpret_cast<uint32_t *>(&r); }
__device__ __forceinline__ uint32_t h2_both(uint32_t a, int high) {
    const __half2 v = *reinterpret_cast<__half2 *>(&a), r = high ? __high2half2(v) : __low2half2(v); return *reinterpret_cast<const uint32_t *>(&r);
}
__device__ __forceinline__ float2 h2_floats(uint32_t a) { return __half22float2(*reinterpret_cast<__half2 *>(&a)); }
__device__ __forceinline__ uint32_t h2_pack(float lo, float hi) { __half2 r = __floats2half2_rn(lo, hi); return *reinterpret_cast<uint32_t *>(&r); }
__device__ __forceinline__ void qg_st16(uint32_t addr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void qg_put16(uint32_t addr, const uint32_t (&d)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(addr), "r"(d[0]), "r"(d[1]), "r"(d[2]), "r"(d[3]), "r"(d[4]), "r"(d[5]), "r"(d[6]), "r"(d[7]),
                   "r"(d[8]), "r"(d[9]), "r"(d[10]), "r"(d[11]), "r"(d[12]), "r"(d[13]), "r"(d[14]), "r"(d[15]) : "memory");
}
__device__ __forceinline__ void qg_ld16(uint32_t (&d)[16], uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]),
                   "=r"(d[8]), "=r"(d[9]), "=r"(d[10]), "=r"(d[11]), "=r"(d[12]), "=r"(d[13]), "=r"(d[14]), "=r"(d[15]) : "r"(addr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// whether `v` holds in all of the 128 threads that meet at this barrier
__device__ __forceinline__ bool qg_all(int bar, bool v) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(r) : "r"((uint32_t)v), "r"(bar) : "memory");
    return r != 0;
}

// LONG: more than FKQ_SUM_STEPS super-blocks of columns.  CLUSTER: the blocks of a cluster split a tile's super-blocks; each leaves its sums in its
// own shared memory (the weight ring, read by then), and after a cluster barrier each adds up its share of the tile's rows of X, read from the others in
// part order.
template <int BN, bool GATEUP, bool LONG, bool CLUSTER>
__global__ void __launch_bounds__(FKQ_THREADS, 1) k_qgemm(FkState *st, const __grid_constant__ CUtensorMap mx, QGemmArgs a) {
    using T = QgTile<BN>;
    constexpr int XS = T::XS, XG = T::XG, NBUF = T::NBUF, AS = T::AS;
    constexpr bool SPLIT = !CLUSTER && BN <= FKQ_SPLIT_ROWS;        // tiles whose parts meet in memory
    constexpr bool LINES = !CLUSTER && T::BOX > 0;                  // .. that are stored by whole lines
    extern __shared__ unsigned char qg_smem[];
    __shared__ __align__(8) uint64_t bars[FKQ_DEQ * FK_STAGES + 2 * XS + 2 * AS + 2 * NBUF + 2];
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x, lane = tid & 31, wid = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t base = (smem_u32(qg_smem) + 1023u) & ~1023u, ring = base + XS * XG * T::XBYTES;
    const uint32_t wfull = smem_u32(bars), xfull = wfull + 8 * FKQ_DEQ * FK_STAGES, xempty = xfull + 8 * XS, afull = xempty + 8 * XS, aempty = afull + 8 * AS,
                   dfull = aempty + 8 * AS, dempty = dfull + 8 * NBUF, drained = dempty + 8 * NBUF;
    pdl_launch_dependents();
    if (tid == 0) {
        for (int i = 0; i < FKQ_DEQ * FK_STAGES; ++i) mbar_init(bars + i, 1);
        uint64_t *b = bars + FKQ_DEQ * FK_STAGES;
        for (int i = 0; i < XS; ++i) { mbar_init(b + i, 1); mbar_init(b + XS + i, 2); }
        b += 2 * XS;
        for (int i = 0; i < AS; ++i) { mbar_init(b + i, FKQ_DEQ); mbar_init(b + AS + i, 2); }
        b += 2 * AS;
        for (int i = 0; i < NBUF; ++i) { mbar_init(b + i, 2); mbar_init(b + NBUF + i, FKQ_EPI); }
        mbar_init(b + 2 * NBUF, 1); mbar_init(b + 2 * NBUF + 1, 1);
        mbar_fence_init();
    }
    if (wid == FKQ_DEQ) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot, tmem_a = tmem + T::DCOLS;      // accumulators, A operand
    const int nsb = a.W.nsb, G = gridDim.x, me = blockIdx.x;
    bool ok = true;
    QWork w;
    auto work = [&](int v, QWork &o) { return CLUSTER ? fkq_cluster_work(-a.whole, a.tiles, nsb, me, v, o) : fkq_work(a.whole, a.tiles, nsb, me, G, v, o); };
    if (wid < FKQ_DEQ) {
        // ---------------------------------------------------------------- weights: packed ring -> fp16 in tensor memory
        const int q = wid & 3, sub = wid >> 3, half = (wid >> 2) & 1, mine = sub * 8 + q * 2 + half;
        const uint32_t bar0 = wfull + 8 * FK_STAGES * wid, ring0 = ring + (uint32_t)(wid * FK_STAGES * FK_UNIT_BYTES);
        const uint32_t dst0 = tmem_a + ((uint32_t)(32 * q + 16 * half) << 16) + (uint32_t)(sub * 32);
        int iv = 0, left = 0, issued = 0, used = 0, as = 0, stages = 0;
        uint32_t aph = 1u, pend = 0;                    // a ring that was never used counts as free; pend: the barrier of what is not announced yet
        const uint4 *iu = nullptr;                      // the next unit of this warp in the block's order of steps, `left` of its piece still to come
        auto piece = [&]() {                            // tiles past the last row tile have none
            for (QWork iw; left == 0 && work(iv, iw); ++iv) {
                const int tile = (iw.tile / a.mtiles) * 16 + mine;
                if (tile < a.W.ntiles) { left = iw.k1 - iw.k0; iu = a.W.units + ((size_t)tile * nsb + iw.k0) * FK_UNIT_VEC; }
            }
        };
        auto issue = [&]() {
            if (left == 0) return;
            if (lane == 0) {
                const int s = issued & (FK_STAGES - 1);
                tc_expect(bar0 + 8 * s, FK_UNIT_BYTES);
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"(ring0 + (uint32_t)(s * FK_UNIT_BYTES)), "l"(iu), "r"((uint32_t)FK_UNIT_BYTES), "r"(bar0 + 8 * s) : "memory");
            }
            ++issued; iu += FK_UNIT_VEC;
            if (--left == 0) piece();
        };
        piece();
        for (int s = 0; s < FK_STAGES; ++s) issue();
        // A k-block is announced when the next one's values are worked out, and its slot is looked at before: both latencies pass under the
        // arithmetic
        auto announce = [&]() {
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0 && pend) tc_arrive(pend);
        };
        auto claim = [&](bool free) {                   // the slot `as` may be written; a wait that runs out gives the kernel up
            announce();
            if (!tc_all(free) && !tc_wait_warp(aempty + 8 * as, aph, a.limit)) ok = false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        };
        auto taken = [&]() { pend = afull + 8 * as; if (++as == AS) { as = 0; aph ^= 1u; } };
        for (int v = 0; ok && work(v, w); ++v) {
            const int tile = (w.tile / a.mtiles) * 16 + mine;
            const bool have = tile < a.W.ntiles;
            const float mul = have ? __ldg(a.rowmul + tile * 16 + (lane >> 2)) : 1.0f, mul8 = have ? __ldg(a.rowmul + tile * 16 + 8 + (lane >> 2)) : 1.0f;
            for (int kb = w.k0; kb < w.k1 && ok; ++kb) {
                const int s = used & (FK_STAGES - 1);
                if (have && !tc_wait_warp(bar0 + 8 * s, (uint32_t)(used / FK_STAGES) & 1u, a.limit)) { ok = false; break; }
                const uint32_t u = ring0 + (uint32_t)(s * FK_UNIT_BYTES + lane * 16);
                // scales and biases of rows g and g + 8, groups 2t and 2t + 1: s and c for the shuffles below, e for the sums' slots
                // (a warp without a unit works on what the ring holds: rows that nobody stores)
                const uint4 sb = lds128(u + 4096u);
                uint4 p = lds128(u);
                uint32_t sc[2], cc[2]; float e[4];      // rows g and g + 8: groups (2t, 2t + 1) in the halves; e of (g, 2t) (g, 2t + 1) (g + 8, 2t) (g + 8, 2t + 1)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t sw = i ? sb.y : sb.x, bw = i ? sb.w : sb.z;
                    const float f = i ? mul8 : mul, s0 = bf_lo(sw) * f, s1 = bf_hi(sw) * f;
                    sc[i] = h2_pack(s0, s1);
                    const float2 sh = h2_floats(sc[i]);
                    asm("cvt.rz.f16x2.f32 %0, %1, %2;" : "=r"(cc[i]) : "f"(-1032.0f * sh.y), "f"(-1032.0f * sh.x));
                    const float2 ch = h2_floats(cc[i]);
                    e[2 * i] = fmaf(8.0f, s0, bf_lo(bw) * f) - fmaf(1032.0f, sh.x, ch.x);
                    e[2 * i + 1] = fmaf(8.0f, s1, bf_hi(bw) * f) - fmaf(1032.0f, sh.y, ch.y);
                }
#pragma unroll 1
                for (int j = 0; j < 4; ++j) {           // groups 2j and 2j + 1
                    const int src = (lane & ~3) | j;
                    // s and c of both groups, and those of nibbles 4 bits up: (1024 + 16 q) s / 16 + c + 960 s
                    const uint32_t s2 = __shfl_sync(0xffffffffu, sc[0], src), c2 = __shfl_sync(0xffffffffu, cc[0], src);
                    const uint32_t s28 = __shfl_sync(0xffffffffu, sc[1], src), c28 = __shfl_sync(0xffffffffu, cc[1], src);
                    const uint32_t h2 = h2_mul(s2, 0x2C002C00u), h28 = h2_mul(s28, 0x2C002C00u), d2 = h2_fma(s2, 0x63806380u, c2), d28 = h2_fma(s28, 0x63806380u, c28);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint4 nx = lds128(u + (uint32_t)((2 * j + h + 1) * 512));      // after the last group: the scales, not used
                        const bool free = tc_look(aempty + 8 * as, aph);
                        // one group's in both halves: operand selectors of the multiply-adds, not instructions
                        const uint32_t sg = h2_both(s2, h), cg = h2_both(c2, h), hg = h2_both(h2, h), dg = h2_both(d2, h);
                        const uint32_t sg8 = h2_both(s28, h), cg8 = h2_both(c28, h), hg8 = h2_both(h28, h), dg8 = h2_both(d28, h);
                        uint32_t r[16];
                        auto expand = [&](uint32_t word, uint32_t s1, uint32_t c1, uint32_t s16, uint32_t c16, int i) {            // pairs (0,4) (1,5) | (2,6) (3,7)
                            const uint32_t hi = word >> 8;
                            r[i] = h2_fma(qg_nibbles<0x000F000Fu>(word), s1, c1); r[i + 1] = h2_fma(qg_nibbles<0x00F000F0u>(word), s16, c16);
                            r[i + 4] = h2_fma(qg_nibbles<0x000F000Fu>(hi), s1, c1); r[i + 5] = h2_fma(qg_nibbles<0x00F000F0u>(hi), s16, c16);
                        };
                        expand(p.x, sg, cg, hg, dg, 0); expand(p.z, sg8, cg8, hg8, dg8, 2); expand(p.y, sg, cg, hg, dg, 8); expand(p.w, sg8, cg8, hg8, dg8, 10);
                        claim(free);
                        qg_st16(dst0 + (uint32_t)(as * 64), r);
                        taken();
                        p = nx;
                    }
                    if (!ok) break;
                }
                if (!ok) break;
                stages += 9;
                {                                       // the sums' slots: columns 8b + 2t (e_hi, e_hi) and 8b + 2t + 1 (e_lo, 0) of group 2t + b
                    const bool free = tc_look(aempty + 8 * as, aph);
                    uint32_t r[8];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {       // e[i] is row g + 8 (i / 2), group 2t + (i & 1)
                        const uint32_t hh = h2_pack(e[i], e[i]);
                        r[(i & 1) * 4 + (i >> 1) * 2] = hh; r[(i & 1) * 4 + (i >> 1) * 2 + 1] = h2_pack(e[i] - h2_floats(hh).x, 0.0f);
                    }
                    if (have) { ++used; __syncwarp(); issue(); }        // the unit is in registers: its ring slot is refilled
                    claim(free);
                    asm volatile("tcgen05.st.sync.aligned.16x256b.x2.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                                 ::"r"(dst0 + (uint32_t)(as * 64)), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
                    taken();
                }
            }
            announce(); pend = 0;                       // the tile's last
        }
        // what is still in flight lands, and the MMAs that read the last stages have been counted, before the block may leave
        for (; used < issued; ++used) if (!tc_wait_warp(bar0 + 8 * (used & (FK_STAGES - 1)), (uint32_t)(used / FK_STAGES) & 1u, TC_DRAIN)) ok = false;
        if (ok) for (int j = stages > AS ? stages - AS : 0; j < stages; ++j) if (!tc_wait_warp(aempty + 8 * (j % AS), (uint32_t)(j / AS) & 1u, a.limit)) ok = false;
        if (!ok && lane == 0) atomicOr(&st->error, FKQ_ERR_WAIT);
    } else if (wid == FKQ_DEQ + FKQ_EPI) {
        // ---------------------------------------------------------------- X
        pdl_wait();
        if (lane == 0) {
            int it = 0;
            for (int v = 0; ok && work(v, w); ++v) {
                const int m0 = (w.tile % a.mtiles) * BN;
                for (int kb = w.k0 * 9; kb < w.k1 * 9; kb += XG, ++it) {
                    const int s = it % XS;
                    if (it >= XS && !tc_wait(xempty + 8 * s, (uint32_t)(it / XS - 1) & 1u, a.limit)) { ok = false; break; }
                    tc_expect(xfull + 8 * s, (uint32_t)(XG * T::XBYTES));
#pragma unroll
                    for (int g = 0; g < XG; ++g)
                        tc_load(base + (s * XG + g) * T::XBYTES, &mx, (kb + g) * 64, m0, xfull + 8 * s);
                }
            }
            for (int j = it > XS ? it - XS : 0; j < it; ++j) {      // landed and, unless a wait ran out, multiplied
                if (!tc_wait(xfull + 8 * (j % XS), (uint32_t)(j / XS) & 1u, TC_DRAIN)) ok = false;
                if (ok && !tc_wait(xempty + 8 * (j % XS), (uint32_t)(j / XS) & 1u, a.limit)) ok = false;
            }
            if (!ok) atomicOr(&st->error, FKQ_ERR_WAIT);
        }
    } else if (wid > FKQ_DEQ + FKQ_EPI) {
        // ---------------------------------------------------------------- MMA issue, a warp per accumulator: the warp stays together and one elected lane
        // issues, so that addresses and descriptors live in uniform registers (a branch on the lane costs moves into them before every
        // instruction: 84 cycles an MMA, 33 with the election); the next k-block's barriers are looked at while this one's MMAs go out,
        // and one warp's waits pass under the other's issue
        pdl_wait();
        const int sub = wid - (FKQ_DEQ + FKQ_EPI + 1);
        const uint32_t idesc = (1u << 4) | ((uint32_t)(BN >> 3) << 17) | ((128u >> 4) << 24);          // fp16 x fp16 -> fp32
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0), tma = tm + (uint32_t)(T::DCOLS + sub * 32);
        const uint64_t db0 = tc_desc(base);
        int s = 0, as = 0;
        uint32_t xph = 0, aph = 0;
        bool xready = false, aready = false;
        int sums = 0;                                   // handed to the storing warps so far
        for (int v = 0; ok && work(v, w); ++v)
        for (int c0 = w.k0, c1; ok && c0 < w.k1; c0 = c1, ++sums) {
            c1 = LONG ? fkq_stretch(w, c0) : w.k1;
            const int d = sums % NBUF;
            if (sums >= NBUF && !tc_wait_warp(dempty + 8 * d, (uint32_t)(sums / NBUF - 1) & 1u, a.limit)) { ok = false; break; }
            const uint32_t dd = tm + (uint32_t)((d * 2 + sub) * BN);
            uint32_t again = 0;                         // 0: the first MMA overwrites
            for (int sb = c0; sb < c1 && ok; ++sb)
#pragma unroll 1
                for (int kk = 0, g = 0; kk < 9; ++kk) {
                    if ((g == 0 && !xready && !tc_wait_warp(xfull + 8 * s, xph, a.limit)) || (!aready && !tc_wait_warp(afull + 8 * as, aph, a.limit))) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t db = db0 + (uint64_t)((s * XG + g) * (T::XBYTES >> 4));
                    const uint32_t aa = tma + (uint32_t)(as * 64), xs_bar = xempty + 8 * s, as_bar = aempty + 8 * as;
                    const bool last = ++g == XG;
                    bool xseen = xready;
                    if (last) { g = 0; if (++s == XS) { s = 0; xph ^= 1u; } xseen = tc_look(xfull + 8 * s, xph); }
                    if (++as == AS) { as = 0; aph ^= 1u; }
                    const bool aseen = tc_look(afull + 8 * as, aph);
                    if (tc_elect()) {
                        qg_mma(dd, aa, db, idesc, again);
                        qg_mma(dd, aa + 8, db + 2, idesc, 1u);
                        if (kk < 8) { qg_mma(dd, aa + 16, db + 4, idesc, 1u); qg_mma(dd, aa + 24, db + 6, idesc, 1u); }
                        tc_commit(as_bar);
                        if (last) tc_commit(xs_bar);
                    }
                    aready = tc_all(aseen);
                    if (last) xready = tc_all(xseen);
                    again = 1;
                }
            if (ok && tc_elect()) tc_commit(dfull + 8 * d);
            __syncwarp();
        }
        if (!tc_drain_mmas(drained + 8 * sub)) ok = false;      // before tensor memory is freed, also where the storing warps gave up
        if (!ok && lane == 0) atomicOr(&st->error, FKQ_ERR_WAIT);
    } else {
        // ---------------------------------------------------------------- finished tiles: lane = weight row, registers = rows of X
        pdl_wait();
        const int ew = wid - FKQ_DEQ, q = ew & 3, sub = ew >> 2, odd = lane & 1;
        // plain rows in pairs: neighbouring lanes trade so that each holds two weight rows of one row of X (even lanes the even one), and
        // loads and stores are 4 bytes wide
        const bool pairs = !GATEUP && !(a.n & 1) && !(a.ldr & 1) && !(((uintptr_t)a.y | (uintptr_t)a.residual | (uintptr_t)a.tail) & 3);
        // counts a part of a tile; true for the last one
        auto count = [&](int tile) {
            const unsigned int most = (unsigned int)fkq_parts(a.tiles, nsb, G, tile) - 1u;
            unsigned int ticket = 0;
            if (lane == 0) {
                unsigned int *word = a.counters + (size_t)tile * FKQ_EPI + ew;
                ticket = atomicAdd(word, 1u);
                if (ticket == most) *word = 0u;         // all parts are in: ready for the next launch
            }
            return __shfl_sync(0xffffffffu, ticket, 0) == most;
        };
        int sums = 0;                                   // taken over so far
        uint32_t src = 0;
        bool met = false;                               // CLUSTER: past the first barrier
        auto take = [&](int, const QWork &w) {
            const int rt = w.tile / a.mtiles, m0 = (w.tile - rt * a.mtiles) * BN, row0 = rt * FKQ_ROWS + sub * 128 + q * 32, n = row0 + lane;
            const bool part = SPLIT && fkq_part(w, nsb);      // whose sums go to memory
            const int rows = min(BN, a.m - m0);         // of X that there are
            uint32_t res[16];                           // residual pairs of 32 rows of X on their way
            auto fetch = [&](int c, auto &r) {
                constexpr int N2 = sizeof(r) / 4;
#pragma unroll
                for (int i = 0; i < N2; ++i)
                    r[i] = pairs && a.residual && n - odd < a.n && c + 2 * i + odd < rows ? __ldcg(reinterpret_cast<const uint32_t *>(a.residual + (size_t)(m0 + c + 2 * i + odd) * a.ldr + n - odd)) : 0u;
            };
            float fac[(BN + 31) / 32];                  // lane -> factor of row lane, + 32 ..
#pragma unroll
            for (int i = 0; i < (BN + 31) / 32; ++i) fac[i] = 32 * i + lane < rows ? __ldcg(a.xscale + m0 + 32 * i + lane) : 0.0f;
            auto factors = [&](int c) {                 // of the 32 rows around row c
                float f = fac[0];
#pragma unroll
                for (int i = 1; i < (BN + 31) / 32; ++i) if (c >= 32 * i) f = fac[i];
                return f;
            };
            const float rmul = row0 + lane < a.W.ntiles * 16 ? __uint_as_float(0x7F000000u - __float_as_uint(__ldg(a.rowmul + row0 + lane))) : 0.0f;       // 2^-k of 2^k
            // LINES: the four weight rows (gate/up: two gate rows and their up rows) that this lane stores of every row of X
            const int first = rt * FKQ_ROWS + sub * 128, four = GATEUP ? first + (lane >> 2) * 16 + (lane & 3) * 2 : first + 4 * lane;
            float rm[4];
            uint2 rs[4];                                // residuals of this warp's next four rows of X on their way
            const bool quads = !GATEUP && !((a.n | a.ldr) & 3) && !(((uintptr_t)a.y | (uintptr_t)a.residual | (uintptr_t)a.tail) & 7);
            auto coming = [&](int m) {
                return quads && a.residual && four < a.n && m < rows ? __ldcg(reinterpret_cast<const uint2 *>(a.residual + (size_t)(m0 + m) * a.ldr + four)) : make_uint2(0, 0);
            };
            if constexpr (LINES) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int r = GATEUP ? four + (i & 1) + (i >> 1) * 8 : four + i;
                    rm[i] = r < a.W.ntiles * 16 ? __uint_as_float(0x7F000000u - __float_as_uint(__ldg(a.rowmul + r))) : 0.0f;
                }
            }
            auto begin = [&]() {
                if constexpr (!GATEUP && LINES)
#pragma unroll
                    for (int i = 0; i < 4; ++i) rs[i] = coming(q + 4 * i);
            };
            // rows c + q, + 4 .. of X from the box, worked on side by side: a warp stores 128 neighbouring results of a row (64 of gate/up)
            auto lines = [&](int c, const float *box) {
                const float fc = factors(c);
                float v[4][4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float f = __shfl_sync(0xffffffffu, fc, (c + 4 * k + q) & 31), *row = box + (4 * k + q) * 128;
                    if constexpr (GATEUP) {
                        const float2 g2 = *reinterpret_cast<const float2 *>(row + 2 * lane), u2 = *reinterpret_cast<const float2 *>(row + 64 + ((2 * lane) ^ 16));
                        v[k][0] = g2.x; v[k][1] = g2.y; v[k][2] = u2.x; v[k][3] = u2.y;
                    } else {
                        const float4 v4 = *reinterpret_cast<const float4 *>(row + 4 * lane);
                        v[k][0] = v4.x; v[k][1] = v4.y; v[k][2] = v4.z; v[k][3] = v4.w;
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[k][i] = v[k][i] * fminf(f, rm[i]) * fmaxf(f, rm[i]);
                }
                if constexpr (GATEUP) {
                    const int out = (first >> 1) + 2 * lane;
                    uint16_t o[8];
                    const float g[8] = {v[0][0], v[0][1], v[1][0], v[1][1], v[2][0], v[2][1], v[3][0], v[3][1]};
                    const float u[8] = {v[0][2], v[0][3], v[1][2], v[1][3], v[2][2], v[2][3], v[3][2], v[3][3]};
                    s_act(a.act, g, u, o);
                    uint16_t *y = a.y + (size_t)(m0 + c + q) * a.n + out;
                    if (!(a.n & 1) && !((uintptr_t)a.y & 3)) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) if (out < a.n && c + 4 * k + q < rows) *reinterpret_cast<uint32_t *>(y + (size_t)(4 * k) * a.n) = (uint32_t)o[2 * k] | ((uint32_t)o[2 * k + 1] << 16);
                    } else {
#pragma unroll
                        for (int k = 0; k < 8; ++k) if (out + (k & 1) < a.n && c + 4 * (k >> 1) + q < rows) y[(size_t)(4 * (k >> 1)) * a.n + (k & 1)] = o[k];
                    }
                } else if (quads) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int m = c + 4 * k + q;
                        const size_t at = (size_t)(m0 + m) * a.n + four;
                        const uint2 o = make_uint2((uint32_t)f2bf(v[k][0] + bf_lo(rs[k].x)) | ((uint32_t)f2bf(v[k][1] + bf_hi(rs[k].x)) << 16),
                                                   (uint32_t)f2bf(v[k][2] + bf_lo(rs[k].y)) | ((uint32_t)f2bf(v[k][3] + bf_hi(rs[k].y)) << 16));
                        if (four < a.n && m < rows) {
                            *reinterpret_cast<uint2 *>(a.y + at) = o;
                            if (a.tail && m0 + m >= a.from) *reinterpret_cast<uint2 *>(a.tail + at - (size_t)a.from * a.n) = o;
                        }
                        rs[k] = coming(m + 16);
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int m = c + 4 * k + q;
                        const size_t at = (size_t)(m0 + m) * a.n + four;
#pragma unroll
                        for (int i = 0; i < 4; ++i) if (four + i < a.n && m < rows) {
                            const uint16_t o = f2bf(v[k][i] + (a.residual ? bf2f(__ldcg(a.residual + (size_t)(m0 + m) * a.ldr + four + i)) : 0.0f));
                            a.y[at + i] = o;
                            if (a.tail && m0 + m >= a.from) a.tail[at + i - (size_t)a.from * a.n] = o;
                        }
                    }
                }
            };
            // waits for the next sums in tensor memory
            auto next = [&]() {
                const int d = sums % NBUF;
                if (!tc_wait_warp(dfull + 8 * d, (uint32_t)(sums / NBUF) & 1u, a.limit)) return false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                src = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)((d * 2 + sub) * BN);
                return true;
            };
            auto taken = [&]() {                        // they are read: the MMAs may go on
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) tc_arrive(dempty + 8 * (sums % NBUF));
                ++sums;
            };
            // Parts of tiles and stretches that others follow leave their sums in the scratch area, added to those of the stretches before; a tile's last
            // stretch adds those to its own in tensor memory.  Sums that are added are requested 16 columns ahead.
            const bool long_sum = LONG && fkq_stretch(w, w.k0) < w.k1;
            bool good = true;
            for (int c0 = w.k0, c1;; c0 = c1) {
                c1 = LONG ? fkq_stretch(w, c0) : w.k1;
                const bool last = !LONG || c1 == w.k1, add = LONG && c0 > w.k0;
                if constexpr (!CLUSTER) { if (!part && !long_sum) { if constexpr (LINES) begin(); else if (!GATEUP) fetch(0, res); } }      // under the MMAs
                if (!next()) { if constexpr (LINES) { good = false; break; } else return false; }
                if constexpr (SPLIT || LONG) if (part || long_sum) {
                    float *mine = a.scratch + (size_t)(a.whole ? me : fkq_slot(a.tiles, nsb, G, me, w.tile)) * fkq_part_floats(BN) + sub * 128 + q * 32 + lane;
                    float p[16];
                    auto before = [&](int c) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) p[i] = add && c < rows ? __ldcg(mine + (size_t)(c + i) * FKQ_ROWS) : 0.0f;
                    };
                    before(0);
#pragma unroll 1
                    for (int c = 0; c < rows; c += 16) {
                        uint32_t r[16]; qg_ld16(r, src + (uint32_t)c);
#pragma unroll
                        for (int i = 0; i < 16; ++i) if (add) r[i] = __float_as_uint(__uint_as_float(r[i]) + p[i]);
                        before(c + 16);
                        if (last && !part) { qg_put16(src + (uint32_t)c, r); continue; }
#pragma unroll
                        for (int i = 0; i < 16; ++i) __stcg(mine + (size_t)(c + i) * FKQ_ROWS, __uint_as_float(r[i]));
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                }
                if (last && !part && long_sum) { if constexpr (LINES) begin(); else if (!GATEUP) fetch(0, res); }
                if (last) break;
                taken();
            }
            // rows c .. of X, whose factors lanes f0 .. hold; r: their residual pairs
            auto store = [&](int c, int f0, float factor, auto &acc, const uint32_t *r) {
                constexpr int NM = sizeof(acc) / 4;
#pragma unroll
                for (int i = 0; i < NM; ++i) {          // the smaller power of two first: no overflow on the way to a result in range
                    const float f = __shfl_sync(0xffffffffu, factor, f0 + i);
                    acc[i] = acc[i] * fminf(f, rmul) * fmaxf(f, rmul);
                }
                if (GATEUP) {
                    // lanes 0-7 / 16-23 hold gate rows, 8-15 / 24-31 the up rows of the same outputs: the lower half takes the even row of X of a
                    // pair, the upper half the odd one
                    const bool up = lane & 8;
                    const int out = (row0 >> 4) * 8 + (lane >> 4) * 8 + (lane & 7);
                    float gate[NM / 2], upv[NM / 2];
                    uint16_t o[NM / 2];
#pragma unroll
                    for (int i = 0; i < NM; i += 2) {
                        const float other = __shfl_xor_sync(0xffffffffu, up ? acc[i] : acc[i + 1], 8);
                        gate[i >> 1] = up ? other : acc[i]; upv[i >> 1] = up ? acc[i + 1] : other;
                    }
                    s_act(a.act, gate, upv, o);
#pragma unroll
                    for (int i = 0; i < NM; i += 2) {
                        const int m = c + i + (up ? 1 : 0);
                        if (m < rows && out < a.n) a.y[(size_t)(m0 + m) * a.n + out] = o[i >> 1];
                    }
                } else if (pairs) {
#pragma unroll
                    for (int i = 0; i < NM; i += 2) {
                        const float other = __shfl_xor_sync(0xffffffffu, odd ? acc[i] : acc[i + 1], 1);
                        const float lo = (odd ? other : acc[i]) + bf_lo(r[i >> 1]), hi = (odd ? acc[i + 1] : other) + bf_hi(r[i >> 1]);
                        const int m = c + i + odd;
                        if (m < rows && n - odd < a.n) {
                            const uint32_t v = (uint32_t)f2bf(lo) | ((uint32_t)f2bf(hi) << 16);
                            *reinterpret_cast<uint32_t *>(a.y + (size_t)(m0 + m) * a.n + n - odd) = v;
                            if (a.tail && m0 + m >= a.from) *reinterpret_cast<uint32_t *>(a.tail + (size_t)(m0 + m - a.from) * a.n + n - odd) = v;
                        }
                    }
                } else if (n < a.n) {
#pragma unroll
                    for (int i = 0; i < NM; ++i) if (c + i < rows) {
                        const float add = a.residual ? bf2f(__ldcg(a.residual + (size_t)(m0 + c + i) * a.ldr + n)) : 0.0f;
                        const uint16_t v = f2bf(acc[i] + add);
                        a.y[(size_t)(m0 + c + i) * a.n + n] = v;
                        if (a.tail && m0 + c + i >= a.from) a.tail[(size_t)(m0 + c + i - a.from) * a.n + n] = v;
                    }
                }
                __syncwarp();
            };
            if constexpr (CLUSTER) {
                const int S = -a.whole, mine = me % S;
                const uint32_t at = ring + (uint32_t)(sub * 128 + q * 32 + lane) * 4u;
#pragma unroll 1
                for (int c = 0; c < BN; c += 16) {      // every column: the others read them without asking how many count
                    uint32_t r[16]; qg_ld16(r, src + (uint32_t)c);
#pragma unroll
                    for (int i = 0; i < 16; ++i) asm volatile("st.shared.u32 [%0], %1;" ::"r"(at + (uint32_t)((c + i) * FKQ_ROWS * 4)), "r"(r[i]) : "memory");
                }
                __syncwarp();
                tc_cluster_sync(); met = true;
                constexpr int CS = BN >= 64 ? 8 : BN == 32 ? 4 : 2;
                const int last = (mine + 1) * (BN / S);
#pragma unroll 1
                for (int c = mine * (BN / S); c < last && c < rows; c += CS) {
                    uint32_t r2[CS / 2];
                    if (!GATEUP) fetch(c, r2);
                    float acc[CS];
#pragma unroll
                    for (int i = 0; i < CS; ++i) acc[i] = 0.0f;
#pragma unroll 1
                    for (int p = 0; p < S; p += 2) {    // in K order, two parts on their way
                        float u[2][CS];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const uint32_t from = tc_remote(at, (uint32_t)(p + h)) + (uint32_t)(c * FKQ_ROWS * 4);
#pragma unroll
                            for (int i = 0; i < CS; ++i) asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(u[h][i]) : "r"(from + (uint32_t)(i * FKQ_ROWS * 4)) : "memory");
                        }
#pragma unroll
                        for (int h = 0; h < 2; ++h)
#pragma unroll
                            for (int i = 0; i < CS; ++i) acc[i] += u[h][i];
                    }
                    store(c, c & 31, factors(c), acc, r2);
                }
            } else if constexpr (LINES) {
                if (!qg_all(1 + sub, good)) return false;              // the four warps of an accumulator meet below: all of them or none
                // 16 rows of X at a time cross shared memory, gate rows before up rows, those 16 banks on
                float *box = reinterpret_cast<float *>(qg_smem + (ring + (uint32_t)(FKQ_DEQ * FK_STAGES * FK_UNIT_BYTES) - smem_u32(qg_smem))) + sub * 2048;
                const int t = q * 32 + lane, up = (t >> 3) & 1, at = GATEUP ? up * 64 + (((t >> 4) * 8 + (t & 7)) ^ (up * 16)) : t;
#pragma unroll 1
                for (int c = 0; c < rows; c += 16) {
                    uint32_t r[16]; qg_ld16(r, src + (uint32_t)c);
                    asm volatile("bar.sync %0, 128;" ::"r"(1 + sub) : "memory");      // the 16 rows before are read
#pragma unroll
                    for (int i = 0; i < 16; ++i) box[i * 128 + at] = __uint_as_float(r[i]);
                    asm volatile("bar.sync %0, 128;" ::"r"(1 + sub) : "memory");
                    lines(c, box);
                }
            } else if (!part) {
#pragma unroll 1
                for (int cc = 0; cc < rows; cc += 32) {
                    const float f = factors(cc);
#pragma unroll
                    for (int h = 0; h < (BN > 16 ? 2 : 1); ++h) {
                        const int c = cc + 16 * h;
                        uint32_t r[16]; qg_ld16(r, src + (uint32_t)c);
                        float acc[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i) acc[i] = __uint_as_float(r[i]);
                        store(c, 16 * h, f, acc, res + 8 * h);
                        if (!GATEUP) {
                            uint32_t nx[8]; fetch(c + 32, nx);
#pragma unroll
                            for (int i = 0; i < 8; ++i) res[8 * h + i] = nx[i];
                        }
                    }
                }
            } else if constexpr (SPLIT) {
                const int first = fkq_owner(a.tiles, nsb, G, w.tile * nsb), last = first + fkq_parts(a.tiles, nsb, G, w.tile) - 1;
                __threadfence();
                __syncwarp();
                if (count(w.tile)) {
                    __threadfence();
                    const float *from = a.scratch + sub * 128 + q * 32 + lane;
#pragma unroll 1
                    for (int c = 0; c < rows; c += 8) {
                        uint32_t r8[4];
                        if (!GATEUP) fetch(c, r8);
                        float acc[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) acc[i] = 0.0f;
#pragma unroll 1
                        for (int p = first; p <= last; p += 3) {          // in K order, three parts on their way
                            float u[3][8];
#pragma unroll
                            for (int h = 0; h < 3; ++h) {
                                const float *f = from + (size_t)fkq_slot(a.tiles, nsb, G, min(p + h, last), w.tile) * fkq_part_floats(BN) + (size_t)c * FKQ_ROWS;
#pragma unroll
                                for (int i = 0; i < 8; ++i) u[h][i] = __ldcg(f + (size_t)i * FKQ_ROWS);
                            }
#pragma unroll
                            for (int h = 0; h < 3; ++h)
#pragma unroll
                                for (int i = 0; i < 8; ++i) if (p + h <= last) acc[i] += u[h][i];
                        }
                        store(c, c & 31, factors(c), acc, r8);
                    }
                }
            }
            taken();
            return true;
        };
        if constexpr (CLUSTER) ok = !work(0, w) || take(0, w);
        else ok = fkq_pieces(a.whole, a.tiles, nsb, me, G, take, [&](const QWork &w) { if constexpr (SPLIT) count(w.tile); });
        if (CLUSTER && !met) tc_cluster_sync();         // gave up: the others are not kept waiting
        if (!ok && lane == 0) atomicOr(&st->error, FKQ_ERR_WAIT);
    }
    if (CLUSTER) {
        __syncwarp();
        if (wid < FKQ_DEQ || wid >= FKQ_DEQ + FKQ_EPI) tc_cluster_sync();
        tc_cluster_sync();                              // nobody leaves while its sums are read
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (wid == FKQ_DEQ) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

// The power of two of every weight row (in the order of the units): what brings the larger of 1024 |s| and |b + 8 s| over the row into
// [2^14, 2^15); values that are not finite do not count.  Once per weight, when it is laid out; a warp per unit row of 16.
__global__ void __launch_bounds__(256) k_row_factors(const uint4 *units, float *mul, int ntiles, int nsb) {
    const int tile = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (tile >= ntiles) return;
    float top[2] = {0.0f, 0.0f};
    for (int i = 0; i < nsb; ++i) {
        const uint4 v = units[((size_t)tile * nsb + i) * FK_UNIT_VEC + 256 + lane];
        const uint32_t s[2] = {v.x, v.y}, b[2] = {v.z, v.w};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            // a 1024th of both, which is finite wherever s and b are
            const float t = 0.0009765625f, c[4] = {fabsf(bf_lo(s[h])), fabsf(bf_hi(s[h])), fabsf(fmaf(8.0f * t, bf_lo(s[h]), t * bf_lo(b[h]))), fabsf(fmaf(8.0f * t, bf_hi(s[h]), t * bf_hi(b[h])))};
#pragma unroll
            for (int j = 0; j < 4; ++j) if (c[j] < INFINITY) top[h] = fmaxf(top[h], c[j]);
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        top[h] = fmaxf(top[h], __shfl_xor_sync(0xffffffffu, top[h], 1)); top[h] = fmaxf(top[h], __shfl_xor_sync(0xffffffffu, top[h], 2));
        int e = top[h] > 0.0f ? (int)(__float_as_uint(top[h]) >> 23) - 117 : 14;
        e = e < -110 ? -110 : e;                        // factor and inverse stay normal numbers
        if ((lane & 3) == 0) mul[tile * 16 + h * 8 + (lane >> 2)] = __uint_as_float((uint32_t)(127 + 14 - e) << 23);
    }
}

// Rows of X as the product reads them: fp16 scaled by a power of two per row, in the k order in which the nibble pairs come out of
// their words (slot 16 b + 4 t + 2 h + e of a group is k = 32 (b / 2) + 8 t + 2 (b & 1) + h + 4 e), the group sums after every 8 groups;
// optionally normalised first (the two roundings of the one-row kernels).  A block per row, the row in registers: bound by the
// latency of one pass over it.
struct StageRowsArgs { const uint16_t *x, *w; __half *out; float *scale; int k, nsb; float eps; };
template <int NT>
__global__ void __launch_bounds__(NT) k_stage_rows(const FkState *st, StageRowsArgs a) {
    __shared__ float red[40];
    const int tid = threadIdx.x, row = blockIdx.x, chunks = a.nsb * 64;
    constexpr int NV = 4;
    uint4 x[NV];
    pdl_wait(); pdl_launch_dependents();
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const int c = v * NT + tid;
        x[v] = c * 8 < a.k ? __ldcg(reinterpret_cast<const uint4 *>(a.x + (size_t)row * a.k) + c) : make_uint4(0, 0, 0, 0);
    }
    if (a.w) {
        float ss = 0.0f;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            float f[8]; unpack8(x[v], f);
#pragma unroll
            for (int j = 0; j < 8; ++j) ss = fmaf(f[j], f[j], ss);
        }
        const float r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(block_sum(ss, red), (float)a.k), a.eps)));
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const int c = v * NT + tid;
            if (c * 8 >= a.k) continue;
            const uint4 wv = __ldg(reinterpret_cast<const uint4 *>(a.w) + c);
            float f[8], n[8]; unpack8(x[v], f); unpack8(wv, n);
            uint32_t o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) o[j] = (uint32_t)f2bf(n[2 * j] * rT(f[2 * j] * r)) | ((uint32_t)f2bf(n[2 * j + 1] * rT(f[2 * j + 1] * r)) << 16);
            x[v] = make_uint4(o[0], o[1], o[2], o[3]);
        }
    }
    uint32_t top = 0;                                   // largest magnitude as bf16 bits; infinities and NaN do not set the scale
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const uint32_t h[4] = {x[v].x, x[v].y, x[v].z, x[v].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t lo = h[j] & 0x7fffu, hi = (h[j] >> 16) & 0x7fffu;
            if (lo < 0x7f80u && lo > top) top = lo;
            if (hi < 0x7f80u && hi > top) top = hi;
        }
    }
    top = __reduce_max_sync(0xffffffffu, top);
    __syncthreads();
    if ((tid & 31) == 0) red[tid >> 5] = __uint_as_float(top);
    __syncthreads();
    top = 0;
#pragma unroll
    for (int i = 0; i < NT / 32; ++i) top = max(top, __float_as_uint(red[i]));
    int e = top ? (int)(top >> 7) - 127 : 8;
    if (e < -118) e = -118;                             // the factor and its inverse stay normal numbers
    const float mul = __uint_as_float((uint32_t)(127 + 8 - e) << 23);
    if (tid == 0) a.scale[row] = __uint_as_float((uint32_t)(127 - 8 + e) << 23);
    __half *out = a.out + (size_t)row * a.nsb * FKQ_SB;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const int c = v * NT + tid;
        if (c >= chunks) break;                         // chunks is a multiple of 64: uniform over a warp
        float f[8]; unpack8(x[v], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] *= mul;
        float sum = ((f[0] + f[1]) + (f[2] + f[3])) + ((f[4] + f[5]) + (f[6] + f[7]));
        sum += __shfl_xor_sync(0xffffffffu, sum, 1); sum += __shfl_xor_sync(0xffffffffu, sum, 2); sum += __shfl_xor_sync(0xffffffffu, sum, 4);
        const int cc = c & 63, j = cc >> 3, b = (cc >> 2) & 1, t = cc & 3;
        __half *block = out + (size_t)(c >> 6) * FKQ_SB, *dst = block + j * 64 + 32 * b + 4 * t;
        *reinterpret_cast<uint2 *>(dst) = make_uint2(h2_pack(f[0], f[4]), h2_pack(f[1], f[5]));
        *reinterpret_cast<uint2 *>(dst + 16) = make_uint2(h2_pack(f[2], f[6]), h2_pack(f[3], f[7]));
        if ((cc & 7) == 0) {
            const float hi = __half2float(__float2half_rn(sum));
            *reinterpret_cast<uint2 *>(block + 512 + 16 * (j & 1) + 4 * (j >> 1)) = make_uint2(h2_pack(hi, sum - hi), h2_pack(hi, 0.0f));
        }
    }
}

// ---------------------------------------------------------------- the other kernels of a prompt
struct EmbedPromptArgs { const uint16_t *table; uint16_t *x; const uint32_t *tokens; int h, vocab; uint16_t *tail; int from; };
__global__ void __launch_bounds__(256) k_embed_prompt(FkState *st, EmbedPromptArgs a) {        // rows of h (a multiple of 8) values
    pdl_wait(); pdl_launch_dependents();
    uint32_t tok = __ldcg(a.tokens + blockIdx.x);
    if (tok >= (uint32_t)a.vocab) { if (threadIdx.x == 0) atomicOr(&st->error, FKL_ERR_TOKEN); tok = 0; }
    const uint4 *src = reinterpret_cast<const uint4 *>(a.table + (size_t)tok * a.h);
    uint4 *dst = reinterpret_cast<uint4 *>(a.x + (size_t)blockIdx.x * a.h);
    uint4 *tail = a.tail && (int)blockIdx.x >= a.from ? reinterpret_cast<uint4 *>(a.tail + (size_t)(blockIdx.x - a.from) * a.h) : nullptr;
    for (int i = threadIdx.x; i < a.h / 8; i += blockDim.x) { const uint4 v = __ldg(src + i); dst[i] = v; if (tail) tail[i] = v; }
}
// greedy token after every row, ties to the lowest index (v a multiple of 8)
__global__ void __launch_bounds__(512) k_argmax_prompt(const FkState *st, const uint16_t *logits, uint32_t *out, int v) {
    __shared__ unsigned long long best_of[16];
    pdl_wait(); pdl_launch_dependents();
    unsigned long long best = argmax_share(logits + (size_t)blockIdx.x * v, v, true);
    best = warp_max_u64(best);
    if ((threadIdx.x & 31) == 0) best_of[threadIdx.x >> 5] = best;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < (int)(blockDim.x >> 5); ++i) best = best_of[i] > best ? best_of[i] : best;
        out[blockIdx.x] = 0xffffffffu - (uint32_t)(best & 0xffffffffull);
    }
}
// RoPE and the cache store of consecutive positions: a block takes a position, works out its angles once for all heads (rope_pair's
// arithmetic) and moves 4 bytes a thread.  Positions past the capacity are an error, and
// nothing is stored.  (A block per head and position, each with its own sine and cosine, took 39 us for 1000 positions
// of the 7B shape: 36000 blocks of 64 threads.)
__global__ void __launch_bounds__(256) k_rope_store_prompt(FkState *st, RopeRowsArgs a) {
    __shared__ float2 turn[256];
    const int m = blockIdx.x, half = a.hd >> 1, quads = half >> 1;       // pairs of dimensions a thread turns together
    pdl_wait(); pdl_launch_dependents();
    const uint32_t pos = st->offset + (uint32_t)m;
    if (a.rows > a.capacity || st->offset > (uint32_t)(a.capacity - a.rows)) {      // two blocks might store one row, and k_flash_rows does not wrap
        if (m == 0 && threadIdx.x == 0) atomicOr(&st->error, FKL_ERR_CAPACITY);
        return;
    }
    for (int d = threadIdx.x; d < half; d += blockDim.x) {
        const float e = __fmul_rn(-__fdiv_rn((float)d, (float)half), a.log2theta), ang = __fmul_rn((float)pos, exp2f(e));
        float s, c; sincosf(ang, &s, &c);
        turn[d] = make_float2(c, s);
    }
    __syncthreads();
    const uint16_t *row = a.qkv + (size_t)m * (a.n_q + 2 * a.n_kv) * a.hd;
    for (int i = threadIdx.x; i < (a.n_q + 2 * a.n_kv) * quads; i += blockDim.x) {
        const int head = i / quads, d = (i - head * quads) * 2;
        uint32_t lo = __ldcg(reinterpret_cast<const uint32_t *>(row + head * a.hd + d)), hi = __ldcg(reinterpret_cast<const uint32_t *>(row + head * a.hd + d + half));
        if (head < a.n_q + a.n_kv) {
            const float2 t0 = turn[d], t1 = turn[d + 1];
            const uint32_t o0 = (uint32_t)f2bf(__fsub_rn(__fmul_rn(bf_lo(lo), t0.x), __fmul_rn(bf_lo(hi), t0.y))) | ((uint32_t)f2bf(__fsub_rn(__fmul_rn(bf_hi(lo), t1.x), __fmul_rn(bf_hi(hi), t1.y))) << 16);
            const uint32_t o1 = (uint32_t)f2bf(__fadd_rn(__fmul_rn(bf_lo(hi), t0.x), __fmul_rn(bf_lo(lo), t0.y))) | ((uint32_t)f2bf(__fadd_rn(__fmul_rn(bf_hi(hi), t1.x), __fmul_rn(bf_hi(lo), t1.y))) << 16);
            lo = o0; hi = o1;
        }
        uint16_t *dst = head < a.n_q ? a.q_out + ((size_t)m * a.n_q + head) * a.hd
                      : head < a.n_q + a.n_kv ? a.cache_k + ((size_t)(head - a.n_q) * a.capacity + pos) * a.hd : a.cache_v + ((size_t)(head - a.n_q - a.n_kv) * a.capacity + pos) * a.hd;
        *reinterpret_cast<uint32_t *>(dst + d) = lo; *reinterpret_cast<uint32_t *>(dst + d + half) = hi;
    }
}
