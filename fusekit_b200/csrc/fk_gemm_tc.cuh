// Matrix product on the 5th-generation tensor cores: Y[m, n] = act(sum_k X[m, k] W[row0 + n, k]), bf16 operands, fp32
// accumulation, optionally grouped by expert (the rows of X between offsets[e] and offsets[e + 1] use the weight rows e * N ..).
//
// Persistent, warp-specialised, one CTA per SM.  A tile is 128 rows of X by BN rows of W.  Warp 0 fetches K slices of 64 by
// TMA (128-byte swizzle) into a ring of shared-memory stages, one thread of warp 1 issues tcgen05.mma (cta_group::1, M = 128,
// N = BN, K = 16) into one of two accumulators in tensor memory, warps 4 .. 7 read finished accumulators back and store them
// while the next tile is being multiplied.  Rows past the end of a tile's range are multiplied and not stored (past the end of
// the tensor TMA delivers zeros).  Waits: fk_tc.cuh.
#pragma once
#include "fk_layers.cuh"
#include "fk_tc.cuh"

#define FKL_TC_BK 64
#define FKL_TC_THREADS 256
template <int BN> struct TcTile {
    static constexpr int STAGES = BN == 256 ? 4 : BN == 128 ? 6 : 8;
    static constexpr int A_BYTES = 128 * FKL_TC_BK * 2, B_BYTES = BN * FKL_TC_BK * 2, STAGE = A_BYTES + B_BYTES, COLS = 2 * BN;
    static constexpr size_t SMEM = (size_t)STAGES * STAGE + 1024;
};
struct TcGemmArgs { void *y; const int *offsets; int m, n, kblocks, row0, ldy, act, out_f32, experts; float scale; BlockCols b; uint32_t limit; };       // b: BLOCK form

template <int BN, bool BLOCK>
__global__ void __launch_bounds__(FKL_TC_THREADS, 1) k_gemm_tc(FkState *st, const __grid_constant__ CUtensorMap mx, const __grid_constant__ CUtensorMap mw, TcGemmArgs a) {
    using T = TcTile<BN>;
    constexpr int S = T::STAGES;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * S + 5];
    __shared__ uint32_t tmem_slot;
    __shared__ int first[FKL_MAX_EXPERTS + 1];          // grouped: first 128-row tile of every expert
    __shared__ int wsum[8];
    const int tid = threadIdx.x, lane = tid & 31, wid = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t base = (tc_smem(smem_raw) + 1023u) & ~1023u;
    const uint32_t full = tc_smem(bars), empty = full + 8 * S, afull = empty + 8 * S, aempty = afull + 16, drained = aempty + 16;
    pdl_launch_dependents();
    if (tid == 0) {
        for (int s = 0; s < S; ++s) { tc_init(full + 8 * s, 1); tc_init(empty + 8 * s, 1); }
        for (int s = 0; s < 2; ++s) { tc_init(afull + 8 * s, 1); tc_init(aempty + 8 * s, 4); }
        tc_init(drained, 1);
        tc_init_fence();
    }
    if (wid == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&tmem_slot)), "r"((uint32_t)T::COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pdl_wait();
    const int ntn = (a.n + BN - 1) / BN;
    int mtiles = (a.m + 127) / 128;
    if (a.offsets) {
        int carry = 0;
        for (int b = 0; b < a.experts; b += FKL_TC_THREADS) {
            const int e = b + tid, c = e < a.experts ? (a.offsets[e + 1] - a.offsets[e] + 127) / 128 : 0;
            int v = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += t; }
            if (lane == 31) wsum[wid] = v;
            __syncthreads();
            int before = carry, total = 0;
            for (int w = 0; w < 8; ++w) { if (w < wid) before += wsum[w]; total += wsum[w]; }
            if (e < a.experts) first[e] = before + v - c;
            carry += total;
            __syncthreads();
        }
        if (tid == 0) first[a.experts] = carry;
        mtiles = carry;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    const int total = mtiles * ntn;
    // tile -> first row of X, end of its rows, first weight row, first column: neighbours share the weight tile (plain) or the
    // rows of X (grouped, where an expert has few rows)
    auto place = [&](int t, int &m0, int &mend, int &wrow, int &n0) {
        if (!a.offsets) { const int nt = t / mtiles; m0 = (t - nt * mtiles) * 128; mend = a.m; n0 = nt * BN; wrow = a.row0 + n0; return; }
        const int mt = t / ntn; n0 = (t - mt * ntn) * BN;
        int lo = 0, hi = a.experts;                     // last expert whose first tile is <= mt
        while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (first[mid] <= mt) lo = mid; else hi = mid; }
        m0 = a.offsets[lo] + (mt - first[lo]) * 128; mend = a.offsets[lo + 1]; wrow = lo * a.n + n0;
    };
    bool ok = true;
    if (wid == 0) {
        if (lane == 0) {
            int it = 0;
            for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
                int m0, mend, wrow, n0; place(t, m0, mend, wrow, n0);
                for (int kb = 0; kb < a.kblocks; ++kb, ++it) {
                    const int s = it % S;
                    if (it >= S && !tc_wait(empty + 8 * s, (uint32_t)(it / S - 1) & 1u, a.limit)) { ok = false; break; }
                    tc_expect(full + 8 * s, (uint32_t)T::STAGE);
                    tc_load(base + s * T::STAGE, &mx, kb * FKL_TC_BK, m0, full + 8 * s);
                    tc_load(base + s * T::STAGE + T::A_BYTES, &mw, kb * FKL_TC_BK, wrow, full + 8 * s);
                }
            }
            // the last stages have landed and, unless a wait ran out, are multiplied before the block may leave
            for (int j = it > S ? it - S : 0; j < it; ++j) {
                if (!tc_wait(full + 8 * (j % S), (uint32_t)(j / S) & 1u, TC_DRAIN)) ok = false;
                if (ok && !tc_wait(empty + 8 * (j % S), (uint32_t)(j / S) & 1u, a.limit)) ok = false;
            }
            if (!ok) atomicOr(&st->error, FKL_ERR_TC_WAIT);
        }
    } else if (wid == 1) {
        // The warp stays together and one elected lane issues: addresses and descriptors live in uniform registers (behind a branch on the
        // lane every instruction waits for moves into them, 84 cycles an MMA where 33 do), and the next slice's barrier is looked at
        // while this one's MMAs go out.
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((128u >> 4) << 24);
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
        const uint64_t da0 = tc_desc(base), db0 = tc_desc(base + T::A_BYTES);
        int s = 0, j = 0;
        uint32_t ph = 0;
        bool ready = false;
        for (int t = blockIdx.x; t < total && ok; t += gridDim.x, ++j) {
            const int b = j & 1;
            if (j >= 2 && !tc_wait_warp(aempty + 8 * b, (uint32_t)(j / 2 - 1) & 1u, a.limit)) { ok = false; break; }
            const uint32_t d = tm + (uint32_t)(b * BN);
            for (int kb = 0; kb < a.kblocks; ++kb) {
                if (!ready && !tc_wait_warp(full + 8 * s, ph, a.limit)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t off = (uint64_t)(s * (T::STAGE >> 4)), da = da0 + off, db = db0 + off;
                const uint32_t bar = empty + 8 * s;
                if (++s == S) { s = 0; ph ^= 1u; }
                const bool seen = tc_look(full + 8 * s, ph);
                if (tc_elect()) {
#pragma unroll
                    for (int k = 0; k < FKL_TC_BK / 16; ++k)
                        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                                     ::"r"(d), "l"(da + (uint64_t)(k * 2)), "l"(db + (uint64_t)(k * 2)), "r"(idesc), "r"(kb | k) : "memory");
                    tc_commit(bar);
                    if (kb + 1 == a.kblocks) tc_commit(afull + 8 * b);
                }
                ready = tc_all(seen);
            }
        }
        if (!tc_drain_mmas(drained)) ok = false;        // before tensor memory is freed, also where the storing warps gave up
        if (!ok && lane == 0) atomicOr(&st->error, FKL_ERR_TC_WAIT);
    } else if (wid >= 4) {
        const int q = wid - 4;
        int j = 0;
        for (int t = blockIdx.x; t < total && ok; t += gridDim.x, ++j) {
            int m0, mend, wrow, n0; place(t, m0, mend, wrow, n0);
            const int b = j & 1, row = m0 + q * 32 + lane;
            if (!tc_wait_warp(afull + 8 * b, (uint32_t)(j / 2) & 1u, a.limit)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int c = 0; c < BN; c += 32) {
                __syncwarp();
                uint32_t d[32];
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                             : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]), "=r"(d[8]), "=r"(d[9]), "=r"(d[10]),
                               "=r"(d[11]), "=r"(d[12]), "=r"(d[13]), "=r"(d[14]), "=r"(d[15]), "=r"(d[16]), "=r"(d[17]), "=r"(d[18]), "=r"(d[19]), "=r"(d[20]), "=r"(d[21]),
                               "=r"(d[22]), "=r"(d[23]), "=r"(d[24]), "=r"(d[25]), "=r"(d[26]), "=r"(d[27]), "=r"(d[28]), "=r"(d[29]), "=r"(d[30]), "=r"(d[31])
                             : "r"(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * BN + c)));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                const int col = n0 + c;
                if (row >= mend || col >= a.n) continue;
                if (BLOCK && col >= a.b.exact) {            // 16 (gate, up) pairs
                    uint16_t *y = (uint16_t *)a.b.y3 + (size_t)row * a.b.ld3 + (col - a.b.exact) / 2;
                    float v[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] = clamped_glu(__uint_as_float(d[2 * i]), __uint_as_float(d[2 * i + 1]), a.b.limit);
                    if (col + 32 <= a.n) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) st4(y + 4 * i, make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]));
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i) if (col + 2 * i < a.n) y[i] = f2bf(v[i]);
                    }
                    continue;
                }
                if (BLOCK) {
                    if (col < a.b.silu) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) if (col + i < a.b.silu) d[i] = __float_as_uint(act_apply(__uint_as_float(d[i]), FKL_ACT_SILU));
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i) d[i] = __float_as_uint(act_apply(__uint_as_float(d[i]), a.act) * a.scale);
                }
                const bool whole = col + 32 <= a.n, exact = BLOCK && col >= a.b.plain;
                if (a.out_f32 || exact) {
                    const int ld = exact ? a.b.exact - a.b.plain : a.ldy;
                    float *y = exact ? a.b.y2 + (size_t)row * ld + col - a.b.plain : (float *)a.y + (size_t)row * ld + col;
                    if (whole && (ld & 3) == 0) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) reinterpret_cast<uint4 *>(y)[i] = make_uint4(d[4 * i], d[4 * i + 1], d[4 * i + 2], d[4 * i + 3]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i) if (col + i < a.n) y[i] = __uint_as_float(d[i]);
                    }
                } else {
                    uint16_t *y = (uint16_t *)a.y + (size_t)row * a.ldy + col;
                    if (whole && (a.ldy & 7) == 0) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            uint32_t w[4];
#pragma unroll
                            for (int p = 0; p < 4; ++p) {
                                const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(d[8 * i + 2 * p]), __uint_as_float(d[8 * i + 2 * p + 1]));
                                w[p] = *reinterpret_cast<const uint32_t *>(&h);
                            }
                            reinterpret_cast<uint4 *>(y)[i] = make_uint4(w[0], w[1], w[2], w[3]);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i) if (col + i < a.n) y[i] = f2bf(__uint_as_float(d[i]));
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc_arrive(aempty + 8 * b);
        }
        if (!ok && lane == 0) atomicOr(&st->error, FKL_ERR_TC_WAIT);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (wid == 2) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)T::COLS) : "memory");
}
