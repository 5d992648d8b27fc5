// Causal attention of M positions on the 5th-generation tensor cores (tcgen05, bf16 operands, fp32 accumulation in tensor memory): the form
// of k_flash_rows (fk_flash.cuh) for heads of 64 or 128 dimensions and enough positions.
//
// A block owns 128 positions and two *sides*: the two query/key maps of one head (same values), or two query heads of one kv head (same
// keys and values).  A side is four warps, a thread per position; both walk the keys 64 at a time.  One warp fetches queries, keys and values
// by TMA (128-byte swizzle, keys and values in rings of three tiles), one issues the MMAs:
//   S = Q K^T   both operands in shared memory, 64 columns of tensor memory a side; the next tile's are formed as soon as this one's are in
//               registers, while its softmax runs
//   O += P V    P goes into 64 columns of its own as two bf16 terms (hi + lo, 32 columns each) and is the A operand from tensor memory; V is
//               read as it lies (rows of keys), i.e. as an N-major operand
// (MMAs of different shapes need not finish in the order they are issued: nothing that one reads or writes is written by the other before
// the first has been waited for.)
// The softmax of a position needs no exchange: its thread reads the 64 scores, keeps maximum and sum, and rescales O (through tensor memory)
// only when some position of its warp has outgrown its maximum by 2^8: until then weights are up to 2^8, which costs them no digit.
// At the end each side scales its rows; of two maps every thread takes half of a row's values from both, combines them, and the halves of a
// row's sum of squares meet in shared memory.
//
// Bound by the special-function unit (an exponential per score: 16 a clock and SM) and about as much by the MMAs, whose value product runs twice
// for hi + lo.  Prompts, us, k_flash_rows before: fatulix-2048, 2048 positions (two maps of 64, values of 128) 9697 -> 7150; kakunex-5120, 1500 (window of
// 1024) 8521 -> 8279; the 7B shape, 1000, 20870 -> 20219; the 0.5B shape, 600, 4782 -> 4621.  Errors against 64 bits agree with k_flash_rows to seven digits,
// results on the wrong side of their bf16 rounding 0.27 -> 0.29 % (two maps, 2048 positions), 0.22 -> 0.24 % (128 x 128, 1000), 0.82 both (64 x 64 at 6000), 4.45 both (two maps at 60000).
// Waits: fk_tc.cuh (the eight softmax warps meet at two barriers of their own, which each of them reaches).
#pragma once
#include "fk_flash.cuh"
#include "fk_tc.cuh"

#define FT_THREADS 320
#define FT_RING 3
template <int KD, int VD> struct FtTile {
    static constexpr int Q_BYTES = 128 * KD * 2, K_BYTES = 64 * KD * 2, V_BYTES = 64 * VD * 2;      // of a side; of a map's tile of keys; of a tile of values
    __host__ __device__ static constexpr size_t smem(int maps) { return 1024 + 2 * (size_t)Q_BYTES + FT_RING * ((size_t)maps * K_BYTES + V_BYTES); }
};
__device__ __forceinline__ void ft_mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t more) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(more) : "memory");
}
__device__ __forceinline__ void ft_mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t more) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(more) : "memory");
}
__device__ __forceinline__ void ft_ld32(uint32_t *d, uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]), "=r"(d[8]), "=r"(d[9]), "=r"(d[10]),
                   "=r"(d[11]), "=r"(d[12]), "=r"(d[13]), "=r"(d[14]), "=r"(d[15]), "=r"(d[16]), "=r"(d[17]), "=r"(d[18]), "=r"(d[19]), "=r"(d[20]), "=r"(d[21]),
                   "=r"(d[22]), "=r"(d[23]), "=r"(d[24]), "=r"(d[25]), "=r"(d[26]), "=r"(d[27]), "=r"(d[28]), "=r"(d[29]), "=r"(d[30]), "=r"(d[31])
                 : "r"(addr) : "memory");
}
__device__ __forceinline__ void ft_st32(uint32_t addr, const uint32_t *d) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                 ::"r"(addr), "r"(d[0]), "r"(d[1]), "r"(d[2]), "r"(d[3]), "r"(d[4]), "r"(d[5]), "r"(d[6]), "r"(d[7]), "r"(d[8]), "r"(d[9]), "r"(d[10]),
                   "r"(d[11]), "r"(d[12]), "r"(d[13]), "r"(d[14]), "r"(d[15]), "r"(d[16]), "r"(d[17]), "r"(d[18]), "r"(d[19]), "r"(d[20]), "r"(d[21]),
                   "r"(d[22]), "r"(d[23]), "r"(d[24]), "r"(d[25]), "r"(d[26]), "r"(d[27]), "r"(d[28]), "r"(d[29]), "r"(d[30]), "r"(d[31]) : "memory");
}
__device__ __forceinline__ void ft_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void ft_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void ft_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void ft_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ float ft_exp2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
// rows of keys (64 columns of values to 128 bytes, groups of 8 keys 1024 bytes apart, the next 64 columns a tile of 64 keys further on), read as an N-major operand
__device__ __forceinline__ uint64_t ft_vdesc(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(8192 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void ft_store16(uint16_t *y, const float *v, float f, int d, int vdim, bool wide) {      // 16 values of a row from dimension d on
    if (wide) {
        uint32_t o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = fl_pack(v[2 * i] * f, v[2 * i + 1] * f);
        reinterpret_cast<uint4 *>(y + d)[0] = make_uint4(o[0], o[1], o[2], o[3]); reinterpret_cast<uint4 *>(y + d)[1] = make_uint4(o[4], o[5], o[6], o[7]);
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) if (d + i < vdim) y[d + i] = f2bf(v[i] * f);
    }
}

template <int KD, int VD, bool WIN>
__global__ void __launch_bounds__(FT_THREADS, 1) k_flash_tc(FkState *st, const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mk, const __grid_constant__ CUtensorMap mv, FlashArgs a, uint32_t limit) {
    using T = FtTile<KD, VD>;
    constexpr int NR = FT_RING;
    extern __shared__ unsigned char ft_smem[];
    __shared__ __align__(8) uint64_t bars[4 * NR + 11];
    __shared__ uint32_t tmem_slot;
    __shared__ float s_inv[2][128], s_sum[2][128];
    const int tid = threadIdx.x, lane = tid & 31, wid = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t base = (tc_smem(ft_smem) + 1023u) & ~1023u, kbase = base + 2 * T::Q_BYTES, kstage = (uint32_t)(a.maps * T::K_BYTES), vbase = kbase + NR * kstage;
    const uint32_t kfull = tc_smem(bars), kempty = kfull + 8 * NR, vfull = kempty + 8 * NR, vempty = vfull + 8 * NR, sfull = vempty + 8 * NR,      // sfull .. odone: one a side
                   sread = sfull + 16, pfull = sread + 16, odone = pfull + 16, qfull = odone + 16, vzero = qfull + 8, drained = vzero + 8;
    if (tid == 0) {
        for (int i = 0; i < 4 * NR; ++i) tc_init(kfull + 8 * i, 1);
        for (int i = 0; i < 2; ++i) { tc_init(sfull + 8 * i, 1); tc_init(sread + 8 * i, 4); tc_init(pfull + 8 * i, 4); tc_init(odone + 8 * i, 1); }
        tc_init(qfull, 1); tc_init(vzero, 1); tc_init(drained, 1);
        tc_init_fence();
    }
    if (wid == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    ft_before();
    __syncthreads();
    ft_after();
    pdl_launch_dependents();            // not before tensor memory is allocated: a dependent block that got it first would wait for this one
    pdl_wait();
    const uint32_t tmem = tmem_slot;
    const int group = a.H / a.G, pairs = a.maps == 2 ? group : (group + 1) / 2, g = (int)blockIdx.x / pairs, pr = (int)blockIdx.x - g * pairs;
    const int head0 = a.maps == 2 ? (int)blockIdx.x : g * group + 2 * pr, sides = a.maps == 2 || 2 * pr + 1 < group ? 2 : 1;
    const int row0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * 128, off = (int)st->offset, last = off + min(row0 + 127, a.rows - 1);
    const bool fits = a.rows <= a.cap && st->offset <= (uint32_t)(a.cap - a.rows);      // else reported by the cache store that came before
    const int wtile = WIN ? max(0, off + row0 - a.window + 1) / 64 : 0, kept = WIN ? min((a.keep + 63) / 64, wtile) : 0, n = fits ? kept + last / 64 - wtile + 1 : 0;
    auto place = [&](int i) { return i < kept ? i : wtile + i - kept; };
    const int beyond = (last & 63) + 1;                 // rows of the last tile from here on are no keys of this prompt
    bool ok = true;
    if (n == 0) {
    } else if (wid == 8) {
        // ---------------------------------------------------------------- queries, keys, values
        if (lane == 0) {
            tc_expect(qfull, (uint32_t)(sides * T::Q_BYTES));
            for (int s = 0; s < sides; ++s)
#pragma unroll
                for (int c = 0; c < KD / 64; ++c) tc_load(base + s * T::Q_BYTES + c * 16384, &mq, (a.maps == 2 ? head0 * 2 + s : head0 + s) * KD + c * 64, row0, qfull);
            int nk = 0, nv = 0;                         // tiles requested
            for (int i = 0; i < n; ++i) {
                const int r = i % NR, key = place(i) * 64;
                if (i >= NR && !tc_wait(kempty + 8 * r, (uint32_t)(i / NR - 1) & 1u, limit)) { ok = false; break; }
                tc_expect(kfull + 8 * r, kstage);
                for (int m = 0; m < a.maps; ++m)
#pragma unroll
                    for (int c = 0; c < KD / 64; ++c) tc_load(kbase + r * kstage + m * T::K_BYTES + c * 8192, &mk, c * 64, (g * a.maps + m) * a.cap + key, kfull + 8 * r);
                ++nk;
                if (i >= NR && !tc_wait(vempty + 8 * r, (uint32_t)(i / NR - 1) & 1u, limit)) { ok = false; break; }
                tc_expect(vfull + 8 * r, T::V_BYTES);
#pragma unroll
                for (int c = 0; c < VD / 64; ++c) tc_load(vbase + r * T::V_BYTES + c * 8192, &mv, c * 64, g * a.cap + key, vfull + 8 * r);
                ++nv;
            }
            // what is in flight lands before the block leaves
            if (!tc_wait(qfull, 0u, TC_DRAIN)) ok = false;
            for (int i = nk > NR ? nk - NR : 0; i < nk; ++i) if (!tc_wait(kfull + 8 * (i % NR), (uint32_t)(i / NR) & 1u, TC_DRAIN)) ok = false;
            for (int i = nv > NR ? nv - NR : 0; i < nv; ++i) if (!tc_wait(vfull + 8 * (i % NR), (uint32_t)(i / NR) & 1u, TC_DRAIN)) ok = false;
        }
        ok = tc_all(ok);
        if (ok && beyond < 64) {        // weights of rows past the newest key are zero, what the cache holds there may be anything
            tc_wait_warp(vfull + 8 * ((n - 1) % NR), (uint32_t)((n - 1) / NR) & 1u, TC_DRAIN);        // every lane sees what landed
            for (int i = lane; i < (64 - beyond) * 8 * (VD / 64); i += 32) {
                const int c = i / ((64 - beyond) * 8), o = i - c * (64 - beyond) * 8;
                asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(vbase + (uint32_t)(((n - 1) % NR) * T::V_BYTES + c * 8192 + beyond * 128 + o * 16)), "r"(0) : "memory");
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc_arrive(vzero);
        }
        if (!ok && lane == 0) atomicOr(&st->error, FKL_ERR_TC_WAIT);
    } else if (wid == 9) {
        // ---------------------------------------------------------------- MMAs (one elected lane issues, the warp stays together)
        constexpr uint32_t SD = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(64 >> 3) << 17) | ((128u >> 4) << 24);
        constexpr uint32_t OD = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(VD >> 3) << 17) | ((128u >> 4) << 24);
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
        ok = tc_wait_warp(qfull, 0u, limit);
        for (int i = 0; i <= n && ok; ++i) {
            if (i < n) {                                // scores of tile i
                const int r = i % NR;
                if (!tc_wait_warp(kfull + 8 * r, (uint32_t)(i / NR) & 1u, limit)) { ok = false; break; }
                for (int s = 0; s < sides && ok; ++s) {
                    if (i > 0 && !tc_wait_warp(sread + 8 * s, (uint32_t)(i - 1) & 1u, limit)) { ok = false; break; }
                    ft_after();
                    const uint64_t dq = tc_desc(base + s * T::Q_BYTES), dk = tc_desc(kbase + r * kstage + (a.maps == 2 ? s * T::K_BYTES : 0));
                    if (tc_elect()) {
#pragma unroll
                        for (int k = 0; k < KD / 16; ++k)
                            ft_mma_ss(tm + 256 + s * 128, dq + (uint64_t)((k >> 2) * (16384 >> 4) + (k & 3) * 2), dk + (uint64_t)((k >> 2) * (8192 >> 4) + (k & 3) * 2), SD, k ? 1u : 0u);
                        tc_commit(sfull + 8 * s);
                        if (s + 1 == sides) tc_commit(kempty + 8 * r);
                    }
                    __syncwarp();
                }
            }
            if (i > 0 && ok) {                          // values of the tile before
                const int j = i - 1, r = j % NR;
                if (!tc_wait_warp(vfull + 8 * r, (uint32_t)(j / NR) & 1u, limit) || (j + 1 == n && beyond < 64 && !tc_wait_warp(vzero, 0u, limit))) { ok = false; break; }
                const uint64_t dv = ft_vdesc(vbase + r * T::V_BYTES);
                for (int s = 0; s < sides && ok; ++s) {
                    if (!tc_wait_warp(pfull + 8 * s, (uint32_t)j & 1u, limit)) { ok = false; break; }
                    ft_after();
                    const uint32_t p = tm + 256 + s * 128 + 64;
                    if (tc_elect()) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            ft_mma_ts(tm + s * 128, p + k * 8, dv + (uint64_t)(k * (2048 >> 4)), OD, (j | k) ? 1u : 0u);
                            ft_mma_ts(tm + s * 128, p + 32 + k * 8, dv + (uint64_t)(k * (2048 >> 4)), OD, 1u);
                        }
                        tc_commit(odone + 8 * s);
                        if (s + 1 == sides) tc_commit(vempty + 8 * r);
                    }
                    __syncwarp();
                }
            }
        }
        if (!tc_drain_mmas(drained)) ok = false;
        if (!ok && lane == 0) atomicOr(&st->error, FKL_ERR_TC_WAIT);
    } else if ((wid >> 2) < sides) {
        // ---------------------------------------------------------------- softmax of a side, a thread per position
        const int s = wid >> 2, lr = (wid & 3) * 32 + lane, row = row0 + lr, pos = off + row, wpos = off + row0 + (wid & 3) * 32;
        const uint32_t tl = tmem + ((uint32_t)((wid & 3) * 32) << 16), to = tl + s * 128, ts = tl + 256 + s * 128;
        const float sc = a.scale * 1.44269504088896341f;        // scores in base-2 exponents
        float m = -INFINITY, l0 = 0.0f, l1 = 0.0f;
        for (int i = 0; i < n && ok; ++i) {
            const int key0 = place(i) * 64;
            if (!tc_wait_warp(sfull + 8 * s, (uint32_t)i & 1u, limit)) { ok = false; break; }
            ft_after();
            uint32_t v[64];
            ft_ld32(v, ts); ft_ld32(v + 32, ts + 32);
            ft_wait_ld();
            ft_before();
            __syncwarp();
            if (lane == 0) tc_arrive(sread + 8 * s);
            if (key0 + 63 > wpos || (WIN && key0 <= wpos + 31 - a.window)) {         // some key is hidden from some position of the warp
#pragma unroll
                for (int j = 0; j < 64; ++j) { const int key = key0 + j; if (key > pos || (WIN && pos - key >= a.window && key >= a.keep)) v[j] = 0xff800000u; }
            }
            float x0 = -INFINITY, x1 = -INFINITY, x2 = -INFINITY, x3 = -INFINITY;
#pragma unroll
            for (int j = 0; j < 64; j += 4) {
                x0 = fmaxf(x0, __uint_as_float(v[j])); x1 = fmaxf(x1, __uint_as_float(v[j + 1])); x2 = fmaxf(x2, __uint_as_float(v[j + 2])); x3 = fmaxf(x3, __uint_as_float(v[j + 3]));
            }
            const float top = fmaxf(fmaxf(x0, x1), fmaxf(x2, x3)) * sc;
            if (i == 0) m = top;
            else if (__any_sync(0xffffffffu, top > m + 8.0f)) {
                if (!tc_wait_warp(odone + 8 * s, (uint32_t)(i - 1) & 1u, limit)) { ok = false; break; }
                ft_after();
                const float nm = fmaxf(m, top), f = nm == -INFINITY ? 1.0f : ft_exp2(m - nm);
                m = nm; l0 *= f; l1 *= f;
#pragma unroll 1
                for (int c = 0; c < VD; c += 32) {
                    uint32_t o[32];
                    ft_ld32(o, to + c); ft_wait_ld();
#pragma unroll
                    for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * f);
                    ft_st32(to + c, o);
                }
                ft_wait_st();
            }
            const float e = m == -INFINITY ? 0.0f : -m;          // no key seen yet: every weight is 0
            uint32_t hi[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                const float p0 = ft_exp2(fmaf(__uint_as_float(v[2 * j]), sc, e)), p1 = ft_exp2(fmaf(__uint_as_float(v[2 * j + 1]), sc, e));
                l0 += p0; l1 += p1;
                hi[j] = fl_pack(p0, p1);
                v[j] = fl_pack(p0 - bf_lo(hi[j]), p1 - bf_hi(hi[j]));
            }
            if (i > 0) {                                // the tile before has been multiplied
                if (!tc_wait_warp(odone + 8 * s, (uint32_t)(i - 1) & 1u, limit)) { ok = false; break; }
                ft_after();
            }
            ft_st32(ts + 64, hi); ft_st32(ts + 96, v);
            ft_wait_st();
            ft_before();
            __syncwarp();
            if (lane == 0) tc_arrive(pfull + 8 * s);
        }
        if (ok && !tc_wait_warp(odone + 8 * s, (uint32_t)(n - 1) & 1u, limit)) ok = false;
        const float inv = 1.0f / (l0 + l1);
        const bool wide = !((a.ldo | a.vdim) & 7) && !((uintptr_t)a.out & 15);
        const bool mine = ok && row < a.rows;
        if (a.maps == 1) {
            if (ok) {
                ft_after();
                const int head = head0 + s;
                const float f = inv * (a.gate && mine ? sigmoid_f(bf2f(a.gate[(size_t)row * a.ldg + head])) : 1.0f);
                uint16_t *y = a.out + (size_t)row * a.ldo + head * a.vdim;
#pragma unroll 1
                for (int c = 0; c < VD; c += 32) {
                    uint32_t o[32];
                    ft_ld32(o, to + c); ft_wait_ld();
                    float v[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(o[j]);
                    if (mine) { ft_store16(y, v, f, c, a.vdim, wide); ft_store16(y, v + 16, f, c + 16, a.vdim, wide); }
                }
            }
        } else {
            // the sides share a head: side s takes the s-th half of every row's values
            if (ok && !tc_wait_warp(odone + 8 * (s ^ 1), (uint32_t)(n - 1) & 1u, limit)) ok = false;
            ft_after();
            s_inv[s][lr] = inv;
            asm volatile("bar.sync 1, 256;" ::: "memory");
            const float i0 = s_inv[0][lr], i1 = s_inv[1][lr];
            float v[VD / 2], ss = 0.0f;
#pragma unroll
            for (int c = 0; c < VD / 2; c += 32) {
                uint32_t o[32];
                ft_ld32(o, tl + s * (VD / 2) + c); ft_wait_ld();
#pragma unroll
                for (int j = 0; j < 32; ++j) v[c + j] = __uint_as_float(o[j]) * i0;
                ft_ld32(o, tl + 128 + s * (VD / 2) + c); ft_wait_ld();
#pragma unroll
                for (int j = 0; j < 32; ++j) { v[c + j] -= a.lambda * (__uint_as_float(o[j]) * i1); if (s * (VD / 2) + c + j < a.vdim) ss = fmaf(v[c + j], v[c + j], ss); }
            }
            s_sum[s][lr] = ss;
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if (mine && ok) {
                float f = inv_rms(s_sum[0][lr] + s_sum[1][lr], a.vdim, a.eps) * (1.0f - a.diff);
                if (a.gate) f *= sigmoid_f(bf2f(a.gate[(size_t)row * a.ldg + head0]));
                uint16_t *y = a.out + (size_t)row * a.ldo + head0 * a.vdim;
#pragma unroll
                for (int c = 0; c < VD / 2; c += 16) ft_store16(y, v + c, f, s * (VD / 2) + c, a.vdim, wide);
            }
        }
        if (!ok && lane == 0) atomicOr(&st->error, FKL_ERR_TC_WAIT);
    }
    ft_before();
    __syncthreads();
    ft_after();
    if (wid == 9) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}
