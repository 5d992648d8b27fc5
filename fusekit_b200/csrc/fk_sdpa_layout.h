// Shared memory of the cluster attention kernels on the tensor cores (k_sdpa_mma, k_sdpa_mma_q).  Plain C++, so that tests look at it without a GPU.
#pragma once
#include <stddef.h>

#if defined(__CUDACC__)
#define FKS_HD __host__ __device__
#else
#define FKS_HD
#endif
#define FK_SDPA_CLMAX 16        // CTAs of the largest cluster (a non-portable size), taken when few kv heads leave SMs idle
#define FK_SDPA_CW 16           // warps per CTA
#define FK_SDPA_MK 16           // keys per warp iteration

// [cpart, fexp) is received: the other CTAs of the cluster store into it as soon as every CTA is running, so nothing of a CTA's own may lie there.
template <int HD, int CW = FK_SDPA_CW> struct SdpaMmaLayout {
    static constexpr int QSTRIDE = HD * 2 + 16;                  // bytes per q row (bf16)
    static constexpr int VSTRIDE = HD * 2 + 16;                  // bytes per V tile row: ldmatrix rows hit distinct banks
    static constexpr int WTILE = FK_SDPA_MK * VSTRIDE;           // bytes of a warp's V tile; later its [G][HD+2] fp32 partial
    static constexpr int QSUMS = (8 * (HD / 64) + 8) * 4;        // bytes: over a quantised cache, [8][HD / 64] sums of q's groups and [8] inverse scales
    FKS_HD static constexpr int q() { return 0; }
    FKS_HD static constexpr int tiles() { return 8 * QSTRIDE; }
    FKS_HD static constexpr int cpart() { return tiles() + CW * WTILE; }
    FKS_HD static constexpr int wexp(int G) { return cpart() + (G * HD + FK_SDPA_CLMAX) * 4; }      // after the received o slices
    FKS_HD static constexpr int fexp(int G) { return wexp(G) + FK_SDPA_CLMAX * G * 2 * 4; }              // [16][G] factors + [G] maxima + [G] 1 / l
    FKS_HD static constexpr int qsum(int G) { return fexp(G) + (16 * G + 2 * G) * 4; }
    FKS_HD static constexpr int bytes(int G) { return qsum(G) + QSUMS; }
};
template <int CW> FKS_HD inline size_t sdpa_mma_smem_bytes(int G, int hd) { return hd == 256 ? SdpaMmaLayout<256, CW>::bytes(G) : hd == 128 ? SdpaMmaLayout<128, CW>::bytes(G) : SdpaMmaLayout<64, CW>::bytes(G); }
