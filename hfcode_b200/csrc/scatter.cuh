// J/K scatter of one shell quartet's ERI block, shared by `nl` lanes, into
// the one-triangle buffer G (F += G + G^T later; shell-pair blocks, block
// (s1, s2) row-major at boff[s1 * nsh + s2]), one FP64 atomic per block
// element:
//   J_ab += 2s P_cd e,  J_cd += 2s P_ab e,
//   K_ac -= s/2 P_bd e, K_ad -= s/2 P_bc e, K_bc -= s/2 P_ad e, K_bd -= s/2 P_ac e.
// The quartet's density blocks go to `w` first; then lane x, x + nl, ... of
// the block elements (16 to 25 per block) each sum their row of products.
// With one thread per quartet the (dd|dd) block is a serial chain of 625
// element loads and 3750 FMAs, which a small molecule has nothing to hide
// behind: 288 us for the 21 (dd|dd) diagonal quartets of benzene.
// Host-compilable with the shims of the test harness (lane 0 of 1).
#pragma once
#include "types.cuh"

namespace hfgpu {

// The six J/K blocks of a quartet as one range of elements: J_ab, J_cd, K_ac,
// K_ad, K_bc, K_bd, each row-major as in G.
template <int NA, int NB, int NC, int ND>
struct Blocks {
    static constexpr int AB = 0, CD = NA * NB, AC = CD + NC * ND, AD = AC + NA * NC, BC = AD + NA * ND,
                         BD = BC + NB * NC, END = BD + NB * ND;
};

// Density elements a quartet's scatter reads: P_cd, P_ab, P_bd, P_bc, P_ad, P_ac.
__host__ __device__ constexpr int scatter_dens(int NA, int NB, int NC, int ND) {
    return NC * ND + NA * NB + NB * ND + NB * NC + NA * ND + NA * NC;
}

// dst(s1, s2, r, c, y): where element (r, c) of the basis, the y-th of the
// block of shells s1 and s2, is added.
template <int NA, int NB, int NC, int ND, typename E, typename Dst>
__device__ __forceinline__ void scatter_lanes(const E* e, double* w, double s, const GPair& bra, const GPair& ket,
                                              const double* __restrict__ P, int nb, Dst dst, bool jonly, int lane,
                                              int nl) {
    const int a0 = bra.aoa, b0 = bra.aob, c0 = ket.aoa, d0 = ket.aob;
    double *pcd = w, *pab = pcd + NC * ND, *pbd = pab + NA * NB, *pbc = pbd + NB * ND, *pad_ = pbc + NB * NC,
           *pac = pad_ + NA * ND;
    // block (r, c) of P, row-major; P is symmetric and column-major
    auto fetch = [&](double* dst, int r0, int nr, int cc0, int nc) {
        for (int x = lane; x < nr * nc; x += nl) dst[x] = __ldg(P + (cc0 + x % nc) + (size_t)(r0 + x / nc) * nb);
    };
    fetch(pcd, c0, NC, d0, ND);
    fetch(pab, a0, NA, b0, NB);
    if (!jonly) {
        fetch(pbd, b0, NB, d0, ND);
        fetch(pbc, b0, NB, c0, NC);
        fetch(pad_, a0, NA, d0, ND);
        fetch(pac, a0, NA, c0, NC);
    }
#ifdef __CUDA_ARCH__
    __syncwarp();
#endif
    constexpr int SI = NB * NC * ND, SJ = NC * ND, SK = ND;  // strides of i, j, k in the block
    using X = Blocks<NA, NB, NC, ND>;
    constexpr int O1 = X::CD, O2 = X::AC, O3 = X::AD, O4 = X::BC, O5 = X::BD;
    const int nel = jonly ? O2 : X::END;
    for (int x = lane; x < nel; x += nl) {
        // element (r, c) of its block, and the two indices it sums over
        int y, r, c, base, n1, s1, n2, s2;
        const double* d;
        double* g;
        if (x < O1) {
            y = x, r = y / NB, c = y % NB;
            base = r * SI + c * SJ, n1 = NC, s1 = SK, n2 = ND, s2 = 1, d = pcd;
            g = dst(bra.sa, bra.sb, a0 + r, b0 + c, y);
        } else if (x < O2) {
            y = x - O1, r = y / ND, c = y % ND;
            base = r * SK + c, n1 = NA, s1 = SI, n2 = NB, s2 = SJ, d = pab;
            g = dst(ket.sa, ket.sb, c0 + r, d0 + c, y);
        } else if (x < O3) {
            y = x - O2, r = y / NC, c = y % NC;
            base = r * SI + c * SK, n1 = NB, s1 = SJ, n2 = ND, s2 = 1, d = pbd;
            g = dst(bra.sa, ket.sa, a0 + r, c0 + c, y);
        } else if (x < O4) {
            y = x - O3, r = y / ND, c = y % ND;
            base = r * SI + c, n1 = NB, s1 = SJ, n2 = NC, s2 = SK, d = pbc;
            g = dst(bra.sa, ket.sb, a0 + r, d0 + c, y);
        } else if (x < O5) {
            y = x - O4, r = y / NC, c = y % NC;
            base = r * SJ + c * SK, n1 = NA, s1 = SI, n2 = ND, s2 = 1, d = pad_;
            g = dst(bra.sb, ket.sa, b0 + r, c0 + c, y);
        } else {
            y = x - O5, r = y / ND, c = y % ND;
            base = r * SJ + c, n1 = NA, s1 = SI, n2 = NC, s2 = SK, d = pac;
            g = dst(bra.sb, ket.sb, b0 + r, d0 + c, y);
        }
        double acc = 0.0;
        for (int u = 0; u < n1; ++u)
            for (int v = 0; v < n2; ++v) acc += d[u * n2 + v] * (double)e[base + u * s1 + v * s2];
        atomicAdd(g, (x < O2 ? 2.0 * s : -0.5 * s) * acc);
    }
}

}  // namespace hfgpu
