// Shared device code of the B200 Fock builder: data layout, Boys function,
// J/K scatter and the kernel templates instantiated once per quartet class
// (one translation unit per class, see generated/cls_*.cu).
#pragma once
#include <cuda_runtime.h>

#include "types.cuh"
#include "lists.cuh"
#include "scatter.cuh"

#include <cstdint>
#include <type_traits>

namespace hfgpu {

// ------------------------------------------------------- class traits ----
// functions of the first / second shell of pair type t
// (SS LS LL DS DL DD PS LP PP DP)
__host__ __device__ constexpr int pt_na(int t) {
    return t == 0 ? 1 : t <= 2 ? 4 : t <= 5 ? 5 : t == 6 ? 3 : t == 7 ? 4 : t == 8 ? 3 : 5;
}
__host__ __device__ constexpr int pt_nb(int t) {
    return t == 0 || t == 1 || t == 3 || t == 6 ? 1 : t == 2 || t == 4 ? 4 : t == 5 ? 5 : 3;
}

#define HF_CLASS_TRAITS(ci, bi, ki, NAME, nout, L)                                                   \
    struct Cls_##NAME {                                                                              \
        static constexpr int CI = ci, BI = bi, KI = ki, NOUT = nout, LL = L;                         \
        __device__ __forceinline__ static void eri(const GPair& b, const GPair& k, const PrimSoA& p, \
                                                   const double* t, const LaneSplit& ls, double* o) { \
            eri_##NAME(b, k, p, t, ls, o);                                                           \
        }                                                                                            \
        __device__ __forceinline__ static void eri32(const GPair& b, const GPair& k, const PrimSoA& p, \
                                                     const float* t, const LaneSplit& ls, float* o) { \
            eri_##NAME##_f32(b, k, p, t, ls, o);                                                     \
        }                                                                                            \
    };

// ------------------------------------------------------- warp output ----
// The J/K sums of a warp's 32 quartets go into G element by element across
// the lanes: the lanes write their quartets' sums of up to N elements to a
// shared buffer ([element][quartet], WST apart), then lane v owns element v
// and walks the quartets, adding up the runs of quartets that share the block
// (consecutive entries of a list mostly share the bra pair and the ket's
// first shell) with one atomic per run.  The lanes of one atomic instruction
// then lie in one or two blocks of G, which are contiguous: a warp's atomics
// touch 2-3 cache lines instead of 32.  With one atomic per element and lane
// the L1 tag stage (one line per cycle) bounded every scatter: 110 atomic
// instructions of 31 lines per warp for LL|DL, l1tex throughput 55-62% in
// all scatter kernels while the FP64 pipe idled.
constexpr int WST = 33;  // odd stride: a column is written and read without bank conflicts

// Block offsets of the warp's quartets in G: [block type][quartet], in the
// order of Blocks (ab, cd, ac, ad, bc, bd); -1 for lanes without a quartet.
constexpr int NBASE = 6 * WST;
__device__ __forceinline__ void set_bases(int* base, const int* __restrict__ boff, int nsh, const GPair& bra,
                                          const GPair& ket, bool act) {
    const int lane = threadIdx.x & 31;
    const int s[6][2] = {{bra.sa, bra.sb}, {ket.sa, ket.sb}, {bra.sa, ket.sa},
                         {bra.sa, ket.sb}, {bra.sb, ket.sa}, {bra.sb, ket.sb}};
#pragma unroll
    for (int x = 0; x < 6; ++x) base[x * WST + lane] = act ? __ldg(boff + s[x][0] * nsh + s[x][1]) : -1;
}

// Adds elements [0, n) of the buffer (n <= N, warp-uniform): map(v, type, off)
// gives element v's block type and place in the block.  N <= 16 lets two, N
// <= 8 four groups of lanes walk a half or a quarter of the quartets each.
// The caller synchronises the warp before (the buffer is written) and after.
template <int N, typename E, typename Map>
__device__ __forceinline__ void walk_add(const E* tb, const int* base, int n, double* __restrict__ G, Map map) {
    constexpr int NG = N <= 8 ? 4 : N <= 16 ? 2 : 1, W = 32 / NG;  // groups; lanes (and quartets) per group
    const int lane = threadIdx.x & 31, q0 = lane / W * W;
#pragma unroll 1
    for (int v = lane % W; v < n; v += W) {
        int type, off;
        map(v, type, off);
        const int* b = base + type * WST + q0;
        const E* t = tb + v * WST + q0;
        double sum = 0.0;
        int cur = -1;
#pragma unroll 4
        for (int q = 0; q < W; ++q) {
            const int x = b[q];
            if (x != cur) {
                if (cur >= 0) atomicAdd(G + cur + off, sum);
                cur = x;
                sum = 0.0;
            }
            sum += (double)t[q];
        }
        if (cur >= 0) atomicAdd(G + cur + off, sum);
    }
}

// ------------------------------------------------------------ scatter ----
// F contributions of the 32 quartets of a warp, blocks in registers (direct
// classes), with weight s, into the one-triangle buffer G (F += G + G^T
// later).  P and G are in shell-pair blocks.  `tb` and `base`: the warp's
// shared buffers.  Every lane of the warp calls it; those with act false add
// nothing.
constexpr int DCH = 16;  // elements per pass through the buffer
template <int NA, int NB, int NC, int ND, typename E>
__device__ __forceinline__ void scatter_quartet(const E* e, double s, const GPair& bra, const GPair& ket, bool act,
                                                const double* __restrict__ Pb, const int* __restrict__ boff, int nsh,
                                                double* __restrict__ G, bool jonly, double* tb, int* base) {
    using X = Blocks<NA, NB, NC, ND>;
    const int lane = threadIdx.x & 31;
    const double* __restrict__ Pab = Pb + __ldg(boff + bra.sa * nsh + bra.sb);
    const double* __restrict__ Pcd = Pb + __ldg(boff + ket.sa * nsh + ket.sb);
    const double* __restrict__ Pac = Pb + __ldg(boff + bra.sa * nsh + ket.sa);
    const double* __restrict__ Pad = Pb + __ldg(boff + bra.sa * nsh + ket.sb);
    const double* __restrict__ Pbc = Pb + __ldg(boff + bra.sb * nsh + ket.sa);
    const double* __restrict__ Pbd = Pb + __ldg(boff + bra.sb * nsh + ket.sb);
    __syncwarp();  // the previous pass has been read
    set_bases(base, boff, nsh, bra, ket, act);
    const double s2 = 2.0 * s, hs = -0.5 * s;
    auto E4 = [&](int i, int j, int k, int l) { return (double)e[((i * NB + j) * NC + k) * ND + l]; };
    const int nel = jonly ? X::AC : X::END;
#pragma unroll
    for (int c = 0; c < X::END; c += DCH) {
        if (c >= nel) break;
        if (c > 0) __syncwarp();  // the previous chunk has been read
#pragma unroll
        for (int x = c; x < (c + DCH < X::END ? c + DCH : X::END); ++x) {
            double acc = 0.0;
            if (x < X::CD) {
#pragma unroll
                for (int k = 0; k < NC; ++k)
#pragma unroll
                    for (int l = 0; l < ND; ++l) acc += __ldg(Pcd + k * ND + l) * E4(x / NB, x % NB, k, l);
            } else if (x < X::AC) {
                const int y = x - X::CD;
#pragma unroll
                for (int i = 0; i < NA; ++i)
#pragma unroll
                    for (int j = 0; j < NB; ++j) acc += __ldg(Pab + i * NB + j) * E4(i, j, y / ND, y % ND);
            } else if (x < X::AD) {
                const int y = x - X::AC;
#pragma unroll
                for (int j = 0; j < NB; ++j)
#pragma unroll
                    for (int l = 0; l < ND; ++l) acc += __ldg(Pbd + j * ND + l) * E4(y / NC, j, y % NC, l);
            } else if (x < X::BC) {
                const int y = x - X::AD;
#pragma unroll
                for (int j = 0; j < NB; ++j)
#pragma unroll
                    for (int k = 0; k < NC; ++k) acc += __ldg(Pbc + j * NC + k) * E4(y / ND, j, k, y % ND);
            } else if (x < X::BD) {
                const int y = x - X::BC;
#pragma unroll
                for (int i = 0; i < NA; ++i)
#pragma unroll
                    for (int l = 0; l < ND; ++l) acc += __ldg(Pad + i * ND + l) * E4(i, y / NC, y % NC, l);
            } else {
                const int y = x - X::BD;
#pragma unroll
                for (int i = 0; i < NA; ++i)
#pragma unroll
                    for (int k = 0; k < NC; ++k) acc += __ldg(Pac + i * NC + k) * E4(i, y / ND, k, y % ND);
            }
            tb[(x - c) * WST + lane] = (x < X::AC ? s2 : hs) * acc;
        }
        __syncwarp();
        walk_add<DCH>(tb, base, min(DCH, nel - c), G, [&](int v, int& type, int& off) {
            const int x = c + v;
            type = x < X::CD ? 0 : x < X::AC ? 1 : x < X::AD ? 2 : x < X::BC ? 3 : x < X::BD ? 4 : 5;
            off = x - (x < X::CD ? 0 : x < X::AC ? X::CD : x < X::AD ? X::AC : x < X::BC ? X::AD
                       : x < X::BD ? X::BC : X::BD);
        });
    }
}

// Elements of G (shell-pair blocks) for scatter_lanes.
struct BlockDst {
    double* G;
    const int* boff;
    int nsh;
    __device__ __forceinline__ double* operator()(int s1, int s2, int, int, int y) const {
        return G + __ldg(boff + s1 * nsh + s2) + y;
    }
};

// ------------------------------------------------------- kernel args ----
struct ClassStats {
    unsigned long long scattered, prim, fp32;
};

// Unit u of the list: false past the end (see unit_place).
__device__ __forceinline__ bool unit_of(const UnitList& L, int u, Unit& w) {
    long long at;
    if (!unit_place(L, u, threadIdx.x & 31, w, at)) return false;
    w.q = L.quartets[at];
    return true;
}

struct NDArgs {
    UnitList list;
    const GPair* bra;
    const GPair* ket;
    PrimSoA prims;
    const double* boys;     // Boys tables of every order, BOYS_BLK values each (types.cuh)
    const float* boysf;
    const double* Pb;       // density in shell-pair blocks
    double* G;              // in shell-pair blocks
    const int* boff;        // block offsets, nsh x nsh
    int nsh;
    double thr;
    int jonly;
    ClassStats* stats;
};

template <int M, typename T>
__device__ __forceinline__ void stage_boys(T* sm, const T* g) {
    const T* src = g + (size_t)M * BOYS_BLK;
    for (int i = threadIdx.x; i < BOYS_BLK; i += blockDim.x) sm[i] = src[i];
    __syncthreads();
}

__device__ __forceinline__ void warp_add_stats(ClassStats* st, unsigned long long sc, unsigned long long pr,
                                               unsigned long long f32) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sc += __shfl_down_sync(0xffffffffu, sc, o);
        pr += __shfl_down_sync(0xffffffffu, pr, o);
        f32 += __shfl_down_sync(0xffffffffu, f32, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (sc) atomicAdd(&st->scattered, sc);
        if (pr) atomicAdd(&st->prim, pr);
        if (f32) atomicAdd(&st->fp32, f32);
    }
}

constexpr int ND_THREADS = 128;
// Threads per block of the staged role kernels, a divisor of ND_THREADS.
// Smaller blocks at the same registers per thread (more blocks per SM) let
// the role kernels of one class stream and the scatters of another share
// the SMs at a finer grain.  C60 FP64 build: 197.6 ms with 128 threads,
// 194.1 with 64, 192.7 with 32; all-FP32 build 124.8, 122.3, 122.3 ms.
#ifndef HF_RB_THREADS
#define HF_RB_THREADS 32
#endif
constexpr int RB_THREADS = HF_RB_THREADS, RB_SCALE = ND_THREADS / RB_THREADS;
static_assert(RB_THREADS * RB_SCALE == ND_THREADS, "role blocks tile a scratch tile exactly");

// Shared memory of a direct kernel's block, per warp: the output buffer and
// the block offsets.
struct NDShared {
    double tbuf[ND_THREADS / 32][DCH * WST];
    int tbase[ND_THREADS / 32][NBASE];
};

// The work units u0, u0 + du, ... of a direct class.
template <class C, bool F32, typename Real>
__device__ __forceinline__ void nondiag_units(const UnitList& list, const GPair* __restrict__ bras,
                                              const GPair* __restrict__ kets, const PrimSoA& prims,
                                              const Real* __restrict__ boys, const double* __restrict__ Pb,
                                              double* __restrict__ G, const int* __restrict__ boff, int nsh,
                                              double thr, bool jonly, ClassStats* stats, int u0, int du,
                                              NDShared& sh) {
    constexpr int NA = pt_na(C::BI), NB = pt_nb(C::BI), NC = pt_na(C::KI), ND = pt_nb(C::KI);
    static_assert(NA * NB * NC * ND == C::NOUT, "class size");
    unsigned long long nsc = 0, npr = 0;
    const int wp = threadIdx.x >> 5;
    Unit w;
    for (int u = u0 + wp; unit_of(list, u, w); u += du) {
        const GPair bra = bras[w.q.x];
        const GPair ket = kets[w.q.y];
        Real e[C::NOUT];
        if constexpr (F32) C::eri32(bra, ket, prims, boys, w.ls, e);
        else C::eri(bra, ket, prims, boys, w.ls, e);
        Real mx = 0;
#pragma unroll
        for (int i = 0; i < C::NOUT; ++i) mx = fmax(mx, fabs(e[i]));
        const bool act = w.store && !((double)mx < thr);  // fock_build_non_diag.f90:69
        npr += w.store ? (unsigned long long)(bra.np * ket.np) : 0ull;
        nsc += act ? 1ull : 0ull;
        const double s = (bra.sa == bra.sb ? 0.5 : 1.0) * (ket.sa == ket.sb ? 0.5 : 1.0);
        scatter_quartet<NA, NB, NC, ND>(e, s, bra, ket, act, Pb, boff, nsh, G, jonly, sh.tbuf[wp], sh.tbase[wp]);
    }
    if (stats) warp_add_stats(stats, nsc, npr, F32 ? nsc : 0ull);
}

template <class C, bool F32>
__global__ void __launch_bounds__(ND_THREADS) k_nondiag(NDArgs a) {
    using Real = typename std::conditional<F32, float, double>::type;
    const int u0 = blockIdx.x * (ND_THREADS / 32);
    if (u0 >= a.list.nunit[2 * a.list.cls + a.list.prec]) return;  // idle block of a captured grid
    __shared__ Real sboys[BOYS_BLK];
    if constexpr (F32) stage_boys<C::LL>(sboys, a.boysf);
    else stage_boys<C::LL>(sboys, a.boys);
    __shared__ NDShared sh;
    nondiag_units<C, F32, Real>(a.list, a.bra, a.ket, a.prims, sboys, a.Pb, a.G, a.boff, a.nsh, a.thr, a.jonly != 0,
                                a.stats, u0, gridDim.x * (ND_THREADS / 32), sh);
}

// Every direct class of a small build in one launch: the blocks are dealt out
// to the lists in turn.  One launch per class leaves a dozen kernels of
// 20-35 us, each too short to fill the GPU, on the class streams.  The Boys
// tables are read through L1 here: most blocks do one unit per warp.
constexpr int MAXDIRECT = 64;
struct NDItem {
    UnitList list;
    const GPair* bra;
    const GPair* ket;
    ClassStats* stats;
    int block0, blocks;  // this list's blocks of the grid
};
struct NDAllArgs {
    int nitem;
    PrimSoA prims;
    const double* boys;
    const float* boysf;
    const double* Pb;
    double* G;
    const int* boff;
    int nsh;
    double thr;
    int jonly;
    NDItem item[MAXDIRECT];
};

struct DiagArgs {
    const GPair* pairs;
    int n;
    PrimSoA prims;
    const double* boys;
    double* schw;          // mode 0: written; mode 1: read
    const double* md;      // mode 1: nsh x nsh maxdm
    int nsh;
    const double* P;
    double* G;             // in shell-pair blocks
    const int* boff;       // block offsets, nsh x nsh
    int nb;
    double thr;
};

// The density screen of the diagonal builder (fock_build_diag.f90:20-21).
__device__ __forceinline__ bool diag_screened(const GPair& pr, double sw, const double* md, int nsh, double thr) {
    const double mv = fmax(md[pr.sa * nsh + pr.sb],
                           fmax(0.25 * md[pr.sb * nsh + pr.sb], 0.25 * md[pr.sa * nsh + pr.sa]));
    return sw * sw * mv < thr;
}

// Shell pairs with themselves, (ab|ab): fock_build_initial_diag.f90 (MODE 0)
// and fock_build_diag.f90 (MODE 1).  One warp per pair: its lanes split the
// np^2 primitive quartets (up to 1296), 4 over the bra and 8 over the ket.
template <class C, int MODE>
__global__ void __launch_bounds__(ND_THREADS) k_diag(DiagArgs a) {
    constexpr int NA = pt_na(C::BI), NB = pt_nb(C::BI);
    const int t = blockIdx.x * (ND_THREADS / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (t >= a.n) return;
    const GPair pr = a.pairs[t];
    if (MODE == 1 && diag_screened(pr, a.schw[t], a.md, a.nsh, a.thr)) return;
    __shared__ double sw[ND_THREADS / 32][scatter_dens(NA, NB, NA, NB)], se[ND_THREADS / 32][C::NOUT];
    const int wp = threadIdx.x >> 5;
    double e[C::NOUT];
    C::eri(pr, pr, a.prims, a.boys + (size_t)C::LL * BOYS_BLK, LaneSplit{lane >> 3, 4, lane & 7, 8, 32}, e);
    if (MODE == 0) {
        double mx = 0;
#pragma unroll
        for (int i = 0; i < C::NOUT; ++i) mx = fmax(mx, fabs(e[i]));
        if (lane == 0) a.schw[t] = sqrt(mx);
    }
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < C::NOUT; ++i) se[wp][i] = fabs(e[i]) > INTTHRESH ? e[i] : 0.0;  // element skip
    }
    const double f = pr.sa == pr.sb ? 1.0 : 2.0;
    scatter_lanes<NA, NB, NA, NB>(se[wp], sw[wp], f * f / 8.0, pr, pr, a.P, a.nb, BlockDst{a.G, a.boff, a.nsh}, false,
                                  lane, 32);
}


// Arguments of the staged classes' kernels: a chunk of the class's quartet
// list, and the scratch it goes through (accumulators, outputs and the
// per-role maxima, each in tiles of TQ quartets: see tcol below).
struct StagedArgs {
    const uint2* quartets;
    int n;                 // quartets in this chunk (an upper bound when ncls is set)
    long long q0;          // chunk start within the list
    const unsigned long long* ncls;  // device-side counts, as in NDArgs (or nullptr)
    int cls, prec;
    const GPair* bra;
    const GPair* ket;
    PrimSoA prims;
    const double* boys;
    const float* boysf;
    double* acc;
    double* out;
    double* mx;
    size_t stride;         // chunk capacity in quartets (a multiple of the tile size TQ)
    int nroles;            // rows of mx
    const double* P;
    double* G;
    int nb;
    double thr;
    int jonly;
    int f32;
    ClassStats* stats;
    const double* Pb;      // density in shell-pair blocks (staged scatter)
    const int* boff;       // block offsets, nsh x nsh
    // diagonal builders only
    double* schw;          // per pair (MODE 0 writes, MODE 1 reads)
    const double* md;      // nsh x nsh density maxima
    int nsh;
    // one launch per stage (gridDim.y = roles): the class's work units, or
    // with list.subs null one quartet per unit (the diagonal builders)
    UnitList list;
};

// Quartets of this chunk: a.n, or with device-side counts the part of the
// list left after q0, at most a.n.
__device__ __forceinline__ int staged_count(const StagedArgs& a) {
    if (!a.ncls) return a.n;
    const long long left = (long long)a.ncls[2 * a.cls + a.prec] - a.q0;
    return (int)(left < 0 ? 0 : left < a.n ? left : a.n);
}

// Units of the chunk in a one-launch stage, [u0, u1): those of the list that
// hold its entries (the first and last may reach into a neighbouring chunk,
// which computes them too), or one per two pairs in the diagonal builders.
__device__ __forceinline__ void chunk_units(const StagedArgs& a, int& u0, int& u1) {
    const UnitList& L = a.list;
    if (!L.subs) {
        u0 = 0;
        u1 = (a.n + 1) / 2;
        return;
    }
    const int n = staged_count(a);
    u0 = u1 = 0;
    if (n > 0) units_of(L, list_start(L) + a.q0, n, u0, u1);
}

// Unit u of a one-launch stage (chunk_units).
__device__ __forceinline__ void stage_unit(const StagedArgs& a, int u, Unit& w) {
    if (a.list.subs) {
        // the entry is counted in 64 bits, but held in 32: the extra register
        // cost the primitive-loop stages 12 bytes of spills, 1-2% of a small
        // build
        long long at = 0;
        unit_place(a.list, u, threadIdx.x & 31, w, at);
        const long long t = at - list_start(a.list) - a.q0;
        w.q = a.list.quartets[at];
        w.store = w.store && t >= 0 && t < a.n;  // entries of other chunks are not stored
        w.t = (int)t;
        return;
    }
    // diagonal builders: two pairs per warp, their at most 9 x 9 primitive
    // quartets over 4 x 4 lanes
    const int lane = threadIdx.x & 31, g = lane & 15, i = 2 * u + (lane >> 4);
    w.t = i < a.n ? i : a.n - 1;
    w.q = a.quartets[a.q0 + w.t];
    w.store = i < a.n && g == 0;
    w.ls = LaneSplit{g >> 2, 4, g & 3, 4, 16};
}

// Scratch layout of a chunk.  Each region (accumulators, outputs, role
// maxima) is a sequence of tiles of TQ quartets; a tile holds the region's R
// rows of its quartets, row-major: element (row, t) sits at
// tcol(t, R) + row * TQ.  A block of ND_THREADS = TQ threads then reads and
// writes one contiguous span of R * TQ elements (a few hundred KB, within
// one or two pages), instead of R rows as far apart as the chunk is long.
constexpr int TQ = 128;
static_assert(TQ == ND_THREADS, "a block of the staged kernels covers one scratch tile");
__device__ __forceinline__ size_t tcol(int t, int R) { return (size_t)(t / TQ) * R * TQ + (t % TQ); }

__device__ __forceinline__ uint2 staged_quartet(const StagedArgs& a, int t) {
    const long long i = a.q0 + t + (a.ncls && a.prec ? (long long)a.ncls[2 * a.cls] : 0);
    return a.quartets[i];
}

// ------------------------------------------- staged scatter, async loads ----
// The staged scatter reads each quartet's ERI block (its column of the
// chunk's output tile) once.  With ~255 registers per thread only 8 warps fit on an
// SM, too few to hide the latency of plain loads, so the block's rows are
// streamed into shared memory with per-thread cp.async copies: slab s (the
// NC*ND rows of one (i, j)) is consumed while slabs s+1 .. s+NBUF-1 are in
// flight.  Every thread copies and reads only its own column, so no block
// barrier is needed; cp.async.wait_group bounds each wait by the thread's own
// copies.  P_bc and P_bd, needed for every i, are staged once in shared
// memory as well.
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

template <typename E>
__device__ __forceinline__ void cp_async_elem(E* dst, const E* src) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (sizeof(E) == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(src) : "memory");
}

// Shared-memory plan of the async scatter (element size es), per warp: NBUF
// slab buffers (three when they fit two blocks per SM, else two), P_bc and
// P_bd, the output buffer of one i (in the slab just consumed where that is
// large enough) and the block offsets.  The last output pass, J_cd, K_bc and
// K_bd, goes through the slab buffers and the P rows, which are free then.
__host__ __device__ constexpr bool scat_over(int NB, int NC, int ND) { return NC * ND * 32 >= (NB + NC + ND) * WST; }
__host__ __device__ constexpr int scat_warp_elems(int nbuf, int NB, int NC, int ND) {
    return (nbuf * NC * ND + NB * (NC + ND)) * 32 + (scat_over(NB, NC, ND) ? 0 : (NB + NC + ND) * WST);
}
__host__ __device__ constexpr int scat_bytes(int nbuf, int NB, int NC, int ND, int es) {
    return (ND_THREADS / 32) * (scat_warp_elems(nbuf, NB, NC, ND) * es + NBASE * 4);
}
__host__ __device__ constexpr int scat_nbuf(int NA, int NB, int NC, int ND, int es = 8) {
    return scat_bytes(3, NB, NC, ND, es) <= 112 * 1024 ? 3 : 2;
}
__host__ __device__ constexpr int scat_smem_bytes(int NA, int NB, int NC, int ND, int es = 8) {
    return scat_bytes(scat_nbuf(NA, NB, NC, ND, es), NB, NC, ND, es);
}

// E is the element type of the scratch rows and of the block sums: double
// for FP64 quartets, float for the FP32 quartets of the mixed form (their
// integrals are FP32 already; the sums go into G with FP64 atomics).
template <int NA, int NB, int NC, int ND, typename E>
__device__ __forceinline__ void scatter_async(const E* __restrict__ e, size_t st, double s, const GPair& bra,
                                              const GPair& ket, const double* __restrict__ Pb,
                                              const int* __restrict__ boff, int nsh,
                                              double* __restrict__ G, bool jonly, bool act, char* smem) {
    constexpr int SLAB = NC * ND, NS = NA * NB;
    constexpr int NBUF = scat_nbuf(NA, NB, NC, ND, (int)sizeof(E));
    constexpr int NI = NB + NC + ND;                 // outputs of one i: J_ab, K_ac, K_ad
    constexpr int NF = NC * ND + NB * NC + NB * ND;  // and at the end: J_cd, K_bc, K_bd
    static_assert((NBUF * SLAB + NB * (NC + ND)) * 32 >= NF * WST, "the last outputs fit the freed buffers");
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    char* mine = smem + wp * (scat_warp_elems(NBUF, NB, NC, ND) * (int)sizeof(E) + NBASE * 4);
    E* wb = reinterpret_cast<E*>(mine + NBASE * 4);  // the warp's buffers
    int* base = reinterpret_cast<int*>(mine);
    // density blocks in shell-pair order (row-major within a block), so each
    // row a thread reads is contiguous instead of one access per column
    const double* __restrict__ Bab = Pb + __ldg(boff + bra.sa * nsh + bra.sb);
    const double* __restrict__ Bac = Pb + __ldg(boff + bra.sa * nsh + ket.sa);
    const double* __restrict__ Bad = Pb + __ldg(boff + bra.sa * nsh + ket.sb);
    const double* __restrict__ Bbc = Pb + __ldg(boff + bra.sb * nsh + ket.sa);
    const double* __restrict__ Bbd = Pb + __ldg(boff + bra.sb * nsh + ket.sb);
    const double* __restrict__ Bcd = Pb + __ldg(boff + ket.sa * nsh + ket.sb);
    E* eb = wb + lane;                       // [NBUF][SLAB][32], this lane's column
    E* pk = wb + NBUF * SLAB * 32 + lane;    // [NB*NC] P_bc then [NB*ND] P_bd
    auto issue = [&](int slab) {
        if (slab < NS) {
            const E* src = e + (size_t)slab * SLAB * st;
            E* dst = eb + (slab % NBUF) * SLAB * 32;
#pragma unroll
            for (int r = 0; r < SLAB; ++r) cp_async_elem(dst + r * 32, src + (size_t)r * st);
        }
        cp_async_commit();  // empty groups keep the count uniform
    };
#pragma unroll
    for (int q = 0; q < NBUF - 1; ++q) issue(q);
    set_bases(base, boff, nsh, bra, ket, act);
#pragma unroll
    for (int j = 0; j < NB; ++j) {
#pragma unroll
        for (int k = 0; k < NC; ++k) pk[(j * NC + k) * 32] = (E)__ldg(Bbc + j * NC + k);
#pragma unroll
        for (int l = 0; l < ND; ++l) pk[(NB * NC + j * ND + l) * 32] = (E)__ldg(Bbd + j * ND + l);
    }
    const E s2 = (E)(2.0 * s), hs = (E)(-0.5 * s);
    E jcd[NC * ND], kbc[NB * NC], kbd[NB * ND], pcd[NC * ND];
#pragma unroll
    for (int x = 0; x < NC * ND; ++x) jcd[x] = 0;
#pragma unroll
    for (int x = 0; x < NB * NC; ++x) kbc[x] = 0;
#pragma unroll
    for (int x = 0; x < NB * ND; ++x) kbd[x] = 0;
#pragma unroll
    for (int k = 0; k < NC; ++k)
#pragma unroll
        for (int l = 0; l < ND; ++l) pcd[k * ND + l] = (E)__ldg(Bcd + k * ND + l);
#pragma unroll 1
    for (int i = 0; i < NA; ++i) {
        E jab[NB], kac[NC], kad[ND], pad_[ND], pac[NC];
#pragma unroll
        for (int j = 0; j < NB; ++j) jab[j] = 0;
#pragma unroll
        for (int k = 0; k < NC; ++k) {
            kac[k] = 0;
            pac[k] = (E)__ldg(Bac + i * NC + k);
        }
#pragma unroll
        for (int l = 0; l < ND; ++l) {
            kad[l] = 0;
            pad_[l] = (E)__ldg(Bad + i * ND + l);
        }
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            const int slab = i * NB + j;
            issue(slab + NBUF - 1);
            cp_async_wait<NBUF - 1>();  // this thread's copies of `slab` have landed
            const E* es = eb + (slab % NBUF) * SLAB * 32;
            const E pab = (E)__ldg(Bab + i * NB + j);
#pragma unroll
            for (int k = 0; k < NC; ++k) {
                const E pbc = pk[(j * NC + k) * 32];
#pragma unroll
                for (int l = 0; l < ND; ++l) {
                    const E v = es[(k * ND + l) * 32];
                    jab[j] += pcd[k * ND + l] * v;
                    jcd[k * ND + l] += pab * v;
                    if (!jonly) {
                        kac[k] += pk[(NB * NC + j * ND + l) * 32] * v;
                        kad[l] += pbc * v;
                        kbc[j * NC + k] += pad_[l] * v;
                        kbd[j * ND + l] += pac[k] * v;
                    }
                }
            }
        }
        // the outputs of this i through the slab just consumed (its next
        // copies are issued in the next iteration) or their own buffer
        E* tb = scat_over(NB, NC, ND) ? wb + (i * NB + NB - 1) % NBUF * SLAB * 32
                                      : wb + (NBUF * SLAB + NB * (NC + ND)) * 32;
        __syncwarp();
#pragma unroll
        for (int j = 0; j < NB; ++j) tb[j * WST + lane] = s2 * jab[j];
#pragma unroll
        for (int k = 0; k < NC; ++k) tb[(NB + k) * WST + lane] = hs * kac[k];
#pragma unroll
        for (int l = 0; l < ND; ++l) tb[(NB + NC + l) * WST + lane] = hs * kad[l];
        __syncwarp();
        walk_add<NI>(tb, base, jonly ? NB : NI, G, [&](int v, int& type, int& off) {
            type = v < NB ? 0 : v < NB + NC ? 2 : 3;
            off = v < NB ? i * NB + v : v < NB + NC ? i * NC + v - NB : i * ND + v - NB - NC;
        });
        __syncwarp();
    }
    cp_async_wait<0>();
    __syncwarp();
#pragma unroll
    for (int x = 0; x < NC * ND; ++x) wb[x * WST + lane] = s2 * jcd[x];
#pragma unroll
    for (int x = 0; x < NB * NC; ++x) wb[(NC * ND + x) * WST + lane] = hs * kbc[x];
#pragma unroll
    for (int x = 0; x < NB * ND; ++x) wb[(NC * ND + NB * NC + x) * WST + lane] = hs * kbd[x];
    __syncwarp();
    walk_add<NF>(wb, base, jonly ? NC * ND : NF, G, [&](int v, int& type, int& off) {
        type = v < NC * ND ? 1 : v < NC * ND + NB * NC ? 4 : 5;
        off = v - (v < NC * ND ? 0 : v < NC * ND + NB * NC ? NC * ND : NC * ND + NB * NC);
    });
}

// Post-screen (max |e| over all roles < thr, fock_build_non_diag.f90:69) and
// J/K scatter of a staged chunk, one thread per quartet.  E is the element
// type of the chunk's output rows (float for the FP32 chunks of staged2
// classes in the mixed form).
template <int NA, int NB, int NC, int ND, typename E = double>
__global__ void __launch_bounds__(ND_THREADS, sizeof(E) == 4 ? 3 : 2) k_scatter_staged(StagedArgs a) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int cnt = staged_count(a);
    const int w0 = t - (threadIdx.x & 31);  // first quartet of this warp
    if (w0 >= cnt) return;                  // a warp with no quartet (whole warps only)
    // every lane of the warp runs the scatter, because the lanes add the
    // warp's block elements together (walk_add); a lane past the end works on
    // the warp's first quartet and adds nothing
    const bool valid = t < cnt;
    const int tq = valid ? t : w0;
    double m = 0.0;
    const double* __restrict__ mxc = a.mx + tcol(tq, a.nroles);
    for (int r = 0; r < a.nroles; ++r) m = fmax(m, mxc[r * TQ]);
    const uint2 q = staged_quartet(a, tq);
    const GPair bra = a.bra[q.x];
    const GPair ket = a.ket[q.y];
    const bool act = valid && !(m < a.thr);  // fock_build_non_diag.f90:69
    const unsigned long long nsc = act ? 1ull : 0ull;
    const unsigned long long npr = valid ? (unsigned long long)(bra.np * ket.np) : 0ull;
    const double s = (bra.sa == bra.sb ? 0.5 : 1.0) * (ket.sa == ket.sb ? 0.5 : 1.0);
    extern __shared__ __align__(16) double hf_scat_smem[];
    scatter_async<NA, NB, NC, ND, E>(reinterpret_cast<const E*>(a.out) + tcol(tq, NA * NB * NC * ND), TQ, s, bra,
                                     ket, a.Pb, a.boff, a.nsh, a.G, a.jonly != 0, act,
                                     reinterpret_cast<char*>(hf_scat_smem));
    if (a.stats) warp_add_stats(a.stats, nsc, npr, a.f32 ? nsc : 0ull);
}

// Small chunks: one warp per quartet, its block in shared memory and the
// block elements over the lanes (scatter_lanes).  The one-thread scatter is a
// serial chain of 100-625 row loads; at a few hundred quartets that chain is
// the kernel's time (25-100 us), while this form takes a few us.  It reads
// each element six times from shared memory, so chunks that fill the SMs keep
// the one-thread form.
constexpr int WPB = ND_THREADS / 32;  // quartets per block
template <int NA, int NB, int NC, int ND, typename E>
__global__ void __launch_bounds__(ND_THREADS) k_scatter_warp(StagedArgs a) {
    constexpr int NOUT = NA * NB * NC * ND;
    __shared__ double sw[WPB][scatter_dens(NA, NB, NC, ND)];
    __shared__ E se[WPB][NOUT];
    const int wp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cnt = staged_count(a);
    unsigned long long nsc = 0, npr = 0;
    for (int t = blockIdx.x * WPB + wp; t < cnt; t += gridDim.x * WPB) {  // whole warps
        __syncwarp();  // the previous quartet's block has been read
        const E* __restrict__ src = reinterpret_cast<const E*>(a.out) + tcol(t, NOUT);
        for (int i = lane; i < NOUT; i += 32) se[wp][i] = src[(size_t)i * TQ];
        double m = 0.0;
        const double* __restrict__ mxc = a.mx + tcol(t, a.nroles);
        for (int r = lane; r < a.nroles; r += 32) m = fmax(m, mxc[r * TQ]);
        const uint2 q = staged_quartet(a, t);
        const GPair bra = a.bra[q.x];
        const GPair ket = a.ket[q.y];
        npr += bra.np * ket.np;
        if (!__any_sync(0xffffffffu, !(m < a.thr))) continue;  // fock_build_non_diag.f90:69
        ++nsc;
        const double s = (bra.sa == bra.sb ? 0.5 : 1.0) * (ket.sa == ket.sb ? 0.5 : 1.0);
        scatter_lanes<NA, NB, NC, ND>(se[wp], sw[wp], s, bra, ket, a.P, a.nb, BlockDst{a.G, a.boff, a.nsh},
                                      a.jonly != 0, lane, 32);
    }
    if (a.stats && lane == 0 && npr) {
        atomicAdd(&a.stats->prim, npr);
        if (nsc) atomicAdd(&a.stats->scattered, nsc);
        if (nsc && a.f32) atomicAdd(&a.stats->fp32, nsc);
    }
}

// Diagonal builders of a staged class (quartets (ab|ab), one warp per pair):
// MODE 0 writes the Schwarz factor sqrt(max|e|) (fock_build_initial_diag),
// MODE 1 applies the density screen schw^2 max(D_ab, D_aa/4, D_bb/4) < thr
// (fock_build_diag.f90:20-21); both skip elements with |e| <= 1e-10 and
// scatter with the weight (bra perms)^2/8.
template <int NA, int NB, int MODE>
__global__ void __launch_bounds__(ND_THREADS) k_scatter_diag(StagedArgs a) {
    constexpr int NOUT = NA * NB * NA * NB;
    __shared__ double sw[WPB][scatter_dens(NA, NB, NA, NB)], se[WPB][NOUT];
    const int wp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * WPB + wp;
    if (t >= staged_count(a)) return;
    const uint2 q = staged_quartet(a, t);
    const GPair pr = a.bra[q.x];
    if (MODE == 0) {
        double m = 0.0;
        for (int r = 0; r < a.nroles; ++r) m = fmax(m, a.mx[tcol(t, a.nroles) + r * TQ]);
        if (lane == 0) a.schw[q.x] = sqrt(m);
    } else if (diag_screened(pr, a.schw[q.x], a.md, a.nsh, a.thr)) {
        return;
    }
    const double* __restrict__ src = a.out + tcol(t, NOUT);
    for (int i = lane; i < NOUT; i += 32) {
        const double v = src[(size_t)i * TQ];
        se[wp][i] = fabs(v) > INTTHRESH ? v : 0.0;  // element skip
    }
    const double f = pr.sa == pr.sb ? 1.0 : 2.0;
    scatter_lanes<NA, NB, NA, NB>(se[wp], sw[wp], f * f / 8.0, pr, pr, a.P, a.nb, BlockDst{a.G, a.boff, a.nsh}, false,
                                  lane, 32);
}

typedef void (*NDKernel)(NDArgs);
typedef void (*NDAllKernel)(const NDAllArgs);
typedef void (*DiagKernel)(DiagArgs);
typedef void (*StagedKernel)(StagedArgs);
constexpr int MAXR = 64;

// Kernels of one quartet class, filled by the class's translation unit.
// mode 0: direct (nd64/nd32); 1: staged output roles (sb*); 2: staged
// accumulator roles (sa*) then output roles (sb*).  All staged classes end
// with scat.
struct ClassKernels {
    int mode;
    NDKernel nd64, nd32;
    DiagKernel diag0, diag1;  // only for classes (X|X)
    int nacc, nrole_a, nrole_b;
    int nrole_b32;            // output roles of the FP32 chunks (staged2: larger roles)
    int nrole_a32;            // accumulator roles of the FP32 chunks (staged3: larger groups)
    StagedKernel sa64[MAXR], sa32[MAXR], sb64[MAXR], sb32[MAXR], scat;
    StagedKernel dscat0, dscat1;  // staged diagonal builders (classes (X|X))
    int scat_smem;                // dynamic shared memory of scat (bytes)
    StagedKernel scat32;          // scatter of FP32 chunks (float rows), or nullptr
    int scat32_smem;
    StagedKernel scatw, scatw32;  // small chunks: one warp per quartet
    // every role of a stage in one launch (gridDim.y = roles), for small
    // chunks; the primitive-loop stages (ma, and mb of mode 1) run on work units
    StagedKernel ma64, ma32;      // stage-A roles (staged3)
    StagedKernel mb64, mb32;      // output / HRR roles
    int bi, ki, L, nout;
};

}  // namespace hfgpu
