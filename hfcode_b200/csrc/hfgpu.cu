// B200 (sm_100a) direct-SCF Fock builder: device kernels and the C ABI.
//
// Replaces the reference's fock_build_initial_diag / fock_build_diag /
// fock_build_non_diag (+ _j_only) subroutines (brichjnh/hfcode, Fortran +
// OpenMP) with CUDA kernels that keep every piece of state resident in HBM:
//
//   k_maxdm        evaluate_maxdm.f90:1-101 -- max |P| per shell-pair block
//                  (incl. the reference's d-l block choice, evaluate_maxdm.f90:82-89)
//   k_diag<C,M>    fock_build_initial_diag.f90 (M=0: Schwarz factors, element
//                  skip |e|>1e-10) and fock_build_diag.f90 (M=1: density
//                  screen schw^2*max(D_ab,D_aa/4,D_bb/4) < thr)
//   k_screen       the per-quartet screen of fock_build_non_diag.f90:63-67
//                  (schw_ab*schw_cd*max(Dcoul,Dexch/4) < thr), evaluated once
//                  for every candidate pair of active shell pairs, as bit masks;
//                  k_expand turns them into per-class quartet lists in order
//   k_offsets      list offsets and work units: how many lanes share a quartet
//   k_nondiag<C>   the work units of a direct class: contracted (ab|cd) from
//                  the generated class function, the post-screen max|e| < thr
//                  (fock_build_non_diag.f90:69), then the J/K scatter with FP64
//                  atomics into a one-triangle buffer G in shell-pair blocks
//   k_symm         F += G + G^T (the reference writes both triangles)
//
// The reference's per-case scatter branches (aa|aa), (aa|bc), (ab|cd), ...
// (fock_build_non_diag.f90:70-117 and 45 more blocks) all add the standard
// RHF J - K/2 contribution of each unique AO quartet; here every ordered
// component of a shell quartet carries the quartet's uniform degeneracy weight
// s = (bra perms)(ket perms)(bra-ket perms)/8, which sums to the same F.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <numeric>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/hfgpu.h"
#include "common.cuh"
#include "generated/class_table.inc"
#include "pairs.hpp"

namespace hfgpu {
#define HF_DECL_REG(ci) void register_class_##ci(ClassKernels* k);
HF_FOR_EACH_CLASS(HF_DECL_REG)
#undef HF_DECL_REG
NDAllKernel direct_all64();
NDAllKernel direct_all32();
static_assert(HF_NPT == NPT && HF_NCLS == NCLS, "generated class table out of date");
}  // namespace hfgpu

using namespace hfgpu;

namespace {

thread_local std::string g_err;

// CUDA forbids device-synchronising calls (cudaMalloc/cudaFree/
// cudaDeviceSynchronize/synchronous copies) in one thread while another
// thread records a stream capture.  Handles live in different threads when
// jobs are served concurrently, so captures and every such call of this
// library take this lock.
std::recursive_mutex g_dev_mu;
#define HF_DEVICE_LOCK std::lock_guard<std::recursive_mutex> dev_lock_(g_dev_mu)
}  // namespace

namespace hfgpu {
// error text for entry points in other translation units (onee.cu)
void set_last_error(const std::string& msg) { g_err = msg; }
std::recursive_mutex& device_mutex() { return g_dev_mu; }

// The library's stream-ordered memory pool on the current device, created
// on first use with no release threshold: memory a finished handle or job
// frees stays in the pool for the next one instead of going back to the
// driver at every synchronisation (which would map it again for the next
// served job).  It is released when the process exits.
cudaMemPool_t memory_pool() {
    static std::mutex mu;
    static cudaMemPool_t pools[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lk(mu);
    if (!pools[dev]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) return nullptr;
        unsigned long long keep = ~0ull;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        pools[dev] = pool;
    }
    return pools[dev];
}

cudaError_t pool_alloc(void** p, size_t bytes, cudaStream_t st) {
    cudaMemPool_t pool = memory_pool();
    if (!pool) return cudaMallocAsync(p, bytes, st);
    return cudaMallocFromPoolAsync(p, bytes, pool, st);
}
}  // namespace hfgpu

namespace {

#define HF_CHECK(call)                                                                   \
    do {                                                                                 \
        cudaError_t e_ = (call);                                                         \
        if (e_ != cudaSuccess) {                                                         \
            g_err = std::string(#call) + ": " + cudaGetErrorString(e_);                  \
            return HFGPU_ERR_CUDA;                                                       \
        }                                                                                \
    } while (0)

constexpr double SHTHRESH = 1e-11;      // molprops.f90:163
constexpr int NSTREAM = 8;              // class streams a handle creates (HFGPU_STREAMS of them used, default 4)
// bra and ket pair types of the quartet classes, in the generator's class order
__constant__ int CLS_BI[NCLS] = {HF_CLASS_BI_LIST};
__constant__ int CLS_KI[NCLS] = {HF_CLASS_KI_LIST};

// evaluate_maxdm.f90: one thread per unordered shell pair.
__global__ void k_maxdm(const int* __restrict__ shtyp, const int* __restrict__ aosh, int nsh, int nb,
                        const double* __restrict__ P, double* __restrict__ md) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long npair = (long long)nsh * (nsh + 1) / 2;
    if (t >= npair) return;
    int a = (int)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
    while ((long long)a * (a + 1) / 2 > t) --a;
    while ((long long)(a + 1) * (a + 2) / 2 <= t) ++a;
    const int b = (int)(t - (long long)a * (a + 1) / 2);
    auto rank = [](int ty) { return ty == 1 ? 0 : ty == 2 ? 1 : ty == 3 ? 2 : 3; };
    auto nf = [](int ty) { return ty == 1 ? 1 : ty == 2 ? 3 : ty == 3 ? 5 : 4; };
    int r = a, c = b;  // the reference's list orientation: lower rank first
    if (rank(shtyp[r]) > rank(shtyp[c])) { int x = r; r = c; c = x; }
    int nr = nf(shtyp[r]), nc = nf(shtyp[c]);
    if (shtyp[r] == 3 && shtyp[c] == 12) { nr = 4; nc = 5; }  // evaluate_maxdm.f90:82-89
    const int r0 = aosh[r], c0 = aosh[c];
    double m = 0.0;
    for (int i = 0; i < nr; ++i)
        for (int j = 0; j < nc; ++j) {
            const int row = r0 + i, col = c0 + j;
            if (row < nb && col < nb) m = fmax(m, fabs(P[row + (size_t)col * nb]));
        }
    md[(size_t)a * nsh + b] = m;
    md[(size_t)b * nsh + a] = m;
}

// Screening tiles: `tw` words of 32 consecutive candidates of one sub-class,
// one warp's work, a word at a time.  Large systems take 64 words (a lane
// keeps two mask words); small ones fewer, so that there are warps enough:
// with 64 words (H2O)12 has 2200 tiles, 15 warps per SM, each a serial chain
// (60 us, the whole screen's time).
constexpr int TWORDS_MAX = 64, TWORDS_MIN = 8;

struct ScreenArgs {
    const ScreenSub* subs;
    int nsub;
    int ntile;
    int tw;                   // words per tile
    const int2* sh[NPT];      // (sa, sb) per active pair, per pair type
    const double* schw[NPT];  // Schwarz factor per active pair
    const double* md;
    int nsh;
    double thr;
    int jonly;
    double f32cut;
    unsigned long long* cnt;  // [2*nsub] survivors per sub-class (FP64, FP32)
    TileEntries* tcnt;        // [ntile] survivors per tile; after k_offsets the entries before it in its sub-class
    unsigned* mask;           // [tw] survivors per tile, then (f32cut > 0) the FP32 ones of every tile
    uint2* qbuf;
};

// The sub-class of a tile: the last one whose first tile is <= t.
__device__ __forceinline__ int tile_sub(const ScreenArgs& a, int t) {
    int lo = 0, hi = a.nsub - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (a.subs[mid].tile0 <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Candidate u of a sub-class as (bra, ket) within its two groups, row by row.
__device__ __forceinline__ void candidate(const ScreenSub& S, long long u, int& i, int& j) {
    long long r;
    if (S.same) {
        r = (long long)((1.0 + sqrt(1.0 + 8.0 * (double)u)) * 0.5);
        while (r * (r - 1) / 2 > u) --r;
        while ((r + 1) * r / 2 <= u) ++r;
        j = (int)(u - r * (r - 1) / 2);
    } else {
        r = u / S.nket;
        j = (int)(u - r * S.nket);
    }
    i = (int)r;
}

// 32 candidates further.
__device__ __forceinline__ void advance(const ScreenSub& S, int& i, int& j) {
    j += 32;
    if (S.same) {
        while (j >= i) j -= i++;
    } else if (S.nket >= 32) {
        if (j >= S.nket) {
            j -= S.nket;
            ++i;
        }
    } else {
        i += j / S.nket;
        j %= S.nket;
    }
}

// Per-quartet screen of fock_build_non_diag.f90:63-67 over every candidate
// pair of active shell pairs, one warp per tile: the survivors as a bit mask
// and their counts.  Bound by the five density gathers of a candidate (L1);
// one search and one division per tile instead of one per 32 candidates, and
// a second pass that expands the masks instead of screening again, took the
// two passes from 1.71 + 1.98 ms to 0.85 + 0.19 ms on C60 (4.2e8 candidates).
__global__ void __launch_bounds__(256) k_screen(ScreenArgs a) {
    const int lane = threadIdx.x & 31;
    const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (t >= a.ntile) return;
    const int c = tile_sub(a, t);
    const ScreenSub S = a.subs[c];
    const int bi = CLS_BI[S.cls], ki = CLS_KI[S.cls];
    const long long u0 = (long long)(t - S.tile0) * (32 * a.tw);
    const int left = (int)min((long long)(32 * a.tw), S.ncand - u0), words = (left + 31) >> 5;
    const int2* __restrict__ bsh = a.sh[bi] + S.b0;
    const int2* __restrict__ ksh = a.sh[ki] + S.k0;
    const double* __restrict__ bsw = a.schw[bi] + S.b0;
    const double* __restrict__ ksw = a.schw[ki] + S.k0;
    const double* __restrict__ md = a.md;
    const int nsh = a.nsh;
    int i, j;
    candidate(S, u0 + lane, i, j);
    unsigned m[2] = {0, 0}, lo[2] = {0, 0};  // words lane and lane + 32
    for (int w = 0; w < words; ++w) {
        bool pass = false, low = false;
        if (w * 32 + lane < left) {
            const int2 ab = __ldg(bsh + i), cd = __ldg(ksh + j);
            double v = fmax(__ldg(md + ab.x * nsh + ab.y), __ldg(md + cd.x * nsh + cd.y));
            if (!a.jonly) {
                const double* __restrict__ ra = md + ab.x * nsh;
                const double* __restrict__ rb = md + ab.y * nsh;
                const double dx = fmax(fmax(__ldg(ra + cd.x), __ldg(ra + cd.y)),
                                       fmax(__ldg(rb + cd.x), __ldg(rb + cd.y)));
                v = fmax(v, 0.25 * dx);
            }
            const double bound = __ldg(bsw + i) * __ldg(ksw + j) * v;
            pass = !(bound < a.thr);
            low = pass && bound < a.f32cut;
        }
        const unsigned mw = __ballot_sync(0xffffffffu, pass), lw = __ballot_sync(0xffffffffu, low);
        if (lane == (w & 31)) {
            if (w < 32) m[0] = mw, lo[0] = lw;
            else m[1] = mw, lo[1] = lw;
        }
        advance(S, i, j);
    }
    const size_t at = (size_t)t * a.tw + lane;
    unsigned* ml = a.mask + (size_t)a.ntile * a.tw;
    for (int x = 0; x < 2; ++x)
        if (lane + 32 * x < a.tw) {
            a.mask[at + 32 * x] = m[x];
            if (a.f32cut > 0.0) ml[at + 32 * x] = lo[x];
        }
    int n32 = __popc(lo[0]) + __popc(lo[1]), n64 = __popc(m[0]) + __popc(m[1]) - n32;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        n64 += __shfl_xor_sync(0xffffffffu, n64, o);
        n32 += __shfl_xor_sync(0xffffffffu, n32, o);
    }
    if (lane == 0) a.tcnt[t] = TileEntries{n64, n32};
    if (lane == 0 && n64) atomicAdd(&a.cnt[2 * c], (unsigned long long)n64);
    if (lane == 1 && n32) atomicAdd(&a.cnt[2 * c + 1], (unsigned long long)n32);
}

// The compacted lists from the masks, one warp per tile.  The entries of a
// sub-class are in candidate order: a warp's 32 quartets share their bra pair
// and mostly the ket's first shell.
__global__ void __launch_bounds__(256) k_expand(ScreenArgs a) {
    const int lane = threadIdx.x & 31;
    const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (t >= a.ntile) return;
    const size_t at = (size_t)t * a.tw + lane;
    const unsigned* ml = a.mask + (size_t)a.ntile * a.tw;
    unsigned m[2] = {0, 0}, lo[2] = {0, 0};
    for (int x = 0; x < 2; ++x)
        if (lane + 32 * x < a.tw) {
            m[x] = a.mask[at + 32 * x];
            if (a.f32cut > 0.0) lo[x] = ml[at + 32 * x];
        }
    if (!__any_sync(0xffffffffu, m[0] | m[1])) return;
    const int c = tile_sub(a, t);
    const ScreenSub S = a.subs[c];
    const long long u0 = (long long)(t - S.tile0) * (32 * a.tw);
    const TileEntries before = a.tcnt[t];
    long long o64 = S.off[0] + before.n64, o32 = S.off[1] + before.n32;
    int i, j;
    candidate(S, u0 + lane, i, j);
    const int words = (int)((min((long long)(32 * a.tw), S.ncand - u0) + 31) >> 5);
    const unsigned lt = (1u << lane) - 1u;
    for (int w = 0; w < words; ++w) {
        const unsigned mw = __shfl_sync(0xffffffffu, w < 32 ? m[0] : m[1], w & 31);
        const unsigned lw = __shfl_sync(0xffffffffu, w < 32 ? lo[0] : lo[1], w & 31), hw = mw & ~lw;
        if (mw >> lane & 1) {
            const uint2 q = make_uint2((unsigned)(S.b0 + i), (unsigned)(S.k0 + j));
            if (lw >> lane & 1) a.qbuf[o32 + __popc(lw & lt)] = q;
            else a.qbuf[o64 + __popc(hw & lt)] = q;
        }
        o64 += __popc(hw);
        o32 += __popc(lw);
        advance(S, i, j);
    }
}

// Sub-class ranges and list regions of the classes (fixed after the Schwarz
// pass), passed by value to k_offsets.
struct OffsetArgs {
    int csub[NCLS + 1];      // sub-classes of class c: [csub[c], csub[c+1])
    long long coff[NCLS];    // first entry of class c in the quartet buffer
    float fill[NCLS][2];     // threads that fill the GPU with this class's kernel, per role (FP64, FP32)
    int lmin[NCLS];          // fewest primitive quartets a lane is given
    int tw;                  // words per screening tile
};

__device__ __forceinline__ long long warp_scan(long long v, int lane) {  // inclusive
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long x = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += x;
    }
    return v;
}

// Write offsets of the compacted lists from the screen's counts, on the device
// so that a build needs no host round trip: per class its FP64 entries, then
// its FP32 entries, sub-classes in order.  Also stores the per-class totals
// that the class kernels read, and cuts each list into work units (see Unit):
// a quartet is spread over as many lanes as it takes for a lane's share of
// its primitive loops to be near the class's primitive work over the threads
// that fill the GPU, and at least lmin.  A class that fills the GPU anyway
// keeps one lane per quartet.  The first NCLS blocks take one class each (one
// warp); the others turn the tile counts of one sub-class each into the
// entries before the tile.
__global__ void __launch_bounds__(OFF_THREADS) k_offsets(OffsetArgs o, ScreenSub* __restrict__ subs,
                                                         const unsigned long long* __restrict__ cnt,
                                                         TileEntries* __restrict__ tcnt,
                                                         unsigned long long* __restrict__ ncls,
                                                         int* __restrict__ nunit) {
    const int c = blockIdx.x, lane = threadIdx.x;
    if (c >= NCLS) {
        const ScreenSub& S = subs[c - NCLS];
        scan_tiles(tcnt + S.tile0, (int)((S.ncand + 32 * o.tw - 1) / (32 * o.tw)));
        return;
    }
    if (lane >= 32) return;
    const int k0 = o.csub[c], k1 = o.csub[c + 1];
    long long n[2] = {0, 0};
    double work[2] = {0.0, 0.0};
    for (int k = k0 + lane; k < k1; k += 32)
        for (int p = 0; p < 2; ++p) {
            const long long m = (long long)cnt[2 * k + p];
            n[p] += m;
            work[p] += (double)m * (subs[k].npb * subs[k].npk);
        }
    for (int p = 0; p < 2; ++p)
        for (int s = 16; s > 0; s >>= 1) {
            n[p] += __shfl_xor_sync(0xffffffffu, n[p], s);
            work[p] += __shfl_xor_sync(0xffffffffu, work[p], s);
        }
    long long at[2] = {o.coff[c], o.coff[c] + n[0]};
    long long unit[2] = {0, 0};
    for (int k = k0; k < k1; k += 32) {
        const int x = k + lane;
        for (int p = 0; p < 2; ++p) {
            const long long m = x < k1 ? (long long)cnt[2 * x + p] : 0;
            const double most = fmax((double)o.lmin[c], work[p] / (double)o.fill[c][p]);
            int lgb = 0, lgk = 0;
            if (x < k1) pick_lanes(subs[x].npb, subs[x].npk, (int)fmin(most, 1e6), lgb, lgk);
            const int per = 32 >> (lgb + lgk);
            const long long u = (m + per - 1) / per;
            const long long sm = warp_scan(m, lane), su = warp_scan(u, lane);
            if (x < k1) {
                subs[x].off[p] = at[p] + sm - m;
                subs[x].unit[p] = (int)(unit[p] + su - u);
                subs[x].lgb[p] = lgb;
                subs[x].lgk[p] = lgk;
            }
            at[p] += __shfl_sync(0xffffffffu, sm, 31);
            unit[p] += __shfl_sync(0xffffffffu, su, 31);
        }
    }
    if (lane < 2) {
        ncls[2 * c + lane] = (unsigned long long)(lane ? n[1] : n[0]);
        nunit[2 * c + lane] = (int)(lane ? unit[1] : unit[0]);
    }
}

// The density in shell-pair blocks: block (s1, s2) holds P[r][c] for the
// functions r of shell s1 and c of shell s2, row-major, at boff[s1*nsh+s2].
// Rows the scatter reads become contiguous (one element per column before).
__global__ void k_pblock(const double* __restrict__ P, double* __restrict__ Pb, const int2* __restrict__ aomap,
                         const int* __restrict__ nfsh, const int* __restrict__ boff, int nb, int nsh) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= (long long)nb * nb) return;
    const int r = (int)(t % nb), c = (int)(t / nb);
    const int2 mr = aomap[r], mc = aomap[c];  // (shell, function within the shell)
    Pb[boff[mr.x * nsh + mc.x] + mr.y * nfsh[mc.x] + mc.y] = P[t];
}

// FMA-chain throughput probe: 8 independent chains per thread so the FP64 and
// FP32 pipes, not latency, bound it.  Used to state the FP64/FP32 roofline.
template <typename T>
__global__ void k_fma_peak(T* out, int iters, T a, T b) {
    T x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = (T)(threadIdx.x + i);
    for (int it = 0; it < iters; ++it)
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = x[i] * a + b;
    T s = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += x[i];
    if (s == (T)-1.2345) out[0] = s;  // keeps the chains live
}

// F += G + G^T; G is in the shell-pair blocks of k_pblock.
__global__ void k_symm(double* __restrict__ F, const double* __restrict__ G, const int2* __restrict__ aomap,
                       const int* __restrict__ nfsh, const int* __restrict__ boff, int nb, int nsh) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= (long long)nb * nb) return;
    const int2 r = aomap[t % nb], c = aomap[t / nb];
    F[t] += G[boff[r.x * nsh + c.x] + r.y * nfsh[c.x] + c.y] + G[boff[c.x * nsh + r.x] + c.y * nfsh[r.x] + r.y];
}

// ------------------------------------------------------------- host ----
}  // namespace

struct hfgpu_handle {
    int nsh = 0, nb = 0, npairs = 0;
    std::vector<int> shtyp, nzet, aosh;
    std::vector<HostPair> pairs[NPT];     // all pairs per GPU type
    std::vector<int> refcount;            // pairs per reference class
    std::vector<double> schw[NPT];        // host copy, by pair index
    std::vector<int> last_ref;            // lastXX per reference class
    bool have_schwarz = false;
    int timing = 0;
    int device = 0;                       // the CUDA device current at hfgpu_init
    long long merge_blocks = 0;           // chunks up to this many role blocks run one launch per stage
    int nstreams = 4;                     // class streams the off-diagonal build uses (<= NSTREAM)
    cudaStream_t stream = nullptr;
    cudaStream_t aux[NSTREAM] = {};    // independent classes run concurrently on these
    cudaEvent_t fork = nullptr, join[NSTREAM] = {};
    // device
    int* d_shtyp = nullptr;
    int* d_aosh = nullptr;
    double* d_psoa = nullptr;      // all-pairs primitive arrays (SoA)
    PrimSoA psoa{};
    double* d_apsoa = nullptr;     // active lists' interleaved primitive arrays (SoA)
    PrimSoA apsoa{};
    std::vector<GPrim> hprims;     // host copy, all-pairs order
    GPair* d_pairs[NPT] = {};
    double* d_schw[NPT] = {};
    GPair* d_apairs[NPT] = {};
    int2* d_ash[NPT] = {};
    double* d_aschw[NPT] = {};
    int nact[NPT] = {};
    std::vector<int> act_np[NPT];
    double* d_boys = nullptr;
    float* d_boysf = nullptr;
    double* d_P = nullptr;
    double* d_F = nullptr;
    double* d_G = nullptr;
    double* d_md = nullptr;
    ScreenSub* d_subs = nullptr;
    std::vector<ScreenSub> hsubs;
    size_t subcap = 0;
    uint2* d_q = nullptr;
    size_t qcap = 0;
    double* d_scratch = nullptr;   // staged classes: accumulators, outputs, maxima
    uint2* d_diaglist[NPT] = {};   // (i, i) for every pair of a type: staged diagonal builders
    double* d_dscratch = nullptr;  // scratch of the staged diagonal builders
    size_t dstride[NPT] = {};
    size_t doff[NPT] = {};         // each staged type's part of d_dscratch (all 0 when they share it)
    bool dshared = false;
    size_t scratch_doubles = 0;
    size_t dscratch_doubles = 0;   // scratch of the staged diagonal builders
    size_t stride[NCLS] = {};      // quartets per chunk of each staged class
    size_t slot_doubles = 0;       // scratch per class stream
    size_t scratch_budget = 0;     // bytes; 0 = default (HFGPU_SCRATCH_MB, or 24 GiB capped at device memory / 6)
    size_t naprims = 0;            // primitive pairs of the active lists
    unsigned long long* d_cnt = nullptr;
    unsigned* d_mask = nullptr;    // survivor masks of the screening tiles (all, then the FP32 ones)
    TileEntries* d_tcnt = nullptr;  // survivors per tile
    size_t tilecap = 0, maskcap = 0;  // tiles and mask words the two hold
    ClassStats* d_stats = nullptr;
    // last build statistics
    double st_ms[NCLS] = {};
    int ntile = 0;                  // screening tiles
    long long ccap[NCLS] = {};      // candidates per class (upper bound of its list)
    long long coff[NCLS] = {};      // class region in the quartet buffer
    long long n64[NCLS] = {}, n32[NCLS] = {};
    int nunit[2 * NCLS] = {};       // work units of the last eager build
    cudaEvent_t ev[2 * NCLS + 2] = {};
    int nsm = 148;
    long long launches = 0;             // kernels enqueued by this handle (graph replays included)
    long long graph_launches = 0;       // kernels in the captured build
    OffsetArgs offs{};                  // sub-class ranges / list regions per class
    // [2 * NCLS] surviving quartets (FP64, FP32) per class, then as ints the work units
    unsigned long long* d_ncls = nullptr;
    long long direct_blocks = 0;        // direct classes of up to this many blocks together run in one launch
    long long warp_scatter = 0;         // chunks up to this many quartets use the one-warp-per-quartet scatter
    double* d_Pb = nullptr;             // density in shell-pair blocks (nb x nb)
    int* d_boff = nullptr;              // block offsets (nsh x nsh)
    int2* d_aomap = nullptr;            // per function: (shell, index within the shell)
    int* d_nfsh = nullptr;              // functions per shell
    cudaGraph_t graph = nullptr;        // captured full build (hfgpu_graph_capture)
    cudaGraphExec_t gexec = nullptr;
    const void* gkey_f = nullptr;       // what the capture was recorded with
    const void* gkey_p = nullptr;
    double gkey_thr[3] = {};
};

struct hfgpu_batch {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    std::vector<hfgpu_handle*> hs;  // launch accounting
};

namespace {

int set_err(int code, const std::string& msg) {
    g_err = msg;
    return code;
}

// Device buffers of a handle come from the library's stream-ordered pool on
// the handle's stream: cudaFreeAsync, unlike cudaFree, does not synchronise
// the whole device, so a served job that finishes does not stall the jobs
// still running on the GPU.  These calls need no lock: a capture in another
// thread (thread-local mode) is unaffected by them.
template <typename T>
int dalloc(T** p, size_t n, cudaStream_t st) {
    if (n == 0) n = 1;
    cudaError_t e = pool_alloc((void**)p, n * sizeof(T), st);
    if (e != cudaSuccess) {
        *p = nullptr;
        g_err = std::string("cudaMallocAsync: ") + cudaGetErrorString(e);
        return HFGPU_ERR_NOMEM;
    }
    return HFGPU_OK;
}

template <typename T>
void dfree(T*& p, cudaStream_t st) {
    if (p) cudaFreeAsync((void*)p, st);
    p = nullptr;
}

// class index of pair types (i <= j) in the generator's class order
int class_index(int i, int j) {
    static const int bi[NCLS] = {HF_CLASS_BI_LIST}, ki[NCLS] = {HF_CLASS_KI_LIST};
    for (int c = 0; c < NCLS; ++c)
        if (bi[c] == i && ki[c] == j) return c;
    return -1;
}

struct ClassTable {
    ClassKernels k[NCLS]{};
    ClassTable() {
#define HF_REG_PTR(ci) register_class_##ci,
        void (*reg[NCLS])(ClassKernels*) = {HF_FOR_EACH_CLASS(HF_REG_PTR)};
#undef HF_REG_PTR
        for (int c = 0; c < NCLS; ++c) {
            reg[c](&k[c]);
            // the staged scatter streams its rows through > 48 KB of shared memory
            if (k[c].scat && k[c].scat_smem > 0)
                cudaFuncSetAttribute(k[c].scat, cudaFuncAttributeMaxDynamicSharedMemorySize, k[c].scat_smem);
            if (k[c].scat32 && k[c].scat32_smem > 0)
                cudaFuncSetAttribute(k[c].scat32, cudaFuncAttributeMaxDynamicSharedMemorySize, k[c].scat32_smem);
            // The role kernels use no shared memory: they prefer the largest
            // L1 carve-out (HFGPU_CARVEOUT=<percent of shared memory> or
            // "none" overrides).  With the four class streams, where role and
            // scatter kernels of different classes share SMs, the C60 FP64
            // build measured 207.6 ms without the preference and 198.4 ms with
            // it; the class times alone are unchanged.  The same preference on
            // the scatters (shared memory first) or on the direct kernels (L1
            // first) measured slower (205.0 and 202.6 ms).
            int pct = 0;
            if (const char* e = getenv("HFGPU_CARVEOUT")) pct = strcmp(e, "none") == 0 ? -2 : atoi(e);
            auto pref = [](StagedKernel f, int v) {
                if (f && v >= -1) cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, v);
            };
            for (int r = 0; r < MAXR; ++r) {
                pref(k[c].sa64[r], pct);
                pref(k[c].sa32[r], pct);
                pref(k[c].sb64[r], pct);
                pref(k[c].sb32[r], pct);
            }
            pref(k[c].ma64, pct);
            pref(k[c].ma32, pct);
            pref(k[c].mb64, pct);
            pref(k[c].mb32, pct);
        }
    }
};
const ClassTable& class_table() {
    static ClassTable t;
    return t;
}
#define CLASS_KERNELS (class_table().k)

DiagKernel diag_kernel(int pt, int mode) {
    const ClassKernels& k = CLASS_KERNELS[class_index(pt, pt)];
    return mode ? k.diag1 : k.diag0;
}

size_t scratch_budget_doubles();

int upload_fp(hfgpu_handle* h, const double* f, const double* p) {
    size_t bytes = (size_t)h->nb * h->nb * sizeof(double);
    HF_CHECK(cudaMemcpyAsync(h->d_P, p, bytes, cudaMemcpyHostToDevice, h->stream));
    HF_CHECK(cudaMemcpyAsync(h->d_F, f, bytes, cudaMemcpyHostToDevice, h->stream));
    return HFGPU_OK;
}

int download_f(hfgpu_handle* h, double* f) {
    size_t bytes = (size_t)h->nb * h->nb * sizeof(double);
    HF_CHECK(cudaMemcpyAsync(f, h->d_F, bytes, cudaMemcpyDeviceToHost, h->stream));
    HF_CHECK(cudaStreamSynchronize(h->stream));
    return HFGPU_OK;
}

int launch_maxdm(hfgpu_handle* h, const double* P, double* md = nullptr) {
    long long np = (long long)h->nsh * (h->nsh + 1) / 2;
    int blocks = (int)((np + 255) / 256);
    ++h->launches;
    k_maxdm<<<blocks, 256, 0, h->stream>>>(h->d_shtyp, h->d_aosh, h->nsh, h->nb, P, md ? md : h->d_md);
    HF_CHECK(cudaGetLastError());
    return HFGPU_OK;
}

int launch_symm(hfgpu_handle* h, double* F, const double* G = nullptr) {
    long long n = (long long)h->nb * h->nb;
    ++h->launches;
    k_symm<<<(int)((n + 255) / 256), 256, 0, h->stream>>>(F, G ? G : h->d_G, h->d_aomap, h->d_nfsh, h->d_boff, h->nb,
                                                          h->nsh);
    HF_CHECK(cudaGetLastError());
    return HFGPU_OK;
}

// Whether a chunk runs every role of a stage in one launch (gridDim.y =
// roles): when all its role blocks together are at most the handle's
// merge_blocks (eight per SM).  Large chunks keep one launch per role, so that every warp on an SM
// runs the same role's code (these FP64 recursions are long straight-line
// programs, and an SM running several of them thrashes its instruction
// cache); small chunks gain more from filling the SMs and launching less.
bool merge_roles(const hfgpu_handle* h, int blocks, int roles) {
    return (long long)blocks * roles <= h->merge_blocks;
}

// Diagonal builder of a staged pair type: chunks of its pairs through the
// class's roles and k_scatter_diag.
int run_staged_diag(hfgpu_handle* h, int t, int mode, const double* P, double thr, double* G, const double* md,
                    cudaStream_t stream) {
    const ClassKernels& K = CLASS_KERNELS[class_index(t, t)];
    const long long n = (long long)h->pairs[t].size();
    const size_t st = h->dstride[t];
    for (long long q0 = 0; q0 < n; q0 += (long long)st) {
        const int m = (int)std::min<long long>((long long)st, n - q0);
        StagedArgs a{};
        a.quartets = h->d_diaglist[t];
        a.n = m;
        a.q0 = q0;
        a.ncls = nullptr;
        a.bra = h->d_pairs[t];
        a.ket = h->d_pairs[t];
        a.prims = h->psoa;
        a.boys = h->d_boys;
        a.boysf = h->d_boysf;
        double* const scratch = h->d_dscratch + h->doff[t];
        a.acc = scratch;
        a.out = scratch + (size_t)K.nacc * st;
        a.mx = scratch + (size_t)(K.nacc + K.nout) * st;
        a.stride = st;
        a.nroles = K.nrole_b;
        a.P = P;
        a.G = G;
        a.boff = h->d_boff;
        a.nb = h->nb;
        a.thr = thr;
        a.stats = nullptr;
        a.schw = h->d_schw[t];
        a.md = md;
        a.nsh = h->nsh;
        // every role of a stage in one launch, two pairs per warp in the
        // primitive-loop stage (stage_unit), then one warp per pair
        const int blocks = (m + ND_THREADS - 1) / ND_THREADS, units = (m + 1) / 2;
        if (K.nrole_a > 0) {
            ++h->launches;
            K.ma64<<<dim3(units, K.nrole_a), RB_THREADS, 0, stream>>>(a);
            HF_CHECK(cudaGetLastError());
        }
        ++h->launches;
        K.mb64<<<dim3(K.nrole_a > 0 ? blocks * RB_SCALE : units, K.nrole_b), RB_THREADS, 0, stream>>>(a);
        HF_CHECK(cudaGetLastError());
        ++h->launches;
        (mode ? K.dscat1 : K.dscat0)<<<(m + WPB - 1) / WPB, ND_THREADS, 0, stream>>>(a);
        HF_CHECK(cudaGetLastError());
    }
    return HFGPU_OK;
}

// Diagonal builder: the direct pair types on streams[0], the staged types on
// the next one, or with `spread` each on one of its own (not when they share
// their scratch).
int launch_diag(hfgpu_handle* h, int mode, const double* P, double thr, double* G, const double* md,
                const cudaStream_t* streams, int ns, bool spread) {
    int next = 0;
    for (int t = 0; t < NPT; ++t) {
        int n = (int)h->pairs[t].size();
        if (n == 0) continue;
        if (CLASS_KERNELS[class_index(t, t)].mode != 0) {
            if ((spread && !h->dshared) || next == 0) ++next;
            int rc = run_staged_diag(h, t, mode, P, thr, G, md, streams[next % ns]);
            if (rc) return rc;
            continue;
        }
        DiagArgs a{h->d_pairs[t], n, h->psoa, h->d_boys, h->d_schw[t], md, h->nsh, P, G, h->d_boff, h->nb, thr};
        ++h->launches;
        diag_kernel(t, mode)<<<(n + WPB - 1) / WPB, ND_THREADS, 0, streams[0]>>>(a);
        HF_CHECK(cudaGetLastError());
    }
    return HFGPU_OK;
}

// The diagonal builder on the class streams, forked from the handle's
// stream: on all of them when nothing else runs (`join`: they join back
// here), on two beside the screening of an off-diagonal build, which joins
// them at its end.
int fork_diag(hfgpu_handle* h, int mode, const double* P, double thr, bool join) {
    const int ns = join ? h->nstreams : std::min(2, h->nstreams);
    HF_CHECK(cudaEventRecord(h->fork, h->stream));
    for (int k = 0; k < ns; ++k) HF_CHECK(cudaStreamWaitEvent(h->aux[k], h->fork, 0));
    const int rc = launch_diag(h, mode, P, thr, h->d_G, h->d_md, h->aux, ns, join);
    if (rc || !join) return rc;
    for (int k = 0; k < ns; ++k) {
        HF_CHECK(cudaEventRecord(h->join[k], h->aux[k]));
        HF_CHECK(cudaStreamWaitEvent(h->stream, h->join[k], 0));
    }
    return HFGPU_OK;
}

// Default scratch budget: 24 GiB, at most a sixth of the device's memory.
// Larger chunks mean fewer role/scatter launches per class and shorter
// tails: C60 builds 226.3 ms at 6 GiB, 220.5 ms at 24 GiB.  A handle
// allocates only what its largest class list needs (the chunk stride is
// capped by the class capacity), so small molecules take far less.
size_t scratch_budget_doubles() {
    size_t mb = 24576;
    size_t freeb = 0, totalb = 0;
    if (cudaMemGetInfo(&freeb, &totalb) == cudaSuccess && totalb > 0)
        mb = std::min(mb, totalb / 6 / (1024 * 1024));
    if (const char* e = getenv("HFGPU_SCRATCH_MB")) {
        long v = atol(e);
        if (v > 0) mb = (size_t)v;
    }
    return mb * 1024 * 1024 / sizeof(double);
}

// Fewest primitive quartets per lane of a work unit: below these the sum of
// the accumulators over the lanes, and the recurrences past the loops that
// every lane then repeats, cost more than the shorter loops save.  Benzene on
// host arrays (direct / staged): 787 us at 3 / 2, 733 at 6 / 4, 684 at 12 / 8,
// 654 at 24 / 8; (H2O)12: 773, 742, 694, 670 us; eight molecules in one batch
// launch: 7.78, 7.50, 7.24, 7.02 ms (the last with half the threads in
// `fill`, which alone gave 7.36).
constexpr int LMIN_DIRECT = 24, LMIN_STAGED = 8;

// Schwarz ordering (index_sort + find_threshold) and the active pair arrays.
int build_active(hfgpu_handle* h) {
    // no library lock here: the allocations are stream-ordered, and holding
    // the lock across this function's stream synchronisations made the jobs
    // of a server queue behind one another's GPU work
    for (int t = 0; t < NPT; ++t) {
        int n = (int)h->pairs[t].size();
        h->schw[t].resize(n);
        if (n)
            HF_CHECK(cudaMemcpyAsync(h->schw[t].data(), h->d_schw[t], n * sizeof(double), cudaMemcpyDeviceToHost,
                                     h->stream));
    }
    HF_CHECK(cudaStreamSynchronize(h->stream));
    h->last_ref.assign(10, 0);
    long long total_q = 0;
    std::vector<GPrim> aprims;
    std::vector<GPair> aps[NPT];
    std::vector<int2> ashs[NPT];
    std::vector<double> ascs[NPT];
    for (int t = 0; t < NPT; ++t) {
        const int n = (int)h->pairs[t].size();
        // reference list order is refpos; pairs[t] is stored in that order
        std::vector<int> ord(n);
        std::iota(ord.begin(), ord.end(), 0);
        std::stable_sort(ord.begin(), ord.end(), [&](int x, int y) { return h->schw[t][x] > h->schw[t][y]; });
        int last = 0;
        if (n > 0) {
            if (h->schw[t][ord[0]] < SHTHRESH) last = 1;
            else if (h->schw[t][ord[n - 1]] > SHTHRESH) last = n;
            else {
                last = n;
                for (int i = 0; i < n; ++i)
                    if (h->schw[t][ord[i]] < SHTHRESH) { last = i + 1; break; }
            }
        }
        h->last_ref[GPU_TO_REF[t]] = last;
        // active set, re-ordered for the GPU: primitive count, first shell, then Schwarz
        std::vector<int> act(ord.begin(), ord.begin() + last);
        std::stable_sort(act.begin(), act.end(), [&](int x, int y) {
            int nx = h->pairs[t][x].g.np, ny = h->pairs[t][y].g.np;
            if (nx != ny) return nx > ny;
            // within a primitive-count group by first shell, so the 32
            // quartets of a warp mostly share it (the scatter adds the runs
            // of quartets that share a block with one atomic per element)
            const int sx = h->pairs[t][x].g.sa, sy = h->pairs[t][y].g.sa;
            if (sx != sy) return sx < sy;
            return h->schw[t][x] > h->schw[t][y];
        });
        std::vector<GPair> ap(last);
        std::vector<int2> ash(last);
        std::vector<double> asc(last);
        for (int i = 0; i < last; ++i) {
            ap[i] = h->pairs[t][act[i]].g;
            ash[i] = make_int2(ap[i].sa, ap[i].sb);
            asc[i] = h->schw[t][act[i]];
        }
        h->nact[t] = last;
        h->act_np[t].resize(last);
        for (int i = 0; i < last; ++i) h->act_np[t][i] = ap[i].np;
        // interleave the primitives of equal-count neighbours: entry ik of
        // pair i of a group [g0, g0+ng) goes to base + ik*ng + (i - g0)
        for (int i = 0; i < last;) {
            int j = i + 1;
            while (j < last && ap[j].np == ap[i].np) ++j;
            const int ng = j - i, np = ap[i].np;
            const size_t base = aprims.size();
            aprims.resize(base + (size_t)np * ng);
            for (int k = i; k < j; ++k) {
                for (int ik = 0; ik < np; ++ik) aprims[base + (size_t)ik * ng + (k - i)] = h->hprims[ap[k].p0 + ik];
                ap[k].p0 = (int)(base + (k - i));
                ap[k].ps = ng;
            }
            i = j;
        }
        aps[t] = std::move(ap);
        ashs[t] = std::move(ash);
        ascs[t] = std::move(asc);
    }
    {
        std::vector<double> soa = prims_soa(aprims);
        dfree(h->d_apsoa, h->stream);
        int rc = dalloc(&h->d_apsoa, std::max<size_t>(soa.size(), 1), h->stream);
        if (rc) return rc;
        h->apsoa = soa_view(h->d_apsoa, aprims.size());
        h->naprims = aprims.size();
        if (!soa.empty())
            HF_CHECK(cudaMemcpyAsync(h->d_apsoa, soa.data(), soa.size() * sizeof(double), cudaMemcpyHostToDevice,
                                     h->stream));
        for (int t = 0; t < NPT; ++t) {
            const int last = h->nact[t];
            if (!last) continue;
            HF_CHECK(cudaMemcpyAsync(h->d_apairs[t], aps[t].data(), last * sizeof(GPair), cudaMemcpyHostToDevice,
                                     h->stream));
            HF_CHECK(cudaMemcpyAsync(h->d_ash[t], ashs[t].data(), last * sizeof(int2), cudaMemcpyHostToDevice,
                                     h->stream));
            HF_CHECK(cudaMemcpyAsync(h->d_aschw[t], ascs[t].data(), last * sizeof(double), cudaMemcpyHostToDevice,
                                     h->stream));
        }
        HF_CHECK(cudaStreamSynchronize(h->stream));
    }
    // screening sub-classes: primitive-count groups of the active lists
    std::vector<std::pair<int, int>> groups[NPT];  // (start, length)
    for (int t = 0; t < NPT; ++t) {
        const int n = h->nact[t];
        for (int i = 0; i < n;) {
            int j = i + 1;
            while (j < n && h->act_np[t][j] == h->act_np[t][i]) ++j;
            groups[t].push_back({i, j - i});
            i = j;
        }
    }
    h->hsubs.clear();
    long long total_words = 0, qoff = 0;
    for (int c = 0; c < NCLS; ++c) {
        const int bi = CLASS_KERNELS[c].bi, ki = CLASS_KERNELS[c].ki;
        long long ccap = 0;
        for (size_t gb = 0; gb < groups[bi].size(); ++gb)
            for (size_t gk = 0; gk < groups[ki].size(); ++gk) {
                if (bi == ki && gk > gb) continue;  // pairs (ii, jj) with ii > jj only
                ScreenSub sub{};
                sub.cls = c;
                sub.same = (bi == ki && gb == gk);
                sub.b0 = groups[bi][gb].first;
                sub.nbra = groups[bi][gb].second;
                sub.k0 = groups[ki][gk].first;
                sub.nket = groups[ki][gk].second;
                sub.npb = h->act_np[bi][sub.b0];
                sub.npk = h->act_np[ki][sub.k0];
                sub.ncand = sub.same ? (long long)sub.nbra * (sub.nbra - 1) / 2 : (long long)sub.nbra * sub.nket;
                if (sub.ncand == 0) continue;
                total_words += (sub.ncand + 31) / 32;
                ccap += sub.ncand;
                h->hsubs.push_back(sub);
            }
        h->ccap[c] = ccap;
        h->coff[c] = qoff;
        h->offs.coff[c] = qoff;
        qoff += ccap;
        h->offs.csub[c + 1] = (int)h->hsubs.size();
        // threads that fill the GPU: 16 warps per SM of a direct kernel, 8 of
        // the 255-register role kernels, whose roles run side by side
        const ClassKernels& K = CLASS_KERNELS[c];
        for (int p = 0; p < 2; ++p) {
            const int roles = K.mode == 0 ? 1 : K.mode == 1 ? (p ? K.nrole_b32 : K.nrole_b)
                                                            : (p ? K.nrole_a32 : K.nrole_a);
            h->offs.fill[c][p] = (float)h->nsm * (K.mode == 0 ? 512.f : 256.f) / (float)roles;
        }
        h->offs.lmin[c] = K.mode == 0 ? LMIN_DIRECT : LMIN_STAGED;
    }
    h->offs.csub[0] = 0;
    // words per tile: the most that leaves 64 tiles per SM
    int tw = TWORDS_MAX;
    while (tw > TWORDS_MIN && total_words < 64LL * h->nsm * tw) tw /= 2;
    long long tiles = 0;
    for (ScreenSub& sub : h->hsubs) {
        sub.tile0 = (int)tiles;
        tiles += (sub.ncand + 32 * tw - 1) / (32 * tw);
    }
    h->offs.tw = tw;
    if (tiles > (1LL << 30)) return set_err(HFGPU_ERR_UNSUPPORTED, "too many candidate quartets");
    h->ntile = (int)tiles;
    total_q = qoff;
    if ((size_t)tiles > h->tilecap || (size_t)tiles * tw > h->maskcap) {
        dfree(h->d_mask, h->stream);
        dfree(h->d_tcnt, h->stream);
        h->tilecap = h->maskcap = 0;
        int rc = dalloc(&h->d_mask, 2 * (size_t)tiles * tw, h->stream);
        if (rc == HFGPU_OK) rc = dalloc(&h->d_tcnt, (size_t)tiles, h->stream);
        if (rc) return rc;
        h->tilecap = (size_t)tiles;
        h->maskcap = (size_t)tiles * tw;
    }
    if (h->hsubs.size() > h->subcap) {
        dfree(h->d_subs, h->stream);
        h->subcap = 0;
        int rc = dalloc(&h->d_subs, h->hsubs.size(), h->stream);
        if (rc) return rc;
        dfree(h->d_cnt, h->stream);
        rc = dalloc(&h->d_cnt, 2 * h->hsubs.size(), h->stream);
        if (rc) return rc;
        h->subcap = h->hsubs.size();
    }
    // the sub-class table stays on the device; k_offsets fills its offsets
    if (!h->hsubs.empty()) {
        HF_CHECK(cudaMemcpyAsync(h->d_subs, h->hsubs.data(), h->hsubs.size() * sizeof(ScreenSub),
                                 cudaMemcpyHostToDevice, h->stream));
        HF_CHECK(cudaStreamSynchronize(h->stream));
    }
    if ((size_t)total_q > h->qcap) {
        dfree(h->d_q, h->stream);
        h->qcap = 0;
        int rc = dalloc(&h->d_q, (size_t)total_q, h->stream);
        if (rc) return rc;
        h->qcap = (size_t)std::max<long long>(total_q, 1);
    }
    // scratch of the staged classes: one chunk of stride quartets holds
    // (accumulators + outputs + role maxima) doubles per quartet
    size_t need = 0;
    const size_t budget = (h->scratch_budget ? h->scratch_budget / sizeof(double) : scratch_budget_doubles()) /
                          h->nstreams;  // one slot per class stream
    for (int c = 0; c < NCLS; ++c) {
        const ClassKernels& K = CLASS_KERNELS[c];
        h->stride[c] = 0;
        if (K.mode == 0 || h->ccap[c] == 0) continue;
        const size_t per = (size_t)K.nacc + K.nout + std::max(K.nrole_b, K.nrole_b32);
        size_t st = std::min<size_t>((size_t)h->ccap[c], budget / per);
        st = (std::max<size_t>(st, TQ) + TQ - 1) / TQ * TQ;  // whole scratch tiles
        h->stride[c] = st;
        need = std::max(need, st * per);
    }
    if (need * h->nstreams > h->scratch_doubles) {
        dfree(h->d_scratch, h->stream);
        h->scratch_doubles = 0;
        int rc = dalloc(&h->d_scratch, need * h->nstreams, h->stream);
        if (rc) return rc;
        h->scratch_doubles = need * h->nstreams;
    }
    h->slot_doubles = need;
    h->have_schwarz = true;
    return HFGPU_OK;
}

// The work units of a class list, as the kernels take them.
UnitList unit_list(const hfgpu_handle* h, int c, int prec) {
    UnitList L{};
    L.subs = h->d_subs;
    L.cnt = h->d_cnt;
    L.ncls = h->d_ncls;
    L.nunit = reinterpret_cast<const int*>(h->d_ncls + 2 * NCLS);
    L.sub0 = h->offs.csub[c];
    L.sub1 = h->offs.csub[c + 1];
    L.coff = h->coff[c];
    L.quartets = h->d_q;
    L.cls = c;
    L.prec = prec;
    return L;
}

// Blocks along x of a kernel that walks its list: as many as the list needs
// where the count is on the host; in a capture, whose counts stay on the
// device, at most `fill` (idle blocks of a grid sized by the capacity cost
// about a nanosecond each, 0.1 ms for a class with many roles).
unsigned walk_blocks(long long need, long long fill, bool capture) {
    return (unsigned)std::max<long long>(1, capture ? std::min(need, fill) : need);
}

// Blocks of a direct class's list of n quartets; in a capture an upper bound,
// from the candidates.  direct_grid is what is launched.
long long direct_need(const hfgpu_handle* h, int c, int prec, long long n, bool capture) {
    return ((capture ? n : h->nunit[2 * c + prec]) + WPB - 1) / WPB;
}
unsigned direct_grid(const hfgpu_handle* h, int c, int prec, long long n, bool capture) {
    return walk_blocks(direct_need(h, c, prec, n, capture), 8LL * h->nsm, capture);
}

// Staged class: chunks of the quartet list through the accumulator roles
// (mode 2), the output roles and the scatter kernel.
int run_staged(hfgpu_handle* h, int c, int prec, long long n, const double* P, double thr, int jonly,
               cudaStream_t stream, double* scratch, bool capture) {
    const ClassKernels& K = CLASS_KERNELS[c];
    const size_t st = h->stride[c];
    for (long long q0 = 0; q0 < n; q0 += (long long)st) {
        const int m = (int)std::min<long long>((long long)st, n - q0);
        StagedArgs a{};
        a.quartets = h->d_q + h->coff[c];
        a.n = m;  // the kernels clamp it by the device-side count
        a.q0 = q0;
        a.ncls = h->d_ncls;
        a.cls = c;
        a.prec = prec;
        a.bra = h->d_apairs[K.bi];
        a.ket = h->d_apairs[K.ki];
        a.prims = h->apsoa;
        a.boys = h->d_boys;
        a.boysf = h->d_boysf;
        a.acc = scratch;
        a.out = scratch + (size_t)K.nacc * st;
        a.mx = scratch + (size_t)(K.nacc + K.nout) * st;
        a.stride = st;
        a.nroles = prec ? K.nrole_b32 : K.nrole_b;
        a.P = P;
        a.Pb = h->d_Pb;
        a.boff = h->d_boff;
        a.nsh = h->nsh;
        a.G = h->d_G;
        a.nb = h->nb;
        a.thr = thr;
        a.jonly = jonly;
        a.f32 = prec;
        a.stats = h->d_stats + c;
        const int blocks = (m + ND_THREADS - 1) / ND_THREADS;
        const int na = prec ? K.nrole_a32 : K.nrole_a;
        if (merge_roles(h, blocks, std::max(na, a.nroles))) {
            // a small list: every role of a stage in one launch, side by side,
            // the primitive-loop stage on the class's work units
            a.list = unit_list(h, c, prec);
            // a unit holds at least one quartet, so m bounds the units; two
            // rounds of the eight resident warps per SM in a capture
            const int nr = std::max(na, a.nroles);
            const long long fill = (16LL * h->nsm + nr - 1) / nr;
            const long long need = capture ? m : (long long)h->nunit[2 * c + prec] * m / n + 32;  // this chunk's share
            const unsigned units = walk_blocks(std::min<long long>(m, need), fill, capture);
            const unsigned hblocks = walk_blocks((long long)blocks * RB_SCALE, fill, capture);
            if (na > 0) {
                ++h->launches;
                (prec ? K.ma32 : K.ma64)<<<dim3(units, na), RB_THREADS, 0, stream>>>(a);
                HF_CHECK(cudaGetLastError());
            }
            ++h->launches;
            (prec ? K.mb32 : K.mb64)<<<dim3(na > 0 ? hblocks : units, a.nroles), RB_THREADS, 0, stream>>>(a);
            HF_CHECK(cudaGetLastError());
        } else {
            for (int r = 0; r < na; ++r) {
                ++h->launches;
                (prec ? K.sa32[r] : K.sa64[r])<<<blocks * RB_SCALE, RB_THREADS, 0, stream>>>(a);
                HF_CHECK(cudaGetLastError());
            }
            for (int r = 0; r < a.nroles; ++r) {
                ++h->launches;
                (prec ? K.sb32[r] : K.sb64[r])<<<blocks * RB_SCALE, RB_THREADS, 0, stream>>>(a);
                HF_CHECK(cudaGetLastError());
            }
        }
        ++h->launches;
        if (m <= h->warp_scatter) {  // one warp per quartet
            const unsigned wblocks = walk_blocks((m + WPB - 1) / WPB, 8LL * h->nsm, capture);
            (prec ? K.scatw32 : K.scatw)<<<wblocks, ND_THREADS, 0, stream>>>(a);
        } else if (prec && K.scat32) {
            K.scat32<<<blocks, ND_THREADS, K.scat32_smem, stream>>>(a);  // float rows
        } else {
            K.scat<<<blocks, ND_THREADS, K.scat_smem, stream>>>(a);
        }
        HF_CHECK(cudaGetLastError());
    }
    return HFGPU_OK;
}

// Off-diagonal build: the screen, the list offsets and the expansion into
// lists, then the class kernels on the handle's concurrent class streams.  With capture set,
// nothing is read back on the host: every launch is sized by the class's
// candidate count (an upper bound) and the kernels read the surviving count
// from d_ncls, so the whole sequence can be recorded into a CUDA graph.
// Eager builds read the counts back once to size the launches exactly.
int run_non_diag(hfgpu_handle* h, const double* P, double thr, int jonly, double f32cut, bool capture = false) {
    if (!h->have_schwarz) return set_err(HFGPU_ERR_STATE, "fock_build_initial_diag has not been called");
    HF_CHECK(cudaMemsetAsync(h->d_stats, 0, NCLS * sizeof(ClassStats), h->stream));
    HF_CHECK(cudaMemsetAsync(h->d_ncls, 0, 3 * NCLS * sizeof(unsigned long long), h->stream));
    const int nsub = (int)h->hsubs.size();
    for (int c = 0; c < NCLS; ++c) h->n64[c] = h->n32[c] = 0;
    if (h->ntile > 0 && nsub > 0) {
        ScreenArgs sa{};
        sa.subs = h->d_subs;
        sa.nsub = nsub;
        sa.ntile = h->ntile;
        sa.tw = h->offs.tw;
        for (int t = 0; t < NPT; ++t) {
            sa.sh[t] = h->d_ash[t];
            sa.schw[t] = h->d_aschw[t];
        }
        sa.md = h->d_md;
        sa.nsh = h->nsh;
        sa.thr = thr;
        sa.jonly = jonly;
        sa.f32cut = f32cut;
        sa.cnt = h->d_cnt;
        sa.tcnt = h->d_tcnt;
        sa.mask = h->d_mask;
        sa.qbuf = h->d_q;
        const int blocks = (h->ntile + 7) / 8;
        HF_CHECK(cudaMemsetAsync(h->d_cnt, 0, 2 * (size_t)nsub * sizeof(unsigned long long), h->stream));
        ++h->launches;
        k_screen<<<blocks, 256, 0, h->stream>>>(sa);  // survivor masks and counts
        HF_CHECK(cudaGetLastError());
        ++h->launches;
        k_offsets<<<NCLS + nsub, OFF_THREADS, 0, h->stream>>>(h->offs, h->d_subs, h->d_cnt, h->d_tcnt, h->d_ncls,
                                                              reinterpret_cast<int*>(h->d_ncls + 2 * NCLS));
        HF_CHECK(cudaGetLastError());
        ++h->launches;
        k_expand<<<blocks, 256, 0, h->stream>>>(sa);  // compacted write
        HF_CHECK(cudaGetLastError());
    }
    {  // the density in shell-pair blocks for the scatters
        const long long n = (long long)h->nb * h->nb;
        ++h->launches;
        k_pblock<<<(int)((n + 255) / 256), 256, 0, h->stream>>>(P, h->d_Pb, h->d_aomap, h->d_nfsh, h->d_boff, h->nb,
                                                                h->nsh);
        HF_CHECK(cudaGetLastError());
    }
    if (!capture) {
        unsigned long long cnt[3 * NCLS];
        HF_CHECK(cudaMemcpyAsync(cnt, h->d_ncls, sizeof(cnt), cudaMemcpyDeviceToHost, h->stream));
        HF_CHECK(cudaStreamSynchronize(h->stream));
        memcpy(h->nunit, cnt + 2 * NCLS, sizeof(h->nunit));
        for (int c = 0; c < NCLS; ++c) {
            h->n64[c] = (long long)cnt[2 * c];
            h->n32[c] = (long long)cnt[2 * c + 1];
        }
    }
    // work items (class, precision) over the class streams, largest
    // first onto the least-loaded stream; with timing on, everything runs in
    // order on the handle's stream
    struct Item { int c, prec; long long n; double w; };
    std::vector<Item> items;
    for (int c = 0; c < NCLS; ++c) {
        h->st_ms[c] = 0.0;
        for (int prec = 0; prec < 2; ++prec) {
            long long n = prec ? h->n32[c] : h->n64[c];
            if (capture) n = (prec && !(f32cut > 0.0)) ? 0 : h->ccap[c];
            if (n > 0) items.push_back({c, prec, n, (double)n * CLASS_KERNELS[c].nout});
        }
    }
    const bool multi = capture || !h->timing;
    if (multi) {
        std::stable_sort(items.begin(), items.end(), [](const Item& x, const Item& y) { return x.w > y.w; });
        HF_CHECK(cudaEventRecord(h->fork, h->stream));
        for (int k = 0; k < h->nstreams; ++k) HF_CHECK(cudaStreamWaitEvent(h->aux[k], h->fork, 0));
    }
    double load[NSTREAM] = {};
    // The direct classes of a small build side by side in one launch per
    // precision.  Small by the work, not by the grid: a capture's grids are
    // capped, and by those every build with few direct classes would be small
    // (C60 in STO-3G with split sp shells: 16.4 ms recorded in one launch,
    // 14.5-15.2 with a launch per class; n-C20H42 in STO-3G 0.52 and 0.48).
    long long direct_blocks = 0;
    for (const Item& it : items)
        if (CLASS_KERNELS[it.c].mode == 0) direct_blocks += direct_need(h, it.c, it.prec, it.n, capture);
    const bool one_launch = multi && direct_blocks <= h->direct_blocks;
    for (int prec = 0; one_launch && prec < 2; ++prec) {
        NDAllArgs a{};
        int blocks = 0;
        double w = 0.0;
        for (const Item& it : items) {
            const ClassKernels& K = CLASS_KERNELS[it.c];
            if (K.mode != 0 || it.prec != prec) continue;
            NDItem& d = a.item[a.nitem++];
            d.list = unit_list(h, it.c, prec);
            d.bra = h->d_apairs[K.bi];
            d.ket = h->d_apairs[K.ki];
            d.stats = h->d_stats + it.c;
            d.block0 = blocks;
            d.blocks = (int)direct_grid(h, it.c, prec, it.n, capture);
            blocks += d.blocks;
            w += it.w;
        }
        if (!a.nitem) continue;
        a.prims = h->apsoa;
        a.boys = h->d_boys;
        a.boysf = h->d_boysf;
        a.Pb = h->d_Pb;
        a.G = h->d_G;
        a.boff = h->d_boff;
        a.nsh = h->nsh;
        a.thr = thr;
        a.jonly = jonly;
        const int k = h->nstreams - 1 - prec % h->nstreams;  // first on its stream: it takes longest
        load[k] += w;
        ++h->launches;
        (prec ? direct_all32() : direct_all64())<<<blocks, ND_THREADS, 0, h->aux[k]>>>(a);
        HF_CHECK(cudaGetLastError());
    }
    for (const Item& it : items) {
        if (one_launch && CLASS_KERNELS[it.c].mode == 0) continue;
        const int c = it.c, prec = it.prec;
        const long long n = it.n;
        const ClassKernels& K = CLASS_KERNELS[c];
        int k = 0;
        for (int q = 1; q < h->nstreams; ++q)
            if (load[q] < load[k]) k = q;
        load[k] += it.w;
        cudaStream_t st = multi ? h->aux[k] : h->stream;
        double* slot = h->d_scratch ? h->d_scratch + (multi ? (size_t)k * h->slot_doubles : 0) : nullptr;
        const bool timed = h->timing && !multi;
        if (timed) HF_CHECK(cudaEventRecord(h->ev[2 * c], h->stream));
        if (K.mode == 0) {
            NDArgs a{};
            a.list = unit_list(h, c, prec);
            a.bra = h->d_apairs[K.bi];
            a.ket = h->d_apairs[K.ki];
            a.prims = h->apsoa;
            a.boys = h->d_boys;
            a.boysf = h->d_boysf;
            a.Pb = h->d_Pb;
            a.G = h->d_G;
            a.boff = h->d_boff;
            a.nsh = h->nsh;
            a.thr = thr;
            a.jonly = jonly;
            a.stats = h->d_stats + c;
            const unsigned blocks = direct_grid(h, c, prec, n, capture);
            ++h->launches;
            (prec ? K.nd32 : K.nd64)<<<blocks, ND_THREADS, 0, st>>>(a);
            HF_CHECK(cudaGetLastError());
        } else {
            int rc = run_staged(h, c, prec, n, P, thr, jonly, st, slot, capture);
            if (rc) return rc;
        }
        if (timed) {
            HF_CHECK(cudaEventRecord(h->ev[2 * c + 1], h->stream));
            HF_CHECK(cudaEventSynchronize(h->ev[2 * c + 1]));
            float ms = 0;
            cudaEventElapsedTime(&ms, h->ev[2 * c], h->ev[2 * c + 1]);
            h->st_ms[c] += ms;
        }
    }
    if (multi) {
        for (int k = 0; k < h->nstreams; ++k) {
            HF_CHECK(cudaEventRecord(h->join[k], h->aux[k]));
            HF_CHECK(cudaStreamWaitEvent(h->stream, h->join[k], 0));
        }
    }
    return HFGPU_OK;
}

}  // namespace

extern "C" {

const char* hfgpu_last_error(void) { return g_err.c_str(); }

int hfgpu_init(const hfgpu_basis* B, hfgpu_handle** out) {
    if (!B || !out || B->nsh <= 0 || B->nb <= 0 || B->maxprim <= 0)
        return set_err(HFGPU_ERR_ARG, "hfgpu_init: bad arguments");
    *out = nullptr;
    hfgpu_handle* h = new hfgpu_handle();
    h->nsh = B->nsh;
    h->nb = B->nb;
    h->shtyp.assign(B->shtyp, B->shtyp + B->nsh);
    h->nzet.assign(B->nzet, B->nzet + B->nsh);
    h->aosh.assign(B->aosh, B->aosh + B->nsh);
    const int MP = B->maxprim;
    for (int s = 0; s < h->nsh; ++s) {
        int t = h->shtyp[s];
        if (t != HFGPU_SHELL_S && t != HFGPU_SHELL_P && t != HFGPU_SHELL_D && t != HFGPU_SHELL_L) {
            delete h;
            return set_err(HFGPU_ERR_ARG, "hfgpu_init: unknown shell type " + std::to_string(t));
        }
        if (h->nzet[s] < 1 || h->nzet[s] > MP) {
            delete h;
            return set_err(HFGPU_ERR_ARG, "hfgpu_init: bad primitive count");
        }
    }
    std::vector<GPrim> prims;
    std::vector<HostPair> plist[NPT];
    h->npairs = build_pairs(B, plist, prims, h->refcount);
    for (int t = 0; t < NPT; ++t) h->pairs[t] = std::move(plist[t]);
    // the same table for every handle: 16200 long-double series, formed once
    struct BoysTables {
        std::vector<double> d;
        std::vector<float> f;
        BoysTables() { build_boys_table(d, f); }
    };
    static const BoysTables tables;
    const std::vector<double>& bt = tables.d;
    const std::vector<float>& btf = tables.f;
    cudaError_t ce = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
    if (ce != cudaSuccess) {
        std::string m = std::string("cudaStreamCreate: ") + cudaGetErrorString(ce);
        delete h;
        return set_err(HFGPU_ERR_CUDA, m);
    }
    {
        int dev = 0;
        if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&h->nsm, cudaDevAttrMultiProcessorCount, dev);
        h->device = dev;
        if (h->nsm <= 0) h->nsm = 148;
        // eight blocks per SM; HFGPU_MERGE_BLOCKS overrides (0: one launch per
        // role always).  Served-size jobs, 200 at once on 8 slots, one box:
        // 10.8 jobs/s without merging, 14.9 at 2 x SMs, 23.9 at 8 x SMs
        h->merge_blocks = 8LL * h->nsm;
        if (const char* e = getenv("HFGPU_MERGE_BLOCKS")) h->merge_blocks = atoll(e);
        // 16 quartets per SM.  At 0 / 4 / 8 / 16 / 32 / 64 / 128 per SM:
        // benzene recorded 499, 499, 482, 468, 475, 505, 536 us, mixed 703,
        // 631, 651, 613, 624, 648 us; C8H18 916, 878, 890, 887, 876, 921, 972
        // us; (H2O)12 882, 856, 862, 877, 891, 905, 957 us.  From C16H34 on the
        // choice is within 1% up to 64
        h->warp_scatter = 16LL * h->nsm;
        // 64 blocks per SM.  A launch per class against one launch: water in
        // STO-3G 106 and 87 us, benzene 567 and 530; C16H34 3.06 and 3.22 ms,
        // C60 in STO-3G with split sp shells 14.3 and 15.9 ms.  In between flat
        // but for n-C20H42 in STO-3G, 524 us up to 32 and 557 from 64 on
        h->direct_blocks = 64LL * h->nsm;
        if (const char* e = getenv("HFGPU_DIRECT")) h->direct_blocks = atoll(e);
        // one form for every list: "single", one thread per quartet, or
        // "grouped", the lanes of a warp together
        if (const char* e = getenv("HFGPU_SCATTER")) {
            if (strcmp(e, "single") == 0) h->warp_scatter = 0;
            if (strcmp(e, "grouped") == 0) h->warp_scatter = INT64_MAX;
        }
        if (const char* e = getenv("HFGPU_WARP_SCATTER")) h->warp_scatter = atoll(e);
        if (const char* e = getenv("HFGPU_STREAMS")) h->nstreams = std::max(1, std::min(NSTREAM, atoi(e)));
    }
    int rc = 0;
    const size_t nb2 = (size_t)h->nb * h->nb;
    rc |= dalloc(&h->d_shtyp, h->nsh, h->stream);
    rc |= dalloc(&h->d_aosh, h->nsh, h->stream);
    rc |= dalloc(&h->d_psoa, 8 * std::max<size_t>(prims.size(), 1), h->stream);
    rc |= dalloc(&h->d_boys, bt.size(), h->stream);
    rc |= dalloc(&h->d_boysf, btf.size(), h->stream);
    rc |= dalloc(&h->d_P, nb2, h->stream);
    rc |= dalloc(&h->d_F, nb2, h->stream);
    rc |= dalloc(&h->d_G, nb2, h->stream);
    rc |= dalloc(&h->d_md, (size_t)h->nsh * h->nsh, h->stream);
    rc |= dalloc(&h->d_cnt, 2 * NCLS, h->stream);
    rc |= dalloc(&h->d_stats, NCLS, h->stream);
    rc |= dalloc(&h->d_ncls, 3 * NCLS, h->stream);
    rc |= dalloc(&h->d_Pb, nb2, h->stream);
    rc |= dalloc(&h->d_boff, (size_t)h->nsh * h->nsh, h->stream);
    rc |= dalloc(&h->d_aomap, (size_t)h->nb, h->stream);
    rc |= dalloc(&h->d_nfsh, (size_t)h->nsh, h->stream);
    for (int t = 0; t < NPT; ++t) {
        size_t n = h->pairs[t].size();
        rc |= dalloc(&h->d_pairs[t], n, h->stream);
        rc |= dalloc(&h->d_schw[t], n, h->stream);
        rc |= dalloc(&h->d_apairs[t], n, h->stream);
        rc |= dalloc(&h->d_ash[t], n, h->stream);
        rc |= dalloc(&h->d_aschw[t], n, h->stream);
    }
    if (rc) {
        hfgpu_finalize(h);
        return HFGPU_ERR_NOMEM;
    }
    cudaEventCreateWithFlags(&h->fork, cudaEventDisableTiming);
    for (int k = 0; k < h->nstreams; ++k) {
        cudaStreamCreateWithFlags(&h->aux[k], cudaStreamNonBlocking);
        cudaEventCreateWithFlags(&h->join[k], cudaEventDisableTiming);
    }
    // uploads on the handle's own stream (pageable sources are staged before
    // the call returns); one synchronisation of that stream at the end
    auto up = [&](void* d, const void* s, size_t bytes) {
        if (bytes == 0) return cudaSuccess;
        return cudaMemcpyAsync(d, s, bytes, cudaMemcpyHostToDevice, h->stream);
    };
    ce = up(h->d_shtyp, h->shtyp.data(), h->nsh * sizeof(int));
    if (ce == cudaSuccess) ce = up(h->d_aosh, h->aosh.data(), h->nsh * sizeof(int));
    if (ce == cudaSuccess) {
        std::vector<double> soa = prims_soa(prims);
        ce = up(h->d_psoa, soa.data(), soa.size() * sizeof(double));
        h->psoa = soa_view(h->d_psoa, prims.size());
    }
    h->hprims = prims;
    if (ce == cudaSuccess) ce = up(h->d_boys, bt.data(), bt.size() * sizeof(double));
    if (ce == cudaSuccess) ce = up(h->d_boysf, btf.data(), btf.size() * sizeof(float));
    {  // shell-pair block layout of the density
        auto nf = [](int t) { return t == HFGPU_SHELL_S ? 1 : t == HFGPU_SHELL_P ? 3 : t == HFGPU_SHELL_D ? 5 : 4; };
        std::vector<int> nfsh(h->nsh), boff((size_t)h->nsh * h->nsh);
        std::vector<int2> aomap(h->nb, make_int2(0, 0));
        for (int a = 0; a < h->nsh; ++a) {
            nfsh[a] = nf(h->shtyp[a]);
            for (int i = 0; i < nfsh[a] && h->aosh[a] + i < h->nb; ++i) aomap[h->aosh[a] + i] = make_int2(a, i);
        }
        long long off = 0;
        for (int a = 0; a < h->nsh; ++a)
            for (int b = 0; b < h->nsh; ++b) {
                boff[(size_t)a * h->nsh + b] = (int)off;
                off += (long long)nfsh[a] * nfsh[b];
            }
        if (off != (long long)h->nb * h->nb) ce = cudaErrorInvalidValue;  // the shells must tile the basis
        if (ce == cudaSuccess) ce = up(h->d_nfsh, nfsh.data(), nfsh.size() * sizeof(int));
        if (ce == cudaSuccess) ce = up(h->d_boff, boff.data(), boff.size() * sizeof(int));
        if (ce == cudaSuccess) ce = up(h->d_aomap, aomap.data(), aomap.size() * sizeof(int2));
    }
    for (int t = 0; t < NPT && ce == cudaSuccess; ++t) {
        std::vector<GPair> gp(h->pairs[t].size());
        for (size_t i = 0; i < gp.size(); ++i) gp[i] = h->pairs[t][i].g;
        ce = up(h->d_pairs[t], gp.data(), gp.size() * sizeof(GPair));
    }
    if (ce != cudaSuccess) {
        std::string m = std::string("hfgpu_init upload: ") + cudaGetErrorString(ce);
        hfgpu_finalize(h);
        return set_err(HFGPU_ERR_CUDA, m);
    }
    // staged diagonal builders: (i, i) lists (their scratch is sized by the
    // handle's budget at the first fock_build_initial_diag)
    {
        for (int t = 0; t < NPT && ce == cudaSuccess; ++t) {
            const ClassKernels& K = CLASS_KERNELS[class_index(t, t)];
            const size_t n = h->pairs[t].size();
            if (K.mode == 0 || n == 0) continue;
            std::vector<uint2> dl(n);
            for (size_t i = 0; i < n; ++i) dl[i] = make_uint2((unsigned)i, (unsigned)i);
            if (dalloc(&h->d_diaglist[t], n, h->stream)) {
                hfgpu_finalize(h);
                return HFGPU_ERR_NOMEM;
            }
            ce = cudaMemcpyAsync(h->d_diaglist[t], dl.data(), n * sizeof(uint2), cudaMemcpyHostToDevice, h->stream);
        }
    }
    if (ce == cudaSuccess) ce = cudaMemsetAsync(h->d_stats, 0, NCLS * sizeof(ClassStats), h->stream);
    if (ce == cudaSuccess) ce = cudaMemsetAsync(h->d_ncls, 0, 3 * NCLS * sizeof(unsigned long long), h->stream);
    // the handle's own stream only: other handles' work on the device goes on
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(h->stream);
    if (ce != cudaSuccess) {
        std::string m = std::string("hfgpu_init: ") + cudaGetErrorString(ce);
        hfgpu_finalize(h);
        return set_err(HFGPU_ERR_CUDA, m);
    }
    *out = h;
    return HFGPU_OK;
}

int hfgpu_finalize(hfgpu_handle* h) {
    if (!h) return HFGPU_OK;
    if (h->stream) cudaStreamSynchronize(h->stream);
    if (h->gexec) cudaGraphExecDestroy(h->gexec);
    if (h->graph) cudaGraphDestroy(h->graph);
    void* bufs[] = {h->d_shtyp, h->d_aosh, h->d_psoa, h->d_apsoa, h->d_boys, h->d_boysf, h->d_P, h->d_F, h->d_G,
                    h->d_md, h->d_subs, h->d_q, h->d_cnt, h->d_mask, h->d_tcnt, h->d_stats, h->d_scratch, h->d_dscratch,
                    h->d_ncls, h->d_Pb, h->d_boff, h->d_aomap, h->d_nfsh};
    for (void* b : bufs)
        if (b) cudaFreeAsync(b, h->stream);
    for (int t = 0; t < NPT; ++t) {
        void* tb[] = {h->d_pairs[t], h->d_schw[t], h->d_apairs[t], h->d_ash[t], h->d_aschw[t], h->d_diaglist[t]};
        for (void* b : tb)
            if (b) cudaFreeAsync(b, h->stream);
    }
    for (int i = 0; i < 2 * NCLS + 2; ++i)
        if (h->ev[i]) cudaEventDestroy(h->ev[i]);
    for (int k = 0; k < NSTREAM; ++k) {
        if (h->aux[k]) {
            cudaStreamSynchronize(h->aux[k]);
            cudaStreamDestroy(h->aux[k]);
        }
        if (h->join[k]) cudaEventDestroy(h->join[k]);
    }
    if (h->fork) cudaEventDestroy(h->fork);
    if (h->stream) {
        cudaStreamSynchronize(h->stream);  // the stream-ordered frees above
        cudaStreamDestroy(h->stream);
    }
    delete h;
    return HFGPU_OK;
}

// Scratch of the staged diagonal builders (one chunk of stride pairs holds
// accumulators, outputs and role maxima per pair), sized once per handle by
// its scratch budget (hfgpu_set_scratch_budget, else the default).
static int alloc_diag_scratch(hfgpu_handle* h) {
    if (h->d_dscratch) return HFGPU_OK;
    const size_t budget = h->scratch_budget ? h->scratch_budget / sizeof(double) : scratch_budget_doubles();
    size_t need = 0, sum = 0;
    for (int t = 0; t < NPT; ++t) {
        const ClassKernels& K = CLASS_KERNELS[class_index(t, t)];
        const size_t n = h->pairs[t].size();
        if (K.mode == 0 || n == 0) continue;
        const size_t per = (size_t)K.nacc + K.nout + K.nrole_b;
        const size_t st = (std::max<size_t>(std::min<size_t>(n, budget / per), TQ) + TQ - 1) / TQ * TQ;  // whole tiles
        h->dstride[t] = st;
        h->doff[t] = sum;
        need = std::max(need, st * per);
        sum += st * per;
    }
    if (!need) return HFGPU_OK;
    // the staged types run side by side where their parts fit the budget
    // together, else one after another through one scratch
    h->dshared = sum > std::max(budget, need);
    if (h->dshared) std::fill(h->doff, h->doff + NPT, 0);
    else need = sum;
    const int rc = dalloc(&h->d_dscratch, need, h->stream);
    if (rc == HFGPU_OK) h->dscratch_doubles = need;
    return rc;
}

static void drop_graph(hfgpu_handle* h) {
    if (h->gexec) cudaGraphExecDestroy(h->gexec);
    if (h->graph) cudaGraphDestroy(h->graph);
    h->gexec = nullptr;
    h->graph = nullptr;
}

int hfgpu_fock_build_initial_diag(hfgpu_handle* h, double* f, const double* p, double thr) {
    if (!h || !f || !p) return set_err(HFGPU_ERR_ARG, "null argument");
    {
        HF_DEVICE_LOCK;
        drop_graph(h);  // the Schwarz pass re-sizes the buffers a captured build points at
        const int rc = alloc_diag_scratch(h);
        if (rc) return rc;
    }
    int rc = upload_fp(h, f, p);
    if (rc) return rc;
    HF_CHECK(cudaMemsetAsync(h->d_G, 0, (size_t)h->nb * h->nb * sizeof(double), h->stream));
    rc = fork_diag(h, 0, h->d_P, thr, true);
    if (rc) return rc;
    rc = launch_symm(h, h->d_F);
    if (rc) return rc;
    rc = download_f(h, f);
    if (rc) return rc;
    return build_active(h);
}

int hfgpu_fock_build_diag(hfgpu_handle* h, double* f, const double* p, double thr) {
    if (!h || !f || !p) return set_err(HFGPU_ERR_ARG, "null argument");
    if (!h->have_schwarz) return set_err(HFGPU_ERR_STATE, "fock_build_initial_diag has not been called");
    int rc = upload_fp(h, f, p);
    if (rc) return rc;
    HF_CHECK(cudaMemsetAsync(h->d_G, 0, (size_t)h->nb * h->nb * sizeof(double), h->stream));
    if ((rc = launch_maxdm(h, h->d_P))) return rc;
    if ((rc = fork_diag(h, 1, h->d_P, thr, true))) return rc;
    if ((rc = launch_symm(h, h->d_F))) return rc;
    return download_f(h, f);
}

static int non_diag_host(hfgpu_handle* h, double* f, const double* p, double thr, int jonly, double f32cut) {
    if (!h || !f || !p) return set_err(HFGPU_ERR_ARG, "null argument");
    if (!h->have_schwarz) return set_err(HFGPU_ERR_STATE, "fock_build_initial_diag has not been called");
    int rc = upload_fp(h, f, p);
    if (rc) return rc;
    HF_CHECK(cudaMemsetAsync(h->d_G, 0, (size_t)h->nb * h->nb * sizeof(double), h->stream));
    if ((rc = launch_maxdm(h, h->d_P))) return rc;
    if ((rc = run_non_diag(h, h->d_P, thr, jonly, f32cut))) return rc;
    if ((rc = launch_symm(h, h->d_F))) return rc;
    return download_f(h, f);
}

int hfgpu_fock_build_non_diag(hfgpu_handle* h, double* f, const double* p, double thr) {
    return non_diag_host(h, f, p, thr, 0, 0.0);
}

int hfgpu_fock_build_non_diag_j_only(hfgpu_handle* h, double* f, const double* p, double thr) {
    return non_diag_host(h, f, p, thr, 1, 0.0);
}

int hfgpu_fock_build_non_diag_mixed(hfgpu_handle* h, double* f, const double* p, double thr, double fp32_cutoff) {
    return non_diag_host(h, f, p, thr, 0, fp32_cutoff);
}

static int device_build(hfgpu_handle* h, double* f_dev, const double* p_dev, double thr_diag, double thr_non_diag,
                        double fp32_cutoff, bool capture) {
    int rc;
    HF_CHECK(cudaMemsetAsync(h->d_G, 0, (size_t)h->nb * h->nb * sizeof(double), h->stream));
    if ((rc = launch_maxdm(h, p_dev))) return rc;
    // beside the screening; joined with the class streams (with per-class
    // timing the classes run on the handle's own stream)
    if ((rc = fork_diag(h, 1, p_dev, thr_diag, h->timing && !capture))) return rc;
    if ((rc = run_non_diag(h, p_dev, thr_non_diag, 0, fp32_cutoff, capture))) return rc;
    return launch_symm(h, f_dev);
}

int hfgpu_fock_build_device(hfgpu_handle* h, double* f_dev, const double* p_dev, double thr_diag,
                            double thr_non_diag, double fp32_cutoff) {
    if (!h || !f_dev || !p_dev) return set_err(HFGPU_ERR_ARG, "null argument");
    if (!h->have_schwarz) return set_err(HFGPU_ERR_STATE, "fock_build_initial_diag has not been called");
    return device_build(h, f_dev, p_dev, thr_diag, thr_non_diag, fp32_cutoff, false);
}

int hfgpu_fock_build_initial_diag_device(hfgpu_handle* h, double* f_dev, const double* p_dev, double thr) {
    if (!h || !f_dev || !p_dev) return set_err(HFGPU_ERR_ARG, "null argument");
    {
        HF_DEVICE_LOCK;
        drop_graph(h);  // the Schwarz pass re-sizes the buffers a captured build points at
        const int rc = alloc_diag_scratch(h);
        if (rc) return rc;
    }
    HF_CHECK(cudaMemsetAsync(h->d_G, 0, (size_t)h->nb * h->nb * sizeof(double), h->stream));
    int rc = fork_diag(h, 0, p_dev, thr, true);
    if (rc) return rc;
    if ((rc = launch_symm(h, f_dev))) return rc;
    return build_active(h);  // reads the Schwarz factors back (synchronises the handle's stream)
}

int hfgpu_fock_build_non_diag_device(hfgpu_handle* h, double* f_dev, const double* p_dev, double thr,
                                     double fp32_cutoff) {
    if (!h || !f_dev || !p_dev) return set_err(HFGPU_ERR_ARG, "null argument");
    if (!h->have_schwarz) return set_err(HFGPU_ERR_STATE, "fock_build_initial_diag has not been called");
    HF_CHECK(cudaMemsetAsync(h->d_G, 0, (size_t)h->nb * h->nb * sizeof(double), h->stream));
    int rc;
    if ((rc = launch_maxdm(h, p_dev))) return rc;
    if ((rc = run_non_diag(h, p_dev, thr, 0, fp32_cutoff))) return rc;
    return launch_symm(h, f_dev);
}

int hfgpu_graph_capture(hfgpu_handle* h, double* f_dev, const double* p_dev, double thr_diag, double thr_non_diag,
                        double fp32_cutoff) {
    if (!h || !f_dev || !p_dev) return set_err(HFGPU_ERR_ARG, "null argument");
    if (!h->have_schwarz) return set_err(HFGPU_ERR_STATE, "fock_build_initial_diag has not been called");
    HF_CHECK(cudaStreamSynchronize(h->stream));
    HF_DEVICE_LOCK;  // held from the start of the capture to its end
    drop_graph(h);
    const long long before = h->launches;
    // thread-local mode: other host threads (other jobs, the caller's own
    // framework) may keep allocating while this thread records
    HF_CHECK(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    const int rc = device_build(h, f_dev, p_dev, thr_diag, thr_non_diag, fp32_cutoff, true);
    cudaGraph_t g = nullptr;
    const cudaError_t ce = cudaStreamEndCapture(h->stream, &g);  // always ends the capture
    if (rc != HFGPU_OK || ce != cudaSuccess) {
        if (g) cudaGraphDestroy(g);
        if (rc != HFGPU_OK) return rc;
        return set_err(HFGPU_ERR_CUDA, std::string("cudaStreamEndCapture: ") + cudaGetErrorString(ce));
    }
    h->graph = g;
    h->graph_launches = h->launches - before;
    h->launches = before;  // recorded, not run
    h->gkey_f = f_dev;
    h->gkey_p = p_dev;
    h->gkey_thr[0] = thr_diag;
    h->gkey_thr[1] = thr_non_diag;
    h->gkey_thr[2] = fp32_cutoff;
    const cudaError_t ie = cudaGraphInstantiate(&h->gexec, g, 0);
    if (ie != cudaSuccess) {
        h->gexec = nullptr;
        drop_graph(h);
        return set_err(HFGPU_ERR_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(ie));
    }
    return HFGPU_OK;
}

int hfgpu_graph_launch(hfgpu_handle* h) {
    if (!h) return set_err(HFGPU_ERR_ARG, "null handle");
    if (!h->gexec) return set_err(HFGPU_ERR_STATE, "hfgpu_graph_capture has not been called");
    HF_CHECK(cudaGraphLaunch(h->gexec, h->stream));
    h->launches += h->graph_launches;
    return HFGPU_OK;
}

// Enqueue one device build on the caller's stream with no host round trip
// (launches sized as for a capture), so that a caller's own CUDA-graph
// capture of a whole SCF iteration can include it.
int hfgpu_fock_build_device_on(hfgpu_handle* h, double* f_dev, const double* p_dev, double thr_diag,
                               double thr_non_diag, double fp32_cutoff, void* stream) {
    if (!h || !f_dev || !p_dev) return set_err(HFGPU_ERR_ARG, "null argument");
    if (!h->have_schwarz) return set_err(HFGPU_ERR_STATE, "fock_build_initial_diag has not been called");
    cudaStream_t own = h->stream;
    h->stream = (cudaStream_t)stream;  // the build forks from and joins back to this stream
    const int rc = device_build(h, f_dev, p_dev, thr_diag, thr_non_diag, fp32_cutoff, true);
    h->stream = own;
    return rc;
}

// Solves the (n x n) system A x = b in place of b on the device (Gaussian
// elimination with partial pivoting, one thread): the DIIS equations of a
// device-resident SCF step, n <= 32.  A is row-major and is overwritten.
__global__ void k_small_solve(double* A, double* b, int n, int* status) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    int ok = 1;
    for (int c = 0; c < n; ++c) {
        int piv = c;
        for (int r = c + 1; r < n; ++r)
            if (fabs(A[r * n + c]) > fabs(A[piv * n + c])) piv = r;
        if (A[piv * n + c] == 0.0) { ok = 0; break; }
        if (piv != c) {
            for (int k = 0; k < n; ++k) { const double t = A[c * n + k]; A[c * n + k] = A[piv * n + k]; A[piv * n + k] = t; }
            const double t = b[c]; b[c] = b[piv]; b[piv] = t;
        }
        for (int r = c + 1; r < n; ++r) {
            const double m = A[r * n + c] / A[c * n + c];
            for (int k = c; k < n; ++k) A[r * n + k] -= m * A[c * n + k];
            b[r] -= m * b[c];
        }
    }
    if (ok)
        for (int r = n - 1; r >= 0; --r) {
            double s = b[r];
            for (int k = r + 1; k < n; ++k) s -= A[r * n + k] * b[k];
            b[r] = s / A[r * n + r];
        }
    if (status) *status = ok;
}

int hfgpu_small_solve(double* a_dev, double* b_dev, int n, int* status_dev, void* stream) {
    if (!a_dev || !b_dev || n <= 0 || n > 32) return set_err(HFGPU_ERR_ARG, "hfgpu_small_solve: bad arguments");
    k_small_solve<<<1, 32, 0, (cudaStream_t)stream>>>(a_dev, b_dev, n, status_dev);
    HF_CHECK(cudaGetLastError());
    return HFGPU_OK;
}

int hfgpu_fock_build_graph(hfgpu_handle* h, double* f, const double* p, double thr_diag, double thr_non_diag,
                           double fp32_cutoff) {
    if (!h || !f || !p) return set_err(HFGPU_ERR_ARG, "null argument");
    if (!h->have_schwarz) return set_err(HFGPU_ERR_STATE, "fock_build_initial_diag has not been called");
    const bool same = h->gexec && h->gkey_f == h->d_F && h->gkey_p == h->d_P && h->gkey_thr[0] == thr_diag &&
                      h->gkey_thr[1] == thr_non_diag && h->gkey_thr[2] == fp32_cutoff;
    int rc;
    if (!same && (rc = hfgpu_graph_capture(h, h->d_F, h->d_P, thr_diag, thr_non_diag, fp32_cutoff))) return rc;
    if ((rc = upload_fp(h, f, p))) return rc;
    HF_CHECK(cudaGraphLaunch(h->gexec, h->stream));
    h->launches += h->graph_launches;
    return download_f(h, f);
}

int hfgpu_synchronize(hfgpu_handle* h) {
    if (!h) return set_err(HFGPU_ERR_ARG, "null handle");
    HF_CHECK(cudaStreamSynchronize(h->stream));
    return HFGPU_OK;
}

int hfgpu_batch_create(hfgpu_handle* const* hs, int n, hfgpu_batch** out) {
    if (!hs || !out || n <= 0) return set_err(HFGPU_ERR_ARG, "hfgpu_batch_create: bad arguments");
    *out = nullptr;
    for (int i = 0; i < n; ++i) {
        if (!hs[i]) return set_err(HFGPU_ERR_ARG, "hfgpu_batch_create: null handle");
        if (!hs[i]->graph)
            return set_err(HFGPU_ERR_STATE, "hfgpu_batch_create: handle " + std::to_string(i) +
                                                " has no captured build (call hfgpu_graph_capture)");
        for (int j = 0; j < i; ++j)
            if (hs[j] == hs[i]) return set_err(HFGPU_ERR_ARG, "hfgpu_batch_create: a handle appears twice");
    }
    HF_DEVICE_LOCK;
    hfgpu_batch* b = new hfgpu_batch();
    b->hs.assign(hs, hs + n);
    cudaError_t ce = cudaGraphCreate(&b->graph, 0);
    // one child graph per instance, no edges between them: the instances
    // share nothing on the device and run concurrently
    for (int i = 0; i < n && ce == cudaSuccess; ++i) {
        cudaGraphNode_t node;
        ce = cudaGraphAddChildGraphNode(&node, b->graph, nullptr, 0, hs[i]->graph);
    }
    if (ce == cudaSuccess) ce = cudaGraphInstantiate(&b->exec, b->graph, 0);
    if (ce != cudaSuccess) {
        hfgpu_batch_destroy(b);
        return set_err(HFGPU_ERR_CUDA, std::string("hfgpu_batch_create: ") + cudaGetErrorString(ce));
    }
    *out = b;
    return HFGPU_OK;
}

int hfgpu_batch_launch(hfgpu_batch* b, void* stream) {
    if (!b || !b->exec) return set_err(HFGPU_ERR_ARG, "null batch");
    HF_CHECK(cudaGraphLaunch(b->exec, (cudaStream_t)stream));
    for (hfgpu_handle* h : b->hs) h->launches += h->graph_launches;
    return HFGPU_OK;
}

int hfgpu_batch_destroy(hfgpu_batch* b) {
    if (!b) return HFGPU_OK;
    HF_DEVICE_LOCK;
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    delete b;
    return HFGPU_OK;
}

int hfgpu_set_scratch_budget(hfgpu_handle* h, size_t bytes) {
    if (!h) return set_err(HFGPU_ERR_ARG, "null handle");
    if (h->have_schwarz) return set_err(HFGPU_ERR_STATE, "set the scratch budget before fock_build_initial_diag");
    h->scratch_budget = bytes;
    return HFGPU_OK;
}

int hfgpu_device_bytes(const hfgpu_handle* h, size_t* bytes) {
    if (!h || !bytes) return set_err(HFGPU_ERR_ARG, "null argument");
    size_t b = 0;
    const size_t nb2 = (size_t)h->nb * h->nb;
    b += 4 * nb2 * sizeof(double);                            // P, F, G, blocked P
    b += ((size_t)h->nsh * h->nsh + 2 * (size_t)h->nb + h->nsh) * sizeof(int);
    b += (size_t)h->nsh * h->nsh * sizeof(double);            // maxdm
    b += 2 * (size_t)h->nsh * sizeof(int);
    b += 8 * h->hprims.size() * sizeof(double);               // all-pairs primitives
    for (int t = 0; t < NPT; ++t) {
        const size_t n = h->pairs[t].size();
        b += n * (2 * sizeof(GPair) + sizeof(double) * 2 + sizeof(int2) + (h->d_diaglist[t] ? sizeof(uint2) : 0));
    }
    b += 8 * h->naprims * sizeof(double);                     // active-list primitives
    b += h->qcap * sizeof(uint2);                             // quartet lists
    b += h->scratch_doubles * sizeof(double);                 // staged scratch
    b += h->dscratch_doubles * sizeof(double);                // staged diagonal builders' scratch
    b += h->maskcap * 2 * sizeof(unsigned) + h->tilecap * sizeof(TileEntries);  // screening masks and counts
    b += h->subcap * (sizeof(ScreenSub) + 2 * sizeof(unsigned long long));
    b += (size_t)(BOYS_MMAX + 1) * BOYS_BLK * (sizeof(double) + sizeof(float));
    *bytes = b;
    return HFGPU_OK;
}

int hfgpu_dims(const hfgpu_handle* h, int* nb, int* nsh, int* npairs) {
    if (!h) return set_err(HFGPU_ERR_ARG, "null handle");
    if (nb) *nb = h->nb;
    if (nsh) *nsh = h->nsh;
    if (npairs) *npairs = h->npairs;
    return HFGPU_OK;
}

int hfgpu_get_schwarz(const hfgpu_handle* h, double* schw_sh, int* last) {
    if (!h) return set_err(HFGPU_ERR_ARG, "null handle");
    if (!h->have_schwarz) return set_err(HFGPU_ERR_STATE, "fock_build_initial_diag has not been called");
    if (schw_sh) {
        for (int t = 0; t < NPT; ++t)
            for (size_t i = 0; i < h->pairs[t].size(); ++i) {
                const GPair& g = h->pairs[t][i].g;
                schw_sh[(size_t)g.sa * h->nsh + g.sb] = h->schw[t][i];
                schw_sh[(size_t)g.sb * h->nsh + g.sa] = h->schw[t][i];
            }
    }
    if (last)
        for (int c = 0; c < 10; ++c) last[c] = h->last_ref[c];
    return HFGPU_OK;
}

int hfgpu_get_class_stats(const hfgpu_handle* h, long long* n_pass, long long* n_scattered, long long* n_prim,
                          long long* n_fp32, double* ms) {
    if (!h) return set_err(HFGPU_ERR_ARG, "null handle");
    // the counters live on the device (a captured build never returns to the
    // host); read them after the handle's stream has drained
    ClassStats st[NCLS];
    unsigned long long cnt[2 * NCLS];
    HF_DEVICE_LOCK;
    HF_CHECK(cudaStreamSynchronize(h->stream));
    HF_CHECK(cudaMemcpy(st, h->d_stats, sizeof(st), cudaMemcpyDeviceToHost));
    HF_CHECK(cudaMemcpy(cnt, h->d_ncls, sizeof(cnt), cudaMemcpyDeviceToHost));
    for (int c = 0; c < NCLS; ++c) {
        if (n_pass) n_pass[c] = (long long)(cnt[2 * c] + cnt[2 * c + 1]);
        if (n_scattered) n_scattered[c] = (long long)st[c].scattered;
        if (n_prim) n_prim[c] = (long long)st[c].prim;
        if (n_fp32) n_fp32[c] = (long long)st[c].fp32;
        if (ms) ms[c] = h->st_ms[c];
    }
    return HFGPU_OK;
}

int hfgpu_launch_count(const hfgpu_handle* h, long long* n) {
    if (!h || !n) return set_err(HFGPU_ERR_ARG, "null argument");
    *n = h->launches;
    return HFGPU_OK;
}

int hfgpu_set_timing(hfgpu_handle* h, int on) {
    if (!h) return set_err(HFGPU_ERR_ARG, "null handle");
    if (on && !h->ev[0])  // the events of the per-class timing
        for (cudaEvent_t& e : h->ev) HF_CHECK(cudaEventCreate(&e));
    h->timing = on;
    return HFGPU_OK;
}

void* hfgpu_stream(hfgpu_handle* h) { return h ? (void*)h->stream : nullptr; }

int hfgpu_measure_fma_peak(double* fp64_gflops, double* fp32_gflops) {
    HF_DEVICE_LOCK;
    int dev = 0, nsm = 0;
    HF_CHECK(cudaGetDevice(&dev));
    HF_CHECK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    double* dd = nullptr;
    HF_CHECK(cudaMalloc(&dd, 64));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int threads = 256, blocks = nsm * 8, iters = 1 << 14;
    double res[2] = {0, 0};
    for (int prec = 0; prec < 2; ++prec) {
        float best = 1e30f;
        for (int rep = 0; rep < 4; ++rep) {
            cudaEventRecord(e0);
            if (prec == 0) k_fma_peak<double><<<blocks, threads>>>(dd, iters, 0.999999, 1e-7);
            else k_fma_peak<float><<<blocks, threads>>>((float*)dd, iters, 0.999999f, 1e-7f);
            cudaEventRecord(e1);
            cudaError_t ce = cudaEventSynchronize(e1);
            if (ce != cudaSuccess) {
                cudaFree(dd);
                g_err = cudaGetErrorString(ce);
                return HFGPU_ERR_CUDA;
            }
            float ms = 0;
            cudaEventElapsedTime(&ms, e0, e1);
            if (rep > 0) best = std::min(best, ms);
        }
        res[prec] = 2.0 * 8.0 * (double)iters * threads * blocks / (best * 1e-3) / 1e9;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(dd);
    if (fp64_gflops) *fp64_gflops = res[0];
    if (fp32_gflops) *fp32_gflops = res[1];
    return HFGPU_OK;
}

}  // extern "C"

// ------------------------------------------------ no-allocation variant ----
// Scratch of hfgpu_fock_build_diag_static: the one-triangle accumulation
// buffer G (nb x nb) and the shell-pair density maxima (nsh x nsh) live in
// this file-scope device array instead of memory from cudaMalloc.  Every GPU
// that loads the library holds it (10,485,760 bytes, 10.0 MiB) until the process exits.
namespace {
constexpr int STATIC_MAX_NB = 1024;
constexpr int STATIC_MAX_NSH = 512;
constexpr size_t STATIC_SCRATCH_DOUBLES =
    (size_t)STATIC_MAX_NB * STATIC_MAX_NB + (size_t)STATIC_MAX_NSH * STATIC_MAX_NSH;
}  // namespace

static __device__ __align__(256) double g_static_scratch[STATIC_SCRATCH_DOUBLES];

namespace {
constexpr int STATIC_MAX_DEVICES = 64;
std::mutex g_static_mu;
double* g_static_ptr[STATIC_MAX_DEVICES] = {};

// Device address of g_static_scratch on the current device.  Host code sees
// only a host-side stand-in under that name, so the address is looked up once
// per device, with that device current, and cached.
int static_scratch(double** out) {
    int dev = 0;
    HF_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= STATIC_MAX_DEVICES) return set_err(HFGPU_ERR_UNSUPPORTED, "device index out of range");
    std::lock_guard<std::mutex> lk(g_static_mu);
    if (!g_static_ptr[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
        if (e != cudaSuccess || !p)
            return set_err(HFGPU_ERR_CUDA, std::string("cudaGetSymbolAddress(g_static_scratch): ") +
                                               cudaGetErrorString(e));
        g_static_ptr[dev] = (double*)p;
    }
    *out = g_static_ptr[dev];
    return HFGPU_OK;
}
}  // namespace

extern "C" int hfgpu_fock_build_diag_static(hfgpu_handle* h, double* f_dev, const double* p_dev, double thr) {
    if (!h || !f_dev || !p_dev) return set_err(HFGPU_ERR_ARG, "null argument");
    if (h->nb > STATIC_MAX_NB || h->nsh > STATIC_MAX_NSH)
        return set_err(HFGPU_ERR_ARG, "hfgpu_fock_build_diag_static: nb " + std::to_string(h->nb) + " / nsh " +
                                          std::to_string(h->nsh) + " exceeds the static scratch limit of nb <= " +
                                          std::to_string(STATIC_MAX_NB) + ", nsh <= " +
                                          std::to_string(STATIC_MAX_NSH));
    if (!h->have_schwarz) return set_err(HFGPU_ERR_STATE, "fock_build_initial_diag has not been called");
    {
        int dev = -1;
        HF_CHECK(cudaGetDevice(&dev));
        if (dev != h->device)
            return set_err(HFGPU_ERR_ARG, "hfgpu_fock_build_diag_static: the current device (" + std::to_string(dev) +
                                              ") is not the device the handle was created on (" +
                                              std::to_string(h->device) + ")");
    }
    double* scratch = nullptr;
    int rc = static_scratch(&scratch);
    if (rc) return rc;
    double* G = scratch;
    double* md = scratch + (size_t)STATIC_MAX_NB * STATIC_MAX_NB;
    // G keeps the previous call's sums: clear it first
    HF_CHECK(cudaMemsetAsync(G, 0, (size_t)h->nb * h->nb * sizeof(double), h->stream));
    if ((rc = launch_maxdm(h, p_dev, md))) return rc;
    if ((rc = launch_diag(h, 1, p_dev, thr, G, md, &h->stream, 1, false))) return rc;
    return launch_symm(h, f_dev, G);
}
