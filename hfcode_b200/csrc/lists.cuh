// Positions in the compacted quartet lists and the work units the kernels
// take from them: plain index arithmetic, in 64 bits wherever a class's list
// is counted (one class of a large molecule passes 2^31 quartets, 17 GB of
// list, well before it fills the GPU's memory).
// Host-compilable with the shims of the test harness (threads as lanes).
#pragma once
#include "types.cuh"

namespace hfgpu {

// One screening sub-class: the candidates of quartet class `cls` whose bra
// pairs come from one primitive-count group of the active bra list and ket
// pairs from one group of the ket list, so that every quartet in the
// compacted sub-list runs its primitive loops with the same trip counts.
struct ScreenSub {
    long long ncand;   // candidates
    int tile0;         // first screening tile
    int cls;
    int same;          // one group against itself: pairs i > j only
    int b0, nbra;      // bra range in the active list
    int k0, nket;      // ket range
    int npb, npk;      // primitives of the bra and ket pairs
    // filled on the device by k_offsets, FP64 and FP32 entries:
    long long off[2];  // write offsets (second pass)
    int unit[2];       // first work unit within the class's list (see Unit)
    int lgb[2], lgk[2];  // log2 of the lanes over the bra and ket primitives
};

// Work unit of a class list: one warp's share, 32 / 2^(lgb + lgk) quartets of
// one sub-class, each spread over 2^(lgb + lgk) lanes that split its
// primitive loops.  A quartet of two six-fold contracted s pairs runs 1296
// primitive quartets: one thread per quartet made that one thread's serial
// chain the time of the whole kernel for a small molecule (benzene SS|SS:
// 255 us at 66 blocks).
struct Unit {
    int t;             // entry within the chunk (stage_unit)
    bool store;        // this lane writes the quartet's results
    uint2 q;           // (bra, ket)
    LaneSplit ls;
};

struct UnitList {
    const ScreenSub* subs;             // the sub-class table
    const unsigned long long* cnt;     // [2 * nsub] entries per sub-class (FP64, FP32)
    const unsigned long long* ncls;    // [2 * NCLS] entries per class
    const int* nunit;                  // [2 * NCLS] work units per class
    int sub0, sub1;                    // sub-classes of this class
    long long coff;                    // first entry of this class in the quartet buffer
    const uint2* quartets;             // the whole quartet buffer
    int cls, prec;
};

// First entry of the list's precision in the quartet buffer.
__device__ __forceinline__ long long list_start(const UnitList& L) {
    return L.coff + (L.prec ? (long long)L.ncls[2 * L.cls] : 0);
}

// Lane `lane` of unit u of the list: everything but the quartet itself, which
// is at `at` of the quartet buffer; false past the end.  The lanes without a
// quartet (the tail of a sub-class) repeat the sub-class's last one and do
// not store.
__device__ __forceinline__ bool unit_place(const UnitList& L, int u, int lane, Unit& w, long long& at) {
    const int p = L.prec;
    if (u >= L.nunit[2 * L.cls + p]) return false;
    int lo = L.sub0, hi = L.sub1 - 1;  // last sub-class whose first unit is <= u
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (L.subs[mid].unit[p] <= u) lo = mid;
        else hi = mid - 1;
    }
    const ScreenSub& S = L.subs[lo];
    const int lgb = S.lgb[p], lgk = S.lgk[p], lg = lgb + lgk;
    const long long first = (long long)(u - S.unit[p]) << (5 - lg);  // within the sub-class
    const long long rest = (long long)L.cnt[2 * lo + p] - first;
    const int n = (int)(rest < 32 ? rest : 32), i = lane >> lg;  // of this unit
    const int g = lane & ((1 << lg) - 1);
    at = S.off[p] + first + (i < n ? i : n - 1);
    w.store = i < n && g == 0;
    w.ls = LaneSplit{g >> lgk, 1 << lgb, g & ((1 << lgk) - 1), 1 << lgk, 1 << lg};
    return true;
}

// The units [u0, u1) that hold entries [first, first + n) of the quartet
// buffer, n > 0, all of the list; the first and last may reach outside them.
__device__ __forceinline__ void units_of(const UnitList& L, long long first, long long n, int& u0, int& u1) {
    const int p = L.prec;
    for (int end = 0; end < 2; ++end) {  // the units of the first and of the last entry
        const long long at = first + (end ? n - 1 : 0);
        int lo = L.sub0, hi = L.sub1 - 1;  // last sub-class whose entries start at or before `at`
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (L.subs[mid].off[p] <= at) lo = mid;
            else hi = mid - 1;
        }
        const ScreenSub& S = L.subs[lo];
        const int u = S.unit[p] + (int)((at - S.off[p]) >> (5 - S.lgb[p] - S.lgk[p]));
        if (end) u1 = u + 1;
        else u0 = u;
    }
}

// Fewest lanes (lgb + lgk) over npb x npk primitives with at most `most`
// primitive quartets per lane, and their best split over bra and ket.
__device__ __forceinline__ void pick_lanes(int npb, int npk, int most, int& lgb, int& lgk) {
    lgb = lgk = 0;
    int best = npb * npk;
    for (int lg = 1; lg <= 5 && best > most; ++lg)
        for (int k = 0; k <= lg; ++k) {
            const int b = lg - k;
            const int c = ((npb + (1 << b) - 1) >> b) * ((npk + (1 << k) - 1) >> k);
            if (c < best) {
                best = c;
                lgb = b;
                lgk = k;
            }
        }
}

// The counts of a sub-class's `nt` tiles (FP64 and FP32 survivors of each
// tile, tile by tile) into the entries before the tile, by one block.  The
// counts of one step of OFF_THREADS tiles fit 32 bits (at most 2048 a tile);
// the entries before the step need not.
constexpr int OFF_THREADS = 128;
struct alignas(16) TileEntries {
    long long n64, n32;
};
__device__ __forceinline__ void scan_tiles(TileEntries* __restrict__ t, int nt) {
    __shared__ int part[OFF_THREADS / 32][2];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    TileEntries run{0, 0};
    for (int k0 = 0; k0 < nt; k0 += OFF_THREADS) {
        const int k = k0 + (int)threadIdx.x;
        const int x0 = k < nt ? (int)t[k].n64 : 0, y0 = k < nt ? (int)t[k].n32 : 0;
        int x = x0, y = y0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int xo = __shfl_up_sync(0xffffffffu, x, o), yo = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= o) x += xo, y += yo;
        }
        if (lane == 31) part[wp][0] = x, part[wp][1] = y;
        __syncthreads();
        TileEntries before = run;
        for (int q = 0; q < OFF_THREADS / 32; ++q) {
            if (q < wp) before.n64 += part[q][0], before.n32 += part[q][1];
            run.n64 += part[q][0], run.n32 += part[q][1];
        }
        if (k < nt) t[k] = TileEntries{before.n64 + x - x0, before.n32 + y - y0};
        __syncthreads();
    }
}

}  // namespace hfgpu
