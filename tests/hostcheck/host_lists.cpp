// Host-compiled check of the quartet lists' index arithmetic (test
// infrastructure): csrc/lists.cuh with threads in the place of a block's
// lanes.  Only tests/test_lists_host.py builds and loads this file.
#include <barrier>
#include <thread>
#include <vector>

#define __device__
#define __host__
#define __forceinline__ inline
#define __restrict__
#define __shared__ static
struct uint2 {
    unsigned x, y;
};
constexpr int BLOCK = 128;
thread_local struct { int x; } threadIdx;
static std::barrier<> g_bar(BLOCK);
static void __syncthreads() { g_bar.arrive_and_wait(); }
static int __shfl_up_sync(unsigned, int v, int o) {
    static int slot[BLOCK];
    slot[threadIdx.x] = v;
    __syncthreads();
    const int r = (threadIdx.x & 31) >= o ? slot[threadIdx.x - o] : v;
    __syncthreads();
    return r;
}
static int __double2int_rn(double x) { return (int)__builtin_nearbyint(x); }
static int __float2int_rn(float x) { return (int)__builtin_nearbyintf(x); }
static double rsqrt(double x) { return 1.0 / __builtin_sqrt(x); }
static float rsqrtf(float x) { return 1.0f / __builtin_sqrtf(x); }
#define __expf(x) __builtin_expf(x)

#include "lists.cuh"

using namespace hfgpu;
static_assert(OFF_THREADS == BLOCK, "one emulated thread per lane");

extern "C" {

// counts[2 * nt] -> entries before each tile, in place
void hl_scan_tiles(long long* counts, int nt) {
    std::vector<std::thread> ts;
    for (int i = 0; i < BLOCK; ++i)
        ts.emplace_back([=] {
            threadIdx.x = i;
            scan_tiles(reinterpret_cast<TileEntries*>(counts), nt);
        });
    for (auto& t : ts) t.join();
}

// A class list of nsub sub-classes, one precision: cnt entries each, off /
// unit their first entry and work unit, 2^lgb x 2^lgk lanes per quartet.
struct Lists {
    std::vector<ScreenSub> subs;
    std::vector<unsigned long long> cnt, ncls;
    std::vector<int> nunit;
    UnitList L;
};

static Lists make(const long long* cnt, const long long* off, const int* unit, const int* lgb, const int* lgk,
                  int nsub, int nunit, long long coff, int prec, long long n64) {
    Lists x;
    x.subs.resize(nsub);
    x.cnt.assign(2 * nsub, 0);
    x.ncls.assign(2, (unsigned long long)n64);
    x.nunit.assign(2, nunit);
    for (int k = 0; k < nsub; ++k) {
        x.cnt[2 * k + prec] = (unsigned long long)cnt[k];
        x.subs[k].off[prec] = off[k];
        x.subs[k].unit[prec] = unit[k];
        x.subs[k].lgb[prec] = lgb[k];
        x.subs[k].lgk[prec] = lgk[k];
    }
    x.L = UnitList{x.subs.data(), x.cnt.data(), x.ncls.data(), x.nunit.data(), 0, nsub, coff, nullptr, 0, prec};
    return x;
}

// out[lane]: place in the quartet buffer, entry in the list, stored or not
int hl_unit(const long long* cnt, const long long* off, const int* unit, const int* lgb, const int* lgk, int nsub,
            int nunit, long long coff, int prec, long long n64, int u, long long* out) {
    Lists x = make(cnt, off, unit, lgb, lgk, nsub, nunit, coff, prec, n64);
    for (int lane = 0; lane < 32; ++lane) {
        Unit w;
        long long at;
        if (!unit_place(x.L, u, lane, w, at)) return 0;
        out[3 * lane] = at;
        out[3 * lane + 1] = at - list_start(x.L);
        out[3 * lane + 2] = w.store;
    }
    return 1;
}

void hl_units_of(const long long* cnt, const long long* off, const int* unit, const int* lgb, const int* lgk,
                 int nsub, int nunit, long long coff, int prec, long long n64, long long q0, long long n, int* out) {
    Lists x = make(cnt, off, unit, lgb, lgk, nsub, nunit, coff, prec, n64);
    units_of(x.L, list_start(x.L) + q0, n, out[0], out[1]);
}

}  // extern "C"
