// The moment sums in the reference's order: each moment component of an
// estimator is one sequential sum over its terms' contributions
// (cauchy_estimator.hpp:340-357), and a reordered sum is not the same double
// (the covariance's cancellation moves it by 1e-9).  The contributions lie
// component by component: component c of row r at contrib[c * pitch + r].
//
// Two routines give the same bits:
//   chain_short  a warp per (estimator, 32 components), a lane per component
//                adding its rows one after another: the additions of many
//                estimators share the FP64 pipe, but one chain cannot run
//                faster than the dependent addition (about 64 cycles a row);
//   chain_scan   a block per (estimator, component): 128 runs of eight rows
//                summed at once from predicted starts, the predictions
//                corrected until every run ends where the next one began.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace mce {

__device__ inline void cp_async16(void* smem_dst, const void* gmem_src, int bytes)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem_src), "r"(bytes) : "memory");
}
__device__ inline void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ inline void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// ---------------------------------------------------------------------------
// chain_short: rows [a, a + n) of this lane's column (null: an idle lane).
// The rows stream through a ring of kMomStages chunks of kMomRows in shared
// memory, 16 bytes a copy, each lane its own column, so the lane's own
// wait_group is the only synchronisation; the additions of a chunk run back
// to back on registers.
constexpr int kMomStages = 3, kMomRows = 64;

__device__ inline double chain_short(const double* col, long long a, long long n, double2 (*ring)[kMomRows / 2][32])
{
    const int lane = threadIdx.x & 31;
    const bool valid = col != nullptr;
    const long long lo = a & ~1LL, end = a + n;  // 16-byte copies start on an even row
    const long long nchunks = (end - lo + kMomRows - 1) / kMomRows;
    auto issue = [&](long long k) {
        if (valid && k < nchunks) {
            const long long r0 = lo + k * kMomRows;
            double2(*slot)[32] = ring[k % kMomStages];
            const double* src = col + r0;
            if (end - r0 >= kMomRows) {
#pragma unroll
                for (int r = 0; r < kMomRows / 2; r++) cp_async16(&slot[r][lane], src + 2 * r, 16);
            } else
                for (int r = 0; 2 * r < end - r0; r++)
                    cp_async16(&slot[r][lane], src + 2 * r, end - r0 - 2 * r >= 2 ? 16 : 8);
        }
        cp_async_commit();
    };
    for (int k = 0; k < kMomStages - 1; k++) issue(k);
    double sum = 0.0;
    for (long long k = 0; k < nchunks; k++) {
        cp_async_wait<kMomStages - 2>();  // chunk k has landed
        // refill the slot of chunk k - 1, whose values were added last iteration
        issue(k + kMomStages - 1);
        if (!valid) continue;
        const long long r0 = lo + k * kMomRows;
        const double2(*slot)[32] = ring[k % kMomStages];
        if (r0 >= a && end - r0 >= kMomRows) {
            // all loads first, then the dependent additions back to back
            double2 v[kMomRows / 2];
#pragma unroll
            for (int r = 0; r < kMomRows / 2; r++) v[r] = slot[r][lane];
#pragma unroll
            for (int r = 0; r < kMomRows / 2; r++) {
                sum += v[r].x;
                sum += v[r].y;
            }
        } else {
            for (int r = 0; r < kMomRows && r0 + r < end; r++) {
                if (r0 + r < a) continue;
                const double2 v = slot[r / 2][lane];
                sum += (r & 1) ? v.y : v.x;
            }
        }
    }
    cp_async_wait<0>();
    return sum;
}

// ---------------------------------------------------------------------------
// chain_scan.  A tile is 128 runs of eight rows, a thread each.  From the true
// sum before the tile and prediction g of the sum before its run, a thread
// adds its rows in floating point, ending at h; when every h is the next
// thread's g, bit for bit, all of them are the sequential sums.  That check
// alone makes the result right; what follows only has to predict well.
//
// First g: the sum before the tile plus a tree sum of the rows between.  It is
// off by some d, and d travels through the run's roundings exactly as
//     d <- RN_u(d + y),
// u the ulp of the step's sum and y the step's rounding error (sum + y is the
// exact value), while the sum stays in its binade.  A step on a grid no coarser
// than an earlier one leaves d alone, so a run acts as d -> RN_U(d + b), U its
// coarsest ulp, b collected at the steps that raise U (a tie counts as a step
// on the doubled grid: it ends even).  With the gap
// a = (previous h) - g, the deviation of a run's end is RN_U(a + d' + b), d' the
// previous run's: such maps compose (ChainMap), and one scan over the threads
// gives every run's start as it will be after all the roundings before it.
// Runs that the sums take from the noise of a cancelled family up to its terms
// and back are predicted like runs on a settled sum; a wrong prediction is
// left where a sum sits next to a power of two, or on a tie, and costs another
// round.  Every round settles at least one more run; a tile that is not settled
// after kChainRounds is finished by plain additions, which bounds the cost.
// Everything about d is integer arithmetic in units of 2^-107 of the tile's
// largest power of two.
constexpr int kChainRun = 8;                          // rows a thread
constexpr int kChainThreads = 128;
constexpr int kChainTile = kChainThreads * kChainRun; // rows a tile
constexpr int kChainPitch = kChainRun + 2;            // doubles between the threads' runs in shared memory
constexpr int kChainStages = 3;
constexpr int kChainRounds = 12;
static_assert(kChainRun % 2 == 0 && kChainPitch % 2 == 0, "a thread's run starts on 16 bytes");

struct ChainMap {  // x -> c + RN_u(x + b), u a power of two (1: exact)
    long long b, c, u;
};
__device__ inline long long chain_rn(long long x, long long u) { return (x + (u >> 1)) & -u; }
__device__ inline long long chain_ceil(long long x, long long u) { return (x + u - 1) & -u; }
// f, then g
__device__ inline ChainMap chain_then(const ChainMap& f, const ChainMap& g)
{
    if (g.u <= f.u) return ChainMap{f.b, g.c + chain_rn(f.c + g.b, g.u), f.u};
    // a step of g at x + b = u/2 mod u, first reached by f's grid at the ceiling
    const long long h = g.u >> 1;
    return ChainMap{f.b + h - chain_ceil(h - f.c - g.b, f.u) + (f.u >> 1), g.c, g.u};
}
// x in units of 2^(q - 1075), towards zero
__device__ inline long long chain_units(double x, int q)
{
    const unsigned hi = (unsigned)__double2hiint(x);
    const int e = (int)((hi >> 20) & 0x7ff);
    const long long m = e ? (((long long)((hi & 0xfffffu) | 0x100000u) << 32) | (unsigned)__double2loint(x)) : 0;
    const int sh = e - q;
    const long long r = sh >= 0 ? m << (sh < 9 ? sh : 9) : m >> (sh > -63 ? -sh : 63);
    return (int)hi < 0 ? -r : r;
}

// (16-byte copies land in v, and are read from it)
struct alignas(16) ChainSmem {
    double v[kChainStages][kChainThreads * kChainPitch];
    double h[kChainThreads / 32], p[kChainThreads / 32], s;
    ChainMap m[kChainThreads / 32];
    int e[kChainThreads / 32], first;
};

// Rows [a, a + n) of one column added in order, by a block of kChainThreads;
// the sum in every thread.
__device__ inline double chain_scan(const double* col, long long a, long long n, ChainSmem& sm)
{
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int kWarps = kChainThreads / 32;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const long long lo = a & ~1LL, end = a + n;
    const long long ntiles = (end - lo + kChainTile - 1) / kChainTile;
    auto issue = [&](long long t) {
        if (t < ntiles) {
            const long long r0 = lo + t * kChainTile + tid * kChainRun;
            double* dst = sm.v[t % kChainStages] + tid * kChainPitch;
#pragma unroll
            for (int c = 0; c < kChainRun / 2; c++) {
                const long long left = end - (r0 + 2 * c);  // beyond the end: zeros
                const int bytes = left >= 2 ? 16 : (left == 1 ? 8 : 0);
                cp_async16(dst + 2 * c, col + (bytes ? r0 + 2 * c : lo), bytes);
            }
        }
        cp_async_commit();
    };
    for (int t = 0; t < kChainStages - 1; t++) issue(t);
    double s = 0.0;
    for (long long t = 0; t < ntiles; t++) {
        cp_async_wait<kChainStages - 2>();
        double* run = sm.v[t % kChainStages] + tid * kChainPitch;
        if (t == 0 && (a & 1) && tid == 0) run[0] = 0.0;  // the row before the first
        double v[kChainRun];
#pragma unroll
        for (int i = 0; i < kChainRun; i += 2) {
            const double2 x = *reinterpret_cast<const double2*>(run + i);
            v[i] = x.x;
            v[i + 1] = x.y;
        }
        // first predictions
        double p = v[0];
#pragma unroll
        for (int i = 1; i < kChainRun; i++) p += v[i];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(kAll, p, o);
            if (lane >= o) p += y;
        }
        if (lane == 31) sm.p[w] = p;
        const double up = __shfl_up_sync(kAll, p, 1);
        __syncthreads();
        double g = s;
        for (int k = 0; k < w; k++) g += sm.p[k];
        if (lane) g += up;
        double h;
        for (int round = 0;; round++) {
            // the run, and (in the even rounds) its rounding errors
            const bool learn = (round & 1) == 0;
            double y[kChainRun], x = g;
            int ex[kChainRun];
            if (learn) {
#pragma unroll
                for (int i = 0; i < kChainRun; i++) {
                    const unsigned long long ax = (unsigned long long)__double_as_longlong(x) << 1;
                    const unsigned long long av = (unsigned long long)__double_as_longlong(v[i]) << 1;
                    const double big = ax >= av ? x : v[i], small = ax >= av ? v[i] : x;
                    const double r = x + v[i];
                    y[i] = small - (r - big);
                    x = r;
                    ex[i] = (__double2hiint(x) >> 20) & 0x7ff;
                }
            } else {
#pragma unroll
                for (int i = 0; i < kChainRun; i++) x += v[i];
            }
            h = x;
            if (lane == 31) sm.h[w] = h;
            if (learn) {
                int em = 0;
#pragma unroll
                for (int i = 0; i < kChainRun; i++) em = em > ex[i] ? em : ex[i];
                em = __reduce_max_sync(kAll, em);
                if (lane == 0) sm.e[w] = em;
            }
            double hp = __shfl_up_sync(kAll, h, 1);
            __syncthreads();
            if (lane == 0) hp = w ? sm.h[w - 1] : s;
            const bool off = __double_as_longlong(hp) != __double_as_longlong(g);
            if (!__syncthreads_or(off)) {
                s = sm.h[kWarps - 1];
                break;
            }
            if (round >= 2 * kChainRounds) {
                // finish from the first run whose start is known but wrong
                if (tid == 0) sm.first = kChainThreads;
                __syncthreads();
                if (off) atomicMin(&sm.first, tid);
                __syncthreads();
                const int f = sm.first;
                if (tid == f) sm.s = hp;
                __syncthreads();
                s = sm.s;
                const double* all = sm.v[t % kChainStages];
                for (int l = f; l < kChainThreads; l++)
#pragma unroll
                    for (int i = 0; i < kChainRun; i++) s += all[l * kChainPitch + i];
                break;
            }
            if (!learn) continue;
            int q = 0;
#pragma unroll
            for (int k = 0; k < kWarps; k++) q = q > sm.e[k] ? q : sm.e[k];
            q -= 107 - 52;
            const long long gap = chain_units(hp - g, q);
            ChainMap m{0, 0, 1};
            int last = (__double2hiint(g) >> 20) & 0x7ff;
#pragma unroll
            for (int i = 0; i < kChainRun; i++) {
                // a tie between sums on the step's own grid ends on an even
                // one whatever d was: a step on the doubled grid
                const unsigned long long ay = (unsigned long long)__double_as_longlong(y[i]) << 1;
                const bool tie = ay == (unsigned long long)(ex[i] - 53) << 53 && last >= ex[i];
                last = ex[i];
                const int j = ex[i] - q + (tie ? 1 : 0);
                const long long u = j > 0 ? 1LL << j : 1;
                if (u > m.u) {
                    const long long hu = u >> 1;
                    long long yu = chain_units(y[i], q);
                    if (tie) yu = yu > 0 ? 0 : -1;
                    yu = yu < hu ? yu : hu - 1;  // (chain_rn takes a half up: one that went down stays below it)
                    m.b += hu - chain_ceil(hu - yu, m.u) + (m.u >> 1);
                    m.u = u;
                }
            }
            m.b += gap;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                ChainMap f;
                f.b = __shfl_up_sync(kAll, m.b, o);
                f.c = __shfl_up_sync(kAll, m.c, o);
                f.u = __shfl_up_sync(kAll, m.u, o);
                if (lane >= o) m = chain_then(f, m);
            }
            if (lane == 31) sm.m[w] = m;
            __syncthreads();
            long long d = 0;  // the deviation of the end before this warp
            for (int k = 0; k < w; k++) d = sm.m[k].c + chain_rn(d + sm.m[k].b, sm.m[k].u);
            long long mine = m.c + chain_rn(d + m.b, m.u);
            const long long before = __shfl_up_sync(kAll, mine, 1);
            d = lane ? before : d;
            if (d == 0) {
                g = hp;  // the run before this one stands
            } else {
                // g += gap + d, in two parts that a double holds exactly
                d += gap;
                const long long dh = (d >> 30) << 30, dl = d - dh;
                const int sc = q - 1075 + 1023;  // the unit's exponent field
                const double one = __hiloint2double((sc > 0 ? sc : 1) << 20, 0);
                g = (g + (double)dh * one) + (double)dl * one;
            }
            __syncthreads();  // sm.m, sm.h, sm.e are read
        }
        __syncthreads();  // the slot and sm.h are read
        issue(t + kChainStages - 1);
    }
    cp_async_wait<0>();
    return s;
}

}  // namespace mce
