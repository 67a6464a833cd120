// Vortex merging, VortexBlobs::merge_blobs (src/VortexBlobs.cpp:110-209),
// hooked at src/DVMBase.cpp:124-132.
//
// The reference merges greedily in index order: each surviving blob i absorbs,
// one after another, every later unmerged j with |gi gj / (gi + gj)| |xi - xj|
// < threshold, where i's position, circulation and core size are updated after
// every absorption; then merged blobs are removed (stable) and IDs renumbered.
// The result depends on that order, so it is reproduced exactly.  At i's turn every
// later blob still has its original position, circulation and core size (only
// absorbers change, and they come in order), so what i absorbs -- its chain --
// depends on its original state and on which later blobs earlier absorbers have
// taken.  That is a fixed-point problem, solved by rounds in parallel:
//   chain of i = what i absorbs, in order, among the j with own[j] >= i (empty
//   when i itself is owned);
//   own[j] = the least i whose chain holds j;
// repeated until no owner changes.  By induction over i a fixed point is the
// sequential result, and each round makes at least one more chain final; a wake's
// settle in about five.  (k_mg_lists finds each blob's qualifying partners once,
// so most blobs of a round only look up whether one is left.)  If the rounds do
// not settle, or the second one takes more than kOrderedShare of all blobs (long
// chains, which one warp each would go through again and again), one block
// walks the absorbers in order instead, searching together for each
// (k_merge_greedy); so it does for a few blobs, for lists that are mostly long, and when there
// is no memory for them.
// Then merged blobs are removed (stable) and IDs renumbered.  Every arithmetic
// step is the reference's, in FP64 with one rounding per operation, so the merged
// state is bit-identical.  A division-free pre-test rejects pairs that cannot
// pass: crit < thr implies (|gi gj| d)^2 < (thr |gi + gj|)^2, and the test keeps
// a 1e-12 relative margin so rounding can never reject a pair the exact formula
// would accept.
//
// Candidates are found through a cell grid when that is safe: since |gi + gj| <=
// |gi| + |gj| a pair can pass only if |xi - xj| < thr (1/|gj| + 1/|gi|).  Blobs
// with the smallest |g| (4 sqrt(n) of them at most, plus any non-finite one) sit in
// a short list scanned at every search; the others are sorted by cell, and a
// search reads the cells within thr (1/g_cut + 1/|gi|) of the absorber (g_cut:
// the smallest |g| in the grid), row by row, falling back to the full scan when
// that radius is large or undefined.  The least qualifying index over the
// candidates is the full scan's first, so the result is unchanged.
//
// Measured (B200, wake, threshold 2e-6, host arrays): 20 k blobs 57.6 -> 1.37 ms
// (a walk of the absorbers in order, one block searching for each, took 53; with
// chains as a first guess it still took 58, since most blobs' partners are taken
// by earlier ones).
#include <cfloat>
#include <algorithm>
#include <cmath>
#include <vector>

#include <cub/cub.cuh>

#include "dvm_device.cuh"
#include "dvm_internal.h"

namespace dvmk {
namespace {

constexpr int kMergeThreads = 1024;
constexpr int kList = 24;              // partners of a blob kept
constexpr uint32_t kFirstMost = 32;    // members in the first two rounds: at a threshold that
                                       // merges everything, each blob would take all later ones
// Share of the blobs taken in the second round from which the ordered walk is the
// faster one (20 k blobs: 32 % merged, rounds 10 ms, walk 62; 58 %, 178 and 73).
constexpr double kOrderedShare = 0.45;
// Share of the blobs with more than kList partners from which that is so in advance (wakes of
// 3000 to 20 000: from 0.67 on the second round takes 49 % and more, at 0.49 32 %).
constexpr double kLongShare = 0.6;
constexpr uint32_t kRoundsMin = 256;   // blobs below which the walk takes less than the rounds' launches
                                       // (10, 100: 180, 190 us against 235, 230; 300: 212, 235 at a
                                       // threshold that merges little, 388 and 336 at one that does)
constexpr int kRoundsMax = 64;         // rounds before the ordered pass takes over
constexpr uint32_t kLookFirst = 32768; // blobs up to which the walk looks who is left first
constexpr uint32_t kLong = 0xFFu;      // as a list's length: more than kList
constexpr uint32_t kSmallList = 2048;  // blobs kept out of the grid, at most
constexpr int kGridMax = 1024;         // cells per axis, at most (and about two per sqrt(n))
constexpr int kCellReach = 8;          // a pass searches at most this many cells of radius

struct MergeGrid {
    double x0, z0, inv_h, h, g_cut;
    int nxc, nzc, enabled;
    const double4* cand;     // (x, z, circ, index), cell-sorted; from cbegin[cells] on the short list
    const uint32_t* svals;   // their indices alone
    const uint32_t* cbegin;  // first candidate of each cell, and of the short list
};

// The reference's test for the pair (i's current state, j): crit < thr.
__device__ __forceinline__ bool merge_test(double xi, double zi, double gi, double xj, double zj,
                                           double gj, double thr) {
    const double gs = dadd(gi, gj);
    if (fabs(gs) < 1e-15) return false;
    const double dx = dsub(xi, xj), dz = dsub(zi, zj);
    const double d2 = dadd(dmul(dx, dx), dmul(dz, dz));
    const double a = fabs(dmul(gi, gj)), b = dmul(thr, fabs(gs));
    if (a < 1e100 && b < 1e100 && a > 1e-140 && b > 1e-140 &&
        dmul(dmul(a, a), d2) > dmul(dmul(b, b), 1.000000000001))
        return false;  // cannot pass the exact test below
    const double crit = dmul(fabs(ddiv(dmul(gi, gj), gs)), __dsqrt_rn(d2));
    return crit < thr;
}

// Cell range to search for absorber state (xi, zi, gi); false: scan everything.
__device__ __forceinline__ bool cell_range(const MergeGrid& G, double xi, double zi, double gi,
                                           double thr, long long& cx0, long long& cx1,
                                           long long& cz0, long long& cz1) {
    if (!G.enabled) return false;
    const double R = thr * (1.0 / G.g_cut + 1.0 / fabs(gi)) * (1.0 + 1e-9);
    if (!(R < kCellReach * G.h) || !(fabs(xi) < 1e300) || !(fabs(zi) < 1e300)) return false;
    // cell coordinates clamped as doubles before the integer conversion
    auto cell = [&](double v, int nc) {
        return (long long)floor(fmin(fmax(v, -2.0), (double)nc + 1.0));
    };
    cx0 = max(0LL, cell((xi - R - G.x0) * G.inv_h, G.nxc) - 1);
    cx1 = min((long long)G.nxc - 1, cell((xi + R - G.x0) * G.inv_h, G.nxc) + 1);
    cz0 = max(0LL, cell((zi - R - G.z0) * G.inv_h, G.nzc) - 1);
    cz1 = min((long long)G.nzc - 1, cell((zi + R - G.z0) * G.inv_h, G.nzc) + 1);
    return true;
}

struct Blobs {
    const double *x, *z, *circ, *sigma;
};
// A blob's state as an absorber.
struct Absorber {
    double x, z, g, s;
};
__device__ __forceinline__ void absorb(Absorber& a, const Blobs& B, uint32_t j) {
    const double gj = B.circ[j], gs = dadd(a.g, gj);
    const double nx = ddiv(dadd(dmul(a.g, a.x), dmul(gj, B.x[j])), gs);
    const double nz = ddiv(dadd(dmul(a.g, a.z), dmul(gj, B.z[j])), gs);
    const double ns = ddiv(dadd(dmul(fabs(a.g), a.s), dmul(fabs(gj), B.sigma[j])),
                           dadd(fabs(a.g), fabs(gj)));
    a = Absorber{nx, nz, gs, ns};
}

// Not taken by an absorber before i.
struct Free {
    const uint32_t* own;
    uint32_t i;
    __device__ __forceinline__ bool operator()(uint32_t j) const { return own[j] >= i; }
};
// The first j >= j0 that the absorber takes among the blobs `there`, by a warp (the
// result is each lane's own least: the warp takes the minimum).
template <typename There>
__device__ __forceinline__ uint32_t search(const Blobs& B, const MergeGrid& G, uint32_t n, double thr,
                                           const Absorber& a, uint32_t j0, const There& there,
                                           uint32_t lane) {
    long long cx0, cx1, cz0, cz1;
    if (!cell_range(G, a.x, a.z, a.g, thr, cx0, cx1, cz0, cz1)) {
        for (uint32_t j = j0; j < n; j += 32) {  // done at the first 32 with a taker
            const uint32_t q = j + lane;
            const bool hit = q < n && there(q) &&
                             merge_test(a.x, a.z, a.g, B.x[q], B.z[q], B.circ[q], thr);
            if (__any_sync(0xffffffffu, hit)) return hit ? q : UINT32_MAX;
        }
        return UINT32_MAX;
    }
    uint32_t best = UINT32_MAX;
    auto look = [&](uint32_t q) {
        const double4 c = G.cand[q];
        const uint32_t j = (uint32_t)__double_as_longlong(c.w);
        if (j >= j0 && j < best && there(j) && merge_test(a.x, a.z, a.g, c.x, c.y, c.z, thr)) best = j;
    };
    for (long long cz = cz0; cz <= cz1; ++cz) {
        const uint64_t r = (uint64_t)cz * G.nxc;
        const uint32_t q1 = G.cbegin[r + cx1 + 1];
        for (uint32_t q = G.cbegin[r + cx0] + lane; q < q1; q += 32) look(q);
    }
    for (uint32_t q = G.cbegin[(uint64_t)G.nxc * G.nzc] + lane; q < n; q += 32) look(q);
    return best;
}

// Partners of every blob in its original state, in no particular order; nl[i] =
// their number, or kLong when there are more than kList (without lists: more than
// none).  One warp per blob.
__global__ void __launch_bounds__(256) k_mg_lists(Blobs B, uint32_t n, double thr, MergeGrid G,
                                                  uint32_t* __restrict__ nl,
                                                  uint32_t* __restrict__ lists,
                                                  uint32_t* __restrict__ n_long) {
    const unsigned all = 0xffffffffu;
    const uint32_t room = lists ? kList : 0;
    uint32_t many = 0;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t i = warp; i < n; i += warps) {
        const double xi = B.x[i], zi = B.z[i], gi = B.circ[i];
        uint32_t* __restrict__ out = lists + (uint64_t)i * room;
        uint32_t m = 0;  // warp-uniform
        auto add = [&](bool hit, uint32_t j) {
            const unsigned b = __ballot_sync(all, hit);
            const uint32_t at = m + __popc(b & ((1u << lane) - 1u));
            if (hit && at < room) out[at] = j;
            m += __popc(b);
        };
        auto look = [&](uint32_t q, bool in) {
            bool hit = false;
            uint32_t j = 0;
            if (in) {
                const double4 c = G.cand[q];
                j = (uint32_t)__double_as_longlong(c.w);
                hit = j > i && merge_test(xi, zi, gi, c.x, c.y, c.z, thr);
            }
            add(hit, j);
        };
        long long cx0, cx1, cz0, cz1;
        if (!cell_range(G, xi, zi, gi, thr, cx0, cx1, cz0, cz1)) {
            for (uint32_t j = i + 1; j < n && m <= room; j += 32) {
                const uint32_t q = j + lane;
                add(q < n && merge_test(xi, zi, gi, B.x[q], B.z[q], B.circ[q], thr), q);
            }
        } else {
            for (long long cz = cz0; cz <= cz1 && m <= room; ++cz) {
                const uint64_t r = (uint64_t)cz * G.nxc;
                const uint32_t q1 = G.cbegin[r + cx1 + 1];
                for (uint32_t q = G.cbegin[r + cx0]; q < q1; q += 32) look(q + lane, q + lane < q1);
            }
            for (uint32_t q = G.cbegin[(uint64_t)G.nxc * G.nzc]; q < n && m <= room; q += 32)
                look(q + lane, q + lane < n);
        }
        if (lane == 0) nl[i] = m > room ? kLong : m;
        many += m > room;
    }
    if (n_long && lane == 0 && many) atomicAdd(n_long, many);
}

// First guess of the owners: as if every blob took all its partners.
__global__ void k_mg_guess(const uint32_t* __restrict__ who, const uint32_t* __restrict__ n_who,
                           const uint32_t* __restrict__ nl, const uint32_t* __restrict__ lists,
                           uint32_t* __restrict__ own) {
    const uint32_t m = n_who[0];
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < m; t += gridDim.x * blockDim.x) {
        const uint32_t i = who[t];
        const uint32_t l = min(nl[i], (uint32_t)kList);
        for (uint32_t q = 0; q < l; ++q) atomicMin(&own[lists[(uint64_t)i * kList + q]], i);
    }
}

// A round in three launches: next owners cleared; every blob that has partners
// absorbs, given the owners, and claims what it takes (one warp per blob); owners
// compared.  flags[0]: some owner changed; flags[-1]: in the round before (when
// none had, there is nothing to do, and both owner arrays stay as they are).
// Nor is there when too many blobs have long lists.
struct Tally {  // of a merge
    uint32_t taken;   // blobs owned after the second round
    uint32_t n_long;  // blobs with more than kList partners
};
__device__ __forceinline__ bool idle(const uint32_t* flags, const Tally* t, uint32_t n) {
    return flags[-1] == 0 || t->n_long > kLongShare * n;
}
__global__ void k_mg_clear(uint32_t n, const uint32_t* __restrict__ flags, const Tally* __restrict__ tally,
                           uint32_t* __restrict__ next) {
    if (idle(flags, tally, n)) return;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x)
        next[p] = UINT32_MAX;
}

__global__ void __launch_bounds__(256) k_mg_round(Blobs B, uint32_t n, double thr, MergeGrid G,
                                                  const uint32_t* __restrict__ who,
                                                  const uint32_t* __restrict__ n_who,
                                                  const uint32_t* __restrict__ nl,
                                                  const uint32_t* __restrict__ lists,
                                                  const uint32_t* __restrict__ own,
                                                  uint32_t* __restrict__ next,
                                                  uint32_t* __restrict__ len,
                                                  double4* __restrict__ after, uint32_t most,
                                                  uint32_t* __restrict__ flags,
                                                  const Tally* __restrict__ tally) {
    if (idle(flags, tally, n)) return;
    const unsigned all = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31, m = n_who[0];
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < m; t += warps) {
        const uint32_t i = who[t], l = nl[i];
        const Free free{own, i};
        uint32_t got = 0;
        if (own[i] == UINT32_MAX) {
            Absorber a{B.x[i], B.z[i], B.circ[i], B.sigma[i]};
            uint32_t j = UINT32_MAX;
            if (l == kLong) {
                j = search(B, G, n, thr, a, i + 1, free, lane);
            } else if (lane < l) {
                const uint32_t q = lists[(uint64_t)i * kList + lane];
                if (free(q)) j = q;
            }
            for (j = __reduce_min_sync(all, j); j != UINT32_MAX; ++got) {
                if (got == most) {  // the round does not count as settled
                    if (lane == 0) flags[0] = 1;
                    break;
                }
                if (lane == 0) atomicMin(&next[j], i);
                absorb(a, B, j);
                j = __reduce_min_sync(all, search(B, G, n, thr, a, j + 1, free, lane));
            }
            if (lane == 0 && got) after[i] = make_double4(a.x, a.z, a.g, a.s);
        }
        if (lane == 0) len[i] = got;
    }
}

__global__ void k_mg_compare(uint32_t n, const uint32_t* __restrict__ own,
                             const uint32_t* __restrict__ next, uint32_t* __restrict__ flags,
                             Tally* tally, bool second) {
    if (idle(flags, tally, n)) return;
    uint32_t mine = 0;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        if (own[p] != next[p]) flags[0] = 1;
        mine += next[p] != UINT32_MAX;
    }
    if (second) {
        mine = __reduce_add_sync(0xffffffffu, mine);
        if ((threadIdx.x & 31) == 0 && mine) atomicAdd(&tally->taken, mine);
    }
}

// The ordered walk: absorbers ascending, each searched for by the whole block, in
// place.
__global__ void __launch_bounds__(kMergeThreads, 1)
    k_merge_greedy(double* __restrict__ x, double* __restrict__ z, double* __restrict__ circ,
                   double* __restrict__ sigma, double* __restrict__ u, double* __restrict__ w,
                   double* __restrict__ uvs, double* __restrict__ wvs, uint32_t n, double thr,
                   MergeGrid G, const uint32_t* __restrict__ absorbers,
                   const uint32_t* __restrict__ n_abs, uint32_t* __restrict__ keep,
                   uint32_t* __restrict__ count) {
    using Reduce = cub::BlockReduce<uint32_t, kMergeThreads>;
    __shared__ typename Reduce::TempStorage red;
    __shared__ double si[4];  // x, z, circ, sigma of the current absorber
    __shared__ uint32_t s_best;
    const uint32_t tid = threadIdx.x;
    for (uint32_t p = tid; p < n; p += kMergeThreads) keep[p] = 1u;
    const uint32_t n_grid = G.enabled ? G.cbegin[(uint64_t)G.nxc * G.nzc] : 0;
    __syncthreads();
    uint32_t merges = 0;
    const uint32_t na = n_abs[0];
    for (uint32_t t = 0; t < na; ++t) {
        const uint32_t i = absorbers[t];  // ascending: the reference's order
        if (!keep[i]) continue;           // every thread reads the same value
        if (tid == 0) {
            si[0] = x[i];
            si[1] = z[i];
            si[2] = circ[i];
            si[3] = sigma[i];
        }
        __syncthreads();
        uint32_t j0 = i + 1;
        while (j0 < n) {
            const double xi = si[0], zi = si[1], gi = si[2];
            uint32_t best = UINT32_MAX;
            // Most of the blobs that this walk meets are merged already, so whether one is left
            // comes before its position and the test, as long as `keep` stays in the L1
            // cache (10 k, 20 k blobs, 98, 82 % merged: 215 and 135 ms the other way round, 134 and
            // 122 so; 60 k, 95 %: 4.6 s and 5.2).
            auto look = [&](uint32_t q) {
                if (n <= kLookFirst) {
                    const uint32_t j = G.svals[q];
                    if (j < j0 || j >= best || !keep[j]) return;
                    const double4 v = G.cand[q];
                    if (merge_test(xi, zi, gi, v.x, v.y, v.z, thr)) best = j;
                } else {
                    const double4 v = G.cand[q];  // (a later blob is as it was)
                    const uint32_t j = (uint32_t)__double_as_longlong(v.w);
                    if (j < j0 || j >= best) return;
                    if (merge_test(xi, zi, gi, v.x, v.y, v.z, thr) && keep[j]) best = j;
                }
            };
            // cell range of this pass (the same decision in every thread)
            long long cx0 = 0, cx1 = -1, cz0 = 0, cz1 = -1;
            const bool full = !cell_range(G, xi, zi, gi, thr, cx0, cx1, cz0, cz1);
            if (full) {
                for (uint32_t j = j0 + tid; j < n; j += kMergeThreads) {
                    if (!keep[j]) continue;
                    if (merge_test(xi, zi, gi, x[j], z[j], circ[j], thr)) {
                        best = j;  // this thread's candidates ascend: its first is its least
                        break;
                    }
                }
            } else {
                // one warp per cell, so the cells' bounds are loaded concurrently
                const long long ncx = cx1 - cx0 + 1, ncell = ncx * (cz1 - cz0 + 1);
                const uint32_t warp = tid >> 5, lane = tid & 31;
                for (long long k = warp; k < ncell; k += kMergeThreads / 32) {
                    const uint64_t c = (uint64_t)(cz0 + k / ncx) * G.nxc + (cx0 + k % ncx);
                    for (uint32_t q = G.cbegin[c] + lane; q < G.cbegin[c + 1]; q += 32) {
                        look(q);
                    }
                }
                for (uint32_t q = n_grid + tid; q < n; q += kMergeThreads) {
                    look(q);
                }
            }
            best = Reduce(red).Reduce(best, cub::Min());
            if (tid == 0) s_best = best;
            __syncthreads();
            best = s_best;
            if (best == UINT32_MAX) break;
            if (tid == 0) {
                const double gj = circ[best], gs = dadd(gi, gj);
                const double nx = ddiv(dadd(dmul(gi, xi), dmul(gj, x[best])), gs);
                const double nz = ddiv(dadd(dmul(gi, zi), dmul(gj, z[best])), gs);
                const double ns = ddiv(dadd(dmul(fabs(gi), si[3]), dmul(fabs(gj), sigma[best])),
                                       dadd(fabs(gi), fabs(gj)));
                si[0] = x[i] = nx;
                si[1] = z[i] = nz;
                si[2] = circ[i] = gs;
                si[3] = sigma[i] = ns;
                u[i] = w[i] = uvs[i] = wvs[i] = 0.0;
                keep[best] = 0u;
                ++merges;
            }
            __syncthreads();
            j0 = best + 1;
        }
        __syncthreads();
    }
    if (tid == 0) count[0] = merges;
}

// The settled rounds: keep flags, the merge count, and the absorbers' new states.
__global__ void k_mg_apply(MergeArrays a, uint32_t n, const uint32_t* __restrict__ nl,
                           const uint32_t* __restrict__ len, const uint32_t* __restrict__ own,
                           const double4* __restrict__ after, uint32_t* __restrict__ keep,
                           uint32_t* __restrict__ count) {
    uint32_t gone = 0;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const uint32_t k = own[p] == UINT32_MAX;
        keep[p] = k;
        gone += 1 - k;
        if (!nl[p] || !len[p]) continue;
        const double4 v = after[p];
        a.x[p] = v.x;
        a.z[p] = v.y;
        a.circ[p] = v.z;
        a.sigma[p] = v.w;
        a.u[p] = a.w[p] = a.uvs[p] = a.wvs[p] = 0.0;
    }
    gone = __reduce_add_sync(0xffffffffu, gone);
    if ((threadIdx.x & 31) == 0 && gone) atomicAdd(count, gone);
}

// |g| as sortable bits (non-finite last) and the bounding box of the finite
// positions, per block.
__global__ void k_mg_stats(const double* __restrict__ x, const double* __restrict__ z,
                           const double* __restrict__ circ, uint32_t n,
                           uint64_t* __restrict__ gbits, double4* __restrict__ part) {
    double xmn = DBL_MAX, xmx = -DBL_MAX, zmn = DBL_MAX, zmx = -DBL_MAX;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const double g = fabs(circ[p]);
        gbits[p] = (g <= DBL_MAX) ? (uint64_t)__double_as_longlong(g) : 0x7FF0000000000000ull;
        if (fabs(x[p]) < 1e300 && fabs(z[p]) < 1e300) {
            xmn = fmin(xmn, x[p]);
            xmx = fmax(xmx, x[p]);
            zmn = fmin(zmn, z[p]);
            zmx = fmax(zmx, z[p]);
        }
    }
    using R = cub::BlockReduce<double, 256>;
    __shared__ typename R::TempStorage t;
    xmn = R(t).Reduce(xmn, cub::Min());
    __syncthreads();
    xmx = R(t).Reduce(xmx, cub::Max());
    __syncthreads();
    zmn = R(t).Reduce(zmn, cub::Min());
    __syncthreads();
    zmx = R(t).Reduce(zmx, cub::Max());
    if (threadIdx.x == 0) part[blockIdx.x] = make_double4(xmn, xmx, zmn, zmx);
}

__global__ void k_mg_classify(const double* __restrict__ x, const double* __restrict__ z,
                              const double* __restrict__ circ, uint32_t n, double x0, double z0,
                              double inv_h, int nxc, int nzc, double g_cut,
                              uint64_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    const uint64_t sentinel = (uint64_t)nxc * nzc;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const double g = fabs(circ[p]);
        uint64_t k = sentinel;
        if (g >= g_cut && g <= DBL_MAX && fabs(x[p]) < 1e300 && fabs(z[p]) < 1e300) {
            const long long cx = (long long)floor((x[p] - x0) * inv_h);
            const long long cz = (long long)floor((z[p] - z0) * inv_h);
            if (cx >= 0 && cx < nxc && cz >= 0 && cz < nzc) k = (uint64_t)cz * nxc + cx;
        }
        keys[p] = k;
        vals[p] = p;
    }
}

// Candidates in cell order, and where each cell's begin (binary search).
__global__ void k_mg_cells(const double* __restrict__ x, const double* __restrict__ z,
                           const double* __restrict__ circ, const uint64_t* __restrict__ skeys,
                           const uint32_t* __restrict__ svals, uint32_t n, uint64_t ncells,
                           double4* __restrict__ cand, uint32_t* __restrict__ cbegin) {
    const uint64_t t0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t q = t0; q < n; q += step) {
        const uint32_t j = svals[q];
        cand[q] = make_double4(x[j], z[j], circ[j], __longlong_as_double((long long)j));
    }
    for (uint64_t c = t0; c <= ncells; c += step) {
        uint32_t lo = 0, hi = n;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (skeys[mid] < c) lo = mid + 1;
            else hi = mid;
        }
        cbegin[c] = lo;
    }
}

__global__ void k_merge_scatter(const uint32_t* __restrict__ count, uint32_t n,
                                const uint32_t* __restrict__ keep, const uint32_t* __restrict__ pos,
                                MergeArrays a, MergeArrays t) {
    if (count[0] == 0) return;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        if (!keep[p]) continue;
        const uint32_t o = pos[p];
        t.x[o] = a.x[p];
        t.z[o] = a.z[p];
        t.circ[o] = a.circ[p];
        t.sigma[o] = a.sigma[p];
        t.u[o] = a.u[p];
        t.w[o] = a.w[p];
        t.uvs[o] = a.uvs[p];
        t.wvs[o] = a.wvs[p];
    }
}

__global__ void k_merge_copyback(const uint32_t* __restrict__ count, uint32_t n, MergeArrays t,
                                 MergeArrays a, uint32_t* __restrict__ id,
                                 uint32_t* __restrict__ n_dev) {
    const uint32_t c = count[0];
    if (c == 0) return;  // nothing merged: IDs unchanged (src/VortexBlobs.cpp:171-173)
    const uint32_t m = n - c;
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < m; q += gridDim.x * blockDim.x) {
        a.x[q] = t.x[q];
        a.z[q] = t.z[q];
        a.circ[q] = t.circ[q];
        a.sigma[q] = t.sigma[q];
        a.u[q] = t.u[q];
        a.w[q] = t.w[q];
        a.uvs[q] = t.uvs[q];
        a.wvs[q] = t.wvs[q];
        if (id) id[q] = q;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && n_dev) n_dev[0] = m;
}

struct MLayout {
    size_t keep, pos, tmp, tmp_bytes, t, count, gbits, gsorted, keys, skeys, vals, svals, cand,
        cbegin, part, scal, len, after, alist, nl, lists, own, flags, bytes;
};

constexpr int kStatBlocks = 256;

int sort_bits(uint64_t v) {
    int b = 1;
    while (b < 64 && (1ull << b) <= v) ++b;
    return b;
}

// Scratch of a merge (about 300 bytes per blob), or, without room for the rounds' lists, of
// the ordered walk alone (half of that; the candidates then lie where the merged
// blobs are gathered later).
MLayout mlayout(uint32_t n, bool rounds) {
    const uint64_t ncells = (uint64_t)kGridMax * kGridMax;
    size_t scan_b = 0, sk_b = 0, sp_b = 0, sel_b = 0;
    const int64_t nn = (int64_t)std::max<uint32_t>(n, 1);
    cub::DeviceScan::ExclusiveSum(nullptr, scan_b, (const uint32_t*)nullptr, (uint32_t*)nullptr, nn);
    cub::DeviceRadixSort::SortKeys(nullptr, sk_b, (const uint64_t*)nullptr, (uint64_t*)nullptr, nn);
    cub::DeviceRadixSort::SortPairs(nullptr, sp_b, (const uint64_t*)nullptr, (uint64_t*)nullptr,
                                    (const uint32_t*)nullptr, (uint32_t*)nullptr, nn, 0,
                                    sort_bits(ncells));
    cub::DeviceSelect::Flagged(nullptr, sel_b, cub::CountingInputIterator<uint32_t>(0),
                               (const uint32_t*)nullptr, (uint32_t*)nullptr, (uint32_t*)nullptr,
                               nn);
    MLayout L{};
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += (bytes + 255) / 256 * 256;
        return o;
    };
    L.keep = take(4ull * n + 4);
    L.pos = take(4ull * n + 4);
    L.tmp_bytes = std::max({scan_b, sk_b, sp_b, sel_b}) + 256;
    L.tmp = take(L.tmp_bytes);
    L.t = take(8 * 8ull * n + 8);
    L.count = take(64);
    L.gbits = take(8ull * n + 8);
    L.gsorted = take(8ull * n + 8);
    L.keys = take(8ull * n + 8);
    L.skeys = take(8ull * n + 8);
    L.vals = take(4ull * n + 4);
    L.svals = take(4ull * n + 4);
    L.cand = rounds ? take(32ull * n + 32) : L.t;
    L.cbegin = take(4 * (ncells + 1));
    L.part = take(sizeof(double4) * kStatBlocks);
    L.scal = take(128);
    L.alist = take(4ull * n + 4);
    L.nl = take(4ull * n + 4);
    if (rounds) {
        L.len = take(4ull * n + 4);
        L.after = take(32ull * n + 32);
        L.lists = take(4ull * kList * n + 4);
        L.own = take(8ull * n + 8);
        L.flags = take(4 * (kRoundsMax + 1) + sizeof(Tally));
    }
    L.bytes = off;
    return L;
}

// Builds the candidate grid with a short list of `small` blobs and at most gmax
// cells per axis (synchronises the stream once to size it); leaves
// G.enabled = 0 when a grid would not narrow the search.
MergeGrid build_grid(const MergeArrays& a, uint32_t n, double thr, uint32_t small, int gmax,
                     const MLayout& L, char* b, cudaStream_t s) {
    MergeGrid G{};
    G.enabled = 0;
    if (n < 4096) return G;  // the full scan is cheap
    uint64_t* gbits = reinterpret_cast<uint64_t*>(b + L.gbits);
    uint64_t* gsorted = reinterpret_cast<uint64_t*>(b + L.gsorted);
    double4* part = reinterpret_cast<double4*>(b + L.part);
    k_mg_stats<<<kStatBlocks, 256, 0, s>>>(a.x, a.z, a.circ, n, gbits, part);
    size_t tb = L.tmp_bytes;
    cub::DeviceRadixSort::SortKeys(b + L.tmp, tb, gbits, gsorted, (int64_t)n, 0, 64, s);
    const uint32_t k = std::min(small, n);
    double g_cut = 0.0, g_med = 0.0;  // (|g| sorted as bits: the bits are the values)
    std::vector<double4> h_part(kStatBlocks);
    cudaMemcpyAsync(&g_cut, gsorted + (k - 1), 8, cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(&g_med, gsorted + n / 2, 8, cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(h_part.data(), part, sizeof(double4) * kStatBlocks, cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) return G;
    double xmn = DBL_MAX, xmx = -DBL_MAX, zmn = DBL_MAX, zmx = -DBL_MAX;
    for (const double4& v : h_part) {
        xmn = std::min(xmn, v.x);
        xmx = std::max(xmx, v.y);
        zmn = std::min(zmn, v.z);
        zmx = std::max(zmx, v.w);
    }
    if (!(g_cut > 0) || !(g_cut <= DBL_MAX) || !(xmx >= xmn) || !(zmx >= zmn)) return G;
    const double span = std::max({xmx - xmn, zmx - zmn, 1e-300});
    const double r_typ = thr * (1.0 / g_cut + 1.0 / g_med);
    if (!(r_typ > 0) || !(r_typ < span / 4)) return G;  // a grid would not narrow the search
    const double h = std::max(r_typ, span / (gmax - 1));
    G.h = h;
    G.inv_h = 1.0 / h;
    G.x0 = xmn;
    G.z0 = zmn;
    G.nxc = std::min(gmax, (int)std::floor((xmx - xmn) * G.inv_h) + 1);
    G.nzc = std::min(gmax, (int)std::floor((zmx - zmn) * G.inv_h) + 1);
    G.g_cut = g_cut;
    const uint64_t ncells = (uint64_t)G.nxc * G.nzc;
    uint64_t* keys = reinterpret_cast<uint64_t*>(b + L.keys);
    uint64_t* skeys = reinterpret_cast<uint64_t*>(b + L.skeys);
    uint32_t* vals = reinterpret_cast<uint32_t*>(b + L.vals);
    uint32_t* svals = reinterpret_cast<uint32_t*>(b + L.svals);
    double4* cand = reinterpret_cast<double4*>(b + L.cand);
    uint32_t* cbegin = reinterpret_cast<uint32_t*>(b + L.cbegin);
    k_mg_classify<<<256, 256, 0, s>>>(a.x, a.z, a.circ, n, G.x0, G.z0, G.inv_h, G.nxc, G.nzc,
                                      g_cut, keys, vals);
    tb = L.tmp_bytes;
    cub::DeviceRadixSort::SortPairs(b + L.tmp, tb, keys, skeys, vals, svals, (int64_t)n, 0,
                                    sort_bits(ncells), s);
    k_mg_cells<<<592, 256, 0, s>>>(a.x, a.z, a.circ, skeys, svals, n, ncells, cand, cbegin);
    G.cand = cand;
    G.cbegin = cbegin;
    G.svals = svals;
    G.enabled = 1;
    return G;
}

}  // namespace

size_t merge_scratch_bytes(uint32_t n, bool rounds) { return mlayout(n, rounds).bytes; }
size_t merge_count_offset(uint32_t n) { return mlayout(n, false).count; }

void merge_run(const MergeArrays& a, uint32_t* id, uint32_t n, double threshold,
               uint32_t* n_dev, uint32_t* count_dev, void* scratch, bool rounds, int sms,
               cudaStream_t s) {
    const MLayout L = mlayout(n, rounds);
    char* b = static_cast<char*>(scratch);
    uint32_t* keep = reinterpret_cast<uint32_t*>(b + L.keep);
    uint32_t* pos = reinterpret_cast<uint32_t*>(b + L.pos);
    double* t0 = reinterpret_cast<double*>(b + L.t);
    MergeArrays t{t0, t0 + n, t0 + 2ull * n, t0 + 3ull * n, t0 + 4ull * n, t0 + 5ull * n,
                  t0 + 6ull * n, t0 + 7ull * n};
    uint32_t* count = count_dev ? count_dev : reinterpret_cast<uint32_t*>(b + L.count);
    if (n < 2 || !(threshold > 0)) {  // crit >= 0 never passes a threshold <= 0
        cudaMemsetAsync(count, 0, sizeof(uint32_t), s);
        return;
    }
    rounds = rounds && n >= kRoundsMin;
    // a warp's search likes a short list and about four cells per blob
    const int root = (int)std::sqrt((double)n);
    const MergeGrid G =
        build_grid(a, n, threshold, std::min<uint32_t>(kSmallList, 4 * root),
                   std::max(64, std::min(kGridMax, 2 * root)), L, b, s);
    uint32_t* len = reinterpret_cast<uint32_t*>(b + L.len);
    double4* after = reinterpret_cast<double4*>(b + L.after);
    uint32_t* alist = reinterpret_cast<uint32_t*>(b + L.alist);
    uint32_t* n_abs = reinterpret_cast<uint32_t*>(b + L.scal) + 4;
    const Blobs B{a.x, a.z, a.circ, a.sigma};
    uint32_t* nl = reinterpret_cast<uint32_t*>(b + L.nl);
    uint32_t* lists = rounds ? reinterpret_cast<uint32_t*>(b + L.lists) : nullptr;
    uint32_t* own[2] = {reinterpret_cast<uint32_t*>(b + L.own),
                        reinterpret_cast<uint32_t*>(b + L.own) + n};
    uint32_t* flags = reinterpret_cast<uint32_t*>(b + L.flags) + 1;  // one per round
    Tally* tally = reinterpret_cast<Tally*>(flags + kRoundsMax);
    if (rounds) {
        cudaMemsetAsync(flags - 1, 1, 4, s);  // (anything but 0: the first round runs)
        cudaMemsetAsync(flags, 0, 4 * kRoundsMax + sizeof(Tally), s);
    }
    k_mg_lists<<<sms * 8, 256, 0, s>>>(B, n, threshold, G, nl, lists, rounds ? &tally->n_long : nullptr);
    size_t sb = L.tmp_bytes;
    cub::DeviceSelect::Flagged(b + L.tmp, sb, cub::CountingInputIterator<uint32_t>(0), nl, alist,
                               n_abs, (int64_t)n, s);
    if (rounds) {
        cudaMemsetAsync(own[0], 0xff, 4 * (size_t)n, s);
        k_mg_guess<<<sms * 2, 256, 0, s>>>(alist, n_abs, nl, lists, own[0]);
    }
    bool settled = false;
    for (int r = 0; rounds && r < kRoundsMax && !settled;) {
        for (const int end = std::min(kRoundsMax, r == 0 ? 2 : r + 4); r < end; ++r) {
            uint32_t *from = own[r & 1], *to = own[(r + 1) & 1];
            k_mg_clear<<<sms * 2, 256, 0, s>>>(n, flags + r, tally, to);
            k_mg_round<<<sms * 8, 256, 0, s>>>(B, n, threshold, G, alist, n_abs, nl, lists, from, to,
                                               len, after, r < 2 ? kFirstMost : UINT32_MAX,
                                               flags + r, tally);
            k_mg_compare<<<sms * 2, 256, 0, s>>>(n, from, to, flags + r, tally, r == 1);
        }
        uint32_t last = 1;
        Tally t{};
        cudaMemcpyAsync(&last, flags + r - 1, 4, cudaMemcpyDeviceToHost, s);
        if (r == 2) cudaMemcpyAsync(&t, tally, sizeof(t), cudaMemcpyDeviceToHost, s);
        if (cudaStreamSynchronize(s) != cudaSuccess || t.n_long > kLongShare * n) break;
        settled = last == 0;
        if (!settled && (double)t.taken > kOrderedShare * n) break;
    }
    if (settled) {
        cudaMemsetAsync(count, 0, sizeof(uint32_t), s);
        k_mg_apply<<<sms * 4, 256, 0, s>>>(a, n, nl, len, own[0], after, keep, count);
    } else {  // with the grid that suits a block's search: fewer, longer lists
        const MergeGrid W = build_grid(a, n, threshold, kSmallList, kGridMax, L, b, s);
        k_merge_greedy<<<1, kMergeThreads, 0, s>>>(a.x, a.z, a.circ, a.sigma, a.u, a.w, a.uvs,
                                                   a.wvs, n, threshold, W, alist, n_abs, keep,
                                                   count);
    }
    size_t tb = L.tmp_bytes;
    cub::DeviceScan::ExclusiveSum(b + L.tmp, tb, keep, pos, (int64_t)n, s);
    const int grid = sms * 4;
    k_merge_scatter<<<grid, 256, 0, s>>>(count, n, keep, pos, a, t);
    k_merge_copyback<<<grid, 256, 0, s>>>(count, n, t, a, id, n_dev);
}

}  // namespace dvmk
