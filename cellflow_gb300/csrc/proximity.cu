// proximity.cu - proximity-graph edges on the cell list.
//
// The reference kernel (cuda-native/src/ParticleSimulation.cu:188-277) scans
// j = i+1 .. N-1 in index order, keeps same-type particles with non-periodic
// squared distance below distance^2 until it holds 2*maxConn of them
// (:215), insertion-sorts them by squared distance (:235-243, stable) and
// emits the first maxConn (:246-275) through an atomicAdd offset (:250).
//
// Here each particle scans only the cells within the distance and keeps the
// 2*maxConn smallest qualifying indices, which is the same candidate set;
// the same stable sort by squared distance then picks the same edges.  For
// the edge list, edges are placed by an exclusive scan of per-particle counts,
// so its order is deterministic: by i, then by distance.  The line vertices
// are written by the selection pass itself at places reserved by one atomic
// per particle: arbitrary order, as the reference's append.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "cf_internal.hpp"

namespace cf {
namespace {

constexpr int kThreads = 128;
constexpr int kMaxHeld = 2 * CF_MAX_PROX_CONN;

// A particle's cell along one axis, computed from its position exactly as the
// cell list's hash computed it (three multiplies instead of dividing the cell
// id back into coordinates).
__device__ __forceinline__ int axis_cell(float x, float inv, int m)
{
    const int c = __float2int_rd(__fmul_rn(x, inv));
    return min(max(c, 0), m - 1);
}

// Calls fn(u) for every sorted slot u in the cells within one cell of (cx, cy,
// cz), clipped at the box (the proximity grid is not periodic), in cell order:
// per-cell start/end arrays (zeros for empty cells).
template <typename Fn>
__device__ __forceinline__ void for_each_candidate(const uint32_t* __restrict__ cell_start,
                                                   const uint32_t* __restrict__ cell_end, const Grid& g, int cx,
                                                   int cy, int cz, Fn fn)
{
    const int mx = g.m[0], my = g.m[1], mz = g.m[2];
    for (int z = max(cz - 1, 0); z <= min(cz + 1, mz - 1); z++)
        for (int y = max(cy - 1, 0); y <= min(cy + 1, my - 1); y++)
            for (int x = max(cx - 1, 0); x <= min(cx + 1, mx - 1); x++) {
                const uint32_t cell = (uint32_t)((z * my + y) * mx + x);
                const uint32_t u_end = cell_end[cell];
                for (uint32_t u = cell_start[cell]; u < u_end; u++) fn(u);
            }
}

// The selection on per-cell start/end arrays (the allocation-free call), one thread per particle.
__global__ void __launch_bounds__(kThreads)
    proximity_select_kernel(const float4* __restrict__ pos_sorted, const uint32_t* __restrict__ vals_sorted,
                            const uint32_t* __restrict__ cell_start, const uint32_t* __restrict__ cell_end, Grid g,
                            int n, float dsq, int max_conn, int32_t* __restrict__ slots, uint32_t* __restrict__ count)
{
    const int t = blockIdx.x * kThreads + threadIdx.x;
    if (t >= n) return;
    const float4 h = pos_sorted[t];
    const uint32_t i = vals_sorted[t];
    const int mx = g.m[0], my = g.m[1], mz = g.m[2];
    const int cx = axis_cell(h.x, g.inv[0], mx);
    const int cy = axis_cell(h.y, g.inv[1], my);
    const int cz = axis_cell(h.z, g.inv[2], mz);
    const int cap = 2 * max_conn;
    if (cap <= 0) {
        count[i] = 0;
        return;
    }

    int held = 0;
    int hj[kMaxHeld];
    float hd[kMaxHeld];
    for_each_candidate(cell_start, cell_end, g, cx, cy, cz, [&](uint32_t u) {
        const float4 q = pos_sorted[u];
        if (__float_as_uint(q.w) != __float_as_uint(h.w)) return;
        const int j = (int)vals_sorted[u];
        if (j <= (int)i) return;
        if (held == cap && j >= hj[cap - 1]) return;
        const float dx = __fsub_rn(q.x, h.x);
        const float dy = __fsub_rn(q.y, h.y);
        const float dz = __fsub_rn(q.z, h.z);
        const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
        if (!(d2 < dsq)) return;
        // insert into the index-ordered set, dropping the largest when full
        int p = held < cap ? held : cap - 1;
        while (p > 0 && hj[p - 1] > j) {
            hj[p] = hj[p - 1];
            hd[p] = hd[p - 1];
            p--;
        }
        hj[p] = j;
        hd[p] = d2;
        if (held < cap) held++;
    });
    // stable insertion sort by squared distance (ParticleSimulation.cu:235-243)
    for (int a = 1; a < held; a++) {
        const float kd = hd[a];
        const int kj = hj[a];
        int b = a - 1;
        while (b >= 0 && hd[b] > kd) {
            hd[b + 1] = hd[b];
            hj[b + 1] = hj[b];
            b--;
        }
        hd[b + 1] = kd;
        hj[b + 1] = kj;
    }
    const int emit = held < max_conn ? held : max_conn;
    for (int e = 0; e < emit; e++) slots[(size_t)i * CF_MAX_PROX_CONN + e] = hj[e];
    count[i] = (uint32_t)emit;
}

// The selections on the CSR cell list: 8, 16 or 32 lanes per particle (sel_lanes).  The list is sorted by type first
// (Grid::by_type), so the particle's clipped stencil, at most nine rows of one contiguous range each,
// holds particles of its own type only: with 8 types an eighth of the candidates.  The
// ranges (one or two rows per lane, concatenated by a prefix sum) are staged as a list of
// sorted slots and the lanes test as many candidates at a time.  Crowded particles, with more in range than their lanes
// hold (16, or 32), are the whole warp's: those of one row of cells together, over the slots around them all (sel_crowd).
// Bound by instruction issue: the work per warp
// is much the same for one particle as for four.  100,000 particles, half of them in clumps (proximity
// / mesh): 49 / 99 us with all types in one list (the mesh one thread per particle), 29 / 34 by
// type with a warp per particle, 26 / 32 with half a warp, 19 / 24 with eight lanes; with four 19 / 30
// and with one 20 / 45 (crowded particles then come 8 or 32 to a warp, one after the other).  Crowded, one type, 300,000
// particles in a layer (the mesh call with 590 in range, limit 2): 7,715 us when each had a first pass over all candidates
// and one of its own in which every candidate in range joined the set; 1,008 with a thread per particle on one
// list; 561 so.
constexpr int kSelWarps = kThreads / 32;

// kLanes lanes per particle: 8, 16 or 32.
template <int kLanes>
struct Sel {
    static constexpr int kGroups = 32 / kLanes;              // particles of a warp
    static constexpr int kCap = 8 * kLanes;                  // candidates staged per particle at a time
    static constexpr int kFound = kLanes == 8 ? 16 : 32;     // in range, without the whole warp
    static constexpr int kRows = (9 + kLanes - 1) / kLanes;  // rows of a lane at most
    static constexpr int kEntries = kFound / kLanes;         // found entries of a lane
    static constexpr uint32_t kMask = kLanes == 32 ? 0xffffffffu : (1u << kLanes) - 1u;
};

template <int kLanes>
struct SelRange {
    uint32_t beg[Sel<kLanes>::kRows];  // this lane's rows (lane, lane + kLanes, ...): first sorted slot
    int len[Sel<kLanes>::kRows], pre[Sel<kLanes>::kRows];  // entries, and those of the rows before
    int total;
};

// Rows of the stencil of a particle at h, for its lanes (lane: 0 .. kLanes - 1).
template <int kLanes>
__device__ __forceinline__ SelRange<kLanes> stencil_rows(const float4& h, const uint32_t* __restrict__ cell_off,
                                                         const Grid& g, int n, int lane)
{
    constexpr int kSelRows = Sel<kLanes>::kRows;
    const int mx = g.m[0], my = g.m[1], mz = g.m[2];
    const int cx = axis_cell(h.x, g.inv[0], mx);
    const int cy = axis_cell(h.y, g.inv[1], my);
    const int cz = axis_cell(h.z, g.inv[2], mz);
    const int xlo = max(cx - 1, 0), xhi = min(cx + 1, mx - 1);
    const int ylo = max(cy - 1, 0), yhi = min(cy + 1, my - 1);
    const int zlo = max(cz - 1, 0), zhi = min(cz + 1, mz - 1);
    const int ny = yhi - ylo + 1, nrows = ny * (zhi - zlo + 1);
    // (a type outside [0, T) is reported by the hash, which counts it as type 0)
    const uint32_t type = __float_as_uint(h.w) & kTypeMask;
    const uint32_t base = (type < (uint32_t)g.worlds ? type : 0u) * (uint32_t)g.cells_w;
    SelRange<kLanes> r;
    r.total = 0;
#pragma unroll
    for (int k = 0; k < kSelRows; k++) {
        r.beg[k] = 0u;
        r.len[k] = 0;
        const int q = lane + kLanes * k;  // row
        if (q < nrows) {
            // q / ny for q < 9 and ny in {1, 2, 3} without a division: (q * 11) >> 5 = q / 3
            const int zq = ny == 3 ? (q * 11) >> 5 : (ny == 2 ? q >> 1 : q);
            const int y = ylo + (q - zq * ny), z = zlo + zq;
            const uint32_t row = base + (uint32_t)((z * my + y) * mx);
            r.beg[k] = cell_off[row + xlo];
            r.len[k] = (int)(cell_off[row + xhi + 1] - r.beg[k]);
            if (!CF_IN_BOUNDS(r.len[k], n + 1) || !CF_IN_BOUNDS(r.beg[k] + r.len[k], n + 1)) r.len[k] = 0;
        }
    }
#pragma unroll
    for (int k = 0; k < kSelRows; k++) {
        int incl = r.len[k];
#pragma unroll
        for (int o = 1; o < kLanes; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o, kLanes);
            if (lane >= o) incl += v;
        }
        r.pre[k] = r.total + incl - r.len[k];
        r.total += __shfl_sync(0xffffffffu, incl, kLanes - 1, kLanes);
    }
    return r;
}

template <int kLanes>
__device__ __forceinline__ void clear_rows(SelRange<kLanes>& r)
{
#pragma unroll
    for (int k = 0; k < Sel<kLanes>::kRows; k++) r.len[k] = 0;
    r.total = 0;
}

// Squared distance, each operation rounded on its own (ParticleSimulation.cu:211-213, :314-317).
__device__ __forceinline__ float sel_distance(const float4& q, const float4& h)
{
    const float dx = __fsub_rn(q.x, h.x), dy = __fsub_rn(q.y, h.y), dz = __fsub_rn(q.z, h.z);
    return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}

// Calls fn(ok, j, d2) for the stencil's candidates, kLanes at a time per particle, the whole warp together: j is the
// candidate's particle index, ok: it is another particle (with kAbove: of a larger index) within the
// distance.  Ends early where more() is false for every particle that has candidates left.  list: the
// particle's staging area.
template <int kLanes, bool kAbove, typename More, typename Fn>
__device__ __forceinline__ void sel_candidates(const SelRange<kLanes>& r, const float4* __restrict__ pos_sorted,
                                               const uint32_t* __restrict__ vals_sorted, const float4& h, uint32_t i,
                                               int n, float dsq, bool skip, uint32_t* list, int lane, More more, Fn fn)
{
    constexpr int kCap = Sel<kLanes>::kCap, kSelRows = Sel<kLanes>::kRows;
    const int total = skip ? 0 : r.total, most = __reduce_max_sync(0xffffffffu, total);
    for (int base = 0; base < most; base += kCap) {
        if (base > 0 && !__any_sync(0xffffffffu, base < total && more())) break;
#pragma unroll
        for (int k = 0; k < kSelRows; k++) {
            if (lane < min(kLanes, 9 - kLanes * k)) {
                const int j0 = max(0, base - r.pre[k]), j1 = skip ? 0 : min(r.len[k], base + kCap - r.pre[k]);
                for (int j = j0; j < j1; j++) list[r.pre[k] + j - base] = r.beg[k] + (uint32_t)j;
            }
        }
        __syncwarp();
        const int lim = min(kCap, total - base), most_here = min(kCap, most - base);
        for (int g0 = 0; g0 < most_here; g0 += kLanes) {
            const int gg = g0 + lane;
            bool ok = false;
            int j = 0;
            float d2 = 0.0f;
            if (gg < lim && CF_IN_BOUNDS(list[gg], n)) {
                const uint32_t u = list[gg];
                const float4 q = pos_sorted[u];
                j = (int)vals_sorted[u];
                d2 = sel_distance(q, h);
                ok = d2 < dsq && (kAbove ? j > (int)i : j != (int)i) && __float_as_uint(q.w) == __float_as_uint(h.w);
            }
            fn(ok, j, d2);
        }
        __syncwarp();
    }
}

// The crowded particles of a warp that lie in one row of cells (groups `members`, their homes in s_home, indices iq),
// by the whole warp over the rows of cells around them all, 32 slots at a time: for each the `cap` (at most 32) smallest
// qualifying indices as (j, d2) in lanes 0 .. held-1, in index order.  Once a set is full a candidate above its
// largest index is dropped, for all of them before its position is read, as most are; a qualifying one joins at its
// place, the largest falling out.
template <int kGroups>
struct Crowd {
    int held[kGroups], hj[kGroups];
    float hd[kGroups];
};

template <int kLanes, bool kAbove>
__device__ __forceinline__ void sel_crowd(const float4* __restrict__ pos_sorted, const uint32_t* __restrict__ vals_sorted,
                                          const uint32_t* __restrict__ cell_off, const Grid& g, int n, float dsq, int cap,
                                          uint32_t members, const float4* s_home, const int (&iq)[Sel<kLanes>::kGroups], int lane,
                                          Crowd<Sel<kLanes>::kGroups>& c)
{
    constexpr int kSelGroups = Sel<kLanes>::kGroups;
    const float4 first = s_home[(__ffs(members) - 1) / kLanes], last = s_home[(31 - __clz(members)) / kLanes];
    const int mx = g.m[0], my = g.m[1], mz = g.m[2];
    const int xlo = max(axis_cell(first.x, g.inv[0], mx) - 1, 0), xhi = min(axis_cell(last.x, g.inv[0], mx) + 1, mx - 1);
    const int cy = axis_cell(first.y, g.inv[1], my), cz = axis_cell(first.z, g.inv[2], mz);
    const int ylo = max(cy - 1, 0), yhi = min(cy + 1, my - 1), zlo = max(cz - 1, 0), zhi = min(cz + 1, mz - 1);
    const int ny = yhi - ylo + 1, nrows = ny * (zhi - zlo + 1);
    const uint32_t type = __float_as_uint(first.w) & kTypeMask;
    uint32_t beg = 0u;
    int len = 0;
    if (lane < nrows) {
        const int zq = ny == 3 ? (lane * 11) >> 5 : (ny == 2 ? lane >> 1 : lane);
        const uint32_t row = (type < (uint32_t)g.worlds ? type : 0u) * (uint32_t)g.cells_w +
                             (uint32_t)(((zlo + zq) * my + ylo + (lane - zq * ny)) * mx);
        beg = cell_off[row + xlo];
        len = (int)(cell_off[row + xhi + 1] - beg);
        if (!CF_IN_BOUNDS(len, n + 1) || !CF_IN_BOUNDS(beg + len, n + 1)) len = 0;
    }
    // chunks of 32 slots, those of each row apart
    int before = (len + 31) >> 5;
    const int own = before;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += v;
    }
    const int chunks = __shfl_sync(0xffffffffu, before, 15);
    before -= own;
    int worst[kSelGroups];  // above every index that the set can still take; of a full set its largest
#pragma unroll
    for (int q = 0; q < kSelGroups; q++) {
        c.held[q] = c.hj[q] = 0;
        c.hd[q] = 0.0f;
        worst[q] = cap > 0 && (members >> (kLanes * q) & 1u) ? 0x7fffffff : -1;
    }
    // chunk k's slot of this lane and its index (none: the largest int)
    const auto fetch = [&](int k, uint32_t& u) {
        const int row = 31 - __clz(__ballot_sync(0xffffffffu, own > 0 && before <= k));
        const int at = 32 * (k - __shfl_sync(0xffffffffu, before, row)) + lane;
        u = __shfl_sync(0xffffffffu, beg, row) + (uint32_t)at;
        return at < __shfl_sync(0xffffffffu, len, row) && CF_IN_BOUNDS(u, n) ? (int)vals_sorted[u] : 0x7fffffff;
    };
    uint32_t u_next = 0u;
    int j_next = chunks > 0 ? fetch(0, u_next) : 0;
    for (int k = 0; k < chunks; k++) {
        const uint32_t u = u_next;
        const int cj = j_next;
        if (k + 1 < chunks) j_next = fetch(k + 1, u_next);
        bool want = false;
#pragma unroll
        for (int q = 0; q < kSelGroups; q++) want |= cj < worst[q] && (kAbove ? cj > iq[q] : cj != iq[q]);
        if (!__any_sync(0xffffffffu, want)) continue;
        float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (want) p = pos_sorted[u];
#pragma unroll
        for (int q = 0; q < kSelGroups; q++) {
            if (worst[q] < 0) continue;
            const float4 h = s_home[q];
            const float cd = sel_distance(p, h);
            uint32_t qm = __ballot_sync(0xffffffffu, cj < worst[q] && (kAbove ? cj > iq[q] : cj != iq[q]) && cd < dsq &&
                                                        __float_as_uint(p.w) == __float_as_uint(h.w));
            if (!qm) continue;
            while (qm) {
                const int src = __ffs(qm) - 1;
                qm &= qm - 1u;
                const int j = __shfl_sync(0xffffffffu, cj, src);
                const float d2 = __shfl_sync(0xffffffffu, cd, src);
                const int pos = __popc(__ballot_sync(0xffffffffu, lane < c.held[q] && c.hj[q] < j));
                if (pos >= cap) continue;
                const int uj = __shfl_up_sync(0xffffffffu, c.hj[q], 1);
                const float ud = __shfl_up_sync(0xffffffffu, c.hd[q], 1);
                if (lane > pos && lane < cap) {
                    c.hj[q] = uj;
                    c.hd[q] = ud;
                }
                if (lane == pos) {
                    c.hj[q] = j;
                    c.hd[q] = d2;
                }
                c.held[q] = min(c.held[q] + 1, cap);
            }
            if (c.held[q] == cap) worst[q] = __shfl_sync(0xffffffffu, c.hj[q], cap - 1);
        }
    }
}

// Per particle fn(lane, lanes, i, h, held, above, entry): by its `lanes` lanes (kLanes, four particles at
// once, or the whole warp), all together: held entries qualify (all of them, or the `cap` smallest
// indices), `above` of them with an index above i; entry(e, j, rank) gives the lane's e-th entry
// (false: none) with its index and rank (kByDistance: by (distance, index), else by index).
// held < 0: not a particle of this call.
template <int kLanes, bool kAbove, bool kByDistance, typename Fn>
__device__ __forceinline__ void select_group(const float4* __restrict__ pos_sorted,
                                             const uint32_t* __restrict__ vals_sorted,
                                             const uint32_t* __restrict__ cell_off, const Grid& g, int n, float dsq, int cap,
                                             int crowd, Fn fn)
{
    constexpr int kSelGroups = Sel<kLanes>::kGroups, kSelFound = Sel<kLanes>::kFound, kSelEntries = Sel<kLanes>::kEntries;
    constexpr uint32_t kGroupMask = Sel<kLanes>::kMask;
    __shared__ uint32_t s_list[kSelWarps][kSelGroups][Sel<kLanes>::kCap];
    __shared__ float2 s_found[kSelWarps][kSelGroups][kSelFound];
    __shared__ float4 s_home[kSelWarps][kSelGroups];
    const int wl = threadIdx.x & 31, warp = threadIdx.x >> 5, group = wl / kLanes, lane = wl % kLanes;
    const int t = ((int)blockIdx.x * kSelWarps + warp) * kSelGroups + group;
    if (__all_sync(0xffffffffu, t >= n)) return;
    const bool mine = t < n;
    const float4 h = pos_sorted[mine ? t : n - 1];
    const uint32_t i = vals_sorted[mine ? t : n - 1];
    SelRange<kLanes> r = stencil_rows<kLanes>(h, cell_off, g, n, lane);
    if (!mine || !CF_IN_BOUNDS(i, n)) clear_rows(r);  // (bounds-checked build)
    float2* found = s_found[warp][group];
    int held = r.total > crowd ? kSelFound + 1 : 0;
    sel_candidates<kLanes, kAbove>(r, pos_sorted, vals_sorted, h, i, n, dsq, held > 0, s_list[warp][group], lane,
                           [&] { return held <= kSelFound; }, [&](bool ok, int j, float d2) {
        const uint32_t qm = (__ballot_sync(0xffffffffu, ok) >> (kLanes * group)) & kGroupMask;
        const int at = held + __popc(qm & ((1u << lane) - 1u));
        if (ok && at < kSelFound) found[at] = make_float2(__int_as_float(j), d2);
        held += __popc(qm);
    });
    __syncwarp();
    const uint32_t again = __ballot_sync(0xffffffffu, mine && held > kSelFound);
    if (held > kSelFound || !mine) held = 0;
    // each lane's entries (in the order in which they were found) and their ranks
    int hj[kSelEntries], rank[kSelEntries] = {};
    float hd[kSelEntries];
#pragma unroll
    for (int e = 0; e < kSelEntries; e++) {
        const float2 f = found[lane + kLanes * e];  // (past held: not used)
        hj[e] = __float_as_int(f.x);
        hd[e] = f.y;
    }
    // those of the `cap` smallest indices, by the group's found entries: all, unless there are more
    uint32_t kept = held < 32 ? (1u << held) - 1u : 0xffffffffu;
    const bool many = __any_sync(0xffffffffu, held > cap);
    if (!kByDistance || many) {
        for (int k = 0; k < held; k++) {
            const int oj = __float_as_int(found[k].x);
#pragma unroll
            for (int e = 0; e < kSelEntries; e++) rank[e] += oj < hj[e];
        }
    }
    if (many) {
#pragma unroll
        for (int e = 0; e < kSelEntries; e++) {
            const uint32_t b = __ballot_sync(0xffffffffu, rank[e] < cap) >> (kLanes * group) & kGroupMask;
            kept &= ~(kGroupMask << (kLanes * e)) | b << (kLanes * e);
            if (kByDistance) rank[e] = 0;
        }
    }
    int above = 0;
#pragma unroll
    for (int e = 0; e < kSelEntries; e++) {
        const bool up = hj[e] > (int)i && (kept >> (lane + kLanes * e) & 1u);
        above += __popc(__ballot_sync(0xffffffffu, up) >> (kLanes * group) & kGroupMask);
    }
    if (kByDistance) {
        for (uint32_t rest = kept; rest; rest &= rest - 1u) {
            const float2 o = found[__ffs(rest) - 1];
            const int oj = __float_as_int(o.x);
#pragma unroll
            for (int e = 0; e < kSelEntries; e++) rank[e] += o.y < hd[e] || (o.y == hd[e] && oj < hj[e]);
        }
    }
    __syncwarp();
    fn(lane, kLanes, i, h, mine && !(again >> wl & 1u) ? __popc(kept) : -1, above, [&](int e, int& j, int& rk) {
        j = hj[e];
        rk = rank[e];
        return (kept >> (lane + kLanes * e) & 1u) != 0u;
    });
    if (!again) return;
    // the crowded ones, those of a row of cells together
    if (lane == 0) s_home[warp][group] = h;
    __syncwarp();
    const int row = (axis_cell(h.z, g.inv[2], g.m[2]) * g.m[1] + axis_cell(h.y, g.inv[1], g.m[1])) * (int)(kTypeMask + 1u) +
                    (int)(__float_as_uint(h.w) & kTypeMask);
    int iq[kSelGroups];
#pragma unroll
    for (int q = 0; q < kSelGroups; q++) iq[q] = (int)__shfl_sync(0xffffffffu, i, kLanes * q);
    for (uint32_t rest = again; rest;) {
        const uint32_t members = __ballot_sync(0xffffffffu, row == __shfl_sync(0xffffffffu, row, __ffs(rest) - 1)) & rest;
        rest &= ~members;
        Crowd<kSelGroups> c;
        sel_crowd<kLanes, kAbove>(pos_sorted, vals_sorted, cell_off, g, n, dsq, cap, members, s_home[warp], iq, wl, c);
#pragma unroll
        for (int q = 0; q < kSelGroups; q++) {
            if (!(members >> (kLanes * q) & 1u)) continue;
            const int all = c.held[q], wj = c.hj[q];
            const float wd = c.hd[q];
            int wr = wl;
            if (kByDistance) {
                wr = 0;
                for (int k = 0; k < all; k++) {
                    const float od = __shfl_sync(0xffffffffu, wd, k);
                    const int oj = __shfl_sync(0xffffffffu, wj, k);
                    wr += (od < wd || (od == wd && oj < wj)) ? 1 : 0;
                }
            }
            const int up = __popc(__ballot_sync(0xffffffffu, wl < all && wj > iq[q]));
            fn(wl, 32, (uint32_t)iq[q], s_home[warp][q], all, up, [&](int e, int& j, int& rk) {
                j = wj;
                rk = wr;
                return e == 0 && wl < all;
            });
        }
    }
}

// The proximity graph's selection: of the 2 * maxConn smallest qualifying indices above i the maxConn
// nearest, in the stable sort's order (ParticleSimulation.cu:235-243), i.e. by (distance, index):
// each held lane counts the entries before it.
// kEmit: instead of the per-particle slots and counts, each particle's warp
// reserves its edges' places with one atomic on *count (the running total) and
// writes their line vertices itself (ParticleSimulation.cu:253-275: per edge the
// vertex of i then of j, each x, y, z, r, g, b with the colour of i's type).
template <int kLanes, bool kEmit>
__global__ void __launch_bounds__(kThreads)
    proximity_select_warp_kernel(const float4* __restrict__ pos_sorted, const uint32_t* __restrict__ vals_sorted,
                                 const uint32_t* __restrict__ cell_off, Grid g, int n, float dsq, int max_conn, int crowd,
                                 int32_t* __restrict__ slots, uint32_t* __restrict__ count,
                                 const float4* __restrict__ pos, ColorTable colors, int n_colors,
                                 float* __restrict__ vertices, int cap_vertices)
{
    select_group<kLanes, true, true>(pos_sorted, vals_sorted, cell_off, g, n, dsq, 2 * max_conn, crowd,
                             [&](int lane, int lanes, uint32_t i, const float4& h, int held, int, auto entry) {
        const int emit = min(held, max_conn);
        uint32_t base = 0u;
        if constexpr (kEmit) {
            if (lane == 0 && emit > 0) base = atomicAdd(count, (uint32_t)emit);
            base = __shfl_sync(0xffffffffu, base, 0, lanes);
        } else {
            if (lane == 0 && held >= 0 && CF_IN_BOUNDS(i, n)) count[i] = (uint32_t)emit;
        }
#pragma unroll
        for (int e = 0; e < Sel<kLanes>::kEntries; e++) {
            int j, rank;
            if (!entry(e, j, rank) || rank >= emit || !CF_IN_BOUNDS(j, n)) continue;
            if constexpr (kEmit) {
                const size_t k = (size_t)base + (size_t)rank;
                if (2 * k + 1 < (size_t)cap_vertices) {
                    // ParticleSimulation.cu:253-275: i then j, each x, y, z, r, g, b with i's colour
                    const float4 q = pos[j];
                    const uint32_t c = (__float_as_uint(h.w) & kTypeMask) % (uint32_t)n_colors;
                    const float cr = colors.c[3 * c], cg = colors.c[3 * c + 1], cb = colors.c[3 * c + 2];
                    float* v = vertices + k * 12;
                    v[0] = h.x; v[1] = h.y; v[2] = h.z; v[3] = cr; v[4] = cg; v[5] = cb;
                    v[6] = q.x; v[7] = q.y; v[8] = q.z; v[9] = cr; v[10] = cg; v[11] = cb;
                }
            } else {
                slots[(size_t)i * CF_MAX_PROX_CONN + rank] = j;
            }
        }
    });
}

__global__ void __launch_bounds__(256)
    proximity_edges_kernel(const int32_t* __restrict__ slots, const uint32_t* __restrict__ offsets, int n,
                           int32_t* __restrict__ edges, int cap)
{
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const uint32_t o = offsets[i], e_count = offsets[i + 1] - o;
    for (uint32_t e = 0; e < e_count; e++) {
        const uint32_t k = o + e;
        if (k < (uint32_t)cap) {
            edges[2 * (size_t)k] = i;
            edges[2 * (size_t)k + 1] = slots[(size_t)i * CF_MAX_PROX_CONN + e];
        }
    }
}

// ---- triangle mesh (ParticleSimulation.cu:280-424) ----------------------------
//
// The reference scans j != i in index order and keeps the first
// min(maxConn, 32) same-type particles with non-periodic squared distance
// below distance^2 * 1.2^2 (the host wrapper's hysteresis, :723-724); every
// pair of them whose indices both exceed i is a triangle (i, a, b), at most 64
// per particle, in pair order (:333-349).  Here each particle keeps the
// min(maxConn, 32) smallest qualifying indices over the cells within range
// (the same list), counts its triangles, and an exclusive scan places them:
// output in i order, then pair order.

constexpr int kMeshHeld = CF_MESH_MAX_CONN;
constexpr int kMeshMaxTriangles = 64;

// slots: the particle's list entries above it, in index order; in the last slot, where fewer than
// all slots are taken, their number, negated.
template <int kLanes>
__global__ void __launch_bounds__(kThreads)
    mesh_select_kernel(const float4* __restrict__ pos_sorted, const uint32_t* __restrict__ vals_sorted,
                       const uint32_t* __restrict__ cell_off, Grid g, int n, float dsq, int max_conn, int crowd,
                       int32_t* __restrict__ slots, uint32_t* __restrict__ count)
{
    // (distances as ParticleSimulation.cu:314-317, each operation rounded on its own in source order)
    select_group<kLanes, false, false>(pos_sorted, vals_sorted, cell_off, g, n, dsq, min(max_conn, kMeshHeld), crowd,
                               [&](int lane, int, uint32_t i, const float4&, int held, int above, auto entry) {
#pragma unroll
        for (int e = 0; e < Sel<kLanes>::kEntries; e++) {
            int j, rank;
            // the entries above i form the list's tail
            if (entry(e, j, rank) && j > (int)i) slots[(size_t)i * kMeshHeld + rank - (held - above)] = j;
        }
        if (lane == 0 && held >= 0 && CF_IN_BOUNDS(i, n)) {
            if (above < kMeshHeld) slots[(size_t)i * kMeshHeld + kMeshHeld - 1] = -above;
            count[i] = (uint32_t)min(above * (above - 1) / 2, kMeshMaxTriangles);
        }
    });
}

// Triangles in particle order, each particle's in the reference's pair order, at offsets[i]; index
// triples and / or vertices of 9 floats (position, flat normal, colour).  One block per
// kEmitParticles particles, whose triangles are consecutive: its warps take them 32 at a time, one
// per lane, vertices through shared memory so that a warp writes one contiguous stretch (27 floats
// a triangle).  Bound by the chain of reads (offsets, list, positions) and, where particles have many triangles, by
// the block with the most: 100,000 particles with 195,000 triangles took 40 us with a thread
// per particle writing its own, 30 with a warp per particle, 19.7 with a warp per 32, 12.0 so.
constexpr int kEmitWarps = 8;
constexpr int kEmitParticles = 128;

__global__ void __launch_bounds__(32 * kEmitWarps)
    mesh_emit_kernel(const int32_t* __restrict__ slots, const uint32_t* __restrict__ offsets, int n,
                     const float4* __restrict__ pos, ColorTable colors, int n_colors,
                     int32_t* __restrict__ tris, float* __restrict__ vertices, long long cap_tris)
{
    __shared__ float s_vertices[kEmitWarps][32 * 27];
    __shared__ uint32_t s_off[kEmitParticles + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i0 = (int)blockIdx.x * kEmitParticles;
    if (threadIdx.x <= kEmitParticles) s_off[threadIdx.x] = offsets[min(i0 + (int)threadIdx.x, n)];
    __syncthreads();
    const uint32_t begin = s_off[0], end = s_off[kEmitParticles];
    float* out = s_vertices[warp];
    for (uint32_t t0 = begin + 32u * warp; t0 < end; t0 += 32u * kEmitWarps) {
        const uint32_t t = min(t0 + (uint32_t)lane, end - 1u);
        // the last particle whose triangles start at or before t
        int p = 0;
#pragma unroll
        for (int step = kEmitParticles / 2; step >= 1; step >>= 1)
            if (s_off[p + step] <= t) p += step;
        // (i0 + p < n: offsets[n] = end > t)
        const int i = i0 + p;
        int rest = (int)(t - s_off[p]);
        const int32_t* list = slots + (size_t)i * kMeshHeld;
        // pair `rest` of (a, b), a < b < m, in order of a then b
        const int last = list[kMeshHeld - 1], m = last < 0 ? -last : kMeshHeld;
        int a = 0;
        while (rest >= m - 1 - a) rest -= m - 1 - a++;
        const int ja = list[a], jb = list[a + 1 + rest];
        const long long room = cap_tris - (long long)t0;
        const int here = (int)min((long long)min(32u, end - t0), max(room, 0ll));  // triangles written
        if (tris && lane < here) {
            int32_t* o = tris + 3 * (long long)t;
            o[0] = i;
            o[1] = ja;
            o[2] = jb;
        }
        if (!vertices) continue;
        const float4 v1 = pos[i], v2 = pos[ja], v3 = pos[jb];
        // ParticleSimulation.cu:365-382, each operation rounded on its own
        const float e1x = __fsub_rn(v2.x, v1.x), e1y = __fsub_rn(v2.y, v1.y), e1z = __fsub_rn(v2.z, v1.z);
        const float e2x = __fsub_rn(v3.x, v1.x), e2y = __fsub_rn(v3.y, v1.y), e2z = __fsub_rn(v3.z, v1.z);
        float nx = __fsub_rn(__fmul_rn(e1y, e2z), __fmul_rn(e1z, e2y));
        float ny = __fsub_rn(__fmul_rn(e1z, e2x), __fmul_rn(e1x, e2z));
        float nz = __fsub_rn(__fmul_rn(e1x, e2y), __fmul_rn(e1y, e2x));
        const float len = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(nx, nx), __fmul_rn(ny, ny)), __fmul_rn(nz, nz)));
        if (len > 0.0001f) {
            nx = __fdiv_rn(nx, len);
            ny = __fdiv_rn(ny, len);
            nz = __fdiv_rn(nz, len);
        }
        const uint32_t c = (__float_as_uint(v1.w) & kTypeMask) % (uint32_t)n_colors;
        const float cr = colors.c[3 * c], cg = colors.c[3 * c + 1], cb = colors.c[3 * c + 2];
        float* v = out + 27 * lane;  // (27 is odd: no two lanes on one bank)
        const float4* vs[3] = {&v1, &v2, &v3};
#pragma unroll
        for (int q = 0; q < 3; q++) {
            v[9 * q + 0] = vs[q]->x;
            v[9 * q + 1] = vs[q]->y;
            v[9 * q + 2] = vs[q]->z;
            v[9 * q + 3] = nx;
            v[9 * q + 4] = ny;
            v[9 * q + 5] = nz;
            v[9 * q + 6] = cr;
            v[9 * q + 7] = cg;
            v[9 * q + 8] = cb;
        }
        __syncwarp();
        float* to = vertices + 27 * (long long)t0;
        for (int e = lane; e < 27 * here; e += 32) to[e] = out[e];
        __syncwarp();
    }
}

// Candidates from which on a particle is taken for crowded without looking, spread evenly over its 27 cells (above: only
// those of larger index count): half as many again in range as its own lanes hold.
template <int kLanes>
int crowd_size(const Grid& g, float dsq, bool above)
{
    const double cells = 27.0 / ((double)g.inv[0] * g.inv[1] * g.inv[2]);  // their volume
    const double reach = std::min(1.0, 4.19 * std::pow((double)dsq, 1.5) / cells) * (above ? 0.5 : 1.0);
    const double size = 1.5 * Sel<kLanes>::kFound / std::max(reach, 1e-9);
    return (int)std::min(size, 1e9);
}

// Blocks of a selection.
template <int kLanes>
int sel_blocks(int n)
{
    return (n + Sel<kLanes>::kGroups * kSelWarps - 1) / (Sel<kLanes>::kGroups * kSelWarps);
}

// Lanes per particle.  Few particles leave most of the GPU idle with eight, and the edge list of a single type, whose list
// has the most candidates out of range, gains in clumps what evenly spread particles lose (device times, eight / sixteen
// lanes: one type, 100,000 particles in blobs 91 / 85 us, evenly spread 26.3 / 27.2; 20,000 of 8 types evenly spread 16.3 / 19.2,
// in blobs equal; with a warp per particle 4,000 in blobs 40.7, with sixteen lanes 43.3, with eight 47.3, host time included).
int sel_lanes(int n, const Grid& g, bool edges)
{
    if (n <= 4096) return 32;
    return n <= 10000 || (edges && g.worlds == 1) ? 16 : 8;
}

template <typename Launch>
void with_lanes(int lanes, Launch launch)
{
    if (lanes == 32)
        launch(std::integral_constant<int, 32>());
    else if (lanes == 16)
        launch(std::integral_constant<int, 16>());
    else
        launch(std::integral_constant<int, 8>());
}

}  // namespace

CF_BOUNDS_READER(proximity)

cudaError_t launch_mesh_select(const float4* pos_sorted, const uint32_t* vals_sorted, const uint32_t* cell_off,
                               const Grid& g, int n, float dsq, int max_conn, int32_t* slots, uint32_t* count,
                               cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    const auto launch = [&](auto lanes) {
        constexpr int kLanes = decltype(lanes)::value;
        mesh_select_kernel<kLanes><<<sel_blocks<kLanes>(n), kThreads, 0, st>>>(
            pos_sorted, vals_sorted, cell_off, g, n, dsq, max_conn, crowd_size<kLanes>(g, dsq, false), slots, count);
    };
    with_lanes(sel_lanes(n, g, false), launch);
    note_launches(st);
    return cudaGetLastError();
}

cudaError_t launch_mesh_emit(const int32_t* slots, const uint32_t* offsets, int n, const float4* pos,
                             const ColorTable& colors, int n_colors, int32_t* tris, float* vertices, long long cap_tris,
                             cudaStream_t st)
{
    if (n <= 0 || cap_tris <= 0) return cudaSuccess;
    mesh_emit_kernel<<<(n + kEmitParticles - 1) / kEmitParticles, 32 * kEmitWarps, 0, st>>>(slots, offsets, n, pos, colors,
                                                                                   n_colors, tris, vertices, cap_tris);
    note_launches(st);
    return cudaGetLastError();
}

cudaError_t launch_proximity_select_cells(const float4* pos_sorted, const uint32_t* vals_sorted,
                                          const uint32_t* cell_start, const uint32_t* cell_end, const Grid& g, int n,
                                          float dsq, int max_conn, int32_t* slots, uint32_t* count, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    proximity_select_kernel<<<(n + kThreads - 1) / kThreads, kThreads, 0, st>>>(pos_sorted, vals_sorted, cell_start,
                                                                               cell_end, g, n, dsq, max_conn, slots, count);
    note_launches(st);
    return cudaGetLastError();
}

namespace {
template <bool kEmit>
cudaError_t launch_proximity_warps(const float4* pos_sorted, const uint32_t* vals_sorted, const uint32_t* cell_off,
                                   const Grid& g, int n, float dsq, int max_conn, int32_t* slots, uint32_t* count,
                                   const float4* pos, const ColorTable& colors, int n_colors, float* vertices,
                                   int cap_vertices, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    const auto launch = [&](auto lanes) {
        constexpr int kLanes = decltype(lanes)::value;
        proximity_select_warp_kernel<kLanes, kEmit><<<sel_blocks<kLanes>(n), kThreads, 0, st>>>(
            pos_sorted, vals_sorted, cell_off, g, n, dsq, max_conn, crowd_size<kLanes>(g, dsq, true), slots, count, pos,
            colors, n_colors, vertices, cap_vertices);
    };
    with_lanes(sel_lanes(n, g, true), launch);
    note_launches(st);
    return cudaGetLastError();
}
}  // namespace

cudaError_t launch_proximity_select(const float4* pos_sorted, const uint32_t* vals_sorted, const uint32_t* cell_off,
                                    const Grid& g, int n, float dsq, int max_conn, int32_t* slots, uint32_t* count,
                                    cudaStream_t st)
{
    return launch_proximity_warps<false>(pos_sorted, vals_sorted, cell_off, g, n, dsq, max_conn, slots, count, nullptr,
                                         ColorTable{}, 1, nullptr, 0, st);
}

cudaError_t launch_proximity_select_vertices(const float4* pos_sorted, const uint32_t* vals_sorted,
                                             const uint32_t* cell_off, const Grid& g, int n, float dsq, int max_conn,
                                             const float4* pos, const ColorTable& colors, int n_colors,
                                             float* vertices, int cap_vertices, uint32_t* total, cudaStream_t st)
{
    return launch_proximity_warps<true>(pos_sorted, vals_sorted, cell_off, g, n, dsq, max_conn, nullptr, total, pos, colors,
                                        n_colors, vertices, cap_vertices, st);
}

cudaError_t launch_proximity_emit_edges(const int32_t* slots, const uint32_t* offsets, int n, int max_conn,
                                        int32_t* edges, int cap, cudaStream_t st)
{
    (void)max_conn;
    if (n <= 0 || cap <= 0) return cudaSuccess;
    proximity_edges_kernel<<<(n + 255) / 256, 256, 0, st>>>(slots, offsets, n, edges, cap);
    note_launches(st);
    return cudaGetLastError();
}


}  // namespace cf
