// step.cu - pairwise smooth force, neighbour density and friction integrator.
//
// Work decomposition.  Particles are in cell order (the sorted snapshot of
// positions).  An item is up to 32 consecutive particles of one row of cells
// (same y and z cell), one home particle per lane.  The candidates of an item
// are the particles of the union of its homes' 27-cell stencils: 9 rows, each
// a run of consecutive cells, i.e. one contiguous range of the sorted snapshot
// (up to three where the run wraps around the box in x), read as one concatenated
// list.  The list is cut into units of at most kUnit candidates.  A warp works
// one unit at a time: it stages the unit into shared memory with its periodic
// shift applied, filters it for all 32 homes and drains the hits.  An item has
// 1, 2, 4, 8 or 16 warps (c.split), which take its units in turn.
//
// Every unit's partial sums start from zero and are added in unit order, so a
// step's result depends on neither the split nor the occupancy variant, bit
// for bit, and a world steps the same alone and in a batch.
//
// Coordinates are staged relative to an origin per item (the centre of the
// stencil box where that keeps c - o exact, else 0 or, in x, the box's right end), periodic shift folded in;
// an unshifted displacement is then the reference's fl(c - h) bit for bit, and one across the box's face is rounded
// at the scale of a few cells at most.
//
// Per unit, two phases:
//   Filter: |c - h|^2 - B = |c|^2 + (|h|^2 - B) - 2 h.c for 32 homes x 8
//     candidates by two m16n8k8 tensor-core products of half-precision
//     operands with 32-bit sums; the sign bits, gathered over the quad of
//     lanes that holds a home's row, give 32-bit masks per home.  Positions
//     are rounded to half precision first and the squares are taken of the
//     rounded positions (as high + low halves), so the value is the rounded
//     points' own squared distance and B only has to cover the rounding of the
//     positions.  The scalar form (four packed FP32 instructions per pair of
//     candidates) cost 4 issue slots a candidate; this costs about 1.7.
//   Drain: each lane walks its home's set bits (three pairs per trip; a
//     warp-uniform trip count, the largest hit count): the contracted distance
//     of the 32-bit displacement; pairs below a second bound (<= the exact
//     test for every pair) interact for certain, pairs above a third do not,
//     and only the rare pairs between (a band ~1e-6 wide) take the
//     reference's exact test on the unshifted coordinates, in the trips where
//     a warp vote finds one.  Interacting pairs add their force term.
//
// Exactness (cuda-native/src/ParticleSimulation.cu:86-165):
//   - the neighbour test is the reference's: d^2 = (dx*dx + dy*dy) + dz*dz and
//     s = d^2 + 1e-4 rounded as the reference (compiled without contraction)
//     rounds them, and sqrtf(s) < eff is replaced by the equivalent s < t,
//     t the smallest float whose correctly rounded square root is >= eff.
//     The bounds bracket that test, so neighbour counts match bit for bit;
//   - a displacement is wrapped like the reference (subtract the extent where
//     its test fires).  With at least 5 cells per axis that is exactly the
//     stencil cells across the box edge: every staged range has one shift for every lane,
//     added after the subtraction (exact path) as the reference does; an item that reaches over the
//     box in x has its last two cells' candidates twice, one period apart, and at most
//     one of the two is within reach of a home.  With
//     fewer cells both phases run the reference's tests per candidate;
//   - force terms use rsqrt and exp approximations (a few ulp) and the
//     contracted distance.
//   The density factor, integrator and wrap are the reference's operations.
//
// What bounds it: instruction issue (42 to 62 % of the slots used) and, in the
// drain, latency and shared-memory bank conflicts at scattered slots.  Counted with two pairs
// a trip and half-precision sums in the filter, at 100k evenly spread particles (3,340 items of 18 groups and 28 trips):
// about 820 instructions for an item's start and end, 97 to stage and 67 to filter a
// group of 32 candidates, 90 per trip.  Three pairs a trip since (532 to 521 us for the step at 1M in
// blobs, 318 to 315 at 64 worlds of 20,000), and the filter's sums in 32 bits (21.1 to 22.3 million warp instructions
// at 100k, 63.4 to 64.2 us; 519 to 535 at 1M, 318 to 326 at the worlds).  What brought the step there,
// against one 32-bit lane per home filtering and draining stretches of the list
// (force kernel, 100k and 1M in blobs): units dealt out entry by entry instead
// of in stretches (28 trips per item instead of 37), band pairs put off to the end
// of the unit instead of an exact test in the trip (61 instructions per trip),
// predicated bit walking, all of a unit's positions in flight at once, the
// tensor-core filter: 62 to 39 us and 737 to 469 us.  One list for an item that reaches over the box
// in x, end cells twice, instead of a second pass for its last cells (and the loop and
// registers that took): 264 to 240 us for 64 worlds of 20,000, 469 to 459 at 1M.  An application
// world of 10,000 particles with ~125 neighbours each (313 items): 276 to 32 us with
// four warps per item, set by the SMs that get a third item.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "cf_internal.hpp"

namespace cf {
namespace {

constexpr int kUnit = 256;          // candidates staged per unit at most
constexpr int kGroups = kUnit / 32; // of 32 candidates
constexpr float kFar = 1e30f;       // the sentinel slot's position, and idle homes' on generic grids (-kFar)
constexpr uint32_t kAll = 0xffffffffu;

__device__ __forceinline__ float wrap_ref(float d, float ext, float half)
{
    // ParticleSimulation.cu:97-102
    if (d > half) d = __fsub_rn(d, ext);
    if (d < -half) d = __fadd_rn(d, ext);
    return d;
}

// Shift code per axis: 0 none, 1 subtract the extent, 2 add it.
__device__ __forceinline__ float code_shift(uint32_t code, float ext)
{
    return code == 1u ? -ext : (code == 2u ? ext : 0.0f);
}

// The shift that was added to a raw coordinate to give its staged value.
__device__ __forceinline__ float staged_shift(float staged, float raw, float ext)
{
    const float d = staged - raw;
    return d > 0.5f * ext ? ext : (d < -0.5f * ext ? -ext : 0.0f);
}

__device__ __forceinline__ int wrap_index(int v, int m) { return v < 0 ? v + m : (v >= m ? v - m : v); }

// A home's x cell, as the cell list's hash computed it.
__device__ __forceinline__ int x_cell(float x, float inv, int m)
{
    const int c = __float2int_rd(__fmul_rn(x, inv));
    return min(max(c, 0), m - 1);
}

// The first of the sorted slots [b, e) of a row of cells whose x cell is at least x (e: none).
__device__ __forceinline__ int first_at_cell(const float4* __restrict__ pos_sorted, int b, int e, int x, float inv, int m)
{
    while (b < e) {
        const int mid = (b + e) >> 1;
        if (x_cell(pos_sorted[mid].x, inv, m) < x)
            b = mid + 1;
        else
            e = mid;
    }
    return b;
}

// fmodf(x, W) of the integrator's wrap (ParticleSimulation.cu:159-161), exact:
// for x in [0, 2W) it is x or x - W, and x - W is exact there (Sterbenz).
__device__ __forceinline__ float wrap_pos(float x, float W)
{
    if (x >= 0.0f && x < 2.0f * W) return x >= W ? __fsub_rn(x, W) : x;
    return fmodf(x, W);
}

// Staging origin on one axis for stencil cells [clo, chi] (shifted cell
// coordinates, cell size cs) and the radius r of the box around it.  The
// centre is used only where it is at least twice the half-width: then every
// raw coordinate c in the box satisfies o/2 <= c <= 2o, so c - o is exact
// (Sterbenz) and an unshifted displacement (c - o) - (h - o) rounds to the
// reference's fl(c - h).  Otherwise the origin is 0 (also exact).
__device__ __forceinline__ void stencil_origin(int clo, int chi, float cs, float& o, float& r)
{
    // (rounded one by one: contracted here and not there, homes and candidates would get two origins)
    const float lo = __fmul_rn((float)clo, cs), hi = __fmul_rn((float)(chi + 1), cs), mg = 0.05f * cs;
    const float ctr = __fmul_rn(0.5f, __fadd_rn(lo, hi)), half = 0.5f * (hi - lo) + mg;
    if (ctr >= 2.0f * half) {
        o = ctr;
        r = half;
    } else {
        o = 0.0f;
        r = fmaxf(fabsf(lo), fabsf(hi)) + mg;
    }
}

// The origin in x and the radius of the box around it for an item of cells [x0, x1], and whether its list is folded.  A
// candidate past the box's right end, staged as x plus the extent less the centre, would be rounded at the scale
// of the item, the whole box in the end; items of a few cells leave it at that.  Others that lie in the right half take
// the right end as their origin: what lies past it keeps its own x, and the rest is exact.  Else the item's homes of the last
// cell are taken one period to the left, with the row's last two cells there too (both exact in the upper half of the
// box) and the first cell as it is, all from the origin 0.  (Choosing between two homes per pair instead took
// 64 worlds of 20,000 from 314 to 348 us and 1M in blobs from 520 to 549; this 318 and 519.)
__device__ __forceinline__ bool stencil_origin_x(int x0, int x1, int mx, float cs, float ext, float& o, float& r)
{
    stencil_origin(x0 - 1, x1 + 1, cs, o, r);
    if (x1 != mx - 1 || (o != 0.0f && x1 - x0 < 4)) return false;
    if (o != 0.0f && 2 * (x0 - 1) > mx) {
        o = ext;
        r = cs * ((float)(mx - x0) + 1.05f);
        return false;
    }
    o = 0.0f;
    r = cs * ((float)mx + 0.05f);
    return true;
}

constexpr int kSegs = 27;  // contiguous ranges of an item's candidates: 9 rows, up to three where a row wraps

// Per-warp staging area.
struct WarpSmem {
    float4 c[1 + kUnit];  // the sentinel (at kFar), then the staged x, y, z and force-table offset (4 type)
    // row 0: the sentinel's masks, then the list's description (below).  Row 1 + g of
    // group g: the filter's half-precision words (x, y), (z, s hi), (s lo, 1), with s = |c|^2, in
    // fragment order, and once the group is filtered, in the first 32 words, the lanes' masks.
    uint32_t row[1 + kGroups][96];
    float4 seg[kSegs];  // per segment: what is added to its positions, and its first sorted index less its list start
    // for each segment with entries in the unit, what gives the sorted index of slot s as x + s * units, and
    // the segment (one more: 16-byte multiples)
    int2 part[kSegs + 1];
};
// Words of row 0: the staging origin; where the segments start in the list.
constexpr int kOriginAt = 32, kStartAt = 36;

// Named barrier of the warps sharing an item: id 1 + slot (at most 4 items per
// block), immediate ids so only five hardware barriers are reserved.
__device__ __forceinline__ void item_barrier(int slot, int threads)
{
    switch (slot) {
    case 0: asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); break;
    case 1: asm volatile("bar.sync 2, %0;" ::"r"(threads) : "memory"); break;
    case 2: asm volatile("bar.sync 3, %0;" ::"r"(threads) : "memory"); break;
    default: asm volatile("bar.sync 4, %0;" ::"r"(threads) : "memory"); break;
    }
}

// Two m16n8k8 products with 32-bit sums (with half-precision accumulators, 237 instead of 244 us a step for 64 worlds of
// 20,000 and 491 instead of 510 for 1M, the instruction promises no more than half precision, 2^-11 of terms
// several times the reach, and the bound below would not hold): 32 homes (fragments a[0..1] rows g and g + 8, a[2..3]
// rows g + 16 and g + 24) against the 8 candidates of one fragment word b.
// d[2 q + j]: row g + 8 q against column 2 t + j.
__device__ __forceinline__ void mma_32x8(const uint32_t (&a)[4], uint32_t b, uint32_t (&d)[8])
{
    asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(b), "f"(0.0f));
    asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
        : "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7])
        : "r"(a[2]), "r"(a[3]), "r"(b), "f"(0.0f));
}

// Quotient and remainder of x by units, x at most kUnit * units (so that the
// rounded quotient is off by one at most).
__device__ __forceinline__ void deal(int x, int units, float per_unit, int& q, int& r)
{
    q = (int)((float)x * per_unit);
    r = x - q * units;
    if (r < 0) {
        q--;
        r += units;
    }
    if (r >= units) {
        q++;
        r -= units;
    }
}

// a where the mask has a bit, b elsewhere.
__device__ __forceinline__ uint32_t bit_select(uint32_t a, uint32_t b, uint32_t mask) { return (a & mask) | (b & ~mask); }

// Two floats rounded to half precision, lo in the low half.
__device__ __forceinline__ uint32_t half2_bits(float lo, float hi)
{
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float half_lo(uint32_t h) { return __low2float(*reinterpret_cast<const __half2*>(&h)); }
__device__ __forceinline__ float half_hi(uint32_t h) { return __high2float(*reinterpret_cast<const __half2*>(&h)); }

// Square root to about 2^-22 (the filter's bound has 2^-16 to spare).
__device__ __forceinline__ float sqrt_approx(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ int top_bit(uint32_t m)
{
    int r;
    asm("bfind.u32 %0, %1;" : "=r"(r) : "r"(m));
    return r;
}

// A value the compiler keeps in a register instead of computing it again from
// the thread index at each use.
__device__ __forceinline__ uint32_t pinned(uint32_t x)
{
    asm volatile("" : "+r"(x));
    return x;
}

// Loads by shared-memory address.
__device__ __forceinline__ float4 lds128(uint32_t at)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at));
    return v;
}
__device__ __forceinline__ float lds32(uint32_t at)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at));
    return v;
}

// 16 bytes from global to shared memory, asynchronously, if `copy`.
__device__ __forceinline__ void copy_async16(bool copy, uint32_t to, const float4* from)
{
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.u32 p, %2, 0;\n\t"
                 "@p cp.async.ca.shared.global [%0], [%1], 16;\n\t}" ::"r"(to), "l"(from), "r"((uint32_t)copy)
                 : "memory");
}
__device__ __forceinline__ void copy_async_wait()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// The reference's exact test for a pair the two bounds left open (within
// rounding of the threshold), on the unshifted coordinates h and o; p is the
// staged candidate.
template <bool kGeneric>
__device__ __forceinline__ bool pair_exact(const StepConsts& c, const float4& h, bool home_left, const float* origin,
                                           const float4& p, const float4& o, float thr)
{
    float ex = __fsub_rn(o.x, h.x), ey = __fsub_rn(o.y, h.y), ez = __fsub_rn(o.z, h.z);
    if (kGeneric) {
        ex = wrap_ref(ex, c.ext[0], c.half[0]);
        ey = wrap_ref(ey, c.ext[1], c.half[1]);
        ez = wrap_ref(ez, c.ext[2], c.half[2]);
    } else {
        ex = __fadd_rn(ex, staged_shift(p.x + origin[0], o.x, c.ext[0]) + (home_left ? c.ext[0] : 0.0f));
        ey = __fadd_rn(ey, staged_shift(p.y + origin[1], o.y, c.ext[1]));
        ez = __fadd_rn(ez, staged_shift(p.z + origin[2], o.z, c.ext[2]));
    }
    const float e2 = __fadd_rn(__fadd_rn(__fmul_rn(ex, ex), __fmul_rn(ey, ey)), __fmul_rn(ez, ez));
    return __fadd_rn(e2, 0.0001f) < thr;
}

// A home's displacement to a staged candidate p, its contracted square, the
// bound below which it interacts for certain, and the weight of the displacement
// in the force: with s = d^2 + 1e-4, dist = sqrt(s) and rs = 1/dist, the
// reference's term (d / dist) F (R exp(-k r^2) - A r), r = dist / eff
// (ParticleSimulation.cu:113-124) is d * F * (R exp2(c1 s) rs - A / eff),
// c1 = -k log2(e) / eff^2.
struct PairTerm {
    float dx, dy, dz, d2, lo, weight;
};

template <bool kGeneric, bool kUniformR>
__device__ __forceinline__ PairTerm pair_term(const StepConsts& c, const float4& p, float hx, float hy, float hz,
                                              uint32_t force_at, uint32_t pair_at)
{
    PairTerm k;
    const uint32_t type4 = __float_as_uint(p.w);
    const float F = lds32(force_at + type4);
    float a_eff = c.att_uniform, c1 = c.c1_uniform;
    k.lo = c.thr_lo_uniform;
    if (!kUniformR) {
        const float4 v = lds128(pair_at + 4 * type4);
        a_eff = v.x;
        c1 = v.y;
        k.lo = v.z;
    }
    k.dx = p.x - hx;
    k.dy = p.y - hy;
    k.dz = p.z - hz;
    if (kGeneric) {
        k.dx = wrap_ref(k.dx, c.ext[0], c.half[0]);
        k.dy = wrap_ref(k.dy, c.ext[1], c.half[1]);
        k.dz = wrap_ref(k.dz, c.ext[2], c.half[2]);
    }
    k.d2 = fmaf(k.dz, k.dz, fmaf(k.dy, k.dy, k.dx * k.dx));
    const float s = k.d2 + 0.0001f;
    float rs, e;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(rs) : "f"(s));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(c1 * s));
    k.weight = F * fmaf(c.repulsion * e, rs, -a_eff);
    return k;
}

// Density-adaptive scale, integrator and wrap of particle i at h with force sum
// f and n neighbours (ParticleSimulation.cu:136-165); vel_in and counts_in: the state before the step,
// in place vel and counts.
__device__ __forceinline__ void integrate(const StepConsts& c, const float4& h, const float4& f, int n, uint32_t i,
                                          const float4* vel_in, const int* counts_in, float4* __restrict__ pos,
                                          float4* __restrict__ vel, float4* __restrict__ acc, int* __restrict__ counts)
{
    const float avg = __fmul_rn((float)(n + counts_in[i]), 0.5f);
    const float density = fminf(__fdiv_rn(avg, (float)c.max_expected_neighbors), 1.0f);
    const float adapt = __fsub_rn(1.0f, __fmul_rn(__fsub_rn(1.0f, c.balance), density));
    const float strength = __fmul_rn(c.force_multiplier, adapt);
    const float fx = __fmul_rn(f.x, strength);
    const float fy = __fmul_rn(f.y, strength);
    const float fz = __fmul_rn(f.z, strength);
    const float4 v = vel_in[i];
    const float vx = __fadd_rn(__fmul_rn(v.x, c.friction), __fmul_rn(fx, c.delta_t));
    const float vy = __fadd_rn(__fmul_rn(v.y, c.friction), __fmul_rn(fy, c.delta_t));
    const float vz = __fadd_rn(__fmul_rn(v.z, c.friction), __fmul_rn(fz, c.delta_t));
    float px = __fadd_rn(h.x, __fmul_rn(vx, c.delta_t));
    float py = __fadd_rn(h.y, __fmul_rn(vy, c.delta_t));
    float pz = __fadd_rn(h.z, __fmul_rn(vz, c.delta_t));
    px = wrap_pos(__fadd_rn(px, c.ext[0]), c.ext[0]);
    py = wrap_pos(__fadd_rn(py, c.ext[1]), c.ext[1]);
    pz = wrap_pos(__fadd_rn(pz, c.ext[2]), c.ext[2]);
    pos[i] = make_float4(px, py, pz, h.w);
    vel[i] = make_float4(vx, vy, vz, 0.0f);
    acc[i] = make_float4(fx, fy, fz, 0.0f);
    counts[i] = n;
}

// kBlockWarps warps per block, kMinBlocks resident blocks the register budget
// is sized for.  Shared memory: the warps' staging, the force tables (one for a
// plain world, one per item of the block in a batch) and, without a uniform
// radius, (A / eff, c1, certain-interaction bound) per type pair.  Forms of their own are kBins, with the
// offsets per bin of cells (the search for a segment's ends in the same form cost the others 3 % at
// 64 worlds of 20,000), and kApart, from one state to another (state arrays that may
// be the same cost the step in place 1.4 % at 100,000 particles).
enum StepForm { kInPlace, kBins, kApart };

template <int kBlockWarps, int kMinBlocks, bool kGeneric, bool kUniformR, StepForm kForm>
__global__ void __launch_bounds__(32 * kBlockWarps, kMinBlocks)
    step_force_kernel(StepConsts c, const PairTables* __restrict__ tables, const float4* __restrict__ pos_sorted,
                      const uint32_t* __restrict__ vals_sorted, const uint32_t* __restrict__ cell_off,
                      const Item* __restrict__ items, const int* __restrict__ n_items, int max_items,
                      float4* __restrict__ pos, float4* __restrict__ vel, float4* __restrict__ acc,
                      int* __restrict__ counts, const float4* __restrict__ vel_in, const int* __restrict__ counts_in)
{
    // pairs per drain trip (two: 459 for 446 us at 1M in blobs; four and more gain nothing with fewer warps)
    constexpr int kPer = 3;
    extern __shared__ __align__(16) unsigned char s_dyn[];
    const int T = c.num_types, TT = T * T;
    const bool one_world = c.grid.worlds == 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    WarpSmem& w = reinterpret_cast<WarpSmem*>(s_dyn)[warp];
    float4* s_pair = reinterpret_cast<float4*>(s_dyn + sizeof(WarpSmem) * kBlockWarps);
    float* s_force = reinterpret_cast<float*>(s_pair + (kUniformR ? 0 : TT));

    // the item and its count are read together (the array holds max_items entries)
    const int split = c.split;
    const int part = warp & (split - 1);
    const int slot_of_item = warp / split;
    const int item = blockIdx.x * (kBlockWarps / split) + slot_of_item;
    Item it{0, 0, 0, 0};
    if (item < max_items) it = items[item];
    if (item >= *n_items) it.count = 0;
    if (!kUniformR) {
        for (int e = threadIdx.x; e < TT; e += 32 * kBlockWarps) {
            const float2 v = tables->pair_compact[e];  // 1 / eff, certain-interaction bound
            s_pair[e] = make_float4(c.attraction * v.x, c.neg_k_log2e * v.x * v.x, v.y, 0.0f);
        }
    }
    if (one_world) {
        for (int e = threadIdx.x; e < TT; e += 32 * kBlockWarps) s_force[e] = c.world_force[e];
    }
    if (one_world || !kUniformR) __syncthreads();
    if (it.count == 0) return;  // the item's other warps leave too: no barrier is pending
    // (bounds-checked build) the item's particles lie in [0, n): else the item's warps skip it
    if (!CF_IN_BOUNDS(it.count - 1, 32) || !CF_IN_BOUNDS(it.first, c.n) || !CF_IN_BOUNDS(it.first + it.count - 1, c.n))
        return;
    if (!one_world) {
        // each of the item's warps writes all of the item's table (the same values)
        s_force += slot_of_item * TT;
        const float* f = c.world_force + (size_t)it.world * TT;
        for (int e = lane; e < TT; e += 32) s_force[e] = f[e];
    }
    // lane 4 g + t holds home g + 8 t: the row whose mask the filter's quad of lanes leaves in it
    const int home = (lane >> 2) + 8 * (lane & 3);
    const bool active = home < it.count;
    const int t = it.first + (active ? home : 0);
    const float4 h = pos_sorted[t];
    const uint32_t i = vals_sorted[t];
    // a type outside [0, T) is reported by the cell list's hash; it stays inside the tables here
    const uint32_t type = min(__float_as_uint(h.w) & kTypeMask, (uint32_t)(T - 1));
    const int mx = c.grid.m[0], my = c.grid.m[1], mz = c.grid.m[2];
    const int yc = it.yz & 0xffff, zc = it.yz >> 16;
    const int hx = x_cell(h.x, c.grid.inv[0], mx);
    const int last = it.count - 1;
    const int x0 = __shfl_sync(kAll, hx, 0);
    const int x1 = __shfl_sync(kAll, hx, ((last & 7) << 2) | (last >> 3));
    if (lane == 0) w.c[0] = make_float4(kFar, kFar, kFar, 0.0f);
    w.row[0][lane] = 0x80000000u;
    // no pair of this home's type interacts at or above thr_f (a contracted squared distance)
    const float thr_f = kUniformR ? c.thr_filter : tables->filter_row[type];
    const uint32_t force_at = pinned((uint32_t)__cvta_generic_to_shared(s_force + type * T));
    const uint32_t pair_at = pinned((uint32_t)__cvta_generic_to_shared(s_pair + type * T));
    // slot b of row r: + (32 r + b) 16
    const uint32_t slots_at = pinned((uint32_t)__cvta_generic_to_shared(&w.c[0]) - 31 * 16);
    const uint32_t masks_at = pinned((uint32_t)__cvta_generic_to_shared(&w.row[0][lane]));

    // the item's sums so far, in part 0 (units are added in order)
    float sum_x = 0.0f, sum_y = 0.0f, sum_z = 0.0f;
    int sum_n = 0;

    // the stencil's x cells: the item's and one each side (on generic grids every cell once), or as stencil_origin_x
    // folds them
    const bool ring = kGeneric && x1 - x0 + 3 >= mx;
    const int xlo = ring ? 0 : x0 - 1;
    const int xhi = ring ? mx - 1 : x1 + 1;  // inclusive
    float ox = 0.0f, rx = 0.0f;
    const bool folded = !kGeneric && stencil_origin_x(x0, x1, mx, c.cell[0], c.ext[0], ox, rx);
    const bool home_left = folded && hx == mx - 1;  // (taken one period to the left)
    const float home_x = home_left ? h.x - c.ext[0] : h.x;

    // segments: lane row + 9 part describes one contiguous range of the snapshot and
    // its periodic shift less the origin (zero on generic grids)
    const int ny = !kGeneric || my > 1 ? 3 : 1, nz = !kGeneric || mz > 1 ? 3 : 1;
    int seg_beg = 0, seg_len = 0;
    uint32_t shift = 0u;
    {
        const uint32_t cx = lane >= 18 ? 2u : (lane >= 9 ? 1u : 0u);
        const int row = lane - 9 * (int)cx;
        const int dz = ny == 3 ? (row * 11) >> 5 : row;  // row / ny (row < 16)
        const int yy = yc + (row - dz * ny) - (ny > 1 ? 1 : 0), zz = zc + dz - (nz > 1 ? 1 : 0);
        const uint32_t cy = yy < 0 ? 1u : (yy >= my ? 2u : 0u);
        const uint32_t cz = zz < 0 ? 1u : (zz >= mz ? 2u : 0u);
        // [xlo, xhi] in the box, left of it and right of it; folded, the last two cells left of it, and the
        // first one in the box if it is not there yet
        int xa = cx == 0u ? max(xlo, 0) : (cx == 1u ? xlo + mx : 0);
        int xb = cx == 0u ? min(xhi, mx - 1) : (cx == 1u ? (xlo < 0 ? mx - 1 : -1) : xhi - mx);
        if (folded) {
            if (cx == 1u) {
                xa = mx - 2;
                xb = mx - 1;
            } else if (cx == 2u) {
                xb = xlo > 0 ? 0 : -1;
            }
        }
        const uint32_t base = (uint32_t)it.world * (uint32_t)c.grid.cells_w +
                              (uint32_t)((wrap_index(zz, mz) * my + wrap_index(yy, my)) * mx);
        if (row < ny * nz && xb >= xa && CF_IN_BOUNDS(base + xb + 1, c.grid.cells + 1)) {
            if (kForm == kBins) {
                // the bins of cells xa..xb, less the particles of their other cells
                const uint32_t bins = base / (uint32_t)mx * (uint32_t)row_bins(c.grid);
                const int first = (int)cell_off[bins + (xa >> c.grid.bin_shift)],
                          last = (int)cell_off[bins + (xb >> c.grid.bin_shift) + 1];
                if (CF_IN_BOUNDS(first, c.n + 1) && CF_IN_BOUNDS(last, c.n + 1)) {
                    seg_beg = first_at_cell(pos_sorted, first, last, xa, c.grid.inv[0], mx);
                    seg_len = first_at_cell(pos_sorted, seg_beg, last, xb + 1, c.grid.inv[0], mx) - seg_beg;
                }
            } else {
                seg_beg = (int)cell_off[base + xa];
                seg_len = (int)cell_off[base + xb + 1] - seg_beg;
            }
            if (!CF_IN_BOUNDS(seg_len, c.n + 1) || !CF_IN_BOUNDS(seg_beg + seg_len, c.n + 1)) seg_len = 0;
        }
        shift = (folded && cx == 2u ? 0u : cx) | cy << 2 | cz << 4;
    }

    // Staging origin per axis (stencil_origin) for the stencil box (cells xlo..xhi,
    // yc-1..yc+1, zc-1..zc+1 in shifted coordinates): every staged candidate and the homes
    // lie within (rx, ry, rz) of it.  The filter works on them scaled by a power of two
    // that puts the box's radius in [64, 128) (squares stay below 65504) and rounded to
    // half precision: at most 2^-11 of the coordinate each, or 2^-25 where it is tiny, and
    // 2^-23 of the box for the contracted scaling, so two points' distance moves by at
    // most the norm of (2^-10 r + 2^-22 box) over the axes.
    // The sums (products exact in 32 bits; |c|^2 and |h|^2 - B as two halves, 2^-22 each;
    // eight terms of at most 4 R^2 together) are off by less than 2^-16 R^2.
    float oy = 0.0f, oz = 0.0f, scale = 1.0f;
    uint32_t a[4];
    if (!kGeneric) {
        float ry, rz;
        stencil_origin(yc - 1, yc + 1, c.cell[1], oy, ry);
        stencil_origin(zc - 1, zc + 1, c.cell[2], oz, rz);
        const int e = (int)(__float_as_uint(fmaxf(rx, fmaxf(ry, rz))) >> 23);
        scale = __uint_as_float((uint32_t)min(max(260 - e, 1), 254) << 23);
        rx *= scale;
        ry *= scale;
        rz *= scale;
        const float r2 = fmaf(rz, rz, fmaf(ry, ry, rx * rx));
        const float ex = fmaf(rx, 0x1p-10f, c.ext[0] * scale * 0x1p-22f),
                    ey = fmaf(ry, 0x1p-10f, c.ext[1] * scale * 0x1p-22f),
                    ez = fmaf(rz, 0x1p-10f, c.ext[2] * scale * 0x1p-22f);
        const float reach = sqrt_approx(fmaxf(thr_f, 0.0f)) * scale + sqrt_approx(fmaf(ez, ez, fmaf(ey, ey, ex * ex)));
        const float bnd = fmaf(reach * reach, 1.0f + 0x1p-16f, r2 * 0x1p-16f);
        const uint32_t xy = half2_bits((home_x - ox) * scale, (h.y - oy) * scale);
        const float qx = half_lo(xy), qy = half_hi(xy), qz = half_lo(half2_bits((h.z - oz) * scale, 0.0f));
        const float k = fmaf(qz, qz, fmaf(qy, qy, qx * qx)) - bnd;
        const float khi = half_lo(half2_bits(k, 0.0f));
        // the home's row of the A operand, k = 0..7: -2 h (3), 1, 1, k hi, 0, k lo (a home that
        // tests nothing: 60000 beside any |c|^2); fragment word t of the four
        // rows that this lane's quad holds, exchanged through shared memory
        __syncwarp();
        *reinterpret_cast<uint4*>(&w.row[1][0] + lane * 4) =
            active && thr_f > 0.0f ? make_uint4(half2_bits(-2.0f * qx, -2.0f * qy), half2_bits(-2.0f * qz, 1.0f),
                                              half2_bits(1.0f, khi), half2_bits(0.0f, k - khi))
                                 : make_uint4(0u, 0x3c000000u, half2_bits(1.0f, 60000.0f), 0u);
        __syncwarp();
        const uint32_t* quad = &w.row[1][0] + (lane & ~3) * 4 + (lane & 3);
#pragma unroll
        for (int q = 0; q < 4; q++) a[q] = quad[4 * q];
    }
    int seg_pre = seg_len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(kAll, seg_pre, o);
        if (lane >= o) seg_pre += v;
    }
    const int total = __shfl_sync(kAll, seg_pre, 31);
    seg_pre -= seg_len;
    // the home's place in the list: its cell is in the centre row's in-box part, or left of it
    const int seg_c = (nz > 1 ? ny : 0) + (ny > 1 ? 1 : 0) + (home_left ? 9 : 0);
    const int own = t - __shfl_sync(kAll, seg_beg - seg_pre, seg_c);
    // the list's segments without the empty ones
    const uint32_t full = __ballot_sync(kAll, seg_len > 0);
    const bool shifted = __any_sync(kAll, seg_len > 0 && shift != 0u);
    int* starts = reinterpret_cast<int*>(&w.row[0][kStartAt]);
    if (seg_len > 0) {
        const int k = __popc(full & ((1u << lane) - 1u));
        starts[k] = seg_pre;
        if (lane == top_bit(full)) starts[k + 1] = 0x7fffffff;
        w.seg[k] = make_float4(code_shift(shift & 3u, c.ext[0]) - ox, code_shift((shift >> 2) & 3u, c.ext[1]) - oy,
                               code_shift(shift >> 4, c.ext[2]) - oz, __int_as_float(seg_beg - seg_pre));
    }
    if (lane == 0) {
        w.row[0][kOriginAt] = __float_as_uint(shifted ? ox : 0.0f);
        w.row[0][kOriginAt + 1] = __float_as_uint(shifted ? oy : 0.0f);
        w.row[0][kOriginAt + 2] = __float_as_uint(shifted ? oz : 0.0f);
    }
    __syncwarp();
    // the drain's coordinates: relative to the origin where some segment is shifted, raw elsewhere
    const float hpx = shifted ? home_x - ox : h.x, hpy = shifted ? h.y - oy : h.y, hpz = shifted ? h.z - oz : h.z;

    // units: the list's entries dealt out in turn (entry g to unit g mod units), so that every
    // unit holds an even share of every home's neighbours and its busiest lane stands out
    // less than it does over a stretch of the list
    const int units = (total + kUnit - 1) / kUnit;
    const float per_unit = __fdividef(1.0f, (float)units);
    int own_slot, own_unit, q0, r0, q1, r1;  // (this lane's segment: its start is entry q0 of unit r0, its end q1 of r1)
    int total_q, total_r;
    deal(total, units, per_unit, total_q, total_r);
    deal(own, units, per_unit, own_slot, own_unit);
    deal(seg_pre, units, per_unit, q0, r0);
    deal(seg_pre + seg_len, units, per_unit, q1, r1);
    for (int u0 = 0; u0 < units; u0 += split) {
        // (before any warp stages over partial sums that part 0 may still be reading)
        if (split > 1 && u0 > 0) item_barrier(slot_of_item, 32 * split);
        const int unit = u0 + part;
        float fx = 0.0f, fy = 0.0f, fz = 0.0f;
        int count = 0;
        if (unit < units) {
            // ---- stage the unit's groups
            const int entries = total_q + (unit < total_r ? 1 : 0);
            const int ngroups = (entries + 31) >> 5;
            // the slot's column and fragment, so that its sign arrives at its bit of the mask: bit
            // 4 k + 3 - t is column 2 t + j of fragment n, k = 0..7: (n, j) = (2, 0), (0, 0),
            // (2, 1), (0, 1), (3, 0), (1, 0), (3, 1), (1, 1)
            uint32_t* frag = w.row[1] + (2 * (3 - (lane & 3)) + ((lane >> 3) & 1)) * 4 + (lane & 4 ? 0 : 2) + (lane >> 4);
            // the unit's part of each segment: slots [slot0, slot1), list entry slot * units + unit
            const int slot0 = q0 + (unit < r0 ? 1 : 0), slot1 = q1 + (unit < r1 ? 1 : 0);
            const bool has = slot1 > slot0;
            const uint32_t parts = __ballot_sync(kAll, has);
            if (has)
                w.part[__popc(parts & ((1u << lane) - 1u))] =
                    make_int2(seg_beg - seg_pre + unit, __popc(full & ((1u << lane) - 1u)));
            __syncwarp();
            // every position in flight at once (asynchronous copies: one round trip to L2 per
            // unit); a slot's segment is the count of segments that start at or before it
            const uint32_t start_bit = has ? 1u << (slot0 & 31) : 0u;
            const int start_group = slot0 >> 5;
            int before = -1;
            for (int gi = 0; gi < ngroups; gi++) {
                const uint32_t begins = __reduce_or_sync(kAll, start_group == gi ? start_bit : 0u);
                const int2 rec = w.part[before + __popc(begins & (0xffffffffu >> (31 - lane)))];
                before += __popc(begins);
                const int slot = gi * 32 + lane, j = rec.x + slot * units;
                copy_async16(slot < entries && CF_IN_BOUNDS(j, c.n), slots_at + 512 + 16 * slot, pos_sorted + j);
                if (shifted) w.row[1 + gi][lane] = (uint32_t)rec.y;
            }
            copy_async_wait();
            __syncwarp();
#pragma unroll 2
            for (int gi = 0; gi < ngroups; gi++) {
                float4& slot = w.c[1 + gi * 32 + lane];
                float4 p = slot;
                const uint32_t other = min(__float_as_uint(p.w) & kTypeMask, (uint32_t)(T - 1));
                p.w = __uint_as_float(4u * other);
                if (!kGeneric) {
                    float fx, fy, fz;
                    if (shifted) {
                        const float4 add = w.seg[w.row[1 + gi][lane]];
                        p.x += add.x;
                        p.y += add.y;
                        p.z += add.z;
                        fx = p.x * scale;
                        fy = p.y * scale;
                        fz = p.z * scale;
                        __syncwarp();  // every lane has read the group's segments
                    } else {
                        fx = fmaf(p.x, scale, -ox * scale);
                        fy = fmaf(p.y, scale, -oy * scale);
                        fz = fmaf(p.z, scale, -oz * scale);
                    }
                    const uint32_t xy = half2_bits(fx, fy);
                    const uint32_t z0 = half2_bits(fz, 0.0f);
                    const float qx = half_lo(xy), qy = half_hi(xy), qz = half_lo(z0);
                    const float sq = fmaf(qz, qz, fmaf(qy, qy, qx * qx));
                    const uint32_t s_hi = half2_bits(0.0f, sq);
                    frag[96 * gi] = xy;
                    frag[96 * gi + 32] = z0 | s_hi;
                    frag[96 * gi + 64] = half2_bits(sq - half_hi(s_hi), 1.0f);
                }
                slot = p;
            }
            __syncwarp();
            if (!kGeneric && (entries & 31) != 0 && lane >= (entries & 31)) {
                // padding up to a whole group: at the origin, with a square (60000 + 60000) that no
                // home passes
                frag[96 * ngroups - 96] = 0u;
                frag[96 * ngroups - 64] = 0x7b530000u;
                frag[96 * ngroups - 32] = 0x3c007b53u;
            }
            __syncwarp();
            int hits = 0;      // set bits of this lane in the unit
            uint32_t nz = 1u;  // bit 0: the sentinel's row; bit 1 + g: group g has a set bit

            // ---- filter: one bit per candidate
            for (int gi = 0; gi < ngroups; gi++) {
                uint32_t m;
                if (kGeneric) {
                    // an idle home sits at -kFar, far from every candidate
                    const float gx = active ? h.x : -kFar, gy = active ? h.y : -kFar, gz = active ? h.z : -kFar;
                    const int lim = entries - gi * 32;
                    m = 0u;
                    for (int q = 0; q < 32 && q < lim; q++) {
                        const float4 p = w.c[1 + gi * 32 + q];
                        const float dx = wrap_ref(p.x - gx, c.ext[0], c.half[0]);
                        const float dy = wrap_ref(p.y - gy, c.ext[1], c.half[1]);
                        const float dz = wrap_ref(p.z - gz, c.ext[2], c.half[2]);
                        if (fmaf(dz, dz, fmaf(dy, dy, dx * dx)) < thr_f) m |= 1u << q;
                    }
                } else {
                    const uint4 b = *reinterpret_cast<const uint4*>(
                        w.row[1 + gi] + min(lane & 3, 2) * 32 + (lane >> 2) * 4);
                    const uint32_t bn[4] = {b.x, b.y, b.z, b.w};
                    // row q's eight sign bits: the top halves of its results two to a word, the top bytes of those
                    // side by side in two words, the second shifted by four, so bit 3 of every nibble is a sign
                    uint32_t r[4], lo[4];
#pragma unroll
                    for (int f = 0; f < 2; f++) {
                        uint32_t d[2][8];
                        mma_32x8(a, bn[2 * f], d[0]);
                        mma_32x8(a, bn[2 * f + 1], d[1]);
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const uint32_t w = __byte_perm(__byte_perm(d[0][2 * q], d[0][2 * q + 1], 0x7632),
                                                           __byte_perm(d[1][2 * q], d[1][2 * q + 1], 0x7632), 0x7531);
                            if (f == 0)
                                lo[q] = w;
                            else
                                r[q] = bit_select(lo[q], w >> 4, 0x80808080u);
                        }
                    }
                    // the four rows' signs into one word, row q at bit 3 - q of every nibble; then a
                    // 4 x 4 transposition of the nibbles' bits over the quad leaves in lane 4 g + t the
                    // whole row g + 8 t, the signs of lane 4 g + t' at bit 3 - t' of every nibble
                    m = bit_select(bit_select(r[0], r[1] >> 1, 0x88888888u),
                                   bit_select(r[2], r[3] >> 1, 0x88888888u) >> 2, 0xccccccccu);
                    uint32_t o = __shfl_xor_sync(kAll, m, 2);
                    m = bit_select(m, __funnelshift_l(o, o, lane & 2 ? 2 : 30), lane & 2 ? 0x33333333u : 0xccccccccu);
                    o = __shfl_xor_sync(kAll, m, 1);
                    m = bit_select(m, __funnelshift_l(o, o, lane & 1 ? 1 : 31), lane & 1 ? 0x55555555u : 0xaaaaaaaau);
                }
                if (unit == own_unit && gi == own_slot >> 5) m &= ~(1u << (own_slot & 31));
                __syncwarp();  // every lane has read the group's words
                w.row[1 + gi][lane] = m;
                hits += __popc(m);
                nz |= m != 0u ? 2u << gi : 0u;
            }

            // ---- drain: every set bit of this lane, highest first, kPer per trip.  The trip
            // count is uniform over the warp; a lane whose mask runs out moves to its next
            // non-empty row with one load, and one with no hit left stays at row 0, whose one
            // bit is the sentinel.
            __syncwarp();
            const int trips = (__reduce_max_sync(kAll, hits) + kPer - 1) / kPer;
            int r = top_bit(nz);
            uint32_t m = r ? w.row[r][lane] : 0x80000000u;
            uint32_t row_at = slots_at + 512 * r;
            // pairs within rounding of the threshold wait: the last one's slot and how many
            uint32_t open_at = 0u;
            int open = 0;
            for (int trip = 0; trip < trips; trip++) {
                uint32_t at[kPer];
                float4 p[kPer];
#pragma unroll
                for (int q = 0; q < kPer; q++) {
                    // the slot of the mask's top bit; the bit cleared; if it was the row's last,
                    // the next row with a bit (predicated: no divergence in the trip)
                    asm volatile("{\n\t.reg .pred z;\n\t.reg .u32 b, o;\n\t"
                                 "bfind.u32 b, %1;\n\t"
                                 "mad.lo.u32 %0, b, 16, %2;\n\t"
                                 "shl.b32 o, 1, b;\n\t"
                                 "xor.b32 %1, %1, o;\n\t"
                                 "setp.eq.u32 z, %1, 0;\n\t"
                                 "@z shl.b32 o, 1, %4;\n\t"
                                 "@z lop3.b32 %3, %3, o, 1, 0xba;\n\t"  // (nz & ~o) | 1
                                 "@z bfind.u32 %4, %3;\n\t"
                                 "@z mad.lo.u32 %2, %4, 512, %5;\n\t"
                                 "@z mad.lo.u32 o, %4, 384, %6;\n\t"
                                 "@z ld.shared.u32 %1, [o];\n\t}"
                                 : "=r"(at[q]), "+r"(m), "+r"(row_at), "+r"(nz), "+r"(r)
                                 : "r"(slots_at), "r"(masks_at));
                    p[q] = lds128(at[q]);
                }
                PairTerm k[kPer];
#pragma unroll
                for (int q = 0; q < kPer; q++)
                    k[q] = pair_term<kGeneric, kUniformR>(c, p[q], hpx, hpy, hpz, force_at, pair_at);
#pragma unroll
                for (int q = 0; q < kPer; q++)
                    asm("{\n\t.reg .pred p, b;\n\t"
                        "setp.lt.f32 p, %6, %7;\n\t"
                        "setp.lt.and.f32 b, %6, %8, !p;\n\t"
                        "@p fma.rn.f32 %0, %9, %12, %0;\n\t"
                        "@p fma.rn.f32 %1, %10, %12, %1;\n\t"
                        "@p fma.rn.f32 %2, %11, %12, %2;\n\t"
                        "@p add.s32 %3, %3, 1;\n\t"
                        "@b mov.u32 %4, %13;\n\t"
                        "@b add.s32 %5, %5, 1;\n\t}"
                        : "+f"(fx), "+f"(fy), "+f"(fz), "+r"(count), "+r"(open_at), "+r"(open)
                        : "f"(k[q].d2), "f"(k[q].lo), "f"(kUniformR ? c.thr_hi_uniform : k[q].lo + c.band), "f"(k[q].dx),
                          "f"(k[q].dy), "f"(k[q].dz), "f"(k[q].weight), "r"(at[q]));
            }
            // the pairs left open take the exact test, after the unit's others: the one of a lane
            // that has one; a lane with more walks its masks again for them
            if (__any_sync(kAll, open > 0)) {
                int row = open > 1 ? ngroups : 0;
                m = row ? w.row[row][lane] : 0u;
                while (open > 0) {
                    if (row) {
                        while (m == 0u) m = w.row[--row][lane];
                        const int bit = top_bit(m);
                        m ^= 1u << bit;
                        open_at = slots_at + 512 * row + 16 * bit;
                    }
                    const float4 p = lds128(open_at);
                    const PairTerm k = pair_term<kGeneric, kUniformR>(c, p, hpx, hpy, hpz, force_at, pair_at);
                    if (!(k.d2 < k.lo) && k.d2 < k.lo + c.band) {
                        open--;
                        // the candidate's sorted index, from its place in the list
                        const int g = ((int)(open_at - slots_at) / 16 - 32) * units + unit;
                        int s = 0;
                        while (starts[s + 1] <= g) s++;
                        const int j = __float_as_int(w.seg[s].w) + g;
                        const float* origin = reinterpret_cast<const float*>(&w.row[0][kOriginAt]);
                        const float thr = kUniformR ? c.thr_uniform
                                                    : tables->threshold[type * kTableStride +
                                                                        (__float_as_uint(p.w) >> 2)];
                        if (g < total && CF_IN_BOUNDS(j, c.n) && pair_exact<kGeneric>(c, h, home_left, origin, p, pos_sorted[j], thr)) {
                            count++;
                            fx = fmaf(k.dx, k.weight, fx);
                            fy = fmaf(k.dy, k.weight, fy);
                            fz = fmaf(k.dz, k.weight, fz);
                        }
                    }
                }
            }
            __syncwarp();
        }
        if (split > 1) {
            // the round's units in order: the other warps leave their partial sums in their own
            // staging area, the item's warps meet at a named barrier (id 1 + item slot,
            // 32 * split threads) and part 0 adds them
            if (part != 0) w.c[1 + lane] = make_float4(fx, fy, fz, __int_as_float(count));
            item_barrier(slot_of_item, 32 * split);
        }
        sum_x += fx;
        sum_y += fy;
        sum_z += fz;
        sum_n += count;
        if (split > 1 && part == 0) {
            const int more = min(split, units - u0);
            for (int q = 1; q < more; q++) {
                const float4 v = (&w)[q].c[1 + lane];
                sum_x += v.x;
                sum_y += v.y;
                sum_z += v.z;
                sum_n += __float_as_int(v.w);
            }
        }
    }
    if (part != 0 || !active || !CF_IN_BOUNDS(i, c.n)) return;
    if (c.integrate_apart)
        acc[i] = make_float4(sum_x, sum_y, sum_z, __int_as_float(sum_n));  // for integrate_kernel
    else
        integrate(c, h, make_float4(sum_x, sum_y, sum_z, 0.0f), sum_n, i, kForm == kApart ? vel_in : vel,
                  kForm == kApart ? counts_in : counts, pos, vel, acc, counts);
}

#ifndef CF_FORCE_WARPS
__global__ void __launch_bounds__(256)
    integrate_kernel(StepConsts c, StepState state)
{
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= c.n) return;
    const float4 f = state.acc[i];
    integrate(c, state.pos[i], f, __float_as_int(f.w), (uint32_t)i, state.vel, state.counts, state.pos_out, state.vel_out,
              state.acc, state.counts_out);
}

// The filter's work of one step, from the cell list alone: per item
// the candidates staged (the union of its homes' stencils, as the force
// kernel concatenates them) and the tests of them by the item's particles.
// One thread per item; out[0] += staged, out[1] += staged * particles.
__global__ void __launch_bounds__(256)
    force_work_kernel(StepConsts c, const uint32_t* __restrict__ keys_sorted, const uint32_t* __restrict__ cell_off,
                      const Item* __restrict__ items, const int* __restrict__ n_items,
                      unsigned long long* __restrict__ out)
{
    const int k = blockIdx.x * 256 + threadIdx.x;
    unsigned long long staged = 0, tested = 0;
    if (k < *n_items) {
        const Item it = items[k];
        const int mx = c.grid.m[0], my = c.grid.m[1], mz = c.grid.m[2];
        const uint32_t world_base = (uint32_t)it.world * (uint32_t)c.grid.cells_w;
        const int yc = it.yz & 0xffff, zc = it.yz >> 16;
        const uint32_t row_base = world_base + (uint32_t)((zc * my + yc) * mx);
        const int x0 = (int)(keys_sorted[it.first] - row_base);
        const int x1 = (int)(keys_sorted[it.first + it.count - 1] - row_base);
        const bool generic = c.grid.generic != 0;
        const int ny = my > 1 ? 3 : 1, nz = mz > 1 ? 3 : 1;
        const bool ring = generic && x1 - x0 + 3 >= mx;
        const int xlo = ring ? 0 : x0 - 1, xhi = ring ? mx - 1 : x1 + 1;
        float o, r;
        const bool folded = !generic && stencil_origin_x(x0, x1, mx, c.cell[0], c.ext[0], o, r);
        for (int row = 0; row < ny * nz; row++) {
            const int dy_row = ny > 1 ? (row % ny) - 1 : 0, dz_row = nz > 1 ? (row / ny) - 1 : 0;
            const int yy = wrap_index(yc + dy_row, my), zz = wrap_index(zc + dz_row, mz);
            const uint32_t base = world_base + (uint32_t)((zz * my + yy) * mx);
            // in the box, left of it, right of it
            staged += cell_off[base + min(xhi, mx - 1) + 1] - cell_off[base + max(xlo, 0)];
            if (folded || xlo < 0) staged += cell_off[base + mx] - cell_off[base + (folded ? mx - 2 : xlo + mx)];
            if (folded ? xlo > 0 : xhi >= mx) staged += cell_off[base + (folded ? 0 : xhi - mx) + 1] - cell_off[base];
        }
        tested = staged * (unsigned long long)it.count;
    }
    // one atomic per warp
    for (int o = 16; o > 0; o >>= 1) {
        staged += __shfl_down_sync(0xffffffffu, staged, o);
        tested += __shfl_down_sync(0xffffffffu, tested, o);
    }
    if ((threadIdx.x & 31) == 0 && (staged | tested)) {
        atomicAdd(&out[0], staged);
        atomicAdd(&out[1], tested);
    }
}

// Items: each row of cells (rows = (y, z) pairs) cut into chunks of at most
// 32 sorted particles.  One block; rows are split into contiguous segments.
__global__ void __launch_bounds__(1024)
    plan_kernel(const uint32_t* __restrict__ cell_off, int mx, int my, int mz, int rows, Item* __restrict__ items,
                int* __restrict__ n_items)
{
    __shared__ uint32_t s_chunk[1024];
    const int tid = threadIdx.x;
    const int per = (rows + 1023) / 1024;
    const int r0 = min(tid * per, rows), r1 = min(r0 + per, rows);
    uint32_t chunks = 0;
    for (int r = r0; r < r1; r++) {
        const uint32_t cnt = cell_off[(r + 1) * mx] - cell_off[r * mx];
        chunks += (cnt + 31u) / 32u;
    }
    s_chunk[tid] = chunks;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const uint32_t b = tid >= o ? s_chunk[tid - o] : 0u;
        __syncthreads();
        s_chunk[tid] += b;
        __syncthreads();
    }
    uint32_t item = s_chunk[tid] - chunks;
    for (int r = r0; r < r1; r++) {
        const uint32_t start = cell_off[r * mx];
        const uint32_t cnt = cell_off[(r + 1) * mx] - start;
        const int yz_w = r / my;
        const int yz = (r - yz_w * my) | ((yz_w % mz) << 16), world = yz_w / mz;
        for (uint32_t k = 0; k < cnt; k += 32u) items[item++] = Item{(int)(start + k), (int)min(32u, cnt - k), yz, world};
    }
    if (tid == 1023) *n_items = (int)s_chunk[1023];
}

#else
constexpr size_t kSmemDefault = 48u << 10;  // of a block, without opting in

// Shared memory of a block: staging per warp, the pair table without a uniform
// radius, and the force table of one world or, in a batch, of each item of the block.
size_t force_smem(int warps, int T, bool uniform, int force_tables)
{
    return sizeof(WarpSmem) * warps + (size_t)T * T * ((uniform ? 0 : sizeof(float4)) + sizeof(float) * force_tables);
}

#endif

}  // namespace

// W = warps per block, B = resident blocks per SM the register budget is sized for.  Every (W, B) is a translation unit of
// its own (this file with CF_FORCE_WARPS and CF_FORCE_BLOCKS), so that a process loads the forms of the one it
// uses: in one unit the 60 forms took a process's first step 6.9 ms, now 0.8.
template <int W, int B>
cudaError_t launch_variant(const StepConsts& c, const PairTables* tables, const float4* pos_sorted,
                           const uint32_t* vals_sorted, const uint32_t* cell_off, const Item* items,
                           const int* n_items, int max_items, const StepState& state, cudaStream_t st);

#ifdef CF_FORCE_WARPS

template <int W, int B>
cudaError_t launch_variant(const StepConsts& c, const PairTables* tables, const float4* pos_sorted,
                           const uint32_t* vals_sorted, const uint32_t* cell_off, const Item* items,
                           const int* n_items, int max_items, const StepState& state, cudaStream_t st)
{
    const size_t smem = force_smem(W, c.num_types, c.uniform_r != 0, c.grid.worlds == 1 ? 1 : W / c.split);
    const int blocks = (int)(((long long)max_items * c.split + W - 1) / W);
    const bool apart = state.pos_out != state.pos;
    cudaError_t e = cudaSuccess;
    const auto launch = [&](auto kernel) {
        // opted in where a launch needs it (to the most that any does, the same from every thread): the attribute
        // loads the kernel, and all 60 at a world's creation took a process's first one from 1.5 to 8 ms
        if (smem > kSmemDefault)
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)force_smem(W, CF_MAX_TYPES, false, W <= 4 ? W : 1));
        if (e != cudaSuccess) return;
        kernel<<<blocks, 32 * W, smem, st>>>(c, tables, pos_sorted, vals_sorted, cell_off, items, n_items, max_items,
                                             state.pos_out, state.vel_out, state.acc, state.counts_out, state.vel,
                                             state.counts);
    };
#define CF_FORCE_FORMS(G, U)                                                                       \
    launch(apart ? step_force_kernel<W, B, G, U, kApart> : step_force_kernel<W, B, G, U, kInPlace>)
    if (c.grid.generic) {
        if (c.uniform_r)
            CF_FORCE_FORMS(true, true);
        else
            CF_FORCE_FORMS(true, false);
    } else if (c.grid.bin_shift) {
        if (apart) return cudaErrorInvalidValue;  // (no caller)
        launch(c.uniform_r ? step_force_kernel<W, B, false, true, kBins> : step_force_kernel<W, B, false, false, kBins>);
    } else {
        if (c.uniform_r)
            CF_FORCE_FORMS(false, true);
        else
            CF_FORCE_FORMS(false, false);
    }
#undef CF_FORCE_FORMS
    if (e != cudaSuccess) return e;
    note_launches(st);
    return cudaGetLastError();
}

template cudaError_t launch_variant<CF_FORCE_WARPS, CF_FORCE_BLOCKS>(
    const StepConsts& c, const PairTables* tables, const float4* pos_sorted, const uint32_t* vals_sorted,
    const uint32_t* cell_off, const Item* items, const int* n_items, int max_items, const StepState& state,
    cudaStream_t st);

#define CF_FORCE_READER(w, b) CF_BOUNDS_READER(step_##w##_##b)
#define CF_FORCE_READER_OF(w, b) CF_FORCE_READER(w, b)
CF_FORCE_READER_OF(CF_FORCE_WARPS, CF_FORCE_BLOCKS)

#else

cudaError_t launch_force_work(const StepConsts& c, const uint32_t* keys_sorted, const uint32_t* cell_off,
                              const Item* items, const int* n_items, int max_items, unsigned long long* out,
                              cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(out, 0, 2 * sizeof(unsigned long long), st);
    if (e != cudaSuccess || max_items <= 0) return e;
    force_work_kernel<<<(max_items + 255) / 256, 256, 0, st>>>(c, keys_sorted, cell_off, items, n_items, out);
    note_launches(st);
    return cudaGetLastError();
}

namespace {
// From this many particles the integrator is a kernel of its own, in particle order: the
// force kernel's scattered access to a particle's state (six sectors) shrinks to one store.  Apart / in the force kernel,
// us a step (evenly spread with many and with few neighbours, in blobs, 64 worlds): 20,000 27.1 / 27.4, 27.0 / 27.5,
// 29.3 / 31.2, 29.1 / 29.2; 70,000 41.4 / 43.5, 33.5 / 35.8, 64.0 / 62.0, 34.2 / 37.5; 100,000 59.9 / 59.8,
// 41.6 / 44.8, 84.5 / 84.8, 39.5 / 43.3; 150,000 90.6 / 89.6, 47.0 / 52.1, 136.5 / 137.3, 49.8 / 54.0; 300,000 74 / 77,
// 68 / 72, 94 / 103, 76 / 93; 1M 253 / 261, 185 / 197, 320 / 340, 225 / 255; below 10,000 up to 2.2 more for the launch.  Worlds
// whose particles have clustered over many steps gain less (100,000 after 25 to 100 steps, launches outside a graph:
// 63.5 / 62.4 and 72.6 / 70.8).  From 150,000 it costs 1 % at most.
constexpr int kIntegrateApart = 150000;
}

int max_step_items(int n, const Grid& g) { return (n + 31) / 32 + g.worlds * g.m[1] * g.m[2]; }

// The force kernel, and the integrator where it is a kernel of its own (the plan is part of the cell list).
int step_launches(int n) { return n > 0 ? 1 + (integrate_apart(n) ? 1 : 0) : 0; }

bool integrate_apart(int n) { return n >= kIntegrateApart; }

// The variant of a world that chose none.  Warps per item: the power of two that
// fills the GPU, at most two per unit that an item of evenly spread particles
// has (one below half a unit, where further warps only add their start: 10.9
// against 13.6 us at 2,048 particles).  Occupancy: the most registers that hold
// all warps at once, else (several waves) the most warps: six blocks of four against ten of
// two 459 / 475 us at 1M in blobs and 240 / 256 at 64 worlds of 20,000.
int default_force_variant(int n, const Grid& g)
{
    const double cells = (double)g.cells, pop = (double)n / cells;
    const double homes = std::min(32.0, std::max(pop * g.m[0], 1.0));
    const double candidates = 9.0 * pop * std::min((double)g.m[0], homes / pop + 3.0);
    const double items = n / 32.0 + 0.5 * std::min(cells / g.m[0], (double)n);
    const double slots = 24.0 * num_sms();
    int split = 1;
    if (candidates >= 0.5 * kUnit)
        while (split < 8 && 2 * split * (n / 32.0) <= slots && split < 2.0 * std::ceil(candidates / kUnit)) split *= 2;
    const double warps = items * split;
    const int occupancy = warps <= 16.0 * num_sms() ? 2 : warps <= 20.0 * num_sms() ? 1 : 0;
    int log2 = 0;
    while ((1 << log2) < split) log2++;
    return occupancy + kForceOccupancies * log2;
}

cudaError_t launch_step_plan(const uint32_t* cell_off, int n, const Grid& g, Item* items, int* n_items,
                             cudaStream_t st)
{
    if (n <= 0) return cudaMemsetAsync(n_items, 0, sizeof(int), st);
    plan_kernel<<<1, 1024, 0, st>>>(cell_off, g.m[0], g.m[1], g.m[2], g.worlds * g.m[1] * g.m[2], items, n_items);
    note_launches(st);
    return cudaGetLastError();
}

cudaError_t launch_step_force(const StepConsts& c, const PairTables* tables, const float4* pos_sorted,
                              const uint32_t* vals_sorted, const uint32_t* cell_off, const Item* items,
                              const int* n_items, int max_items, const StepState& state, cudaStream_t st)
{
    if (c.n <= 0 || max_items <= 0) return cudaSuccess;
    if (c.split < 1 || c.split > 16 || (c.split & (c.split - 1)) != 0) return cudaErrorInvalidValue;
    cudaError_t e;
#define CF_FORCE_VARIANT(W, B) \
    launch_variant<W, B>(c, tables, pos_sorted, vals_sorted, cell_off, items, n_items, max_items, state, st)
    if (c.split <= 2)
        e = c.variant == 0 ? CF_FORCE_VARIANT(4, 6) : c.variant == 1 ? CF_FORCE_VARIANT(2, 10) : CF_FORCE_VARIANT(4, 4);
    else if (c.split == 4)
        e = c.variant == 0 ? CF_FORCE_VARIANT(4, 6) : c.variant == 1 ? CF_FORCE_VARIANT(4, 5) : CF_FORCE_VARIANT(4, 4);
    else
        e = c.split == 8 ? CF_FORCE_VARIANT(8, 2) : CF_FORCE_VARIANT(16, 1);
#undef CF_FORCE_VARIANT
    if (e != cudaSuccess || !c.integrate_apart) return e;
    integrate_kernel<<<(c.n + 255) / 256, 256, 0, st>>>(c, state);
    note_launches(st);
    return cudaGetLastError();
}

#endif  // CF_FORCE_WARPS

}  // namespace cf
