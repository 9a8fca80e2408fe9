// All-pairs histograms over spatially sorted atoms (full_pairs_histograms_coords,
// Extensions/pairs_histograms.pyx:289-335).
//
// k_full_tiles (hist_kernels.cu) evaluates every pair i < j, although at
// r <= 20 A in a 103 A box only 3.5 % of them are in range.  Here the atoms
// are sorted along a serpentine of columns first, so that 32 consecutive
// atoms (a block) fill about a cube, and only pairs of blocks that can hold a
// pair in range are evaluated:
//
//   k_cell_bounds   range of the atoms' real-space positions;
//   k_cell_count    cell of every atom and its rank there;
//   k_cell_scan     exclusive scan of the cell counts (one CTA);
//   k_cell_scatter  atoms to their sorted places;
//   k_cell_blocks   bounding boxes of each block, in box coordinates and in
//                   real space (one warp per block);
//   k_cell_list     the pairs of blocks that can hold a pair in range;
//   k_cell_hist     those pairs of blocks: a warp holds one atom of the row
//                   block per lane and takes the columns in turn.
//
// What makes it exact: the float32 difference a - b and the reference's
// round() are monotone, so if round() of the smallest and of the largest
// difference two blocks can have agree on every axis, it is that constant k
// for every pair of the two blocks, and box = (a - b) - k needs no rounding
// of its own (most blocks: k = 0 and no subtraction).  Then every real-space
// vector of the two blocks lies within their bounding boxes' difference minus
// k B, whose distance from the origin bounds the pairs' distances from below.
// Where k is not constant, |real| >= |g| w with g the wrapped difference of
// one axis and w the box's perpendicular width bounds them, and the pairs
// that are left take the whole minimum image (pair_s).  A block pair is
// skipped only beyond maxD plus a margin far above the float32 rounding of
// positions and distances.  Distances are symmetric bit for bit, so a pair is
// evaluated once, in either order, and counted at [el(i)][el(j)] for the
// original indexes i < j.
//
// Where the boxes' largest distance is below maxD (and their smallest above
// minD) by the same margin, every pair of the two blocks is in range.
//
// Bound: SM issue and the FMA pipe (blocks wholly in range: issue and the
// shared-memory pipe, 77 % of its wavefronts).  Two columns at a time go through
// add/fma.rn.f32x2 (one issue slot for two IEEE float32 operations, at the
// FMA pipe's scalar rate), the bin comes from an approximate quotient that is
// checked against the distance to the next integer, and one lane in three of
// an evaluated pair counts; per-lane queues of the counted pairs, as in
// k_full_tiles, measured slower here (1.10 against 0.90 ms per call: the lanes
// of a block have unequal numbers of neighbours).  Measured (whole host calls):
// 100,000 atoms, 103 A box with gamma = 120, r 0-20 A: 6.92 -> 0.63 ms, the
// kernel 6.81 -> 0.55 ms for 5.2e5 of 4.9e6 block pairs, 31 issue slots per
// column of 32 rows; 11,303 atoms, r 0-12 A: 335 -> 84 us; a 100,000-atom
// particle with every pair counted (shape function): 12.5 -> 4.1 ms, 24 issue
// slots per column (5.3 ms and 32 with each pair tested).
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "cell_walk.cuh"
#include "frmc_ptx.cuh"

namespace frmc {

constexpr int kCellCap = 1 << 16;     // cells at most (one CTA scans them)
constexpr long long kCellList = 1 << 23;  // entries of a list of block pairs at most (64 MB)
constexpr int kCellSub = 8;           // cells per block along a column

struct CellSort {
    // the caller's arrays (k_cell_bounds packs them; host memory where the
    // device reads it), or null: the atoms are packed already
    const float *coords;     // (n, 3)
    const int *el, *src_mol;
    float4 *atoms4;          // (x, y, z, el bits)
    int *mol;
    int n, nb, ne, hs, pbc;
    Basis B;
    double volume;           // of the box (0: of the range of positions)
    CellScalars *sc;
    int *cells;              // counts, then starts
    int2 *place;             // per atom: cell, rank
    float *x, *y, *z;        // sorted, negated; NaN past the last atom
    int4 *meta;              // el ne hs, el hs, molecule, original index
    float4 *bounds;          // per block: 3 float4 (box lo, box hi, real lo, real hi)
};

struct CellHist {
    CellWalk walk;
    float s_lo, s_hi, minD, binw;
    float inv, off, slack;   // 1 / bin, 1 - min / bin, see CellBins
    unsigned total;
    unsigned *intra, *inter;
    int smem_hist;
};

__device__ __forceinline__ unsigned ordered_bits(float f)
{
    const unsigned u = __float_as_uint(f);
    return u & 0x80000000u ? ~u : u | 0x80000000u;
}

__device__ __forceinline__ float from_ordered(unsigned u)
{
    return __uint_as_float(u & 0x80000000u ? u & 0x7fffffffu : ~u);
}

// Position in real space (sorting and bounds only; the margin covers its rounding).
__device__ __forceinline__ float3 cell_real(const CellSort &p, float3 c)
{
    if (!p.pbc)
        return c;
    return make_float3(c.x * p.B.b[0] + c.y * p.B.b[3] + c.z * p.B.b[6],
                       c.x * p.B.b[1] + c.y * p.B.b[4] + c.z * p.B.b[7],
                       c.x * p.B.b[2] + c.y * p.B.b[5] + c.z * p.B.b[8]);
}

// The atoms' range, and their packed form where they come as three arrays:
// 256 atoms a turn, whose 768 coordinates are read in order.  Bound by the link
// to host memory: 100,000 atoms (2 MB) in 14 us, where three copies and an 8 us
// kernel went before.
__global__ void __launch_bounds__(256) k_cell_bounds(CellSort p)
{
    grid_launch_dependents();
    __shared__ float tile[3 * 256];
    __shared__ unsigned red[7];
    const int tid = threadIdx.x;
    if (tid < 7)
        red[tid] = 0u;
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY}, am = 0.f;
    bool strange = false;
    for (int i0 = blockIdx.x * 256; i0 < p.n; i0 += gridDim.x * 256) {
        const int i = i0 + tid;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p.coords) {
            int el = 0, mol = 0;
            if (i < p.n) {
                el = p.el[i];
                mol = p.src_mol[i];
            }
            const int m = 3 * min(256, p.n - i0);
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 3; ++k)
                if (tid + 256 * k < m)
                    tile[tid + 256 * k] = p.coords[3ll * i0 + tid + 256 * k];
            __syncthreads();
            if (i < p.n) {
                a = make_float4(tile[3 * tid], tile[3 * tid + 1], tile[3 * tid + 2], __int_as_float(el));
                p.atoms4[i] = a;
                p.mol[i] = mol;
            }
        } else if (i < p.n) {
            a = p.atoms4[i];
        }
        if (i >= p.n)
            continue;  // (every thread takes the same turns)
        const float3 r = cell_real(p, make_float3(a.x, a.y, a.z));
        am = fmaxf(am, fmaxf(fabsf(a.x), fmaxf(fabsf(a.y), fabsf(a.z))));
        strange |= !(fabsf(a.x) < INFINITY && fabsf(a.y) < INFINITY && fabsf(a.z) < INFINITY);
        lo[0] = fminf(lo[0], r.x); lo[1] = fminf(lo[1], r.y); lo[2] = fminf(lo[2], r.z);
        hi[0] = fmaxf(hi[0], r.x); hi[1] = fmaxf(hi[1], r.y); hi[2] = fmaxf(hi[2], r.z);
    }
    __syncthreads();
    unsigned v[7];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        v[k] = ~ordered_bits(lo[k]);
        v[3 + k] = ordered_bits(hi[k]);
    }
    v[6] = __float_as_uint(am);
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        v[k] = __reduce_max_sync(0xffffffffu, v[k]);
        if ((tid & 31) == 0)
            atomicMax(&red[k], v[k]);
    }
    if (strange)
        p.sc->strange = 1u;
    __syncthreads();
    if (tid < 7)
        atomicMax(tid < 3 ? &p.sc->nlo[tid] : tid < 6 ? &p.sc->hi[tid - 3] : &p.sc->amax, red[tid]);
}

struct CellGeom {
    float lo[3], inv[3];
    int n[3];
};

// Columns (x, y) about as wide as the cube that holds one block at the mean
// density, cut into cells of an eighth of it along z.  A free system without
// extent on an axis has no density: one cell, in no order (a sheet of 11,000 atoms,
// all pairs within 20 A: 115 us, and 295 with every pair evaluated).
__device__ CellGeom cell_geom(const CellSort &p)
{
    CellGeom g;
    float ext[3];
    for (int k = 0; k < 3; ++k) {
        g.lo[k] = from_ordered(~p.sc->nlo[k]);
        ext[k] = from_ordered(p.sc->hi[k]) - g.lo[k];
        if (!(ext[k] > 0.f && ext[k] < INFINITY))
            ext[k] = 0.f;
    }
    const float vol = p.volume > 0.0 ? (float)p.volume : ext[0] * ext[1] * ext[2];
    const float a = cbrtf(vol * (float)kCellBlock / (float)p.n);
    for (int k = 0; k < 3; ++k) {
        const float m = a > 0.f ? ext[k] / a * (k == 2 ? (float)kCellSub : 1.f) : 1.f;
        g.n[k] = m < 1.f ? 1 : (m > 4096.f ? 4096 : (int)(m + 0.5f));
    }
    while ((long long)g.n[0] * g.n[1] > kCellCap) {
        g.n[0] = (g.n[0] + 1) / 2;
        g.n[1] = (g.n[1] + 1) / 2;
    }
    g.n[2] = min(g.n[2], max(1, kCellCap / (g.n[0] * g.n[1])));
    for (int k = 0; k < 3; ++k) g.inv[k] = ext[k] > 0.f ? (float)g.n[k] / ext[k] : 0.f;
    return g;
}

__device__ __forceinline__ int cell_axis(const CellGeom &g, int k, float v)
{
    const float t = (v - g.lo[k]) * g.inv[k];
    return t > 0.f ? (t < (float)g.n[k] ? (int)t : g.n[k] - 1) : 0;  // NaN: 0
}

__global__ void __launch_bounds__(256) k_cell_count(CellSort p)
{
    grid_dependency_wait();
    grid_launch_dependents();
    __shared__ CellGeom g;
    if (threadIdx.x == 0) {
        g = cell_geom(p);
        if (blockIdx.x == 0)
            p.sc->ncells = g.n[0] * g.n[1] * g.n[2];
    }
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n)
        return;
    const float4 a = p.atoms4[i];
    const float3 r = cell_real(p, make_float3(a.x, a.y, a.z));
    const int ix = cell_axis(g, 0, r.x), iy = cell_axis(g, 1, r.y), iz = cell_axis(g, 2, r.z);
    // serpentine: neighbouring columns join at the same end
    const int col = ix * g.n[1] + (ix & 1 ? g.n[1] - 1 - iy : iy);
    const int cell = col * g.n[2] + (col & 1 ? g.n[2] - 1 - iz : iz);
    p.place[i] = make_int2(cell, atomicAdd(p.cells + cell, 1));
}

// Exclusive scan in place of n counts (the sort's cells where n is 0), 4,096 a
// turn; the array is zero up to the next multiple of 4,096.
__global__ void __launch_bounds__(1024) k_cell_scan(int *cells, const CellScalars *sc, int n)
{
    grid_dependency_wait();
    grid_launch_dependents();
    __shared__ int warp[2][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int turns = ((n ? n : sc->ncells) + 4095) / 4096;
    int carry = 0;
    int4 *v = reinterpret_cast<int4 *>(cells) + threadIdx.x;
    int4 c = *v;
    for (int t = 0; t < turns; ++t, v += 1024) {
        const int4 nxt = t + 1 < turns ? v[1024] : make_int4(0, 0, 0, 0);
        const int mine = c.x + c.y + c.z + c.w;
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, o);
            incl += lane >= o ? u : 0;
        }
        if (lane == 31)
            warp[t & 1][w] = incl;
        __syncthreads();
        // every warp scans the 32 warp totals itself
        int all = warp[t & 1][lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, all, o);
            all += lane >= o ? u : 0;
        }
        const int before = w ? __shfl_sync(0xffffffffu, all, w - 1) : 0;
        const int at = carry + before + incl - mine;
        *v = make_int4(at, at + c.x, at + c.x + c.y, at + c.x + c.y + c.z);
        carry += __shfl_sync(0xffffffffu, all, 31);
        c = nxt;
    }
}

// el * f, or a value beyond every histogram (the caller's element indexes are
// not checked).
__device__ __forceinline__ int cell_offset(int el, long long f)
{
    const long long v = el * f;
    return v > (1ll << 30) || v < -(1ll << 30) ? 1 << 30 : (int)v;
}

__global__ void __launch_bounds__(256) k_cell_scatter(CellSort p)
{
    grid_dependency_wait();
    grid_launch_dependents();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.nb * kCellBlock)
        return;
    if (i >= p.n) {
        p.x[i] = p.y[i] = p.z[i] = __int_as_float(0x7fc00000);  // no pair in range
        p.meta[i] = make_int4(0, 0, 0, 0);
        return;
    }
    const int2 pl = p.place[i];
    const int at = p.cells[pl.x] + pl.y;
    const float4 c = p.atoms4[i];
    const int el = __float_as_int(c.w);
    p.x[at] = -c.x;
    p.y[at] = -c.y;
    p.z[at] = -c.z;
    if ((unsigned)el >= (unsigned)p.ne)
        p.sc->bad = 1u;
    p.meta[at] = make_int4(cell_offset(el, (long long)p.ne * p.hs), cell_offset(el, p.hs), p.mol[i], i);
}

__device__ __forceinline__ float warp_min(float v)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__global__ void __launch_bounds__(256) k_cell_blocks(CellSort p)
{
    grid_dependency_wait();
    grid_launch_dependents();
    const int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (b >= p.nb)
        return;
    const int lane = threadIdx.x & 31, i = b * kCellBlock + lane;
    const float3 c = make_float3(-p.x[i], -p.y[i], -p.z[i]);
    const float3 r = cell_real(p, c);
    // NaN atoms are in no pair; fminf and fmaxf pass over them
    const float v[6] = {c.x, c.y, c.z, r.x, r.y, r.z};
    float lo[6], hi[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        lo[k] = warp_min(v[k]);
        hi[k] = -warp_min(-v[k]);
    }
    if (lane == 0) {
        p.bounds[3 * b] = make_float4(lo[0], lo[1], lo[2], hi[0]);
        p.bounds[3 * b + 1] = make_float4(hi[1], hi[2], lo[3], lo[4]);
        p.bounds[3 * b + 2] = make_float4(lo[5], hi[3], hi[4], hi[5]);
    }
}

constexpr int kListThreads = 256, kListPer = 8;  // offsets a thread tests

// A CTA per row block and 2,048 offsets: the pairs of blocks that can hold a
// pair within reach, appended to the list (their order changes no count).
// Bound by the bounds it reads (48 bytes a test, from L2): 4.9e6 tests 26 us.
template <int BM>
__global__ void __launch_bounds__(kListThreads) k_cell_list(CellWalk p)
{
    grid_dependency_wait();
    grid_launch_dependents();
    const int I = p.i0 + blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float reach = p.reach0 + p.reach1 * __uint_as_float(p.sc->amax);
    const BlockBox a = block_box(p.bounds, I);
    const int o0 = blockIdx.y * (kListThreads * kListPer) + threadIdx.x;
    unsigned code[kListPer], found = 0u;
#pragma unroll
    for (int k = 0; k < kListPer; ++k) {
        const int o = o0 + k * kListThreads;
        const int J = o < p.half ? column_block(I, o, p.nb) : -1;
        unsigned pack = 0u;
        int what = -1;
        if (J >= 0)
            what = block_test<BM>(p, a, block_box(p.bounds, J), reach, pack);
        code[k] = what >= 0 ? list_code(what, pack) : ~0u;
        found += what >= 0;
    }
    // places: the threads before this one, and one claim per CTA
    __shared__ unsigned sums[kListThreads / 32], base;
    unsigned at = found;
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
        const unsigned v = __shfl_up_sync(0xffffffffu, at, d);
        at += lane >= d ? v : 0u;
    }
    if (lane == 31)
        sums[warp] = at;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned all = 0u;
        for (int w = 0; w < kListThreads / 32; ++w) {
            const unsigned v = sums[w];
            sums[w] = all;
            all += v;
        }
        base = all ? atomicAdd(&p.sc->listed, all) : 0u;
    }
    __syncthreads();
    at += base + sums[warp] - found;
#pragma unroll
    for (int k = 0; k < kListPer; ++k)
        if (code[k] != ~0u)
            p.list[at++] = list_entry(I, o0 + k * kListThreads, code[k]);
}

__device__ __forceinline__ float rsqrt_approx(float s)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(s));
    return r;
}

// What every pair needs, in registers: limits and the bin quotient's constants.
struct CellBins {
    f2 inv, off, magic;
    float s_lo, s_hi;
    float slack;             // the fast bin holds where |fraction - 0.5| < slack
    unsigned limit;          // bytes of a histogram in global memory, 0: in shared memory
    unsigned spare;          // shared-memory address of the lane's spare counter
    __device__ CellBins(const CellHist &p, unsigned shaddr) : inv(dup2(p.inv)), off(dup2(p.off)), magic(dup2(kMagic))
    {
        s_lo = p.s_lo;
        s_hi = p.s_hi;
        slack = p.walk.sc->bad ? -1.0f : p.slack;
        limit = p.smem_hist ? 0u : 4u * p.total;
        spare = shaddr + 4u * (p.total + 1u + (threadIdx.x & 31u));
    }
};

// The pairs that the fast path leaves: the IEEE root and quotient, counts of
// atoms of one molecule and checked offsets.  j: the column's sorted index.
__device__ __noinline__ void bin_exact(const CellHist &p, float s, int i, int j, unsigned *shist)
{
    const int4 row = p.walk.meta[i], col = p.walk.meta[j];
    const unsigned flat =
        (unsigned)(row.w < col.w ? row.x + col.y : col.x + row.y) + (unsigned)pair_bin(s, p.minD, p.binw);
    if (flat < p.total) {
        if (row.z == col.z)
            atomicAdd(p.intra + flat, 1u);
        else if (shist)
            atomicAdd(shist + flat, 1u);
        else
            atomicAdd(p.inter + flat, 1u);
    }
}

// Counts four columns' pairs (squared distances s, two and two) with one row
// atom per lane.  A quotient from rsqrt.approx (2^-22.9) differs from the
// reference's by less than a known bound, so where it is further than that
// from an integer its floor is the bin; the others (0.2 % of the pairs at
// 2,000 bins) and pairs of one molecule go through bin_exact.  IN: every pair
// is in range (but NaNs), so where all of the warp's bins hold there is nothing
// to select.  Offsets in
// `row` and `meta` are in bytes and count from `shaddr` and 2^23's bits.
template <bool LO, bool IN>
__device__ __forceinline__ void bin_quad(const CellHist &p, const CellBins &k, f2 s01, f2 s23, const CellRow &row,
                                         const int4 *meta, int j0, unsigned *shist, f2 nz)
{
    const float s[4] = {lo2(s01), hi2(s01), lo2(s23), hi2(s23)};
    bool in[4];
    if (!IN) {
#pragma unroll
        for (int h = 0; h < 4; ++h) in[h] = (!LO || s[h] >= k.s_lo) && s[h] < k.s_hi;  // s >= 0 or NaN
        if (!__any_sync(0xffffffffu, in[0] || in[1] || in[2] || in[3]))
            return;
    }
    bool sure[4];
    unsigned at[4];
#pragma unroll
    for (int h = 0; h < 4; h += 2) {
        const f2 d = mul2(h ? s23 : s01, pack2(rsqrt_approx(s[h]), rsqrt_approx(s[h + 1])), nz);
        const f2 t = fma2(d, k.inv, k.off);            // quotient + 1
        const f2 r = add2_down(t, k.magic);            // 2^23 + floor
        // fraction - 0.5: t - (floor + 0.5), every step exact
        const f2 u = fma2(add2(r, dup2(0.5f - kMagic)), dup2(-1.0f), t);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const int4 col = meta[h + g];
            at[h + g] = (4u * __float_as_uint(g ? hi2(r) : lo2(r)) + row.meta.y) + col.y +
                        (row.meta.w < col.w ? row.meta.x : col.x);
            sure[h + g] = fabsf(g ? hi2(u) : lo2(u)) < k.slack && row.meta.z != col.z;
        }
    }
    if (IN) {
        if (__all_sync(0xffffffffu, sure[0] && sure[1] && sure[2] && sure[3])) {
#pragma unroll
            for (int h = 0; h < 4; ++h) asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(at[h]) : "memory");
            return;
        }
#pragma unroll
        for (int h = 0; h < 4; ++h) in[h] = s[h] < k.s_hi;  // not a NaN
    }
    bool fast[4], rare = false;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        fast[h] = in[h] && sure[h];
        rare |= in[h] && !fast[h];
    }
    if (k.limit == 0u) {
        // the other lanes add to a spare counter: a predicated shared-memory
        // atomic compiles to a branch around it (three more issue slots)
#pragma unroll
        for (int h = 0; h < 4; ++h)
            asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(fast[h] ? at[h] : k.spare) : "memory");
    } else {
#pragma unroll
        for (int h = 0; h < 4; ++h)
            if (fast[h] && at[h] < k.limit)
                atomicAdd(p.inter + at[h] / 4u, 1u);
    }
    if (__any_sync(0xffffffffu, rare)) {
        unsigned left = 0u;
#pragma unroll
        for (int h = 0; h < 4; ++h) left |= in[h] && !fast[h] ? 1u << h : 0u;
        while (left) {
            const int h = __ffs(left) - 1;
            left &= left - 1;
            bin_exact(p, h < 2 ? (h ? s[1] : s[0]) : (h == 2 ? s[2] : s[3]), row.index, j0 + h, shist);
        }
    }
}

template <int BM, bool LO>
__global__ void __launch_bounds__(kCellThreads, 1) k_cell_hist(CellHist p)
{
    grid_dependency_wait();
    grid_launch_dependents();
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x;
    unsigned *shist = nullptr;
    if (p.smem_hist) {
        shist = reinterpret_cast<unsigned *>(smem + kCellThreads / 32 * sizeof(CellStage));
        for (unsigned k = tid; k < p.total; k += kCellThreads) shist[k] = 0u;
        __syncthreads();
    }
    // byte offsets of a row: from the counters, less 2^23 and the quotient's 1
    const unsigned rowbase = (shist ? smem_addr(shist) : 0u) - 4u * (kMagicBits + 1u);
    const CellBins bins(p, shist ? smem_addr(shist) : 0u);
    const f2 nz = dup2(p.walk.negzero);
    walk_blocks<BM, true>(
        p.walk, reinterpret_cast<CellStage *>(smem)[tid >> 5],
        [&](const int4 &m, bool row) {
            // (el (ne - 1) hs, el hs): a pair's offset is the sum of both
            // second terms and the first of the atom with the smaller index
            return make_int4(4 * (m.x - m.y), (int)(4u * m.y + (row ? rowbase : 0u)), m.z, m.w);
        },
        [&](f2 s01, f2 s23, const CellRow &row, const int4 *meta, int j0, auto in) {
            bin_quad<LO, decltype(in)::value>(p, bins, s01, s23, row, meta, j0, shist, nz);
        });
    __syncthreads();
    if (shist)
        for (unsigned k = tid; k < p.total; k += kCellThreads) {
            const unsigned v = shist[k];
            if (v)
                atomicAdd(p.inter + k, v);
        }
}

// ================================================================ launchers
static size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }

// Smallest |b w|-like widths of the box: w_k = 1 / |column k of B^-1|
// (|real| >= |g_k| w_k, g = real B^-1).  False for a singular basis.
static bool box_widths(const float *b, float w[3], double *volume)
{
    double B[9];
    for (int k = 0; k < 9; ++k) B[k] = b[k];
    const double c[9] = {B[4] * B[8] - B[5] * B[7], B[2] * B[7] - B[1] * B[8], B[1] * B[5] - B[2] * B[4],
                         B[5] * B[6] - B[3] * B[8], B[0] * B[8] - B[2] * B[6], B[2] * B[3] - B[0] * B[5],
                         B[3] * B[7] - B[4] * B[6], B[1] * B[6] - B[0] * B[7], B[0] * B[4] - B[1] * B[3]};
    const double det = B[0] * c[0] + B[1] * c[3] + B[2] * c[6];
    *volume = std::fabs(det);
    if (!(*volume > 0.0) || !std::isfinite(*volume))
        return false;
    for (int k = 0; k < 3; ++k)
        w[k] = (float)(*volume / std::sqrt(c[k] * c[k] + c[3 + k] * c[3 + k] + c[6 + k] * c[6 + k]));
    return true;
}

// Largest bin a pair in range can take (the reference's float32 quotient).
static long long largest_bin(float s_hi, float minD, float binw)
{
    const float d = std::sqrt(std::nextafterf(s_hi, 0.0f));
    const float t = d - minD;
    const float v = t / binw;
    return v >= 0.0f && v < 1e9f ? (long long)v : -1;
}

bool cell_walk_applies(long long n, int bm, const Basis &B, float reach)
{
    float w[3];
    double vol;
    return n >= 2 && n <= (1ll << 24) && reach > 0.0f && std::isfinite(reach) &&
           (bm == BM_IBC || box_widths(B.b, w, &vol));
}

bool cell_hist_applies(long long n, int bm, const Basis &B, float minD, float maxD, float binw, int ne, int hs)
{
    float s_lo, s_hi;
    const long long total = (long long)ne * ne * hs;
    if (!cell_walk_applies(n, bm, B, maxD) || !std::isfinite(minD))
        return false;
    sq_limits(minD, maxD, &s_lo, &s_hi);
    if (!(s_hi > 0.0f) || !std::isfinite(s_hi))
        return false;
    const long long top = largest_bin(s_hi, minD, binw);
    return top >= 0 && top < (1ll << 22) && top <= total;
}

size_t cell_hist_scratch(int n, size_t zeroed)
{
    const size_t nb = (size_t)(n + kCellBlock - 1) / kCellBlock, np = nb * kCellBlock, half = nb / 2 + 1;
    return up256(8 * std::min(nb, (size_t)kCellList / half) * half) + 256 + up256(4 * (size_t)kCellCap) + up256(zeroed) + up256(8 * (size_t)n) + 3 * up256(4 * np) +
           up256(16 * np) + up256(48 * (np / kCellBlock)) + up256(16 * (size_t)n) + up256(4 * (size_t)n);
}

int sort_cells(int sms, const float *coords, const float4 *atoms4, const int *el, const int *mol, int n, int bm,
               const Basis &B, float reach, int ne, int hs, void *scratch, CellWalk *walk, cudaStream_t st,
               size_t zeroed, void **zero)
{
    CellSort c{};
    c.coords = coords;
    c.el = el;
    c.src_mol = mol;
    c.n = n;
    c.nb = (n + kCellBlock - 1) / kCellBlock;
    c.ne = ne;
    c.hs = hs;
    c.pbc = bm != BM_IBC;
    c.B = B;
    CellWalk &h = *walk;
    h = CellWalk{};
    h.B = B;
    h.negzero = -0.0f;
    h.w[0] = h.w[1] = h.w[2] = 1.0f;
    double scale = 1.0;
    if (c.pbc) {
        if (!box_widths(B.b, h.w, &c.volume))
            return set_error(FRMC_E_ARG, "sorted pairs: singular basis");
        scale = 0.0;
        for (int k = 0; k < 9; ++k) scale += std::fabs((double)B.b[k]);
    }
    // margin: float32 positions are off by a few 1e-7 of |coordinate| |B|
    h.reach0 = (float)((double)reach * 1.0001 + 1e-5 * scale);
    h.reach1 = (float)(1e-5 * scale);
    unsigned char *at = static_cast<unsigned char *>(scratch);
    auto take = [&](size_t bytes) {
        unsigned char *r = at;
        at += up256(bytes);
        return r;
    };
    const size_t np = (size_t)c.nb * kCellBlock;
    c.sc = reinterpret_cast<CellScalars *>(take(sizeof(CellScalars)));
    c.cells = reinterpret_cast<int *>(take(4 * (size_t)kCellCap));
    unsigned char *extra = take(zeroed);
    if (zero)
        *zero = extra;
    c.place = reinterpret_cast<int2 *>(take(8 * (size_t)n));
    c.x = reinterpret_cast<float *>(take(4 * np));
    c.y = reinterpret_cast<float *>(take(4 * np));
    c.z = reinterpret_cast<float *>(take(4 * np));
    c.meta = reinterpret_cast<int4 *>(take(16 * np));
    c.bounds = reinterpret_cast<float4 *>(take(48 * (size_t)c.nb));
    c.atoms4 = reinterpret_cast<float4 *>(take(16 * (size_t)n));
    c.mol = reinterpret_cast<int *>(take(4 * (size_t)n));
    if (!coords) {  // packed already; read only
        c.atoms4 = const_cast<float4 *>(atoms4);
        c.mol = const_cast<int *>(mol);
    }
    h.nb = c.nb;
    h.x = c.x;
    h.y = c.y;
    h.z = c.z;
    h.meta = c.meta;
    h.bounds = c.bounds;
    h.sc = c.sc;
    h.half = c.nb / 2 + 1;
    h.rows = (int)std::min<long long>(c.nb, kCellList / h.half);
    h.list = reinterpret_cast<unsigned long long *>(take(8 * (size_t)h.rows * h.half));

    // scalars, cell counts and what the caller wants zero
    FRMC_CUDA(cudaMemsetAsync(scratch, 0, 256 + 4 * (size_t)kCellCap + zeroed, st));
    k_cell_bounds<<<std::min((n + 255) / 256, sms), 256, 0, st>>>(c);
    FRMC_CUDA(cudaGetLastError());
    FRMC_TRY(launch_after(k_cell_count, (n + 255) / 256, 256, 0, st, c));
    FRMC_TRY(launch_after(k_cell_scan, 1, 1024, 0, st, c.cells, c.sc, 0));
    FRMC_TRY(launch_after(k_cell_scatter, (int)((np + 255) / 256), 256, 0, st, c));
    return launch_after(k_cell_blocks, (c.nb * 32 + 255) / 256, 256, 0, st, c);
}

int launch_cell_scan(int *counts, int n, cudaStream_t st)
{
    return launch_after(k_cell_scan, 1, 1024, 0, st, counts, (CellScalars *)nullptr, n);
}

int launch_cell_list(const CellWalk &w, int bm, cudaStream_t st)
{
    const dim3 grid(w.rows, (w.half + kListThreads * kListPer - 1) / (kListThreads * kListPer));
    return bm == BM_IBC ? launch_after(k_cell_list<BM_IBC>, grid, kListThreads, 0, st, w)
                        : launch_after(k_cell_list<BM_GENERAL>, grid, kListThreads, 0, st, w);
}

template <int BM>
static int launch_cell_hist_bm(const CellHist &p, int grid, size_t smem, int max_smem, cudaStream_t st)
{
    auto kern = p.s_lo > 0.0f ? k_cell_hist<BM, true> : k_cell_hist<BM, false>;
    // the limit, not this launch's size: another thread's launch may come between
    FRMC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem));
    return launch_after(kern, grid, kCellThreads, smem, st, p);
}

int launch_cell_hist(int sms, int max_smem_optin, const float *coords, const float4 *atoms4, const int *el,
                     const int *mol, int n, int bm, const Basis &B, float minD, float maxD, float binw, int ne, int hs,
                     unsigned *intra, unsigned *inter, void *scratch, cudaStream_t st)
{
    CellHist h{};
    FRMC_TRY(sort_cells(sms, coords, atoms4, el, mol, n, bm, B, maxD, ne, hs, scratch, &h.walk, st, 0, nullptr));
    sq_limits(minD, maxD, &h.s_lo, &h.s_hi);
    h.minD = minD;
    h.binw = binw;
    // relative errors: rsqrt.approx 2^-22.9, its product, 1 / bin and the fma
    // 2^-24 each, the reference's square root, difference and quotient 2^-24
    // each: 4.9e-7 of (d + |min|) / bin in all
    // (the quotient is taken one higher, so that it is never negative)
    h.inv = 1.0f / binw;
    h.off = 1.0f - minD * h.inv;
    h.slack = 0.5f - (5e-7f * (maxD + std::fabs(minD)) * std::fabs(h.inv) + 1e-6f);
    if (largest_bin(h.s_hi, minD, binw) > hs)
        h.slack = -1.0f;  // offsets past the histogram are possible: bin_exact checks them
    h.total = (unsigned)((long long)ne * ne * hs);
    h.intra = intra;
    h.inter = inter;
    const size_t stage = kCellThreads / 32 * sizeof(CellStage);
    const size_t hist = 4 * ((size_t)h.total + 33);  // + bin hs of the last row, 32 spare counters
    h.smem_hist = stage + hist <= (size_t)max_smem_optin;
    const size_t smem = stage + (h.smem_hist ? hist : 0);
    // the walk's margins on both limits (reach0 is maxD and its own)
    const float own = h.walk.reach0 - maxD;
    h.walk.in0 = h.smem_hist ? maxD - own : -1.0f;
    h.walk.from0 = h.s_lo > 0.0f ? minD + own : -1.0f;
    return walk_lists(sms, h.walk, bm, st, [&](int grid) {
        switch (bm) {
        case BM_IBC: return launch_cell_hist_bm<BM_IBC>(h, grid, smem, max_smem_optin, st);
        case BM_DIAG: return launch_cell_hist_bm<BM_DIAG>(h, grid, smem, max_smem_optin, st);
        case BM_XYTRI: return launch_cell_hist_bm<BM_XYTRI>(h, grid, smem, max_smem_optin, st);
        case BM_LOWER: return launch_cell_hist_bm<BM_LOWER>(h, grid, smem, max_smem_optin, st);
        default: return launch_cell_hist_bm<BM_GENERAL>(h, grid, smem, max_smem_optin, st);
        }
    });
}

}  // namespace frmc
