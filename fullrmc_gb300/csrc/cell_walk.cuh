// The walk over pairs of spatially sorted atoms within a reach: a warp takes runs
// of a list of block pairs (k_cell_list tests and lists them), holds one atom of
// the row block per lane and hands the squared distances of the column block's
// atoms to the caller four columns at a time.  cell_pairs.cu sorts the atoms and
// says what makes the test exact.
#pragma once
#include <cstdint>
#include <type_traits>

#include "frmc_math.cuh"
#include "frmc_runtime.h"

namespace frmc {

constexpr int kCellBlock = 32;        // atoms of a block: one per lane
constexpr int kCellThreads = 768;

// Range of the positions as ordered unsigned bits, the largest coordinate
// magnitude and the work counter; zeroed (lo: inverted) by k_cell_bounds' memset.
struct CellScalars {
    unsigned nlo[3];   // ~ordered(lo): an atomicMax from zero
    unsigned hi[3];
    unsigned amax;     // bits of max |coordinate|
    unsigned next;     // entries of the list claimed after each warp's first
    unsigned listed;   // entries of the list
    int ncells;        // cells of the sort
    unsigned bad;      // an element index is outside the histogram
    unsigned strange;  // a coordinate is not finite
};

// What the walk over block pairs needs (walk_blocks).
struct CellWalk {
    int nb, half;            // blocks; offsets of a row block's columns: 0 .. half - 1
    int i0, rows;            // the list holds the pairs of `rows` row blocks from i0 at a time
    unsigned long long *list;
    const float *x, *y, *z;
    const int4 *meta;
    const float4 *bounds;
    CellScalars *sc;
    Basis B;
    float w[3];              // perpendicular widths of the box
    float reach0, reach1;    // reach = reach0 + reach1 * max |coordinate|
    float in0, from0;        // distances of block pairs wholly in range: past from0 + reach1 * max, up to in0 less
                             // that (in0 < 0: none)
    float negzero;           // -0 (mul2)
};

// Whether the walk can find the pairs of n atoms within `reach`.
bool cell_walk_applies(long long n, int bm, const Basis &B, float reach);
// Sorts the atoms on `st` into `scratch` (cell_hist_scratch(n, zeroed) bytes,
// its first 256 the CellScalars) and fills the walk over their pairs within
// `reach`.  The atoms come as three arrays (device memory, or host memory that
// the device reads) or packed with their molecules.  An atom's meta is
// (el * ne * hs, el * hs, molecule, index).  `zeroed` bytes at *zero start as 0.
int sort_cells(int sms, const float *coords, const float4 *atoms4, const int *el, const int *mol, int n, int bm,
               const Basis &B, float reach, int ne, int hs, void *scratch, CellWalk *walk, cudaStream_t st,
               size_t zeroed, void **zero);
// Lists the block pairs of w.rows row blocks from w.i0 that can hold a pair
// within reach.
int launch_cell_list(const CellWalk &w, int bm, cudaStream_t st);
// Runs launch(CTAs of kCellThreads) after each list of row blocks.
template <class Launch>
int walk_lists(int sms, CellWalk &w, int bm, cudaStream_t st, const Launch &launch)
{
    const int rows = w.rows;
    const long long tests = (long long)rows * w.half;
    const int grid = (int)(tests < sms * (kCellThreads / 32ll) ? (tests + kCellThreads / 32 - 1) / (kCellThreads / 32) : sms);
    for (w.i0 = 0; w.i0 < w.nb; w.i0 += rows) {
        w.rows = w.nb - w.i0 < rows ? w.nb - w.i0 : rows;
        if (w.i0)
            FRMC_CUDA(cudaMemsetAsync(&w.sc->next, 0, 2 * sizeof(unsigned), st));
        FRMC_TRY(launch_cell_list(w, bm, st));
        FRMC_TRY(launch(grid));
    }
    return FRMC_OK;
}
// Exclusive scan in place of n counts, zero up to the next multiple of 4,096.
int launch_cell_scan(int *counts, int n, cudaStream_t st);

// ------------------------------------------------------------ float32 pairs
typedef unsigned long long f2;  // two float32 in one 64-bit register

__device__ __forceinline__ f2 dup2(float v)
{
    const unsigned u = __float_as_uint(v);
    return (f2)u << 32 | u;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b)
{
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// a b, rounded once.  ptxas contracts mul.rn.f32x2 and add.rn.f32x2 into one
// fma.rn.f32x2 (unlike the scalar forms, whose .rn keeps them apart), which
// would change the last bit of a distance.  So a product is an fma that adds
// nz = -0, which is exact for every product (x + -0 = x, also for x = +-0),
// and nz comes from the kernel's parameters, so it is no constant to fold.
__device__ __forceinline__ f2 mul2(f2 a, f2 b, f2 nz)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(nz));
    return r;
}

// The basis terms that pair_s<BM> keeps, duplicated for f32x2, and -0.
template <int BM>
struct Basis2 {
    f2 b[BM == BM_IBC ? 1 : 9], nz;
    __device__ Basis2(const Basis &B, float negzero)
    {
        if (BM != BM_IBC)
#pragma unroll
            for (int k = 0; k < 9; ++k) b[k] = dup2(B.b[k]);
        nz = dup2(negzero);
    }
};

// Squared distances of two pairs from their wrapped box differences, in the
// operation order of pair_s<BM>.
template <int BM>
__device__ __forceinline__ f2 square2(f2 dx, f2 dy, f2 dz, const Basis2<BM> &B)
{
    f2 x = dx, y = dy, z = dz;
    if (BM == BM_DIAG) {
        x = mul2(dx, B.b[0], B.nz);
        y = mul2(dy, B.b[4], B.nz);
        z = mul2(dz, B.b[8], B.nz);
    } else if (BM == BM_XYTRI) {
        x = add2(mul2(dx, B.b[0], B.nz), mul2(dy, B.b[3], B.nz));
        y = mul2(dy, B.b[4], B.nz);
        z = mul2(dz, B.b[8], B.nz);
    } else if (BM == BM_LOWER) {
        x = add2(add2(mul2(dx, B.b[0], B.nz), mul2(dy, B.b[3], B.nz)), mul2(dz, B.b[6], B.nz));
        y = add2(mul2(dy, B.b[4], B.nz), mul2(dz, B.b[7], B.nz));
        z = mul2(dz, B.b[8], B.nz);
    } else if (BM == BM_GENERAL) {
        x = add2(add2(mul2(dx, B.b[0], B.nz), mul2(dy, B.b[3], B.nz)), mul2(dz, B.b[6], B.nz));
        y = add2(add2(mul2(dx, B.b[1], B.nz), mul2(dy, B.b[4], B.nz)), mul2(dz, B.b[7], B.nz));
        z = add2(add2(mul2(dx, B.b[2], B.nz), mul2(dy, B.b[5], B.nz)), mul2(dz, B.b[8], B.nz));
    }
    return add2(add2(mul2(x, x, B.nz), mul2(y, y, B.nz)), mul2(z, z, B.nz));
}

// round() of one difference as pair_s takes it.
__device__ __forceinline__ float round_ref(float d)
{
    return truncf(__fadd_rn(d, copysignf(0.5f, d)));
}

__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 pack2(float a, float b)
{
    return (f2)__float_as_uint(b) << 32 | __float_as_uint(a);
}
__device__ __forceinline__ float lo2(f2 a) { return __uint_as_float((unsigned)a); }
__device__ __forceinline__ float hi2(f2 a) { return __uint_as_float((unsigned)(a >> 32)); }

// One warp's column block in shared memory: x, y, z negated, and the atoms'
// histogram offsets, molecule and original index.
struct __align__(16) CellStage {
    float x[kCellBlock], y[kCellBlock], z[kCellBlock];
    int4 meta[kCellBlock];
};

// A row atom: sorted index, position, histogram offsets, molecule and original index.
struct CellRow {
    int index;
    float x, y, z;
    int4 meta;
};

constexpr float kMagic = 8388608.0f;           // 2^23: t + 2^23 rounded down is 2^23 + floor(t), 0 <= t < 2^22
constexpr unsigned kMagicBits = 0x4b000000u;

__device__ __forceinline__ f2 add2_down(f2 a, f2 b)
{
    f2 r;
    asm("add.rz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// The minimum image of two differences: x - trunc(x + copysign(0.5, x)) with
// the sign set aside and the truncation by adding 2^23 rounded down, exact
// for |x| < 2^22 (FRND runs on the quarter-rate pipe).
__device__ __forceinline__ f2 wrap2(f2 x, f2 magic)
{
    const f2 sign = 0x8000000080000000ull;
    const f2 a = x & ~sign;
    const f2 n = add2(add2_down(add2(a, dup2(0.5f)), magic), dup2(-kMagic));
    return fma2(n, dup2(-1.0f), a) ^ (x & sign);
}

// What two blocks need for the pairs' minimum image.
enum CellWrap : int {
    CW_NONE = 0,   // every image shift is 0
    CW_SHIFT = 1,  // one constant shift
    CW_WRAP = 2,   // the whole minimum image
    CW_FAR = 3,    // the same for coordinates beyond wrap2's range
};

// One lane's row atom against the 32 staged columns (sorted indexes from j0).
// CW_WRAP and CW_FAR take only the columns past `after` (a block against
// itself: past the lane's own).
// `quad` gets the squared distances of four columns, two and two, and whether
// (IN) every pair of the blocks without a NaN is known to be in range.
template <int BM, int WRAP, bool IN, class Quad>
__device__ __forceinline__ void block_pairs(const CellWalk &p, const CellStage &c, const CellRow &row, const float *sh,
                                            const Basis2<BM> &B2, int j0, int after, const Quad &quad)
{
    const f2 magic = dup2(kMagic);
    const f2 rx2 = dup2(row.x), ry2 = dup2(row.y), rz2 = dup2(row.z);
    const f2 kx = dup2(-sh[0]), ky = dup2(-sh[1]), kz = dup2(-sh[2]);
    // the short body of blocks in range pays for its loop (4.54 -> 4.10 ms of
    // the particle's call; 2: 4.37, 8: 4.09), the longer one does not
#pragma unroll(IN ? 4 : 1)
    for (int g = 0; g < kCellBlock; g += 4) {
        f2 s[2];
        if (WRAP != CW_FAR) {
            const ulonglong2 X = *reinterpret_cast<const ulonglong2 *>(c.x + g);
            const ulonglong2 Y = *reinterpret_cast<const ulonglong2 *>(c.y + g);
            const ulonglong2 Z = *reinterpret_cast<const ulonglong2 *>(c.z + g);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                f2 dx = add2(rx2, h ? X.y : X.x), dy = add2(ry2, h ? Y.y : Y.x), dz = add2(rz2, h ? Z.y : Z.x);
                if (WRAP == CW_SHIFT) {
                    dx = add2(dx, kx);
                    dy = add2(dy, ky);
                    dz = add2(dz, kz);
                } else if (WRAP == CW_WRAP && BM != BM_IBC) {
                    dx = wrap2(dx, magic);
                    dy = wrap2(dy, magic);
                    dz = wrap2(dz, magic);
                }
                s[h] = square2<BM>(dx, dy, dz, B2);
            }
        } else {
#pragma unroll
            for (int h = 0; h < 2; ++h)
                s[h] = pack2(pair_s<BM>(row.x, row.y, row.z, -c.x[g + 2 * h], -c.y[g + 2 * h], -c.z[g + 2 * h], p.B),
                             pair_s<BM>(row.x, row.y, row.z, -c.x[g + 2 * h + 1], -c.y[g + 2 * h + 1],
                                        -c.z[g + 2 * h + 1], p.B));
        }
        if (WRAP >= CW_WRAP)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                s[h] = pack2(g + 2 * h > after ? lo2(s[h]) : INFINITY, g + 2 * h + 1 > after ? hi2(s[h]) : INFINITY);
        quad(s[0], s[1], row, c.meta + g, j0 + g, std::integral_constant<bool, IN>());
    }
}

struct BlockBox {
    float lo[3], hi[3], rlo[3], rhi[3];
};

__device__ __forceinline__ BlockBox block_box(const float4 *bounds, int b)
{
    const float4 u = bounds[3 * b], v = bounds[3 * b + 1], w = bounds[3 * b + 2];
    BlockBox r;
    r.lo[0] = u.x; r.lo[1] = u.y; r.lo[2] = u.z; r.hi[0] = u.w;
    r.hi[1] = v.x; r.hi[2] = v.y; r.rlo[0] = v.z; r.rlo[1] = v.w;
    r.rlo[2] = w.x; r.rhi[0] = w.y; r.rhi[1] = w.z; r.rhi[2] = w.w;
    return r;
}

constexpr int kBlockIn = 4;  // or-ed to CW_NONE and CW_SHIFT where every pair is in range

// The CellWrap of two blocks (`pack`: the shift of CW_SHIFT as three int8), or
// -1 where every pair is out of range.
template <int BM>
__device__ __forceinline__ int block_test(const CellWalk &p, const BlockBox &a, const BlockBox &b, float reach,
                                          unsigned &pack)
{
    pack = 0u;
    float k[3] = {0.f, 0.f, 0.f};
    bool same = true, near = true;
    if (BM != BM_IBC) {
        bool far = false;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const float lo = __fsub_rn(a.lo[d], b.hi[d]), hi = __fsub_rn(a.hi[d], b.lo[d]);
            const float k0 = round_ref(lo), k1 = round_ref(hi);
            same &= k0 == k1 && fabsf(k0) < 100.f;
            near &= lo > -4e6f && hi < 4e6f;
            k[d] = k0;
            // smallest |g| over the interval: 0 where it holds an integer
            const float n = floorf(hi);
            const float m = n >= lo ? 0.f : fminf(lo - n, n + 1.f - hi);
            far |= m * p.w[d] > reach;
        }
        if (far)
            return -1;
        if (!same)
            return near ? CW_WRAP : CW_FAR;
    }
    float gap2 = 0.f, far2 = 0.f;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float t = BM == BM_IBC ? 0.f : k[0] * p.B.b[d] + k[1] * p.B.b[3 + d] + k[2] * p.B.b[6 + d];
        const float lo = a.rlo[d] - b.rhi[d] - t, hi = a.rhi[d] - b.rlo[d] - t;
        const float gap = fmaxf(0.f, fmaxf(lo, -hi));
        gap2 += gap * gap;
        const float far = fmaxf(-lo, hi);
        far2 += far * far;
    }
    if (gap2 > reach * reach)
        return -1;
    const float margin = reach - p.reach0, top = p.in0 - margin, from = p.from0 + margin;
    const int in = top > 0.f && far2 < top * top && (p.from0 < 0.f || gap2 > from * from) ? kBlockIn : 0;
    if (BM == BM_IBC)
        return CW_NONE | in;
    const int kx = (int)k[0], ky = (int)k[1], kz = (int)k[2];
    pack = (unsigned)(kx & 255) | (unsigned)(ky & 255) << 8 | (unsigned)(kz & 255) << 16;
    return (pack ? CW_SHIFT : CW_NONE) | in;
}

// Column block of offset o from row block I, or -1: each unordered pair of
// blocks belongs to one row block, and every row block gets half of the others.
__device__ __forceinline__ int column_block(int I, int o, int nb)
{
    if (2 * o > nb || (2 * o == nb && I >= o))
        return -1;
    const int J = I + o;
    return J < nb ? J : J - nb;
}

// An entry of the list: row block and offset of the column block (19 bits each),
// shift (24, of CW_SHIFT, never 0 there) and one of these.
enum ListKind : unsigned { LK_SAME = 0, LK_IN = 1, LK_WRAP = 2, LK_FAR = 3 };

__device__ __forceinline__ unsigned long long list_entry(int I, int o, unsigned code)
{
    return (unsigned long long)I << 45 | (unsigned long long)o << 26 | code;
}
__device__ __forceinline__ unsigned list_code(int what, unsigned pack)
{
    const unsigned kind = what == CW_FAR ? LK_FAR : what == CW_WRAP ? LK_WRAP : what & kBlockIn ? LK_IN : LK_SAME;
    return pack << 2 | kind;
}

// Walks the listed pairs of blocks, a warp per run of entries.  `prepare` turns
// an atom's meta into what `quad` expects of a row (true) and of a column.
// INNER: blocks wholly in range (p.in0) are told apart.
//
// The list is made by a kernel of its own (k_cell_list): with the tests in the
// walk, 32 offsets of a row block at a time, the last warps to hold a full test
// ended 65 us after the others (100,000 atoms, 605 us), and shorter items paid
// more for their tests than they gained (16 offsets 724 us a call, 32 692;
// with the list 634).
template <int BM, bool INNER = false, class Prepare, class Quad>
__device__ __forceinline__ void walk_blocks(const CellWalk &p, CellStage &stage, const Prepare &prepare,
                                            const Quad &quad)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Basis2<BM> B2(p.B, p.negzero);
    const unsigned listed = p.sc->listed;
    const unsigned nwarps = gridDim.x * (kCellThreads / 32);
    // about 16 runs per warp, so that the last ones end together (8: 642 us a call, 16: 634)
    const unsigned run = min(max(listed / (nwarps * 16u), 1u), 16u);

    // the next run is claimed while this one is evaluated
    unsigned next = (blockIdx.x * (kCellThreads / 32) + warp) * run;
    CellRow row;
    int I = -1;
    while (next < listed) {
        const unsigned first = next, count = min(run, listed - first);
        if (lane == 0)
            next = nwarps * run + atomicAdd(&p.sc->next, run);
        const unsigned long long mine = lane < (int)count ? p.list[first + lane] : 0ull;
        // the next block's columns are loaded while one is evaluated
        float nx = 0.f, ny = 0.f, nz = 0.f;
        int4 nm = make_int4(0, 0, 0, 0);
        int J = 0;
        unsigned long long e = 0ull;
        auto load = [&](unsigned k) {
            e = __shfl_sync(0xffffffffu, mine, k);
            J = (int)(e >> 45) + (int)(e >> 26 & 0x7ffffu);
            J = J < p.nb ? J : J - p.nb;
            const int c = J * kCellBlock + lane;
            nx = p.x[c];
            ny = p.y[c];
            nz = p.z[c];
            nm = p.meta[c];
        };
        load(0);
        for (unsigned k = 0; k < count; ++k) {
            const unsigned kind = (unsigned)e & 3u, pk = (unsigned)e >> 2 & 0xffffffu;
            const int row_block = (int)(e >> 45);
            const int j0 = J * kCellBlock;
            if (row_block != I) {
                I = row_block;
                const int i = row.index = I * kCellBlock + lane;
                row.x = -p.x[i];
                row.y = -p.y[i];
                row.z = -p.z[i];
                row.meta = prepare(p.meta[i], true);
            }
            const bool diag = J == I;
            __syncwarp();
            stage.x[lane] = nx;
            stage.y[lane] = ny;
            stage.z[lane] = nz;
            stage.meta[lane] = prepare(nm, false);
            __syncwarp();
            if (k + 1 < count)
                load(k + 1);
            const float sh[3] = {(float)(signed char)(pk & 255u), (float)(signed char)(pk >> 8 & 255u),
                                 (float)(signed char)(pk >> 16 & 255u)};
            const int after = diag ? lane : -1;
            if (kind == LK_FAR)
                block_pairs<BM, CW_FAR, false>(p, stage, row, sh, B2, j0, after, quad);
            else if (diag || kind == LK_WRAP)
                block_pairs<BM, CW_WRAP, false>(p, stage, row, sh, B2, j0, after, quad);
            else if (INNER && kind == LK_IN && !pk)
                block_pairs<BM, CW_NONE, INNER>(p, stage, row, sh, B2, j0, -1, quad);
            else if (INNER && kind == LK_IN)
                block_pairs<BM, CW_SHIFT, INNER>(p, stage, row, sh, B2, j0, -1, quad);
            else if (!pk)
                block_pairs<BM, CW_NONE, false>(p, stage, row, sh, B2, j0, -1, quad);
            else
                block_pairs<BM, CW_SHIFT, false>(p, stage, row, sh, B2, j0, -1, quad);
        }
        next = __shfl_sync(0xffffffffu, next, 0);
    }
}

}  // namespace frmc
