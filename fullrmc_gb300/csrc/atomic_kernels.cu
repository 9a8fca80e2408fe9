// Atomic distance constraints (Extensions/atomic_distances.pyx): for atom
// rows against every other atom, the pairs whose distance falls inside (or
// outside) per-element-pair limits are counted, and their distance -- or its
// difference to the nearest / upper / lower limit -- is summed, into
// [ne][ne] intra- and inter-molecular accumulators.
//
// The counts are integers and order-free, but the sums are float32 additions
// in the reference's loop order (rows in the order given, then columns in
// increasing index), and float32 addition is not associative.  So the pairs
// are evaluated in parallel and every contributing pair is listed in that
// order, then each accumulator adds its values in list order:
//   k_atomic_pairs<true>   one CTA per (row, chunk of kAtomicCols columns):
//                          the number of contributing pairs of its block;
//   k_scan_*               exclusive scan of those numbers (block offsets);
//   k_atomic_pairs<false>  the same blocks list their contributors, in column
//                          order, at their offsets;
//   k_atomic_sum           adds the list in order into the accumulators.
#include <cstdint>
#include <cstring>

#include "cell_walk.cuh"
#include "frmc_ptx.cuh"

namespace frmc {

constexpr int kAtomicThreads = 256;
constexpr int kAtomicPerThread = 4;
constexpr int kAtomicCols = kAtomicThreads * kAtomicPerThread;

enum AtomicFlags {
    AF_INTER = 1,
    AF_INTRA = 2,
    AF_WITHIN = 4,
    AF_RED_UPPER = 8,
    AF_RED_LOWER = 16,
    AF_RED = 32,
};

struct AtomicParams {
    const float *coords;  // (n, 3) box coordinates, or null when dists is given
    const float *dists;   // (n, K) distances, column k for row k (or null)
    const int *rows;      // (K,) atom index of each row
    int K, n, nchunks, allAtoms, flags, ne;
    Basis B;
    int bm;
    const int *mol, *el;
    const float *lower, *upper;  // (ne, ne) limits, indexed [el(column)][el(row)]
    long long *block_count;      // per (row, chunk): contributors, then their list offset
    int *list_bucket;            // contributors: (0 intra / 1 inter) * ne*ne + el(row) * ne + el(column)
    float *list_value;           // their values
};

// Whether a pair at distance d counts under its limits; d becomes what is
// summed (atomic_distances.pyx:100-126).
__device__ __forceinline__ bool contact_value(int flags, float lower, float upper, float &d)
{
    if (flags & AF_WITHIN) {
        if (d < lower || d >= upper)
            return false;
    } else if (d >= lower && d < upper) {
        return false;
    }
    if (flags & AF_RED_UPPER) {
        d = fabsf(__fsub_rn(upper, d));
    } else if (flags & AF_RED_LOWER) {
        d = fabsf(__fsub_rn(lower, d));
    } else if (flags & AF_RED) {
        d = d > __fdiv_rn(__fadd_rn(lower, upper), 2.0f) ? fabsf(__fsub_rn(upper, d)) : fabsf(__fsub_rn(lower, d));
    }
    return true;
}

template <int BM>
__device__ __forceinline__ bool atomic_pair(const AtomicParams &p, int ela, int mola, float ax, float ay, float az,
                                            int k, int j, float &value, int &bucket)
{
    const int molj = p.mol[j];
    const bool same = molj == mola;
    if (!(p.flags & AF_INTRA) && same)
        return false;
    if (!(p.flags & AF_INTER) && !same)
        return false;
    float d;
    if (p.dists) {
        d = p.dists[(long long)j * p.K + k];
    } else {
        const float *c = p.coords + 3ll * j;
        d = __fsqrt_rn(pair_s<BM>(ax, ay, az, c[0], c[1], c[2], p.B));
    }
    const int elj = p.el[j];
    if (!contact_value(p.flags, p.lower[elj * p.ne + ela], p.upper[elj * p.ne + ela], d))
        return false;
    value = d;
    bucket = (same ? 0 : p.ne * p.ne) + ela * p.ne + elj;
    return true;
}

template <int BM, bool COUNT>
__global__ void __launch_bounds__(kAtomicThreads) k_atomic_pairs(AtomicParams p)
{
    __shared__ int s_warp[kAtomicThreads / 32];
    const long long blk = blockIdx.x;
    const int k = (int)(blk / p.nchunks);
    const int chunk = (int)(blk % p.nchunks);
    const int a = p.rows[k];
    const int start = p.allAtoms ? 0 : a;
    const int j0 = chunk * kAtomicCols;
    const int ela = p.el[a], mola = p.mol[a];
    float ax = 0.f, ay = 0.f, az = 0.f;
    if (!p.dists) {
        ax = p.coords[3ll * a];
        ay = p.coords[3ll * a + 1];
        az = p.coords[3ll * a + 2];
    }
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    // each thread takes kAtomicPerThread consecutive columns, so the block's
    // column order is (thread, column) order
    bool hit[kAtomicPerThread];
    float val[kAtomicPerThread];
    int bkt[kAtomicPerThread];
    int mine = 0;
#pragma unroll
    for (int u = 0; u < kAtomicPerThread; ++u) {
        const int j = j0 + threadIdx.x * kAtomicPerThread + u;
        hit[u] = false;
        if (j < p.n && j >= start && j != a)
            hit[u] = atomic_pair<BM>(p, ela, mola, ax, ay, az, k, j, val[u], bkt[u]);
        mine += hit[u];
    }
    int incl = mine;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, off);
        if ((int)lane >= off)
            incl += v;
    }
    if (lane == 31)
        s_warp[warp] = incl;
    __syncthreads();
    int before = 0, total = 0;
    for (int w = 0; w < kAtomicThreads / 32; ++w) {
        const int c = s_warp[w];
        if (w < (int)warp)
            before += c;
        total += c;
    }
    if (COUNT) {
        if (threadIdx.x == 0)
            p.block_count[blk] = total;
        return;
    }
    long long pos = p.block_count[blk] + before + incl - mine;
#pragma unroll
    for (int u = 0; u < kAtomicPerThread; ++u)
        if (hit[u]) {
            p.list_bucket[pos] = bkt[u];
            p.list_value[pos] = val[u];
            ++pos;
        }
}

// Exclusive scan of v[0..n) in place (int64), three launches: each CTA of
// 1024 scans its segment and stores the segment total; one CTA scans the
// totals; the totals' prefix is added back.
__global__ void __launch_bounds__(1024) k_scan_segments(long long *v, long long n, long long *totals)
{
    __shared__ long long s[1024];
    const long long i = (long long)blockIdx.x * 1024 + threadIdx.x;
    const long long x = i < n ? v[i] : 0;
    s[threadIdx.x] = x;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
        const long long t = threadIdx.x >= (unsigned)off ? s[threadIdx.x - off] : 0;
        __syncthreads();
        s[threadIdx.x] += t;
        __syncthreads();
    }
    if (i < n)
        v[i] = s[threadIdx.x] - x;
    if (threadIdx.x == 1023)
        totals[blockIdx.x] = s[1023];
}

__global__ void __launch_bounds__(1024) k_scan_totals(long long *totals, long long m, long long *grand)
{
    __shared__ long long s[1024];
    __shared__ long long carry;
    if (threadIdx.x == 0)
        carry = 0;
    __syncthreads();
    for (long long c0 = 0; c0 < m; c0 += 1024) {
        const long long i = c0 + threadIdx.x;
        const long long x = i < m ? totals[i] : 0;
        s[threadIdx.x] = x;
        __syncthreads();
        for (int off = 1; off < 1024; off <<= 1) {
            const long long t = threadIdx.x >= (unsigned)off ? s[threadIdx.x - off] : 0;
            __syncthreads();
            s[threadIdx.x] += t;
            __syncthreads();
        }
        if (i < m)
            totals[i] = carry + s[threadIdx.x] - x;
        __syncthreads();
        if (threadIdx.x == 0)
            carry += s[1023];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        *grand = carry;
}

__global__ void k_scan_add(long long *v, long long n, const long long *totals)
{
    const long long i = (long long)blockIdx.x * 1024 + threadIdx.x;
    if (i < n)
        v[i] += totals[blockIdx.x];
}

// A list that did not fit its buffers, or atoms that the sorted walk does not
// list (coordinates that are not finite), leave the sums as they are.
struct ListGuard {
    const long long *length;     // null: always good
    long long cap;
    const unsigned *strange;
    __device__ bool closed() const { return length && (*length > cap || *strange != 0u); }
};

// The ordered float32 sum of one bucket (one CTA each): dsum[b] plus the
// bucket's values in list order, every addition rounded, and their number.
// dsum and nsum are (2, ne, ne) and start from the caller's values.
//
// A chain of float32 additions is not associative, but while the sum stays in
// one binade it is an integer sum: with u the sum's unit in the last place,
// M = s / u goes to M + x / u rounded to an integer, ties to even, so adding x
// >= 0 moves M by an amount that depends on M's parity alone (and on that only
// where x / u is exactly halfway).  Such steps are pairs (move of an even M,
// move of an odd M), and pairs compose associatively: a tile of the list is
// scanned in parallel.  Where M would reach 2^24 the thread that holds that
// element adds its own elements as floats, and the scan goes on from there in
// the next binade.  Sums that are not positive and finite (the start: 0) are
// added one by one until they are.
//
// Bound: latency of the tiles (a scan each) and of the passes of two scans, one
// per 4,096 values and one per binade.  A bucket's values, one entry in 18, are
// brought together first, so that a pass has one or few per thread.  43,000
// entries in 18 buckets: one warp adding the list through shared memory 3.93 ms
// (90 ns an entry), passes over tiles of the list 44 us, over the bucket's
// values 34 (2,000 entries 21 and 11 us).
constexpr int kSumThreads = 512;
constexpr int kSumPer = 8;
constexpr int kSumTile = kSumThreads * kSumPer;
constexpr int kSumFull = 1 << 24;

struct SumStep {
    int even, odd;  // move of an even and of an odd M (clamped to 2^25: past the binade)
};

__device__ __forceinline__ SumStep sum_then(SumStep a, SumStep b)
{
    SumStep r;
    r.even = min(a.even + (a.even & 1 ? b.odd : b.even), 2 * kSumFull);
    r.odd = min(a.odd + (a.odd & 1 ? b.even : b.odd), 2 * kSumFull);
    return r;
}

// Adding x in units of u: x / u = q (exact, a power of two apart).
__device__ __forceinline__ SumStep sum_step(float q)
{
    if (!(q >= 0.0f && q < (float)kSumFull))
        return SumStep{2 * kSumFull, 2 * kSumFull};  // NaN, negative or past the binade: added as a float
    const float f = floorf(q), h = q - f;
    const int n = (int)f;
    SumStep r;
    r.even = n + (h > 0.5f ? 1 : (h == 0.5f ? n & 1 : 0));
    r.odd = n + (h > 0.5f ? 1 : (h == 0.5f ? (n + 1) & 1 : 0));
    return r;
}

__device__ __forceinline__ SumStep sum_shfl_up(SumStep v, int o)
{
    return SumStep{__shfl_up_sync(0xffffffffu, v.even, o), __shfl_up_sync(0xffffffffu, v.odd, o)};
}

__global__ void __launch_bounds__(kSumThreads) k_atomic_sum(const int *__restrict__ list_bucket,
                                                            const float *__restrict__ list_value,
                                                            const long long *length, ListGuard guard, float *dsum,
                                                            int *nsum)
{
    __shared__ SumStep wtot[kSumThreads / 32];
    __shared__ int wcount[kSumThreads / 32];
    __shared__ float vals[2 * kSumTile];
    __shared__ float s_next;
    __shared__ int pos_next;
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (guard.closed())
        return;
    const long long len = *length;
    float s = dsum[b];
    int n = 0;
    // the next tile is loaded while one is sorted out
    int4 b0, b1;
    float4 v0, v1;
    auto load = [&](long long first) {
        if (first < len) {  // the lists are padded to a multiple of 8 entries
            b0 = *reinterpret_cast<const int4 *>(list_bucket + first);
            b1 = *reinterpret_cast<const int4 *>(list_bucket + first + 4);
            v0 = *reinterpret_cast<const float4 *>(list_value + first);
            v1 = *reinterpret_cast<const float4 *>(list_value + first + 4);
        }
    };
    load((long long)tid * kSumPer);
    long long base = 0;
    while (base < len) {
        // the bucket's values in list order, of as many tiles as surely fit
        int filled = 0;
        while (base < len && filled <= kSumTile) {
            const long long first = base + tid * kSumPer;
            const float v[kSumPer] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
            unsigned has = 0u;
            if (first < len) {
                const int bk[kSumPer] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
                for (int k = 0; k < kSumPer; ++k) has |= bk[k] == b && first + k < len ? 1u << k : 0u;
            }
            load(first + kSumTile);
            int at = __popc(has);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, at, o);
                at += lane >= o ? t : 0;
            }
            if (lane == 31)
                wcount[warp] = at;
            __syncthreads();
            int w = lane < kSumThreads / 32 ? wcount[lane] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, w, o);
                w += lane >= o ? t : 0;
            }
            at += filled - __popc(has) + (warp ? __shfl_sync(0xffffffffu, w, warp - 1) : 0);
            filled += __shfl_sync(0xffffffffu, w, 31);
#pragma unroll
            for (int k = 0; k < kSumPer; ++k)
                if (has >> k & 1u)
                    vals[at++] = v[k];
            base += kSumTile;
            __syncthreads();  // wcount is written again
        }
        n += filled;
        int pos = 0;
        while (pos < filled) {
            const unsigned bits = __float_as_uint(s);
            const int e = (int)(bits >> 23);  // > 254 where s < 0
            if (e > 30 && e < 220) {
                // this thread's values: per of them from first
                const int per = min((filled - pos + kSumThreads - 1) / kSumThreads, kSumPer), first = pos + tid * per;
                const int end = min(first + per, filled);
                const float scale = __uint_as_float((unsigned)(277 - e) << 23);  // 1 / u, u = 2^(e - 150)
                const int M = (int)((bits & 0x7fffffu) | 0x800000u);
                SumStep own{0, 0};
                for (int k = first; k < end; ++k) own = sum_then(own, sum_step(__fmul_rn(vals[k], scale)));
                SumStep incl = own;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const SumStep t = sum_shfl_up(incl, o);
                    if (lane >= o)
                        incl = sum_then(t, incl);
                }
                if (lane == 31)
                    wtot[warp] = incl;
                __syncthreads();
                // every warp scans the warp totals itself
                SumStep w = lane < kSumThreads / 32 ? wtot[lane] : SumStep{0, 0};
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const SumStep t = sum_shfl_up(w, o);
                    if (lane >= o)
                        w = sum_then(t, w);
                }
                SumStep before = sum_shfl_up(incl, 1);
                if (lane == 0)
                    before = SumStep{0, 0};
                const SumStep wb{__shfl_sync(0xffffffffu, w.even, warp ? warp - 1 : 0),
                                 __shfl_sync(0xffffffffu, w.odd, warp ? warp - 1 : 0)};
                if (warp)
                    before = sum_then(wb, before);
                const int all = M & 1 ? __shfl_sync(0xffffffffu, w.odd, 31) : __shfl_sync(0xffffffffu, w.even, 31);
                const int m0 = M + (M & 1 ? before.odd : before.even);
                const int m1 = m0 + (m0 & 1 ? own.odd : own.even);
                const float u = __uint_as_float((unsigned)(e - 23) << 23);
                if (M + all < kSumFull) {
                    if (tid == 0) {
                        s_next = __fmul_rn((float)(M + all), u);
                        pos_next = min(pos + per * kSumThreads, filled);
                    }
                } else if (m0 < kSumFull && m1 >= kSumFull) {  // one thread: the moves are not negative
                    float t = __fmul_rn((float)m0, u);
                    for (int k = first; k < end; ++k) t = __fadd_rn(t, vals[k]);
                    s_next = t;
                    pos_next = end;
                }
            } else if (tid == 0) {
                // some entries more than needed: the first binades are short
                float t = s;
                int k = pos;
                while (k < filled) {
                    t = __fadd_rn(t, vals[k++]);
                    const unsigned te = __float_as_uint(t) >> 23;
                    if (k - pos >= 64 && te > 30u && te < 220u)
                        break;
                }
                s_next = t;
                pos_next = k;
            }
            __syncthreads();
            s = s_next;
            pos = pos_next;
            __syncthreads();  // the shared state is written again
        }
    }
    if (tid == 0) {
        dsum[b] = s;
        nsum[b] += n;
    }
}

// pair_elements_stats (atomic_distances.pyx:632-672): for i < j, count
// [el(i)][el(j)] intra (same molecule) or inter.  One CTA per row i; lanes
// with the same counter are merged with __match_any_sync before the shared
// atomic, and each CTA adds its counts to the result once.
__global__ void __launch_bounds__(256) k_pair_stats(const int *el, const int *mol, int n, int ne, int *nintra,
                                                   int *ninter)
{
    extern __shared__ int cnt[];  // [2][ne][ne]
    const int total = 2 * ne * ne;
    for (int k = threadIdx.x; k < total; k += blockDim.x) cnt[k] = 0;
    __syncthreads();
    const int i = blockIdx.x;
    const int ei = el[i], mi = mol[i];
    const unsigned lane = threadIdx.x & 31u;
    for (int jb = i + 1; jb < n; jb += blockDim.x) {
        const int j = jb + threadIdx.x;
        const int off = j < n ? (mol[j] == mi ? 0 : ne * ne) + ei * ne + el[j] : -1;
        const unsigned same = __match_any_sync(0xffffffffu, off);
        if (off >= 0 && lane == (unsigned)(__ffs(same) - 1))
            atomicAdd(cnt + off, __popc(same));
    }
    __syncthreads();
    for (int k = threadIdx.x; k < total; k += blockDim.x) {
        const int v = cnt[k];
        if (v)
            atomicAdd((k < ne * ne ? nintra + k : ninter + (k - ne * ne)), v);
    }
}

// The whole pipeline for one call: lists the contributors (device buffers
// grown as needed) and adds them in order into dsum / nsum (device, (2, ne,
// ne), holding the starting values).
static int atomic_distances_device(AtomicParams p, DevBuf &counts, DevBuf &totals, DevBuf &list_b, DevBuf &list_v,
                                   float *dsum, int *nsum, cudaStream_t st)
{
    p.nchunks = (p.n + kAtomicCols - 1) / kAtomicCols;
    const long long nblocks = (long long)p.K * p.nchunks;
    if (nblocks <= 0)
        return FRMC_OK;
    if (nblocks > 0x7fffffffll)
        return set_error(FRMC_E_ARG, "atomic distances: too many rows x columns");
    if (p.ne > 16)
        return set_error(FRMC_E_ARG, "atomic distances: at most 16 elements");
    const long long nseg = (nblocks + 1023) / 1024;
    FRMC_TRY(counts.ensure(8 * (size_t)nblocks));
    FRMC_TRY(totals.ensure(8 * (size_t)(nseg + 1)));
    p.block_count = counts.as<long long>();
    const unsigned g = (unsigned)nblocks;
#define FRMC_ATOMIC_LAUNCH(C)                                                                                        \
    switch (p.bm) {                                                                                              \
    case BM_IBC: k_atomic_pairs<BM_IBC, C><<<g, kAtomicThreads, 0, st>>>(p); break;                            \
    case BM_DIAG: k_atomic_pairs<BM_DIAG, C><<<g, kAtomicThreads, 0, st>>>(p); break;                          \
    case BM_XYTRI: k_atomic_pairs<BM_XYTRI, C><<<g, kAtomicThreads, 0, st>>>(p); break;                        \
    case BM_LOWER: k_atomic_pairs<BM_LOWER, C><<<g, kAtomicThreads, 0, st>>>(p); break;                        \
    default: k_atomic_pairs<BM_GENERAL, C><<<g, kAtomicThreads, 0, st>>>(p); break;                            \
    }
    FRMC_ATOMIC_LAUNCH(true);
    FRMC_CUDA(cudaGetLastError());
    long long *tot = totals.as<long long>();
    k_scan_segments<<<(unsigned)nseg, 1024, 0, st>>>(p.block_count, nblocks, tot);
    k_scan_totals<<<1, 1024, 0, st>>>(tot, nseg, tot + nseg);
    k_scan_add<<<(unsigned)nseg, 1024, 0, st>>>(p.block_count, nblocks, tot);
    FRMC_CUDA(cudaGetLastError());
    long long len = 0;
    FRMC_CUDA(cudaMemcpyAsync(&len, tot + nseg, 8, cudaMemcpyDeviceToHost, st));
    FRMC_CUDA(cudaStreamSynchronize(st));
    if (len > 0) {
        FRMC_TRY(list_b.ensure(4 * (size_t)len + 4 * kSumPer));
        FRMC_TRY(list_v.ensure(4 * (size_t)len + 4 * kSumPer));
        p.list_bucket = list_b.as<int>();
        p.list_value = list_v.as<float>();
        FRMC_ATOMIC_LAUNCH(false);
        FRMC_CUDA(cudaGetLastError());
        k_atomic_sum<<<2 * p.ne * p.ne, kSumThreads, 0, st>>>(p.list_bucket, p.list_value, tot + nseg, ListGuard{},
                                                              dsum, nsum);
        FRMC_CUDA(cudaGetLastError());
    }
#undef FRMC_ATOMIC_LAUNCH
    return FRMC_OK;
}

// ------------------------------------------------ all pairs within a reach
// full_atomic_distances_coords counts contacts of a few Angstrom: 2 of the
// 10,000 columns a row of a 19,994-atom system meets.  With limits that bound
// the distance from above, the pairs come from the walk over sorted atoms
// (cell_walk.cuh) instead of from two passes over all of them:
//   k_contacts       lists the pairs i < j that count, in any order, with
//                    their rank among row i's;
//   launch_cell_scan the rows' places in the list;
//   k_contact_place  every entry to its row's part of the list;
//   k_contact_order  every entry to its place by column within the row.
// Measured: 19,994 atoms (43,000 contacts): two passes 1,814 us, the walk 44 us
// and its sort, scan and ordering 37 us; the whole call 2.07 -> 0.23 ms.
struct ContactParams {
    CellWalk walk;
    float s_hi;              // s < s_hi for every distance below the largest upper limit
    int flags, ne;
    const float *lower, *upper;
    long long *count;
    long long cap;
    int *row;                // contacts of row i, then their start
    int4 *hits, *placed;     // (i, j, bucket, value bits)
    int *rank;               // of hits[e] among its row's
    int *list_bucket;
    float *list_value;
};

// A warp's contacts wait in shared memory until there are 32 to write: one
// addition to the list's length for each hit serialises at its address (a
// system of 43,000 contacts took 72 us that way, 44 us this way).
constexpr int kContactQueue = 64;

struct ContactQueue {
    int4 hit[kContactQueue];
};

__device__ __forceinline__ void contact_flush(const ContactParams &p, ContactQueue &q, int &fill, int take)
{
    const int lane = threadIdx.x & 31;
    __syncwarp();
    long long at = 0;
    if (lane == 0)
        at = (long long)atomicAdd(reinterpret_cast<unsigned long long *>(p.count), (unsigned long long)take);
    at = __shfl_sync(0xffffffffu, at, 0) + lane;
    fill -= take;
    if (lane < take) {
        const int4 h = q.hit[fill + lane];
        const int rank = atomicAdd(p.row + h.x, 1);
        if (at < p.cap) {
            p.hits[at] = h;
            p.rank[at] = rank;
        }
    }
    __syncwarp();
}

template <int BM>
__global__ void __launch_bounds__(kCellThreads, 1) k_contacts(ContactParams p)
{
    grid_dependency_wait();
    grid_launch_dependents();
    __shared__ CellStage stage[kCellThreads / 32];
    __shared__ ContactQueue queue[kCellThreads / 32];
    ContactQueue &q = queue[threadIdx.x >> 5];
    const float s_hi = p.s_hi;
    const unsigned before = (1u << (threadIdx.x & 31)) - 1u;
    int fill = 0;
    walk_blocks<BM>(
        p.walk, stage[threadIdx.x >> 5], [](const int4 &m, bool) { return m; },
        [&](f2 s01, f2 s23, const CellRow &row, const int4 *meta, int, auto) {
            const float s[4] = {lo2(s01), hi2(s01), lo2(s23), hi2(s23)};
            unsigned in = 0u;
#pragma unroll
            for (int h = 0; h < 4; ++h) in |= s[h] < s_hi ? 1u << h : 0u;
            in = __reduce_or_sync(0xffffffffu, in);
            while (in) {
                const int h = __ffs(in) - 1;
                in &= in - 1;
                const float sh = h < 2 ? (h ? s[1] : s[0]) : (h == 2 ? s[2] : s[3]);
                // meta: (el * ne, el, molecule, original index); row i, column j, i < j
                const int4 a = row.meta, b = meta[h];
                const bool first = a.w < b.w, same = a.z == b.z;
                bool hit = sh < s_hi && (p.flags & (same ? AF_INTRA : AF_INTER));
                float d = 0.f;
                int bucket = 0;
                if (hit) {
                    const int eli = first ? a.y : b.y, elj = first ? b.y : a.y;
                    d = __fsqrt_rn(sh);
                    bucket = (same ? 0 : p.ne * p.ne) + eli * p.ne + elj;
                    hit = contact_value(p.flags, p.lower[elj * p.ne + eli], p.upper[elj * p.ne + eli], d);
                }
                const unsigned hits = __ballot_sync(0xffffffffu, hit);
                if (hit)
                    q.hit[fill + __popc(hits & before)] =
                        make_int4(first ? a.w : b.w, first ? b.w : a.w, bucket, __float_as_int(d));
                fill += __popc(hits);
                if (fill >= 32)
                    contact_flush(p, q, fill, 32);
            }
        });
    if (fill)
        contact_flush(p, q, fill, fill);
}

__global__ void __launch_bounds__(256) k_contact_place(ContactParams p, ListGuard guard, unsigned *strange)
{
    grid_dependency_wait();
    grid_launch_dependents();
    if (blockIdx.x == 0 && threadIdx.x == 0)
        *strange = *guard.strange;  // to the host with the results
    if (guard.closed())
        return;
    const long long len = *p.count;
    for (long long e = blockIdx.x * 256ll + threadIdx.x; e < len; e += gridDim.x * 256ll) {
        const int4 h = p.hits[e];
        p.placed[p.row[h.x] + p.rank[e]] = h;
    }
}

__global__ void __launch_bounds__(256) k_contact_order(ContactParams p, ListGuard guard)
{
    grid_dependency_wait();
    grid_launch_dependents();
    if (guard.closed())
        return;
    const long long len = *p.count;
    for (long long e = blockIdx.x * 256ll + threadIdx.x; e < len; e += gridDim.x * 256ll) {
        const int4 h = p.placed[e];
        const int b = p.row[h.x], end = p.row[h.x + 1];
        int at = b;
        for (int q = b; q < end; ++q) at += p.placed[q].y < h.y ? 1 : 0;
        p.list_bucket[at] = h.z;
        p.list_value[at] = __int_as_float(h.w);
    }
}

// Contacts listed at most, per atom, by the walk; more are left to the passes
// over all pairs (a row's entries are ordered by counting).
constexpr long long kContactsPerAtom = 128;

// The all-pairs sums by the walk.  *done is 0 (and the sums are as they were)
// where the limits do not bound the distance, or the atoms have coordinates
// that are not finite or more contacts than the walk lists.
int atomic_contacts_run(Context *c, const float *coords, int n, int flags, int ne, const float *basis_host, int isPBC,
                        const int *mol, const int *el, const float *lower_host, const float *upper_host,
                        const AtomicBlock &block, unsigned char *results, int *done, cudaStream_t st)
{
    *done = 0;
    float reach = 0.0f;
    for (int k = 0; k < ne * ne; ++k) {
        if (!(lower_host[k] == lower_host[k]) || !(upper_host[k] <= 3.0e38f))
            return FRMC_OK;  // NaN limits and infinite ones count pairs at any distance
        reach = upper_host[k] > reach ? upper_host[k] : reach;
    }
    static const float kId[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
    const float *Bh = isPBC && basis_host ? basis_host : kId;
    const int bm = basis_mode(Bh, isPBC);
    const Basis B = make_basis(Bh);
    if (!(flags & AF_WITHIN) || !cell_walk_applies(n, bm, B, reach))
        return FRMC_OK;
    ContactParams p{};
    float s_lo;
    sq_limits(0.0f, reach, &s_lo, &p.s_hi);
    p.flags = flags;
    p.ne = ne;
    p.lower = block.lower();
    p.upper = block.upper();
    p.count = block.length();
    p.cap = 4ll * n + 1024;
    for (int turn = 0; turn < 2; ++turn) {
        const size_t rows = 4 * (((size_t)n + 1 + 4095) / 4096 * 4096);
        FRMC_TRY(c->buf[BUF_CELLS].ensure(cell_hist_scratch(n, rows)));
        FRMC_TRY(c->buf[BUF_ATOMIC_TOTALS].ensure(36 * (size_t)p.cap));
        FRMC_TRY(c->buf[BUF_ATOMIC_LIST_B].ensure(4 * (size_t)p.cap + 4 * kSumPer));
        FRMC_TRY(c->buf[BUF_ATOMIC_LIST_V].ensure(4 * (size_t)p.cap + 4 * kSumPer));
        p.hits = c->buf[BUF_ATOMIC_TOTALS].as<int4>();
        p.placed = p.hits + p.cap;
        p.rank = reinterpret_cast<int *>(p.placed + p.cap);
        p.list_bucket = c->buf[BUF_ATOMIC_LIST_B].as<int>();
        p.list_value = c->buf[BUF_ATOMIC_LIST_V].as<float>();
        if (turn)
            FRMC_CUDA(cudaMemsetAsync(p.count, 0, 8, st));
        FRMC_TRY(sort_cells(c->sms, coords, nullptr, el, mol, n, bm, B, reach, ne, 1, c->buf[BUF_CELLS].p, &p.walk, st,
                            rows, reinterpret_cast<void **>(&p.row)));
        const unsigned *strange = &p.walk.sc->strange;
        FRMC_TRY(walk_lists(c->sms, p.walk, bm, st, [&](int grid) {
            switch (bm) {
            case BM_IBC: return launch_after(k_contacts<BM_IBC>, grid, kCellThreads, 0, st, p);
            case BM_DIAG: return launch_after(k_contacts<BM_DIAG>, grid, kCellThreads, 0, st, p);
            case BM_XYTRI: return launch_after(k_contacts<BM_XYTRI>, grid, kCellThreads, 0, st, p);
            case BM_LOWER: return launch_after(k_contacts<BM_LOWER>, grid, kCellThreads, 0, st, p);
            default: return launch_after(k_contacts<BM_GENERAL>, grid, kCellThreads, 0, st, p);
            }
        }));
        FRMC_TRY(launch_cell_scan(p.row, n + 1, st));
        const ListGuard guard{p.count, p.cap, strange};
        const int g = (int)((p.cap + 255) / 256 < 4ll * c->sms ? (p.cap + 255) / 256 : 4ll * c->sms);
        FRMC_TRY(launch_after(k_contact_place, g, 256, 0, st, p, guard, block.strange()));
        FRMC_TRY(launch_after(k_contact_order, g, 256, 0, st, p, guard));
        // in full order: its few large CTAs, placed while the one ahead runs, come
        // two to an SM (the call 229 -> 259 us)
        k_atomic_sum<<<2 * ne * ne, kSumThreads, 0, st>>>(p.list_bucket, p.list_value, p.count, guard, block.dsum(),
                                                          block.nsum());
        FRMC_CUDA(cudaGetLastError());
        FRMC_CUDA(cudaMemcpyAsync(results, block.p, block.results(), cudaMemcpyDeviceToHost, st));
        FRMC_CUDA(cudaStreamSynchronize(st));
        long long count;
        unsigned odd;
        memcpy(&count, results + 16 * block.m, sizeof(count));
        memcpy(&odd, results + 16 * block.m + 8, sizeof(odd));
        if (odd)
            return FRMC_OK;
        if (count <= p.cap) {
            *done = 1;
            return FRMC_OK;
        }
        if (count > kContactsPerAtom * n)
            return FRMC_OK;
        p.cap = count;
    }
    return FRMC_OK;
}

// ------------------------------------------------------------ a few rows
// The constraint's call on a moved molecule: K rows against every column, read
// once from the caller's arrays; the contacts (a few dozen) go to one list,
// and one CTA per accumulator orders and adds its own.  Six launches, a wait
// for the list's length and nine copies made a whole call of 161 us for 13 rows
// of 19,994 atoms; with these two launches and two copies it takes 75 us.
constexpr int kFewHits = 2048;

struct FewParams {
    AtomicParams a;
    long long *length;
    int4 *hits;  // (row position, column, bucket, value bits)
};

template <int BM>
__global__ void __launch_bounds__(256) k_few_rows(FewParams p)
{
    grid_launch_dependents();
    __shared__ float4 row[kFewRows];
    __shared__ int atom[kFewRows], mol[kFewRows];
    const AtomicParams &a = p.a;
    if ((int)threadIdx.x < a.K) {
        const int r = a.rows[threadIdx.x];
        row[threadIdx.x] =
            make_float4(a.coords[3ll * r], a.coords[3ll * r + 1], a.coords[3ll * r + 2], __int_as_float(a.el[r]));
        atom[threadIdx.x] = r;
        mol[threadIdx.x] = a.mol[r];
    }
    __syncthreads();
    const int j = blockIdx.x * 256 + threadIdx.x;
    if (j >= a.n)
        return;
    const float x = a.coords[3ll * j], y = a.coords[3ll * j + 1], z = a.coords[3ll * j + 2];
    const int elj = a.el[j], molj = a.mol[j];
    for (int k = 0; k < a.K; ++k) {
        if (j == atom[k] || (!a.allAtoms && j < atom[k]))
            continue;
        const bool same = molj == mol[k];
        if (!(a.flags & (same ? AF_INTRA : AF_INTER)))
            continue;
        const int ela = __float_as_int(row[k].w);
        float d = __fsqrt_rn(pair_s<BM>(row[k].x, row[k].y, row[k].z, x, y, z, a.B));
        if (!contact_value(a.flags, a.lower[elj * a.ne + ela], a.upper[elj * a.ne + ela], d))
            continue;
        const long long at = (long long)atomicAdd(reinterpret_cast<unsigned long long *>(p.length), 1ull);
        if (at < kFewHits)
            p.hits[at] = make_int4(k, j, (same ? 0 : a.ne * a.ne) + ela * a.ne + elj, __float_as_int(d));
    }
}

// One CTA per accumulator: its contacts in (row, column) order, added one
// after the other.
__global__ void __launch_bounds__(256) k_few_sum(FewParams p, float *dsum, int *nsum)
{
    grid_dependency_wait();
    grid_launch_dependents();
    __shared__ unsigned long long key[kFewHits];
    __shared__ float value[kFewHits], sorted[kFewHits];
    __shared__ int count;
    const long long len = *p.length;
    if (len > kFewHits)
        return;
    if (threadIdx.x == 0)
        count = 0;
    __syncthreads();
    for (int e = threadIdx.x; e < (int)len; e += 256) {
        const int4 h = p.hits[e];
        if (h.z == (int)blockIdx.x) {
            const int at = atomicAdd(&count, 1);
            key[at] = (unsigned long long)h.x << 32 | (unsigned)h.y;
            value[at] = __int_as_float(h.w);
        }
    }
    __syncthreads();
    const int m = count;
    for (int e = threadIdx.x; e < m; e += 256) {
        int at = 0;
        for (int q = 0; q < m; ++q) at += key[q] < key[e] ? 1 : 0;
        sorted[at] = value[e];
    }
    __syncthreads();
    if (threadIdx.x == 0 && m) {
        float s = dsum[blockIdx.x];
        for (int e = 0; e < m; ++e) s = __fadd_rn(s, sorted[e]);
        dsum[blockIdx.x] = s;
        nsum[blockIdx.x] += m;
    }
}

int atomic_few_run(Context *c, const float *coords, const int *rows, int K, int n, int allAtoms, int flags, int ne,
                   const float *basis_host, int isPBC, const int *mol, const int *el, const AtomicBlock &block,
                   unsigned char *results, int *done, cudaStream_t st)
{
    *done = 0;
    static const float kId[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
    const float *Bh = isPBC && basis_host ? basis_host : kId;
    FewParams p{};
    p.a.coords = coords;
    p.a.rows = rows;
    p.a.K = K;
    p.a.n = n;
    p.a.allAtoms = allAtoms;
    p.a.flags = flags;
    p.a.ne = ne;
    p.a.B = make_basis(Bh);
    p.a.mol = mol;
    p.a.el = el;
    p.a.lower = block.lower();
    p.a.upper = block.upper();
    p.length = block.length();
    FRMC_TRY(c->buf[BUF_ATOMIC_TOTALS].ensure(16 * kFewHits));
    p.hits = c->buf[BUF_ATOMIC_TOTALS].as<int4>();
    const unsigned g = (unsigned)((n + 255) / 256);
    switch (basis_mode(Bh, isPBC)) {
    case BM_IBC: k_few_rows<BM_IBC><<<g, 256, 0, st>>>(p); break;
    case BM_DIAG: k_few_rows<BM_DIAG><<<g, 256, 0, st>>>(p); break;
    case BM_XYTRI: k_few_rows<BM_XYTRI><<<g, 256, 0, st>>>(p); break;
    case BM_LOWER: k_few_rows<BM_LOWER><<<g, 256, 0, st>>>(p); break;
    default: k_few_rows<BM_GENERAL><<<g, 256, 0, st>>>(p); break;
    }
    FRMC_CUDA(cudaGetLastError());
    FRMC_TRY(launch_after(k_few_sum, 2 * ne * ne, 256, 0, st, p, block.dsum(), block.nsum()));
    FRMC_CUDA(cudaMemcpyAsync(results, block.p, block.results(), cudaMemcpyDeviceToHost, st));
    FRMC_CUDA(cudaStreamSynchronize(st));
    long long len;
    memcpy(&len, results + 16 * block.m, sizeof(len));
    *done = len <= kFewHits;
    return FRMC_OK;
}

int atomic_distances_run(Context *c, const float *coords, const float *dists, const int *rows, int K, int n,
                         int allAtoms, int flags, int ne, const float *basis_host, int isPBC, const int *mol,
                         const int *el, const float *lower, const float *upper, float *dsum, int *nsum,
                         cudaStream_t st)
{
    static const float kId[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
    AtomicParams p{};
    p.coords = coords;
    p.dists = dists;
    p.rows = rows;
    p.K = K;
    p.n = n;
    p.allAtoms = allAtoms;
    p.flags = flags;
    p.ne = ne;
    const float *B = isPBC && basis_host ? basis_host : kId;
    p.bm = basis_mode(B, isPBC);
    p.B = make_basis(B);
    p.mol = mol;
    p.el = el;
    p.lower = lower;
    p.upper = upper;
    return atomic_distances_device(p, c->buf[BUF_ATOMIC_COUNTS], c->buf[BUF_ATOMIC_TOTALS], c->buf[BUF_ATOMIC_LIST_B],
                                   c->buf[BUF_ATOMIC_LIST_V], dsum, nsum, st);
}

int launch_pair_stats(const int *el, const int *mol, int n, int ne, int *nintra, int *ninter, cudaStream_t st)
{
    if (n < 2)
        return FRMC_OK;
    k_pair_stats<<<n - 1, 256, 8 * ne * ne, st>>>(el, mol, n, ne, nintra, ninter);
    FRMC_CUDA(cudaGetLastError());
    return FRMC_OK;
}

}  // namespace frmc
