// Coordination numbers (Extensions/atomic_coordination.pyx, used by
// AtomicCoordinationNumberConstraint).  Every entry point of that module is a
// sequence of terms
//     coordNumData[def] += count{ j in list : lower[def] <= d(row, j) <= upper[def] }
// where d is the minimum-image distance of two atoms (or an entry of a
// caller's distance row) and the count is a float32 sum of ones
// (atomic_coordination.pyx:31-44), so it is exact below 2^24 and stops at
// 2^24 above.  The additions into coordNumData are float32 and happen in term
// order (atomic_coordination.pyx:184-198, 220-240), which only matters when a
// partial sum is not an integer below 2^24.
//
//   k_coord_count       one CTA per (term, chunk of kCoordChunk list entries):
//                       distances, window test, one integer atomicAdd per CTA;
//   k_coord_accumulate  one warp per definition: the sum of its terms' counts
//                       when every partial sum is an exact integer, else the
//                       float32 additions one by one in term order.
#include <cmath>
#include <cstdint>
#include <cstring>

#include "cell_walk.cuh"
#include "frmc_ptx.cuh"

namespace frmc {

constexpr int kCoordThreads = 256;
constexpr int kCoordPerThread = 4;
constexpr int kCoordChunk = kCoordThreads * kCoordPerThread;
constexpr int kCoordSaturate = 1 << 24;  // 2^24 + 1 rounds back to 2^24 in float32

struct CoordParams {
    const float *coords;         // (n, 3) box coordinates, or null for distance rows
    const float *dists;          // concatenated distance rows
    const long long *dist_off;   // start of row r in dists
    const int *dist_len;         // length of row r
    int n;
    Basis B;
    const int *lists;            // concatenated index lists
    const CoordTerm *terms;
    const int2 *items;           // (term, first list entry of the chunk)
    const float *lower, *upper;  // per definition
    int *counts;                 // per term, zeroed before the launch
};

template <int BM>
__global__ void __launch_bounds__(kCoordThreads) k_coord_count(CoordParams p)
{
    __shared__ int s_warp[kCoordThreads / 32];
    const int2 it = p.items[blockIdx.x];
    const CoordTerm t = p.terms[it.x];
    const float lo = p.lower[t.def], up = p.upper[t.def];
    float ax = 0.f, ay = 0.f, az = 0.f;
    const float *row = nullptr;
    int rowlen;
    if (p.coords) {
        ax = p.coords[3ll * t.row];
        ay = p.coords[3ll * t.row + 1];
        az = p.coords[3ll * t.row + 2];
        rowlen = p.n;
    } else {
        row = p.dists + p.dist_off[t.row];
        rowlen = p.dist_len[t.row];
    }
    int hits = 0;
#pragma unroll
    for (int u = 0; u < kCoordPerThread; ++u) {
        const int e = it.y + u * kCoordThreads + (int)threadIdx.x;
        if (e < t.len) {
            int j = p.lists[t.begin + e];
            if (j < 0)  // numpy indexing of the list (checked on the host)
                j += rowlen;
            float d;
            if (p.coords)
                d = __fsqrt_rn(pair_s<BM>(ax, ay, az, p.coords[3ll * j], p.coords[3ll * j + 1], p.coords[3ll * j + 2],
                                          p.B));
            else
                d = row[j];
            hits += (lo <= d && d <= up) ? 1 : 0;
        }
    }
    hits = __reduce_add_sync(0xffffffffu, hits);
    if ((threadIdx.x & 31u) == 0)
        s_warp[threadIdx.x >> 5] = hits;
    __syncthreads();
    if (threadIdx.x == 0) {
        int total = 0;
#pragma unroll
        for (int w = 0; w < kCoordThreads / 32; ++w) total += s_warp[w];
        if (total)
            atomicAdd(p.counts + it.x, total);
    }
}

__device__ __forceinline__ int coord_saturate(int c)
{
    return c < kCoordSaturate ? c : kCoordSaturate;
}

// def_ids[u]: the u-th definition touched; its terms, in call order, are
// def_terms[def_off[u] .. def_off[u+1]).
__global__ void k_coord_accumulate(const int *counts, const int *def_ids, const int *def_off, const int *def_terms,
                                   int ndefs, float *data)
{
    const int u = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const unsigned lane = threadIdx.x & 31u;
    if (u >= ndefs)
        return;
    const int b = def_off[u], e = def_off[u + 1];
    long long total = 0;
    for (int i = b + (int)lane; i < e; i += 32) total += coord_saturate(counts[def_terms[i]]);
#pragma unroll
    for (int off = 16; off; off >>= 1) total += __shfl_xor_sync(0xffffffffu, total, off);
    if (lane)
        return;
    const int def = def_ids[u];
    const float c0 = data[def];
    // all partial sums c0 + k lie in [c0, c0 + total]: exact when that range
    // holds only integers of magnitude <= 2^24
    if (c0 == rintf(c0) && fabsf(c0) <= (float)kCoordSaturate && (double)c0 + (double)total <= (double)kCoordSaturate) {
        data[def] = (float)((long long)c0 + total);
        return;
    }
    float c = c0;
    for (int i = b; i < e; ++i) c = __fadd_rn(c, (float)coord_saturate(counts[def_terms[i]]));
    data[def] = c;
}

int coordination_run(const CoordLaunch &L, cudaStream_t st)
{
    if (L.nitems > 0) {
        CoordParams p{};
        p.coords = L.coords;
        p.dists = L.dists;
        p.dist_off = L.dist_off;
        p.dist_len = L.dist_len;
        p.n = L.n;
        static const float kId[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
        const float *B = L.isPBC && L.basis ? L.basis : kId;
        const int bm = L.coords ? basis_mode(B, L.isPBC) : BM_IBC;
        p.B = make_basis(B);
        p.lists = L.lists;
        p.terms = L.terms;
        p.items = L.items;
        p.lower = L.lower;
        p.upper = L.upper;
        p.counts = L.counts;
        const unsigned g = (unsigned)L.nitems;
        switch (bm) {
        case BM_IBC: k_coord_count<BM_IBC><<<g, kCoordThreads, 0, st>>>(p); break;
        case BM_DIAG: k_coord_count<BM_DIAG><<<g, kCoordThreads, 0, st>>>(p); break;
        case BM_XYTRI: k_coord_count<BM_XYTRI><<<g, kCoordThreads, 0, st>>>(p); break;
        case BM_LOWER: k_coord_count<BM_LOWER><<<g, kCoordThreads, 0, st>>>(p); break;
        default: k_coord_count<BM_GENERAL><<<g, kCoordThreads, 0, st>>>(p); break;
        }
        FRMC_CUDA(cudaGetLastError());
    }
    if (L.ndefs > 0) {
        const int threads = 128;
        const unsigned g = (unsigned)(((long long)L.ndefs * 32 + threads - 1) / threads);
        k_coord_accumulate<<<g, threads, 0, st>>>(L.counts, L.def_ids, L.def_off, L.def_terms, L.ndefs, L.data);
        FRMC_CUDA(cudaGetLastError());
    }
    return FRMC_OK;
}

// ------------------------------------------------- all atoms, by the walk
// all_atoms_coord_number_coords meets every core with every shell atom of a
// definition: 2.2e9 distances for 52,000 atoms, of which a few per atom lie in
// a window.  Where every window's upper end bounds the distance, every list
// holds an atom once and every row a (list, definition) once, the counts come
// from the walk over sorted atoms: an atom carries one bit per slot (list,
// definition) as a row and one as a member of the slot's list, and a pair
// adds to the slots where one atom is a row and the other a member, both ways
// round.  The sums are whole numbers, so their order is free; k_coord_count
// takes the rest.  Measured, 52,000 atoms, four definitions: 4.82 ms -> 68 us
// and 27 us for the sort; the native call 6.2 -> 0.6 ms.
struct CoordWalk {
    CellWalk walk;
    float s_hi;              // s < s_hi for every distance up to the largest upper end
    const float *lower, *upper;  // per slot
    unsigned long long *totals;  // per slot
};

template <int BM>
__global__ void __launch_bounds__(kCellThreads, 1) k_coord_walk(CoordWalk p)
{
    grid_dependency_wait();
    grid_launch_dependents();
    __shared__ CellStage stage[kCellThreads / 32];
    __shared__ unsigned count[kCoordSlots];
    __shared__ float lower[kCoordSlots], upper[kCoordSlots];
    if (threadIdx.x < kCoordSlots) {
        count[threadIdx.x] = 0u;
        lower[threadIdx.x] = p.lower[threadIdx.x];
        upper[threadIdx.x] = p.upper[threadIdx.x];
    }
    __syncthreads();
    const float s_hi = p.s_hi;
    walk_blocks<BM>(
        p.walk, stage[threadIdx.x >> 5], [](const int4 &m, bool) { return m; },
        [&](f2 s01, f2 s23, const CellRow &row, const int4 *meta, int, auto) {
            const float s[4] = {lo2(s01), hi2(s01), lo2(s23), hi2(s23)};
            unsigned in = 0u;
#pragma unroll
            for (int h = 0; h < 4; ++h) in |= s[h] < s_hi ? 1u << h : 0u;
            while (in) {
                const int h = __ffs(in) - 1;
                in &= in - 1;
                // meta: (slots as a row, the same, slots as a member, original index)
                const int4 b = meta[h];
                const unsigned ab = (unsigned)(row.meta.x & b.z), ba = (unsigned)(b.x & row.meta.z);
                unsigned left = ab | ba;
                if (!left)
                    continue;
                const float d = __fsqrt_rn(h < 2 ? (h ? s[1] : s[0]) : (h == 2 ? s[2] : s[3]));
                while (left) {
                    const int k = __ffs(left) - 1;
                    left &= left - 1;
                    if (lower[k] <= d && d <= upper[k])
                        atomicAdd(count + k, (ab >> k & 1u) + (ba >> k & 1u));
                }
            }
        });
    __syncthreads();
    if (threadIdx.x < kCoordSlots && count[threadIdx.x])
        atomicAdd(p.totals + threadIdx.x, (unsigned long long)count[threadIdx.x]);
}

int coordination_walk(Context *c, const float *coords, const int *row_mask, const int *member_mask, int n,
                      const float *basis, int isPBC, const float *lower, const float *upper, int nslots,
                      long long *totals, int *done, cudaStream_t st)
{
    *done = 0;
    float low[kCoordSlots], up[kCoordSlots], reach = 0.0f;
    for (int k = 0; k < kCoordSlots; ++k) {
        low[k] = k < nslots ? lower[k] : 0.0f;
        up[k] = k < nslots ? upper[k] : -1.0f;
        if (!(up[k] <= 3.0e38f) || !(low[k] == low[k]))
            return FRMC_OK;
        reach = up[k] > reach ? up[k] : reach;
    }
    static const float kId[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
    const float *Bh = isPBC && basis ? basis : kId;
    const int bm = basis_mode(Bh, isPBC);
    const Basis B = make_basis(Bh);
    reach = nextafterf(reach, 3.4e38f);  // windows include their upper end
    if (!cell_walk_applies(n, bm, B, reach))
        return FRMC_OK;
    CoordWalk p{};
    float s_lo;
    sq_limits(0.0f, reach, &s_lo, &p.s_hi);
    FRMC_TRY(c->buf[BUF_CELLS].ensure(cell_hist_scratch(n)));
    FRMC_TRY(c->buf[BUF_ATOMIC_ACC].ensure(16 * kCoordSlots));
    p.totals = c->buf[BUF_ATOMIC_ACC].as<unsigned long long>();
    float *limits = reinterpret_cast<float *>(p.totals + kCoordSlots);
    p.lower = limits;
    p.upper = limits + kCoordSlots;
    unsigned char block[16 * kCoordSlots] = {0};
    memcpy(block + 8 * kCoordSlots, low, sizeof(low));
    memcpy(block + 12 * kCoordSlots, up, sizeof(up));
    FRMC_CUDA(cudaMemcpyAsync(p.totals, block, sizeof(block), cudaMemcpyHostToDevice, st));
    FRMC_TRY(sort_cells(c->sms, coords, nullptr, row_mask, member_mask, n, bm, B, reach, 1, 1, c->buf[BUF_CELLS].p,
                        &p.walk, st, 0, nullptr));
    FRMC_TRY(walk_lists(c->sms, p.walk, bm, st, [&](int grid) {
        switch (bm) {
        case BM_IBC: return launch_after(k_coord_walk<BM_IBC>, grid, kCellThreads, 0, st, p);
        case BM_DIAG: return launch_after(k_coord_walk<BM_DIAG>, grid, kCellThreads, 0, st, p);
        case BM_XYTRI: return launch_after(k_coord_walk<BM_XYTRI>, grid, kCellThreads, 0, st, p);
        case BM_LOWER: return launch_after(k_coord_walk<BM_LOWER>, grid, kCellThreads, 0, st, p);
        default: return launch_after(k_coord_walk<BM_GENERAL>, grid, kCellThreads, 0, st, p);
        }
    }));
    FRMC_CUDA(cudaGetLastError());
    long long got[kCoordSlots];
    unsigned odd = 0;
    FRMC_CUDA(cudaMemcpyAsync(got, p.totals, sizeof(got), cudaMemcpyDeviceToHost, st));
    FRMC_CUDA(cudaMemcpyAsync(&odd, &p.walk.sc->strange, sizeof(odd), cudaMemcpyDeviceToHost, st));
    FRMC_CUDA(cudaStreamSynchronize(st));
    if (odd)
        return FRMC_OK;
    for (int k = 0; k < nslots; ++k) totals[k] = got[k];
    *done = 1;
    return FRMC_OK;
}

int coordination_chunk()
{
    return kCoordChunk;
}

}  // namespace frmc
