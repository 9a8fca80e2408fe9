// Distances, differences and coordinate transforms
// (fullrmc Extensions/pairs_distances.pyx and
//  Extensions/boundary_conditions_collection.pyx:88-110).
//
// Distances use the same squared-distance arithmetic as the histogram kernels
// followed by an IEEE sqrt; differences keep every basis term so that even
// signed zeros match the reference.
#include <algorithm>

#include "frmc_math.cuh"
#include "frmc_runtime.h"

namespace frmc {

struct PointSrc {
    const float *pts;   // explicit points: component c of point k at pts[c*ps + k]
    long long ps;
    const int *idx;     // or atom indexes into coords
    InlinePoints few;   // or (neither given) at most kInlinePoints points by value
};

constexpr int kDistAtoms = 256;  // threads of a block, and its largest tile of atoms
// Outputs that a block forms at most: 16 a thread, and fewer where that leaves
// less than two blocks an SM (differences of 5,000 atoms to 70 points: tiles of
// 256 atoms, 40 blocks, 75.7 us a call, of 21 atoms 60.4; 13 distances of 3,000
// atoms: 12 blocks 37, 188 blocks 28).
constexpr int kDistOutputs = 4096;
constexpr int kDistBlocks = 304;
constexpr int kDistLeast = 4;  // atoms of a tile

// W = 1: out[i, k] = |bc(point k - coords[i])|; W = 3: out[i, c, k] = component c
// of the difference.
//
// Bound by the bytes over the host link (coordinates in, rows out; an output is
// 4 bytes and about 25 instructions), so that each is moved once and in whole
// lines: a block stages its atoms' coordinates and up to kInlinePoints points in
// shared memory and writes the block's outputs in the order they are stored.  A
// difference is formed once per component for that.  13 rows of 52,000 atoms,
// whole call: one thread per (atom, row) between copies 65.5 us, so 50.
template <int BM, int W>
__global__ void __launch_bounds__(kDistAtoms) k_distances(const float *__restrict__ coords, int n,
                                                          const __grid_constant__ PointSrc src, int tile, int points, int K,
                                                          int fromIndex, Basis B, float *__restrict__ out)
{
    __shared__ float sc[3 * kDistAtoms], sx[kInlinePoints], sy[kInlinePoints], sz[kInlinePoints];
    __shared__ int sa[kInlinePoints];
    const int i0 = blockIdx.x * tile, k0 = blockIdx.y * points;
    const int na = min(tile, n - i0), kt = min(points, K - k0);
    for (int e = threadIdx.x; e < 3 * na; e += kDistAtoms) sc[e] = coords[3 * (long long)i0 + e];
    if ((int)threadIdx.x < kt) {
        const int t = threadIdx.x, k = k0 + t;
        if (src.idx) {
            const int a = src.idx[k];
            sa[t] = a;
            sx[t] = coords[3 * (long long)a];
            sy[t] = coords[3 * (long long)a + 1];
            sz[t] = coords[3 * (long long)a + 2];
        } else if (src.pts) {
            sa[t] = -1;
            sx[t] = src.pts[k];
            sy[t] = src.pts[src.ps + k];
            sz[t] = src.pts[2 * src.ps + k];
        } else {
            sa[t] = src.few.atom[t];
            sx[t] = src.few.x[t];
            sy[t] = src.few.y[t];
            sz[t] = src.few.z[t];
        }
    }
    __syncthreads();
    // row r = W * atom + component; consecutive threads take consecutive outputs
    const int dr = kDistAtoms / kt, dk = kDistAtoms % kt;
    int r = threadIdx.x / kt, k = threadIdx.x % kt;
    while (r < W * na) {
        const int a = W == 1 ? r : r / 3;
        if (!(fromIndex && i0 + a < sa[k])) {
            float v;
            if (W == 1) {
                v = __fsqrt_rn(pair_s<BM>(sx[k], sy[k], sz[k], sc[3 * a], sc[3 * a + 1], sc[3 * a + 2], B));
            } else {
                float d[3];
                pair_diff(sx[k], sy[k], sz[k], sc[3 * a], sc[3 * a + 1], sc[3 * a + 2], B, BM != BM_IBC, d[0], d[1],
                          d[2]);
                const int c = r - 3 * a;
                v = c == 0 ? d[0] : c == 1 ? d[1] : d[2];
            }
            out[((long long)i0 * W + r) * K + k0 + k] = v;
        }
        r += dr;
        k += dk;
        if (k >= kt) {
            k -= kt;
            ++r;
        }
    }
}

// out[i] = bc(to[i] - from[i])  (pairs_distances.pyx:71-93, :113-126)
__global__ void __launch_bounds__(256) k_from_to(const float *__restrict__ from, const float *__restrict__ to, int n,
                                                 Basis B, int isPBC, float *__restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    float ox, oy, oz;
    pair_diff(to[3 * (long long)i], to[3 * (long long)i + 1], to[3 * (long long)i + 2], from[3 * (long long)i],
              from[3 * (long long)i + 1], from[3 * (long long)i + 2], B, isPBC, ox, oy, oz);
    out[3 * (long long)i] = ox;
    out[3 * (long long)i + 1] = oy;
    out[3 * (long long)i + 2] = oz;
}

// out[i] = coords[i] . M in the reference's order
// (boundary_conditions_collection.pyx:104-106).
__global__ void __launch_bounds__(256) k_transform(Basis M, const float *__restrict__ coords, int n,
                                                   float *__restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const float x = coords[3 * (long long)i], y = coords[3 * (long long)i + 1], z = coords[3 * (long long)i + 2];
#pragma unroll
    for (int c = 0; c < 3; ++c)
        out[3 * (long long)i + c] =
            __fadd_rn(__fadd_rn(__fmul_rn(x, M.b[c]), __fmul_rn(y, M.b[3 + c])), __fmul_rn(z, M.b[6 + c]));
}

int launch_distances(int diff, const float *coords, int n, const float *pts, long long ps, const int *idx,
                     const InlinePoints *few, int K, int fromIndex, int isPBC, const float *basis, float *out,
                     cudaStream_t st)
{
    if (n <= 0 || K <= 0)
        return FRMC_OK;
    if (K > 65535)
        return set_error(FRMC_E_ARG, "too many points (%d)", K);
    PointSrc src{pts, ps, idx, few ? *few : InlinePoints()};
    Basis B = make_basis(basis);
    // as many points for each block of a row of blocks (65: 33 and 32)
    const int turns = (K + kInlinePoints - 1) / kInlinePoints, points = (K + turns - 1) / turns;
    int tile = std::min(kDistAtoms, kDistOutputs / ((diff ? 3 : 1) * points));
    tile = std::max(kDistLeast, std::min(tile, (n + kDistBlocks - 1) / kDistBlocks * turns));
    dim3 grid((n + tile - 1) / tile, turns);
    if (diff) {
        // one form for every basis: no term that is zero may be left out
        auto kern = isPBC ? k_distances<BM_GENERAL, 3> : k_distances<BM_IBC, 3>;
        kern<<<grid, kDistAtoms, 0, st>>>(coords, n, src, tile, points, K, fromIndex, B, out);
        FRMC_CUDA(cudaGetLastError());
        return FRMC_OK;
    }
    switch (basis_mode(basis, isPBC)) {
    case BM_IBC: k_distances<BM_IBC, 1><<<grid, kDistAtoms, 0, st>>>(coords, n, src, tile, points, K, fromIndex, B, out); break;
    case BM_DIAG: k_distances<BM_DIAG, 1><<<grid, kDistAtoms, 0, st>>>(coords, n, src, tile, points, K, fromIndex, B, out); break;
    case BM_XYTRI: k_distances<BM_XYTRI, 1><<<grid, kDistAtoms, 0, st>>>(coords, n, src, tile, points, K, fromIndex, B, out); break;
    case BM_LOWER: k_distances<BM_LOWER, 1><<<grid, kDistAtoms, 0, st>>>(coords, n, src, tile, points, K, fromIndex, B, out); break;
    default: k_distances<BM_GENERAL, 1><<<grid, kDistAtoms, 0, st>>>(coords, n, src, tile, points, K, fromIndex, B, out); break;
    }
    FRMC_CUDA(cudaGetLastError());
    return FRMC_OK;
}

int launch_from_to(const float *from, const float *to, int n, int isPBC, const float *basis, float *out,
                   cudaStream_t st)
{
    if (n <= 0)
        return FRMC_OK;
    k_from_to<<<(n + 255) / 256, 256, 0, st>>>(from, to, n, make_basis(basis), isPBC, out);
    FRMC_CUDA(cudaGetLastError());
    return FRMC_OK;
}

int launch_transform(const float *M, const float *coords, int n, float *out, cudaStream_t st)
{
    if (n <= 0)
        return FRMC_OK;
    k_transform<<<(n + 255) / 256, 256, 0, st>>>(make_basis(M), coords, n, out);
    FRMC_CUDA(cudaGetLastError());
    return FRMC_OK;
}

}  // namespace frmc
