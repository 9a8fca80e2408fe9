// FP64 sine transforms between real and reciprocal space
// (fullrmc Extensions/reciprocal_space.pyx, recomputed in double precision).
//
//   gr_to_sq  (reciprocal_space.pyx:42-73):
//       S(q) = 1 + 4 pi rho / q * sum_r dr r (g(r) - 1) sin(q r)
//   Gr_to_sq  (reciprocal_space.pyx:82-109):
//       S(q) = 1 + 1 / q * sum_r dr G(r) sin(q r)
//   sq_to_Gr  (reciprocal_space.pyx:118-145):
//       G(r) = 2 / pi * sum_q dq q (S(q) - 1) sin(q r)
//
// The float32 inputs are promoted exactly, so every sine argument q*r is the
// exact double product; only the summation order differs from a float64
// numpy evaluation.
//
// Bound: GB300's narrow FP64 pipe (2 lanes a clock and SM: 16 cycles for a
// warp's instruction).  sin() costs about 30 FP64 instructions a term; the
// grids of the transforms let four do (k_sine_fixed).  k_sine_rows, one CTA per
// output point with sin(), takes the grids that do not.  Whole calls, r 0-20 A
// by 0.01 to Q 0.5-30 by 0.01 (5.9e6 terms): 278 -> 93.5 us.  Rms error against
// 80-bit sums, over 21 grids (500-2,000 r by 0.01, 450-2,950 Q, three transforms):
// 0.86 to 1.16 of k_sine_rows', mean 0.997; over each call's 20 smallest
// arguments 0.91.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "frmc_runtime.h"

namespace frmc {

enum SineKind : int { SK_GR_TO_SQ = 0, SK_BIGGR_TO_SQ = 1, SK_SQ_TO_GR = 2 };

// ----------------------------------------------------------------- shape function
// fullrmc's ShapeFunction (Constraints/Collection.py:15-160) on the device in
// FP64: a StructureFactorConstraint's total G(r) from all-pairs counts
// (StructureFactorConstraints.py:836-896), its S(q) (:302-312, 772-773) and
// G(r) back from S(q) (Collection.py:131-139).

// G(b) = 4 pi r_b rho0 (g(b) - 1), g(b) = sum_p coef_p n_p(b) / vol_b with
// n_p the pair's intra + inter counts (both orientations for unlike
// elements) and coef_p = w_p V / N_p; also w1[b] = dr G(b) for S(q).
__global__ void k_shape_G(const unsigned *__restrict__ counts, int ne, int hs, int npairs, const int *__restrict__ pi,
                          const int *__restrict__ pj, const double *__restrict__ pc, const double *__restrict__ r,
                          const double *__restrict__ vol, double rho0, double dr, double *__restrict__ G,
                          double *__restrict__ w1)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= hs)
        return;
    const long long total = (long long)ne * ne * hs;
    const unsigned *intra = counts, *inter = counts + total;
    double g = 0.0;
    for (int q = 0; q < npairs; ++q) {
        const int i = pi[q], j = pj[q];
        const long long ij = ((long long)i * ne + j) * hs + b;
        long long n = (long long)intra[ij] + inter[ij];
        if (i != j) {
            const long long ji = ((long long)j * ne + i) * hs + b;
            n += (long long)intra[ji] + inter[ji];
        }
        g += pc[q] * (double)n;
    }
    g /= vol[b];
    const double Gb = (4.0 * M_PI * r[b] * rho0) * (g - 1.0);
    G[b] = Gb;
    w1[b] = dr * Gb;
}

// w2[k] = dq q_k (S(q_k) - 1), the weights of the transform back to r.
__global__ void k_shape_wq(const double *__restrict__ q, const double *__restrict__ S, int nq, double dq,
                           double *__restrict__ w2)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < nq)
        w2[k] = dq * q[k] * (S[k] - 1.0);
}

// out[m] = add + mul * sum_l w[l] sin(x_m y_l) (divided by x_m when div): one
// CTA per output point; thread t sums l = t, t + 128, ... in order, and a
// fixed tree combines the 128 partial sums, so the result does not depend on
// anything but the inputs.
constexpr int kSineRowThreads = 128;
__global__ void __launch_bounds__(kSineRowThreads) k_sine_rows(const double *__restrict__ x,
                                                               const double *__restrict__ y,
                                                               const double *__restrict__ w, int ny, double add,
                                                               double mul, int div, double *__restrict__ out)
{
    __shared__ double part[kSineRowThreads / 32];
    const int m = blockIdx.x;
    const double xm = x[m];
    double acc = 0.0;
    for (int l = threadIdx.x; l < ny; l += kSineRowThreads) acc = fma(w[l], sin(xm * y[l]), acc);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31u) == 0)
        part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        const double s = (part[0] + part[1]) + (part[2] + part[3]);
        out[m] = add + mul * (div ? s / xm : s);
    }
}

// The sine transforms with one CTA per output point (k_sine_rows): the
// float32 grids are promoted exactly and the summand weights formed first.
__global__ void k_sine_prep(int kind, const float *__restrict__ xs, int nx, const float *__restrict__ ys,
                            const float *__restrict__ f, int ny, double *__restrict__ xd, double *__restrict__ yd,
                            double *__restrict__ w)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nx)
        xd[i] = (double)xs[i];
    if (i < ny) {
        const double dy = (double)ys[1] - (double)ys[0];
        const double y = (double)ys[i], v = (double)f[i];
        yd[i] = y;
        w[i] = kind == SK_BIGGR_TO_SQ ? dy * v : dy * y * (v - 1.0);
    }
}

// ------------------------------------------------- sines in fixed point
// Both grids are float32, so on a common scale the summation grid is integers,
// y = Y 2^-e with Y < 2^37, and each output point is the fraction of a turn
// X = x 2^-e / (2 pi) modulo 1, to 96 bits (Payne and Hanek's reduction: the
// product of a float's integer with as many bits of 1 / (2 pi) as it needs).
// The phase X Y modulo 1 is then a few integer multiply-adds, exact to 2^-59 of
// a turn, and the integer pipes are thirty times as wide as the FP64 pipe.  Its
// top 12 bits name one of 4,096 arcs, the others the place r in [-1/2, 1/2) of
// its arc, and with h = 2 pi / 4096
//   sin = T0 + T1 r + T2 r^2  (FP64: sin, h cos, -h^2/2 sin of the arc's centre)
//       + (T0's rounding - h^3/6 cos r^3 + h^4/24 sin r^4)   (float32),
// the last line below 1.6e-10 and so good to 5e-18 in float32, the next term of
// the series below 2.3e-18 (with 2,048 arcs 7e-17, as large as a sine's own
// rounding).  Four FP64 instructions a term: r, two for the polynomial, one for
// the weighted sum.
//
// The last line's sum over a lane's terms is formed first and the FP64 sum starts
// from it, so that it costs no rounding of its own: added at the end it made the
// error 3 to 9 % larger.  (The integer and float32 pipes have the room to form the
// phases twice; this, the larger table and the check below take 2 to 3 us of a
// call, 91.0 -> 93.5 us at 5.9e6 terms, 38.5 -> 40.5 at 3.5e5.)  What is left is an
// absolute error of a sine, where sin() has a relative one, so an output whose
// sines are small throughout -- sum |w| t below 1/32 sum |w|, with t = 2 / pi asin
// |sin| -- is summed again with sin(), or where an argument is small its series.
constexpr int kArcs = 4096;
// Rms error of an output over that of correctly rounded sines: 0.91 to 1.06 from
// t = 1/24 on, 0.97 to 1.24 at 1/32, 1.15 to 1.5 at 1/64 (sin() itself rounds
// a little worse: against k_sine_rows 0.91 over the 20 smallest arguments).
constexpr float kSineSmall = 1.0f / 32;
constexpr int kSineThreads = 384;  // 512 and 768: 0.5 and 2 us more a call of 5.9e6 terms
constexpr int kSineWarps = kSineThreads / 32;
constexpr int kSineParts = 4;    // parts of an output point's sum, a warp each
constexpr int kSineBatch = 64;   // output points of a CTA between two barriers

struct __align__(16) SineArc {
    double t0, t1, t2;
    float low, t3;  // T0's rounding, -h^3/6 cos
};
struct SineTable {
    SineArc arc[kArcs];
    float t4[kArcs];  // h^4/24 sin
};
struct SineTerm {
    unsigned y0, y1;
    double w;
};
struct SinePoint {
    unsigned x0, x1, x2;  // X, low word first
    int zero;             // x is 0: every sine is
    double x;
};

// Fixed-point fractions of 112 bits: a b.
static unsigned __int128 fixed_mul(unsigned __int128 a, unsigned __int128 b)
{
    const unsigned long long al = (unsigned long long)a, ah = (unsigned long long)(a >> 64);
    const unsigned long long bl = (unsigned long long)b, bh = (unsigned long long)(b >> 64);
    return ((unsigned __int128)ah * bh << 16) + (((unsigned __int128)ah * bl + (unsigned __int128)al * bh) >> 48);
}

// The nearest double of a fraction, and what is left of it.
static void fixed_split(unsigned __int128 v, double *hi, double *lo)
{
    *hi = std::ldexp((double)(unsigned long long)(v >> 48), -64);
    const __int128 rest = (__int128)v - ((__int128)(unsigned long long)std::ldexp(*hi, 64) << 48);
    *lo = std::ldexp((double)(long long)(rest >> 16), -96);
}

// The arcs' table from the Taylor series in fixed point (pi to 112 bits).
static void sine_table(SineTable *t)
{
    const unsigned __int128 pi = (unsigned __int128)0x3243f6a8885a3ull << 64 | 0x08d313198a2e0370ull;
    const double h = 2.0 * M_PI / kArcs;
    for (int k = 0; k < kArcs / 4; ++k) {
        const unsigned __int128 x = pi * (2 * k + 1) >> 12;  // the centre's angle in the first quadrant
        const unsigned __int128 x2 = fixed_mul(x, x);
        // cos above 1/2 and below: 1 - x^2/2 + ...; the terms fall below 2^-112
        unsigned __int128 one = (unsigned __int128)1 << 112, sn = x, cs = one, ts = x, tc = one;
        for (int i = 1; i < 20; ++i) {
            tc = fixed_mul(tc, x2) / (unsigned)((2 * i - 1) * (2 * i));
            ts = fixed_mul(ts, x2) / (unsigned)((2 * i) * (2 * i + 1));
            cs = i & 1 ? cs - tc : cs + tc;
            sn = i & 1 ? sn - ts : sn + ts;
        }
        double s, sl, c, cl;
        fixed_split(sn, &s, &sl);
        fixed_split(cs, &c, &cl);
        for (int q = 0; q < 4; ++q) {
            const double sv = q == 0 ? s : q == 1 ? c : q == 2 ? -s : -c;
            const double lv = q == 0 ? sl : q == 1 ? cl : q == 2 ? -sl : -cl;
            const double cv = q == 0 ? c : q == 1 ? -s : q == 2 ? -c : s;
            SineArc &a = t->arc[q * (kArcs / 4) + k];
            a.t0 = sv;
            a.t1 = cv * h;
            a.t2 = -sv * (h * h / 2.0);
            a.low = (float)lv;
            a.t3 = (float)(-cv * (h * h * h / 6.0));
            t->t4[q * (kArcs / 4) + k] = (float)(sv * (h * h * h * h / 24.0));
        }
    }
}

// The scale of a summation grid: the smallest e with every y 2^e an integer,
// below 2^37.  False for grids, weights and output grids that the fixed-point
// sines do not take (host arrays): the sines' last line is summed with float32
// weights, so a weight and any sum of weights has to be finite there and the
// largest far from its smallest numbers.
bool sine_fixed_scale(int kind, const float *xs, int64_t nx, const float *ys, const float *f, int64_t ny, int *scale)
{
    int e = -200, top = -200;
    float ymax = 0.0f;
    double wmax = 0.0;
    const double dy = (double)ys[1] - (double)ys[0];
    for (int64_t i = 0; i < ny; ++i) {
        const float y = ys[i];
        const double w = kind == SK_BIGGR_TO_SQ ? dy * f[i] : dy * y * ((double)f[i] - 1.0);
        if (!(y >= 0.0f && y < 1e30f) || !(std::fabs(f[i]) < 1e30f) || !(std::fabs(w) < 1e28))
            return false;
        wmax = std::max(wmax, std::fabs(w));
        if (y == 0.0f)
            continue;
        uint32_t u;
        memcpy(&u, &y, 4);
        int ex = (int)(u >> 23);
        uint32_t m = u & 0x7fffffu;
        if (ex)
            m |= 0x800000u;
        else
            ex = 1;
        e = std::max(e, 150 - ex - __builtin_ctz(m));  // y = m 2^(ex - 150)
        ymax = std::max(ymax, y);
    }
    if (!(ymax > 0.0f) || (wmax > 0.0 && wmax < 1e-20))
        return false;
    std::frexp(ymax, &top);
    if (top + e > 37 || e > 64 || e < -32)
        return false;
    for (int64_t i = 0; i < nx; ++i) {
        const float x = xs[i];
        // sines that are all small are left to sin() (kSineSmall)
        if (x != 0.0f && !(x > 0.0f && x < 1e6f && (double)x * ymax >= 0.02))
            return false;
    }
    *scale = e;
    return true;
}

__global__ void __launch_bounds__(256) k_sine_fixed_prep(int kind, const float *__restrict__ xs, int nx,
                                                         const float *__restrict__ ys, const float *__restrict__ f,
                                                         int ny, int e, SinePoint *__restrict__ point,
                                                         SineTerm *__restrict__ term, float *__restrict__ wf)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nx) {
        const float x = xs[i];
        const unsigned u = __float_as_uint(x), ex = max(u >> 23, 1u);
        const unsigned m = (u & 0x7fffffu) | (u >> 23 ? 0x800000u : 0u);
        // m times 1 / (2 pi) to 160 bits, then the 96 bits below the point
        const unsigned inv[5] = {0x36d8a566u, 0x7d4d3770u, 0x7f09d5f4u, 0x9391054au, 0x28be60dbu};
        unsigned p[7];
        unsigned long long carry = 0;
        for (int k = 0; k < 5; ++k) {
            carry += (unsigned long long)m * inv[k];
            p[k] = (unsigned)carry;
            carry >>= 32;
        }
        p[5] = (unsigned)carry;
        p[6] = 0u;
        const int shift = 64 + e - ((int)ex - 150);  // value = m 2^(ex - 150 - e) / (2 pi)
        unsigned w[3];
        for (int k = 0; k < 3; ++k) {
            const int b = shift + 32 * k, q = b >> 5, r = b & 31;
            const unsigned lo = q >= 0 && q < 7 ? p[q] : 0u, hi = q + 1 >= 0 && q + 1 < 7 ? p[q + 1] : 0u;
            w[k] = __funnelshift_r(lo, hi, r);
        }
        SinePoint pt;
        pt.x0 = w[0];
        pt.x1 = w[1];
        pt.x2 = w[2];
        pt.zero = x == 0.0f;
        pt.x = (double)x;
        point[i] = pt;
    }
    if (i < ny) {
        const double dy = (double)ys[1] - (double)ys[0];
        const double y = (double)ys[i], v = (double)f[i];
        const unsigned long long Y = (unsigned long long)ldexp(y, e);
        SineTerm t;
        t.y0 = (unsigned)Y;
        t.y1 = (unsigned)(Y >> 32);
        t.w = Y == 0 ? 0.0 : kind == SK_BIGGR_TO_SQ ? dy * v : dy * y * (v - 1.0);
        term[i] = t;
        wf[i] = (float)t.w;
    }
}

// The phase of one term in 2^-64 of a turn.
__device__ __forceinline__ unsigned long long sine_phase(const SinePoint &x, unsigned y0, unsigned y1)
{
    unsigned long long d = (unsigned long long)x.x0 * y0 >> 32;
    d += (unsigned long long)x.x1 * y0;
    d += (unsigned long long)x.x0 * y1;
    return d + ((unsigned long long)(x.x2 * y0 + x.x1 * y1) << 32);
}

// A lane's float32 sums over its terms.
struct SineSide {
    float low = 0.0f;    // weights times the sines' last line
    float small = 0.0f;  // |w| times the quarter turns from the sine's next zero
    float all = 0.0f;    // |w|
    __device__ __forceinline__ void add(const SineTable &t, unsigned long long d, float w)
    {
        const int k = (int)(d >> 52);
        const float r = (float)(int)((unsigned)(d >> 20) ^ 0x80000000u) * 2.3283064365386963e-10f;  // 2^-32
        const float2 a = *reinterpret_cast<const float2 *>(&t.arc[k].low);  // low, t3
        const float c = __fmaf_rn(__fmul_rn(__fmaf_rn(t.t4[k], r, a.y), r), __fmul_rn(r, r), a.x);
        low = __fmaf_rn(w, c, low);
        const float q = fabsf((float)(int)((unsigned)(d >> 32) << 1)) * 4.656612873077393e-10f;  // 2^-31
        small = __fmaf_rn(fabsf(w), q, small);
        all = __fadd_rn(all, fabsf(w));
    }
};

// sin(a) for 0 <= a <= 1/2 by its Taylor series (the next term is below 2^-65 a):
// a third of sin()'s FP64 instructions.
__device__ __forceinline__ double sine_series(double a)
{
    const double z = a * a;
    double p = -1.0 / 1307674368000.0;
    p = fma(p, z, 1.0 / 6227020800.0);
    p = fma(p, z, -1.0 / 39916800.0);
    p = fma(p, z, 1.0 / 362880.0);
    p = fma(p, z, -1.0 / 5040.0);
    p = fma(p, z, 1.0 / 120.0);
    p = fma(p, z, -1.0 / 6.0);
    return fma(a * z, p, a);
}

__device__ __forceinline__ double lane_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// CTA b takes the output points b, b + gridDim.x, ...; a warp sums a quarter
// of a point's terms, lane by lane in order, and the parts are added in a fixed
// tree, so the result depends on nothing but the inputs.
__global__ void __launch_bounds__(kSineThreads, 1) k_sine_fixed(const SineTable *__restrict__ table,
                                                                const SinePoint *__restrict__ point, int nx,
                                                                const SineTerm *__restrict__ term,
                                                                const float *__restrict__ wf, int ny, double unit,
                                                                double add, double mul, int div,
                                                                double *__restrict__ out)
{
    extern __shared__ __align__(16) unsigned char smem[];
    SineTable &t = *reinterpret_cast<SineTable *>(smem);
    __shared__ double part[kSineBatch * kSineParts];
    __shared__ float2 size[kSineBatch * kSineParts];  // sums of |w| t and |w|
    __shared__ bool again[kSineBatch];
    static_assert(kSineWarps % kSineParts == 0, "a warp keeps its part");
    {
        const uint4 *src = reinterpret_cast<const uint4 *>(table);
        uint4 *dst = reinterpret_cast<uint4 *>(smem);
        for (int k = threadIdx.x; k < (int)(sizeof(SineTable) / 16); k += kSineThreads) dst[k] = src[k];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int mine = (nx - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;  // output points of this CTA
    for (int o0 = 0; o0 < mine; o0 += kSineBatch) {
        const int batch = min(kSineBatch, mine - o0);
        const int items = batch * kSineParts, l0 = warp % kSineParts * 32 + lane;  // a warp's items are one part
        auto point_of = [&](int item) { return point[blockIdx.x + (o0 + item / kSineParts) * gridDim.x]; };
        SineSide next;
        SinePoint ahead{};
        if (warp < items) {
            ahead = point_of(warp);
            for (int l = l0; l < ny; l += 32 * kSineParts)
                next.add(t, sine_phase(ahead, term[l].y0, term[l].y1), wf[l]);
        }
        for (int item = warp; item < items; item += kSineWarps) {
            // this item's FP64 sum beside the float32 sums of the one after
            const SinePoint pt = ahead;
            const SineSide side = next;
            next = SineSide();
            if (item + kSineWarps < items)
                ahead = point_of(item + kSineWarps);
            double acc = (double)side.low;
#pragma unroll 2
            for (int l = l0; l < ny; l += 32 * kSineParts) {
                const SineTerm y = term[l];
                const unsigned long long d = sine_phase(pt, y.y0, y.y1);
                const double r = __longlong_as_double((long long)(d & 0xfffffffffffffull | 0x3ff0000000000000ull)) - 1.5;
                const SineArc &a = t.arc[d >> 52];
                acc = fma(y.w, fma(fma(a.t2, r, a.t1), r, a.t0), acc);
                next.add(t, sine_phase(ahead, y.y0, y.y1), wf[l]);
            }
            acc = lane_sum(acc);
            float small = side.small, all = side.all;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                small += __shfl_down_sync(0xffffffffu, small, o);
                all += __shfl_down_sync(0xffffffffu, all, o);
            }
            if (lane == 0) {
                part[item] = pt.zero ? 0.0 : acc;
                size[item] = make_float2(pt.zero ? all : small, all);
            }
        }
        __syncthreads();
        bool low = false;
        if ((int)threadIdx.x < batch) {
            const float2 *z = size + threadIdx.x * kSineParts;
            low = again[threadIdx.x] =
                (z[0].x + z[1].x) + (z[2].x + z[3].x) < kSineSmall * ((z[0].y + z[1].y) + (z[2].y + z[3].y));
        }
        if (__syncthreads_or(low)) {
            for (int item = warp; item < items; item += kSineWarps) {
                if (!again[item / kSineParts])
                    continue;
                const double x = point_of(item).x * unit;
                double acc = 0.0;
                for (int l = l0; l < ny; l += 32 * kSineParts) {
                    const SineTerm y = term[l];
                    // the integer y in a double's last place at 2^52
                    const double a = x * (__hiloint2double(0x43300000 | (int)y.y1, (int)y.y0) - 4503599627370496.0);
                    acc = fma(y.w, a <= 0.5 ? sine_series(a) : sin(a), acc);
                }
                acc = lane_sum(acc);
                if (lane == 0)
                    part[item] = acc;
            }
            __syncthreads();
        }
        if ((int)threadIdx.x < batch) {
            const double *p = part + threadIdx.x * kSineParts;
            const double s = (p[0] + p[1]) + (p[2] + p[3]);
            const int m = (int)blockIdx.x + (o0 + (int)threadIdx.x) * (int)gridDim.x;
            out[m] = add + mul * (div ? s / point[m].x : s);
        }
        __syncthreads();
    }
}

size_t sine_fixed_scratch(int64_t nx, int64_t ny)
{
    return sizeof(SinePoint) * (size_t)nx + sizeof(SineTerm) * (size_t)ny + 4 * (size_t)ny + 64;
}

size_t sine_table_bytes() { return sizeof(SineTable); }

// The arcs' table to `dst` (once per allocation).
int sine_table_upload(void *dst, cudaStream_t st)
{
    static const SineTable *table = [] {
        SineTable *t = new SineTable();
        sine_table(t);
        return t;
    }();
    FRMC_CUDA(cudaMemcpyAsync(dst, table, sizeof(SineTable), cudaMemcpyHostToDevice, st));
    return FRMC_OK;
}

// The transform on grids that sine_fixed_scale took; the arrays and `out` in
// device memory or host memory that the device reads and writes.
int launch_sine_fixed(int sms, int kind, const float *xs, int nx, const float *ys, const float *f, int ny, double rho,
                      int scale, double *out, const void *table, void *scratch, cudaStream_t st)
{
    SinePoint *point = static_cast<SinePoint *>(scratch);
    SineTerm *term = reinterpret_cast<SineTerm *>(point + nx);
    float *wf = reinterpret_cast<float *>(term + ny);
    const int n = nx > ny ? nx : ny;
    k_sine_fixed_prep<<<(n + 255) / 256, 256, 0, st>>>(kind, xs, nx, ys, f, ny, scale, point, term, wf);
    FRMC_CUDA(cudaFuncSetAttribute(k_sine_fixed, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SineTable)));
    const double add = kind == SK_SQ_TO_GR ? 0.0 : 1.0;
    const double mul = kind == SK_GR_TO_SQ ? 4.0 * M_PI * rho : kind == SK_BIGGR_TO_SQ ? 1.0 : 2.0 / M_PI;
    k_sine_fixed<<<sms < nx ? sms : nx, kSineThreads, sizeof(SineTable), st>>>(
        static_cast<const SineTable *>(table), point, nx, term, wf, ny, std::ldexp(1.0, -scale), add, mul,
        kind != SK_SQ_TO_GR, out);
    FRMC_CUDA(cudaGetLastError());
    return FRMC_OK;
}

int launch_sine(int kind, const float *xs, int nx, const float *ys, const float *f, int ny, double rho, double *out,
                double *scratch, cudaStream_t st)
{
    if (nx <= 0)
        return FRMC_OK;
    if (ny < 2)
        return set_error(FRMC_E_ARG, "sine transform needs at least two grid points");
    double *xd = scratch, *yd = xd + nx, *w = yd + ny;
    const int n = nx > ny ? nx : ny;
    k_sine_prep<<<(n + 255) / 256, 256, 0, st>>>(kind, xs, nx, ys, f, ny, xd, yd, w);
    if (kind == SK_GR_TO_SQ)
        k_sine_rows<<<nx, kSineRowThreads, 0, st>>>(xd, yd, w, ny, 1.0, 4.0 * M_PI * rho, 1, out);
    else if (kind == SK_BIGGR_TO_SQ)
        k_sine_rows<<<nx, kSineRowThreads, 0, st>>>(xd, yd, w, ny, 1.0, 1.0, 1, out);
    else
        k_sine_rows<<<nx, kSineRowThreads, 0, st>>>(xd, yd, w, ny, 0.0, 2.0 / M_PI, 0, out);
    FRMC_CUDA(cudaGetLastError());
    return FRMC_OK;
}

int launch_shape_function(const unsigned *counts, int ne, int hs, int npairs, const int *pi, const int *pj,
                          const double *pc, const double *r, const double *vol, double rho0, double dr,
                          const double *q, int nq, double dq, const double *rv, int nr, double *G, double *S,
                          double *Gs, double *w1, double *w2, cudaStream_t st)
{
    if (hs < 1 || nq < 1)
        return FRMC_OK;
    k_shape_G<<<(hs + 255) / 256, 256, 0, st>>>(counts, ne, hs, npairs, pi, pj, pc, r, vol, rho0, dr, G, w1);
    k_sine_rows<<<nq, kSineRowThreads, 0, st>>>(q, r, w1, hs, 1.0, 1.0, 1, S);
    k_shape_wq<<<(nq + 255) / 256, 256, 0, st>>>(q, S, nq, dq, w2);
    if (nr > 0)
        k_sine_rows<<<nr, kSineRowThreads, 0, st>>>(rv, q, w2, nq, 0.0, 2.0 / M_PI, 0, Gs);
    FRMC_CUDA(cudaGetLastError());
    return FRMC_OK;
}

}  // namespace frmc
