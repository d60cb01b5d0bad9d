// lp_hull.cu — per-cluster convex hull and oriented bounding boxes.
//
// Reference: lidar_processing_lib/src/polygonizer.cpp and Processor::run's per-cluster gather
// (src/processor/src/processor.cpp:627-671). Persistent CTAs take clusters from a work queue
// (clusters above 512 members one CTA each, then the others one warp each). The cluster scatter
// has already written each member's x, y contiguously and the cluster's z range. Per cluster:
//   1. the members extreme in 16 directions (an inscribed polygon of members),
//   2. Quickhull refinement: the member farthest outside each polygon edge is inserted, for a
//      few rounds; members proven strictly inside leave the active set. Every polygon vertex is a
//      member, so a member strictly inside the polygon (an FP32 test with a 1e-5 relative margin,
//      far above its rounding error) cannot be a hull vertex,
//   3. sort of the remaining candidates by (x, y, member order), Andrew's monotone chain with the
//      reference's FP64 orientation predicate (polygonizer.cpp:45-50, 62-85) decided in FP32
//      wherever that is provably the same decision: the same output as the reference's chain over
//      all members,
//   4. local hull indices = rank of each hull vertex among the cluster's members in input
//      order (the reference gathers a cluster's points in obstacle order, processor.cpp:640),
//   5. in a kernel of its own (k_hull_boxes), rotating-calipers box (Shamos antipodal pairs, best area
//      kept as a float exactly like BoundingBox::area; comparisons screened in FP32) and the PCA box,
//      one warp each.
#include <atomic>
#include <cfloat>
#include <climits>
#include <mutex>

#include "lp_introsort.cuh"
#include "lp_batch.cuh"
#include "lp_common.cuh"
#include "lp_math.cuh"
#include "lp_stages.hpp"

namespace lpg
{
namespace
{
constexpr int kHullThreads = 256;
constexpr int kHullSmem = 1024; // candidates sorted in shared memory; larger sets use global scratch

template <typename T>
struct HPt
{
    T x, y;
    uint32_t key; // tie-break and identity: member input order
};

template <typename T>
__device__ __forceinline__ bool hpt_less(const HPt<T>& a, const HPt<T>& b)
{
    // (without branches: the sorts compare every pair or exchange every step)
    return (a.x < b.x) | ((a.x == b.x) & ((a.y < b.y) | ((a.y == b.y) & (a.key < b.key))));
}

// Members with a NaN coordinate are no candidates: hpt_less would not order them (the sorts by counting
// need a total order), and the chain, which never pops them, would hold more vertices than the cluster members.
__device__ __forceinline__ bool has_place(float x, float y)
{
    return x == x && y == y;
}

// polygonizer.cpp:45-50: counter-clockwise or collinear, evaluated in FP64 exactly as written
__device__ __noinline__ bool ccw_or_colinear(double ax, double ay, double bx, double by, double cx, double cy)
{
    return (bx - ax) * (cy - ay) - (by - ay) * (cx - ax) <= 0;
}

__device__ __forceinline__ uint32_t ford(float f)
{
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ unsigned long long warp_max64(unsigned long long v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
    {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, v, o);
        v = t > v ? t : v;
    }
    return v;
}
// The smaller / larger of an accumulator that is not a NaN and a value (a NaN leaves the accumulator).
__device__ __forceinline__ double min_d(double acc, double v)
{
    return v < acc ? v : acc;
}
__device__ __forceinline__ double max_d(double acc, double v)
{
    return v > acc ? v : acc;
}
// The warp's smallest / largest of values that are not NaNs: integer reductions of the two halves of the order-preserving
// bit pattern (an FP64 tree takes five dependent comparisons of the FP64 unit and ten shuffles).
__device__ __noinline__ double warp_min_d(double v)
{
    const long long u = __double_as_longlong(v);
    const unsigned long long k = static_cast<unsigned long long>(u ^ ((u >> 63) | LLONG_MIN));
    const uint32_t h = static_cast<uint32_t>(k >> 32);
    const uint32_t hi = __reduce_min_sync(0xffffffffu, h);
    const uint32_t lo = __reduce_min_sync(0xffffffffu, h == hi ? static_cast<uint32_t>(k) : 0xffffffffu);
    const long long m = static_cast<long long>((static_cast<unsigned long long>(hi) << 32) | lo);
    return __longlong_as_double(m ^ (~(m >> 63) | LLONG_MIN));
}
__device__ __forceinline__ double warp_max_d(double v)
{
    return -warp_min_d(-v);
}

// ---------------------------------------------------------------------------------------------
// Shamos antipodal pairs (polygonizer.cpp:93-163) for the hull P[0..n), written to `pairs`.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ double tri_area(double ax, double ay, double bx, double by, double cx, double cy)
{
    // areaOfTriangle, polygonizer.hpp:227-231
    return fabs((ax * (by - cy) + bx * (cy - ay) + cx * (ay - by)) * 0.5);
}

// What bounds these kernels on a scan is the code itself: a cluster's warp runs most of it once, and waits
// for each instruction line to arrive. So every FP64 division and square root is one shared function (a
// call costs a few tens of cycles, the inlined sequence about 2 KB), what runs rarely stands out of line, and
// loops over a hull's few vertices are not unrolled further than their latency needs.
__device__ __noinline__ double div_d(double a, double b)
{
    return a / b;
}
__device__ __noinline__ double sqrt_d(double a)
{
    return sqrt(a);
}

// The FP64 areas of two triangles of P compared, as the reference evaluates them (side by side: the two
// chains overlap): 1 larger, 0 equal, -1 neither.
__device__ __noinline__ int area_order(const double2* P, int a1, int b1, int c1, int a2, int b2, int c2)
{
    const double u = tri_area(P[a1].x, P[a1].y, P[b1].x, P[b1].y, P[c1].x, P[c1].y);
    const double v = tri_area(P[a2].x, P[a2].y, P[b2].x, P[b2].y, P[c2].x, P[c2].y);
    return u > v ? 1 : (u == v ? 0 : -1);
}

// The error of s = fl(b - a) (Knuth's TwoSum of b and -a): s + diff_err = b - a exactly.
__device__ __forceinline__ float diff_err(float b, float a, float s)
{
    const float a1 = s - b;
    const float b1 = s - a1;
    return ((-a) - a1) + (b - b1);
}

// Twice the signed area of (a, b, c), hi + lo, from exact two-term differences and products (the last cross terms dropped).
__device__ __forceinline__ float2 cross2(float2 a, float2 b, float2 c)
{
    const float u = b.x - a.x, v = c.y - a.y, w = b.y - a.y, z = c.x - a.x;
    const float ul = diff_err(b.x, a.x, u), vl = diff_err(c.y, a.y, v), wl = diff_err(b.y, a.y, w), zl = diff_err(c.x, a.x, z);
    const float t1 = u * v, t2 = w * z;
    const float e1 = __fmaf_rn(u, v, -t1), e2 = __fmaf_rn(w, z, -t2);
    const float s = t1 - t2;
    const float lo = diff_err(t1, t2, s) + ((e1 + (u * vl + ul * v)) - (e2 + (w * zl + wl * z)));
    const float hi = s + lo;
    const float rest = (s - hi) + lo;
    return hi < 0.0f ? make_float2(-hi, -rest) : make_float2(hi, rest);
}

// area_order of float vertices. Twice the areas from cross2 are within 2^-41 R^2 each (its products lie below 4 R^2
// and err by 2^-45 of that, its sums of small terms by less), the FP64 ones within 2e-14 M R (R, M as
// below): a difference beyond tol2 = 4e-12 R^2 + 4e-13 M R has the FP64 comparison's sign. Opposite edges of a box are
// near parallel, so many of a walk's comparisons come here; an FP64 chain costs 64 cycles an operation.
__device__ __noinline__ int area_order_near(const double2* P, const float2* Pf, float tol2, int a1, int b1, int c1, int a2,
                                            int b2, int c2)
{
    const float2 u = cross2(Pf[a1], Pf[b1], Pf[c1]), v = cross2(Pf[a2], Pf[b2], Pf[c2]);
    const float d = (u.x - v.x) + (u.y - v.y);
    if (fabsf(d) > tol2)
        return d > 0.0f ? 1 : -1;
    return area_order(P, a1, b1, c1, a2, b2, c2);
}

// Triangle-area comparisons of the pair walk, evaluated in FP64 exactly as the reference does.
struct AreaCmpFp64
{
    const double2* P;
    __device__ __forceinline__ bool gt(int a1, int b1, int c1, int a2, int b2, int c2) const
    {
        return area_order(P, a1, b1, c1, a2, b2, c2) > 0;
    }
    __device__ __forceinline__ bool eq(int a1, int b1, int c1, int a2, int b2, int c2) const
    {
        return area_order(P, a1, b1, c1, a2, b2, c2) == 0;
    }
};

// The same comparisons decided in FP32 where the float areas differ by more than `tol`, else by
// area_order_near. Float areas use coordinates relative to vertex 0: with every |local vertex| <= R the
// float area is within 1.02e-6 R^2 of the exact area of the (float-valued) vertices, and the FP64
// area of the reference within 1e-14 M R (M the largest |coordinate|). tol is at least twice the
// sum of both bounds, so a decision taken in FP32 is the one FP64 takes. The margins are the constructor's:
// one left at zero would let the approximate areas decide the ties of parallel edges.
struct AreaCmpFiltered
{
    const double2* P;
    const float2* Pf; // the same vertices as floats (exact: they are float points)
    float ox, oy, tol;
    float tol2; // of twice the areas, evaluated with two-term differences and products (area_order_near)
    // m: M; r2: at least R^2
    __device__ __forceinline__ AreaCmpFiltered(const double2* p, const float2* pf, float m, float r2)
        : P(p), Pf(pf), ox(pf[0].x), oy(pf[0].y), tol(2.0f * (4e-6f * r2 + 1e-13f * (m * sqrtf(r2))) + 1e-30f),
          tol2(4e-12f * r2 + 4e-13f * (m * sqrtf(r2)) + 1e-30f)
    {
    }
    __device__ __forceinline__ float af(int a, int b, int c) const
    {
        const float ax = Pf[a].x - ox, ay = Pf[a].y - oy;
        const float bx = Pf[b].x - ox, by = Pf[b].y - oy;
        const float cx = Pf[c].x - ox, cy = Pf[c].y - oy;
        return fabsf((ax * (by - cy) + bx * (cy - ay) + cx * (ay - by)) * 0.5f);
    }
    __device__ __forceinline__ bool gt(int a1, int b1, int c1, int a2, int b2, int c2) const
    {
        const float d = af(a1, b1, c1) - af(a2, b2, c2);
        if (d > tol)
            return true;
        if (d < -tol)
            return false;
        return area_order_near(P, Pf, tol2, a1, b1, c1, a2, b2, c2) > 0;
    }
    __device__ __forceinline__ bool eq(int a1, int b1, int c1, int a2, int b2, int c2) const
    {
        if (fabsf(af(a1, b1, c1) - af(a2, b2, c2)) > tol)
            return false;
        return area_order_near(P, Pf, tol2, a1, b1, c1, a2, b2, c2) == 0;
    }
};

template <typename Cmp>
__device__ __noinline__ int antipodal_pairs(const Cmp& cmp, int n, int2* pairs, int cap)
{
    int np = 0;
    if (n < 2)
        return 0;
    auto nx = [n](int i) { return (i + 1 == n) ? 0 : i + 1; };
    auto push = [&](int a, int b) {
        if (np < cap)
            pairs[np] = make_int2(a, b);
        ++np;
    };
    const int i0 = n - 1;
    int i = 0, j = 1;
    int guard = 0;
    // areaOfTriangle(i, i+1, j+1) > areaOfTriangle(i, i+1, j)
    while (cmp.gt(i, nx(i), nx(j), i, nx(i), j) && guard++ < 4 * n + 8)
        j = nx(j);
    const int j0 = j;
    guard = 0;
    while (i != j0 && guard++ < 4 * n + 8)
    {
        i = nx(i);
        push(i, j);
        int g2 = 0;
        while (cmp.gt(i, nx(i), nx(j), i, nx(i), j) && g2++ < 4 * n + 8)
        {
            j = nx(j);
            if (!(i == j0 && j == i0))
                push(i, j);
            else
                return np;
        }
        if (cmp.eq(j, nx(i), nx(j), i, nx(i), j))
        {
            if (!(i == j0 && j == i0))
                push(i, nx(j));
            else
                push(nx(i), j);
        }
    }
    return np;
}

__device__ __forceinline__ float warp_min_f(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_max_f(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Rotating calipers (polygonizer.cpp:165-278) by one warp: all lanes return the same box.
__device__ __noinline__ void calipers_warp(const double2* P, int n, const int2* pairs, int npairs, lp_bounding_box* out)
{
    const uint32_t lane = lane_id();
    lp_bounding_box box;
    for (int k = 0; k < 4; ++k)
        box.corners[k][0] = box.corners[k][1] = 0.0;
    box.area = 0.0f;
    box.angle_rad = 0.0f;
    box.is_valid = 0;
    if (n < 3)
    {
        if (lane == 0)
            *out = box;
        return;
    }
    double cx = 0.0, cy = 0.0;
    for (int k = 0; k < n; ++k)
    {
        cx += P[k].x;
        cy += P[k].y;
    }
    cx = div_d(cx, n);
    cy = div_d(cy, n);
    float best = __double2float_rn(DBL_MAX); // BoundingBox::area is a float: DBL_MAX -> +inf
    for (int pi = 0; pi < npairs; ++pi)
    {
        const int2 pr = pairs[pi];
        for (int e = 0; e < 2; ++e)
        {
            const int index = e == 0 ? pr.x : pr.y;
            for (int o = 0; o < 2; ++o)
            {
                int nb = index + (o == 0 ? -1 : 1);
                if (nb < 0)
                    nb += n;
                else if (nb >= n)
                    nb -= n;
                const double ex = P[nb].x - P[index].x;
                const double ey = P[nb].y - P[index].y;
                const double len = sqrt_d(ex * ex + ey * ey);
                if (len < 1.0e-6)
                    continue;
                const double ux = div_d(ex, len), uy = div_d(ey, len);
                double mnx = DBL_MAX, mxx = -DBL_MAX, mny = DBL_MAX, mxy = -DBL_MAX;
                for (int k = static_cast<int>(lane); k < n; k += 32)
                {
                    const double tx = P[k].x - cx, ty = P[k].y - cy;
                    const double rx = tx * ux + ty * uy;
                    const double ry = -tx * uy + ty * ux;
                    mnx = min_d(mnx, rx);
                    mxx = max_d(mxx, rx);
                    mny = min_d(mny, ry);
                    mxy = max_d(mxy, ry);
                }
                mnx = warp_min_d(mnx);
                mxx = warp_max_d(mxx);
                mny = warp_min_d(mny);
                mxy = warp_max_d(mxy);
                const double area = (mxx - mnx) * (mxy - mny);
                if (area < static_cast<double>(best))
                {
                    best = __double2float_rn(area);
                    box.area = best;
                    box.corners[0][0] = mnx * ux - mny * uy + cx;
                    box.corners[0][1] = mnx * uy + mny * ux + cy;
                    box.corners[1][0] = mxx * ux - mny * uy + cx;
                    box.corners[1][1] = mxx * uy + mny * ux + cy;
                    box.corners[2][0] = mxx * ux - mxy * uy + cx;
                    box.corners[2][1] = mxx * uy + mxy * ux + cy;
                    box.corners[3][0] = mnx * ux - mxy * uy + cx;
                    box.corners[3][1] = mnx * uy + mxy * ux + cy;
                    box.angle_rad = lpm::atan2_approx(__double2float_rn(uy), __double2float_rn(ux));
                    box.is_valid = 1;
                }
            }
        }
    }
    if (lane == 0)
        *out = box;
}

// Principal components of the 2x2 covariance as the reference gets them: V of Eigen 3.4's
// JacobiSVD (svd_.compute, polygonizer.cpp:326), in binary64 and in that library's operation order
// (this file is compiled without multiply-add contraction), so the axes are bit-identical to the
// host's. Steps: divide by the largest |coefficient|; while an off-diagonal entry exceeds
// max(DBL_MIN, 2 eps max|diagonal|), a left rotation symmetrises the (1, 0) block and a Jacobi
// rotation diagonalises it (W rotated on both sides, V on the right); columns ordered by
// descending |diagonal| with a strict comparison. Below the threshold nothing rotates, so a
// near-diagonal covariance keeps the identity axes. Sweeps stop after 64 (one or two in practice;
// the library loops until the test passes). Returns false for a non-finite covariance (the
// library's InvalidInput: the reference's box stays invalid, :327-330).
struct Rot2
{
    double c, s;
};

__device__ __forceinline__ void rot2_apply(double& x0, double& x1, double& y0, double& y1, Rot2 r)
{
    if (r.c == 1.0 && r.s == 0.0)
        return;
    const double a0 = x0, a1 = x1, b0 = y0, b1 = y1;
    x0 = r.c * a0 + r.s * b0;
    x1 = r.c * a1 + r.s * b1;
    y0 = -r.s * a0 + r.c * b0;
    y1 = -r.s * a1 + r.c * b1;
}

__device__ bool pca_axes(double sxx, double sxy, double syy, double& v00, double& v01, double& v10, double& v11)
{
    if (!(isfinite(sxx) && isfinite(sxy) && isfinite(syy)))
        return false;
    double scale = max_d(max_d(fabs(sxx), fabs(sxy)), fabs(syy));
    if (scale == 0.0)
        scale = 1.0;
    // the divisions by the scale on lanes 0, 1 and 2 (one division sequence)
    const uint32_t lane = lane_id();
    const double wq = div_d(((lane == 0u) ? sxx : ((lane == 1u) ? sxy : syy)), scale);
    double w00 = __shfl_sync(0xffffffffu, wq, 0), w01 = __shfl_sync(0xffffffffu, wq, 1), w10 = w01,
           w11 = __shfl_sync(0xffffffffu, wq, 2);
    v00 = 1.0, v01 = 0.0, v10 = 0.0, v11 = 1.0;
    const double precision = 2.0 * DBL_EPSILON;
    double max_diag = max_d(fabs(w00), fabs(w11));
#pragma unroll 1
    for (int sweep = 0; sweep < 64; ++sweep)
    {
        const double threshold = max_d(DBL_MIN, precision * max_diag);
        if (!(fabs(w10) > threshold || fabs(w01) > threshold))
            break;
        // block of the index pair (1, 0): m = [[W11, W10], [W01, W00]]
        double m00 = w11, m01 = w10, m10 = w01, m11 = w00;
        Rot2 r1{1.0, 0.0};
        const double t = m00 + m11, d = m10 - m01;
        if (!(fabs(d) < DBL_MIN))
        {
            const double u = div_d(t, d);
            const double tmp = sqrt_d(1.0 + u * u);
            r1 = Rot2{div_d(u, tmp), div_d(1.0, tmp)};
        }
        rot2_apply(m00, m01, m10, m11, r1);
        Rot2 rr{1.0, 0.0}; // the Jacobi rotation of [[m00, m01], [m01, m11]]
        const double deno = 2.0 * fabs(m01);
        if (!(deno < DBL_MIN))
        {
            const double tau = div_d(m00 - m11, deno);
            const double w = sqrt_d(tau * tau + 1.0);
            const double tt = div_d(1.0, tau > 0.0 ? tau + w : tau - w);
            const double sign_t = tt > 0.0 ? 1.0 : -1.0;
            const double n = div_d(1.0, sqrt_d(tt * tt + 1.0));
            rr = Rot2{n, -sign_t * copysign(1.0, m01) * fabs(tt) * n}; // (m01 / |m01|, m01 finite and not zero)
        }
        const Rot2 rl{r1.c * rr.c - r1.s * -rr.s, r1.c * -rr.s + r1.s * rr.c}; // r1 composed with rr^T
        const Rot2 rt{rr.c, -rr.s};
        rot2_apply(w10, w11, w00, w01, rl); // rows 1 and 0 of W
        rot2_apply(w01, w11, w00, w10, rt); // columns 1 and 0 of W
        rot2_apply(v01, v11, v00, v10, rt); // columns 1 and 0 of V
        max_diag = max_d(max_d(max_diag, fabs(w11)), fabs(w00));
    }
    if (fabs(w11) * scale > fabs(w00) * scale)
    {
        const double a = v00, b = v10;
        v00 = v01;
        v10 = v11;
        v01 = a;
        v11 = b;
    }
    return true;
}

// No box: every field zero, by one warp.
__device__ __forceinline__ void no_box(lp_bounding_box* out)
{
    const uint32_t lane = lane_id();
    if (lane < 8u)
        out->corners[lane >> 1][lane & 1u] = 0.0;
    if (lane == 0)
    {
        out->area = 0.0f;
        out->angle_rad = 0.0f;
        out->is_valid = 0;
    }
}

// Sums of the x and of the y coordinates of P[0..n) as the reference's loop computes them in
// binary64 (left to right), by one warp; every lane returns both. Each term is a multiple of
// 2^g (g from its exponent and the trailing zeros of its significand) and below 2^t in
// magnitude; when log2(n) + max t - min g <= 53 every partial sum of any order is exact, so a warp
// tree gives the loop's result. Otherwise (tiny next to large coordinates) the loop runs as written.
__device__ __noinline__ void sum_xy_fp64(const double2* P, int n, double& sx, double& sy)
{
    const uint32_t lane = lane_id();
    int tmax = -4096, gmin = 4096;
    bool ok = true;
    double px = 0.0, py = 0.0;
    auto scan = [&](double v) {
        const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(v));
        const int e = static_cast<int>((u >> 52) & 0x7ffull);
        if ((u << 1) == 0ull)
            return; // zero
        if (e == 0 || e == 0x7ff)
        {
            ok = false; // subnormal, infinite or nan
            return;
        }
        const unsigned long long m = (u & 0xfffffffffffffull) | (1ull << 52);
        tmax = max(tmax, e - 1022);
        gmin = min(gmin, e - 1075 + (__ffsll(static_cast<long long>(m)) - 1));
    };
#pragma unroll 1
    for (int k = static_cast<int>(lane); k < n; k += 32)
    {
        scan(P[k].x);
        scan(P[k].y);
        px += P[k].x;
        py += P[k].y;
    }
    ok = __all_sync(0xffffffffu, ok);
    tmax = __reduce_max_sync(0xffffffffu, tmax);
    gmin = __reduce_min_sync(0xffffffffu, gmin);
    const int lg = 32 - __clz(n); // >= log2(n)
    if (ok && lg + tmax - gmin <= 53)
    {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
        {
            px += __shfl_xor_sync(0xffffffffu, px, o);
            py += __shfl_xor_sync(0xffffffffu, py, o);
        }
        sx = px;
        sy = py;
        return;
    }
    sx = 0.0;
    sy = 0.0;
#pragma unroll 1
    for (int k = 0; k < n; ++k)
    {
        sx += P[k].x;
        sy += P[k].y;
    }
}

// PCA box by one warp, every step in FP64 in the reference's order: the mean, the covariance sums
// (the principal axis is ill-conditioned exactly where they nearly cancel), the JacobiSVD axes
// (pca_axes, evaluated by every lane alike), the rotated extents (lanes stride over the vertices;
// min and max do not depend on order) and the corners. The box equals the reference loop's bit
// for bit.
__device__ __noinline__ void pca_box_warp(const double2* P, int n, lp_bounding_box* out)
{
    const uint32_t lane = lane_id();
    if (n >= 3)
    {
        double sx, sy;
        sum_xy_fp64(P, n, sx, sy);
        // mx = sx / n and my = sy / n on lanes 0 and 1 (one division sequence)
        const double mq = div_d((lane & 1u) ? sy : sx, static_cast<double>(n));
        const double mx = __shfl_sync(0xffffffffu, mq, 0), my = __shfl_sync(0xffffffffu, mq, 1);
        // the three covariance sums keep the reference's order: the products of vertex k come from
        // lane k mod 32, lanes 0, 1 and 2 accumulate sxx, sxy and syy in one instruction per step
        double acc = 0.0;
#pragma unroll 1
        for (int base = 0; base < n; base += 32)
        {
            const int k = base + static_cast<int>(lane);
            double txx = 0.0, txy = 0.0, tyy = 0.0;
            if (k < n)
            {
                const double dx = P[k].x - mx, dy = P[k].y - my;
                txx = dx * dx;
                txy = dx * dy;
                tyy = dy * dy;
            }
            const int cnt = min(32, n - base);
#pragma unroll 2
            for (int j = 0; j < cnt; ++j)
            {
                const double a0 = __shfl_sync(0xffffffffu, txx, j);
                const double a1 = __shfl_sync(0xffffffffu, txy, j);
                const double a2 = __shfl_sync(0xffffffffu, tyy, j);
                acc += (lane == 0u) ? a0 : ((lane == 1u) ? a1 : a2);
            }
        }
        const double cq = div_d(acc, static_cast<double>(n - 1));
        const double sxx = __shfl_sync(0xffffffffu, cq, 0), sxy = __shfl_sync(0xffffffffu, cq, 1),
                     syy = __shfl_sync(0xffffffffu, cq, 2);
        double v00, v01, v10, v11;
        if (pca_axes(sxx, sxy, syy, v00, v01, v10, v11))
        {
            double mnx = DBL_MAX, mxx = -DBL_MAX, mny = DBL_MAX, mxy = -DBL_MAX;
#pragma unroll 1
            for (int i = static_cast<int>(lane); i < n; i += 32)
            {
                const double dx = P[i].x - mx, dy = P[i].y - my;
                const double rx = dx * v00 + dy * v10;
                const double ry = dx * v01 + dy * v11;
                mnx = min_d(mnx, rx);
                mxx = max_d(mxx, rx);
                mny = min_d(mny, ry);
                mxy = max_d(mxy, ry);
            }
            mnx = warp_min_d(mnx);
            mxx = warp_max_d(mxx);
            mny = warp_min_d(mny);
            mxy = warp_max_d(mxy);
            // coordinate c of corner k from lane 2 k + c (one sequence for all eight)
            const int k = static_cast<int>(lane >> 1) & 3;
            const bool cy = (lane & 1u) != 0u;
            const double xk = (k == 1 || k == 2) ? mxx : mnx, yk = (k >= 2) ? mxy : mny;
            const double at = xk * (cy ? v10 : v00) + yk * (cy ? v11 : v01) + (cy ? my : mx);
            if (lane < 8u)
                out->corners[k][cy] = at;
            if (lane == 0)
            {
                out->area = __double2float_rn((mxx - mnx) * (mxy - mny));
                out->angle_rad = __double2float_rn(atan2(v10, v00));
                out->is_valid = 1;
            }
            return;
        }
    }
    no_box(out);
}

// FP64 rotated extents of P about (cx, cy) for the unit direction (ux, uy), by one warp.
__device__ __noinline__ void extents_fp64(const double2* P, int n, double cx, double cy, double ux, double uy,
                                             double& mnx, double& mxx, double& mny, double& mxy)
{
    mnx = DBL_MAX, mxx = -DBL_MAX, mny = DBL_MAX, mxy = -DBL_MAX;
#pragma unroll 1
    for (int k = static_cast<int>(lane_id()); k < n; k += 32)
    {
        const double tx = P[k].x - cx, ty = P[k].y - cy;
        const double rx = tx * ux + ty * uy;
        const double ry = -tx * uy + ty * ux;
        mnx = min_d(mnx, rx);
        mxx = max_d(mxx, rx);
        mny = min_d(mny, ry);
        mxy = max_d(mxy, ry);
    }
    mnx = warp_min_d(mnx);
    mxx = warp_max_d(mxx);
    mny = warp_min_d(mny);
    mxy = warp_max_d(mxy);
}

// Rotating calipers with the candidate boxes screened in FP32 (same result as calipers_warp).
//
// The reference walks the edges named by the antipodal pairs and keeps a box when its FP64 area
// is below the float `best` of the boxes kept so far. An edge's box is the same for both
// directions of the edge (every term only changes sign, exactly), so it is evaluated once per
// hull edge j (P[j] -> P[j+1]): ea[j] = FP32 area, within e = 1e-4 R^2 of the FP64 area (the
// rounding of the float frame, direction and extents stays below 6e-6 R^2, R = largest
// |P - P[0]|). Edges with ea[j] <= T are the contenders, with T grown from the smallest ea until
// no other edge lies within G = 2e + 1e-6 (T + 2e) above it. Every other edge then has a float
// area above every contender's FP64 area and above the float of the smallest area, so (i) the
// last box the reference keeps is a contender's and (ii) replaying the reference's walk over the
// contenders alone, with their FP64 areas, keeps the same boxes among them. Each contender's FP64
// extents are kept by one lane; the winner's corners come from them, negated for the reverse
// direction (exact), so they are the reference's. The skip test (edge length < 1e-6) is screened
// in FP32 too (|float len^2 - len^2| < 2^-21 len^2) and evaluated in FP64 only near 1e-12.
// Only the edges the walk visits take part (an unvisited edge's area is +inf): a pair walk that
// misses a vertex never looks at its edges, and a contender set made only of unvisited edges
// would leave no box where the reference keeps one.
// Up to 32 contenders (one per lane) are handled; more fall back to calipers_warp.
__device__ __noinline__ void calipers_fast(const double2* P, const float2* Pf, int n, const int2* pairs, int npairs, float* ea,
                              float r2, lp_bounding_box* out)
{
    const uint32_t lane = lane_id();
    if (n < 3)
    {
        no_box(out);
        return;
    }
    const float ox = Pf[0].x, oy = Pf[0].y;
    const float e = 1e-4f * r2 + 1e-30f;
    // Only edges the walk visits can hold the reference's box: on a near-degenerate hull the pair
    // walk can miss a vertex, and with it an edge that may have the smallest area. Mark the
    // visited edges (ea[j] = 0, the edge mapping of `visit` below) before choosing contenders.
#pragma unroll 1
    for (int j = static_cast<int>(lane); j < n; j += 32)
        ea[j] = -1.0f;
    __syncwarp();
#pragma unroll 1
    for (int v = static_cast<int>(lane); v < 4 * npairs; v += 32)
    {
        const int2 pr = pairs[v >> 2];
        const int index = ((v >> 1) & 1) ? pr.y : pr.x;
        ea[(v & 1) ? index : ((index == 0) ? n - 1 : index - 1)] = 0.0f; // offset +1: edge index; -1: index - 1
    }
    __syncwarp();
    float amin = INFINITY;
#pragma unroll 1
    for (int j = static_cast<int>(lane); j < n; j += 32)
    {
        const int j1 = (j + 1 == n) ? 0 : j + 1;
        const float fx = Pf[j1].x - Pf[j].x, fy = Pf[j1].y - Pf[j].y;
        const float fl2 = fx * fx + fy * fy;
        bool skip = fl2 < 0.9999e-12f || ea[j] != 0.0f; // unvisited edges never compete
        if (!skip && !(fl2 > 1.0001e-12f))
        {
            const double dx = P[j1].x - P[j].x, dy = P[j1].y - P[j].y;
            skip = sqrt_d(dx * dx + dy * dy) < 1.0e-6;
        }
        float a = INFINITY; // edges the reference skips never compete
        if (!skip)
        {
            const float fl = sqrtf(fl2);
            const float ux = fx / fl, uy = fy / fl;
            float mnx = INFINITY, mxx = -INFINITY, mny = INFINITY, mxy = -INFINITY;
#pragma unroll 2
            for (int k = 0; k < n; ++k)
            {
                const float tx = Pf[k].x - ox, ty = Pf[k].y - oy;
                const float rx = tx * ux + ty * uy;
                const float ry = -tx * uy + ty * ux;
                mnx = fminf(mnx, rx);
                mxx = fmaxf(mxx, rx);
                mny = fminf(mny, ry);
                mxy = fmaxf(mxy, ry);
            }
            a = (mxx - mnx) * (mxy - mny);
        }
        ea[j] = a;
        amin = fminf(amin, a);
    }
    amin = warp_min_f(amin);
    __syncwarp();
    if (amin == INFINITY)
    {
        no_box(out); // every edge is skipped, as in the reference
        return;
    }
    float T = amin;
#pragma unroll 1
    for (int it = 0; it <= n; ++it)
    {
        const float G = 2.0f * e + 1e-6f * (T + 2.0f * e);
        float nt = T;
    #pragma unroll 1
    for (int j = static_cast<int>(lane); j < n; j += 32)
            if (ea[j] > T && ea[j] <= T + G)
                nt = fmaxf(nt, ea[j]);
        nt = warp_max_f(nt);
        if (nt == T)
            break;
        T = nt;
    }
    // FP64 centroid of the hull vertices, as the reference's loop sums them
    double sx, sy;
    sum_xy_fp64(P, n, sx, sy);
    const double cq = div_d((lane & 1u) ? sy : sx, static_cast<double>(n));
    const double cx = __shfl_sync(0xffffffffu, cq, 0), cy = __shfl_sync(0xffffffffu, cq, 1);
    // contender c (in edge order) is held by lane c: its edge, direction, FP64 extents and area
    int my_j = -1;
    int ncont = 0;
#pragma unroll 1
    for (int base = 0; base < n; base += 32)
    {
        const int j = base + static_cast<int>(lane);
        const uint32_t mask = __ballot_sync(0xffffffffu, j < n && ea[j] <= T);
#pragma unroll 1
        for (uint32_t mm = mask; mm != 0u; mm &= mm - 1u, ++ncont)
            if (static_cast<int>(lane) == ncont) // contender ncont goes to lane ncont
                my_j = base + __ffs(mm) - 1;
        if (ncont > 32)
            break;
    }
    if (ncont > 32)
    {
        calipers_warp(P, n, pairs, npairs, out);
        return;
    }
    // each contender's unit direction on its own lane (one square root and division sequence)
    double my_ux = 0.0, my_uy = 0.0, my_mnx = 0.0, my_mxx = 0.0, my_mny = 0.0, my_mxy = 0.0, my_area = 0.0;
    if (my_j >= 0)
    {
        const int j1 = (my_j + 1 == n) ? 0 : my_j + 1;
        const double ex = P[j1].x - P[my_j].x, ey = P[j1].y - P[my_j].y;
        const double len = sqrt_d(ex * ex + ey * ey);
        my_ux = div_d(ex, len);
        my_uy = div_d(ey, len);
    }
#pragma unroll 1
    for (int c = 0; c < ncont; ++c)
    {
        const double ux = __shfl_sync(0xffffffffu, my_ux, c), uy = __shfl_sync(0xffffffffu, my_uy, c);
        double mnx, mxx, mny, mxy;
        extents_fp64(P, n, cx, cy, ux, uy, mnx, mxx, mny, mxy);
        if (static_cast<int>(lane) == c)
        {
            my_mnx = mnx;
            my_mxx = mxx;
            my_mny = mny;
            my_mxy = mxy;
            my_area = (mxx - mnx) * (mxy - mny);
        }
    }
    // The reference's walk over the contenders. Its float `best` only ever takes contenders' float
    // areas F = fl32(A), and rounding is monotone, so a visit's test A < (double)best is F < best,
    // or at F == best the contender's bit `below` = (A < (double)F). The final best is therefore
    // the smallest F of all visits, and the kept box is the last visit with that F which passes:
    // the first one (it meets a larger best; at F = +inf only with `below`) and every later one
    // with `below`. Each lane takes every 32nd visit (pair pi, side e2, neighbour o).
    float my_f = INFINITY;
    int my_below = 0;
    if (my_j >= 0)
    {
        my_f = __double2float_rn(my_area);
        my_below = my_area < static_cast<double>(my_f);
    }
    const int nvis = 4 * npairs;
    auto visit = [&](int v, int& j, bool& rev, float& f, int& below) {
        const int2 pr = pairs[v >> 2];
        const int index = ((v >> 1) & 1) ? pr.y : pr.x;
        const int o = v & 1;
        int nb = index + (o == 0 ? -1 : 1);
        if (nb < 0)
            nb += n;
        else if (nb >= n)
            nb -= n;
        j = (o == 1) ? index : nb; // hull edge j joins P[j] and P[j+1]
        rev = (o == 0);            // walked from P[j+1] to P[j]
        const bool cont = ea[j] <= T;
        f = INFINITY;
        below = 0;
#pragma unroll 1
        for (int c = 0; c < ncont; ++c)
        {
            const int jc = __shfl_sync(0xffffffffu, my_j, c);
            const float fc = __shfl_sync(0xffffffffu, my_f, c);
            const int bc = __shfl_sync(0xffffffffu, my_below, c);
            if (cont && j == jc)
            {
                f = fc;
                below = bc;
            }
        }
        return cont;
    };
    float fmin = INFINITY;
    bool any = false;
#pragma unroll 1
    for (int v0 = 0; v0 < nvis; v0 += 32)
    {
        const int v = v0 + static_cast<int>(lane);
        int j, below;
        bool rev;
        float f;
        const bool cont = visit(min(v, nvis - 1), j, rev, f, below) && v < nvis;
        if (cont)
            fmin = fminf(fmin, f);
        any |= cont;
    }
    fmin = warp_min_f(fmin);
    any = __any_sync(0xffffffffu, any);
    int first = INT32_MAX, lastb = -1;
#pragma unroll 1
    for (int v0 = 0; any && v0 < nvis; v0 += 32)
    {
        const int v = v0 + static_cast<int>(lane);
        int j, below;
        bool rev;
        float f;
        const bool cont = visit(min(v, nvis - 1), j, rev, f, below) && v < nvis;
        if (cont && f == fmin)
        {
            first = min(first, v);
            if (below)
                lastb = max(lastb, v);
        }
    }
    first = static_cast<int>(__reduce_min_sync(0xffffffffu, static_cast<unsigned>(first)));
    lastb = static_cast<int>(__reduce_max_sync(0xffffffffu, static_cast<unsigned>(lastb + 1))) - 1;
    const int win = (lastb >= 0) ? lastb : ((any && fmin < INFINITY) ? first : -1);
    float best = __double2float_rn(DBL_MAX);
    int wj = -1;
    bool wrev = false;
    if (win >= 0)
    {
        int below;
        float f;
        visit(win, wj, wrev, f, below);
        best = fmin;
    }
    if (wj >= 0)
    {
        const int src = __ffs(__ballot_sync(0xffffffffu, my_j == wj)) - 1;
        double ux = __shfl_sync(0xffffffffu, my_ux, src), uy = __shfl_sync(0xffffffffu, my_uy, src);
        double mnx = __shfl_sync(0xffffffffu, my_mnx, src), mxx = __shfl_sync(0xffffffffu, my_mxx, src);
        double mny = __shfl_sync(0xffffffffu, my_mny, src), mxy = __shfl_sync(0xffffffffu, my_mxy, src);
        if (wrev)
        {
            // reverse direction: u and every projection change sign exactly
            ux = -ux;
            uy = -uy;
            const double a0 = mnx, a1 = mny;
            mnx = -mxx;
            mxx = -a0;
            mny = -mxy;
            mxy = -a1;
        }
        // coordinate c of corner k from lane 2 k + c (one sequence for all eight): x ux - y uy + cx and
        // x uy + y ux + cy
        const int k = static_cast<int>(lane >> 1) & 3;
        const bool yy = (lane & 1u) != 0u;
        const double xk = (k == 1 || k == 2) ? mxx : mnx, yk = (k >= 2) ? mxy : mny;
        const double at = xk * (yy ? uy : ux) + (yy ? yk * ux : -(yk * uy)) + (yy ? cy : cx);
        if (lane < 8u)
            out->corners[k][yy] = at;
        if (lane == 0)
        {
            out->area = best;
            out->angle_rad = lpm::atan2_approx(__double2float_rn(uy), __double2float_rn(ux));
            out->is_valid = 1;
        }
        return;
    }
    no_box(out);
}

// Antipodal pairs and the rotating-calipers box of hull P (h vertices) by one warp. With float
// copies Pf and h floats of scratch ea the comparisons are screened in FP32; without them
// (Pf == nullptr) everything runs in FP64.
__device__ __noinline__ void calipers_box(ScanState* st, const double2* P, const float2* Pf, float* ea, int h, int2* pairs,
                             lp_bounding_box* out)
{
    const uint32_t lane = lane_id();
    const int cap = 4 * h + 16;
    int npairs = 0;
    if (Pf != nullptr)
    {
        const float ox = Pf[0].x, oy = Pf[0].y;
        float r2 = 0.0f, mabs = 0.0f;
        for (int k = static_cast<int>(lane); k < h; k += 32)
        {
            const float lx = Pf[k].x - ox, ly = Pf[k].y - oy;
            r2 = fmaxf(r2, lx * lx + ly * ly);
            mabs = fmaxf(mabs, fmaxf(fabsf(Pf[k].x), fabsf(Pf[k].y)));
        }
        r2 = warp_max_f(r2) * 1.001f;
        mabs = warp_max_f(mabs);
        if (lane == 0)
            npairs = antipodal_pairs(AreaCmpFiltered(P, Pf, mabs, r2), h, pairs, cap);
        npairs = __shfl_sync(0xffffffffu, npairs, 0);
        if (npairs > cap)
        {
            if (lane == 0)
                raise_err(st, ERR_INTERNAL);
            npairs = cap;
        }
        __syncwarp();
        calipers_fast(P, Pf, h, pairs, npairs, ea, r2, out);
    }
    else
    {
        if (lane == 0)
            npairs = antipodal_pairs(AreaCmpFp64{P}, h, pairs, cap);
        npairs = __shfl_sync(0xffffffffu, npairs, 0);
        if (npairs > cap)
        {
            if (lane == 0)
                raise_err(st, ERR_INTERNAL);
            npairs = cap;
        }
        __syncwarp();
        calipers_warp(P, h, pairs, npairs, out);
    }
}

// u * v has an exact binary32 error term: the product neither underflows nor overflows (an infinite one
// would compare as equal to any other).
__device__ __forceinline__ bool prod_err_exact(float u, float v, float t)
{
    return fabsf(t) <= FLT_MAX && (fabsf(t) >= 1e-30f || u == 0.0f || v == 0.0f);
}

// The near-ties of chain_pops, out of line: along an exactly straight wall every test is one.
__device__ __noinline__ bool ccw_or_colinear_near(float ax, float ay, float bx, float by, float cx, float cy)
{
    const float u = bx - ax, v = cy - ay, w = by - ay, z = cx - ax;
    const float t1 = u * v;
    const float t2 = w * z;
    if (prod_err_exact(u, v, t1) && prod_err_exact(w, z, t2))
    {
        const float ul = diff_err(bx, ax, u), vl = diff_err(cy, ay, v), wl = diff_err(by, ay, w), zl = diff_err(cx, ax, z);
        const float e1 = __fmaf_rn(u, v, -t1), e2 = __fmaf_rn(w, z, -t2);
        // When the four differences are exact binary32 values, each product of two of them
        // is exact in binary64 (48 significant bits), so the binary64 expression has the sign
        // of u v - w z exactly. Rounding to binary32 is monotone, so t1 < t2 implies u v < w z (and
        // t1 > t2 the converse); at t1 == t2 the difference is e1 - e2, the exact product errors.
        if (ul == 0.0f && vl == 0.0f && wl == 0.0f && zl == 0.0f)
            return t1 != t2 ? t1 < t2 : e1 <= e2;
        // Otherwise the products of the exact two-term differences up to their last cross term: t + e + (u vl +
        // ul v) errs by less than 2^-46 |t| (the dropped ul vl is below 2^-48, each rounding of the small
        // terms too), t1 - t2 is exact (both lie within 2^-20 of each other), the sums of the small terms
        // round by less than 2^-46 (|t1| + |t2|): beyond 2^-42 of that sum, the sign is the exact one, and
        // the binary64 expression, within 3 * 2^-53 of it, has it too.
        const float d = (t1 - t2) + ((e1 + (u * vl + ul * v)) - (e2 + (w * zl + wl * z)));
        if (fabsf(d) > 2.2737367544323206e-13f * (fabsf(t1) + fabsf(t2)))
            return d < 0.0f;
    }
    return ccw_or_colinear(ax, ay, bx, by, cx, cy);
}

// Does the candidate c pop b (a below it)? Decided in FP32 when the float determinant exceeds 2^-21 (|t1| +
// |t2|) in magnitude (its rounding error stays below 6 * 2^-24 of that sum, the FP64 form's below
// 3 * 2^-53); `near`: it does not, ask chain_pops_near.
__device__ __forceinline__ bool chain_pops(float ax, float ay, float bx, float by, float cx, float cy, bool& near)
{
    const float u = bx - ax, v = cy - ay, w = by - ay, z = cx - ax;
    const float t1 = u * v;
    const float t2 = w * z;
    const float d = t1 - t2;
    near = !(fabsf(d) > (fabsf(t1) + fabsf(t2)) * 4.76837158203125e-7f + 1e-30f);
    return d < 0.0f;
}
__device__ __forceinline__ bool chain_pops_near(float ax, float ay, float bx, float by, float cx, float cy)
{
    return ccw_or_colinear_near(ax, ay, bx, by, cx, cy);
}
__device__ __forceinline__ bool chain_pops(double ax, double ay, double bx, double by, double cx, double cy, bool& near)
{
    near = false;
    return ccw_or_colinear(ax, ay, bx, by, cx, cy);
}
__device__ __forceinline__ bool chain_pops_near(double ax, double ay, double bx, double by, double cx, double cy)
{
    return ccw_or_colinear(ax, ay, bx, by, cx, cy);
}

// One half of the monotone chain over sorted candidates C[0..m) (polygonizer.cpp:62-88) by W lanes
// (32: a warp; 16: half of one, the other half walks the other half of the chain): the lower
// half walks C forwards, the upper half backwards from C[m - 1]. The reference's
// second loop continues on the stack of the first but never pops below C[m - 1] (its k >= t
// test), so the upper half is the same walk on its own stack starting from that point. Writes the stack
// to S, returns its size.
// The walk is a chain of orientation tests, each a chain of its own: one thread took 400 cycles a candidate. Here lane l
// holds the l-th point from the top of the stack and the one below it, and tests whether the candidate pops it once
// those above are gone; the pops are the lanes up to the first that says no, so a candidate costs one test, a ballot and
// the shuffles, without a divergent branch (each costs some 40 cycles). Points deeper than W come back from memory when
// they are uncovered, and only the first lane that does not pop for certain has its near-tie decided.
template <int W, typename T>
__device__ __noinline__ int chain_half(const HPt<T>* C, int m, int* S, bool upper)
{
    const int l = static_cast<int>(lane_id()) & (W - 1);
    const int first = static_cast<int>(lane_id()) - l;
    int k = 0;
    T ax = T(0), ay = T(0), bx = T(0), by = T(0); // below, and the l-th from the top
    auto at = [&](int depth, T& x, T& y) { // the stack's entry `depth` from the bottom, if there is one
        if (depth >= 0)
        {
            const HPt<T> p = C[S[depth]];
            x = p.x;
            y = p.y;
        }
    };
    auto group = [&](uint32_t mask) { return (W == 32) ? mask : ((mask >> first) & ((1u << (W & 31)) - 1u)); };
    int i = upper ? m - 1 : 0;
    const int step = upper ? -1 : 1;
    HPt<T> next = (m > 0) ? C[i] : HPt<T>{};
    for (int j = 0; j < m; ++j, i += step)
    {
        const HPt<T> c = next;
        next = C[min(max(i + step, 0), m - 1)];
        const bool deep = (W == 32) ? k > W : __any_sync(0xffffffffu, k > W); // (only then can every lane pop)
        bool near, live = l + 1 < k;
        bool pop = chain_pops(ax, ay, bx, by, c.x, c.y, near);
        near = near & live;
        pop = pop & live & !near;
        const uint32_t keep = __ballot_sync(0xffffffffu, !pop), ties = __ballot_sync(0xffffffffu, near);
        int pops = __ffs(group(keep)) - 1;
        const uint32_t lowest = (W == 32) ? (keep & (0u - keep))
                                          : ((keep & (0u - keep)) | ((keep >> 16) & (0u - (keep >> 16))) << 16);
        if ((lowest & ties) != 0u || deep) // (the same for all lanes)
        {
            __syncwarp(); // the entries written so far, before they are read here and below
            for (;;)
            {
                if (near)
                    pop = chain_pops_near(ax, ay, bx, by, c.x, c.y);
                const uint32_t mine = group(__ballot_sync(0xffffffffu, !pop));
                pops = mine ? __ffs(mine) - 1 : W;
                if (!__any_sync(0xffffffffu, pops == W))
                    break;
                if (pops == W)
                {
                    k -= W;
                    at(k - 1 - l, bx, by);
                    at(k - 2 - l, ax, ay);
                    live = l + 1 < k;
                    pop = chain_pops(ax, ay, bx, by, c.x, c.y, near);
                    near = near & live;
                    pop = pop & live & !near;
                }
            }
        }
        k -= pops;
        const int own = l - 1 + pops, below = l + pops;
        T nx = __shfl_sync(0xffffffffu, bx, first + (own & (W - 1))), ny = __shfl_sync(0xffffffffu, by, first + (own & (W - 1)));
        T mx = __shfl_sync(0xffffffffu, bx, first + (below & (W - 1))),
          my = __shfl_sync(0xffffffffu, by, first + (below & (W - 1)));
        if (deep)
        {
            if (own >= W)
                at(k - l, nx, ny);
            if (below >= W)
                at(k - 1 - l, mx, my);
        }
        ax = mx;
        ay = my;
        bx = (l == 0) ? c.x : nx;
        by = (l == 0) ? c.y : ny;
        if (l == 0)
            S[k] = i;
        ++k;
    }
    __syncwarp();
    return k;
}

// Strictly left of a -> b by a relative margin of 1e-5: the float cross product errs by less
// than 2.4e-7 (|ex| + |ey|)(|qx| + |qy|), so a point passing is strictly left in exact arithmetic.
__device__ __forceinline__ bool left_strict_f(float ax, float ay, float bx, float by, float px, float py)
{
    const float ex = bx - ax, ey = by - ay, qx = px - ax, qy = py - ay;
    const float cr = ex * qy - ey * qx;
    const float scale = (fabsf(ex) + fabsf(ey)) * (fabsf(qx) + fabsf(qy));
    return cr > 1e-5f * scale + 1e-30f;
}

// Bitonic sort of n candidates (capacity next_pow2(n)) in global memory by one block.
template <typename T>
__device__ void block_sort_global(HPt<T>* a, uint32_t n)
{
    const uint32_t np2 = next_pow2(n);
    for (uint32_t k = n + threadIdx.x; k < np2; k += blockDim.x)
        a[k] = HPt<T>{static_cast<T>(INFINITY), static_cast<T>(INFINITY), 0xffffffffu};
    __syncthreads();
    for (uint32_t k = 2; k <= np2; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1)
        {
            for (uint32_t i = threadIdx.x; i < np2; i += blockDim.x)
            {
                const uint32_t ixj = i ^ j;
                if (ixj > i)
                {
                    const bool up = ((i & k) == 0);
                    const HPt<T> x = a[i], y = a[ixj];
                    if (up ? hpt_less(y, x) : hpt_less(x, y))
                    {
                        a[i] = y;
                        a[ixj] = x;
                    }
                }
            }
            __syncthreads();
        }
}

constexpr int kDirs = 16;         // extreme-point directions of the initial polygon
constexpr int kPolyCap = 256;     // refined polygon capacity
constexpr int kRefineRounds = 12; // farthest-point insertion rounds
constexpr int kCountLater = 128;   // hulls of at most this many vertices have a large cluster's members counted later
constexpr uint32_t kHullEnough = 96; // active members few enough to end them (a round costs about 30 candidates' sort and chain)
constexpr uint32_t kBigCluster = 512; // larger clusters take a whole CTA; smaller ones one warp

struct HullSmem
{
    HPt<float> cand[kHullSmem];
    int stack[2 * kHullSmem + 2];
    uint32_t hkey[kHullSmem]; // hull vertex member keys, sorted
    int32_t diff[kHullSmem + 1];
    float2 poly[kPolyCap];
    float2 poly2[kPolyCap];
    float4 erec[kPolyCap]; // refinement edge e: start point and direction
    float2 emar[kPolyCap]; // its inside and outside margins per unit of |q|_1
    unsigned long long pkey[kPolyCap];
    unsigned long long ext[kDirs][kHullThreads / 32];
    float2 dirs[kDirs];
    uint32_t scan[33];
    int npoly;
    int grew;
    int ncand;
    int nhull;
    uint32_t work;
};

__device__ __forceinline__ unsigned long long fkey_payload(float v, uint32_t i)
{
    return (static_cast<unsigned long long>(ford(v)) << 32) | i;
}

// A cluster's z range from the ordered keys the cluster scatter accumulates (max of ~ord(z), max
// of ord(z)).
__device__ __forceinline__ float zkey_unord(uint32_t u)
{
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}
__device__ __forceinline__ float zkey_min(uint32_t k)
{
    return zkey_unord(~k);
}
__device__ __forceinline__ float zkey_max(uint32_t k)
{
    return zkey_unord(k);
}

// Members extreme in the kDirs = 16 directions 2 pi d / 16 (counter-clockwise). Directions d and
// d + 8 are opposite, so eight projections give both: the largest along d, and for d + 8 the
// smallest along d. Any extreme member serves (the polygon only has to consist of members); ties
// keep the first member a thread sees and, across threads, the larger member position.
struct Extremes16
{
    float hi[8], lo[8];
    uint32_t ih[8], il[8];
    __device__ __forceinline__ void init()
    {
#pragma unroll
        for (int d = 0; d < 8; ++d)
        {
            hi[d] = -INFINITY;
            lo[d] = INFINITY;
            ih[d] = il[d] = 0u;
        }
    }
    __device__ __forceinline__ void add(const float2* dirs, float x, float y, uint32_t i)
    {
#pragma unroll
        for (int d = 0; d < 8; ++d)
        {
            const float v = x * dirs[d].x + y * dirs[d].y;
            if (v > hi[d])
            {
                hi[d] = v;
                ih[d] = i;
            }
            if (v < lo[d])
            {
                lo[d] = v;
                il[d] = i;
            }
        }
    }
    __device__ __forceinline__ unsigned long long key(int d) const
    {
        return d < 8 ? fkey_payload(hi[d], ih[d]) : fkey_payload(-lo[d - 8], il[d - 8]);
    }
    // The warp's largest key of direction d, on lane d (the other lanes: unspecified). Two integer
    // reductions a direction, of the value and of the positions that hold it.
    __device__ __forceinline__ unsigned long long warp_key() const
    {
        unsigned long long mine = 0ull;
#pragma unroll
        for (int d = 0; d < kDirs; ++d)
        {
            const unsigned long long k = key(d);
            const uint32_t v = static_cast<uint32_t>(k >> 32);
            const uint32_t top = __reduce_max_sync(0xffffffffu, v);
            const uint32_t at = __reduce_max_sync(0xffffffffu, v == top ? static_cast<uint32_t>(k) : 0u);
            if (static_cast<int>(lane_id()) == d)
                mine = (static_cast<unsigned long long>(top) << 32) | at;
        }
        return mine;
    }
};

// The polygon of the extreme members in direction order (counter-clockwise), repeats dropped, by one
// warp: lane d < kDirs holds direction d's key, so the members load side by side. Returns its size.
__device__ __forceinline__ int extreme_polygon(const float2* xy, uint32_t n, unsigned long long key, float2* poly)
{
    const uint32_t lane = lane_id();
    const uint32_t i = static_cast<uint32_t>(key);
    const uint32_t prev = __shfl_up_sync(0xffffffffu, i, 1);
    const bool take = n > 0u && lane < static_cast<uint32_t>(kDirs) && (lane == 0u || i != prev);
    const uint32_t mask = __ballot_sync(0xffffffffu, take);
    if (take)
        poly[__popc(mask & ((1u << lane) - 1u))] = xy[i];
    __syncwarp();
    int np = __popc(mask);
    if (np > 1 && poly[np - 1].x == poly[0].x && poly[np - 1].y == poly[0].y)
        --np;
    return np;
}

// Large clusters: the two passes over every member (the 16 direction extremes, the first
// refinement round against the polygon they span) run grid-wide before the hull kernel, in
// (cluster, chunk of kPreChunk members) items, so the cluster's CTA starts at the second round.
// Both reduce exactly (packed-key maxima; the survivors are a set, listed in any order), with
// the hull kernel's expressions, so the hull kernel continues from the same state.
constexpr uint32_t kPreMin = 8192;
constexpr uint32_t kPreChunk = 4096;

__device__ __forceinline__ void hull_dirs(float2* dirs)
{
    if (threadIdx.x < kDirs)
    {
        const float a = 6.28318530717958647692f * static_cast<float>(threadIdx.x) / kDirs;
        dirs[threadIdx.x] = make_float2(cosf(a), sinf(a));
    }
}

// The first polygon from the extremes' packed keys: extreme members in direction order (counter-
// clockwise), repeats dropped. Thread 0.
__device__ int first_polygon(const float2* xy, uint32_t n, const unsigned long long* best, float2* poly)
{
    int np = 0;
    uint32_t prev = 0xffffffffu;
    for (int d = 0; d < kDirs; ++d)
    {
        const uint32_t i = static_cast<uint32_t>(best[d] & 0xffffffffull);
        if (n > 0 && i != prev)
        {
            poly[np++] = xy[i];
            prev = i;
        }
    }
    if (np > 1 && poly[np - 1].x == poly[0].x && poly[np - 1].y == poly[0].y)
        --np;
    return np;
}

__global__ void __launch_bounds__(256) k_hull_pre_ext(BatchDev b)
{
    pdl_enter();
    __shared__ float2 dirs[kDirs];
    __shared__ unsigned long long ext[kDirs][8];
    hull_dirs(dirs);
    __syncthreads();
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const uint32_t nitems = b.queue[6];
    for (uint32_t it = blockIdx.x; it < nitems; it += gridDim.x)
    {
        const uint2 w = b.pre_items[it];
        const uint32_t g = w.x, start = b.cl_start[g], n = b.cl_cnt[g];
        const uint32_t i0 = w.y * kPreChunk, i1 = min(n, i0 + kPreChunk);
        const float2* xy = b.mxy + start;
        Extremes16 ex;
        ex.init();
        for (uint32_t i = i0 + threadIdx.x; i < i1; i += blockDim.x)
        {
            const float2 q = xy[i];
            ex.add(dirs, q.x, q.y, i);
        }
#pragma unroll
        for (int d = 0; d < kDirs; ++d)
        {
            const unsigned long long v = warp_max64(ex.key(d));
            if (lane == 0)
                ext[d][warp] = v;
        }
        __syncthreads();
        if (threadIdx.x < kDirs)
        {
            unsigned long long best = ext[threadIdx.x][0];
            for (uint32_t k = 1; k < (blockDim.x >> 5); ++k)
                best = ext[threadIdx.x][k] > best ? ext[threadIdx.x][k] : best;
            atomicMax(&b.pre_ext[16ull * g + threadIdx.x], best);
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256) k_hull_pre_ref(BatchDev b)
{
    pdl_enter();
    __shared__ float2 poly[kDirs];
    __shared__ float4 erec[kDirs];
    __shared__ float2 emar[kDirs];
    __shared__ unsigned long long pkey[kDirs];
    __shared__ int npoly;
    const uint32_t lane = lane_id();
    const uint32_t nitems = b.queue[6];
    for (uint32_t it = blockIdx.x; it < nitems; it += gridDim.x)
    {
        const uint2 w = b.pre_items[it];
        const uint32_t g = w.x, start = b.cl_start[g], n = b.cl_cnt[g];
        const uint32_t i0 = w.y * kPreChunk, i1 = min(n, i0 + kPreChunk);
        const float2* xy = b.mxy + start;
        if (threadIdx.x == 0)
            npoly = first_polygon(xy, n, b.pre_ext + 16ull * g, poly);
        __syncthreads();
        const int np = npoly;
        if (np >= 3)
        {
            for (int e = threadIdx.x; e < np; e += blockDim.x)
            {
                pkey[e] = 0ull;
                const float2 a = poly[e], c = poly[(e + 1 == np) ? 0 : e + 1];
                const float ex = c.x - a.x, ey = c.y - a.y;
                const float l1 = fabsf(ex) + fabsf(ey);
                erec[e] = make_float4(a.x, a.y, ex, ey);
                emar[e] = make_float2(1e-5f * l1, 1e-6f * l1);
            }
            __syncthreads();
            uint32_t* act0 = reinterpret_cast<uint32_t*>(b.hs_stack + 2ull * start + 2ull * b.cl_rank[g]);
            for (uint32_t base = i0; base < i1; base += blockDim.x)
            {
                const uint32_t i = base + threadIdx.x;
                bool keep = false;
                if (i < i1)
                {
                    // the hull kernel's round-0 test: strictly inside every edge by the margin, and
                    // the farthest member outside each edge
                    const float2 q = xy[i];
                    bool in = true;
                    for (int e = 0; e < np; ++e)
                    {
                        const float4 r = erec[e];
                        const float2 mg = emar[e];
                        const float qx = q.x - r.x, qy = q.y - r.y;
                        const float cr = r.z * qy - r.w * qx;
                        const float aq = fabsf(qx) + fabsf(qy);
                        if (!(cr > mg.x * aq))
                            in = false;
                        if (cr < -(mg.y * aq))
                        {
                            const unsigned long long key = fkey_payload(-cr, i);
                            if (key > pkey[e])
                                atomicMax(&pkey[e], key);
                        }
                    }
                    keep = !in;
                }
                const uint32_t mask = __ballot_sync(0xffffffffu, keep);
                uint32_t at = 0;
                if (lane == 0 && mask)
                    at = atomicAdd(&b.pre_nact[g], static_cast<uint32_t>(__popc(mask)));
                at = __shfl_sync(0xffffffffu, at, 0);
                if (keep)
                    act0[at + static_cast<uint32_t>(__popc(mask & ((1u << lane) - 1u)))] = i;
            }
            __syncthreads();
            if (threadIdx.x < static_cast<uint32_t>(np) && pkey[threadIdx.x] != 0ull)
                atomicMax(&b.pre_pk[16ull * g + threadIdx.x], pkey[threadIdx.x]);
        }
        __syncthreads();
    }
}

// Local indices of a hull's h vertices (H: their candidates in C), more than shared memory takes: the members
// [start, start + n) before each, by a CTA. A vertex per lane, every member once for all of a warp's (from
// aligned quadruples, the same for all lanes). A warp per vertex read the members for each of them: of the 117 ms that
// k_hull took for a cluster of 112,000 members and 2,048 vertices all but 10.
__device__ __noinline__ void count_members(const uint32_t* members, uint32_t start, uint32_t n, const HPt<float>* C, const int* H,
                                           int h, int32_t* out)
{
    const uint32_t a4 = start & 3u;
    const uint4* mv = reinterpret_cast<const uint4*>(members + (start - a4));
    const uint32_t nq = (n + a4 + 3u) / 4u;
    for (int j = static_cast<int>(threadIdx.x); j - static_cast<int>(lane_id()) < h; j += kHullThreads)
    {
        const uint32_t key = (j < h) ? C[H[j]].key : 0u;
        uint32_t cnt = 0;
#pragma unroll 4
        for (uint32_t v = 0; v < nq; ++v)
        {
            const uint4 o = mv[v];
            const uint32_t i = 4u * v - a4; // (wraps below the first member: not less than n)
            cnt += (o.x < key && i < n) ? 1u : 0u;
            cnt += (o.y < key && i + 1u < n) ? 1u : 0u;
            cnt += (o.z < key && i + 2u < n) ? 1u : 0u;
            cnt += (o.w < key && i + 3u < n) ? 1u : 0u;
        }
        if (j < h)
            out[j] = static_cast<int32_t>(cnt);
    }
}

// Cluster g of scan s: z range, hull (local indices into hull_tmp at cl_start), boxes.
__device__ void hull_one(const BatchDev& b, HullSmem& sm, uint32_t g, int compute_obb)
{
    const uint32_t n = b.cl_cnt[g];
    const uint32_t start = b.cl_start[g];
    const uint32_t* mem = b.members + start;
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    if (threadIdx.x == 0)
        sm.ncand = 0;

    // 1. the extreme member in each of kDirs directions (float projections: any member is a valid
    //    polygon vertex, exactness is not needed here), from the members' x, y stored contiguously
    //    by the cluster scatter; the z range is already known. The members are read as aligned
    //    pairs (slot v: members 2v - a and 2v - a + 1, a = start mod 2), four 16-byte loads in
    //    flight per thread; the halves outside [0, n) are skipped (the loads stay inside the
    //    allocation: it starts at or before member start - a and has 16 bytes after its end).
    const float2* xy = b.mxy + start;
    HPt<float>* gs = reinterpret_cast<HPt<float>*>(b.hs_cand) + 2ull * start; // capacity 2n >= next_pow2(n)
    const int32_t a2 = static_cast<int32_t>(start & 1u);
    const float4* xv = reinterpret_cast<const float4*>(b.mxy + (start - static_cast<uint32_t>(a2)));
    const uint32_t npair = (n + static_cast<uint32_t>(a2) + 1u) / 2u;
    const bool pre = n > kPreMin; // extremes and round 0 came from the grid-wide passes
    Extremes16 ex;
    ex.init();
    for (uint32_t v0 = threadIdx.x; !pre && v0 < npair; v0 += 4u * blockDim.x)
    {
        float4 q[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
        {
            const uint32_t v = v0 + static_cast<uint32_t>(u) * blockDim.x;
            q[u] = (v < npair) ? xv[v] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
        {
            const int32_t i = 2 * static_cast<int32_t>(v0 + static_cast<uint32_t>(u) * blockDim.x) - a2;
            if (i >= 0 && i < static_cast<int32_t>(n))
                ex.add(sm.dirs, q[u].x, q[u].y, static_cast<uint32_t>(i));
            if (i + 1 >= 0 && i + 1 < static_cast<int32_t>(n))
                ex.add(sm.dirs, q[u].z, q[u].w, static_cast<uint32_t>(i + 1));
        }
    }
    if (!pre)
    {
        const unsigned long long key = ex.warp_key();
        if (lane < static_cast<uint32_t>(kDirs))
            sm.ext[lane][warp] = key;
    }
    else if (threadIdx.x < kDirs * (kHullThreads / 32))
    {
        const uint32_t d = threadIdx.x / (kHullThreads / 32), w = threadIdx.x % (kHullThreads / 32);
        sm.ext[d][w] = (w == 0) ? b.pre_ext[16ull * g + d] : 0ull;
    }
    __syncthreads();
    if (warp == 0)
    {
        unsigned long long best = 0ull;
        if (lane < static_cast<uint32_t>(kDirs))
            for (int w = 0; w < kHullThreads / 32; ++w)
                best = sm.ext[lane][w] > best ? sm.ext[lane][w] : best;
        const int np = extreme_polygon(xy, n, best, sm.poly);
        if (lane == 0)
        {
            b.cl_zmin[g] = zkey_min(b.cl_zkey[2u * g]);
            b.cl_zmax[g] = zkey_max(b.cl_zkey[2u * g + 1u]);
            sm.npoly = np;
        }
    }
    __syncthreads();

    int32_t* hull_dst = b.hull_tmp + start;
    if (n < 3)
    {
        // convexHull with fewer than 3 points returns 0..n-1 (polygonizer.cpp:36-41)
        if (threadIdx.x == 0)
        {
            for (uint32_t i = 0; i < n; ++i)
                hull_dst[i] = static_cast<int32_t>(i);
            b.hull_cnt[g] = n;
            if (compute_obb)
            {
                lp_bounding_box z;
                memset(&z, 0, sizeof(z));
                b.obb_c[g] = z;
                b.obb_p[g] = z;
            }
        }
        __syncthreads();
        return;
    }

    // 2. refine the polygon: insert the member farthest outside each edge (Quickhull step),
    //    while it grows and fits. Every vertex is a member, so the polygon stays inside the hull.
    //    Members proven strictly inside the current polygon leave the active set: the float test
    //    keeps a 1e-5 relative margin, far above its rounding error, so no hull vertex is dropped.
    uint32_t* act[2] = {reinterpret_cast<uint32_t*>(b.hs_stack + 2ull * start + 2ull * b.cl_rank[g]), nullptr};
    act[1] = act[0] + n; // two member lists of n entries in the chain-stack scratch (2n + 2)
    int cur = -1;        // -1: the active set is all members
    uint32_t nact = n;
    int np = sm.npoly;
    float2 *poly = sm.poly, *grown = sm.poly2;
    for (int round = 0; round < kRefineRounds && np >= 3; ++round)
    {
        for (int e = threadIdx.x; e < np; e += blockDim.x)
        {
            sm.pkey[e] = 0ull;
            const float2 a = poly[e], c = poly[(e + 1 == np) ? 0 : e + 1];
            const float ex = c.x - a.x, ey = c.y - a.y;
            const float l1 = fabsf(ex) + fabsf(ey);
            sm.erec[e] = make_float4(a.x, a.y, ex, ey);
            sm.emar[e] = make_float2(1e-5f * l1, 1e-6f * l1);
        }
        if (threadIdx.x == 0)
            sm.ncand = 0;
        __syncthreads();
        const int nxt = (cur == 0) ? 1 : 0;
        // two members per thread and edge load; q = p - a, cr < 0: right of the edge, outside
        auto edge = [&](const float4& r, const float2& mg, int e, float px, float py, uint32_t i, bool& in) {
            const float qx = px - r.x, qy = py - r.y;
            const float cr = r.z * qy - r.w * qx;
            const float aq = fabsf(qx) + fabsf(qy);
            if (!(cr > mg.x * aq))
                in = false;
            if (cr < -(mg.y * aq))
            {
                const unsigned long long key = fkey_payload(-cr, i);
                if (key > sm.pkey[e])
                    atomicMax(&sm.pkey[e], key);
            }
        };
        // members ok0 / ok1 (at least one): a missing one repeats the other and is not listed
        auto test2 = [&](float2 p0, uint32_t i0, bool ok0, float2 p1, uint32_t i1, bool ok1) {
            if (!ok0)
            {
                p0 = p1;
                i0 = i1;
            }
            if (!ok1)
            {
                p1 = p0;
                i1 = i0;
            }
            bool in0 = true, in1 = true;
            for (int e = 0; e < np; ++e)
            {
                const float4 r = sm.erec[e];
                const float2 mg = sm.emar[e];
                edge(r, mg, e, p0.x, p0.y, i0, in0);
                edge(r, mg, e, p1.x, p1.y, i1, in1);
            }
            if (ok0 && !in0)
                act[nxt][atomicAdd(&sm.ncand, 1)] = i0;
            if (ok1 && !in1)
                act[nxt][atomicAdd(&sm.ncand, 1)] = i1;
        };
        if (cur < 0 && pre)
        {
            // round 0 ran grid-wide against this polygon: its survivors are in act[0], and the
            // farthest member outside each edge is in the pass's record
            for (int e = threadIdx.x; e < np; e += blockDim.x)
                sm.pkey[e] = b.pre_pk[16ull * g + e];
            if (threadIdx.x == 0)
                sm.ncand = static_cast<int>(b.pre_nact[g]);
        }
        else if (cur < 0)
        {
            // all members: the aligned pairs of step 1, one 16-byte load each
            for (uint32_t v = threadIdx.x; v < npair; v += blockDim.x)
            {
                const float4 q = xv[v];
                const int32_t i = 2 * static_cast<int32_t>(v) - a2;
                test2(make_float2(q.x, q.y), static_cast<uint32_t>(max(i, 0)), i >= 0,
                      make_float2(q.z, q.w), static_cast<uint32_t>(i + 1), i + 1 < static_cast<int32_t>(n));
            }
        }
        else
        {
            for (uint32_t t = threadIdx.x; t < nact; t += 2u * blockDim.x)
            {
                const uint32_t t1 = t + blockDim.x;
                const bool two = t1 < nact;
                const uint32_t i0 = act[cur][t];
                const uint32_t i1 = two ? act[cur][t1] : i0;
                test2(xy[i0], i0, true, xy[i1], i1, two);
            }
        }
        __syncthreads();
        cur = nxt;
        const uint32_t had = nact;
        nact = static_cast<uint32_t>(sm.ncand);
        // each edge's farthest member goes in behind the edge's start, a thread per edge
        static_assert(kPolyCap <= kHullThreads);
        const int me = static_cast<int>(threadIdx.x);
        const unsigned long long far = (me < np) ? sm.pkey[me] : 0ull;
        uint32_t add;
        const int at = me + static_cast<int>(block_excl_scan(far != 0ull ? 1u : 0u, sm.scan, &add));
        const int w = np + static_cast<int>(add);
        if (add == 0u || w > kPolyCap)
            break;
        if (me < np)
        {
            grown[at] = poly[me];
            if (far != 0ull)
                grown[at + 1] = xy[static_cast<uint32_t>(far & 0xffffffffull)];
        }
        float2* const was = poly;
        poly = grown;
        grown = was;
        np = w;
        __syncthreads();
        if (nact <= kHullEnough || 4u * nact > 3u * had)
            break; // sorting the rest costs less than another round
    }

    // 3. candidates: active members not strictly inside the polygon by a relative margin far
    //    above float rounding (a hull vertex is never strictly inside a polygon of members)
    const int npf = np;
    auto inside = [&](float px, float py) {
        if (npf < 3)
            return false;
        for (int d = 0; d < npf; ++d)
        {
            const float2 a = poly[d], c = poly[(d + 1 == npf) ? 0 : d + 1];
            if (!left_strict_f(a.x, a.y, c.x, c.y, px, py))
                return false;
        }
        return true;
    };
    if (threadIdx.x == 0)
        sm.ncand = 0;
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < nact; t += blockDim.x)
    {
        const uint32_t i = (cur < 0) ? t : act[cur][t];
        const uint32_t o = mem[i];
        const float2 p = xy[i];
        if (!inside(p.x, p.y) && has_place(p.x, p.y))
        {
            const int pos = atomicAdd(&sm.ncand, 1);
            if (pos < kHullSmem)
                sm.cand[pos] = HPt<float>{p.x, p.y, o};
            gs[pos] = HPt<float>{p.x, p.y, o};
        }
    }
    __syncthreads();
    const int m = sm.ncand;
    const bool small = m <= kHullSmem;

    // 4. sort by (x, y, input order) and the monotone chain
    const HPt<float>* C;
    int* H;
    if (m <= kHullThreads)
    {
        // a candidate per thread, its place the number of smaller ones (a total order)
        const bool mine = static_cast<int>(threadIdx.x) < m;
        const HPt<float> v = mine ? sm.cand[threadIdx.x] : HPt<float>{INFINITY, INFINITY, 0xffffffffu};
        uint32_t rank = 0;
        if (static_cast<int>(warp * 32u) < m)
#pragma unroll 4
            for (int k = 0; k < m; ++k)
                rank += hpt_less(sm.cand[k], v) ? 1u : 0u;
        __syncthreads();
        if (mine)
            sm.cand[rank] = v;
        C = sm.cand;
        H = sm.stack;
    }
    else if (small)
    {
        const uint32_t np2 = next_pow2(static_cast<uint32_t>(m));
        for (uint32_t i = m + threadIdx.x; i < np2; i += blockDim.x)
            sm.cand[i] = HPt<float>{INFINITY, INFINITY, 0xffffffffu};
        __syncthreads();
        block_bitonic_sort(sm.cand, np2, [](const HPt<float>& a, const HPt<float>& c) { return hpt_less(a, c); });
        C = sm.cand;
        H = sm.stack;
    }
    else
    {
        block_sort_global(gs, static_cast<uint32_t>(m));
        C = gs;
        H = b.hs_stack + 2ull * start + 2ull * b.cl_rank[g]; // capacity 2n + 2 >= 2m + 2
    }
    __syncthreads();
    // lower half on warp 0, upper half on warp 1 into H + m + 1; then the
    // upper half moves down behind the lower one (forwards: the source lies above the target)
    if (warp < 2u)
    {
        const int k = chain_half<32>(C, m, H + (warp ? m + 1 : 0), warp == 1u);
        if (lane == 0)
            (warp ? sm.grew : sm.nhull) = k;
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        const int kl = sm.nhull, ku = sm.grew;
        for (int j = 1; j < ku - 1; ++j)
            H[kl - 1 + j] = H[m + 1 + j];
        sm.nhull = (m < 2) ? m : kl + ku - 2;
    }
    __syncthreads();
    const int h = sm.nhull;
    bool tied;
    {
        // a hull vertex with an identical candidate next to it: the reference's pick among them
        // follows std::sort's order (k_hull_boxes replays it)
        bool tie = false;
        for (int j = threadIdx.x; j < h; j += blockDim.x)
        {
            const int q = H[j];
            const HPt<float> c = C[q];
            tie |= (q > 0 && C[q - 1].x == c.x && C[q - 1].y == c.y) ||
                   (q + 1 < static_cast<int>(m) && C[q + 1].x == c.x && C[q + 1].y == c.y);
        }
        tied = __syncthreads_or(tie);
        if (tied && threadIdx.x == 0)
            b.tie_list[atomicAdd(&b.queue[5], 1u)] = g;
    }

    // 5. The vertices' coordinates for k_hull_boxes and their local indices: the number of
    //    members before each in input order.
    const bool fast = h <= kHullSmem;
    for (int j = threadIdx.x; j < h; j += blockDim.x)
    {
        const HPt<float> c = C[H[j]];
        b.hs_pts[start + j] = make_double2(static_cast<double>(c.x), static_cast<double>(c.y));
    }
    if (pre && small && h <= kCountLater)
    {
        // a cluster of the grid-wide passes: its members are counted grid-wide too (k_hull_boxes, one item per
        // kPreChunk members); not where a tie repair needs the indices first
        if (threadIdx.x == 0)
            b.pre_nact[g] = tied ? 0u : static_cast<uint32_t>(h);
        if (!tied)
        {
            int* keys = b.hs_stack + 2ull * start + 2ull * b.cl_rank[g];
            for (int j = threadIdx.x; j < h; j += blockDim.x)
            {
                keys[j] = static_cast<int>(C[H[j]].key);
                hull_dst[j] = 0;
            }
            if (threadIdx.x == 0)
                b.hull_cnt[g] = static_cast<uint32_t>(h);
            __syncthreads();
            return;
        }
    }
    else if (pre && threadIdx.x == 0)
        b.pre_nact[g] = 0u;
    const uint32_t np2 = next_pow2(static_cast<uint32_t>(h));
    int place = -1; // of the thread's vertex in key order (up to a vertex per thread)
    if (h <= kHullThreads)
    {
        if (static_cast<int>(threadIdx.x) < h)
            sm.diff[threadIdx.x] = static_cast<int32_t>(C[H[threadIdx.x]].key);
        __syncthreads();
        if (static_cast<int>(threadIdx.x) < h)
        {
            const uint32_t key = static_cast<uint32_t>(sm.diff[threadIdx.x]);
            place = 0;
#pragma unroll 4
            for (int k = 0; k < h; ++k)
                place += (static_cast<uint32_t>(sm.diff[k]) < key) ? 1 : 0;
            sm.hkey[place] = key;
        }
        for (uint32_t j = h + threadIdx.x; j < np2; j += blockDim.x)
            sm.hkey[j] = 0xffffffffu;
        __syncthreads();
    }
    else if (fast)
    {
        for (int j = threadIdx.x; j < h; j += blockDim.x)
            sm.hkey[j] = C[H[j]].key;
        for (uint32_t j = h + threadIdx.x; j < np2; j += blockDim.x)
            sm.hkey[j] = 0xffffffffu;
        __syncthreads();
        block_bitonic_sort(sm.hkey, np2, [](uint32_t a, uint32_t c) { return a < c; });
    }
    if (fast)
    {
        for (int j = threadIdx.x; j <= h; j += blockDim.x)
            sm.diff[j] = 0;
        __syncthreads();
        // member o adds 1 to every hull vertex with a larger key: diff[upper_bound(o)] += 1. Each
        // thread walks a contiguous chunk of the member list as aligned quadruples (slot v:
        // members 4v - a .. 4v - a + 3, a = start mod 4; entries outside [0, n) skipped, the loads
        // stay inside the allocation), four at a time: a search is a chain of shared-memory loads, sixteen of
        // them overlap (one after the other, 37,990 members took 45,000 cycles). Members come in ascending index
        // runs, so consecutive ones mostly fall into the same bin: a bin's count is added when the bin changes.
        const uint32_t a4 = start & 3u;
        const uint4* mv = reinterpret_cast<const uint4*>(b.members + (start - a4));
        const uint32_t nq = (n + a4 + 3u) / 4u;
        const uint32_t per = (nq + kHullThreads - 1u) / kHullThreads;
        const uint32_t q0 = threadIdx.x * per, q1 = min(nq, q0 + per);
        int cb = h, cc = 0; // current bin and its pending count
        for (uint32_t v = q0; v < q1; v += 4u)
        {
            uint32_t o[16], l[16];
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u)
            {
                const uint4 q = (v + u < q1) ? mv[v + u] : make_uint4(0u, 0u, 0u, 0u);
                o[4 * u] = q.x;
                o[4 * u + 1] = q.y;
                o[4 * u + 2] = q.z;
                o[4 * u + 3] = q.w;
            }
#pragma unroll
            for (int c = 0; c < 16; ++c)
                l[c] = 0u;
#pragma unroll 1
            for (uint32_t step = np2 >> 1; step > 0u; step >>= 1)
#pragma unroll
                for (int c = 0; c < 16; ++c)
                    l[c] += (sm.hkey[l[c] + step - 1u] <= o[c]) ? step : 0u;
            const uint32_t i = 4u * v - a4; // (wraps below the first member: not less than n)
            const uint32_t end = min(n, 4u * q1 - a4);
#pragma unroll
            for (int c = 0; c < 16; ++c)
            {
                const int bin = static_cast<int>(l[c] + ((sm.hkey[l[c]] <= o[c]) ? 1u : 0u));
                const bool in = i + c < end;
                if (in && bin != cb)
                {
                    if (cc > 0 && cb < h)
                        atomicAdd(&sm.diff[cb], cc);
                    cb = bin;
                    cc = 0;
                }
                cc += in ? 1 : 0;
            }
        }
        if (cc > 0 && cb < h)
            atomicAdd(&sm.diff[cb], cc);
    }
    else // (candidates and stack lie in global memory)
        count_members(b.members, start, n, reinterpret_cast<const HPt<float>*>(b.hs_cand) + 2ull * start,
                      b.hs_stack + 2ull * start + 2ull * b.cl_rank[g], h, hull_dst);
    __syncthreads();
    if (fast)
    {
        if (threadIdx.x == 0)
        {
            int run = 0;
            for (int t = 0; t < h; ++t)
            {
                run += sm.diff[t];
                sm.diff[t] = run; // members with a smaller key than hkey[t]
            }
        }
        __syncthreads();
        if (place >= 0)
            hull_dst[threadIdx.x] = sm.diff[place];
        for (int j = threadIdx.x; h > kHullThreads && j < h; j += blockDim.x)
        {
            const uint32_t key = C[H[j]].key;
            int lo = 0, hi = h - 1;
            while (lo < hi)
            {
                const int mid = (lo + hi) >> 1;
                if (sm.hkey[mid] < key)
                    lo = mid + 1;
                else
                    hi = mid;
            }
            hull_dst[j] = sm.diff[lo];
        }
    }
    if (threadIdx.x == 0)
        b.hull_cnt[g] = static_cast<uint32_t>(h);
    __syncthreads();
}

// ---------------------------------------------------------------------------------------------
// Warp path for clusters of at most kBigCluster members: the same steps as hull_one without CTA
// barriers (the 16-direction polygon is the prefilter; candidates rarely exceed a warp's buffer,
// and then the sort and the chain stack move to global scratch).
// ---------------------------------------------------------------------------------------------
constexpr int kWarpCand = 256;
constexpr uint32_t kWarpRefineMin = 64; // more candidates than this: refine the polygon first
constexpr int kWarpPoly = 64;           // refined polygon capacity of the warp path

// Scratch of the warp path's polygon refinement.
struct WarpRefine
{
    float2 rp[kWarpPoly], rp2[kWarpPoly];
    float4 erec[kWarpPoly];
    float2 emar[kWarpPoly];
    unsigned long long pkey[kWarpPoly];
};

struct WarpSmem
{
    WarpRefine refine;
    HPt<float> cand[kWarpCand];
    int stack[2 * kWarpCand + 2];
    float2 poly[kDirs];
};

// Quickhull rounds over the candidates C[0..m) (at most 16 per lane), starting from the warp's
// 16-direction polygon: each round tests every candidate against the polygon's edges (keeping
// the farthest candidate outside each edge), compacts away the candidates strictly inside, and
// inserts the farthest ones. Returns the number of candidates left in C.
__device__ uint32_t warp_refine(WarpSmem& ws, HPt<float>* C, uint32_t m, int np)
{
    WarpRefine& wr = ws.refine;
    const uint32_t lane = lane_id();
    for (int e = static_cast<int>(lane); e < np; e += 32)
        wr.rp[e] = ws.poly[e];
    __syncwarp();
    for (int round = 0; round < 4 && m > kWarpRefineMin; ++round)
    {
        for (int e = static_cast<int>(lane); e < np; e += 32)
        {
            const float2 a = wr.rp[e], c = wr.rp[(e + 1 == np) ? 0 : e + 1];
            const float ex = c.x - a.x, ey = c.y - a.y;
            const float l1 = fabsf(ex) + fabsf(ey);
            wr.erec[e] = make_float4(a.x, a.y, ex, ey);
            wr.emar[e] = make_float2(1e-5f * l1, 1e-6f * l1);
            wr.pkey[e] = 0ull;
        }
        __syncwarp();
        uint32_t inbits = 0u;
        for (uint32_t base = 0, q = 0; base < m; base += 32, ++q)
        {
            const uint32_t k = base + lane;
            bool in = false;
            if (k < m)
            {
                const HPt<float> c = C[k];
                in = true;
                for (int e = 0; e < np; ++e)
                {
                    const float4 r = wr.erec[e];
                    const float2 mg = wr.emar[e];
                    const float qx = c.x - r.x, qy = c.y - r.y;
                    const float cr = r.z * qy - r.w * qx; // < 0: right of the edge, outside
                    const float aq = fabsf(qx) + fabsf(qy);
                    if (!(cr > mg.x * aq))
                        in = false;
                    if (cr < -(mg.y * aq))
                    {
                        const unsigned long long key = fkey_payload(-cr, k);
                        if (key > wr.pkey[e])
                            atomicMax(&wr.pkey[e], key);
                    }
                }
            }
            inbits |= (in ? 1u : 0u) << q;
        }
        __syncwarp();
        // each edge's farthest outside candidate goes in behind the edge's start (positions before compaction)
        static_assert(kWarpPoly == 64);
        const int e0 = static_cast<int>(lane), e1 = e0 + 32;
        const unsigned long long f0 = (e0 < np) ? wr.pkey[e0] : 0ull, f1 = (e1 < np) ? wr.pkey[e1] : 0ull;
        const uint32_t m0 = __ballot_sync(0xffffffffu, f0 != 0ull), m1 = __ballot_sync(0xffffffffu, f1 != 0ull);
        const int add = __popc(m0) + __popc(m1);
        const bool grew = add > 0 && np + add <= kWarpPoly;
        if (grew)
        {
            auto put = [&](int e, unsigned long long f, int before) {
                if (e >= np)
                    return;
                wr.rp2[e + before] = wr.rp[e];
                if (f != 0ull)
                {
                    const HPt<float> c = C[static_cast<uint32_t>(f & 0xffffffffull)];
                    wr.rp2[e + before + 1] = make_float2(c.x, c.y);
                }
            };
            put(e0, f0, __popc(m0 & ((1u << lane) - 1u)));
            put(e1, f1, __popc(m0) + __popc(m1 & ((1u << lane) - 1u)));
            __syncwarp();
            np += add;
            for (int e = e0; e < np; e += 32)
                wr.rp[e] = wr.rp2[e];
        }
        __syncwarp();
        // compact in place (every chunk is read before any of its positions is written)
        uint32_t wpos = 0;
        for (uint32_t base = 0, q = 0; base < m; base += 32, ++q)
        {
            const uint32_t k = base + lane;
            const bool keep = k < m && !((inbits >> q) & 1u);
            HPt<float> c{0.0f, 0.0f, 0u};
            if (keep)
                c = C[k];
            const uint32_t mask = __ballot_sync(0xffffffffu, keep);
            __syncwarp();
            if (keep)
                C[wpos + __popc(mask & ((1u << lane) - 1u))] = c;
            wpos += __popc(mask);
        }
        m = wpos;
        __syncwarp();
        if (!grew)
            break;
    }
    return m;
}

__device__ void hull_one_warp(const BatchDev& b, WarpSmem& ws, const float2* dirs, uint32_t g, int compute_obb)
{
    const uint32_t n = b.cl_cnt[g];
    const uint32_t start = b.cl_start[g];
    const uint32_t* mem = b.members + start;
    const uint32_t lane = lane_id();
    const float2* xy = b.mxy + start;
    Extremes16 ex;
    ex.init();
    for (uint32_t i0 = lane; i0 < n; i0 += 128u)
    {
        float2 p[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u)
            p[u] = (i0 + 32u * u < n) ? xy[i0 + 32u * u] : make_float2(NAN, NAN); // (never an extreme)
#pragma unroll 1
        for (uint32_t u = 0; u < 4 && i0 + 32u * u < n; ++u)
            ex.add(dirs, u < 2 ? (u == 0 ? p[0].x : p[1].x) : (u == 2 ? p[2].x : p[3].x),
                   u < 2 ? (u == 0 ? p[0].y : p[1].y) : (u == 2 ? p[2].y : p[3].y), i0 + 32u * u);
    }
    const int npf = extreme_polygon(xy, n, ex.warp_key(), ws.poly);
    if (lane == 0)
    {
        b.cl_zmin[g] = zkey_min(b.cl_zkey[2u * g]);
        b.cl_zmax[g] = zkey_max(b.cl_zkey[2u * g + 1u]);
    }
    int32_t* hull_dst = b.hull_tmp + start;
    if (n < 3)
    {
        if (lane == 0)
        {
            for (uint32_t i = 0; i < n; ++i)
                hull_dst[i] = static_cast<int32_t>(i);
            b.hull_cnt[g] = n;
            if (compute_obb)
            {
                lp_bounding_box z;
                memset(&z, 0, sizeof(z));
                b.obb_c[g] = z;
                b.obb_p[g] = z;
            }
        }
        __syncwarp();
        return;
    }
    // the polygon's edges (start, direction; |direction|_1), in the refinement's scratch
    if (lane < static_cast<uint32_t>(npf))
    {
        const float2 a = ws.poly[lane], c = ws.poly[(static_cast<int>(lane) + 1 == npf) ? 0 : lane + 1];
        ws.refine.erec[lane] = make_float4(a.x, a.y, c.x - a.x, c.y - a.y);
        ws.refine.emar[lane].x = fabsf(c.x - a.x) + fabsf(c.y - a.y);
    }
    __syncwarp();
    auto inside = [&](float px, float py) { // left_strict_f of every edge
        bool in = npf >= 3;
#pragma unroll 4
        for (int d = 0; d < npf; ++d)
        {
            const float4 r = ws.refine.erec[d];
            const float qx = px - r.x, qy = py - r.y;
            const float cr = r.z * qy - r.w * qx;
            const float scale = ws.refine.emar[d].x * (fabsf(qx) + fabsf(qy));
            in = in && cr > 1e-5f * scale + 1e-30f;
        }
        return in;
    };
    HPt<float>* gs = reinterpret_cast<HPt<float>*>(b.hs_cand) + 2ull * start; // capacity 2n >= next_pow2(n)
    uint32_t m = 0;
    uint32_t o_next = mem[min(lane, n - 1u)];
    float2 p_next = xy[min(lane, n - 1u)];
#pragma unroll 1
    for (uint32_t base = 0; base < n; base += 32)
    {
        const uint32_t i = base + lane;
        const HPt<float> c{p_next.x, p_next.y, o_next};
        const uint32_t ahead = min(i + 32u, n - 1u); // (on its way during the tests)
        o_next = mem[ahead];
        p_next = xy[ahead];
        const bool keep = !inside(c.x, c.y) && i < n && has_place(c.x, c.y);
        const uint32_t mask = __ballot_sync(0xffffffffu, keep);
        if (keep)
        {
            const uint32_t pos = m + __popc(mask & ((1u << lane) - 1u));
            if (pos < static_cast<uint32_t>(kWarpCand))
                ws.cand[pos] = c;
            gs[pos] = c;
        }
        m += __popc(mask);
    }
    __syncwarp();
    // Many candidates (members spread along the boundary, e.g. an arc): refine the polygon as the
    // CTA path does (insert the candidate farthest outside each edge, drop the candidates proven
    // strictly inside by the 1e-5 relative margin), a few rounds.
    HPt<float>* C0 = (m <= static_cast<uint32_t>(kWarpCand)) ? ws.cand : gs;
    if (m > kWarpRefineMin && npf >= 3)
        m = warp_refine(ws, C0, m, npf);
    const bool small = m <= static_cast<uint32_t>(kWarpCand);
    if (small && C0 == gs)
    {
        for (uint32_t k = lane; k < m; k += 32)
            ws.cand[k] = gs[k];
        __syncwarp();
    }
    HPt<float>* C = small ? ws.cand : gs;
    int* H = small ? ws.stack : (b.hs_stack + 2ull * start + 2ull * b.cl_rank[g]);
    if (small)
    {
        // two candidates per lane, the place of each the number of smaller ones (hpt_less is a total order), into
        // the refinement's scratch: 120 candidates take a tenth of the exchange sort's 50,000 cycles
        static_assert(sizeof(WarpRefine) >= sizeof(HPt<float>) * kWarpCand);
        HPt<float>* D = reinterpret_cast<HPt<float>*>(&ws.refine);
        const HPt<float> last{INFINITY, INFINITY, 0xffffffffu};
        for (uint32_t base = lane; base < m + lane; base += 64u)
        {
            const HPt<float> v0 = (base < m) ? ws.cand[base] : last, v1 = (base + 32u < m) ? ws.cand[base + 32u] : last;
            uint32_t r0 = 0, r1 = 0;
#pragma unroll 2
            for (uint32_t k = 0; k < m; ++k)
            {
                const HPt<float> c = ws.cand[k];
                r0 += hpt_less(c, v0) ? 1u : 0u;
                r1 += hpt_less(c, v1) ? 1u : 0u;
            }
            if (base < m)
                D[r0] = v0;
            if (base + 32u < m)
                D[r1] = v1;
        }
        __syncwarp();
        C = D;
    }
    else
    {
        const uint32_t np2 = next_pow2(m);
        for (uint32_t i = m + lane; i < np2; i += 32)
            C[i] = HPt<float>{INFINITY, INFINITY, 0xffffffffu};
        __syncwarp();
        warp_bitonic_smem(C, np2, [](const HPt<float>& x, const HPt<float>& y) { return hpt_less(x, y); });
    }
    // lanes 0 to 15 walk the lower half, the others the upper one into H + m + 1, which then moves down behind
    // the lower half (chunk by chunk, forwards: the source lies above the target)
    const int kh = chain_half<16>(C, static_cast<int>(m), H + (lane >= 16u ? m + 1u : 0u), lane >= 16u);
    const int kl = __shfl_sync(0xffffffffu, kh, 0), ku = __shfl_sync(0xffffffffu, kh, 16);
    __syncwarp();
    for (int j0 = 1; j0 < ku - 1; j0 += 32)
    {
        const int j = j0 + static_cast<int>(lane);
        const int v = (j < ku - 1) ? H[static_cast<int>(m) + 1 + j] : 0;
        __syncwarp();
        if (j < ku - 1)
            H[kl - 1 + j] = v;
        __syncwarp();
    }
    const int h = (m < 2u) ? static_cast<int>(m) : kl + ku - 2;
    {
        bool tie = false;
        for (int j = static_cast<int>(lane); j < h; j += 32)
        {
            const int q = H[j];
            const HPt<float> c = C[q];
            tie |= (q > 0 && C[q - 1].x == c.x && C[q - 1].y == c.y) ||
                   (q + 1 < static_cast<int>(m) && C[q + 1].x == c.x && C[q + 1].y == c.y);
        }
        if (__any_sync(0xffffffffu, tie) && lane == 0)
            b.tie_list[atomicAdd(&b.queue[5], 1u)] = g;
    }
    // the members once in registers (n <= kBigCluster), then counted for every vertex
    uint32_t mk[kBigCluster / 32u];
#pragma unroll
    for (uint32_t q = 0; q < kBigCluster / 32u; ++q)
        mk[q] = (32u * q + lane < n) ? mem[32u * q + lane] : 0xffffffffu; // (never below a key)
    for (int j0 = 0; j0 < h; j0 += 32)
    {
        const int j = j0 + static_cast<int>(lane);
        const HPt<float> c = (j < h) ? C[H[j]] : HPt<float>{0.0f, 0.0f, 0u};
        uint32_t before = 0;
        for (int u = 0; u < min(32, h - j0); ++u)
        {
            const uint32_t key = __shfl_sync(0xffffffffu, c.key, u);
            uint32_t cnt = 0;
#pragma unroll
            for (uint32_t q = 0; q < kBigCluster / 32u; ++q)
                cnt += (mk[q] < key) ? 1u : 0u;
            cnt = __reduce_add_sync(0xffffffffu, cnt);
            if (static_cast<int>(lane) == u)
                before = cnt;
        }
        if (j < h)
        {
            hull_dst[j] = static_cast<int32_t>(before);
            b.hs_pts[start + j] = make_double2(static_cast<double>(c.x), static_cast<double>(c.y));
        }
    }
    if (lane == 0)
        b.hull_cnt[g] = static_cast<uint32_t>(h);
    __syncwarp();
}

// Work items: every cluster of the batch. queue[2] counts clusters of more than kBigCluster
// members (listed from the front of hull_work, taken by whole CTAs first), queue[3] the others
// (listed from the back, taken one warp each). A cluster's member range is reserved here too, with its rank
// in the order of the ranges (queue[8..9]; scratch that has a fixed part per cluster lies at a multiple
// of the start plus one of the rank), and its counters start at zero.
__global__ void k_hull_worklist(BatchDev b)
{
    pdl_enter();
    uint32_t* work = b.hull_work;
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= b.ncl)
        return;
    const int s = scan_of_cluster(b, g);
    if (g - b.scans[s].cl_off >= b.state[s].n_clusters)
        return;
    const uint32_t n = b.cl_cnt[g];
    const unsigned long long got = atomicAdd(reinterpret_cast<unsigned long long*>(&b.queue[8]), (1ull << 32) | n);
    b.cl_start[g] = static_cast<uint32_t>(got);
    b.cl_rank[g] = static_cast<uint32_t>(got >> 32);
    b.cl_fill[g] = 0u;
    b.cl_zkey[2u * g] = b.cl_zkey[2u * g + 1u] = 0u;
    if (n > b.hull_cta_min) // hull_cta_min <= kBigCluster: the warp path's limit
        work[atomicAdd(&b.queue[2], 1u)] = g;
    else
        work[b.ncl - 1u - atomicAdd(&b.queue[3], 1u)] = g;
    if (n > kPreMin)
    {
        // the grid-wide member passes: records cleared, one item per kPreChunk members (queue[6])
        for (int d = 0; d < 16; ++d)
        {
            b.pre_ext[16ull * g + d] = 0ull;
            b.pre_pk[16ull * g + d] = 0ull;
        }
        b.pre_nact[g] = 0u;
        const uint32_t nch = (n + kPreChunk - 1u) / kPreChunk;
        const uint32_t at = atomicAdd(&b.queue[6], nch);
        for (uint32_t c = 0; c < nch; ++c)
            b.pre_items[at + c] = make_uint2(g, c);
    }
}

constexpr size_t kHullDynSmem = sizeof(HullSmem) > (kHullThreads / 32) * sizeof(WarpSmem)
                                    ? sizeof(HullSmem)
                                    : (kHullThreads / 32) * sizeof(WarpSmem);

// Persistent CTAs: first every large cluster (one CTA each, queue[1] is the head), then every
// small cluster (one warp each, queue[4] is the head).
__global__ void __launch_bounds__(kHullThreads) k_hull(BatchDev b, int compute_obb, const uint32_t* work)
{
    pdl_enter();
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ float2 dirs[kDirs];
    HullSmem& sm = *reinterpret_cast<HullSmem*>(smraw);
    if (threadIdx.x < kDirs)
    {
        const float a = 6.28318530717958647692f * static_cast<float>(threadIdx.x) / kDirs;
        dirs[threadIdx.x] = make_float2(cosf(a), sinf(a));
        sm.dirs[threadIdx.x] = dirs[threadIdx.x];
    }
    const uint32_t nbig = b.queue[2];
    const uint32_t nsmall = b.queue[3];
    for (;;)
    {
        __syncthreads();
        if (threadIdx.x == 0)
            sm.work = atomicAdd(&b.queue[1], 1u);
        __syncthreads();
        const uint32_t w = sm.work;
        if (w >= nbig)
            break;
        const uint32_t g = work[w];
        hull_one(b, sm, g, compute_obb);
    }
    __syncthreads(); // the CTA's shared memory now becomes eight per-warp regions
    WarpSmem& ws = reinterpret_cast<WarpSmem*>(smraw)[threadIdx.x >> 5];
    for (;;)
    {
        uint32_t w = 0;
        if (lane_id() == 0)
            w = atomicAdd(&b.queue[4], 1u);
        w = __shfl_sync(0xffffffffu, w, 0);
        if (w >= nsmall)
            break;
        const uint32_t g = work[b.ncl - 1u - w];
        hull_one_warp(b, ws, dirs, g, compute_obb);
    }
}

// ---------------------------------------------------------------------------------------------
// The reference's order among identical points (Polygonizer::convexHull, polygonizer.cpp:51-59):
// std::sort orders the point indices by x, then (|dx| < DBL_EPSILON) y, and leaves points that
// compare equal in whatever order its introsort produced. The monotone chain keeps, of a run of
// identical points, the first in that order at the leftmost vertex and on the upper chain, and
// the last on the lower chain up to the rightmost vertex. The hull kernels order ties by input
// index; where a hull vertex has an identical point, the whole cluster's std::sort is replayed
// (lp_introsort.cuh) and each vertex re-picked from its run.
// ---------------------------------------------------------------------------------------------
template <typename T>
struct HRec
{
    T x, y;
    uint32_t idx;
};

template <typename T>
struct HullLess // the reference's sort comparator on its binary64 PointXY
{
    __device__ __forceinline__ bool operator()(const HRec<T>& a, const HRec<T>& b) const
    {
        const double ax = static_cast<double>(a.x), bx = static_cast<double>(b.x);
        return ax < bx || (fabs(ax - bx) < DBL_EPSILON && static_cast<double>(a.y) < static_cast<double>(b.y));
    }
};

// The same comparator on binary32 coordinates widened to binary64, decided in binary32 where that
// is exact: equal finite x compare by y (|dx| = 0; infinite x give inf - inf = NaN, not below
// DBL_EPSILON); distinct x of which one is at least 2^-20 in magnitude differ by at least 2^-44, so
// only x both below 2^-20 need the binary64 difference.
template <>
struct HullLess<float>
{
    __device__ __forceinline__ bool operator()(const HRec<float>& a, const HRec<float>& b) const
    {
        if (a.x < b.x)
            return true;
        if (a.x == b.x)
            return fabsf(a.x) < INFINITY && a.y < b.y;
        if (fabsf(a.x) < 0x1p-20f && fabsf(b.x) < 0x1p-20f)
            return fabs(static_cast<double>(a.x) - static_cast<double>(b.x)) < DBL_EPSILON && a.y < b.y;
        return false;
    }
};

template <typename T>
struct IdxLess
{
    __device__ __forceinline__ bool operator()(const HRec<T>& a, const HRec<T>& b) const { return a.idx < b.idx; }
};

// rec: the n points in input order (idx = position). hull (h local indices, in input-order ties)
// is rewritten with the reference's picks; vxy(j): the coordinates of hull vertex j (read before
// hull[j] is rewritten); ge/le: n entries each.
template <typename T, class VertexXY>
__device__ void hull_repair_ties(HRec<T>* rec, uint32_t n, int32_t* hull, int h, VertexXY vxy, uint32_t* ge,
                                 uint32_t* le, isort::SortShared& ss)
{
    __shared__ int s_jr;
    isort::cta_sort(rec, n, HullLess<T>{}, ge, le, ss);
    if (threadIdx.x == 0)
    {
        // the rightmost vertex ends the lower chain: the lexicographic maximum, its last occurrence
        // (a cloud of identical points has the hull [first, last] of one coordinate)
        int jr = 0;
        double2 best = vxy(0);
        for (int j = 1; j < h; ++j)
        {
            const double2 v = vxy(j);
            if (v.x > best.x || (v.x == best.x && v.y >= best.y))
            {
                jr = j;
                best = v;
            }
        }
        s_jr = jr;
    }
    __syncthreads();
    const int jr = s_jr;
    const HullLess<T> less{};
    for (int j = threadIdx.x; j < h; j += blockDim.x)
    {
        const double2 v = vxy(j);
        const HRec<T> t{static_cast<T>(v.x), static_cast<T>(v.y), 0u};
        // equal range of the vertex's point in the sorted records
        uint32_t lo = 0, hi = n;
        while (lo < hi)
        {
            const uint32_t mid = (lo + hi) / 2;
            if (less(rec[mid], t))
                lo = mid + 1;
            else
                hi = mid;
        }
        uint32_t lo2 = lo, hi2 = n;
        while (lo2 < hi2)
        {
            const uint32_t mid = (lo2 + hi2) / 2;
            if (!less(t, rec[mid]))
                lo2 = mid + 1;
            else
                hi2 = mid;
        }
        if (lo2 > lo)
            hull[j] = static_cast<int32_t>(rec[(j == 0 || j > jr) ? lo : lo2 - 1].idx);
    }
    __syncthreads();
}

// Clusters listed by k_hull (a hull vertex with an identical candidate): the members' records in
// input order (sorted by member key), then the repair. The sorts are chains of dependent accesses,
// so clusters of at most kTieSmemRecs members are sorted in shared memory (records, then the ge / le
// lists); larger ones use the cluster's scratch: the candidate area (records), the chain stack
// area (ge / le). The vertices' coordinates go to the FP64 hull area.
constexpr uint32_t kTieSmemRecs = 4096;
constexpr size_t kTieDynSmem = static_cast<size_t>(kTieSmemRecs) * (sizeof(HRec<float>) + 8);

// Cluster g's tie repair, by one CTA with kTieDynSmem bytes of shared memory.
__device__ __noinline__ void repair_cluster(const BatchDev& b, uint32_t g, unsigned char* tsm, isort::SortShared& ss)
{
    const uint32_t start = b.cl_start[g], n = b.cl_cnt[g];
    const int h = static_cast<int>(b.hull_cnt[g]);
    const bool local = n <= kTieSmemRecs;
    HRec<float>* rec = local ? reinterpret_cast<HRec<float>*>(tsm)
                             : reinterpret_cast<HRec<float>*>(reinterpret_cast<HPt<float>*>(b.hs_cand) + 2ull * start);
    uint32_t* ge = local ? reinterpret_cast<uint32_t*>(tsm + kTieSmemRecs * sizeof(HRec<float>))
                         : reinterpret_cast<uint32_t*>(b.hs_stack + 2ull * start + 2ull * b.cl_rank[g]);
    uint32_t* le = ge + (local ? kTieSmemRecs : n);
    for (uint32_t k = threadIdx.x; k < n; k += blockDim.x)
    {
        const float2 p = b.mxy[start + k];
        rec[k] = HRec<float>{p.x, p.y, b.members[start + k]};
    }
    __syncthreads();
    isort::cta_sort(rec, n, IdxLess<float>{}, ge, le, ss);
    for (uint32_t k = threadIdx.x; k < n; k += blockDim.x)
        rec[k].idx = k; // local index: position in input order
    __syncthreads();
    const double2* hv = b.hs_pts + start; // the vertices' coordinates, from k_hull
    hull_repair_ties(rec, n, b.hull_tmp + start, h, [=](int j) { return hv[j]; }, ge, le, ss);
    __syncthreads();
}

// A cluster's hull vertices while its boxes are computed, N at most.
template <int N>
struct BoxSmem
{
    double2 hp[N];
    float2 pf[N];
    float ea[N];
};
constexpr int kBoxWarpVerts = 256; // more: the warps of a CTA share one region, up to kHullSmem
static_assert(sizeof(BoxSmem<kBoxWarpVerts>) * (kHullThreads / 32) <= kTieDynSmem && sizeof(BoxSmem<kHullSmem>) <= kTieDynSmem);

// The tie repairs (rare), the member counts of the large clusters' hulls, then both boxes of every cluster, a warp for each box. The boxes' FP64 chains
// (the SM retires an FP64 instruction of a warp every 16 cycles) take longer than finding the hull: one after the other
// behind the hull, they were more than half of the 62 us that a small scan's longest cluster took; here the two boxes run
// on different SMs where the scan is small, and the hull kernel's code fits the instruction cache better without them.
// Item i of 2 K (K clusters, the large ones first; calipers, then PCA) goes to CTA i mod grid, so that a small
// scan's boxes share no SM's FP64 unit. A tie repair moves no coordinate: the boxes need not wait for it.
__global__ void __launch_bounds__(kHullThreads) k_hull_boxes(BatchDev b, int compute_obb, const uint32_t* work)
{
    pdl_enter();
    __shared__ isort::SortShared ss;
    extern __shared__ __align__(16) unsigned char tsm[];
    const uint32_t ntie = b.queue[5]; // the tie count (queue[4] is the small-cluster head)
    for (uint32_t t = blockIdx.x; t < ntie; t += gridDim.x)
        repair_cluster(b, b.tie_list[t], tsm, ss);
    const uint32_t warp = threadIdx.x >> 5, lane = lane_id();
    // the large clusters' member counts (37,990 members took the cluster's own CTA 44,000 cycles)
    const uint32_t nitems = b.queue[6];
    for (uint32_t it = blockIdx.x; it < nitems; it += gridDim.x)
    {
        const uint2 item = b.pre_items[it];
        const uint32_t g = item.x;
        const uint32_t h = b.pre_nact[g]; // 0: counted with the hull
        if (h == 0u)
            continue;
        const uint32_t start = b.cl_start[g], n = b.cl_cnt[g];
        const uint32_t* mem = b.members + start;
        const int* keys = b.hs_stack + 2ull * start + 2ull * b.cl_rank[g];
        constexpr uint32_t kEach = kPreChunk / kHullThreads;
        uint32_t o[kEach];
#pragma unroll
        for (uint32_t u = 0; u < kEach; ++u)
        {
            const uint32_t i = item.y * kPreChunk + u * kHullThreads + threadIdx.x;
            o[u] = (i < n) ? mem[i] : 0xffffffffu; // (never below a key)
        }
#pragma unroll 2
        for (uint32_t j = 0; j < h; ++j)
        {
            const uint32_t key = static_cast<uint32_t>(keys[j]);
            uint32_t cnt = 0;
#pragma unroll
            for (uint32_t u = 0; u < kEach; ++u)
                cnt += (o[u] < key) ? 1u : 0u;
            cnt = __reduce_add_sync(0xffffffffu, cnt);
            if (lane == 0)
                atomicAdd(&b.hull_tmp[start + j], static_cast<int32_t>(cnt));
        }
    }
    if (!compute_obb)
        return;
    const uint32_t nbig = b.queue[2], nsmall = b.queue[3];
    const uint32_t K = nbig + nsmall;
    auto cluster = [&](uint32_t w) { return w < nbig ? work[w] : work[b.ncl - 1u - (w - nbig)]; };
    // hulls of more vertices than a warp's region holds: one per CTA, one box a warp
    for (uint32_t w = blockIdx.x; w < K; w += gridDim.x)
    {
        const uint32_t g = cluster(w);
        const int h = static_cast<int>(b.hull_cnt[g]);
        if (h <= kBoxWarpVerts)
            continue;
        const uint32_t start = b.cl_start[g];
        BoxSmem<kHullSmem>& bs = *reinterpret_cast<BoxSmem<kHullSmem>*>(tsm);
        const bool fast = h <= kHullSmem;
        if (fast)
            for (int j = threadIdx.x; j < h; j += kHullThreads)
            {
                const double2 p = b.hs_pts[start + j];
                bs.hp[j] = p;
                bs.pf[j] = make_float2(static_cast<float>(p.x), static_cast<float>(p.y)); // (float vertices: exact)
            }
        __syncthreads();
        const double2* P = fast ? bs.hp : (b.hs_pts + start);
        if (warp == 0)
            calipers_box(&b.state[scan_of_cluster(b, g)], P, fast ? bs.pf : nullptr, bs.ea, h,
                         b.hs_pairs + 4ull * start + 16ull * b.cl_rank[g], &b.obb_c[g]);
        else if (warp == 1)
            pca_box_warp(P, h, &b.obb_p[g]);
        __syncthreads();
    }
    BoxSmem<kBoxWarpVerts>& bs = reinterpret_cast<BoxSmem<kBoxWarpVerts>*>(tsm)[warp];
    for (uint32_t i = blockIdx.x + gridDim.x * warp; i < 2u * K; i += gridDim.x * (kHullThreads / 32))
    {
        const uint32_t g = cluster(i < K ? i : i - K);
        const int h = static_cast<int>(b.hull_cnt[g]);
        if (h > kBoxWarpVerts || b.cl_cnt[g] < 3u) // (fewer than three members: zero, written with the hull)
            continue;
        const uint32_t start = b.cl_start[g];
        for (int j = static_cast<int>(lane); j < h; j += 32)
        {
            const double2 p = b.hs_pts[start + j];
            bs.hp[j] = p;
            bs.pf[j] = make_float2(static_cast<float>(p.x), static_cast<float>(p.y));
        }
        __syncwarp();
        if (i < K)
            calipers_box(&b.state[scan_of_cluster(b, g)], bs.hp, bs.pf, bs.ea, h,
                         b.hs_pairs + 4ull * start + 16ull * b.cl_rank[g], &b.obb_c[g]);
        else
            pca_box_warp(bs.hp, h, &b.obb_p[g]);
        __syncwarp();
    }
}

// Dense hull output, one CTA per scan: hull_cnt becomes the exclusive scan of its hulls' sizes, from
// the scan's pt_off (K + 1 entries), and the hulls move behind one another into hull_out.
constexpr uint32_t kFinishThreads = 1024;

__global__ void __launch_bounds__(kFinishThreads) k_hull_finish(BatchDev b)
{
    pdl_enter();
    __shared__ uint32_t sm[33];
    __shared__ uint32_t soff[kFinishThreads + 1], sst[kFinishThreads];
    const ScanDev& sd = b.scans[blockIdx.x];
    const uint32_t K = min(b.state[blockIdx.x].n_clusters, sd.cluster_cap - 1u);
    uint32_t base = sd.pt_off;
    for (uint32_t k0 = 0; k0 <= K; k0 += kFinishThreads)
    {
        const uint32_t k = k0 + threadIdx.x, g = sd.cl_off + k;
        const uint32_t h = (k < K) ? b.hull_cnt[g] : 0u;
        uint32_t total;
        const uint32_t at = base + block_excl_scan(h, sm, &total); // (its barriers: the counts are read)
        if (k <= K)
            b.hull_cnt[g] = at;
        soff[threadIdx.x] = at;
        sst[threadIdx.x] = (k < K) ? b.cl_start[g] : 0u;
        if (threadIdx.x == 0)
            soff[kFinishThreads] = base + total;
        __syncthreads();
        // vertex by vertex: its hull is the last that starts at or before it
        for (uint32_t v = base + threadIdx.x; v < base + total; v += kFinishThreads)
        {
            uint32_t lo = 0u, hi = kFinishThreads - 1u;
            while (lo < hi)
            {
                const uint32_t mid = (lo + hi + 1u) / 2u;
                if (soff[mid] <= v)
                    lo = mid;
                else
                    hi = mid - 1u;
            }
            b.hull_out[v] = b.hull_tmp[sst[lo] + (v - soff[lo])];
        }
        base += total;
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------------
// Standalone single-polygon entry points (double inputs): one CTA.
//
// What bounds them: nearly every point of a cluster lies inside its hull, and sorting all of them
// (24-byte records, about log2(n)^2 / 2 passes) and walking them with one thread's FP64 orientation
// tests took most of the 62 ms that twelve polygons of 3 to 20,000 points needed for hull and both
// boxes (now 1.9 ms, 52 us a call). The points proven inside a polygon of input points
// are dropped first (Quickhull rounds as in hull_one, coordinates as floats), so the sort and the
// chain see a few dozen to a few hundred; 1,024 threads because the rounds stream over all points.
// Points whose coordinates are binary32 values (the processor's are) also take the FP32-screened
// orientation test, whose decisions are those of the FP64 expression.
// ---------------------------------------------------------------------------------------------
constexpr int kSingleThreads = 1024;
constexpr uint32_t kSingleCand = 512;     // candidates sorted in shared memory
constexpr uint32_t kSingleFilterMin = 64; // fewer points go straight to the sort
constexpr uint32_t kSingleEnough = 96;    // candidates few enough to end the rounds

struct SingleSmem
{
    HPt<double> cand[kSingleCand]; // as HPt<float> for binary32 points
    int stack[2 * kSingleCand + 2];
    float2 poly[2][kPolyCap];
    float4 erec[kPolyCap];
    float2 emar[kPolyCap];
    unsigned long long pkey[kPolyCap];
    unsigned long long ext[kDirs][kSingleThreads / 32];
    float2 dirs[kDirs];
    float red[kSingleThreads / 32];
    int npoly, grew, nact;
};

// Lists (act[0], n entries) the points not proven inside the hull and returns their number, or n
// when nothing can be dropped (the list is then not valid). `lf` receives the points as floats:
// themselves when `exact` (all binary32 values), else relative to the first point, where each
// coordinate is within 2^-24 R of the exact difference (R: the largest); the tests' margins add that
// error (a cross product of |e|, |q| errs by less than 2^-22 R (|e| + |q|)).
__device__ uint32_t single_filter(SingleSmem& sm, const double2* pts, uint32_t n, bool exact, float2* lf, uint32_t* act0,
                                  uint32_t* act1)
{
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5, tid = threadIdx.x, nt = blockDim.x;
    hull_dirs(sm.dirs);
    const double ox = exact ? 0.0 : pts[0].x, oy = exact ? 0.0 : pts[0].y;
    __syncthreads();
    Extremes16 ex;
    ex.init();
    float R = 0.0f;
    for (uint32_t i = tid; i < n; i += nt)
    {
        const double2 p = pts[i];
        const float2 q = make_float2(static_cast<float>(p.x - ox), static_cast<float>(p.y - oy));
        lf[i] = q;
        R = fmaxf(R, fmaxf(fabsf(q.x), fabsf(q.y)));
        ex.add(sm.dirs, q.x, q.y, i);
    }
    R = warp_max_f(R);
    if (lane == 0)
        sm.red[warp] = R;
#pragma unroll
    for (int d = 0; d < kDirs; ++d)
    {
        const unsigned long long v = warp_max64(ex.key(d));
        if (lane == 0)
            sm.ext[d][warp] = v;
    }
    __syncthreads();
    R = warp_max_f(sm.red[lane]); // every warp alike (kSingleThreads / 32 == 32)
    if (!(R > 1e-12f && R < 1e15f))
        return n; // float products would leave the normal range
    const float slack = exact ? 0.0f : 1e-6f * R;
    if (warp < static_cast<uint32_t>(kDirs))
    {
        const unsigned long long v = warp_max64(sm.ext[warp][lane]);
        if (lane == 0)
            sm.pkey[warp] = v;
    }
    __syncthreads();
    if (tid == 0)
        sm.npoly = first_polygon(lf, n, sm.pkey, sm.poly[0]);
    __syncthreads();
    uint32_t* act[2] = {act0, act1};
    int cur = -1, pb = 0; // -1: the active set is all points
    uint32_t nact = n;
    for (int round = 0; round < kRefineRounds && (round == 0 || nact > kSingleEnough); ++round)
    {
        const int np = sm.npoly;
        if (np < 3)
            break;
        const float2* poly = sm.poly[pb];
        for (int e = static_cast<int>(tid); e < np; e += static_cast<int>(nt))
        {
            sm.pkey[e] = 0ull;
            const float2 a = poly[e], c = poly[(e + 1 == np) ? 0 : e + 1];
            const float dx = c.x - a.x, dy = c.y - a.y;
            const float l1 = fabsf(dx) + fabsf(dy);
            sm.erec[e] = make_float4(a.x, a.y, dx, dy);
            sm.emar[e] = make_float2(1e-5f * l1 + slack, slack * l1 + 1e-30f);
        }
        if (tid == 0)
            sm.nact = 0;
        __syncthreads();
        const int nxt = (cur == 0) ? 1 : 0;
        for (uint32_t t = tid; t < ((nact + 31u) & ~31u); t += nt)
        {
            const bool live = t < nact;
            const uint32_t i = live ? ((cur < 0) ? t : act[cur][t]) : 0u;
            const float2 q = lf[i];
            bool in = true;
            for (int e = 0; live && e < np; ++e)
            {
                const float4 r = sm.erec[e];
                const float2 mg = sm.emar[e];
                const float qx = q.x - r.x, qy = q.y - r.y;
                const float cr = r.z * qy - r.w * qx;
                const float aq = fabsf(qx) + fabsf(qy);
                if (!(cr > mg.x * aq + mg.y))
                    in = false;
                if (cr < -(mg.x * aq + mg.y)) // any outside point may become a vertex
                {
                    const unsigned long long key = fkey_payload(-cr, i);
                    if (key > sm.pkey[e])
                        atomicMax(&sm.pkey[e], key);
                }
            }
            const uint32_t m = __ballot_sync(0xffffffffu, live && !in);
            uint32_t at = 0u;
            if (lane == 0 && m)
                at = static_cast<uint32_t>(atomicAdd(&sm.nact, __popc(m)));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (live && !in)
                act[nxt][at + static_cast<uint32_t>(__popc(m & ((1u << lane) - 1u)))] = i;
        }
        __syncthreads();
        cur = nxt;
        nact = static_cast<uint32_t>(sm.nact);
        // each edge's farthest outside point becomes a vertex behind the edge's first one (warp 0)
        if (warp == 0)
        {
            int add = 0;
            for (int e = static_cast<int>(lane); e < np; e += 32)
                add += (sm.pkey[e] != 0ull) ? 1 : 0;
            add = static_cast<int>(warp_sum(static_cast<uint32_t>(add)));
            const bool grow = add > 0 && np + add <= kPolyCap;
            int w = 0;
            for (int base = 0; grow && base < np; base += 32)
            {
                const int e = base + static_cast<int>(lane);
                const bool ins = e < np && sm.pkey[e] != 0ull;
                const uint32_t im = __ballot_sync(0xffffffffu, ins);
                const int at = w + static_cast<int>(lane) + __popc(im & ((1u << lane) - 1u));
                if (e < np)
                    sm.poly[pb ^ 1][at] = sm.poly[pb][e];
                if (ins)
                    sm.poly[pb ^ 1][at + 1] = lf[static_cast<uint32_t>(sm.pkey[e] & 0xffffffffull)];
                w += 32 + __popc(im);
            }
            if (lane == 0)
            {
                sm.grew = grow ? 1 : 0;
                if (grow)
                    sm.npoly = np + add;
            }
        }
        __syncthreads();
        if (!sm.grew)
            break;
        pb ^= 1;
    }
    if (cur < 0)
        return n;
    if (cur == 1)
    {
        for (uint32_t t = tid; t < nact; t += nt)
            act0[t] = act1[t];
        __syncthreads();
    }
    return nact;
}

// Sort and chain of m candidates (list: their input positions, null for all points; `placed` of them without a NaN
// coordinate, which alone take part: has_place): hull indices to out, returns the hull size; *tie: a vertex has an
// identical candidate.
template <typename T>
__device__ int single_chain(SingleSmem& sm, const double2* pts, const uint32_t* list, uint32_t m, uint32_t placed, HPt<T>* gl,
                            int* gstack, int32_t* out, bool* tie)
{
    auto run = [&](HPt<T>* C, int* H) {
        const uint32_t np2 = next_pow2(m);
        for (uint32_t t = threadIdx.x; t < np2; t += blockDim.x)
        {
            HPt<T> c{static_cast<T>(INFINITY), static_cast<T>(INFINITY), 0xffffffffu};
            if (t < m)
            {
                const uint32_t i = list ? list[t] : t;
                const double2 p = pts[i];
                if (p.x == p.x && p.y == p.y) // (the others end behind all points)
                    c = HPt<T>{static_cast<T>(p.x), static_cast<T>(p.y), i};
            }
            C[t] = c;
        }
        m = placed;
        __syncthreads();
        block_bitonic_sort(C, np2, [](const HPt<T>& x, const HPt<T>& y) { return hpt_less(x, y); });
        if (threadIdx.x < 64u)
        {
            const bool upper = threadIdx.x >= 32u;
            const int k = chain_half<32>(C, static_cast<int>(m), H + (upper ? m + 1 : 0), upper);
            if (lane_id() == 0)
                (upper ? sm.grew : sm.npoly) = k;
        }
        __syncthreads();
        const int kl = sm.npoly;
        // (a chain without orientations, where they overflow binary64, pops nothing: no more than out holds)
        const int h = (m < 2u) ? static_cast<int>(m) : min(kl + sm.grew - 2, static_cast<int>(m) + 1);
        bool t = false;
        for (int j = static_cast<int>(threadIdx.x); j < h; j += static_cast<int>(blockDim.x))
        {
            const int q = (j < kl) ? H[j] : H[static_cast<int>(m) + 2 + j - kl];
            const HPt<T> c = C[q];
            out[j] = static_cast<int32_t>(c.key);
            t |= (q > 0 && C[q - 1].x == c.x && C[q - 1].y == c.y) ||
                 (q + 1 < static_cast<int>(m) && C[q + 1].x == c.x && C[q + 1].y == c.y);
        }
        *tie = t;
        return h;
    };
    return (m <= kSingleCand) ? run(reinterpret_cast<HPt<T>*>(sm.cand), sm.stack) : run(gl, gstack);
}

// scratch: next_pow2(n) records of 24 bytes, stack: 2n + 8 ints (8-byte aligned). The floats of the
// filter lie in the stack area (the chain needs it only for candidates beyond shared memory, after the
// filter), its two lists at the end of the record area.
__global__ void __launch_bounds__(kSingleThreads) k_hull_single(const double2* pts, uint32_t n, HPt<double>* scratch,
                                                              int* stack, int32_t* out, uint32_t* n_out)
{
    pdl_enter();
    __shared__ __align__(16) unsigned char raw[sizeof(SingleSmem) > sizeof(isort::SortShared) ? sizeof(SingleSmem)
                                                                                             : sizeof(isort::SortShared)];
    SingleSmem& sm = *reinterpret_cast<SingleSmem*>(raw);
    bool exact = true, finite = true;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x)
    {
        const double2 p = pts[i];
        exact &= static_cast<double>(static_cast<float>(p.x)) == p.x && static_cast<double>(static_cast<float>(p.y)) == p.y;
        finite &= isfinite(p.x) && isfinite(p.y);
    }
    exact = __syncthreads_and(exact);
    finite = __syncthreads_and(finite);
    uint32_t placed = n;
    if (!finite)
    {
        if (threadIdx.x == 0)
            sm.nact = 0;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < n; i += blockDim.x)
            if (pts[i].x == pts[i].x && pts[i].y == pts[i].y)
                atomicAdd(&sm.nact, 1);
        __syncthreads();
        placed = static_cast<uint32_t>(sm.nact);
    }
    const size_t bytes = static_cast<size_t>(next_pow2(n)) * sizeof(HPt<double>);
    const size_t lists = bytes - 8ull * n; // the two lists of n entries start here
    uint32_t* act0 = reinterpret_cast<uint32_t*>(reinterpret_cast<unsigned char*>(scratch) + lists);
    uint32_t m = n;
    if (finite && n > kSingleFilterMin)
        m = single_filter(sm, pts, n, exact, reinterpret_cast<float2*>(stack), act0, act0 + n);
    // without a gain, or when the candidates' records would meet the list, every point takes part
    const bool all = m == n || (m > kSingleCand && static_cast<size_t>(next_pow2(m)) * sizeof(HPt<double>) > lists);
    if (all)
        m = n;
    __syncthreads();
    bool tie;
    int h;
    if (exact && finite)
        h = single_chain(sm, pts, all ? nullptr : act0, m, m, reinterpret_cast<HPt<float>*>(scratch), stack, out, &tie);
    else
        h = single_chain(sm, pts, all ? nullptr : act0, m, finite ? m : placed, scratch, stack, out, &tie);
    if (threadIdx.x == 0)
        *n_out = static_cast<uint32_t>(h);
    if (__syncthreads_or(tie))
    {
        // a vertex with an identical point: the reference's std::sort order decides which one. The
        // sort buffer takes the records (24 bytes each, as its entries) and the chain stack (2n + 8
        // ints, free now) the partition lists; the vertices' coordinates are read from the input.
        isort::SortShared& ss = *reinterpret_cast<isort::SortShared*>(raw);
        auto* rec = reinterpret_cast<HRec<double>*>(scratch);
        for (uint32_t i = threadIdx.x; i < n; i += blockDim.x)
            rec[i] = HRec<double>{pts[i].x, pts[i].y, i};
        __syncthreads();
        uint32_t* ge = reinterpret_cast<uint32_t*>(stack);
        hull_repair_ties(rec, n, out, h, [=](int j) { return pts[out[j]]; }, ge, ge + n, ss);
    }
}

// Antipodal pairs and a box of one polygon by one warp. A polygon of at most kBoxVerts binary32
// vertices takes the FP32-screened walk and calipers of the pipeline's hulls (same pairs, same box);
// others run in FP64 throughout (every visited edge's extents: 4 n^2 / 32 FP64 steps).
constexpr uint32_t kBoxVerts = 1024;

__global__ void __launch_bounds__(32) k_boxes_single(const double2* P, uint32_t n, int2* pairs, int cap, int kind,
                                                    lp_bounding_box* out, int* npairs_out)
{
    pdl_enter();
    __shared__ double2 sp[kBoxVerts];
    __shared__ float2 spf[kBoxVerts];
    __shared__ float ea[kBoxVerts];
    const uint32_t lane = lane_id();
    const bool local = n <= kBoxVerts;
    bool exact = true;
    float mabs = 0.0f, r2 = 0.0f;
    if (local)
    {
        for (uint32_t k = lane; k < n; k += 32)
        {
            const double2 p = P[k];
            const float2 f = make_float2(static_cast<float>(p.x), static_cast<float>(p.y));
            exact &= static_cast<double>(f.x) == p.x && static_cast<double>(f.y) == p.y;
            mabs = fmaxf(mabs, fmaxf(fabsf(f.x), fabsf(f.y)));
            sp[k] = p;
            spf[k] = f;
        }
        __syncwarp();
        for (uint32_t k = lane; k < n; k += 32)
        {
            const float lx = spf[k].x - spf[0].x, ly = spf[k].y - spf[0].y;
            r2 = fmaxf(r2, lx * lx + ly * ly);
        }
        mabs = warp_max_f(mabs);
        r2 = warp_max_f(r2) * 1.001f;
    }
    const bool fast = __all_sync(0xffffffffu, exact) && local && mabs < 1e15f;
    const double2* V = local ? sp : P;
    if (kind == 1)
    {
        if (lane == 0 && npairs_out)
            *npairs_out = 0;
        pca_box_warp(V, static_cast<int>(n), out);
        return;
    }
    int np = 0;
    if (lane == 0)
    {
        if (fast)
            np = antipodal_pairs(AreaCmpFiltered(V, spf, mabs, r2), static_cast<int>(n), pairs, cap);
        else
            np = antipodal_pairs(AreaCmpFp64{V}, static_cast<int>(n), pairs, cap);
    }
    np = __shfl_sync(0xffffffffu, np, 0);
    if (lane == 0 && npairs_out)
        *npairs_out = np;
    if (np > cap)
        np = cap;
    __syncwarp();
    if (kind == 0)
    {
        if (fast)
            calipers_fast(V, spf, static_cast<int>(n), pairs, np, ea, r2, out);
        else
            calipers_warp(V, static_cast<int>(n), pairs, np, out);
    }
}
} // namespace

namespace
{
// The vehicle gates (processor.cpp:679-755), one warp per cluster. Lane 0 checks the hull size, the
// point count, the height against the table's limits and the volume of the hull area (polygonArea,
// polygonizer.hpp:186-198, binary64 in hull order); a cluster that passes is boxed by rotating
// calipers over all its points in input order, which is what the reference passes
// (polygonizer_points_), with the same routine the hulls' boxes use; lane 0 then checks the hull's
// share of the box (> 0.4) and the box's edges against the vehicle types in order.
__global__ void k_obj_gate(ObjDev o, VehicleTableDev vt, int enabled, double2* P, float2* Pf, float* ea, int2* pairs,
                           ScanState* st)
{
    pdl_enter();
    const uint32_t l = blockIdx.x * (blockDim.x / 32u) + threadIdx.x / 32u;
    if (l >= o.K)
        return;
    const uint32_t lane = lane_id();
    const uint32_t off = o.cl_off[l], nc = o.cl_off[l + 1] - off;
    const uint32_t h0 = o.hull_off[l], h = o.hull_off[l + 1] - h0;
    const double height = static_cast<double>(o.zmax[l]) - static_cast<double>(o.zmin[l]);
    double area = 0.0, volume = 0.0;
    int pass = 0;
    if (lane == 0)
    {
        lp_bounding_box none;
        for (int k = 0; k < 4; ++k)
            none.corners[k][0] = none.corners[k][1] = 0.0;
        none.area = 0.0f;
        none.angle_rad = 0.0f;
        none.is_valid = 0;
        o.boxes[l] = none;
        o.cls[l] = -1;
        if (enabled && h >= 3 && nc > 150 && height > vt.min_h && height < vt.max_h)
        {
            auto vx = [&](uint32_t k) { return static_cast<double>(o.cloud[off + static_cast<uint32_t>(o.hull_idx[h0 + k])].x); };
            auto vy = [&](uint32_t k) { return static_cast<double>(o.cloud[off + static_cast<uint32_t>(o.hull_idx[h0 + k])].y); };
            double a = 0.0;
            for (uint32_t k = 0; k + 1 < h; ++k)
                a += (vx(k) * vy(k + 1)) - (vx(k + 1) * vy(k));
            a += (vx(h - 1) * vy(0)) - (vx(0) * vy(h - 1));
            area = fabs(a) * 0.5;
            volume = area * height;
            pass = (volume > vt.min_v && volume < vt.max_v) ? 1 : 0;
        }
    }
    pass = __shfl_sync(0xffffffffu, pass, 0);
    if (!pass)
        return;
    area = __shfl_sync(0xffffffffu, area, 0);
    volume = __shfl_sync(0xffffffffu, volume, 0);
    for (uint32_t k = lane; k < nc; k += 32)
    {
        const lp_xyzrgb& p = o.cloud[off + k];
        P[off + k] = make_double2(static_cast<double>(p.x), static_cast<double>(p.y));
        Pf[off + k] = make_float2(p.x, p.y);
    }
    __syncwarp();
    calipers_box(st, P + off, Pf + off, ea + off, static_cast<int>(nc), pairs + 4ull * off + 16ull * l, &o.boxes[l]);
    __syncwarp();
    if (lane != 0)
        return;
    const lp_bounding_box box = o.boxes[l];
    if (!box.is_valid || !(area / static_cast<double>(box.area) > 0.4))
        return;
    auto dist = [&](int a, int c) {
        const double dx = box.corners[a][0] - box.corners[c][0];
        const double dy = box.corners[a][1] - box.corners[c][1];
        return sqrt(dx * dx + dy * dy);
    };
    const double e1 = dist(0, 1), e2 = dist(1, 2);
    const double len = fmax(e1, e2), wid = fmin(e1, e2);
    for (int v = 0; v < 5; ++v)
    {
        const double* d = vt.dims[v];
        const double* bb = vt.bounds[v];
        if (len > d[0] && len < d[1] && wid > d[2] && wid < d[3] && height > d[4] && height < d[5] && volume > bb[0] &&
            volume < bb[1] && area > bb[2] && area < bb[3])
        {
            o.cls[l] = v;
            break;
        }
    }
}
} // namespace

void launch_objects_gates(cudaStream_t st, const ObjDev& o, const VehicleTableDev& vt, int enabled, double2* P,
                          float2* Pf, float* ea, int2* pairs, ScanState* state, uint64_t& launches)
{
    if (o.K == 0)
        return;
    k_obj_gate<<<div_up(o.K, 4u), 128, 0, st>>>(o, vt, enabled, P, Pf, ea, pairs, state);
    launches += 1;
}

void launch_polygons(Launcher& L, const BatchDev& b, const BatchHost& hb, int compute_obb)
{
    LP_LAUNCH(L, k_hull_worklist, div_up(b.ncl, 256u), 256, b);
    launch_cluster_scatter(L, b);
    LP_LAUNCH(L, k_hull_pre_ext, static_cast<uint32_t>(sm_count()) * 4u, 256, b);
    LP_LAUNCH(L, k_hull_pre_ref, static_cast<uint32_t>(sm_count()) * 4u, 256, b);
    const int sms = sm_count();
    LP_LAUNCH_SMEM(L, k_hull, static_cast<uint32_t>(sms) * hb.hull_ctas_per_sm, kHullThreads, kHullDynSmem, b, compute_obb,
                   static_cast<const uint32_t*>(b.hull_work));
    LP_LAUNCH_SMEM(L, k_hull_boxes, static_cast<uint32_t>(sms) * (compute_obb ? 2u : 1u), kHullThreads, kTieDynSmem, b, compute_obb,
                   static_cast<const uint32_t*>(b.hull_work));
    LP_LAUNCH(L, k_hull_finish, static_cast<uint32_t>(b.nscan), kFinishThreads, b);
}

void init_kernel_attributes()
{
    init_kdtree_attributes();
    cudaFuncSetAttribute(k_hull, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kHullDynSmem));
    cudaFuncSetAttribute(k_hull_boxes, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kTieDynSmem));
}

int sm_count()
{
    // asked for at most launches of a run: the attribute is read once per device
    static std::atomic<int> known[64];
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && (n = known[dev].load(std::memory_order_relaxed)) > 0)
        return n;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    n = n > 0 ? n : 1;
    if (dev >= 0 && dev < 64)
        known[dev].store(n, std::memory_order_relaxed);
    return n;
}

void launch_hull_single(Launcher& L, const double2* pts, uint32_t n, void* scratch, int* stack, int32_t* out,
                        uint32_t* n_out)
{
    LP_LAUNCH(L, k_hull_single, 1, kSingleThreads, pts, n, reinterpret_cast<HPt<double>*>(scratch), stack, out, n_out);
}

void launch_boxes_single(Launcher& L, const double2* P, uint32_t n, int2* pairs, int cap, int kind, lp_bounding_box* out,
                         int* npairs_out)
{
    LP_LAUNCH(L, k_boxes_single, 1, 32, P, n, pairs, cap, kind, out, npairs_out);
}
} // namespace lpg

// =============================================================================================
// Convex hull without any allocation (lp_convex_hull_noalloc, lidar_gb300.h).
//
// For callers that must not allocate device memory: code that runs inside a real-time loop
// whose memory is reserved up front (cudaMalloc can synchronise the device and stall other
// work), plugin hosts whose allocator policy forbids it, or code paths where an allocation
// failure cannot be handled. The caller passes device buffers for the input and the output; the
// kernel's working memory is the file-scope array below, which every GPU that loads this library
// holds (2.1 MiB) until the process exits.
// =============================================================================================
namespace
{
constexpr uint32_t kNoallocMaxPoints = LP_NOALLOC_HULL_MAX_POINTS;
// sort buffer: next_pow2(n) points of 24 bytes; chain stack: 2n + 8 ints
constexpr size_t kNoallocSortBytes = static_cast<size_t>(kNoallocMaxPoints) * 24;
constexpr size_t kNoallocStackBytes = (2 * static_cast<size_t>(kNoallocMaxPoints) + 8) * 4;

static __device__ __align__(256) unsigned char g_noalloc_hull_scratch[kNoallocSortBytes + kNoallocStackBytes];

constexpr int kNoallocMaxDevices = 64;
std::mutex g_noalloc_mutex;
void* g_noalloc_ptr[kNoallocMaxDevices] = {};

__global__ void k_hull_noalloc_small(uint32_t n, int32_t* out, uint32_t* n_out)
{
    // fewer than 3 points: indices 0..n-1 (polygonizer.cpp:36-41)
    if (threadIdx.x < n)
        out[threadIdx.x] = static_cast<int32_t>(threadIdx.x);
    if (threadIdx.x == 0)
        *n_out = n;
}
} // namespace

extern "C" lp_status lp_convex_hull_noalloc(const double* d_xy, uint32_t n, int32_t* d_indices_out, uint32_t* d_n_out,
                                            void* stream)
{
    if (!d_n_out || (n && (!d_xy || !d_indices_out)))
        return LP_ERR_BAD_ARG;
    if (n > kNoallocMaxPoints)
        return LP_ERR_CAPACITY; // more points than the static working array holds
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoallocMaxDevices)
    {
        cudaGetLastError();
        return LP_ERR_NO_DEVICE;
    }
    void* scratch = nullptr;
    {
        // once per device, with that device current: the device address of the static array
        std::lock_guard<std::mutex> lock(g_noalloc_mutex);
        if (!g_noalloc_ptr[dev])
        {
            void* p = nullptr;
            const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_hull_scratch);
            if (e != cudaSuccess || !p)
            {
                cudaGetLastError();
                return LP_ERR_CUDA;
            }
            g_noalloc_ptr[dev] = p;
        }
        scratch = g_noalloc_ptr[dev];
    }
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    // the status is this launch's own (cudaLaunchKernel's return value), so an error left behind
    // by some other code in the process is neither reported as this call's nor cleared
    cudaError_t e;
    if (n < 3)
    {
        void* args[] = {&n, &d_indices_out, &d_n_out};
        e = cudaLaunchKernel(reinterpret_cast<const void*>(&k_hull_noalloc_small), dim3(1), dim3(32), args, 0, st);
    }
    else
    {
        // every scratch element the kernel reads is written earlier in the same launch, so the
        // previous call's contents never leak into this one
        auto* sort_buf = reinterpret_cast<lpg::HPt<double>*>(scratch);
        int* stack = reinterpret_cast<int*>(static_cast<unsigned char*>(scratch) + kNoallocSortBytes);
        const double2* xy = reinterpret_cast<const double2*>(d_xy);
        void* args[] = {&xy, &n, &sort_buf, &stack, &d_indices_out, &d_n_out};
        e = cudaLaunchKernel(reinterpret_cast<const void*>(&lpg::k_hull_single), dim3(1), dim3(lpg::kSingleThreads), args,
                             0, st);
    }
    return e == cudaSuccess ? LP_OK : LP_ERR_CUDA;
}
