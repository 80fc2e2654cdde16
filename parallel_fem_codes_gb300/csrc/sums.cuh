// Device sums and the Givens step shared by the streaming and the on-chip
// restart cycles.
#pragma once
#include "system.h"

namespace fg {

// Running sum of T values with the error of a 48-bit (FP32) or plain (FP64)
// accumulator: FP32 by error-free two-sums, because this part's FP64 pipe
// issues one warp instruction in 16 cycles.
template <typename T> struct Sum;
template <> struct Sum<double> {
    double h = 0.0;
    __device__ __forceinline__ void add(double v) { h += v; }
    __device__ __forceinline__ void add_square(double v) { h += v * v; }
    __device__ __forceinline__ void fold(int o) { h += __shfl_xor_sync(0xffffffffu, h, o); }
    // plus what lane ^ o gives
    __device__ __forceinline__ void take(const Sum &give, int o) { h += __shfl_xor_sync(0xffffffffu, give.h, o); }
    __device__ __forceinline__ double rounded() const { return h; }
    __device__ __forceinline__ double value() const { return h; }
};
template <> struct Sum<float> {
    float h = 0.f, l = 0.f;
    __device__ __forceinline__ void add(float v)
    {
        const float s = __fadd_rn(h, v), t = __fsub_rn(s, h);
        l = __fadd_rn(l, __fadd_rn(__fsub_rn(h, __fsub_rn(s, t)), __fsub_rn(v, t)));
        h = s;
    }
    __device__ __forceinline__ void add_square(float v)
    {
        const float p = __fmul_rn(v, v);
        l = __fadd_rn(l, __fmaf_rn(v, v, -p));
        add(p);
    }
    // (ah + al) b, the high product exactly
    __device__ __forceinline__ void add_product(float ah, float al, float b)
    {
        const float p = __fmul_rn(ah, b);
        l = __fadd_rn(l, __fmaf_rn(al, b, __fmaf_rn(ah, b, -p)));
        add(p);
    }
    __device__ __forceinline__ void fold(int o)
    {
        const float oh = __shfl_xor_sync(0xffffffffu, h, o), ol = __shfl_xor_sync(0xffffffffu, l, o);
        // the two partners add in the same order, so both hold the same sum
        const bool up = (threadIdx.x & o) != 0;
        const float ah = up ? oh : h, al = up ? ol : l, bh = up ? h : oh, bl = up ? l : ol;
        h = ah;
        l = __fadd_rn(al, bl);
        add(bh);
    }
    __device__ __forceinline__ void take(const Sum &give, int o)
    {
        l = __fadd_rn(l, __shfl_xor_sync(0xffffffffu, give.l, o));
        add(__shfl_xor_sync(0xffffffffu, give.h, o));
    }
    __device__ __forceinline__ float rounded() const { return __fadd_rn(h, l); }
    __device__ __forceinline__ double value() const { return (double)h + (double)l; }
};

// The power of two that brings m into [1, 2) (1 where m is 0 or not finite): what
// is kept in FP32 is kept times it, so that its range is FP64's.  The
// newest basis vector is stored unscaled, times this for an m of the size of
// M^-1 A v_0: its products with the basis then grow with the operator's scale,
// not with its cube, and a power of two changes no rounding.
// (A power whose reciprocal is normal too; by the exponent's bits.)
__device__ __forceinline__ float unit_scale(float m)
{
    const int e = (__float_as_int(m) >> 23) & 0xff;
    return m == 0.f || e == 0xff ? 1.f : __int_as_float((254 - max(1, min(e, 253))) << 23);
}
__device__ __forceinline__ double unit_scale(double m)
{
    const int e = (__double2hiint(m) >> 20) & 0x7ff;
    return m == 0.0 || e == 0x7ff ? 1.0 : __hiloint2double((2046 - max(1, min(e, 2045))) << 20, 0);
}

// Givens step i (pgmres.c:111-157) by one warp: the coefficients h[0..i] and
// h(i+1, i) = hn of column i; rotations and right-hand side in cs, sn, g
// (kmax, kmax, kmax + 1), the rotated column to H; t, a: scratch of kmax.  The
// recurrence down the column is one FMA a row (its products are formed by the
// lanes).  Returns true when the cycle ends.
struct Rot {
    double *cs, *sn, *g, *t, *a;
    int iters, steps, breakdown;
    double rho;
};
template <typename T>
__device__ __forceinline__ bool givens(double *H, int km, Rot &R, int i, const T *h, double hn, double target)
{
    const int lane = threadIdx.x & 31;
    for (int j = lane; j < i; j += 32) R.t[j] = R.cs[j] * (double)h[j + 1];
    __syncwarp();
    if (lane == 0) {
        double a = (double)h[0];
        for (int j = 0; j < i; ++j) {
            R.a[j] = a;
            a = fma(-R.sn[j], a, R.t[j]);
        }
        R.a[i] = a;
    }
    __syncwarp();
    for (int j = lane; j < i; j += 32) H[j * km + i] = R.cs[j] * R.a[j] + R.sn[j] * (double)h[j + 1];
    const double a = R.a[i], q = a * a + hn * hn, ri = rsqrt(q), r = q * ri;
    const double cs = a * ri, sn = hn * ri, gi = R.g[i];
    __syncwarp();
    if (lane == 0) {
        R.cs[i] = cs;
        R.sn[i] = sn;
        H[i * km + i] = r;
        R.g[i + 1] = -sn * gi;
        R.g[i] = cs * gi;
    }
    __syncwarp();
    R.rho = fabs(sn * gi);
    R.iters = R.steps = i + 1;
    if (!(q > 0.0) || !isfinite(R.rho)) {
        R.breakdown = 1;
        if (!(q > 0.0)) R.steps = i;         // column i unusable
        return true;
    }
    return !(R.rho > target) || i + 1 >= km - 1 || !(hn > 0.0);
}

// y of the cycle's triangular system (pgmres.c:163-171) by one warp: columns
// from the last to the first, each lane keeping two rows of the right-hand side
__device__ __forceinline__ void back_substitute(const double *H, int km, const double *g, int m, double *y)
{
    const int lane = threadIdx.x & 31;
    double g0 = lane < m ? g[lane] : 0.0, g1 = lane + 32 < m ? g[lane + 32] : 0.0;
    const double d0 = lane < m ? 1.0 / H[lane * km + lane] : 0.0;
    const double d1 = lane + 32 < m ? 1.0 / H[(lane + 32) * km + lane + 32] : 0.0;
    for (int c1 = m - 1; c1 >= 0; c1 -= 4) {
        double h0[4], h1[4];                 // four columns' loads together
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int c = c1 - q;
            h0[q] = lane < c ? H[lane * km + c] : 0.0;
            h1[q] = lane + 32 < c ? H[(lane + 32) * km + c] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int c = c1 - q;
            if (c < 0) break;
            const double yc = __shfl_sync(0xffffffffu, c < 32 ? g0 * d0 : g1 * d1, c & 31);
            if (lane == 0) y[c] = yc;
            g0 -= h0[q] * yc;
            g1 -= h1[q] * yc;
        }
    }
    __syncwarp();
}

// y as FP32 pairs times a power of two, by one warp, m <= 64: yh, yl and the
// power's reciprocal.  Sums of V y are then formed in error-free FP32 pairs (the
// FP64 FMA and the conversion a value would bind: 513 x 513 FP32 26.0 -> 27.4 ms a solve, 32
// streaming systems 229 -> 256), with the range of FP64.  The solution is off from the exact
// one by as much as with FP64 sums (432 solves of 961 to 25k equations, FP64 /
// pairs 1.00 where the last bits show, 1.0 to 1.2 at a tolerance of 1e-11).
__device__ __forceinline__ void split_y(const double *y, const double *scale, int m, float *yh, float *yl, int stride, double *back)
{
    const int lane = threadIdx.x & 31;
    double a = lane < m ? y[lane] : 0.0, b = lane + 32 < m ? y[lane + 32] : 0.0;
    if (scale) {
        if (lane < m) a *= scale[lane];
        if (lane + 32 < m) b *= scale[lane + 32];
    }
    double t = fmax(fabs(a), fabs(b));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t = fmax(t, __shfl_xor_sync(0xffffffffu, t, o));
    const double u = unit_scale(t);
    a *= u;
    b *= u;
    if (lane < m) {
        yh[stride * lane] = (float)a;
        yl[stride * lane] = (float)(a - (double)(float)a);
    }
    if (lane + 32 < m) {
        yh[stride * (lane + 32)] = (float)b;
        yl[stride * (lane + 32)] = (float)(b - (double)(float)b);
    }
    if (lane == 0) *back = 1.0 / u;
}

}  // namespace fg
