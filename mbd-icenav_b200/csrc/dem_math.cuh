// dem_math.cuh — scalar helpers with the NumPy/JAX semantics the frame step relies on.
//
// The reference computes with jnp (XLA) ops whose NaN and rounding semantics
// differ from C's fmin/fmax: jnp.maximum/minimum/clip propagate NaN, jnp.sign(0)
// is 0, float `%` is a floor-mod whose result takes the divisor's sign.  The
// kernels are compiled with -fmad=false so that a*b+c rounds twice, as NumPy
// and XLA-CPU do, which keeps contact and fracture predicates computed from
// identical inputs identical.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

namespace dem {

template <typename T> struct vec2_of;
template <> struct vec2_of<float> { typedef float2 type; };
template <> struct vec2_of<double> { typedef double2 type; };

template <typename T>
__device__ __forceinline__ typename vec2_of<T>::type ld2(const T* p, int i) {
    return reinterpret_cast<const typename vec2_of<T>::type*>(p)[i];
}
template <typename T>
__device__ __forceinline__ void st2(T* p, int i, T x, T y) {
    typename vec2_of<T>::type v;
    v.x = x;
    v.y = y;
    reinterpret_cast<typename vec2_of<T>::type*>(p)[i] = v;
}

// jnp.maximum / jnp.minimum: NaN in either operand gives NaN.
template <typename T> __device__ __forceinline__ T jmax(T a, T b) {
    return (a != a) ? a : ((b != b) ? b : (a > b ? a : b));
}
template <typename T> __device__ __forceinline__ T jmin(T a, T b) {
    return (a != a) ? a : ((b != b) ? b : (a < b ? a : b));
}
// float has the NaN-propagating forms as one instruction (five otherwise)
template <> __device__ __forceinline__ float jmax<float>(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
template <> __device__ __forceinline__ float jmin<float>(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
// jnp.clip(x, lo, hi) == minimum(maximum(x, lo), hi)
template <typename T> __device__ __forceinline__ T jclip(T x, T lo, T hi) {
    return jmin(jmax(x, lo), hi);
}
template <typename T> __device__ __forceinline__ T jsign(T x) {
    return (x > T(0)) ? T(1) : ((x < T(0)) ? T(-1) : x);  // 0 -> 0, NaN -> NaN
}
// Python / NumPy float remainder: result in [0, m) for m > 0.
template <typename T> __device__ __forceinline__ T pymod(T x, T m) {
    if (x > T(0) && x < m) return x;  // fmod returns it too, at the length of its general path
    T r = fmod(x, m);
    if (r != T(0)) {
        if ((m < T(0)) != (r < T(0))) r += m;
    } else {
        r = copysign(T(0), m);
    }
    return r;
}
template <typename T> __device__ __forceinline__ bool jfinite(T x) { return isfinite(x); }

__device__ __forceinline__ float jpow(float a, float b) { return powf(a, b); }
__device__ __forceinline__ double jpow(double a, double b) { return pow(a, b); }
__device__ __forceinline__ float jsqrt(float a) { return sqrtf(a); }
__device__ __forceinline__ double jsqrt(double a) { return sqrt(a); }
__device__ __forceinline__ void jsincos(float a, float* s, float* c) { sincosf(a, s, c); }
__device__ __forceinline__ void jsincos(double a, double* s, double* c) { sincos(a, s, c); }
__device__ __forceinline__ float jcos(float a) { return cosf(a); }
__device__ __forceinline__ double jcos(double a) { return cos(a); }
__device__ __forceinline__ float jsin(float a) { return sinf(a); }
__device__ __forceinline__ double jsin(double a) { return sin(a); }

// ─── correctly rounded division and square root without branches ────────────
// Newton iterations from the hardware's seed and Markstein's final steps
// (P. Markstein, IBM J. Res. Dev. 34, 1990): with y = 1/d rounded to nearest and q
// within an ulp of x/d, the exact remainder e = x - q d gives x/d rounded to nearest
// as q + e y; an iteration from a y within an ulp of 1/d rounds it to nearest unless
// d's significand is all ones.  With g within an ulp of sqrt(x) and h close to
// 1/(2 sqrt(x)), the exact x - g^2 gives the root rounded to nearest as g + (x - g^2) h.
// The operators' values while operands stay within kFastLo..kFastHi, where no
// remainder underflows, or the numerator is zero (the quotient's sign is then not the
// operator's: callers add it to sums, which it does not change); callers test that
// and leave the rest to the operators.  tests/test_gpu_fast_math.py compares them:
// every float significand of the root, the roots and quotients closest to half way
// between two results, 2^30 random and edge operands of each.  One after another, the
// operators' range checks and branches are what a substep of a single warp waits
// for: a block of these interleaves instead, and a reciprocal serves several quotients.
template <typename T> struct FastRange;
template <> struct FastRange<float> {
    static __device__ __forceinline__ float lo() { return 8.6736174e-19f; }  // 2^-60
    static __device__ __forceinline__ float hi() { return 1.1529215e18f; }   // 2^60
};
template <> struct FastRange<double> {
    static __device__ __forceinline__ double lo() { return 3.8725919148493183e-121; }  // 2^-400
    static __device__ __forceinline__ double hi() { return 2.5822498780869086e120; }   // 2^400
};
// a numerator or divisor that the fast forms may take
template <typename T> __device__ __forceinline__ bool fast_ok(T x) {
    const T ax = fabs(x);
    return ax >= FastRange<T>::lo() && ax <= FastRange<T>::hi();
}
template <typename T> __device__ __forceinline__ bool fast_num(T x) { return x == T(0) || fast_ok(x); }

__device__ __forceinline__ float rcp_nr(float d) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
    return fmaf(fmaf(-d, y, 1.0f), y, y);
}
__device__ __forceinline__ double rcp_nr(double d) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = fma(-d, y, 1.0);  // 2^-19 at most: e + e^2 leaves 2^-57
    y = fma(fma(e, e, e), y, y);
    y = fma(fma(-d, y, 1.0), y, y);
    // 2^k (1 - 2^-53): 1/d is half way and a little more above 2^-k, where y has stayed
    constexpr long long kOnes = 0xfffffffffffffll;
    const bool ones = (__double_as_longlong(d) & kOnes) == kOnes;
    return __longlong_as_double(__double_as_longlong(y) + (ones ? 1 : 0));
}
// x / d with y = rcp_nr(d)
__device__ __forceinline__ float div_nr(float x, float d, float y) {
    float q = x * y;
    q = fmaf(fmaf(-d, q, x), y, q);
    return fmaf(fmaf(-d, q, x), y, q);
}
__device__ __forceinline__ double div_nr(double x, double d, double y) {
    double q = x * y;
    q = fma(fma(-d, q, x), y, q);
    return fma(fma(-d, q, x), y, q);
}
// sqrt(x); h gets 1 / (2 sqrt(x)) to working accuracy
__device__ __forceinline__ float sqrt_nr(float x, float& h) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    float g = x * y;
    h = 0.5f * y;
    const float r = fmaf(-h, g, 0.5f);
    g = fmaf(g, r, g);
    h = fmaf(h, r, h);
    return fmaf(fmaf(-g, g, x), h, g);
}
__device__ __forceinline__ double sqrt_nr(double x, double& h) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double g = x * y;
    h = 0.5 * y;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const double r = fma(-h, g, 0.5);
        g = fma(g, r, g);
        h = fma(h, r, h);
    }
    return fma(fma(-g, g, x), h, g);
}

// NumPy's pairwise summation for a contiguous reduction of n <= 128 items
// (numpy/_core/src/umath/loops_utils.h): sequential below 8 items, otherwise
// eight interleaved partial sums combined as ((r0+r1)+(r2+r3))+((r4+r5)+(r6+r7))
// followed by the tail.  Used for the masked vertex mean of ship-contact pass 2.
template <typename T>
__device__ __forceinline__ T np_pairwise_sum(const T* a, int n) {
    if (n < 8) {
        T res = T(0);
        // NumPy starts from -0.0 for n < 8 and adds in order
        res = -T(0);
        for (int i = 0; i < n; ++i) res += a[i];
        return res;
    }
    T r[8];
    for (int j = 0; j < 8; ++j) r[j] = a[j];
    int i = 8;
    for (; i < n - (n % 8); i += 8)
        for (int j = 0; j < 8; ++j) r[j] += a[i + j];
    T res = ((r[0] + r[1]) + (r[2] + r[3])) + ((r[4] + r[5]) + (r[6] + r[7]));
    for (; i < n; ++i) res += a[i];
    return res;
}

// Monotone bit patterns of non-negative floats for atomicMax.
__device__ __forceinline__ unsigned f2ord(float x) { return __float_as_uint(x); }
__device__ __forceinline__ unsigned long long d2ord(double x) {
    return (unsigned long long)__double_as_longlong(x);
}

__device__ __forceinline__ unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ unsigned atom_add_release_u32(unsigned* p, unsigned v) {
    unsigned old;
    asm volatile("atom.add.release.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}
__device__ __forceinline__ unsigned atom_add_acqrel_u32(unsigned* p, unsigned v) {
    unsigned old;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}
__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long atom_add_release_u64(unsigned long long* p, unsigned long long v) {
    unsigned long long old;
    asm volatile("atom.add.release.gpu.global.u64 %0, [%1], %2;" : "=l"(old) : "l"(p), "l"(v) : "memory");
    return old;
}
__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_u32(unsigned* p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

}  // namespace dem
