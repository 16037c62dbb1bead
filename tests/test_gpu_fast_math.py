"""The branch-free division, square root and overlap^1.5 of the resident substeps against
the operators and the branching form, on the device: the same value wherever callers
take them (kFastLo..kFastHi, a zero numerator), bit for bit but for the sign of zero."""
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include "dem_kernels.cuh"
using namespace dem;
typedef unsigned long long u64;

__device__ u64 mix(u64 z) {  // splitmix64
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
template <typename T> struct Bits;
template <> struct Bits<float> {
    static const int sig = 23, ends = 60;
    __device__ static float make(u64 s, int e) {
        return __uint_as_float((unsigned)(s & 0x7fffffu) | (unsigned)(e + 127) << 23);
    }
};
template <> struct Bits<double> {
    static const int sig = 52, ends = 400;
    __device__ static double make(u64 s, int e) {
        return __longlong_as_double((long long)((s & 0xfffffffffffffull) | (u64)(e + 1023) << 52));
    }
};
// a significand: random, or one of the edges (few low or high bits set or clear)
template <typename T> __device__ u64 significand(u64 r) {
    const u64 all = (1ull << Bits<T>::sig) - 1;
    const u64 low = (r >> 8) & 7, a = (r >> 16) % Bits<T>::sig;
    switch (r & 7) {
        case 0: return low;                                  // next above a power of two
        case 1: return all - low;                            // next below
        case 2: return (1ull << a) + low;                    // a single bit, and close to it
        case 3: return (all << a) & all;                     // a run of ones
        default: return (mix(r) >> 5) & all;
    }
}
// a positive operand of the fast range, its ends among them
template <typename T> __device__ T operand(u64 r) {
    const int E = Bits<T>::ends, e = (int)(mix(r ^ 1) % (2 * E + 1)) - E;
    return e == E ? Bits<T>::make(0, E) : Bits<T>::make(significand<T>(r), e);
}
template <typename T> __device__ void expect(T got, T want, u64* bad) {
    if (!(got == want)) atomicAdd(bad, 1ull);
}
template <typename T> __global__ void divisions(u64 n, u64* bad) {
    for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        const u64 r = mix(2 * i), q = mix(2 * i + 1);
        T x = operand<T>(r), d = operand<T>(q);
        if (r >> 63) x = -x;
        if (q >> 62 == 3) d = -d;
        if ((i & 1023) == 0) x = (i & 1024) ? T(0) : -T(0);
        if (!fast_num(x) || !fast_ok(d)) atomicAdd(bad, 1ull);
        expect(div_nr(x, d, rcp_nr(d)), x / d, bad);
    }
}
// What the double form takes from the hardware's reciprocal: 19 bits.
__global__ void seeds(u64 n, u64* bad) {
    for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        const double d = operand<double>(mix(i));
        double y;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
        if (!(fabs(fma(-d, y, 1.0)) <= 0x1p-19)) atomicAdd(bad, 1ull);
    }
}
// The quotients that are hardest to round: with p-bit x and d, x 2^s = m d + c for a
// (p + 1)-bit odd m (half way between two results) and a small odd c.
template <typename T> __global__ void hard_divisions(u64 n, u64* bad, u64* cases) {
    const int p = Bits<T>::sig + 1;
    typedef unsigned __int128 u128;
    for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        u64 D = (1ull << (p - 1)) | (sizeof(T) == 4 ? i : significand<T>(mix(i))) & ((1ull << (p - 1)) - 1) | 1ull;
        u64 inv = D;  // of an odd number modulo 2^64: three more correct bits, then twice as many each
        for (int k = 0; k < 5; ++k) inv *= 2 - D * inv;
        for (int c = -15; c <= 15; c += 2)
            for (int s = p; s <= p + 1; ++s) {
                u64 m = (0 - (u64)(long long)c) * inv & ((1ull << s) - 1);
                if (s == p) m |= 1ull << p;
                const u128 v = (u128)m * D + (u128)(__int128)c;
                if (m < 1ull << p || (v >> (s + p - 1)) != 1) continue;
                const T x = Bits<T>::make((u64)(v >> s), 0), d = Bits<T>::make(D, 0);
                expect(div_nr(x, d, rcp_nr(d)), x / d, bad);
                if ((v & (((u128)1 << s) - 1)) == 0) atomicAdd(cases, 1ull);
            }
    }
}
template <typename T> __device__ void one_root(T x, u64* bad) {
    T h;
    if (!fast_ok(x)) atomicAdd(bad, 1ull);
    expect(sqrt_nr(x, h), jsqrt(x), bad);
    const T one = h * T(2) * jsqrt(x);  // 1 / (2 sqrt(x)) to working accuracy
    if (!(fabs(one - T(1)) < T(8) * (sizeof(T) == 4 ? T(1.2e-7) : T(2.3e-16)))) atomicAdd(bad, 1ull);
}
// every float significand in an even and an odd binade, and in the lowest and the highest
__global__ void float_roots(u64* bad) {
    const int e[4] = {0, 1, -60, 59};
    for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < (1u << 23); s += gridDim.x * blockDim.x)
        for (int k = 0; k < 4; ++k) one_root(Bits<float>::make(s, e[k]), bad);
    one_root(Bits<float>::make(0, 60), bad);
}
template <typename T> __global__ void roots(u64 n, u64* bad) {
    for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x)
        one_root(operand<T>(mix(3 * i)), bad);
}
// The roots that are hardest to round: x 2^s = m^2 + c with m as above.
template <typename T> __global__ void hard_roots(u64 n, u64* bad, u64* cases) {
    const int p = Bits<T>::sig + 1;
    typedef unsigned __int128 u128;
    for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        const long long c = -(1 + 8 * ((long long)i - (long long)(n / 2)));
        // r^2 = -c modulo 2^64, a bit at a time from -c = 1 modulo 8
        u64 r = 1;
        for (int k = 3; k < 63; ++k)
            if ((r * r + (u64)c) >> k & 1) r += 1ull << (k - 1);
        for (int s = p + 1; s <= p + 2; ++s)
            for (int k = 0; k < 4; ++k) {
                const u64 m = ((k & 1 ? 0 - r : r) + (k & 2 ? 1ull << (s - 1) : 0)) & ((1ull << s) - 1);
                const u128 v = (u128)m * m + (u128)(__int128)c;
                if (m < 1ull << p || m >= 1ull << (p + 1) || (v >> (s + p - 1)) != 1) continue;
                one_root(Bits<T>::make((u64)(v >> s), s & 1), bad);
                if ((v & (((u128)1 << s) - 1)) == 0) atomicAdd(cases, 1ull);
            }
    }
}
template <typename T> __global__ void hertz(u64 n, u64* bad, u64* open) {
    for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        const u64 q = mix(5 * i);
        const T o = operand<T>(q);
        bool ok = true;
        const T got = hertz15_nr(o, ok);
        if (ok)
            expect(got, hertz15(o), bad);
        else if ((q & 7) > 3)  // of the random significands
            atomicAdd(open, 1ull);
    }
}
int main() {
    u64* c;
    if (cudaMallocManaged(&c, 12 * sizeof(u64)) != cudaSuccess) return 2;
    for (int i = 0; i < 12; ++i) c[i] = 0;
    const u64 N = 1ull << 30, M = 1ull << 28;
    divisions<float><<<1184, 256>>>(N, c);
    divisions<double><<<1184, 256>>>(N, c + 1);
    float_roots<<<1184, 256>>>(c + 2);
    roots<float><<<1184, 256>>>(M, c + 2);
    roots<double><<<1184, 256>>>(N, c + 3);
    hertz<float><<<1184, 256>>>(N, c + 4, c + 5);
    hertz<double><<<1184, 256>>>(M, c + 6, c + 7);
    seeds<<<1184, 256>>>(M, c + 1);
    hard_divisions<float><<<1184, 256>>>(1 << 23, c, c + 8);  // every odd divisor
    hard_divisions<double><<<1184, 256>>>(1 << 24, c + 1, c + 9);
    hard_roots<float><<<1184, 256>>>(1 << 16, c + 2, c + 10);
    hard_roots<double><<<1184, 256>>>(1 << 22, c + 3, c + 11);
    if (cudaDeviceSynchronize() != cudaSuccess) return 3;
    for (int i = 0; i < 12; ++i) printf("%llu ", c[i]);
    return 0;
}
"""


def test_branch_free_forms_are_the_operators(tmp_path):
    from mbd_icenav_b200 import build
    src, exe = tmp_path / "fast.cu", tmp_path / "fast"
    src.write_text(PROGRAM)
    subprocess.run([build.nvcc_path(), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false",
                    "--expt-relaxed-constexpr", "-I", f"{ROOT}/include", "-I", build.CSRC, "-o", str(exe), str(src)],
                   check=True, capture_output=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, done
    div32, div64, root32, root64, hertz32, open32, hertz64, open64, *hard = map(int, done.stdout.split())
    assert (div32, div64, root32, root64, hertz32, hertz64) == (0, 0, 0, 0, 0, 0)
    assert min(hard) > 10000  # of each kind, all of them as constructed
    # overlap^1.5 is left open in one case of 2^18: about 2^11 of the 2^29 random significands
    assert 2 ** 9 < open32 < 2 ** 13 and open64 == 0
