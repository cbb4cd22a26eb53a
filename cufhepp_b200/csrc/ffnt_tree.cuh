// FP64 negacyclic FFNT for N = 1024 by two warps (64 threads, 8 points each).
//
// The folded polynomial z (512 complex coefficients) is evaluated at the
// roots of Y^512 = i, Y = psi^{1 + 4 f}, psi = e^{i pi / 1024}, by halving:
// modulo Y^m - r a polynomial (u, v) splits into u + w v and u - w v with
// w^2 = r, modulo Y^{m/2} - w and Y^{m/2} + w.  The twist of the textbook form
// (src/ntt_small_modulus.cu:207-244) is part of the twiddles, and a butterfly
// is six fused multiply-adds:
//   s = u + w v (four), d = 2 u - s (two).
// Nine levels run as three passes of three levels on 8 registers, with two
// transposes through shared memory in between: the first among all 64
// threads, the second among 8 neighbouring lanes of a warp.
//
//   forward: thread T holds z[T + 64 m], m = 0..7; afterwards v[q] is bin
//            tree_bin(T) + 64 rev8(q) of the spectrum
//   inverse: thread T holds bins tree_bin(T) + 64 k, k = 0..7; afterwards
//            v[q] is coefficient T + 64 neg8(q), untwisted and scaled
// so a coefficient stays in its thread from an inverse to the next forward
// transform.
//
// Why 8 points per thread: 16 points need over 64 registers of data, and a
// warp alone issues an FP64 instruction every 3.3 cycles at best (measured;
// two warps per scheduler reach 0.83 and four 0.96 of the pipe), so the
// transforms want many warps of few registers.
#pragma once
#include "engine.h"
#include "fft64.cuh"

namespace cufhe {

// Conversions by exponent bias: one FP64 add, where the conversion
// instructions run at a quarter of the FP64 rate (14 against 61 per clock and
// SM measured).
// v - off, v and off small non-negative integers
__device__ __forceinline__ double small_to_double(uint32_t v, int off)
{
    return __hiloint2double(0x43300000, (int)v) - (4503599627370496.0 + off);
}
// nearest integer of x modulo 2^32, |x| < 2^51
__device__ __forceinline__ uint32_t round_mod32(double x)
{
    return (uint32_t)__double2loint(x + 6755399441055744.0);
}

// bit reversal of 3 bits, and the index of the opposite root
__host__ __device__ constexpr int rev8(int q) { return ((q & 1) << 2) | (q & 2) | ((q & 4) >> 2); }
__host__ __device__ constexpr int neg8(int q) { return (8 - rev8(q)) & 7; }
// lowest bin of thread T
__host__ __device__ constexpr int tree_bin(int T) { return (T >> 3) + 8 * (T & 7); }
// position of bin f in a spectrum row: conflict-free for the transforms
// (bins of one thread group, stride 8) and for consecutive bins
__host__ __device__ constexpr int spec_ix(int f) { return f ^ ((f >> 3) & 7); }

// barrier of the two warps of a transform
__device__ __forceinline__ void pair_sync(int id)
{
    asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory");
}

// (u, v) -> (u + w v, u - w v)
__device__ __forceinline__ void tree_bf(double2& u, double2& v, double2 w)
{
    double2 s;
    s.x = fma(w.x, v.x, fma(-w.y, v.y, u.x));
    s.y = fma(w.x, v.y, fma(w.y, v.x, u.y));
    v.x = fma(2.0, u.x, -s.x);
    v.y = fma(2.0, u.y, -s.y);
    u = s;
}
// the same with w times i
__device__ __forceinline__ void tree_bfi(double2& u, double2& v, double2 w)
{
    tree_bf(u, v, make_double2(-w.y, w.x));
}
__device__ __forceinline__ void tree_bf1(double2& u, double2& v)
{
    const double2 s = cadd(u, v);
    v = csub(u, v);
    u = s;
}
__device__ __forceinline__ void tree_bf1i(double2& u, double2& v)
{
    const double2 s = make_double2(u.x - v.y, u.y + v.x);
    v = make_double2(u.x + v.y, u.y - v.x);
    u = s;
}

// v[0..7], coefficients of a polynomial modulo Y^8 - r -> its values: v[q] at
// Y = c e^{2 pi i rev8(q) / 8}; a, b, c: level twiddles (r = a^2, a = b^2,
// b = c^2), c4 = e^{i pi / 4} c
__device__ __forceinline__ void tree8(double2 (&v)[8], double2 a, double2 b, double2 c, double2 c4)
{
#pragma unroll
    for (int m = 0; m < 4; m++) tree_bf(v[m], v[m + 4], a);
#pragma unroll
    for (int m = 0; m < 2; m++) {
        tree_bf(v[m], v[m + 2], b);
        tree_bfi(v[m + 4], v[m + 6], b);
    }
    tree_bf(v[0], v[1], c);
    tree_bfi(v[2], v[3], c);
    tree_bf(v[4], v[5], c4);
    tree_bfi(v[6], v[7], c4);
}
__device__ __forceinline__ void tree8(double2 (&v)[8], const double2* __restrict__ tw)
{
    constexpr double R2 = 0.70710678118654752440;
    const double2 c = __ldg(tw + 128);
    tree8(v, __ldg(tw), __ldg(tw + 64), c, make_double2(R2 * (c.x - c.y), R2 * (c.x + c.y)));
}
// the same for r = 1
__device__ __forceinline__ void tree8_one(double2 (&v)[8])
{
    constexpr double R2 = 0.70710678118654752440;
#pragma unroll
    for (int m = 0; m < 4; m++) tree_bf1(v[m], v[m + 4]);
#pragma unroll
    for (int m = 0; m < 2; m++) {
        tree_bf1(v[m], v[m + 2]);
        tree_bf1i(v[m + 4], v[m + 6]);
    }
    tree_bf1(v[0], v[1]);
    tree_bf1i(v[2], v[3]);
    tree_bf(v[4], v[5], make_double2(R2, R2));
    tree_bfi(v[6], v[7], make_double2(R2, R2));
}

// e^{-i pi k / 16} 2^23: the part of the inverse's untwist that a register
// needs, and the Torus32 scale over the 512 points (a power of two)
static __constant__ double2 c_untw[8];

// Forward transform (see above).  tile: the pair's 512 double2 of shared
// memory, free on entry; ltw: the thread's column of the twiddle table
// (engine.h); bar: the pair's barrier.  The caller stores the bins (the tile
// is free again).
__device__ __forceinline__ void tree_forward(double2 (&v)[8], double2* tile,
                                             const double2* __restrict__ ltw, int T, int bar)
{
    tree8(v, make_double2(0.70710678118654752440, 0.70710678118654752440),   // pi/4
          make_double2(0.92387953251128675613, 0.38268343236508977173),      // pi/8
          make_double2(0.98078528040323044913, 0.19509032201612826785),      // pi/16
          make_double2(0.55557023301960222474, 0.83146961230254523708));     // 5 pi/16
    // v[q]: coefficient T of the sub-polynomial r = rev8(q) (modulo Y^64 -
    // psi^{64 (1 + 4 r)})
#pragma unroll
    for (int q = 0; q < 8; q++) tile[rev8(q) * 64 + T] = v[q];
    pair_sync(bar);
    const int w = T & 7;
    double2* const t = tile + (T & ~7) * 8;
#pragma unroll
    for (int m = 0; m < 8; m++) v[m] = t[w + 8 * m];
    __syncwarp();
    tree8(v, ltw);
    // v[q]: coefficient w of sub-polynomial T / 8 + 8 rev8(q) (of 64, modulo Y^8 - ..)
#pragma unroll
    for (int q = 0; q < 8; q++) t[rev8(q) * 8 + (w ^ rev8(q))] = v[q];
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = t[w * 8 + (u ^ w)];
    pair_sync(bar);
    tree8(v, ltw + 3 * 64);
}

__device__ __forceinline__ void tree_store(const double2 (&v)[8], double2* row, int T)
{
    const int f = tree_bin(T);
#pragma unroll
    for (int q = 0; q < 8; q++) row[spec_ix(f) + 64 * rev8(q)] = v[q];
}

// Inverse transform (see above), times 2^23 = 2^32 / 512.  In v[k] = bin
// tree_bin(T) + 64 k; the tile may hold them (it is rewritten after the
// pair's barrier).
__device__ __forceinline__ void tree_inverse(double2 (&v)[8], double2* tile,
                                             const double2* __restrict__ ltw, int T, int bar)
{
    const int w = T & 7;
    double2* const t = tile + (T & ~7) * 8;
    pair_sync(bar);
    tree8_one(v);
    // v[q] = sum_k Z[f + 64 k] w8^{-m k}, m = neg8(q)
#pragma unroll
    for (int q = 0; q < 8; q++) t[w * 8 + (neg8(q) ^ w)] = v[q];
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = t[u * 8 + (w ^ u)];
    __syncwarp();
    tree8(v, ltw + 6 * 64);
#pragma unroll
    for (int q = 0; q < 8; q++) t[w + 8 * neg8(q)] = v[q];
    pair_sync(bar);
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = tile[u * 64 + T];
    tree8(v, ltw + 9 * 64);
    // untwist psi^{-n} 2^23, n = T + 64 neg8(q)
    const double2 u = __ldg(ltw + 12 * 64);
#pragma unroll
    for (int q = 0; q < 8; q++) v[q] = cmul(cmul(v[q], u), c_untw[neg8(q)]);
}

}  // namespace cufhe
