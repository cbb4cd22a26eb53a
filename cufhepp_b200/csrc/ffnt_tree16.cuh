// The transform of ffnt_tree.cuh by one warp (16 points per lane): four levels
// with compile-time twiddles, a transpose through shared memory, and five
// levels with per-lane twiddles (the inverse: four, one and four).
//
//   forward: a lane holds z[l + 32 n], n = 0..15, l = tree_low(lane);
//            afterwards v[q] is bin l + 32 tree_pos(q) of the spectrum
//   inverse: the lane holds bins l + 32 k, k = 0..15; afterwards v[q] is
//            coefficient l + 32 tree_neg(q), untwisted and scaled
// so a coefficient stays in its lane and register from an inverse to the next
// forward transform.  tree_low puts l and l + 16, which read the same words
// after the transpose, in neighbouring lanes: a 128-bit shared-memory load
// whose neighbouring lanes agree takes two cycles instead of four (measured).
// 464 FP64 operations per lane, against 568 for twist, 16-point DFT, twiddles,
// 16-point DFT and a cross-lane radix-2 step.
#pragma once
#include <math.h>

#include "ffnt_tree.cuh"

namespace cufhe {

// bit reversal of 4 bits, and the index of the opposite root
__host__ __device__ constexpr int tree_pos(int q)
{
    return ((q & 1) << 3) | ((q & 2) << 1) | ((q & 4) >> 1) | ((q & 8) >> 3);
}
__host__ __device__ constexpr int tree_neg(int q) { return (16 - tree_pos(q)) & 15; }
__host__ __device__ constexpr int tree_low(int lane) { return (lane >> 1) + 16 * (lane & 1); }

// Twiddles of a 16-point tree: level twiddles a, b, c, d (each a square root
// of the one before; the first a square root of the tree's Y^16 = r) and the
// multiples that further blocks of the last two levels need.
struct TreeTw {
    double2 a, b, c, c4, d, d8, d4, d38;
};

__device__ __forceinline__ double2 rot4(double2 w)  // e^{i pi/4} w
{
    constexpr double R2 = 0.70710678118654752440;
    return make_double2(R2 * (w.x - w.y), R2 * (w.x + w.y));
}
__device__ __forceinline__ double2 rot8(double2 w)  // e^{i pi/8} w
{
    return cmul(w, make_double2(0.92387953251128675613, 0.38268343236508977173));
}
__device__ __forceinline__ TreeTw tree_tw(double2 a, double2 b, double2 c, double2 d)
{
    TreeTw t;
    t.a = a;
    t.b = b;
    t.c = c;
    t.c4 = rot4(c);
    t.d = d;
    t.d8 = rot8(d);
    t.d4 = rot4(d);
    t.d38 = cmul(d, make_double2(0.38268343236508977173, 0.92387953251128675613));
    return t;
}
// the first four levels of the forward transform (Y^16 = i)
__device__ __forceinline__ TreeTw tree_tw_twist()
{
    TreeTw t;
    t.a = make_double2(0.70710678118654752440, 0.70710678118654752440);    // pi/4
    t.b = make_double2(0.92387953251128675613, 0.38268343236508977173);    // pi/8
    t.c = make_double2(0.98078528040323044913, 0.19509032201612826785);    // pi/16
    t.c4 = make_double2(0.55557023301960222474, 0.83146961230254523708);   // 5 pi/16
    t.d = make_double2(0.99518472667219688624, 0.09801714032956060199);    // pi/32
    t.d8 = make_double2(0.88192126434835502971, 0.47139673682599764856);   // 5 pi/32
    t.d4 = make_double2(0.63439328416364549822, 0.77301045336273696081);   // 9 pi/32
    t.d38 = make_double2(0.29028467725446236764, 0.95694033573220886494);  // 13 pi/32
    return t;
}

// v[0..15], coefficients of a polynomial modulo Y^16 - r -> its values: v[q]
// at Y = d e^{2 pi i tree_pos(q) / 16}
__device__ __forceinline__ void tree16(double2 (&v)[16], const TreeTw& t)
{
#pragma unroll
    for (int m = 0; m < 8; m++) tree_bf(v[m], v[m + 8], t.a);
#pragma unroll
    for (int m = 0; m < 4; m++) {
        tree_bf(v[m], v[m + 4], t.b);
        tree_bfi(v[m + 8], v[m + 12], t.b);
    }
#pragma unroll
    for (int m = 0; m < 2; m++) {
        tree_bf(v[m], v[m + 2], t.c);
        tree_bfi(v[m + 4], v[m + 6], t.c);
        tree_bf(v[m + 8], v[m + 10], t.c4);
        tree_bfi(v[m + 12], v[m + 14], t.c4);
    }
    tree_bf(v[0], v[1], t.d);
    tree_bfi(v[2], v[3], t.d);
    tree_bf(v[4], v[5], t.d4);
    tree_bfi(v[6], v[7], t.d4);
    tree_bf(v[8], v[9], t.d8);
    tree_bfi(v[10], v[11], t.d8);
    tree_bf(v[12], v[13], t.d38);
    tree_bfi(v[14], v[15], t.d38);
}

// the same for r = 1: v[q] = sum_k x[k] e^{2 pi i k tree_pos(q) / 16}
__device__ __forceinline__ void tree16_one(double2 (&v)[16])
{
    constexpr double R2 = 0.70710678118654752440, C1 = 0.92387953251128675613,
                     S1 = 0.38268343236508977173;
#pragma unroll
    for (int m = 0; m < 8; m++) tree_bf1(v[m], v[m + 8]);
#pragma unroll
    for (int m = 0; m < 4; m++) {
        tree_bf1(v[m], v[m + 4]);
        tree_bf1i(v[m + 8], v[m + 12]);
    }
#pragma unroll
    for (int m = 0; m < 2; m++) {
        tree_bf1(v[m], v[m + 2]);
        tree_bf1i(v[m + 4], v[m + 6]);
        tree_bf(v[m + 8], v[m + 10], make_double2(R2, R2));
        tree_bfi(v[m + 12], v[m + 14], make_double2(R2, R2));
    }
    tree_bf1(v[0], v[1]);
    tree_bf1i(v[2], v[3]);
    tree_bf(v[4], v[5], make_double2(R2, R2));
    tree_bfi(v[6], v[7], make_double2(R2, R2));
    tree_bf(v[8], v[9], make_double2(C1, S1));
    tree_bfi(v[10], v[11], make_double2(C1, S1));
    tree_bf(v[12], v[13], make_double2(S1, C1));
    tree_bfi(v[14], v[15], make_double2(S1, C1));
}

// position of bin f in a spectrum row: lane order of the transforms, with bit
// 3 of the lane XORed into bit 0, so that both the transforms (consecutive
// lanes) and a multiply-accumulate (consecutive bins, every second lane)
// spread over the banks
__device__ __forceinline__ int spec16_lane(int lane) { return lane ^ ((lane >> 3) & 1); }
__device__ __forceinline__ int spec16_ix(int f)
{
    return spec16_lane(2 * (f & 15) + ((f >> 4) & 1)) + (f & ~31);
}

// e^{-i pi k / 32} 2^23: the part of the inverse's untwist that a register
// needs, and the Torus32 scale over the 512 points (a power of two)
static __constant__ double2 c_untw16[16];

inline void untwist16(double2 (&u)[16])
{
    const long double pi = 3.141592653589793238462643383279502884L;
    for (int k = 0; k < 16; k++) {
        const long double a = -pi * k / 32;
        u[k] = make_double2((double)(cosl(a) * 0x1p23L), (double)(sinl(a) * 0x1p23L));
    }
}

// Forward transform (see above).  tile: this warp's 512 double2 of shared
// memory, free on entry and left free.
__device__ __forceinline__ void tree16_forward(double2 (&v)[16], double2* tile,
                                             const double2* __restrict__ ltw, int lane)
{
    tree16(v, tree_tw_twist());
    // v[q]: coefficient l of the sub-polynomial r = tree_pos(q) (modulo
    // Y^32 - psi^{32 (1 + 4 r)}); XOR swizzle: both sides conflict-free
#pragma unroll
    for (int q = 0; q < 16; q++) {
        const int r = tree_pos(q);
        tile[r * 32 + (lane ^ (r & 7))] = v[q];
    }
    __syncwarp();
    const int r = lane >> 1;
    const double2* t = tile + r * 32;
    const double2 w = __ldg(&ltw[0 * 32 + lane]);
#pragma unroll
    for (int m = 0; m < 16; m++) {
        // even lanes take the + half of the fifth level, odd lanes the - half
        // (the sign is in w); coefficients m and m + 16 of sub-polynomial r
        const double2 a = t[(2 * m) ^ (r & 7)], b = t[(2 * m + 1) ^ (r & 7)];
        v[m].x = fma(w.x, b.x, fma(-w.y, b.y, a.x));
        v[m].y = fma(w.x, b.y, fma(w.y, b.x, a.y));
    }
    __syncwarp();
    tree16(v, tree_tw(__ldg(&ltw[1 * 32 + lane]), __ldg(&ltw[2 * 32 + lane]),
                      __ldg(&ltw[3 * 32 + lane]), __ldg(&ltw[4 * 32 + lane])));
}

// Inverse transform (see above), times 2^23 = 2^32 / 512.  In v[k] = bin
// l + 32 k.
__device__ __forceinline__ void tree16_inverse(double2 (&v)[16], double2* tile,
                                             const double2* __restrict__ ltw, int lane)
{
    tree16_one(v);
    // v[q] = sum_k Z[l + 32 k] w16^{-m k}, m = tree_neg(q)
#pragma unroll
    for (int q = 0; q < 16; q++) tile[lane * 16 + (tree_neg(q) ^ (lane & 7))] = v[q];
    __syncwarp();
    const double2 w = __ldg(&ltw[9 * 32 + lane]);
    const int m = lane >> 1;
#pragma unroll
    for (int r = 0; r < 16; r++) {
        const double2 a = tile[(2 * r) * 16 + (m ^ ((2 * r) & 7))];
        const double2 b = tile[(2 * r + 1) * 16 + (m ^ ((2 * r + 1) & 7))];
        v[r].x = fma(w.x, b.x, fma(-w.y, b.y, a.x));
        v[r].y = fma(w.x, b.y, fma(w.y, b.x, a.y));
    }
    __syncwarp();
    tree16(v, tree_tw(__ldg(&ltw[5 * 32 + lane]), __ldg(&ltw[6 * 32 + lane]),
                      __ldg(&ltw[7 * 32 + lane]), __ldg(&ltw[8 * 32 + lane])));
    // untwist psi^{-n} 2^23, n = l + 32 tree_neg(q)
    const double2 u = __ldg(&ltw[10 * 32 + lane]);
#pragma unroll
    for (int q = 0; q < 16; q++) v[q] = cmul(cmul(v[q], u), c_untw16[tree_neg(q)]);
}

}  // namespace cufhe
