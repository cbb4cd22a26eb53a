// FP64 FFNT blind rotation (the drop-in precision form) with fused
// SampleExtract.
//
// Semantics: __BlindRotate__ / __BlindRotateKeyBundle__ with Accumulate /
// AccumulateKeyBundle (include/gatebootstrapping_gpu.cuh:69-221, :801-884,
// :895-1033, :1335-1380) and __SampleExtractIndex__<P,0>
// (src/bootstrap_gpu.cu:1201-1221):
//   bar = 2N - (b >> 21)  (no rounding), abar_i = (a_i + 2^20) >> 21,
//   acc = X^bar * (0, vec(mu)),
//   non-KB step i : acc += round(IFFNT(sum_r FFNT(dec_r(X^abar acc - acc)) BK_i[r]))
//   KB pair p     : acc  = round(IFFNT(sum_r FFNT(dec_r(acc)) KB_p[r])),
//                   KB = H + bk0 (X^{a0+a1}-1) + bk1 (X^{a0}-1) + bk2 (X^{a1}-1).
// The H term of a KeyBundle step adds the value of the digits; it is added as
// an integer after the rounding, (acc + 2^15) & 0xffff0000, instead of through
// the transforms.
//
// Two forms, by the number of lanes (gates) per SM:
//   k_br_fp64      two lanes per CTA, one warp per polynomial: batches that
//                  fill the GPU
//   k_br_fp64_one  one lane per CTA or per cluster of four CTAs, two warps per
//                  digit row: up to three lanes per SM
// A step is, in both: forward transforms of the digits -> spectra in shared
// memory | multiply-accumulate with the key, bin by bin | inverse transforms,
// rounding.  At lvl1 the rounded values are the exact integers (products below
// 2^44 against 53 bits), so every form gives the same words.
//
// What bounds it: the FP64 pipe takes a warp's fused multiply-add in two
// cycles, but an instruction with three register operands needs three (43
// against 63 per clock and SM measured; two register operands and a constant
// run at full rate).  A KeyBundle step is 154 K FP64 operations per lane, 62 K
// of them the products with three register operands; counted with their
// operands a lane step cannot take less than 3.4 K cycles of an SM.  4789
// lanes: 26.9 -> 23.3 ms (4.5 K cycles); plain key 42.0 -> 38.4 ms.
#include <stdlib.h>

#include <cooperative_groups.h>

#include "engine.h"
#include "ffnt_tree16.cuh"

namespace cufhe {

namespace {

constexpr uint32_t kDecOffset = (128u << 24) + (128u << 16) + (1u << 15);  // offsetgen + round
constexpr int kRootEntries = 514;  // psi^t, t <= 512, padded to an even count

// Shared-memory position of psi^t (t in [0, 512]): the low 3 bits XORed with
// the next 3, so that the strided gathers psi^{(1 + 4 f) a} spread over the
// banks.
__device__ __forceinline__ int root_pos(uint32_t t) { return (int)(t ^ ((t >> 3) & 7u)); }

// psi^t for any t (mod 2N): psi^512 = i
__device__ __forceinline__ double2 root_at(const double2* tab, uint32_t t)
{
    double2 v = tab[root_pos(t & 511u)];
    if (t & 512u) v = make_double2(-v.y, v.x);
    if (t & 1024u) v = make_double2(-v.x, -v.y);
    return v;
}

// i^m v (exact)
__device__ __forceinline__ double2 mul_ipow(double2 v, uint32_t m)
{
    if (m & 1u) v = make_double2(-v.y, v.x);
    if (m & 2u) v = make_double2(-v.x, -v.y);
    return v;
}

// The gadget needs only the upper halves of acc + kDecOffset: digit 0 (most
// significant) is byte 1 of a half minus 128, digit 1 byte 0 minus 128, and
// the value the digits stand for is (half - 0x8080) << 16.  A thread keeps
// coefficient n's half in the lower and n + 512's in the upper 16 bits.
__device__ __forceinline__ uint32_t pack_halves(uint32_t lo, uint32_t hi)
{
    return ((lo + kDecOffset) >> 16) | ((hi + kDecOffset) & 0xffff0000u);
}
__device__ __forceinline__ double2 digits_of(uint32_t h, int d)
{
    const int sh = 8 - 8 * d;
    return make_double2(small_to_double((h >> sh) & 255u, 128),
                        small_to_double((h >> (16 + sh)) & 255u, 128));
}
__device__ __forceinline__ uint32_t recompose_lo(uint32_t h) { return (h << 16) - 0x80800000u; }
__device__ __forceinline__ uint32_t recompose_hi(uint32_t h) { return (h & 0xffff0000u) - 0x80800000u; }

// coefficient i of the test vector X^bar (mu + mu X + ..)
__device__ __forceinline__ uint32_t test_coef(uint32_t bar, uint32_t i, uint32_t mu)
{
    if (bar == 2u * kN) return mu;
    return ((i < (bar & (kN - 1))) ^ (bar >> 10)) ? 0u - mu : mu;
}

// CTAs of a grid that all run at once and share the work of prefetching
constexpr unsigned kPrefetchCtas = 444;


// ---- two lanes per CTA, one warp per polynomial.
// The warp keeps its polynomial's digits in registers from the rounding of a
// step to the transforms of the next (KeyBundle; the plain form rotates the
// accumulator and keeps it in shared memory), so a step has two barriers and
// no warp idles in the inverse transforms.  Three CTAs per SM (168 registers,
// 76 KB): six lanes whose phases drift apart, so that one CTA's key loads run
// under the others' transforms.  4789 lanes KeyBundle: 23.3 ms; two CTAs per
// SM with the registers that leaves 25.2 ms, but 3.18 against 3.24 ms for 592
// lanes, which is one round of them.  Measured and not kept: neighbouring
// threads sharing a bin, one output polynomial each, with the key words of the
// next bin loaded ahead (25.5 ms); eight lanes per SM whose spectra stay in
// tensor memory (24.9 ms for 4736); six lanes in one CTA (31.5 ms); 8 points
// per thread and twice the warps (28.4 ms); the transforms' twiddles in shared
// memory instead of the L1 (25.5 against 24.6 ms).
template <bool KB>
constexpr size_t two_smem_bytes()
{
    return sizeof(double2) * (2 * 4 * kHalfN + (KB ? kRootEntries : 0)) +
           (KB ? 0 : sizeof(uint32_t) * 2 * kTrlwe) + sizeof(uint16_t) * 2 * kN0;
}
static_assert(two_smem_bytes<true>() <= 76800, "three KeyBundle CTAs per SM");
static_assert(two_smem_bytes<false>() <= 113 * 1024, "two plain CTAs per SM");

template <bool KB, int MINB>
__global__ void __launch_bounds__(128, MINB)
    k_br_fp64(const uint32_t* __restrict__ lane_in, int lanes, uint32_t mu,
              const double2* __restrict__ bkf, const double2* __restrict__ psi, int steps,
              uint32_t* __restrict__ acc_out, uint32_t* __restrict__ lane_out)
{
    constexpr int G = 2, NT = 128;
    constexpr int E = KB ? 3 : 1;               // keys per step
    constexpr size_t kTrgswF = 4 * 2 * kHalfN;  // double2 per Fourier TRGSW
    extern __shared__ __align__(16) unsigned char smem[];
    double2* spec = reinterpret_cast<double2*>(smem);  // [G][4][512]
    double2* roots = spec + G * 4 * kHalfN;            // KeyBundle only
    uint32_t* acc = reinterpret_cast<uint32_t*>(roots + (KB ? kRootEntries : 0));  // plain only
    uint16_t* abar = reinterpret_cast<uint16_t*>(acc + (KB ? 0 : G * kTrlwe));
    const double2* const ltw = psi + kTw16At;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int lane_base = blockIdx.x * G;
    const int wg = warp >> 1, wj = warp & 1;
    const int low = tree_low(lane);

    if (KB)
        for (int t = tid; t <= 512; t += NT) roots[root_pos((uint32_t)t)] = psi[t];
    for (int g = 0; g < G; g++) {
        const int l = lane_base + g;
        const bool ok = l < lanes;
        const uint32_t* x = lane_in + (size_t)(ok ? l : 0) * kTlwe0;
        for (int i = tid; i < kN0; i += NT)
            abar[g * kN0 + i] = ok ? (uint16_t)((x[i] + (1u << 20)) >> 21) : 0;
    }
    const int total = KB ? kN0 / 2 : kN0;
    const int nsteps = (steps < 0 || steps > total) ? total : steps;
    // this warp's polynomial; KeyBundle: the accumulators land in the spectra's
    // place after the last step
    uint32_t* const own = (KB ? reinterpret_cast<uint32_t*>(spec) : acc) + (wg * 2 + wj) * kN;
    uint32_t P[16];
    {
        const int l = lane_base + wg;
        const uint32_t bar = l < lanes ? 2u * kN - (lane_in[(size_t)l * kTlwe0 + kN0] >> 21) : 2u * kN;
#pragma unroll
        for (int m = 0; m < 16; m++) {
            const uint32_t n = (uint32_t)(low + 32 * m);
            const uint32_t lo = wj ? test_coef(bar, n, mu) : 0u, hi = wj ? test_coef(bar, n + 512, mu) : 0u;
            if (!KB || nsteps == 0) {
                own[n] = lo;
                own[n + 512] = hi;
            }
            P[m] = pack_halves(lo, hi);
        }
    }
    __syncthreads();

    double2* const slot = spec + (wg * 4 + 2 * wj) * kHalfN;
    const int sl = spec16_lane(lane);

#pragma unroll 1
    for (int p = 0; p < nsteps; p++) {
        if (tid == 0 && p + 2 < nsteps && gridDim.x <= kPrefetchCtas)
            prefetch_part(bkf + (size_t)(p + 2) * E * kTrgswF, E * kTrgswF * sizeof(double2),
                          blockIdx.x, gridDim.x);
        if (!KB) {
            // X^abar acc - acc (include/gatebootstrapping_gpu.cuh:114-138)
            const uint32_t ab = abar[wg * kN0 + p], abm = ab & (kN - 1), abn = ab >> 10;
#pragma unroll
            for (int m = 0; m < 16; m++) {
                const uint32_t n = (uint32_t)(low + 32 * m);
                uint32_t rl = own[(n - ab) & (kN - 1)], rh = own[(n + 512 - ab) & (kN - 1)];
                rl = ((n < abm) ^ abn) ? 0u - rl : rl;
                rh = ((n + 512 < abm) ^ abn) ? 0u - rh : rh;
                P[m] = pack_halves(rl - own[n], rh - own[n + 512]);
            }
        }
        // ---- forward transforms of both digits of this warp's polynomial
#pragma unroll 1
        for (int d = 0; d < 2; d++) {
            double2 v[16];
#pragma unroll
            for (int n = 0; n < 16; n++) v[n] = digits_of(P[n], d);
            tree16_forward(v, slot + d * kHalfN, ltw, lane);
#pragma unroll
            for (int q = 0; q < 16; q++) slot[d * kHalfN + sl + 32 * tree_pos(q)] = v[q];
        }

        // ---- key multiply-accumulate, thread = bins tid + 128 i.  The key
        // words of the two output polynomials lie side by side (one 256-bit
        // load); one key at a time keeps four of them in flight per thread
        // beside both lanes' spectra and sums.  The KeyBundle roots of the
        // bins 128 apart follow from the first's: psi^{512 a} = i^a (exact).
        {
            const double2* bk = bkf + (size_t)p * E * kTrgswF + 2 * tid;
            double2 root[G][3];
            uint32_t rot[G];
            if constexpr (KB) {
                const uint32_t ex = 1u + 4u * (uint32_t)tid;
#pragma unroll
                for (int g = 0; g < G; g++) {
                    const uint32_t a0 = abar[g * kN0 + 2 * p], a1 = abar[g * kN0 + 2 * p + 1];
                    root[g][0] = root_at(roots, ex * (a0 + a1));
                    root[g][1] = root_at(roots, ex * a0);
                    root[g][2] = root_at(roots, ex * a1);
                    rot[g] = (a0 & 3u) | ((a1 & 3u) << 2);
                }
            }
            __syncthreads();
            const int ix0 = spec16_ix(tid);
#pragma unroll 1
            for (int i = 0; i < 4; i++) {
                const int ix = ix0 + 128 * i;
                double2 D[G][4], o[G][2];
#pragma unroll
                for (int g = 0; g < G; g++) {
                    o[g][0] = o[g][1] = make_double2(0.0, 0.0);
#pragma unroll
                    for (int r = 0; r < 4; r++) D[g][r] = spec[(g * 4 + r) * kHalfN + ix];
                }
#pragma unroll
                for (int e = 0; e < E; e++) {
                    double2 k[4][2];
#pragma unroll
                    for (int r = 0; r < 4; r++) key_pair(k[r][0], k[r][1], &bk[(e * 4 + r) * 1024 + i * 256]);
#pragma unroll
                    for (int g = 0; g < G; g++) {
                        double2 s0 = cfma(make_double2(0.0, 0.0), D[g][0], k[0][0]);
                        double2 s1 = cfma(make_double2(0.0, 0.0), D[g][0], k[0][1]);
#pragma unroll
                        for (int r = 1; r < 4; r++) {
                            s0 = cfma(s0, D[g][r], k[r][0]);
                            s1 = cfma(s1, D[g][r], k[r][1]);
                        }
                        if constexpr (KB) {
                            double2 x = root[g][e];
                            x.x -= 1.0;
                            o[g][0] = cfma(o[g][0], x, s0);
                            o[g][1] = cfma(o[g][1], x, s1);
                        } else {
                            o[g][0] = s0;
                            o[g][1] = s1;
                        }
                    }
                }
#pragma unroll
                for (int g = 0; g < G; g++) {
                    // into digit 0's row of either polynomial, which its warp owns
                    spec[(g * 4 + 0) * kHalfN + ix] = o[g][0];
                    spec[(g * 4 + 2) * kHalfN + ix] = o[g][1];
                    if constexpr (KB) {
                        const uint32_t a0 = rot[g], a1 = rot[g] >> 2;
                        root[g][0] = mul_ipow(root[g][0], a0 + a1);
                        root[g][1] = mul_ipow(root[g][1], a0);
                        root[g][2] = mul_ipow(root[g][2], a1);
                    }
                }
            }
        }
        __syncthreads();

        // ---- inverse transform of this warp's polynomial, rounding
        {
            double2 v[16];
#pragma unroll
            for (int k = 0; k < 16; k++) v[k] = slot[sl + 32 * k];
            __syncwarp();
            tree16_inverse(v, slot, ltw, lane);
            if constexpr (KB) {
                const bool last = p + 1 == nsteps;
                if (last) __syncthreads();  // the accumulators overwrite the spectra
#pragma unroll
                for (int q = 0; q < 16; q++) {
                    const int m = tree_neg(q);
                    const uint32_t lo = round_mod32(v[q].x) + recompose_lo(P[m]);
                    const uint32_t hi = round_mod32(v[q].y) + recompose_hi(P[m]);
                    P[m] = pack_halves(lo, hi);
                    if (last) {
                        own[low + 32 * m] = lo;
                        own[low + 32 * m + 512] = hi;
                    }
                }
            } else {
#pragma unroll
                for (int q = 0; q < 16; q++) {
                    const int n = low + 32 * tree_neg(q);
                    own[n] += round_mod32(v[q].x);
                    own[n + 512] += round_mod32(v[q].y);
                }
                __syncwarp();  // the next step's rotation reads other lanes' coefficients
            }
        }
    }
    __syncthreads();

    // ---- epilogue: accumulator and/or SampleExtract (index 0)
    for (int g = 0; g < G; g++) {
        const int l = lane_base + g;
        if (l >= lanes) break;
        const uint32_t* a = (KB ? reinterpret_cast<uint32_t*>(spec) : acc) + g * kTrlwe;
        if (acc_out)
            for (int i = tid; i < kTrlwe; i += NT) acc_out[(size_t)l * kTrlwe + i] = a[i];
        if (lane_out) {
            uint32_t* o = lane_out + (size_t)l * kTlwe1;
            for (int i = tid; i <= kN; i += NT)
                o[i] = i == kN ? a[kN] : (i == 0 ? a[0] : 0u - a[kN - i]);
        }
    }
}

template <bool KB, int MINB>
cudaError_t launch_two(const uint32_t* lane_in, int lanes, uint32_t mu, const double2* bkf,
                       const Fp64Tables& t, int steps, uint32_t* acc_out, uint32_t* lane_out,
                       cudaStream_t st)
{
    constexpr size_t smem = two_smem_bytes<KB>();
    static DeviceAttrFlags attr;
    {
        const cudaError_t e = set_smem_attr_once(attr, k_br_fp64<KB, MINB>, smem);
        if (e != cudaSuccess) return e;
    }
    k_br_fp64<KB, MINB><<<(lanes + 1) / 2, 128, smem, st>>>(lane_in, lanes, mu, bkf, t.psi, steps,
                                                          acc_out, lane_out);
    return cudaGetLastError();
}

// BK polynomial -> Fourier domain: read as signed int32, scale 2^-32, fold,
// twist, forward FFT (src/bootstrap_gpu.cu:59-112).  One warp per polynomial.
__global__ void __launch_bounds__(128) k_bk_to_fft(const uint32_t* __restrict__ bk, int npolys,
                                                   const double2* __restrict__ psi,
                                                   const double2* __restrict__ tw512,
                                                   double2* __restrict__ out, int pairs)
{
    __shared__ __align__(16) double2 tiles[4][kSlotStride];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int poly = blockIdx.x * 4 + warp;
    if (poly >= npolys) return;
    const uint32_t* src = bk + (size_t)poly * kN;
    double2 v[16];
#pragma unroll
    for (int n2 = 0; n2 < 16; n2++) {
        const int n = lane + 32 * n2;
        const double2 z = make_double2((double)(int32_t)src[n] * 0x1p-32,
                                       (double)(int32_t)src[n + kHalfN] * 0x1p-32);
        v[n2] = cmul(z, __ldg(&psi[n]));
    }
    fft512_warp<1>(v, tiles[warp], tw512, lane);
    // pairs: bins of the two polynomials of a row interleaved
    double2* dst = pairs ? out + (size_t)(poly >> 1) * 2 * kHalfN + (poly & 1)
                         : out + (size_t)poly * kHalfN;
    const int step = pairs ? 2 : 1;
#pragma unroll
    for (int m = 0; m < 16; m++) dst[step * ((lane & 15) + 16 * m + 256 * (lane >> 4))] = v[m];
}

// ---- one lane per CTA (R = 1), or per cluster of R = 4 CTAs on 4 SMs; two warps per
// digit row (8 points per thread), since a warp alone cannot keep the FP64 pipe
// busy.  In a cluster every CTA runs the lane's transforms (redundantly, on its
// own copy of the accumulator) but multiplies only its 512 / R frequency bins
// with the key, and the inverse transforms gather the parts from the peers'
// shared memory (distributed shared memory).  The key rows of a step do not
// depend on the step before, so each thread fetches those of its first items
// into registers before the forward transforms and those of a further one while
// it multiplies, and the rows of the step after next are brought into the L2:
// a gate's key switching key and this key together do not stay there (32 lanes
// between key switches: one CTA per lane without the prefetch 2.30 ms, with it
// 1.25, in clusters 1.05; nothing else between the rotations 1.6 ms).  The products of a cluster alternate
// between two buffers, so that one cluster barrier per step is enough: a buffer
// is rewritten two steps later, after the next step's barrier, which every
// peer's gather precedes.
// One lane: 1.22 -> 1.06 ms (R = 4); 148 lanes 1.66 -> 1.15 (R = 1); 296 lanes,
// two CTAs per SM, 2.18 -> 1.95; 444 lanes, three, 2.95 -> 2.75.  Plain key:
// 148 lanes 2.71 -> 1.71, 296 lanes 3.44 -> 2.88, 444 lanes 4.56 -> 4.18 ms.
// Measured and not kept: clusters of two up to 74 lanes (no gain over one CTA;
// plain key 2.06 against 1.67 ms), neighbouring threads sharing a bin with one
// output each (148 lanes 1.21 ms), the twiddles in shared memory (1.17-1.21 ms).
constexpr int kCluMaxLanes = 32;
constexpr size_t kOneSmem = 120 * 1024;  // > half an SM: one CTA per SM
template <int R>
constexpr size_t one_smem_bytes()
{
    return sizeof(double2) * ((R > 1 ? 8 : 4) * kHalfN + kRootEntries) + sizeof(uint32_t) * kTrlwe +
           sizeof(uint16_t) * kN0;
}
static_assert(one_smem_bytes<4>() <= kOneSmem && one_smem_bytes<1>() <= 75 * 1024, "CTA layouts");

template <bool KB, int R, int MINB>
__global__ void __launch_bounds__(256, MINB)
    k_br_fp64_one(const uint32_t* __restrict__ lane_in, int lanes, uint32_t mu,
                  const double2* __restrict__ bkf, const double2* __restrict__ psi, int steps,
                  uint32_t* __restrict__ acc_out, uint32_t* __restrict__ lane_out)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char smem[];
    double2* spec = reinterpret_cast<double2*>(smem);  // [4][512] digit spectra
    // [2][2][512] products, by step parity; one CTA: in the place of rows 0 and 2
    double2* prod = R > 1 ? spec + 4 * kHalfN : spec;
    double2* roots = R > 1 ? prod + 4 * kHalfN : spec + 4 * kHalfN;
    uint32_t* acc = reinterpret_cast<uint32_t*>(roots + kRootEntries);
    uint16_t* abar = reinterpret_cast<uint16_t*>(acc + kTrlwe);

    const int tid = threadIdx.x;
    const int pair = tid >> 6, T = tid & 63, bar_id = 1 + pair;
    const int rank = R > 1 ? (int)cluster.block_rank() : 0;
    const double2* const ltw = psi + 2 * kN + T;
    const int l = blockIdx.x / R;
    const bool ok = l < lanes;

    for (int t = tid; t <= 512; t += 256) roots[root_pos((uint32_t)t)] = psi[t];
    {
        const uint32_t* x = lane_in + (size_t)(ok ? l : 0) * kTlwe0;
        for (int i = tid; i < kN0; i += 256) abar[i] = ok ? (uint16_t)((x[i] + (1u << 20)) >> 21) : 0;
        const uint32_t bar = ok ? 2u * kN - (x[kN0] >> 21) : 2u * kN;
        for (int i = tid; i < kN; i += 256) {
            acc[i] = 0;
            acc[kN + i] = test_coef(bar, (uint32_t)i, mu);
        }
    }
    const double2* peer[R];
#pragma unroll
    for (int k = 0; k < R; k++) peer[k] = R > 1 ? cluster.map_shared_rank(prod, k) : prod;
    if (R > 1) cluster.sync(); else __syncthreads();

    const int total = KB ? kN0 / 2 : kN0;
    const int nsteps = (steps < 0 || steps > total) ? total : steps;
    constexpr int E = KB ? 3 : 1;                    // keys per step
    constexpr int NB = R == 1 ? 2 : 1;               // bins per thread
    constexpr size_t kTrgswF = 4 * 2 * kHalfN;
    const int f0 = rank * (512 / R) + tid;
    const bool mac = R < 4 || tid < 512 / R;

#pragma unroll 1
    for (int p = 0; p < nsteps; p++) {
        if (tid == 0 && p + 2 < nsteps)
            prefetch_part(bkf + (size_t)(p + 2) * E * kTrgswF, E * kTrgswF * sizeof(double2), blockIdx.x,
                          gridDim.x);
        const double2* bk = bkf + (size_t)p * E * kTrgswF + 2 * f0;
        constexpr int NPRE = MINB > 2 ? 0 : MINB > 1 ? 1 : E;  // keys fetched ahead
        double2 b[E][4][2];
        if (mac)
#pragma unroll
            for (int e = 0; e < NPRE; e++)
#pragma unroll
                for (int r = 0; r < 4; r++) key_words(b[e][r], &bk[(e * 4 + r) * 1024]);
        // ---- phase 1 (every rank): decompose + fold + forward transform, pair r
        {
            const int d = pair & 1;
            const uint32_t* a = acc + (pair >> 1) * kN;
            double2 v[8];
            const uint32_t ab = KB ? 0u : abar[p];
            const uint32_t abm = ab & (kN - 1), abn = ab >> 10;
#pragma unroll
            for (int m = 0; m < 8; m++) {
                const uint32_t n = (uint32_t)(T + 64 * m);
                uint32_t lo = a[n], hi = a[n + 512];
                if constexpr (!KB) {
                    uint32_t rl = a[(n - ab) & (kN - 1)], rh = a[(n + 512 - ab) & (kN - 1)];
                    rl = ((n < abm) ^ abn) ? 0u - rl : rl;
                    rh = ((n + 512 < abm) ^ abn) ? 0u - rh : rh;
                    lo = rl - lo;
                    hi = rh - hi;
                }
                v[m] = digits_of(pack_halves(lo, hi), d);
            }
            tree_forward(v, spec + pair * kHalfN, ltw, T, bar_id);
            tree_store(v, spec + pair * kHalfN, T);
        }
        __syncthreads();

        // ---- phase 2: key multiply-accumulate of this rank's bins
        if (mac)
#pragma unroll
            for (int u = 0; u < NB; u++) {
                const int f = f0 + 256 * u;
                const int ix = spec_ix(f);
                double2 D[4], o[2];
                o[0] = o[1] = make_double2(0.0, 0.0);
#pragma unroll
                for (int r = 0; r < 4; r++) D[r] = spec[r * kHalfN + ix];
                const uint32_t ef = 1u + 4u * (uint32_t)f;
                const uint32_t a0 = abar[KB ? 2 * p : 0], a1 = abar[KB ? 2 * p + 1 : 0];
                const uint32_t am[3] = {a0 + a1, a0, a1};
#pragma unroll
                for (int e = 0; e < E; e++) {
                    if (u == 0 && e >= NPRE)
#pragma unroll
                        for (int r = 0; r < 4; r++) key_words(b[e][r], &bk[(e * 4 + r) * 1024]);
                    double2 s[2];
#pragma unroll
                    for (int r = 0; r < 4; r++)
#pragma unroll
                        for (int j = 0; j < 2; j++)
                            s[j] = cfma(r ? s[j] : make_double2(0.0, 0.0), D[r], b[e][r][j]);
                    if (u + 1 < NB)
#pragma unroll
                        for (int r = 0; r < 4; r++) key_words(b[e][r], &bk[(e * 4 + r) * 1024 + 512]);
                    if constexpr (KB) {
                        // sum of (X^a - 1) bk terms; H is added as an integer (phase 3)
                        double2 x = root_at(roots, ef * am[e]);
                        x.x -= 1.0;
                        o[0] = cfma(o[0], x, s[0]);
                        o[1] = cfma(o[1], x, s[1]);
                    } else {
                        o[0] = s[0];
                        o[1] = s[1];
                    }
                }
                double2* const out = R > 1 ? prod + (p & 1) * 2 * kHalfN : spec;
                out[ix] = o[0];
                out[(R > 1 ? 1 : 2) * kHalfN + ix] = o[1];
            }
        if (R > 1) cluster.sync(); else __syncthreads();  // every rank's products are written

        // ---- phase 3 (every rank): gather, inverse transform, round, pair j
        if (pair < 2) {
            const int f = spec_ix(tree_bin(T));
            double2 v[8];
#pragma unroll
            for (int k = 0; k < 8; k++) 
                v[k] = R > 1 ? peer[k * R / 8][((p & 1) * 2 + pair) * kHalfN + f + 64 * k]
                             : spec[2 * pair * kHalfN + f + 64 * k];
            tree_inverse(v, spec + 2 * pair * kHalfN, ltw, T, bar_id);
            uint32_t* a = acc + pair * kN;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const int n = T + 64 * neg8(q);
                const uint32_t lo = round_mod32(v[q].x), hi = round_mod32(v[q].y);
                a[n] = lo + (KB ? (a[n] + (1u << 15)) & 0xffff0000u : a[n]);
                a[n + 512] = hi + (KB ? (a[n + 512] + (1u << 15)) & 0xffff0000u : a[n + 512]);
            }
        }
        __syncthreads();
    }
    if (R > 1) cluster.sync();  // no CTA leaves while a peer still gathers from it

    if (ok && rank == 0) {
        if (acc_out)
            for (int i = tid; i < kTrlwe; i += 256) acc_out[(size_t)l * kTrlwe + i] = acc[i];
        if (lane_out) {
            uint32_t* o = lane_out + (size_t)l * kTlwe1;
            for (int i = tid; i <= kN; i += 256)
                o[i] = i == kN ? acc[kN] : (i == 0 ? acc[0] : 0u - acc[kN - i]);
        }
    }
}

template <bool KB, int R, int MINB>
cudaError_t launch_one(const uint32_t* lane_in, int lanes, uint32_t mu, const double2* bkf,
                       const Fp64Tables& t, int steps, uint32_t* acc_out, uint32_t* lane_out,
                       cudaStream_t st)
{
    static DeviceAttrFlags attr;
    constexpr size_t smem = MINB == 1 ? kOneSmem : one_smem_bytes<R>();
    {
        const cudaError_t e = set_smem_attr_once(attr, k_br_fp64_one<KB, R, MINB>, smem);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(lanes * R);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = R;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = R > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k_br_fp64_one<KB, R, MINB>, lane_in, lanes, mu, bkf, t.psi, steps,
                              acc_out, lane_out);
}
}  // namespace

// Lanes per CTA: 1 or 2 (4, an earlier form, is taken as 2).
// CUFHE_BR_LANES_PER_CTA overrides the default for tuning.
static int br_lanes_per_cta()
{
    static int g = 0;
    if (!g) {
        const char* e = getenv("CUFHE_BR_LANES_PER_CTA");
        g = (e && atoi(e) == 4) ? 4 : (e && atoi(e) == 2) ? 2 : (e && atoi(e) == 1) ? 1 : 2;
    }
    return g;
}

namespace {
struct BrTuning {
    int n = 0;
    int bound[32];
    int g[32];
};
BrTuning g_br_tuning[64];
}  // namespace

void br_fp64_set_tuning(int dev, int n, const int* bound, const int* g)
{
    BrTuning& t = g_br_tuning[dev & 63];
    t.n = n < 0 ? 0 : (n > 32 ? 32 : n);
    for (int i = 0; i < t.n; i++) {
        t.bound[i] = bound[i];
        t.g[i] = g[i];
    }
}

int br_fp64_get_tuning(int dev, int* bound, int* g, int cap)
{
    const BrTuning& t = g_br_tuning[dev & 63];
    for (int i = 0; i < t.n && i < cap; i++) {
        bound[i] = t.bound[i];
        g[i] = t.g[i];
    }
    return t.n;
}

cudaError_t launch_br_fp64(bool kb, const uint32_t* lane_in, int lanes, uint32_t mu,
                           const double2* bkf, const Fp64Tables& t, int steps, uint32_t* acc_out,
                           uint32_t* lane_out, cudaStream_t st)
{
    if (lanes <= 0) return cudaSuccess;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    int g;
    const BrTuning& tun = g_br_tuning[dev & 63];
    if (getenv("CUFHE_BR_LANES_PER_CTA")) {
        g = br_lanes_per_cta();
    } else if (tun.n > 0) {
        int i = 0;
        while (i + 1 < tun.n && lanes > tun.bound[i]) i++;
        g = tun.g[i];
    } else {
        // untuned: one lane per CTA while the batch fits one round of three
        // per SM (444 lanes: 2.75 ms against 3.2 ms with two lanes per CTA),
        // two lanes per CTA beyond (592 lanes: 3.18 against 3.9 ms)
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        g = lanes <= 3 * sms ? 1 : 2;
    }
    return launch_br_fp64_g(g, kb, lane_in, lanes, mu, bkf, t, steps, acc_out, lane_out, st);
}

cudaError_t launch_br_fp64_g(int g, bool kb, const uint32_t* lane_in, int lanes, uint32_t mu,
                             const double2* bkf, const Fp64Tables& t, int steps,
                             uint32_t* acc_out, uint32_t* lane_out, cudaStream_t st)
{
    if (lanes <= 0) return cudaSuccess;
    int sms = 148, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
#define BR_ARGS lane_in, lanes, mu, bkf, t, steps, acc_out, lane_out, st
    if (g != 1) {
        // plain: shared memory for two CTAs per SM.  KeyBundle: two when that
        // is one round (4 lanes per SM), three beyond.
        if (!kb) return launch_two<false, 2>(BR_ARGS);
        return lanes <= 4 * sms ? launch_two<true, 2>(BR_ARGS) : launch_two<true, 3>(BR_ARGS);
    }
    // KeyBundle: one lane per cluster of four SMs while the clusters fit at once
    // (32 lanes: 1.05 against 1.14 ms; 37 clusters no longer fit: 2.2 ms).  The
    // plain key has a third of the key rows per step and gains nothing (one lane
    // 2.03 against 1.64 ms).  CUFHE_BR_CLUSTER=0 keeps one CTA per lane; a device
    // that cannot place the clusters runs one CTA per lane instead.
    const char* e = getenv("CUFHE_BR_CLUSTER");
    if (kb && !(e && atoi(e) == 0) && lanes <= kCluMaxLanes && 4 * lanes <= sms) {
        const cudaError_t r = launch_one<true, 4, 1>(BR_ARGS);
        if (r == cudaSuccess) return r;
        cudaGetLastError();
    }
    if (lanes <= sms) return kb ? launch_one<true, 1, 1>(BR_ARGS) : launch_one<false, 1, 1>(BR_ARGS);
    if (lanes <= 2 * sms) return kb ? launch_one<true, 1, 2>(BR_ARGS) : launch_one<false, 1, 2>(BR_ARGS);
    return kb ? launch_one<true, 1, 3>(BR_ARGS) : launch_one<false, 1, 3>(BR_ARGS);
#undef BR_ARGS
}

cudaError_t launch_bk_to_fft(const uint32_t* bk, int npolys, const Fp64Tables& t, double2* out,
                             cudaStream_t st, bool pairs)
{
    k_bk_to_fft<<<(npolys + 3) / 4, 128, 0, st>>>(bk, npolys, t.psi, t.tw512, out, pairs ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t upload_fft_constants(void)
{
    double2 w[16], un[8];
    const long double pi = 3.141592653589793238462643383279502884L;
    for (int k = 0; k < 16; k++) {
        const long double a = 2 * pi * k / 32;
        w[k] = make_double2((double)cosl(a), (double)sinl(a));
    }
    for (int k = 0; k < 8; k++) {
        const long double b = -pi * k / 16;  // psi^{-64 k}, times 2^23
        un[k] = make_double2((double)(cosl(b) * 0x1p23L), (double)(sinl(b) * 0x1p23L));
    }
    double2 un16[16];
    untwist16(un16);
    cudaError_t e = cudaMemcpyToSymbol(c_w32, w, sizeof(w));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_untw, un, sizeof(un));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_untw16, un16, sizeof(un16));
    return e;
}

}  // namespace cufhe
