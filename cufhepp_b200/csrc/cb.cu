// CMUX and CMUX lookup tables (the private key switching of circuit
// bootstrapping runs on the tensor cores, iks_tc.cu).
//
//   k_cmux     CMUX d0 + ExtProd(C, d1 - d0) with a Fourier-domain TRGSW<lvl1>
//              of L digits of BGBIT bits (the reference's CMUX,
//              src/bootstrap_gpu.cu:704-813, with its lvl1 gadget l = 2,
//              Bgbit = 8, or the circuit-bootstrapping gadget l = 3, Bgbit = 6).
//   k_lut_leaves / k_extract8
//              leaves and outputs of 8-bit -> 8-bit lookup tables evaluated as
//              CMUX trees with the 8 output bits packed in coefficients 0..7.

#include "cufhe_b200.h"
#include "engine.h"
#include "ffnt_tree.cuh"

namespace cufhe {

namespace {


// digit d (0 = most significant) of an offset Torus32 value, BGBIT bits, plus
// half the base
template <int L, int BGBIT>
__device__ __forceinline__ uint32_t gadget_digit(uint32_t t, int d)
{
    return (t >> (32 - (d + 1) * BGBIT)) & ((1u << BGBIT) - 1);
}

template <int L, int BGBIT>
constexpr uint32_t gadget_offset()
{
    uint32_t off = 0;
    for (int i = 1; i <= L; i++) off += (1u << (BGBIT - 1)) << (32 - i * BGBIT);
    return off + (1u << (32 - L * BGBIT - 1));
}

// G CMUXes per CTA on one key, 2L warps: warp r = (input poly j, digit d)
// transforms that digit row of each; thread f (bin) multiplies-accumulates with
// the key, each word read once for all G; the warps share the 2 G inverse
// transforms and add d0.
// A row whose digits are all zero is skipped, transform and products: exactly
// zero is added.  The leaves of a lookup table are constants in eight
// coefficients of one polynomial and one digit, so at the lowest level, half of
// a tree's CMUXes, one row of six is left.
template <int L, int BGBIT, int G>
__global__ void __launch_bounds__(64 * L, 2) k_cmux(CmuxPlan p, const double2* __restrict__ psi,
                                                    const double2* __restrict__ tw512)
{
    constexpr int W = 2 * L;  // warps, and rows per CMUX
    constexpr uint32_t kHalf = 1u << (BGBIT - 1);
    extern __shared__ __align__(16) unsigned char cmux_smem[];
    double2 (*slots)[kSlotStride] = reinterpret_cast<double2 (*)[kSlotStride]>(cmux_smem);  // [G * 2L]
    __shared__ int some[G * W];  // the row has a digit that is not zero
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = blockIdx.x * G;  // the G CMUXes belong to one group
    const int g = c / p.per, m = c % p.per;
    const size_t node = (size_t)g * p.node_stride_g + (size_t)m * p.node_stride_m;
    const double2* key = p.trgsw + (size_t)g * p.trgsw_stride;
    uint32_t* out = p.out + ((size_t)g * p.per + m) * kTrlwe;
    constexpr uint32_t kOffG = gadget_offset<L, BGBIT>();
#pragma unroll 1
    for (int i = 0; i < G; i++) {
        const int d = warp % L;
        const size_t at = (node + (size_t)i * p.node_stride_m) * kTrlwe + (warp / L) * kN;
        const uint32_t *d0 = p.d0 + at, *d1 = p.d1 + at;
        double2 v[16];
        uint32_t any = 0;
#pragma unroll
        for (int n2 = 0; n2 < 16; n2++) {
            const int n = lane + 32 * n2;
            const uint32_t lo = gadget_digit<L, BGBIT>(d1[n] - d0[n] + kOffG, d);
            const uint32_t hi = gadget_digit<L, BGBIT>(d1[n + kHalfN] - d0[n + kHalfN] + kOffG, d);
            any |= (lo ^ kHalf) | (hi ^ kHalf);
            v[n2] = make_double2(small_to_double(lo, kHalf), small_to_double(hi, kHalf));
        }
        const bool nz = __any_sync(0xffffffffu, any != 0);
        double2* row = slots[i * W + warp];
        if (nz) {
#pragma unroll
            for (int n2 = 0; n2 < 16; n2++) v[n2] = cmul(v[n2], __ldg(&psi[lane + 32 * n2]));
            fft512_warp<1>(v, row, tw512, lane);
#pragma unroll
            for (int mm = 0; mm < 16; mm++) row[(lane & 15) + 16 * mm + 256 * (lane >> 4)] = v[mm];
        }
        if (lane == 0) some[i * W + warp] = nz;
    }
    __syncthreads();
    for (int f = threadIdx.x; f < kHalfN; f += 64 * L) {
        double2 o[G][2];
#pragma unroll
        for (int i = 0; i < G; i++) o[i][0] = o[i][1] = make_double2(0.0, 0.0);
#pragma unroll
        for (int r = 0; r < W; r++) {
            bool use = false;
#pragma unroll
            for (int i = 0; i < G; i++) use |= some[i * W + r] != 0;
            if (!use) continue;
            const double2 k0 = __ldg(&key[(r * 2 + 0) * kHalfN + f]);
            const double2 k1 = __ldg(&key[(r * 2 + 1) * kHalfN + f]);
#pragma unroll
            for (int i = 0; i < G; i++) {
                if (some[i * W + r]) {
                    const double2 z = slots[i * W + r][f];
                    o[i][0] = cfma(o[i][0], z, k0);
                    o[i][1] = cfma(o[i][1], z, k1);
                }
            }
        }
        // only this thread reads or writes bin f
#pragma unroll
        for (int i = 0; i < G; i++) {
            slots[i * W + 0][f] = o[i][0];
            slots[i * W + 1][f] = o[i][1];
        }
    }
    __syncthreads();
    for (int t = warp; t < 2 * G; t += W) {
        const int i = t >> 1, oj = t & 1;
        const uint32_t* d0 = p.d0 + (node + (size_t)i * p.node_stride_m) * kTrlwe + oj * kN;
        uint32_t* dst = out + (size_t)i * kTrlwe + oj * kN;
        double2* row = slots[i * W + oj];
        double2 v[16];
#pragma unroll
        for (int n2 = 0; n2 < 16; n2++) v[n2] = row[lane + 32 * n2];
        __syncwarp();
        fft512_warp<-1>(v, row, tw512, lane);
#pragma unroll
        for (int mm = 0; mm < 16; mm++) {
            const int n = (lane & 15) + 16 * mm + 256 * (lane >> 4);
            // untwist conj(psi^n), / 512, x 2^32 => x 2^23; rounded as the reference
            const double2 u = cmulc(v[mm], __ldg(&psi[n]));
            dst[n] = d0[n] + round_mod32(u.x * 0x1p23);
            dst[n + kHalfN] = d0[n + kHalfN] + round_mod32(u.y * 0x1p23);
        }
    }
}

// leaves of q lookup tables: node (q, x) = (0, sum_b (bit b of lut[x] ? mu : -mu) X^b)
__global__ void k_lut_leaves(const uint8_t* __restrict__ luts, int q, uint32_t mu,
                             uint32_t* __restrict__ nodes)
{
    const size_t node = blockIdx.x;  // q * 256 + x
    if (node >= (size_t)q * 256) return;
    const uint8_t v = luts[node];
    uint32_t* t = nodes + node * kTrlwe;
    for (int i = threadIdx.x; i < kTrlwe; i += blockDim.x) {
        uint32_t w = 0;
        if (i >= kN && i < kN + 8) w = ((v >> (i - kN)) & 1) ? mu : 0u - mu;
        t[i] = w;
    }
}

// SampleExtract at coefficients 0..7 of each root TRLWE -> TLWE<lvl1> [q][8][1025]
__global__ void k_extract8(const uint32_t* __restrict__ roots, int q, uint32_t* __restrict__ out)
{
    const int idx = blockIdx.x;  // q * 8 + b
    if (idx >= q * 8) return;
    const int b = idx & 7;
    const uint32_t* acc = roots + (size_t)(idx >> 3) * kTrlwe;
    uint32_t* o = out + (size_t)idx * kTlwe1;
    for (int n = threadIdx.x; n <= kN; n += blockDim.x)
        o[n] = n == kN ? acc[kN + b] : (n <= b ? acc[b - n] : 0u - acc[kN + b - n]);
}

}  // namespace

// The FFT constants of this translation unit (fft64.cuh keeps them per file)
cudaError_t upload_cb_constants(void)
{
    double2 w[16];
    const long double pi = 3.141592653589793238462643383279502884L;
    for (int k = 0; k < 16; k++) {
        const long double a = 2 * pi * k / 32;
        w[k] = make_double2((double)cosl(a), (double)sinl(a));
    }
    return cudaMemcpyToSymbol(c_w32, w, sizeof(w));
}

template <int L, int BGBIT, int G>
static cudaError_t launch_cmux_t(const CmuxPlan& p, const Fp64Tables& t, cudaStream_t st)
{
    constexpr size_t smem = sizeof(double2) * G * 2 * L * kSlotStride;
    static DeviceAttrFlags attr;
    {
        const cudaError_t e = set_smem_attr_once(attr, k_cmux<L, BGBIT, G>, smem);
        if (e != cudaSuccess) return e;
    }
    k_cmux<L, BGBIT, G><<<p.count / G, 64 * L, smem, st>>>(p, t.psi, t.tw512);
    return cudaGetLastError();
}

cudaError_t launch_cmux(int gadget, const CmuxPlan& p, const Fp64Tables& t, cudaStream_t st)
{
    if (p.count <= 0) return cudaSuccess;
    int sms = 148, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // two CMUXes of a group share the key words once there are enough for two
    // CTAs of one on every SM; a lone CMUX finishes sooner with the CTA to itself
    const bool two = p.per % 2 == 0 && p.count % 2 == 0 && p.count > 2 * sms;
    if (gadget == CUFHE_GADGET_CB)
        return two ? launch_cmux_t<3, 6, 2>(p, t, st) : launch_cmux_t<3, 6, 1>(p, t, st);
    return two ? launch_cmux_t<2, 8, 2>(p, t, st) : launch_cmux_t<2, 8, 1>(p, t, st);
}

cudaError_t launch_lut_leaves(const uint8_t* luts, int q, uint32_t mu, uint32_t* nodes,
                              cudaStream_t st)
{
    if (q <= 0) return cudaSuccess;
    k_lut_leaves<<<q * 256, 256, 0, st>>>(luts, q, mu, nodes);
    return cudaGetLastError();
}

cudaError_t launch_extract8(const uint32_t* roots, int q, uint32_t* out, cudaStream_t st)
{
    if (q <= 0) return cudaSuccess;
    k_extract8<<<q * 8, 256, 0, st>>>(roots, q, out);
    return cudaGetLastError();
}

}  // namespace cufhe
