// Identity key switching lvl1 -> lvl0 on the tensor cores (integer,
// bit-exact).
//
// IdentityKeySwitchPreAdd / KeySwitchFromTLWE (include/keyswitch_gpu.cuh:
// 128-256) compute, for x = ca*A + cb*B (+off on b),
//   res[o] = [o == n0] x_b + sum_{i < 1024, j < 7} c(v_ij) . KSK[i][j][.][o]
// with digits v_ij in [-2, 1]: v = -1 adds KSK[i][j][0], v = +1 subtracts it,
// v = -2 adds KSK[i][j][1].  Written over K = (i, j, e) with e in {0, 1} this
// is an exact GEMM with a one-hot operand:
//   A[gate][k] in {-1, 0, +1}  (per gate, from the digits)
//   B[k][(o, c)] = limb_c(KSK[k][o])  (balanced signed bytes, shared by all gates)
//   res[o] = x_b[o == n0] + sum_c (A B_c)[o] << 8c   mod 2^32
// K = 14336, |sum| <= 7168 * 128, so INT32 accumulation is exact.
//
// k_iks_prep combines the inputs and packs each digit into two bits; k_iks_gemm
// expands them to the one-hot bytes in shared memory itself, so the operand A
// never exists in memory (it was 14 KB per key switch, written once and read by
// every column tile), and streams the key tiles once for two unit tiles.
#include "engine.h"
#include "engine.h"
#include "tc_util.cuh"

namespace cufhe {

namespace {

constexpr int kT = CUFHE_LVL10_T;
constexpr int kChunkK = 128;
constexpr int kMGates = 128;                // gates per tile (M)
constexpr int kNCols = 256;                 // 64 outputs x 4 limbs per tile (N)
constexpr int kOutPerTile = kNCols / 4;     // 64
constexpr int kNTiles = (kTlwe0 + kOutPerTile - 1) / kOutPerTile;  // 10
constexpr int kATile = kMGates * kChunkK;   // 16 KB
constexpr int kBTile = kNCols * kChunkK;    // 32 KB
constexpr uint32_t kIdescIks = idesc_i8(kMGates, kNCols);
constexpr uint32_t kTmemColsIks = 256;
// Private key switching: MT unit tiles per CTA share every key chunk (MT
// accumulators of 256 TMEM columns): a stage holds MT A tiles and one B tile.
// MT = 2 halves the key bytes streamed per unit (2.5 GB per function).
template <int MT>
constexpr int iks_stages() { return MT == 1 ? 4 : 3; }
template <int MT>
constexpr size_t iks_smem() { return 1024 + (size_t)iks_stages<MT>() * (MT * kATile + kBTile) + 256; }

// K = (i, j, e) of an input with NIN mask coefficients: NIN * 7 * 2
template <int NIN>
constexpr int iks_chunks() { return NIN * kT * 2 / kChunkK; }  // 112 (lvl1), 224 (lvl2)
constexpr int kChunks = iks_chunks<kN>();

__host__ __device__ constexpr uint32_t iks_offset_tc()
{
    uint32_t off = 0;
    for (int i = 1; i <= kT; i++) off += 2u << (32 - i * CUFHE_LVL10_BASEBIT);
    return off + (1u << (32 - (1 + CUFHE_LVL10_BASEBIT * kT)));
}

// lvl20: the same decomposition of a Torus64 value (include/keyswitch_gpu.cuh
// :128-187 at lvl20param)
__host__ __device__ constexpr uint64_t iks20_offset_tc()
{
    uint64_t off = 0;
    for (int i = 1; i <= (int)CUFHE_LVL20_T; i++) off += 2ull << (64 - i * CUFHE_LVL20_BASEBIT);
    return off + (1ull << (64 - (1 + CUFHE_LVL20_BASEBIT * CUFHE_LVL20_T)));
}

// Place of a pair (i, j) in a run of 16: the digit codes of consecutive pairs are
// consecutive bit pairs of a word, and the expansion takes every fourth.
__host__ __device__ constexpr int pair_at(int place) { return 4 * (place & 3) + (place >> 2); }

// key tiles [nt][kc][32 KB]: row = o_local * 4 + c, K-major, 128B-swizzled.
// Key row k (k < KTOT) has OUTW words; rows k >= KTOT and columns o >= OUTW
// are zero.  PAIRS: k = (pair, e) with the pairs of each run of 16 in the order
// of pair_at.
template <int CH, int NT, int OUTW, int KTOT, bool PAIRS>
__global__ void k_iks_key(const uint32_t* __restrict__ ksk, uint8_t* __restrict__ out)
{
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t total = (size_t)NT * CH * kBTile / 4;
    if (q >= total) return;
    const size_t byte = q * 4;
    const int tile = (int)(byte / kBTile);
    const uint32_t w = (uint32_t)(byte % kBTile);
    const int nt = tile / CH, kc = tile % CH;
    const uint32_t row = (w / 1024) * 8 + (w % 1024) / 128;
    const uint32_t kl = ((((w % 128) / 16) ^ (row & 7)) << 4) + (w % 16);
    const int o = nt * kOutPerTile + (int)(row / 4);
    const int c = (int)(row % 4);
    uint32_t packed = 0;
    for (int e = 0; e < 4; e++) {
        size_t k = (size_t)kc * kChunkK + kl + e;
        if (PAIRS) k = (k & ~(size_t)31) + 2 * pair_at((int)(k & 31) >> 1) + (k & 1);
        const int8_t v = (o < OUTW && k < (size_t)KTOT) ? limb(ksk[k * OUTW + o], c) : (int8_t)0;
        packed |= (uint32_t)(uint8_t)v << (8 * e);
    }
    reinterpret_cast<uint32_t*>(out)[q] = packed;
}

// The seven digits of an input word as two-bit codes (v = code - 2), digit j at
// bits 2 j.  top: the upper 16 bits of the word plus the decomposition offset.
__device__ __forceinline__ uint32_t digit_field(uint32_t top)
{
    const uint32_t r = __brev(top << 16) & 0x3fffu;  // bit pairs in reverse, each swapped
    return ((r & 0x1555u) << 1) | ((r >> 1) & 0x1555u);
}

// The codes of a chunk (64 pairs, 128 bits of the string of fields) of one unit
__device__ __forceinline__ uint4 chunk_codes(const uint16_t* field, int kc)
{
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int bit = 128 * kc + 32 * q, i = bit / 14;
        const uint64_t f = (uint64_t)field[i] | (uint64_t)field[i + 1] << 14 |
                           (uint64_t)field[i + 2] << 28 | (uint64_t)field[i + 3] << 42;
        w[q] = (uint32_t)(f >> (bit - 14 * i));
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

constexpr int kPrepUnits = 8;  // per CTA, one warp each: eight rows' codes of a chunk are 128 bytes

// Rows of the result before the products: zero, with b in the last word.  Not
// done when dst may overlap the inputs (k_iks_init does it afterwards).
__device__ __forceinline__ void init_row(uint32_t* row, uint32_t b, int part, int parts)
{
    for (int o = part; o < kTlwe0; o += parts) row[o] = o == kTlwe0 - 1 ? b : 0u;
}

// digit codes of the units (lanes in mode 0, gates in mode 1):
// codes[u / 128][kc][u % 128]; xb[u] = b part; valid[u]
__global__ void __launch_bounds__(256) k_iks_prep(int mode, Plan plan, int units,
                                                  const uint32_t* __restrict__ in0,
                                                  const uint32_t* __restrict__ in1,
                                                  const uint32_t* __restrict__ in2,
                                                  const uint32_t* __restrict__ lane_out,
                                                  uint4* __restrict__ codes,
                                                  uint32_t* __restrict__ xb, int* __restrict__ valid,
                                                  uint32_t* __restrict__ dst,
                                                  const int32_t* __restrict__ out_idx)
{
    __shared__ uint16_t field[kPrepUnits][kN + 4];  // four past the end are read, not used
    // one warp per unit: its digit fields (coalesced)
    const int here = units - (int)blockIdx.x * kPrepUnits < kPrepUnits
                         ? units - (int)blockIdx.x * kPrepUnits : kPrepUnits;
    const int lane = threadIdx.x & 31, wr = threadIdx.x >> 5;
    if (wr < here) {
        const int u = blockIdx.x * kPrepUnits + wr;
        LanePreadd p = {nullptr, nullptr, 0, 0, 0};
        int ok = 0;
        if (mode == 0) {
            p = plan_lane_preadd(plan, u, in0, in1, in2, kTlwe1);
            ok = 1;
        } else {
            const int l0 = plan_lane0(plan, u);
            if (l0 >= 0) {
                p = gate_combine(plan_op(plan, u), lane_out + (size_t)l0 * kTlwe1,
                                 lane_out + (size_t)(l0 + 1) * kTlwe1);
                ok = 1;
            }
        }
        uint32_t b = 0;
        if (ok) {
            const uint32_t* pb = p.cb ? p.b : p.a;  // cb = 0: not used
#pragma unroll 8
            for (int i = lane; i < kN; i += 32) {
                const uint32_t x = (uint32_t)p.ca * p.a[i] + (uint32_t)p.cb * pb[i];
                field[wr][i] = (uint16_t)digit_field((x + iks_offset_tc()) >> 16);
            }
            b = (uint32_t)p.ca * p.a[kN] + (uint32_t)p.cb * pb[kN] + p.off;
            if (dst) init_row(dst + (out_idx ? (size_t)out_idx[u] : (size_t)u) * kTlwe0, b, lane, 32);
        }
        if (lane == 0) {
            xb[u] = b;
            valid[u] = ok;
        }
    }
    __syncthreads();
    const int r = threadIdx.x % kPrepUnits, u = blockIdx.x * kPrepUnits + r;
    if (r < here)
        for (int kc = threadIdx.x / kPrepUnits; kc < kChunks; kc += 256 / kPrepUnits)
            codes[((size_t)(u / kMGates) * kChunks + kc) * kMGates + u % kMGates] =
                chunk_codes(field[r], kc);
}

// lvl02 gates: the digit codes of gate u from its lane outputs at lvl2
// (uint64 TLWE<lvl2>), combined as binary -> lane0, Mux -> lane0 + lane1 +
// mu2, NMux -> -(lane0 + lane1) - mu2 (src/cufhe_gates_gpu.cu:826-979);
// xb[u] = the combined b rounded to Torus32 (include/keyswitch_gpu.cuh:33-50).
__global__ void __launch_bounds__(256) k_iks20_prep(Plan plan, int units,
                                                    const uint64_t* __restrict__ lane_out,
                                                    uint4* __restrict__ codes,
                                                    uint32_t* __restrict__ xb, int* __restrict__ valid,
                                                    uint32_t* __restrict__ dst)
{
    constexpr int kCh = iks_chunks<CUFHE_LVL2_N>();
    constexpr int kTl2 = CUFHE_TLWE2_WORDS;
    __shared__ uint16_t field[kPrepUnits][CUFHE_LVL2_N + 4];
    const int here = units - (int)blockIdx.x * kPrepUnits < kPrepUnits
                         ? units - (int)blockIdx.x * kPrepUnits : kPrepUnits;
    const int lane = threadIdx.x & 31, wr = threadIdx.x >> 5;
    if (wr < here) {
        const int u = blockIdx.x * kPrepUnits + wr;
        const int l0 = plan_lane0(plan, u);
        uint32_t b = 0;
        if (l0 >= 0) {
            const int op = plan_op(plan, u);
            const uint64_t* A = lane_out + (size_t)l0 * kTl2;
            const bool two = op == kMux || op == kNMux;
            const uint64_t* B = two ? A + kTl2 : A;
            const uint64_t use = two ? 1ull : 0ull;
            const uint64_t neg = op == kNMux ? ~0ull : 0ull;  // x -> -x when set
#pragma unroll 8
            for (int i = lane; i < (int)CUFHE_LVL2_N; i += 32) {
                uint64_t x = A[i] + use * B[i];
                x = (x ^ neg) - neg;
                field[wr][i] = (uint16_t)digit_field((uint32_t)((x + iks20_offset_tc()) >> 48));
            }
            uint64_t x = A[CUFHE_LVL2_N] + use * (B[CUFHE_LVL2_N] + CUFHE_MU64);
            x = (x ^ neg) - neg;
            b = (uint32_t)((x + (1ull << 31)) >> 32);
            if (dst) init_row(dst + plan_out_row(plan, u) * kTlwe0, b, lane, 32);
        }
        if (lane == 0) {
            xb[u] = b;
            valid[u] = l0 >= 0;
        }
    }
    __syncthreads();
    const int r = threadIdx.x % kPrepUnits, u = blockIdx.x * kPrepUnits + r;
    if (r < here)
        for (int kc = threadIdx.x / kPrepUnits; kc < kCh; kc += 256 / kPrepUnits)
            codes[((size_t)(u / kMGates) * kCh + kc) * kMGates + u % kMGates] = chunk_codes(field[r], kc);
}

// init_row of every valid unit, after the inputs have been read
__global__ void __launch_bounds__(256) k_iks_init(int units, const uint32_t* __restrict__ xb,
                                                  const int* __restrict__ valid,
                                                  uint32_t* __restrict__ dst,
                                                  const int32_t* __restrict__ out_idx)
{
    const int u = blockIdx.x;
    if (u < units && valid[u])
        init_row(dst + (out_idx ? (size_t)out_idx[u] : (size_t)u) * kTlwe0, xb[u], threadIdx.x, 256);
}

// ---- private key switching TLWE<lvl2> -> TRLWE<lvl1> as a one-hot GEMM:
// K = (i, j, u) = 2049 x 10 x 15 (i: input word, j: 4-bit digit level, u:
// digit value - 1), A[unit][k] = -1 where digit j of word i of the unit is
// u + 1, B[k][(o, c)] = limb c of key row k, word o (2048 words); each
// digit selects one row, so |sum| <= 20490 x 128 fits INT32 exactly.
constexpr int kPksT = 10;
constexpr int kPksNu = 15;
constexpr int kPksK = (CUFHE_LVL2_N + 1) * kPksT * kPksNu;           // 307,350
constexpr int kPksChunks = (kPksK + kChunkK - 1) / kChunkK;          // 2402
constexpr int kPksWordsOut = 2 * CUFHE_LVL1_N;                       // 2048
constexpr int kPksNTiles = kPksWordsOut / kOutPerTile;               // 32

__global__ void __launch_bounds__(256) k_pks_prep(const uint64_t* __restrict__ tlwe, int units,
                                                  PksMap map, uint8_t* __restrict__ atiles)
{
    const int u = blockIdx.x;
    if (u >= units) return;
    const uint64_t* t = tlwe + (size_t)u * (CUFHE_LVL2_N + 1);
    const uint64_t badd = map.badd[u / map.per];
    constexpr uint64_t kOff = 1ull << (64 - (1 + 4 * kPksT));
    const uint32_t row = (uint32_t)(u % kMGates);
    uint8_t* tb = atiles + (size_t)(u / kMGates) * kPksChunks * kATile;
    for (int q = threadIdx.x; q < kPksChunks * kChunkK / 16; q += blockDim.x) {
        uint32_t wv[4] = {0, 0, 0, 0};
        int ci = -1;
        uint64_t ab = 0;
#pragma unroll
        for (int e = 0; e < 16; e++) {
            const int k = 16 * q + e;
            if (k >= kPksK) break;
            const int c = k / (kPksT * kPksNu), rem = k % (kPksT * kPksNu);
            const int j = rem / kPksNu, uu = rem % kPksNu;
            if (c != ci) {
                ci = c;
                ab = t[c] + (c == CUFHE_LVL2_N ? badd : 0ull) + kOff;
            }
            const uint32_t d = (uint32_t)(ab >> (60 - 4 * j)) & 15u;
            if (d == (uint32_t)uu + 1) wv[e >> 2] |= 0xFFu << (8 * (e & 3));
        }
        const int k0 = 16 * q;
        *reinterpret_cast<uint4*>(tb + (size_t)(k0 / kChunkK) * kATile +
                                  swz_offset(row, (uint32_t)(k0 % kChunkK))) =
            make_uint4(wv[0], wv[1], wv[2], wv[3]);
    }
}

// Output rows of the one-hot GEMM: unit u writes OUTW words at
// dst + (idx ? idx[u] : u % per) * stride_lo + (u / per) * stride_hi.
struct OutMap {
    const int32_t* idx;
    int per;
    size_t stride_lo, stride_hi;
};

// xb (optional) is added to output word OUTW - 1; valid (optional) masks units.
template <int CH, int NT, int OUTW, int MT = 1>
__global__ void __launch_bounds__(128, 1) k_onehot_gemm(const uint8_t* __restrict__ atiles,
                                                     const uint8_t* __restrict__ btiles,
                                                     const uint32_t* __restrict__ xb,
                                                     const int* __restrict__ valid, int units,
                                                     uint32_t* __restrict__ dst, OutMap om,
                                                     int* __restrict__ err)
{
    constexpr int S = iks_stages<MT>();
    constexpr int SB = MT * kATile + kBTile;  // stage bytes: MT A tiles, then the B tile
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    unsigned char* smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)S * SB);
    uint64_t* empty = full + S;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(empty + S);
    __shared__ int s_fail;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int gt = blockIdx.x / NT, nt = blockIdx.x % NT;
    // this CTA's unit tiles: gt * MT + m for m < mc
    const int gtiles = (units + kMGates - 1) / kMGates;
    const int mc = gtiles - gt * MT < MT ? gtiles - gt * MT : MT;
    const uint8_t* ga = atiles + (size_t)gt * MT * CH * kATile;
    const uint8_t* gb = btiles + (size_t)nt * CH * kBTile;
    int pend[S];  // thread 0: 1 + parity of an outstanding fill
#pragma unroll
    for (int s = 0; s < S; s++) pend[s] = 0;
    int last_commit = -1;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(kTmemColsIks * MT));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        s_fail = 0;
        for (int s = 0; s < S; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (tid == 0) {
        auto fill = [&](int s, int kc) {
            unsigned char* st = smem + (size_t)s * SB;
            mbar_expect_tx(&full[s], (uint32_t)(mc * kATile + kBTile));
            for (int m = 0; m < mc; m++)
                bulk_g2s(st + m * kATile, ga + ((size_t)m * CH + kc) * kATile, kATile, &full[s]);
            bulk_g2s(st + MT * kATile, gb + (size_t)kc * kBTile, kBTile, &full[s]);
            pend[s] = 1 + ((kc / S) & 1);
        };
        for (int s = 0; s < S; s++) fill(s, s);
        for (int kc = 0; kc < CH; kc++) {
            const int s = kc % S;
            if (!mbar_wait(&full[s], (kc / S) & 1)) {
                s_fail = 1;
                break;
            }
            pend[s] = 0;
            tc_fence_after();
            const uint32_t a0 = smem_u32(smem + (size_t)s * SB);
            const uint32_t b0 = a0 + MT * kATile;
            for (int m = 0; m < mc; m++)
#pragma unroll
                for (int k = 0; k < kChunkK / 32; k++)
                    tc_mma_i8_ss(tmem + kTmemColsIks * m, desc_kmajor_sw128(a0 + m * kATile + 32 * k),
                                 desc_kmajor_sw128(b0 + 32 * k), kIdescIks, (kc | k) != 0);
            tc_commit(&empty[s]);
            last_commit = kc;
            // refill the stage of chunk kc-1 with chunk kc+S-1 once its MMAs are done
            if (kc >= 1 && kc + S - 1 < CH) {
                const int sp = (kc - 1) % S;
                if (!mbar_wait(&empty[sp], ((kc - 1) / S) & 1)) {
                    s_fail = 1;
                    break;
                }
                fill(sp, kc + S - 1);
            }
        }
        if (!s_fail && !mbar_wait(&empty[(CH - 1) % S], ((CH - 1) / S) & 1))
            s_fail = 1;
        if (s_fail) {
            atomicOr(err, 1);
            for (int s = 0; s < S; s++)
                if (pend[s]) mbar_wait(&full[s], (uint32_t)(pend[s] - 1));
            if (last_commit >= 0)
                mbar_wait(&empty[last_commit % S], (uint32_t)((last_commit / S) & 1));
        }
    }
    __syncthreads();
    tc_fence_after();
#pragma unroll 1
    for (int m = 0; m < mc && !s_fail; m++) {
        // this thread's TMEM lane = unit row of tile gt * MT + m
        const int u = (gt * MT + m) * kMGates + warp * 32 + lane;
        const bool live = u < units && (!valid || valid[u]);
        uint32_t* rowp = dst;
        if (live)
            rowp += (om.idx ? (size_t)om.idx[u] : (size_t)(u % om.per)) * om.stride_lo +
                    (size_t)(u / om.per) * om.stride_hi;
        const uint32_t lane_base = (uint32_t)(32 * warp) << 16;
#pragma unroll 1
        for (int cc = 0; cc < kNCols / 32; cc++) {
            uint32_t v[32];
            tmem_ld32(tmem + lane_base + kTmemColsIks * m + 32 * cc, v);
            tmem_wait_ld();
            if (live) {
#pragma unroll
                for (int oo = 0; oo < 8; oo++) {
                    const int o = nt * kOutPerTile + cc * 8 + oo;
                    uint32_t r = v[4 * oo] + (v[4 * oo + 1] << 8) + (v[4 * oo + 2] << 16) +
                                 (v[4 * oo + 3] << 24);
                    if (xb && o == OUTW - 1) r += xb[u];
                    if (o < OUTW) rowp[o] = r;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(kTmemColsIks * MT));
}

// ---- the identity key switches' GEMM.  The work is the sequence of chunks of
// all (pair of unit tiles, column tile) accumulators; CTA c of G takes the c-th
// G-th of it, so that the last round is as full as the others (4096 units: 160
// accumulators on 148 SMs) and a single key switch is spread over all SMs (8
// chunks each instead of 112 in a row).  An accumulator cut between CTAs is
// summed in dst, mod 2^32 in any order: every CTA adds its part with atomics.
//   warps 0..7  expand the digit codes of one row per thread into the one-hot
//               tiles (two tables of four bytes, selected with PRMT), and
//               afterwards drain the accumulator
//   warp 8      streams the key tiles (bulk copies) and issues the MMAs
// A chunk of a pair of tiles takes about 2,100 cycles: 1,024 are MMA (4096 units
// cannot take less than 63 us of them), and the MMAs' operand reads with the
// tiles' writes keep shared memory busy for 1,250.  Leaving out the expansion,
// its stores, the key copies or three quarters of the MMAs in a copy saves 10,
// 9, 9 and 33 us of 165: no single part is the bound, the hand-over from warp to
// warp is.
// Key switches of 4096 units, prep and GEMM: 264 -> 150 us; of one 76 -> 30 us.
// A 32 KB copy lands about 1.3 us after its issue, hence five key stages; the
// one-hot tiles are made on the SM and two do (three and four: the same time).
constexpr int kKeyStages = 5;
constexpr int kHotStages = 2;
constexpr int kHotBytes = 2 * kATile;
constexpr int kIksThreads = 288;
constexpr int kDrainWords = 32 * 33;  // per warp: 32 rows x 32 words, padded; in the one-hot stages
constexpr size_t kIksSmem = 1024 + (size_t)kHotStages * kHotBytes + (size_t)kKeyStages * kBTile + 256;
static_assert(kIksSmem <= 232448 && 8 * kDrainWords * 4 <= kHotStages * kHotBytes,
              "shared memory of the key-switch GEMM");

// 8 one-hot bytes of four digits (set s of a code word): digit v = -1 -> (1, 0),
// v = +1 -> (-1, 0), v = -2 -> (0, 1), v = 0 -> (0, 0)
__device__ __forceinline__ uint2 expand4(uint32_t w, int s)
{
    const uint32_t sel = ((w >> (2 * s)) & 0x03030303u) * 0x11u + 0x40404040u;
    return make_uint2(__byte_perm(0xFF000100u, 0x00000001u, sel),
                      __byte_perm(0xFF000100u, 0x00000001u, sel >> 16));
}

template <int CH>
__global__ void __launch_bounds__(kIksThreads, 1)
    k_iks_gemm(const uint4* __restrict__ codes, const uint8_t* __restrict__ btiles,
               const int* __restrict__ valid, int units, uint32_t* __restrict__ dst,
               const int32_t* __restrict__ out_idx, int* __restrict__ err)
{
    constexpr int S = kKeyStages, SA = kHotStages;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    unsigned char* hot = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
    unsigned char* keys = hot + (size_t)SA * kHotBytes;
    uint32_t* drain = reinterpret_cast<uint32_t*>(hot);
    uint64_t* full = reinterpret_cast<uint64_t*>(keys + (size_t)S * kBTile);
    uint64_t* empty = full + S;
    uint64_t* hot_full = empty + S;
    uint64_t* hot_empty = hot_full + SA;
    uint64_t* acc_full = hot_empty + SA;
    uint64_t* acc_free = acc_full + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + 1);
    __shared__ int s_fail;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int gtiles = (units + kMGates - 1) / kMGates, groups = (gtiles + 1) / 2;
    const long long total = (long long)groups * kNTiles * CH;
    const int lo = (int)(total * blockIdx.x / gridDim.x);
    const int hi = (int)(total * (blockIdx.x + 1) / gridDim.x);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;"
                     ::"r"(smem_u32(tmem_slot)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        s_fail = 0;
        for (int s = 0; s < S; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < SA; s++) {
            mbar_init(&hot_full[s], 8);
            mbar_init(&hot_empty[s], 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_free, 8);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 8) {
        if (lane == 0) {
            const int n = hi - lo;
            int filled = 0, committed = 0;  // chunks
            bool ok = true;
            auto fill = [&](int it) {
                const int pos = lo + it, tile = pos / CH, kc = pos % CH;
                const int s = it % S;
                mbar_expect_tx(&full[s], (uint32_t)kBTile);
                bulk_g2s(keys + (size_t)s * kBTile,
                         btiles + ((size_t)(tile % kNTiles) * CH + kc) * kBTile, kBTile, &full[s]);
                filled = it + 1;
            };
            for (int it = 0; it < S && it < n; it++) fill(it);
            int seg = 0;
            for (int it = 0; it < n && ok; it++) {
                const int pos = lo + it, tile = pos / CH, kc = pos % CH;
                const int s = it % S;
                const int mc = gtiles - 2 * (tile / kNTiles) < 2 ? 1 : 2;
                const bool first = it == 0 || kc == 0;
                if (first && seg > 0 && !mbar_wait(acc_free, (uint32_t)((seg - 1) & 1))) ok = false;
                if (ok && !mbar_wait(&full[s], (uint32_t)((it / S) & 1))) ok = false;
                if (ok && !mbar_wait(&hot_full[it % SA], (uint32_t)((it / SA) & 1))) ok = false;
                if (!ok) break;
                tc_fence_after();
                const uint32_t a0 = smem_u32(hot + (size_t)(it % SA) * kHotBytes);
                const uint32_t b0 = smem_u32(keys + (size_t)s * kBTile);
                for (int m = 0; m < mc; m++)
#pragma unroll
                    for (int k = 0; k < kChunkK / 32; k++)
                        tc_mma_i8_ss(tmem + kTmemColsIks * m, desc_kmajor_sw128(a0 + m * kATile + 32 * k),
                                     desc_kmajor_sw128(b0 + 32 * k), kIdescIks, !first || k != 0);
                tc_commit(&empty[s]);
                tc_commit(&hot_empty[it % SA]);
                committed = it + 1;
                if (kc == CH - 1 || it == n - 1) {
                    tc_commit(acc_full);
                    seg++;
                }
                // refill the stage of the chunk before once its MMAs are done
                if (it >= 1 && it + S - 1 < n) {
                    if (mbar_wait(&empty[(it - 1) % S], (uint32_t)(((it - 1) / S) & 1)))
                        fill(it + S - 1);
                    else
                        ok = false;
                }
            }
            if (!ok) {
                s_fail = 1;
                atomicOr(err, 1);
                // the copies and MMAs in flight end before the memory they use is freed
                for (int it = committed; it < filled; it++)
                    mbar_wait(&full[it % S], (uint32_t)((it / S) & 1));
                if (committed > 0)
                    mbar_wait(&empty[(committed - 1) % S], (uint32_t)(((committed - 1) / S) & 1));
            }
        }
    } else {
        const int m = warp >> 2, row = 32 * (warp & 3) + lane;
        uint32_t* buf = drain + warp * kDrainWords;
        int seg = 0;
        bool ok = true;
        auto load = [&](int it) {
            const int pos = lo + it, tile = pos / CH, kc = pos % CH, gt = 2 * (tile / kNTiles) + m;
            return gt < gtiles ? __ldg(&codes[((size_t)gt * CH + kc) * kMGates + row])
                               : make_uint4(0, 0, 0, 0);
        };
        uint4 c = load(0);
        for (int it = 0; it < hi - lo && ok; it++) {
            const int pos = lo + it, tile = pos / CH, kc = pos % CH, s = it % SA;
            const int gt = 2 * (tile / kNTiles) + m;
            const uint4 cur = c;
            if (it + 1 < hi - lo) c = load(it + 1);
            if (it >= SA && !mbar_wait(&hot_empty[s], (uint32_t)((it / SA - 1) & 1))) ok = false;
            if (gt < gtiles) {
                unsigned char* a = hot + (size_t)s * kHotBytes + m * kATile;
                const uint32_t w[4] = {cur.x, cur.y, cur.z, cur.w};
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const uint2 x = expand4(w[q >> 1], 2 * (q & 1)), y = expand4(w[q >> 1], 2 * (q & 1) + 1);
                    *reinterpret_cast<uint4*>(a + swz_offset((uint32_t)row, 16u * q)) =
                        make_uint4(x.x, x.y, y.x, y.y);
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the MMAs read these stores
            __syncwarp();
            if (lane == 0) mbar_arrive(&hot_full[s]);
            if (kc == CH - 1 || it == hi - lo - 1) {
                // ---- drain: recombine the limbs, transpose, add to the rows
                // (through the one-hot stages: every MMA that reads them has ended, and
                // the next chunk is expanded by warps that have all left the drain)
                if (!mbar_wait(acc_full, (uint32_t)(seg & 1))) ok = false;
                seg++;
                tc_fence_after();
                const int u = gt * kMGates + row;
                const bool live = ok && gt < gtiles && u < units && valid[u];
                const long long at = live ? (long long)(out_idx ? out_idx[u] : u) * kTlwe0 : -1;
                const int o0 = (tile % kNTiles) * kOutPerTile;
                const unsigned any = __ballot_sync(0xffffffffu, live);
                if (any) {
#pragma unroll 1
                    for (int h = 0; h < 2; h++) {
#pragma unroll
                        for (int cc = 0; cc < 4; cc++) {
                            uint32_t v[32];
                            tmem_ld32(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + kTmemColsIks * m +
                                          128 * h + 32 * cc, v);
                            tmem_wait_ld();
#pragma unroll
                            for (int oo = 0; oo < 8; oo++)
                                buf[lane * 33 + 8 * cc + oo] = v[4 * oo] + (v[4 * oo + 1] << 8) +
                                                               (v[4 * oo + 2] << 16) + (v[4 * oo + 3] << 24);
                        }
                        __syncwarp();
                        const int o = o0 + 32 * h + lane;
#pragma unroll 4
                        for (int r = 0; r < 32; r++) {
                            const long long ra = __shfl_sync(0xffffffffu, at, r);
                            if (ra >= 0 && o < kTlwe0) atomicAdd(dst + ra + o, buf[r * 33 + lane]);
                        }
                        __syncwarp();
                    }
                }
                tc_fence_before();
                asm volatile("bar.sync 1, 256;" ::: "memory");
                if (lane == 0) mbar_arrive(acc_free);
            }
        }
        if (!ok && lane == 0) atomicOr(err, 1);
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

}  // namespace

size_t iks_tc_key_bytes() { return (size_t)kNTiles * kChunks * kBTile; }
size_t iks20_tc_key_bytes() { return (size_t)kNTiles * iks_chunks<CUFHE_LVL2_N>() * kBTile; }

cudaError_t iks_tc_key_build(const uint32_t* ksk_dev, uint8_t* key_tiles, cudaStream_t st)
{
    const size_t units = iks_tc_key_bytes() / 4;
    k_iks_key<kChunks, kNTiles, kTlwe0, kChunks * kChunkK, true>
        <<<(unsigned)((units + 255) / 256), 256, 0, st>>>(ksk_dev, key_tiles);
    return cudaGetLastError();
}

cudaError_t iks20_tc_key_build(const uint32_t* ksk_dev, uint8_t* key_tiles, cudaStream_t st)
{
    const size_t units = iks20_tc_key_bytes() / 4;
    constexpr int kCh2 = iks_chunks<CUFHE_LVL2_N>();
    k_iks_key<kCh2, kNTiles, kTlwe0, kCh2 * kChunkK, true>
        <<<(unsigned)((units + 255) / 256), 256, 0, st>>>(ksk_dev, key_tiles);
    return cudaGetLastError();
}

// bytes_per_row: operand bytes of one unit in one chunk (digit codes 16,
// one-hot tiles of the private key switch 128)
static cudaError_t iks_tc_workspace(IksWorkspace& w, int units, int chunks, int bytes_per_row,
                                    cudaStream_t st)
{
    if ((size_t)units <= w.cap && chunks == w.chunks) return cudaSuccess;
    iks_tc_workspace_free(w);
    const size_t bytes = (size_t)((units + kMGates - 1) / kMGates) * chunks * kMGates * bytes_per_row;
    cudaError_t e;
    if ((e = cudaMalloc(&w.atiles, bytes)) != cudaSuccess) return e;
    // zeroed in stream order: the engine's streams are non-blocking, so a
    // memset on the legacy stream could land after the first prep's stores
    if ((e = cudaMemsetAsync(w.atiles, 0, bytes, st)) != cudaSuccess) return e;
    if ((e = cudaMalloc(&w.xb, (size_t)units * 4)) != cudaSuccess) return e;
    if ((e = cudaMalloc(&w.valid, (size_t)units * 4)) != cudaSuccess) return e;
    w.cap = (size_t)units;
    w.chunks = chunks;
    return cudaSuccess;
}

cudaError_t iks_tc_reserve(IksWorkspace& w, int units, bool lvl2, cudaStream_t st)
{
    return iks_tc_workspace(w, units, lvl2 ? iks_chunks<CUFHE_LVL2_N>() : kChunks, 16, st);
}

void iks_tc_workspace_free(IksWorkspace& w)
{
    cudaFree(w.atiles);
    cudaFree(w.xb);
    cudaFree(w.valid);
    w = IksWorkspace();
}

template <int CH, int NT, int OUTW, int MT = 1>
static cudaError_t gemm_attr()
{
    static DeviceAttrFlags attr;
    {
        const cudaError_t e = set_smem_attr_once(attr, k_onehot_gemm<CH, NT, OUTW, MT>, iks_smem<MT>());
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// the GEMM on as many CTAs as there are SMs, but at least two chunks each
template <int CH>
static cudaError_t launch_iks_gemm(const IksWorkspace& w, const uint8_t* key_tiles, int units,
                                   uint32_t* dst, const int32_t* out_idx, int* err, cudaStream_t st)
{
    static DeviceAttrFlags attr;
    const cudaError_t e = set_smem_attr_once(attr, k_iks_gemm<CH>, kIksSmem);
    if (e != cudaSuccess) return e;
    int sms = 148, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    k_iks_gemm<CH><<<sms, kIksThreads, kIksSmem, st>>>(reinterpret_cast<const uint4*>(w.atiles), key_tiles,
                                                       w.valid, units, dst, out_idx, err);
    return cudaGetLastError();
}

cudaError_t launch_iks_tc(int mode, const Plan& plan, const uint32_t* in0, const uint32_t* in1,
                          const uint32_t* in2, const uint32_t* lane_out, const uint8_t* key_tiles,
                          uint32_t* dst, IksWorkspace& w, int* err, cudaStream_t st,
                          int* launches)
{
    *launches = 0;
    const int units = mode == 0 ? plan.lanes : plan.count;
    if (units <= 0) return cudaSuccess;
    cudaError_t e = iks_tc_workspace(w, units, kChunks, 16, st);
    if (e != cudaSuccess) return e;
    const int32_t* out_idx = mode == 1 ? plan.out_idx : nullptr;
    // the rows of dst are cleared before the products are added: with the
    // digits, unless dst overlaps the inputs (a caller's in-place key switch; the
    // gates' inputs of mode 0 and dst, the engine's lane buffer, never do)
    const char* d0 = reinterpret_cast<const char*>(dst);
    const char* a0 = reinterpret_cast<const char*>(lane_out);
    const bool inplace = mode == 1 && !out_idx && d0 < a0 + (size_t)plan.lanes * kTlwe1 * 4 &&
                         a0 < d0 + (size_t)units * kTlwe0 * 4;
    k_iks_prep<<<(units + kPrepUnits - 1) / kPrepUnits, 256, 0, st>>>(
        mode, plan, units, in0, in1, in2, lane_out, reinterpret_cast<uint4*>(w.atiles), w.xb, w.valid,
        inplace ? nullptr : dst, out_idx);
    if (inplace) k_iks_init<<<units, 256, 0, st>>>(units, w.xb, w.valid, dst, out_idx);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    *launches = inplace ? 3 : 2;
    return launch_iks_gemm<kChunks>(w, key_tiles, units, dst, out_idx, err, st);
}

cudaError_t launch_iks20_tc(const Plan& plan, const uint64_t* lane_out, const uint8_t* key_tiles,
                            uint32_t* dst, IksWorkspace& w, int* err, cudaStream_t st,
                            int* launches)
{
    constexpr int kCh = iks_chunks<CUFHE_LVL2_N>();
    *launches = 0;
    const int units = plan.count;
    if (units <= 0) return cudaSuccess;
    cudaError_t e = iks_tc_workspace(w, units, kCh, 16, st);
    if (e != cudaSuccess) return e;
    const char* d0 = reinterpret_cast<const char*>(dst);
    const char* a0 = reinterpret_cast<const char*>(lane_out);
    const bool inplace = !plan.out_idx && d0 < a0 + (size_t)plan.lanes * CUFHE_TLWE2_WORDS * 8 &&
                         a0 < d0 + (size_t)units * kTlwe0 * 4;
    k_iks20_prep<<<(units + kPrepUnits - 1) / kPrepUnits, 256, 0, st>>>(
        plan, units, lane_out, reinterpret_cast<uint4*>(w.atiles), w.xb, w.valid, inplace ? nullptr : dst);
    if (inplace) k_iks_init<<<units, 256, 0, st>>>(units, w.xb, w.valid, dst, nullptr);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    *launches = inplace ? 3 : 2;
    return launch_iks_gemm<kCh>(w, key_tiles, units, dst, plan.out_idx, err, st);
}

size_t privks_tc_key_bytes() { return (size_t)kPksNTiles * kPksChunks * kBTile; }

cudaError_t privks_tc_key_build(const uint32_t* key_dev, uint8_t* key_tiles, cudaStream_t st)
{
    const size_t units = privks_tc_key_bytes() / 4;
    k_iks_key<kPksChunks, kPksNTiles, kPksWordsOut, kPksK, false>
        <<<(unsigned)((units + 255) / 256), 256, 0, st>>>(key_dev, key_tiles);
    return cudaGetLastError();
}

cudaError_t launch_privks_tc(const uint64_t* tlwe, int units, const uint8_t* key_tiles,
                             const PksMap& map, uint32_t* out, IksWorkspace& w, int* err,
                             cudaStream_t st, int* launches, bool prep)
{
    *launches = 0;
    if (units <= 0) return cudaSuccess;
    cudaError_t e = iks_tc_workspace(w, units, kPksChunks, kChunkK, st);
    constexpr int kMT = 2;  // two unit tiles per CTA share each 2.5 GB key's chunks
    if (e == cudaSuccess) e = gemm_attr<kPksChunks, kPksNTiles, kPksWordsOut, kMT>();
    if (e != cudaSuccess) return e;
    if (prep) k_pks_prep<<<units, 256, 0, st>>>(tlwe, units, map, w.atiles);
    const int gtiles = (units + kMGates - 1) / kMGates;
    const int ggroups = (gtiles + kMT - 1) / kMT;
    const OutMap om = {nullptr, map.per, map.stride_lo, map.stride_hi};
    k_onehot_gemm<kPksChunks, kPksNTiles, kPksWordsOut, kMT>
        <<<ggroups * kPksNTiles, 128, iks_smem<kMT>(), st>>>(w.atiles, key_tiles, nullptr, nullptr,
                                                             units, out, om, err);
    *launches = prep ? 2 : 1;
    return cudaGetLastError();
}

}  // namespace cufhe
