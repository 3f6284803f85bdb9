// Genomic relationship matrix from PLINK BED on sm_103a tensor cores.
//
// Replaces GrmBuilder::compute(const PlinkReader&) for VanRaden (algorithm 1),
// reference src/core/grm_builder.cpp:63-405.
//
// The reference forms Z (n x m, FP64) with Z_ij = x_ij - mu_j for observed
// calls and 0 for missing ones, then G = Z Z^T / sum_2pq (FP64 GEMM, :351).
// Here the same quantity is computed in integer arithmetic on the f16 tensor
// cores and rounded once at the end.  XX and L are exact; Q uses mu_j^2
// rounded to a multiple of 2^-45, so |G - G_exact| <= n_valid 2^-46 / sum_2pq
// (plus the final rounding) -- below the FP64 GEMM rounding of the reference
// for realistic SNP counts:
//
//   (Z Z^T)_ik = XX_ik - L_ik 2^-29 + Q_ik 2^-45, with
//   XX_ik = sum_j x_ij x_kj                               (integer cross-products)
//   L_ik  = sum_j (x_ij o_kj + o_ij x_kj) a_j,  a_j = mu_j 2^29 (exact, < 2^30)
//   Q_ik  = sum_j o_ij o_kj e_j,                e_j = round(a_j^2 / 2^13) (< 2^47)
//
// o_ij = 1 for an observed call.  mu_j is a float >= 2^-6 (MAF >= 0.01), so
// a_j is an exact integer.  a_j is split into balanced base-2048 digits, e_j into
// balanced base-4096 digits (|digit| <= 2048, exactly representable in f16), so
// every product the tensor core forms is an exact small integer.  The SNPs are cut
// into chunks over which no partial sum can reach 2^24 (sum of 4 |digit| of a_j,
// of |digit| of e_j: up to 8192 SNPs), so the FP32 accumulators are exact; at the
// end of a chunk they are added to exact totals in shared memory.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>
#include <cuda_fp16.h>
#include "handle.h"

namespace cbx {
namespace grm {

constexpr int TILE_M = 128;   // samples per tile row block (= TMEM lanes)
constexpr int TILE_N = 32;    // samples per tile column block
constexpr int KSTEP = 64;     // SNPs per operand stage
constexpr int NSTAGE = 3;     // operand stages (A in TMEM, B in shared memory)
constexpr int NRAW = 4;       // raw 2-bit stages
constexpr int NVAR = 11;      // B-side operand variants: X, O a (3), X a (3), O e (4)
constexpr int NDIG = 7;       // digits per SNP (3 for a_j, 4 for e_j)
constexpr int MAX_CHUNK = 128;         // steps per chunk (8192 SNPs)
constexpr int64_t SUM_LIMIT = 1 << 22; // sum of |digit| of a_j per chunk
constexpr int64_t Q_EXACT = 1 << 16;   // SNPs up to which a sum of e_j fits an int64
// 24 warps: 0 MMA, 1 loader, 2-3 idle, 4-11 A producers, 12-19 B producers, 20-23
// epilogue.  Four A and four B warps make a stage, the others the next one: a job is a
// chain of waits, loads, stores and a fence, which takes longer than a stage's products.
constexpr int THREADS = 768;
constexpr int NPROD = 8;      // producer warps of a stage

constexpr int B_VAR_BYTES = TILE_N * KSTEP * 2;                    // 4096
constexpr int STAGE_BYTES = NVAR * B_VAR_BYTES;                    // 45056
constexpr int RAW_A = TILE_M * KSTEP / 4;                          // 2048
constexpr int RAW_B = TILE_N * KSTEP / 4;                          // 512
constexpr int RAW_D = NDIG * KSTEP * 2;                            // 896
constexpr int RAW_BYTES = RAW_A + RAW_B + RAW_D;                   // 3456
constexpr int OFF_STAGE = 0;
constexpr int OFF_RAW = OFF_STAGE + NSTAGE * STAGE_BYTES;          // 135168
constexpr int OFF_XX = OFF_RAW + NRAW * RAW_BYTES;                 // 148992
constexpr int OFF_L = OFF_XX + TILE_N * TILE_M * 4;                // 165376
constexpr int OFF_Q = OFF_L + TILE_N * TILE_M * 8;                 // 198144
constexpr int OFF_BAR = OFF_Q + TILE_N * TILE_M * 8;               // 230912
constexpr int SMEM_BYTES = OFF_BAR + 256;                          // 231168
static_assert(SMEM_BYTES <= 232448, "shared memory budget");
// TMEM columns: XX, three digits of L, four of Q (32 each), then the A stages
// (X and O, 32 columns of f16 pairs each)
constexpr int COL_L = 32, COL_Q = 128, COL_A = 256;
static_assert(COL_A + NSTAGE * 64 <= 512, "TMEM budget");

// Sample-major codes: x (0, 1, 2) or 3 for a missing call.  A word holds 16 SNPs, SNP k
// in the field of bits 2 (k / 2) of its lower (k even) or upper (k odd) half, so that
// masking one field leaves the f16 pair of SNPs k, k + 1 (neighbours along K): bits 0-9
// are the subnormals' mantissa, linear in the code, 4^p 2^-24 for field p = 0..4, and
// fields 5-7 are 0-2 of the word shifted by 10.  The digits carry the 4^-p.
__host__ __device__ constexpr int field_pow(int j) { return j < 5 ? j : j - 5; }
constexpr float DIGIT_SCALE = 16.0f;  // of the digits as stored: below f16's largest
// the accumulators' unit: A x 2^24, B's codes (2^-14) x 2^14, digits
constexpr float ACC_SCALE = 17179869184.0f;  // 2^34 = 2^24 2^14 / DIGIT_SCALE

struct Args {
  const uint8_t* xt;    // sample-major 2-bit genotypes, n_pad rows x row_bytes
  const uint16_t* dig;  // f16 digits, [Kp/64][NDIG][64]
  const int2* tiles;    // (row block, column block) per tile
  const int* chunk;     // first step of each chunk, and the end
  const int* part;      // first chunk of each part of the SNPs, and the end
  int ntiles;
  int parts;
  int64_t row_bytes;    // Kp / 4
  int n;
  int q_exact;          // sums of e_j fit an int64
  double s2pq;
  double* G;            // n x n
  int32_t* xx;          // n x n or null
  // parts > 1: totals of each (tile, part), [col][row]; k_grm_sum adds them
  int32_t* pxx;
  int64_t* pl;
  int64_t* pq;          // int64 or the bits of a double, as q_exact says
  int* status;
};

struct Bars {
  uint64_t op_full[NSTAGE];
  uint64_t op_empty[NSTAGE];
  uint64_t raw_full[NRAW];
  uint64_t raw_empty[NRAW];
  uint64_t acc_full;
  uint64_t acc_empty;
  uint64_t drain;
  uint32_t tmem_base;
  int abort;
};

__device__ __forceinline__ void fail(Bars* b, int* status) {
  b->abort = 1;
  atomicExch(status, DEV_TIMEOUT);
}

// no memory clobber: loads of the raw stage may pass the stores to the operand stage
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c,
                                             uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c),
               "r"(d));
}

// codes -> x (0 where missing) and observed (1 or 0), two bits a field
__device__ __forceinline__ void split_codes(uint32_t w, uint32_t& x, uint32_t& o) {
  const uint32_t mis = w & (w >> 1) & 0x55555555u;
  x = w & ~(mis * 3u);
  o = ~mis & 0x55555555u;
}

__device__ __forceinline__ uint32_t half2_bits(float v) {
  const __half2 h = __float2half2_rn(v);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// one answer for the whole warp, whose next instructions are warp-wide
__device__ __forceinline__ bool wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort));
}

__device__ __forceinline__ uint32_t hmul2u(uint32_t a, uint32_t b) {
  __half2 r = __hmul2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
  return *reinterpret_cast<uint32_t*>(&r);
}

// D[tmem] (+)= A[tmem] * B[smem]^T
__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// 32 lanes x 16 consecutive 32-bit columns
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

// digit of the residue v in [0, base): base / 2 and up go to the next digit's side
__host__ __device__ __forceinline__ int balanced(int v, int base) {
  return v >= base / 2 ? v - base : v;
}

__device__ __forceinline__ int32_t acc_int(uint32_t v) {
  return __float2int_rn(__uint_as_float(v) * ACC_SCALE);
}

// totals of Q: int64 or double bits
__device__ __forceinline__ int64_t q_add(int64_t a, int64_t b, bool exact) {
  return exact ? a + b : __double_as_longlong(__longlong_as_double(a) + __longlong_as_double(b));
}

__device__ __forceinline__ double grm_value(int32_t xx, int64_t l, int64_t qt, bool exact, double s2pq) {
  const double q = exact ? (double)qt : __longlong_as_double(qt);
  const int64_t xl = (int64_t)xx * (int64_t(1) << 29) - l;
  const double raw = (double)xl * 0x1p-29 + q * 0x1p-45;
  return s2pq > 0 ? raw / s2pq : raw;
}

// One item = a 128 x 32 tile of G over one part of the SNPs.  The A operands (X and O of
// the 128 rows) are written straight to TMEM, the 11 variants of the 32 columns to shared
// memory; 16 SNPs are X (X, O a) and O (X a, O e), two products of 128 and 224 columns
// whose results lie side by side in TMEM.
// Bound by the two products (950 cycles per 64 SNPs; the B stores and reads keep the
// shared-memory pipe busy for 700 of them); a step takes 1,010 to 1,070.  With A in shared
// memory too, products of 96 and 128 columns, steps of 32 SNPs made by all producers
// together and a flush every 2048 SNPs it was 2,300: at n = 12,000, m = 40,001 90.2 ms,
// now 40.
__global__ void __launch_bounds__(THREADS, 1) k_grm_tc(Args args) {
  extern __shared__ __align__(1024) uint8_t smem[];
  Bars* bars = reinterpret_cast<Bars*>(smem + OFF_BAR);
  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;

  if (tid == 0) {
    for (int i = 0; i < NSTAGE; ++i) {
      mbar_init(&bars->op_full[i], NPROD);
      mbar_init(&bars->op_empty[i], 1);
    }
    for (int i = 0; i < NRAW; ++i) {
      mbar_init(&bars->raw_full[i], 32);
      mbar_init(&bars->raw_empty[i], NPROD);
    }
    mbar_init(&bars->acc_full, 1);
    mbar_init(&bars->acc_empty, 4);
    mbar_init(&bars->drain, 1);
    bars->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  volatile int* abort_flag = &bars->abort;
  const int nitems = args.ntiles * args.parts;

  if (warp == 0) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      constexpr uint32_t ID96 = idesc_f16_f32(128, 96);
      constexpr uint32_t ID128 = idesc_f16_f32(128, 128);
      constexpr uint32_t ID224 = idesc_f16_f32(128, 224);
      uint32_t g = 0, c = 0;
      bool ok = true;
      for (int it = blockIdx.x; it < nitems && ok; it += gridDim.x) {
        const int pt = it % args.parts;
        for (int ch = args.part[pt]; ch < args.part[pt + 1] && ok; ++ch, ++c) {
          if (!mbar_wait(&bars->acc_empty, (c & 1) ^ 1, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const int ns = args.chunk[ch + 1] - args.chunk[ch];
          for (int s = 0; s < ns; ++s, ++g) {
            const uint32_t slot = g % NSTAGE;
            if (!mbar_wait(&bars->op_full[slot], (g / NSTAGE) & 1, abort_flag)) { ok = false; break; }
            tc_fence_after();
            const uint32_t bB = smem_addr(smem + OFF_STAGE + slot * STAGE_BYTES);
            const uint32_t aX = tmem_base + COL_A + slot * 64, aO = aX + 32;
#pragma unroll
            for (int ks = 0; ks < KSTEP / 16; ++ks) {
              const uint32_t ko = ks * 256;  // two 8-element core matrices along K
              const uint32_t ka = ks * 8;    // 16 f16 of K per lane
              if (s == 0 && ks == 0) {
                // a chunk's first products replace the accumulators: XX and the
                // three L's by X (X, O a), Q by O O e
                umma_f16_ts(tmem_base, aX, sdesc_noswizzle(bB, 128, 1024), ID128, 0u);
                umma_f16_ts(tmem_base + COL_L, aO, sdesc_noswizzle(bB + 4 * B_VAR_BYTES, 128, 1024),
                            ID96, 1u);
                umma_f16_ts(tmem_base + COL_Q, aO, sdesc_noswizzle(bB + 7 * B_VAR_BYTES, 128, 1024),
                            ID128, 0u);
              } else {
                umma_f16_ts(tmem_base, aX + ka, sdesc_noswizzle(bB + ko, 128, 1024), ID128, 1u);
                umma_f16_ts(tmem_base + COL_L, aO + ka,
                            sdesc_noswizzle(bB + 4 * B_VAR_BYTES + ko, 128, 1024), ID224, 1u);
              }
            }
            umma_commit(&bars->op_empty[slot]);
          }
          if (ok) umma_commit(&bars->acc_full);
        }
      }
      if (!ok) fail(bars, args.status);
      // make sure no MMA is in flight before TMEM is released
      umma_commit(&bars->drain);
      if (!mbar_wait(&bars->drain, 0, abort_flag)) {
        // abort already set; the final wait below is bounded by time only
        const uint64_t t0 = global_ns();
        while (!mbar_try(&bars->drain, 0) && global_ns() - t0 < kWaitLimitNs) {}
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- raw loader (cp.async) ----------------
    uint32_t g = 0;
    bool ok = true;
    for (int it = blockIdx.x; it < nitems && ok; it += gridDim.x) {
      const int2 tl = args.tiles[it / args.parts];
      const int pt = it % args.parts;
      const uint8_t* rowA = args.xt + (int64_t)tl.x * TILE_M * args.row_bytes;
      const uint8_t* rowB = args.xt + (int64_t)tl.y * TILE_N * args.row_bytes;
      const int p1 = args.chunk[args.part[pt + 1]];
      for (int p = args.chunk[args.part[pt]]; p < p1; ++p, ++g) {
        const uint32_t slot = g % NRAW;
        if (!mbar_wait(&bars->raw_empty[slot], ((g / NRAW) & 1) ^ 1, abort_flag)) { ok = false; break; }
        uint8_t* raw = smem + OFF_RAW + slot * RAW_BYTES;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int r = lane + 32 * q;
          cp_async_16(raw + r * 16, rowA + (int64_t)r * args.row_bytes + (int64_t)p * 16);
        }
        cp_async_16(raw + RAW_A + lane * 16, rowB + (int64_t)lane * args.row_bytes + (int64_t)p * 16);
        const uint16_t* dg = args.dig + (int64_t)p * NDIG * KSTEP;
#pragma unroll
        for (int q = 0; q < 2; ++q)
          if (lane + 32 * q < RAW_D / 16)
            cp_async_16(raw + RAW_A + RAW_B + (lane + 32 * q) * 16, dg + (lane + 32 * q) * 8);
        cp_async_arrive(&bars->raw_full[slot]);
      }
    }
    if (!ok) fail(bars, args.status);
    cp_async_wait_all();
  } else if (warp >= 4 && warp < 20) {
    // ---------------- producers: 2-bit codes -> f16 operands ----------------
    const bool side_a = warp < 12;
    const int q = warp & 3;
    const uint32_t grp = ((warp >> 2) & 1) ^ 1;  // warps 4-7 and 12-15: the even steps
    constexpr float S0 = DIGIT_SCALE;
    const uint32_t scale[5] = {half2_bits(S0), half2_bits(S0 / 4), half2_bits(S0 / 16),
                               half2_bits(S0 / 64), half2_bits(S0 / 256)};
    uint32_t g = 0;
    bool ok = true;
    for (int it = blockIdx.x; it < nitems && ok; it += gridDim.x) {
      const int pt = it % args.parts;
      const int p1 = args.chunk[args.part[pt + 1]];
      for (int p = args.chunk[args.part[pt]]; p < p1; ++p, ++g) {
        if ((g & 1) != grp) continue;
        const uint32_t rslot = g % NRAW, oslot = g % NSTAGE;
        const uint32_t ophase = ((g / NSTAGE) & 1) ^ 1;
        if (!wait_warp(&bars->raw_full[rslot], (g / NRAW) & 1, abort_flag)) { ok = false; break; }
        const uint8_t* raw = smem + OFF_RAW + rslot * RAW_BYTES;
        if (side_a) {
          // thread = row of the tile: 64 SNPs of X and of O into its TMEM lane
          const uint4 w4 = *reinterpret_cast<const uint4*>(raw + (q * 32 + lane) * 16);
          const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
          const uint32_t ta = tmem_base + (uint32_t(q * 32) << 16) + COL_A + oslot * 64;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t X[16], O[16];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              uint32_t x, o;
              split_codes(w[2 * h + u], x, o);
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const uint32_t m = 0x00030003u << (2 * field_pow(j));
                X[8 * u + j] = (j < 5 ? x : x >> 10) & m;
                O[8 * u + j] = (j < 5 ? o : o >> 10) & m;
              }
            }
            if (h == 0) {
              __syncwarp();
              if (lane == 0) mbar_arrive(&bars->raw_empty[rslot]);
              if (!wait_warp(&bars->op_empty[oslot], ophase, abort_flag)) { ok = false; break; }
              tc_fence_after();
            }
            tmem_st16(ta + 16 * h, X);
            tmem_st16(ta + 32 + 16 * h, O);
          }
          if (!ok) break;
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          tc_fence_before();
        } else {
          // thread = (row of the tile's columns, 16 SNPs), 11 variants; codes as 2^-14 x
          const uint32_t w = *reinterpret_cast<const uint32_t*>(raw + RAW_A + lane * 16 + q * 4);
          uint32_t x, o;
          split_codes(w, x, o);
          const uint8_t* dg = raw + RAW_A + RAW_B + q * 32;
          const uint32_t vb = smem_addr(smem + OFF_STAGE + oslot * STAGE_BYTES) + (lane >> 3) * 1024 +
                              (lane & 7) * 16 + q * 256;
          if (!wait_warp(&bars->op_empty[oslot], ophase, abort_flag)) { ok = false; break; }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t X[4], O[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint32_t xs = h ? x >> 8 : x, os = h ? o >> 8 : o;
              X[j] = (xs << (10 - 2 * j)) & 0x0C000C00u;
              O[j] = (os << (10 - 2 * j)) & 0x0C000C00u;
            }
            const uint32_t vh = vb + h * 128;
            uint32_t Y[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) Y[j] = hmul2u(X[j], scale[field_pow(4 * h + j)]);
            st_shared_v4(vh, Y[0], Y[1], Y[2], Y[3]);
#pragma unroll
            for (int d = 0; d < NDIG; ++d) {
              const uint4 dv = *reinterpret_cast<const uint4*>(dg + h * 16 + d * (KSTEP * 2));
              const int v = d < 3 ? 1 + d : 4 + d;
              st_shared_v4(vh + v * B_VAR_BYTES, hmul2u(O[0], dv.x), hmul2u(O[1], dv.y),
                           hmul2u(O[2], dv.z), hmul2u(O[3], dv.w));
              if (d < 3)
                st_shared_v4(vh + (4 + d) * B_VAR_BYTES, hmul2u(X[0], dv.x), hmul2u(X[1], dv.y),
                             hmul2u(X[2], dv.z), hmul2u(X[3], dv.w));
            }
          }
          fence_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->raw_empty[rslot]);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->op_full[oslot]);
      }
    }
    if (!ok) fail(bars, args.status);
  } else if (warp >= 20) {
    // ---------------- epilogue: exact chunk flush + final write ----------------
    const int q = warp & 3;
    const int row = q * 32 + lane;
    int32_t* XX = reinterpret_cast<int32_t*>(smem + OFF_XX);
    int64_t* LT = reinterpret_cast<int64_t*>(smem + OFF_L);
    int64_t* QT = reinterpret_cast<int64_t*>(smem + OFF_Q);
    const bool exact = args.q_exact;
    const uint32_t ta = tmem_base + (uint32_t(q * 32) << 16);
    uint32_t c = 0;
    bool ok = true;
    for (int it = blockIdx.x; it < nitems && ok; it += gridDim.x) {
      const int2 tl = args.tiles[it / args.parts];
      const int pt = it % args.parts;
      const int c0 = args.part[pt], c1 = args.part[pt + 1];
      for (int ch = c0; ch < c1; ++ch, ++c) {
        if (!__all_sync(0xffffffffu, mbar_wait_idle(&bars->acc_full, c & 1, abort_flag, 200))) {
          ok = false;
          break;
        }
        tc_fence_after();
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          {
            uint32_t vx[16], l0[16], l1[16];
            tmem_ld16(ta + 16 * h, vx);
            tmem_ld16(ta + COL_L + 16 * h, l0);
            tmem_ld16(ta + COL_L + 32 + 16 * h, l1);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const int e = (16 * h + j) * TILE_M + row;
              const int32_t xi = acc_int(vx[j]);
              const int64_t L = (int64_t)acc_int(l0[j]) +
                                (int64_t)acc_int(l1[j]) * 2048;
              XX[e] = ch == c0 ? xi : XX[e] + xi;
              LT[e] = ch == c0 ? L : LT[e] + L;
            }
            tmem_ld16(ta + COL_L + 64 + 16 * h, l0);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j)
              LT[(16 * h + j) * TILE_M + row] +=
                  (int64_t)acc_int(l0[j]) * 4194304;
          }
          int64_t Q[16];
          {
            uint32_t q0[16], q1[16];
            tmem_ld16(ta + COL_Q + 16 * h, q0);
            tmem_ld16(ta + COL_Q + 32 + 16 * h, q1);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j)
              Q[j] = (int64_t)acc_int(q0[j]) +
                     (int64_t)acc_int(q1[j]) * 4096;
            tmem_ld16(ta + COL_Q + 64 + 16 * h, q0);
            tmem_ld16(ta + COL_Q + 96 + 16 * h, q1);
            tmem_ld_wait();
            if (h == 1) {
              // everything is in registers: the next chunk may replace the accumulators
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(&bars->acc_empty);
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const int e = (16 * h + j) * TILE_M + row;
              const int64_t t = Q[j] + (((int64_t)acc_int(q0[j]) +
                                         (int64_t)acc_int(q1[j]) * 4096)
                                        * 16777216);
              const int64_t v = exact ? t : __double_as_longlong((double)t);
              QT[e] = ch == c0 ? v : q_add(QT[e], v, exact);
            }
          }
        }
      }
      if (!ok) break;
      if (args.parts > 1) {
        // this part's totals, summed by k_grm_sum
        const int64_t base = (int64_t)it * (TILE_M * TILE_N) + row;
        for (int col = 0; col < TILE_N; ++col) {
          const int e = col * TILE_M + row;
          args.pxx[base + col * TILE_M] = XX[e];
          args.pl[base + col * TILE_M] = LT[e];
          args.pq[base + col * TILE_M] = QT[e];
        }
        continue;
      }
      // final write of this tile (both triangles)
      const int gi = tl.x * TILE_M + row;
      if (gi < args.n) {
        for (int col = 0; col < TILE_N; ++col) {
          const int gk = tl.y * TILE_N + col;
          if (gk >= args.n) break;
          const int e = col * TILE_M + row;
          const int32_t xi = XX[e];
          const double gv = grm_value(xi, LT[e], QT[e], exact, args.s2pq);
          args.G[(int64_t)gi * args.n + gk] = gv;
          args.G[(int64_t)gk * args.n + gi] = gv;
          if (args.xx) {
            args.xx[(int64_t)gi * args.n + gk] = xi;
            args.xx[(int64_t)gk * args.n + gi] = xi;
          }
        }
      }
    }
    if (!ok) fail(bars, args.status);
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem_base, 512);
}

// The totals of a tile's parts, in order, to G and the counts: grid (tile, 8 column groups).
__global__ void __launch_bounds__(512) k_grm_sum(Args args) {
  const int t = blockIdx.x, row = threadIdx.x, col = blockIdx.y * 4 + threadIdx.y;
  const int2 tl = args.tiles[t];
  const int64_t base = (int64_t)t * args.parts * (TILE_M * TILE_N) + col * TILE_M + row;
  int32_t x = 0;
  int64_t l = 0, q = 0;  // the zero of both forms of q
  for (int p = 0; p < args.parts; ++p) {
    const int64_t e = base + (int64_t)p * (TILE_M * TILE_N);
    x += args.pxx[e];
    l += args.pl[e];
    q = q_add(q, args.pq[e], args.q_exact);
  }
  const int gi = tl.x * TILE_M + row, gk = tl.y * TILE_N + col;
  if (gi >= args.n || gk >= args.n) return;
  const double gv = grm_value(x, l, q, args.q_exact, args.s2pq);
  args.G[(int64_t)gi * args.n + gk] = gv;
  args.G[(int64_t)gk * args.n + gi] = gv;
  if (args.xx) {
    args.xx[(int64_t)gi * args.n + gk] = x;
    args.xx[(int64_t)gk * args.n + gi] = x;
  }
}

// Digits of a_j = mean_j 2^29 (base 2048) and e_j = round(a_j^2 / 2^13) (base 4096) as
// f16, in the order of the operand stages; zeros beyond K.
__global__ void k_grm_digits(const float* __restrict__ mean, int64_t K, int64_t Kp,
                             uint16_t* __restrict__ dig) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= Kp) return;
  int d[NDIG] = {0, 0, 0, 0, 0, 0, 0};
  if (k < K) {
    const int64_t a = (int64_t)((double)mean[k] * 536870912.0);
    int64_t r = a;
    for (int q = 0; q < 2; ++q) {
      d[q] = balanced((int)(r & 2047), 2048);
      r = (r - d[q]) >> 11;
    }
    d[2] = (int)r;
    int64_t e = (int64_t)(((uint64_t)a * (uint64_t)a + (uint64_t(1) << 12)) >> 13);
    for (int q = 3; q < 6; ++q) {
      d[q] = balanced((int)(e & 4095), 4096);
      e = (e - d[q]) >> 12;
    }
    d[6] = (int)e;
  }
  const float scale = DIGIT_SCALE / (float)(1 << (2 * field_pow((int)(k & 15) >> 1)));
  for (int q = 0; q < NDIG; ++q)
    dig[((k / KSTEP) * NDIG + q) * KSTEP + k % KSTEP] = __half_as_ushort(__float2half_rn(d[q] * scale));
}

// Per-SNP tallies of 2-bit codes over the first n samples (codes beyond n ignored).
__global__ void k_snp_counts(const uint8_t* __restrict__ payload, int64_t n, int64_t m,
                             int64_t bps, int32_t* n_obs, int32_t* sum_x, int32_t* n_hom1,
                             int32_t* n_het, int32_t* n_hom2) {
  const int64_t j = blockIdx.x;
  if (j >= m) return;
  const uint8_t* row = payload + j * bps;
  int hom1 = 0, het = 0, hom2 = 0;
  for (int64_t b = threadIdx.x; b < bps; b += blockDim.x) {
    const uint32_t v = row[b];
    const int64_t left = n - 4 * b;
    const uint32_t mask = left >= 4 ? 0x55u : (0x55u >> (2 * (4 - left)));
    const uint32_t lo = v & 0x55u, hi = (v >> 1) & 0x55u;
    hom1 += __popc(~lo & ~hi & mask);
    het += __popc(~lo & hi & mask);
    hom2 += __popc(lo & hi & mask);
  }
  __shared__ int red[3][32];
  for (int off = 16; off > 0; off >>= 1) {
    hom1 += __shfl_down_sync(0xffffffffu, hom1, off);
    het += __shfl_down_sync(0xffffffffu, het, off);
    hom2 += __shfl_down_sync(0xffffffffu, hom2, off);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) { red[0][w] = hom1; red[1][w] = het; red[2][w] = hom2; }
  __syncthreads();
  if (threadIdx.x == 0) {
    int a = 0, b2 = 0, c = 0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) { a += red[0][i]; b2 += red[1][i]; c += red[2][i]; }
    if (n_obs) n_obs[j] = a + b2 + c;
    if (sum_x) sum_x[j] = 2 * a + b2;
    if (n_hom1) n_hom1[j] = a;
    if (n_het) n_het[j] = b2;
    if (n_hom2) n_hom2[j] = c;
  }
}

// Transpose the valid SNPs into sample-major 2-bit rows, coded as above, in the fields
// named there.  Samples >= n and SNP columns >= K are missing.
__global__ void k_repack(const uint8_t* __restrict__ payload, int64_t n, int64_t bps,
                         const int32_t* __restrict__ valid_idx, int64_t K, int64_t row_bytes,
                         uint8_t* __restrict__ xt) {
  __shared__ uint8_t raw[64][33];
  const int kb = blockIdx.x, ib = blockIdx.y, t = threadIdx.x;
  for (int idx = t; idx < 64 * 32; idx += 128) {
    const int sl = idx >> 5, byte = idx & 31;
    const int64_t k = (int64_t)kb * 64 + sl;
    const int64_t sb = (int64_t)ib * 32 + byte;
    uint8_t v = 0x55;
    if (k < K && sb < bps) v = payload[(int64_t)valid_idx[k] * bps + sb];
    raw[sl][byte] = v;
  }
  __syncthreads();
  const int64_t i = (int64_t)ib * 128 + t;
  uint32_t out[4] = {0, 0, 0, 0};
#pragma unroll 4
  for (int s = 0; s < 64; ++s) {
    uint32_t code = (raw[s][t >> 2] >> (2 * (t & 3))) & 3u;
    if (i >= n) code = 1;
    code = (0x1Eu >> (2 * code)) & 3u;  // BED 00, 01, 10, 11 -> 2, 3, 1, 0
    out[s >> 4] |= code << (16 * (s & 1) + (s & 14));
  }
  uint4* dst = reinterpret_cast<uint4*>(xt + i * row_bytes + (int64_t)kb * 16);
  *dst = make_uint4(out[0], out[1], out[2], out[3]);
}

// Parts that the SNPs of every tile are cut into: more only where that fills the SMs
// better, by the rounds of items times the steps of one (each item adds about ten
// steps' time of filling the stages and of the flush).  At n = 501, m = 5,003 (40 tiles)
// three parts: the tiles 28 + 12 us for the sum, 96 us by 40 SMs before.
static int choose_parts(int64_t ntiles, int np, int sms) {
  int best = 1;
  int64_t cost = INT64_MAX;
  for (int p = 1; p <= 16 && p <= np; ++p) {
    if (p > 1 && ntiles * p > 8 * (int64_t)sms) break;
    const int64_t c = ((ntiles * p + sms - 1) / sms) * ((np + p - 1) / p + 10);
    if (c < cost) {
      cost = c;
      best = p;
    }
  }
  return best;
}

// G is copied to pinned host memory behind the tiles, in groups of whole rounds of tiles:
// the row blocks that a group completes are, with the entries below them, two rectangles.
// From two rounds a group on.  The call at n = 12,000, m = 40,001 (59 rounds): 48.1 ms with one copy
// after the tiles, 43.8 in four groups, 43.0 in eight, 42.9 in 16; at n = 6,000, m = 20,000 (14
// rounds) 7.3, 6.4, 6.3 and 6.4.
constexpr int COPY_GROUPS = 8;

static bool is_pinned(const void* p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeHost;
}

// Copies on the second stream; none is left running when the call ends, by an error or not.
struct CopyBehind {
  cbx_handle* h;
  bool used = false;
  // rows r0 .. r1 - 1 from column r0 on and the columns below them
  void add(cudaStream_t s, const double* src, double* dst, int64_t n, int64_t r0, int64_t r1) {
    if (r1 <= r0) return;
    used = true;
    CBX_CUDA(cudaEventRecord(h->ev_fork, s));
    CBX_CUDA(cudaStreamWaitEvent(h->stream2, h->ev_fork, 0));
    rect(src + r0 * n + r0, dst + r0 * n + r0, n, r1 - r0, n - r0);
    if (r1 < n) rect(src + r1 * n + r0, dst + r1 * n + r0, n, n - r1, r1 - r0);
  }
  void rect(const double* src, double* dst, int64_t n, int64_t rows, int64_t cols) {
    CBX_CUDA(cudaMemcpy2DAsync(dst, n * 8, src, n * 8, cols * 8, rows, cudaMemcpyDeviceToHost, h->stream2));
  }
  void finish() {
    if (used) CBX_CUDA(cudaStreamSynchronize(h->stream2));
    used = false;
  }
  ~CopyBehind() {
    if (used) cudaStreamSynchronize(h->stream2);
  }
};

}  // namespace grm
}  // namespace cbx

using namespace cbx;

static const uint8_t* check_bed_bytes(const uint8_t* bed, int64_t bed_bytes, int64_t n, int64_t m) {
  CBX_REQUIRE(bed != nullptr, CBX_ERR_ARG, "bed is null");
  CBX_REQUIRE(n > 0 && m > 0, CBX_ERR_ARG, "Empty dataset provided to GrmBuilder");
  CBX_REQUIRE(n < (int64_t(1) << 31) && m < (int64_t(1) << 31), CBX_ERR_ARG, "n or m too large");
  CBX_REQUIRE(bed_bytes >= 3, CBX_ERR_FORMAT, "Invalid .bed file (too small)");
  CBX_REQUIRE(bed[0] == 0x6C && bed[1] == 0x1B, CBX_ERR_FORMAT, "Invalid .bed file magic number");
  CBX_REQUIRE(bed[2] == 0x01, CBX_ERR_FORMAT, "Only SNP-major mode (0x01) .bed files are supported");
  const int64_t bps = (n + 3) / 4;
  CBX_REQUIRE(bed_bytes >= 3 + m * bps, CBX_ERR_FORMAT,
              ".bed file is truncated: " + std::to_string(bed_bytes) + " < " +
                  std::to_string(3 + m * bps) + " bytes");
  return bed + 3;
}

extern "C" int cbx_bed_snp_counts(cbx_handle* h, const uint8_t* bed, int64_t bed_bytes, int64_t n,
                                  int64_t m, int32_t* n_obs, int32_t* sum_x, int32_t* n_hom1,
                                  int32_t* n_het, int32_t* n_hom2) {
  return cbx_guard(h, [&] {
    const uint8_t* payload = check_bed_bytes(bed, bed_bytes, n, m);
    CBX_CUDA(cudaSetDevice(h->device));
    const int64_t bps = (n + 3) / 4;
    DevBuf<uint8_t> d_bed;
    d_bed.resize(m * bps);
    CBX_CUDA(cudaMemcpyAsync(d_bed.p, payload, m * bps, cudaMemcpyHostToDevice, h->stream));
    DevBuf<int32_t> cnt;
    cnt.resize(5 * m);
    grm::k_snp_counts<<<(unsigned)m, 128, 0, h->stream>>>(d_bed.p, n, m, bps, cnt.p, cnt.p + m,
                                                          cnt.p + 2 * m, cnt.p + 3 * m, cnt.p + 4 * m);
    h->launched("k_snp_counts");
    int32_t* outs[5] = {n_obs, sum_x, n_hom1, n_het, n_hom2};
    for (int i = 0; i < 5; ++i)
      if (outs[i])
        CBX_CUDA(cudaMemcpyAsync(outs[i], cnt.p + i * m, m * sizeof(int32_t), cudaMemcpyDeviceToHost,
                                 h->stream));
    CBX_CUDA(cudaStreamSynchronize(h->stream));
  });
}

extern "C" int cbx_grm_bed(cbx_handle* h, const uint8_t* bed, int64_t bed_bytes, int64_t n, int64_t m,
                           float min_maf, int algorithm, int64_t block_size, double* G,
                           int32_t* xx_counts, float* allele_freqs, double* sum2pq,
                           int64_t* n_valid) {
  return cbx_guard(h, [&] {
    CBX_REQUIRE(algorithm == 1, CBX_ERR_UNSUPPORTED,
                "GPU GRM implements algorithm 1 (VanRaden) only; got " + std::to_string(algorithm));
    CBX_REQUIRE(block_size > 0, CBX_ERR_ARG, "block_size must be positive");
    const uint8_t* payload = check_bed_bytes(bed, bed_bytes, n, m);
    CBX_CUDA(cudaSetDevice(h->device));
    cudaStream_t s = h->stream;
    const int64_t bps = (n + 3) / 4;

    // scratch: the BED bytes and tallies, then everything sized by the valid SNPs;
    // kept by the handle up to 64 MB each
    struct Scratch {
      cbx_handle* h;
      uint8_t* get(int i, size_t bytes) {
        if (h->grm_ws[i].n < bytes) h->grm_ws[i].resize(bytes);
        return h->grm_ws[i].p;
      }
      ~Scratch() {
        for (auto& w : h->grm_ws)
          if (w.n > (size_t(64) << 20)) w.release();
      }
    } scratch{h};
    auto up = [](size_t b) { return (b + 255) & ~size_t(255); };

    // 1. per-SNP integer tallies on the device
    uint8_t* d_bed = scratch.get(0, up(m * bps) + m * 8);
    int32_t* d_cnt = reinterpret_cast<int32_t*>(d_bed + up(m * bps));
    CBX_CUDA(cudaMemcpyAsync(d_bed, payload, m * bps, cudaMemcpyHostToDevice, s));
    grm::k_snp_counts<<<(unsigned)m, 128, 0, s>>>(d_bed, n, m, bps, d_cnt, d_cnt + m, nullptr,
                                                  nullptr, nullptr);
    h->launched("k_snp_counts");
    std::vector<int32_t> n_obs(m), sum_x(m);
    CBX_CUDA(cudaMemcpyAsync(n_obs.data(), d_cnt, m * 4, cudaMemcpyDeviceToHost, s));
    CBX_CUDA(cudaMemcpyAsync(sum_x.data(), d_cnt + m, m * 4, cudaMemcpyDeviceToHost, s));
    CBX_CUDA(cudaStreamSynchronize(s));

    // 2. host: validity, float mean / 2pq, blocked sum 2pq (grm_builder.cpp:219-277,353)
    std::vector<int32_t> valid_idx;
    std::vector<float> mean;
    valid_idx.reserve(m);
    double total_sum_2pq = 0.0;
    const double thr = static_cast<double>(min_maf);
    for (int64_t start = 0; start < m; start += block_size) {
      const int64_t end = std::min(start + block_size, m);
      double block_sum = 0.0;
      for (int64_t j = start; j < end; ++j) {
        if (allele_freqs) allele_freqs[j] = -1.0f;
        if (n_obs[j] == 0) continue;
        const double freq = (double)sum_x[j] / (2.0 * n_obs[j]);
        const double maf = std::min(freq, 1.0 - freq);
        if (maf < thr || std::abs(maf) < 1e-8) continue;
        const float two_pq = (float)(1.0f * 2.0 * freq * (1.0 - freq));
        if (allele_freqs) allele_freqs[j] = (float)freq;
        mean.push_back((float)(freq * 2.0));
        valid_idx.push_back((int32_t)j);
        block_sum += two_pq;
      }
      total_sum_2pq += block_sum;
    }
    const int64_t K = (int64_t)valid_idx.size();
    if (sum2pq) *sum2pq = total_sum_2pq;
    if (n_valid) *n_valid = K;

    h->G.resize(n * n);
    h->G_n = n;
    if (K == 0) {
      // no usable SNP: the reference leaves G at zero
      h->G.zero(s);
      if (G) CBX_CUDA(cudaMemsetAsync(h->G.p, 0, n * n * sizeof(double), s));
      if (G) std::memset(G, 0, n * n * sizeof(double));
      if (xx_counts) std::memset(xx_counts, 0, n * n * sizeof(int32_t));
      CBX_CUDA(cudaStreamSynchronize(s));
      return;
    }
    // L stays an exact int64 below 2^53 for up to 2^21 SNPs
    CBX_REQUIRE(K <= 2000000, CBX_ERR_UNSUPPORTED, "more than 2e6 valid SNPs");

    // 3. tiles of the upper triangle (128-row x 32-column blocks), parts and chunks
    // of the SNPs
    const int64_t Kp = (K + 63) / 64 * 64;
    const int64_t n_pad = (n + 127) / 128 * 128;
    const int64_t row_bytes = Kp / 4;
    const int nib = (int)(n_pad / 128), njb = (int)(n_pad / 32);
    std::vector<int2> tiles;
    for (int ib = 0; ib < nib; ++ib)
      for (int jb = 4 * ib; jb < njb; ++jb) tiles.push_back(make_int2(ib, jb));
    const int np = (int)(Kp / 64);
    const int parts = grm::choose_parts((int64_t)tiles.size(), np, h->num_sms);
    std::vector<int> chunk, part;
    {
      int64_t s0 = 0, s1 = 0;
      int len = 0, next = 0;
      for (int p = 0; p < np; ++p) {
        int64_t t0 = 0, t1 = 0;
        for (int64_t k = 64 * (int64_t)p; k < std::min<int64_t>(64 * (int64_t)(p + 1), K); ++k) {
          const double ad = (double)mean[k] * 536870912.0;  // 2^29
          const int64_t a = (int64_t)ad;
          CBX_REQUIRE((double)a == ad && a > 0 && a < (int64_t(1) << 30), CBX_ERR_ARG,
                      "allele mean outside the exact-integer range (MAF filter below 2^-7?)");
          const int d0 = grm::balanced((int)(a & 2047), 2048);
          t0 += std::abs(d0);
          t1 += std::abs(grm::balanced((int)(((a - d0) >> 11) & 2047), 2048));
        }
        const bool first = p == next;  // a part starts here
        if (first || len == grm::MAX_CHUNK || s0 + t0 > grm::SUM_LIMIT || s1 + t1 > grm::SUM_LIMIT) {
          if (first) {
            part.push_back((int)chunk.size());
            next = (int)((int64_t)np * (int64_t)part.size() / parts);
          }
          chunk.push_back(p);
          s0 = s1 = 0;
          len = 0;
        }
        s0 += t0;
        s1 += t1;
        ++len;
      }
      part.push_back((int)chunk.size());
      chunk.push_back(np);
    }

    // 4. upload tables, digits, repack to sample-major 2-bit rows
    const size_t items = parts > 1 ? tiles.size() * parts : 0;
    const size_t pel = (size_t)grm::TILE_M * grm::TILE_N;
    const size_t o_valid = 0, o_mean = o_valid + up(K * 4), o_tiles = o_mean + up(K * 4),
                 o_chunk = o_tiles + up(tiles.size() * sizeof(int2)),
                 o_part = o_chunk + up(chunk.size() * 4), o_dig = o_part + up(part.size() * 4),
                 o_xt = o_dig + up(Kp * grm::NDIG * 2), o_xx = o_xt + up(n_pad * row_bytes),
                 o_pl = o_xx + (xx_counts ? up((size_t)n * n * 4) : 0),
                 o_pq = o_pl + items * pel * 8, o_pxx = o_pq + items * pel * 8,
                 o_end = o_pxx + items * pel * 4;
    uint8_t* ws = scratch.get(1, o_end);
    int32_t* d_valid = reinterpret_cast<int32_t*>(ws + o_valid);
    CBX_CUDA(cudaMemcpyAsync(d_valid, valid_idx.data(), K * 4, cudaMemcpyHostToDevice, s));
    CBX_CUDA(cudaMemcpyAsync(ws + o_mean, mean.data(), K * 4, cudaMemcpyHostToDevice, s));
    CBX_CUDA(cudaMemcpyAsync(ws + o_tiles, tiles.data(), tiles.size() * sizeof(int2),
                             cudaMemcpyHostToDevice, s));
    CBX_CUDA(cudaMemcpyAsync(ws + o_chunk, chunk.data(), chunk.size() * 4, cudaMemcpyHostToDevice, s));
    CBX_CUDA(cudaMemcpyAsync(ws + o_part, part.data(), part.size() * 4, cudaMemcpyHostToDevice, s));
    uint16_t* d_dig = reinterpret_cast<uint16_t*>(ws + o_dig);
    grm::k_grm_digits<<<(unsigned)((Kp + 127) / 128), 128, 0, s>>>(
        reinterpret_cast<float*>(ws + o_mean), K, Kp, d_dig);
    h->launched("k_grm_digits");
    grm::k_repack<<<dim3((unsigned)(Kp / 64), (unsigned)(n_pad / 128)), 128, 0, s>>>(
        d_bed, n, bps, d_valid, K, row_bytes, ws + o_xt);
    h->launched("k_repack");

    // 5. the tiles
    int32_t* d_xx = reinterpret_cast<int32_t*>(ws + o_xx);
    grm::Args args;
    args.xt = ws + o_xt;
    args.dig = d_dig;
    args.tiles = reinterpret_cast<int2*>(ws + o_tiles);
    args.chunk = reinterpret_cast<int*>(ws + o_chunk);
    args.part = reinterpret_cast<int*>(ws + o_part);
    args.ntiles = (int)tiles.size();
    args.parts = parts;
    args.row_bytes = row_bytes;
    args.n = (int)n;
    args.q_exact = K <= grm::Q_EXACT;
    args.s2pq = total_sum_2pq;
    args.G = h->G.p;
    args.xx = xx_counts ? d_xx : nullptr;
    args.pl = reinterpret_cast<int64_t*>(ws + o_pl);
    args.pq = reinterpret_cast<int64_t*>(ws + o_pq);
    args.pxx = reinterpret_cast<int32_t*>(ws + o_pxx);
    args.status = h->status.p;
    ensure_smem((const void*)grm::k_grm_tc, grm::SMEM_BYTES, h->device);
    const int grid = (int)std::min<int64_t>(h->num_sms, (int64_t)args.ntiles * parts);
    cbx_handle::ProfRec pr{};
    if (h->prof_on) {
      CBX_CUDA(cudaEventCreate(&pr.a));
      CBX_CUDA(cudaEventCreate(&pr.b));
      CBX_CUDA(cudaEventRecord(pr.a, s));
    }
    const int rounds = args.ntiles / h->num_sms;
    const bool follow = G && parts == 1 && rounds >= 2 * grm::COPY_GROUPS && grm::is_pinned(G);
    grm::CopyBehind copies{h};
    if (follow) {
      int t0 = 0, ib = 0;
      for (int gr = 1; gr <= grm::COPY_GROUPS; ++gr) {
        const int t1 = gr == grm::COPY_GROUPS ? args.ntiles : rounds * gr / grm::COPY_GROUPS * h->num_sms;
        grm::Args part_args = args;
        part_args.tiles = args.tiles + t0;
        part_args.ntiles = t1 - t0;
        grm::k_grm_tc<<<std::min(h->num_sms, t1 - t0), grm::THREADS, grm::SMEM_BYTES, s>>>(part_args);
        h->launched("k_grm_tc");
        // row blocks whose tiles, and so all rows' and columns' entries from them on, are done
        const int64_t r0 = 128 * (int64_t)ib;
        while (ib < nib && (ib + 1 < nib ? (int)(std::lower_bound(tiles.begin(), tiles.end(), ib + 1,
                                                                  [](const int2& t, int b) { return t.x < b; }) -
                                                 tiles.begin())
                                         : args.ntiles) <= t1)
          ++ib;
        copies.add(s, h->G.p, G, n, r0, std::min<int64_t>(n, 128 * (int64_t)ib));
        t0 = t1;
      }
    } else {
      grm::k_grm_tc<<<grid, grm::THREADS, grm::SMEM_BYTES, s>>>(args);
      h->launched("k_grm_tc");
    }
    if (h->prof_on) {
      CBX_CUDA(cudaEventRecord(pr.b, s));
      pr.bucket = 2;
      // algorithmic integer work 2 n^2 K (the full square of X X^T)
      pr.bytes = 2.0 * (double)n * (double)n * (double)K;
      h->prof.push_back(pr);
    }
    if (parts > 1) {
      grm::k_grm_sum<<<dim3((unsigned)args.ntiles, grm::TILE_N / 4), dim3(grm::TILE_M, 4), 0, s>>>(args);
      h->launched("k_grm_sum");
    }
    h->check_status("cbx_grm_bed");
    if (G && !follow) CBX_CUDA(cudaMemcpyAsync(G, h->G.p, n * n * sizeof(double), cudaMemcpyDeviceToHost, s));
    if (xx_counts)
      CBX_CUDA(cudaMemcpyAsync(xx_counts, d_xx, n * n * sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    CBX_CUDA(cudaStreamSynchronize(s));
    copies.finish();
  });
}
