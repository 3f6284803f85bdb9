// FP64-accurate dense algebra on the tensor cores: C = A B', Cholesky factors and
// SPD inverses, for the set-up (G^-1, A22^-1, H^-1) and the dense AI-REML steps
// (reference: matrix_io.cpp:488-501, vce.cpp:2859-3195, relationship_builder.cpp:
// 573-584).  GB300 runs FP64 at 1/64 of its FP32 rate (1.2 TFLOP/s), so these
// were bound by cuSOLVER's FP64 GEMMs.
//
// Products.  Row i of an operand is scaled by 2^(61 - e_i), 2^e_i above its largest
// magnitude, and rounded to an integer |F| < 2^61 (below 2^-62 of the row maximum, the
// rounding of a double itself is 2^-54).  F is cut into eight balanced base-256
// digits (-128 .. 127, exact in f16).  The 36 digit pairs with s + t <= 7 are multiplied
// by kind::f16 MMAs; pairs of one weight s + t share an FP32 accumulator ("class"), whose
// partial sums are integers of at most 8 * 128 * 2^14 = 2^24, hence exact, over chunks
// of 128 K elements.  Each chunk is flushed into two int64 totals per output and the
// product is rounded to FP64 once.  The dropped pairs weigh below 2^-58 of the product
// of the two row maxima per term, less than an FP64 multiply-add's rounding.
//
// Factorization.  Right-looking in blocks of 32 inside outer panels of 256 or 512
// columns, in a row-major lower triangle W.  Step k (k_panel) factors the 32 x 32
// pivot block by FP64 elimination, giving X = L_kk^-1, and substitutes L_ik L_kk' = S_ik for
// the rows below; for the inverse also row k of M = L^-1, L_kk M_kj = R_kj for j < k, where
// R_ij = -sum_l L_il M_lj is kept in the slot of W that L_ij has left.  Digit MMAs then
// apply S_ij -= L_ik L_jk' and R_ij -= L_ik M_kj, within the panel after each step
// (K = 32) and to the rest once per panel (K = the panel's width).  A^-1 = M'M is one
// triangular product at the end.
//
// Bound: below n = 3,000 the chain of 32-wide steps (a pivot factor and a K = 32 update,
// 26 us); above it the digit MMAs (36 per FP64 multiply-add) and the L2 reads that feed
// them (96 KB a step of 2,304 tensor clocks).  Measured, inverse with its factor, against
// cuSOLVER potrf + potri: n = 500 0.61 ms (4.2), 2,000 2.7 (31), 8,000 35 (1,194), 20,000
// 322 (about 11,000).  The product at n = 2,000: 0.60 ms (15.3 by cuBLAS DGEMM).  128 x 64
// tiles: eight classes of 64 columns fill the 512 TMEM columns, and a narrower tile reads
// the A digits more often.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include "fx64.h"
#include "tma.cuh"

namespace cbx {
namespace fx {

constexpr int NPL = 8;                         // digit planes
constexpr int PLANE_A = 128 * 32 * 2;          // one plane of a 128-row, 32-wide block
constexpr int BLK = NPL * PLANE_A;             // 64 KB: one (row tile, K step) block
constexpr int NSTAGE = 2;
// Output tiles are 128 x NT, NT = 64 or 32: eight classes of NT TMEM columns.
template <int NT> struct Tile {
  static constexpr int PLANE_B = NT * 32 * 2;
  static constexpr int STAGE = BLK + NPL * PLANE_B;  // 96 or 80 KB
  static constexpr int EW = NT / 4;                  // epilogue warps: 16 columns of a TMEM lane quadrant each
  static constexpr int THREADS = 128 + 32 * EW;
  static constexpr int OFF_OUT = NSTAGE * STAGE;     // 2 KB per epilogue warp
  static constexpr int OFF_BAR = OFF_OUT + EW * 2048;
  static constexpr int SMEM = OFF_BAR + 256 + 1024;
  };
constexpr int CHUNK = 4;                       // K steps per exact FP32 chunk
constexpr int EX_MIN = -900, EX_BAD = 1 << 20; // exponent of a zero row; of a row with NaN / Inf
constexpr unsigned long long BIAS = 0x8080808080808080ull;  // 128 in each digit byte

// canonical K-major no-swizzle offset of (row, k) in a 32-wide f16 plane
__device__ __forceinline__ uint32_t cm_off(int r, int k) {
  return (uint32_t)((r >> 3) * 512 + (r & 7) * 16 + (k >> 3) * 128 + (k & 7) * 2);
}
// digit byte j of two elements as an f16 pair: byte - 128, exact
__device__ __forceinline__ uint32_t digit_pair(uint32_t ga, uint32_t gb, uint32_t j) {
  const uint32_t u = __byte_perm(ga, gb, j | ((j + 4) << 4));
  const uint32_t v = __byte_perm(u, 0x64646464u, 0x4140);  // f16 1024 + byte
  uint32_t d;
  asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(v), "r"(0xE480E480u));  // - 1152
  return d;
}
__device__ __forceinline__ double pow2d(int n) { return __longlong_as_double((long long)(n + 1023) << 52); }
// smallest e with |v| < 2^e (v finite, not zero), from the bits of |v|
__device__ __forceinline__ int expo(double v) {
  const int e = (int)((__double_as_longlong(v) >> 52) & 0x7FF);
  return e == 0x7FF ? EX_BAD : max(EX_MIN, e - 1022);
}
// (hi 2^32 + lo) 2^n, rounded to nearest (ties away from zero), for -900 < n < 900, in about 30 integer
// instructions without a branch: on GB300 each FP64 instruction or int64 conversion of a
// warp holds its quarter of the SM's FP64 pipe for 64 clocks.
__device__ __forceinline__ unsigned long long from_totals(long long hi, long long lo, int n) {
  const long long h = hi + (lo >> 32);
  const uint32_t m = (uint32_t)(h >> 63);
  const unsigned long long l = (unsigned long long)((uint32_t)lo ^ m) + (m & 1u);
  const unsigned long long t = ((unsigned long long)h ^ ((unsigned long long)m << 32 | m)) + (l >> 32);
  uint32_t w2 = (uint32_t)(t >> 32), w1 = (uint32_t)t, w0 = (uint32_t)l;  // |x| in 96 bits
  int e = 1023 + 32 + 62 + n;  // biased exponent, less the leading bit the mantissa adds
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const bool z = w2 == 0;
    w2 = z ? w1 : w2;
    w1 = z ? w0 : w1;
    w0 = z ? 0u : w0;
    e -= z ? 32 : 0;
  }
  const int c = __clz((int)w2);
  const uint32_t b1 = __funnelshift_l(w1, w2, c), b0 = __funnelshift_l(w0, w1, c);
  const unsigned long long b = ((unsigned long long)b1 << 32) | b0;
  const unsigned long long v = ((unsigned long long)(uint32_t)(e - c) << 52) + (b >> 11) + ((b >> 10) & 1);
  return w2 ? v | ((unsigned long long)(m & 1u) << 63) : 0ull;
}
// the same for any exponent (EX_BAD: a row with NaN or Inf)
__device__ __noinline__ double from_totals_any(long long hi, long long lo, int n) {
  if (n > EX_BAD / 2) return __longlong_as_double(0x7FF8000000000000ll);
  return ldexp(fma((double)hi, 0x1p32, (double)lo), n);
}
// Programmatic dependent launch: k_fx64's set-up overlaps the end of k_panel, whose writes
// are visible after the wait.  Not the other way round: blocks of k_panel that arrive
// early settle two on one SM while others idle, and share its FP64 pipe (15.7 ms became
// 23 at n = 5,000).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// digit planes of N = 8 or 4 consecutive K elements of one row, from element N kg on
template <int N>
__device__ __forceinline__ void put_digits(const double (&v)[N], int ex, uint8_t* blk, int row, int kg) {
  const double sc = pow2d(61 - (ex == EX_BAD ? 0 : ex));
  uint32_t lo[N], hi[N];
#pragma unroll
  for (int e = 0; e < N; ++e) {
    const unsigned long long G =
        BIAS + (ex == EX_BAD ? 0ull : (unsigned long long)__double2ll_rn(v[e] * sc));
    lo[e] = (uint32_t)G;
    hi[e] = (uint32_t)(G >> 32);
  }
#pragma unroll
  for (int pl = 0; pl < NPL; ++pl) {
    const int j = 7 - pl;
    uint32_t w[N / 2];
#pragma unroll
    for (int e = 0; e < N / 2; ++e)
      w[e] = j < 4 ? digit_pair(lo[2 * e], lo[2 * e + 1], j) : digit_pair(hi[2 * e], hi[2 * e + 1], j - 4);
    uint8_t* const dst = blk + pl * PLANE_A + cm_off(row, kg * N);
    if constexpr (N == 8) *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
    else *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
  }
}

// ---- products --------------------------------------------------------------
// A segment of output tiles: row tiles [ra, rb) with column tiles [ca, cb), or
// [ca, CPT (rt + 1)) (the lower triangle, CPT = 128 / NT) when tri.
struct Seg {
  int ra, rb, ca, cb, tri, cmin;
  __host__ __device__ int upto(int cpt, int x) const {  // tiles in the row tiles [ra, x)
    return tri ? cpt * (x - ra) * (x + ra + 1) / 2 - ca * (x - ra) : (x - ra) * (cb - ca);
  }
  __host__ __device__ int count(int cpt) const { return rb <= ra || (!tri && cb <= ca) ? 0 : upto(cpt, rb); }
};
struct Job {
  const uint8_t *A, *B;
  const int32_t *ea, *eb;
  int ka, kb;        // K steps per row tile in storage
  int ks0, ks1;      // K steps summed
  int ktri;          // storage and sum start at the row tile's own K step (4 rt)
  Seg seg[2];
  int tiles;
  int mode;          // 0: C -= T; 1: C = T; 2: C = C' = T (lower triangle computed)
  int rmin;          // rows below rmin, columns below the segment's cmin are left alone (mode 0)
  int m, n;          // output bounds (modes 1, 2)
  double* C;
  int64_t ldc;
  // split sum (mode 1): nz slices of kper K steps, slice z writes C + z * cz
  int nz, kper;
  int64_t cz;
  const int* active;  // nothing to do when it points to 0
  int late;           // the kernel before writes nothing read here: wait for it at the end
};
struct Bars {
  uint64_t full[NSTAGE], empty[NSTAGE], acc_full, acc_empty, drain;
  uint32_t tmem;
  int abort;
};

// Tile t: row and column tile, the segment's cmin, and the K steps [k0, k1) it sums.
struct Where {
  int rt, ct, cmin, k0, k1, z;
};
template <int NT>
__device__ __forceinline__ Where tile_of(const Job& J, int t) {
  constexpr int CPT = 128 / NT;
  Where o;
  o.z = 0;
  if (J.nz > 1) {
    const int per = J.tiles / J.nz;
    o.z = t / per;
    t -= o.z * per;
  }
  const int c0 = J.seg[0].count(CPT);
  const Seg& s = t < c0 ? J.seg[0] : J.seg[1];
  if (t >= c0) t -= c0;
  o.cmin = s.cmin;
  int x;
  if (s.tri) {
    // the root of upto(x) = t, then the exact row tile beside it
    const float h = 0.5f * CPT, b = h - s.ca;
    x = (int)((sqrtf(b * b + 4.0f * h * ((float)t + (float)s.ra * (h * (s.ra + 1) - s.ca))) - b) / (2.0f * h));
    x = max(s.ra, min(x, s.rb - 1));
    while (x > s.ra && s.upto(CPT, x) > t) --x;
    while (s.upto(CPT, x + 1) <= t) ++x;
  } else {
    x = s.ra + t / (s.cb - s.ca);
  }
  o.rt = x;
  o.ct = s.ca + t - s.upto(CPT, x);
  o.k0 = J.ktri ? 4 * x : J.ks0 + o.z * J.kper;
  o.k1 = J.nz > 1 ? min(J.ks1, o.k0 + J.kper) : J.ks1;
  return o;
}
// first block of a row tile in a panel's storage (triangular panels keep K steps >= 4 rt)
__device__ __forceinline__ size_t blk_of(int rt, int ks, int stride, int tri) {
  return tri ? (size_t)rt * stride - 2 * (size_t)rt * (rt - 1) + (ks - 4 * rt) : (size_t)rt * stride + ks;
}

// Warp roles: 0 bulk loads, 1 TMEM owner and MMA issuer, 4 and up epilogue (NT / 16 warps
// per TMEM lane quadrant, 16 columns each: wider shares unroll to more code than the
// instruction cache holds, and every launch starts cold).  The epilogue is kept off the two slow
// pipes: totals are read from the floats' bits (an F2I takes four times an add) and become
// doubles in integer instructions; C is read and written in whole sectors through a
// swizzled 32 x 8 staging block per warp.
template <int NT>
__global__ void __launch_bounds__(Tile<NT>::THREADS, 1) k_fx64(const __grid_constant__ Job J, int* status) {
  using T = Tile<NT>;
  if (J.active && *J.active == 0) {
    pdl_wait();
    return;
  }
  extern __shared__ uint8_t dsm_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dsm_raw) + 1023) & ~uintptr_t(1023));
  Bars* bars = reinterpret_cast<Bars*>(smem + T::OFF_BAR);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < NSTAGE; ++i) {
      mbar_init(&bars->full[i], 1);
      mbar_init(&bars->empty[i], 1);
    }
    mbar_init(&bars->acc_full, 1);
    mbar_init(&bars->acc_empty, T::EW);
    mbar_init(&bars->drain, 1);
    bars->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem, 8 * NT);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem;
  volatile int* abort_flag = &bars->abort;
  auto fail = [&]() {
    bars->abort = 1;
    atomicExch(status, DEV_TIMEOUT);
  };
  if (!J.late) pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      uint32_t g = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < J.tiles && ok; t += gridDim.x) {
        const Where o = tile_of<NT>(J, t);
        const int rt = o.rt, ct = o.ct;
        for (int k = o.k0; k < o.k1; ++k, ++g) {
          const uint32_t s = g % NSTAGE;
          if (!mbar_wait(&bars->empty[s], ((g / NSTAGE) & 1) ^ 1, abort_flag)) { ok = false; break; }
          mbar_expect_tx(&bars->full[s], T::STAGE);
          const uint32_t dst = smem_addr(smem + s * T::STAGE);
          bulk_load(dst, J.A + blk_of(rt, k, J.ka, J.ktri) * BLK, BLK, &bars->full[s]);
          const uint8_t* b = J.B + blk_of(ct / (128 / NT), k, J.kb, J.ktri) * BLK + (ct % (128 / NT)) * T::PLANE_B;
#pragma unroll
          for (int pl = 0; pl < NPL; ++pl)
            bulk_load(dst + BLK + pl * T::PLANE_B, b + pl * PLANE_A, T::PLANE_B, &bars->full[s]);
        }
      }
      if (!ok) fail();
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      uint32_t g = 0, c = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < J.tiles && ok; t += gridDim.x) {
        const Where o = tile_of<NT>(J, t);
        for (int k = o.k0; k < o.k1; ++k, ++g) {
          const int ci = (k - o.k0) % CHUNK;
          if (ci == 0) {
            if (!mbar_wait(&bars->acc_empty, (c & 1) ^ 1, abort_flag)) { ok = false; break; }
            tc_fence_after();
          }
          const uint32_t s = g % NSTAGE;
          if (!mbar_wait(&bars->full[s], (g / NSTAGE) & 1, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t op = smem_addr(smem + s * T::STAGE);
#pragma unroll
          for (int kh = 0; kh < 2; ++kh) {
            const uint32_t acc0 = (ci == 0 && kh == 0) ? 0u : 1u;
            const uint32_t bb = op + BLK + kh * 256;
#pragma unroll
            for (int pl = 0; pl < NPL; ++pl) {
              // digit plane pl of A against planes 0 .. 7 - pl of B: classes pl .. 7
              const uint64_t dA = sdesc_noswizzle(op + pl * PLANE_A + kh * 256, 128, 512);
              const int n1 = (NPL - pl) * NT;
              umma_f16(tmem + pl * NT, dA, sdesc_noswizzle(bb, 128, 512), idesc_f16_f32(128, n1 > 256 ? 256 : n1),
                       pl == 0 ? acc0 : 1u);
              if (n1 > 256)
                umma_f16(tmem + pl * NT + 256, dA, sdesc_noswizzle(bb + (256 / NT) * T::PLANE_B, 128, 512),
                         idesc_f16_f32(128, n1 - 256), pl == 0 ? acc0 : 1u);
            }
          }
          umma_commit(&bars->empty[s]);
          if (ci == CHUNK - 1 || k == o.k1 - 1) {
            umma_commit(&bars->acc_full);
            ++c;
          }
        }
      }
      if (!ok) fail();
      umma_commit(&bars->drain);
      const uint64_t t0 = global_ns();
      while (!mbar_try(&bars->drain, 0) && global_ns() - t0 < kWaitLimitNs) {}
    }
    __syncwarp();
  } else if (warp >= 4) {
    constexpr int MAGIC = 0x4B400000;  // bits of 1.5 2^23: those of 1.5 2^23 + v are MAGIC + v, |v| <= 2^22
    const int q = warp & 3, j0 = ((warp - 4) >> 2) * 16;
    uint8_t* out = smem + T::OFF_OUT + (warp - 4) * 2048;
    uint32_t c = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < J.tiles && ok; t += gridDim.x) {
      const Where o = tile_of<NT>(J, t);
      const int rt = o.rt, ct = o.ct, cmin = o.cmin;
      const int nch = (o.k1 - o.k0 + CHUNK - 1) / CHUNK;
      double* const C = J.C + o.z * J.cz;
      const int rb = rt * 128 + q * 32, row = rb + lane, col0 = ct * NT + j0;
      const int ea = J.ea[row] - 66;  // 56 - 2 * 61
      const int el = J.eb[col0 + (lane & 15)];
      // modulo 2^64: the offsets' sum leaves the range of an int64 from 432 chunks on
      unsigned long long hi[16], lo[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) hi[j] = lo[j] = 0ull - (unsigned long long)MAGIC * 0x01010101ull * (unsigned)nch;
      for (int ch = 0; ch < nch; ++ch, ++c) {
        if (!mbar_wait_idle(&bars->acc_full, c & 1, abort_flag, 20)) { ok = false; break; }
        tc_fence_after();
        const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + j0;
        float big = 0.0f;
#pragma unroll
        for (int u = 0; u < NPL; ++u) {
          uint32_t r[16];
          tmem_ld16(ta + u * NT, r);
          tmem_ld_wait();
          const int mul = 1 << ((3 - (u & 3)) * 8);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float f = __uint_as_float(r[j]);
            big = fmaxf(big, fabsf(f));
            const long long v = (long long)__float_as_int(__fadd_rn(f, 12582912.0f)) * mul;
            if (u < 4) hi[j] += (unsigned long long)v;
            else lo[j] += (unsigned long long)v;
          }
        }
        // sums past 2^22 (possible over more than 32 K elements, and rare) do not fit the bits
        // trick: replace its value by the F2I's
        if (__any_sync(~0u, big > 4194304.0f)) {
#pragma unroll
          for (int u = 0; u < NPL; ++u) {
            uint32_t r[16];
            tmem_ld16(ta + u * NT, r);
            tmem_ld_wait();
            const int mul = 1 << ((3 - (u & 3)) * 8);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const float f = __uint_as_float(r[j]);
              const long long v =
                  (long long)(__float2int_rn(f) + MAGIC - __float_as_int(__fadd_rn(f, 12582912.0f))) * mul;
              if (u < 4) hi[j] += (unsigned long long)v;
              else lo[j] += (unsigned long long)v;
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->acc_empty);
      }
      if (!ok) break;
      // usual exponents take the branch-free conversion
      const bool usual = !__any_sync(~0u, ea + 66 < -400 || ea + 66 > 400 || el < -400 || el > 400);
      const int chunk = lane & 3;
#pragma unroll
      for (int h = 0; h < 16; h += 8) {
        const int cb = col0 + h;
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
          double2 x;
          const int e0 = ea + __shfl_sync(~0u, el, h + j), e1 = ea + __shfl_sync(~0u, el, h + j + 1);
          if (usual) {
            x.x = __longlong_as_double((long long)from_totals((long long)hi[h + j], (long long)lo[h + j], e0));
            x.y = __longlong_as_double((long long)from_totals((long long)hi[h + j + 1], (long long)lo[h + j + 1], e1));
          } else {
            x.x = from_totals_any((long long)hi[h + j], (long long)lo[h + j], e0);
            x.y = from_totals_any((long long)hi[h + j + 1], (long long)lo[h + j + 1], e1);
          }
          *reinterpret_cast<double2*>(out + lane * 64 + (((j >> 1) ^ ((lane >> 1) & 3)) << 4)) = x;
          if (J.mode == 2 && row < J.m) {
            if (cb + j <= row) J.C[(int64_t)(cb + j) * J.ldc + row] = x.x;
            if (cb + j + 1 <= row) J.C[(int64_t)(cb + j + 1) * J.ldc + row] = x.y;
          }
        }
        __syncwarp();
        if (J.mode == 0) {
          double2 o[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int r = rb + 8 * i + (lane >> 2);
            if (r >= J.rmin && cb >= cmin)
              o[i] = *reinterpret_cast<const double2*>(J.C + (int64_t)r * J.ldc + cb + 2 * chunk);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int rl = 8 * i + (lane >> 2);
            const double2 x = *reinterpret_cast<const double2*>(out + rl * 64 + ((chunk ^ ((rl >> 1) & 3)) << 4));
            if (rb + rl >= J.rmin && cb >= cmin) {
              o[i].x -= x.x;
              o[i].y -= x.y;
              *reinterpret_cast<double2*>(J.C + (int64_t)(rb + rl) * J.ldc + cb + 2 * chunk) = o[i];
            }
          }
        } else {
          const int col = lane & 7, cc = cb + col;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int rl = 4 * i + (lane >> 3), r = rb + rl;
            const double x =
                *reinterpret_cast<const double*>(out + rl * 64 + (((col >> 1) ^ ((rl >> 1) & 3)) << 4) + (col & 1) * 8);
            if (r < J.m && cc < J.n && (J.mode == 1 || cc <= r)) C[(int64_t)r * J.ldc + cc] = x;
          }
        }
      }
    }
    if (!ok) fail();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem, 8 * NT);
  if (J.late) pdl_wait();
}

// ---- digits of a matrix ------------------------------------------------------
// ex[r]: exponent of the largest magnitude of row r (rows past `rows` are zero).
// One warp per row; trans: one thread per row, K over blockDim.y.
__global__ void __launch_bounds__(256) k_rowexp(const double* __restrict__ src, int64_t ld, int64_t rows, int64_t k,
                                                int32_t* __restrict__ ex) {
  const int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  int e = EX_MIN;
  if (r < rows)
    for (int64_t j = threadIdx.x & 31; j < k; j += 32) {
      const double v = src[r * ld + j];
      if (v != 0.0) e = max(e, expo(v));
    }
  for (int o = 16; o; o >>= 1) e = max(e, __shfl_xor_sync(~0u, e, o));
  if ((threadIdx.x & 31) == 0) ex[r] = e;
}
__global__ void __launch_bounds__(256) k_rowexp_t(const double* __restrict__ src, int64_t ld, int64_t rows, int64_t k,
                                                  int32_t* __restrict__ ex) {
  __shared__ int red[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t r = (int64_t)blockIdx.x * 32 + lane;
  int e = EX_MIN;
  if (r < rows)
    for (int64_t j = w; j < k; j += 8) {
      const double v = src[j * ld + r];
      if (v != 0.0) e = max(e, expo(v));
    }
  red[w][lane] = e;
  __syncthreads();
  if (w == 0) {
    for (int i = 1; i < 8; ++i) e = max(e, red[i][lane]);
    ex[r] = e;
  }
}
// blocks (row tile, K step): thread = row, 8 K elements at a time
__global__ void __launch_bounds__(128) k_digits(const double* __restrict__ src, int64_t ld, int64_t rows, int64_t k,
                                                int trans, int ks, const int32_t* __restrict__ ex,
                                                uint8_t* __restrict__ dig) {
  const int64_t r = (int64_t)blockIdx.x * 128 + threadIdx.x;
  const int64_t k0 = (int64_t)blockIdx.y * 32;
  uint8_t* blk = dig + ((size_t)blockIdx.x * ks + blockIdx.y) * BLK;
  const int e = ex[r];
#pragma unroll
  for (int kg = 0; kg < 4; ++kg) {
    double v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int64_t kk = k0 + kg * 8 + i;
      v[i] = (r < rows && kk < k) ? (trans ? src[kk * ld + r] : src[r * ld + kk]) : 0.0;
    }
    put_digits(v, e, blk, threadIdx.x, kg);
  }
}

// Columns of an interleaved block as rows of an operand: element (c, k) is
// X[(p + gmap[k]) * xs + c].  Exponents (columns from ncols on are zero), then digits.
__global__ void __launch_bounds__(256) k_colexp(const double* __restrict__ X, int xs, int64_t p,
                                                const int32_t* __restrict__ gmap, int64_t ng, int ncols,
                                                int32_t* __restrict__ ex, const int* active) {
  if (active && *active == 0) return;
  __shared__ int red[8];
  const int c = blockIdx.x;
  int e = EX_MIN;
  if (c < ncols)
    for (int64_t k = threadIdx.x; k < ng; k += 256) {
      const double v = X[(p + gmap[k]) * xs + c];
      if (v != 0.0) e = max(e, expo(v));
    }
  e = __reduce_max_sync(~0u, e);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; ++i) e = max(e, red[i]);
    ex[c] = e;
  }
}
__global__ void __launch_bounds__(128) k_coldigits(const double* __restrict__ X, int xs, int64_t p,
                                                   const int32_t* __restrict__ gmap, int64_t ng, int ncols, int ks,
                                                   const int32_t* __restrict__ ex, uint8_t* __restrict__ dig,
                                                   const int* active) {
  if (active && *active == 0) return;
  const int64_t total = (int64_t)ks * ncols * 4;
  for (int64_t i = blockIdx.x * 128ll + threadIdx.x; i < total; i += gridDim.x * 128ll) {
    const int c = (int)(i % ncols), kg = (int)(i / ncols & 3);
    const int64_t st = i / (4 * ncols);
    double v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int64_t k = st * 32 + kg * 8 + j;
      v[j] = k < ng ? X[(p + gmap[k]) * xs + c] : 0.0;
    }
    put_digits(v, ex[c], dig + (size_t)st * BLK, c, kg);
  }
}
// out[i * os + c] = the slices' sum in slice order for c < ncols, 0 for ncols <= c < oc
__global__ void __launch_bounds__(256) k_slices(const double* __restrict__ part, int nz, int64_t cz, int ldp, int64_t ng,
                                                int ncols, double* __restrict__ out, int os, int oc,
                                                const int* active) {
  if (active && *active == 0) return;
  const int64_t total = ng * oc;
  for (int64_t i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll) {
    const int64_t r = i / oc;
    const int c = (int)(i - r * oc);
    double s = 0.0;
    if (c < ncols)
      for (int z = 0; z < nz; ++z) s += part[z * cz + r * ldp + c];
    out[r * os + c] = s;
  }
}

// ---- Cholesky ------------------------------------------------------------------
// The factorization runs on D A D, D_ii = 2^-k_i with 4^k_i <= A_ii < 4^(k_i + 1): its entries
// are below 4, so that no 2 x 2 determinant over- or underflows, and the scaling is exact.
__global__ void k_scales(const double* __restrict__ A, int64_t n, int64_t np, FxAdd add, int32_t* __restrict__ sc) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= np) return;
  const double v = i < n ? A[i * n + i] + add.diag + add.all : 1.0;
  sc[i] = v > 0.0 && isfinite(v) ? ilogb(v) >> 1 : 0;
}
// W (np x np row-major) = lower triangle of D A D (A column-major), identity on the padding
__global__ void __launch_bounds__(256) k_load_lower(const double* __restrict__ A, int64_t n, int64_t np, FxAdd add,
                                                    const int32_t* __restrict__ sc, double* __restrict__ W) {
  __shared__ double t[32][33];
  const int64_t i0 = (int64_t)blockIdx.x * 32, j0 = (int64_t)blockIdx.y * 32;
  if (j0 > i0) return;
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  for (int c = y; c < 32; c += 8) {
    const int64_t i = i0 + x, j = j0 + c;
    t[c][x] = (i < n && j < n)
                  ? (A[j * n + i] + (i == j ? add.diag : 0.0) + add.all) * pow2d(max(-1022, min(1023, -sc[i] - sc[j])))
                  : (i == j ? 1.0 : 0.0);
  }
  __syncthreads();
  for (int r = y; r < 32; r += 8) W[(i0 + r) * np + j0 + x] = t[x][r];
}

struct Panel {
  double* W;
  int64_t np;
  int k0, K0, K1, B;
  int inverse;
  uint8_t* dig;       // inner digits (K = 32)
  int32_t* ex;        // their exponents
  int32_t* exo;       // exponents of the outer panel's rows, so far
  int32_t* exm;       // exponents of the columns of M, so far
  double* P;          // L of the outer panel (np x B)
  double* D;          // diagonal blocks of M (or L), np x 32: other CTAs still read the pivot block in W
  double* piv;
  int* bad;
};

// One 32-wide step.  Every CTA factors the pivot block (it is small, and a separate
// launch would cost more than the repeat), then takes 16-row groups: x L_kk' = v with v
// the row's 32 entries in the pivot columns (rows below the pivot), the column's
// entries in the pivot rows (columns left of it), or a unit vector (the pivot rows, whose x
// are the columns of X = L_kk^-1).
//
// A chain of FP64 latencies bounds it: a dependent multiply-add takes 68 clocks, a reciprocal
// 230, a publish and barrier 120, and one warp-wide FP64 instruction holds its
// quarter of the SM's FP64 pipe for 64.  Hence 2 x 2 pivots (one reciprocal and one
// barrier for two columns), the next pivot's rows and its publication ahead of the other
// rows of a step, no square root inside the chain, and groups of 16 rows, which put a
// problem of 2,000 rows on 128 SMs.
//
// A pivot pair is applied as L D L', never by its explicit inverse: with l = p12 / p11, the
// second row less l times the first (w) is eliminated by p2 = p22 - l p12.  The inverse's
// two terms cancel to the same small difference, but each is rounded at the size of p12 / p2
// first, and the condition of the pair enters twice.  The groups' rows are forward
// substitutions by the same pairs and not products with X, which lose the root of L_kk's
// condition where two adjacent rows are near-duplicates.  Measured with the pair's inverse
// and X before, both this way now (panels of 128): factor at n = 2,000 2.59 ms, now 2.47, inverse 2.81 both; at
// 8,000 18.3, now 18.1, and 34.4, now 34.8 (a substitution issues 92 FP64 instructions a warp and group,
// the product 80; the digits took 16 on half of the lanes, now 8).  L L' - A at n = 96 with adjacent
// rows 1e-3 apart: 0.01 of 4 n u sqrt(A_ii A_jj), 1e5 times it before, when rows 1e-4 apart were
// found not positive definite.
__global__ void __launch_bounds__(128) k_panel(const __grid_constant__ Panel a) {
  __shared__ double X[32][33], V[4][32][5], pa[16][32], pb[16][32], ra[16][32], rw[16][32];
  __shared__ double pv[32], lp[16], i1[16], l2[16], i2[16];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int64_t np = a.np;
  const double* Wk = a.W + (int64_t)a.k0 * np + a.k0;
  // lane = column; registers 2 s, 2 s + 1 = rows 2 (w + 4 s), 2 (w + 4 s) + 1
  double d[8];
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const int r = 2 * (w + 4 * (t >> 1)) + (t & 1);
    d[t] = lane <= r ? Wk[r * np + lane] : Wk[lane * np + r];
  }
  // groups of 16 rows: a warp takes four, eight lanes a row, columns c + 8 m.  The first
  // group's entries are in flight during the factorization
  const int c = lane & 7, row = 4 * w + (lane >> 3);
  const int gk = a.k0 / 16, ng = (int)(np / 16);
  int g = (a.inverse ? 0 : gk) + blockIdx.x;
  double pre[4] = {0.0, 0.0, 0.0, 0.0};
  auto fetch = [&](int gg) {
    if (gg == gk || gg == gk + 1) return;  // the pivot rows: from X
    const int r = gg * 16 + row;
#pragma unroll
    for (int m = 0; m < 4; ++m)
      pre[m] = gg > gk ? a.W[(int64_t)r * np + a.k0 + c + 8 * m] : a.W[(int64_t)(a.k0 + c + 8 * m) * np + r];
  };
  if (g < ng) fetch(g);
  // rows 2 j, 2 j + 1 (registers 2 s, 2 s + 1 of warp j & 3): the first (ra), the second less
  // l times it (rw), and both over their pivots (pa, pb); their own columns take those of
  // the pair's inverse
  auto publish = [&](int j, double& da, double& db) {
    const int k = 2 * j;
    const double p11 = __shfl_sync(~0u, da, k), p12 = __shfl_sync(~0u, da, k + 1), p22 = __shfl_sync(~0u, db, k + 1);
    const double det = fma(p11, p22, -p12 * p12);
    // both reciprocals in one pass of the chain, half a warp each
    const double rcp = reciprocal(lane < 16 ? p11 : det);
    const double r1 = __shfl_sync(~0u, rcp, 0), r2 = p11 * __shfl_sync(~0u, rcp, 16);  // 1 / p2 = p11 / det
    const double l = p12 * r1;
    da = lane == k ? 1.0 : lane == k + 1 ? 0.0 : da;
    db = lane == k ? 0.0 : lane == k + 1 ? 1.0 : db;
    const double wb = fma(-l, da, db);
    ra[j][lane] = da;
    rw[j][lane] = wb;
    pa[j][lane] = da * r1;
    pb[j][lane] = wb * r2;
    if (lane == 0) {
      pv[k] = p11;
      pv[k + 1] = det;  // over p11 below
      lp[j] = l;
      l2[j] = p12;
    }
    __syncwarp();  // this warp does not wait at the barrier it arrives at
    asm volatile("bar.arrive %0, 128;" ::"r"(1 + (j & 7)) : "memory");
  };
  if (w == 0) publish(0, d[0], d[1]);
#pragma unroll
  for (int ss = 0; ss < 4; ++ss) {
#pragma unroll 1
    for (int ww = 0; ww < 4; ++ww) {
      const int j = 4 * ss + ww;
      if (w != ww) asm volatile("bar.sync %0, 128;" ::"r"(1 + (j & 7)) : "memory");
      const double qa = pa[j][lane], qb = pb[j][lane];
      const bool piv = (lane >> 1) == j;
      // a row's entries in the pivot columns are the pivot rows' in its own (symmetry)
      auto update = [&](int t) {
        const int r = 2 * (w + 4 * (t >> 1)) + (t & 1);
        d[t] = fma(-rw[j][r], qb, fma(-ra[j][r], qa, piv ? 0.0 : d[t]));
      };
      // the next pivot's rows first, and their pivot, before the other rows
      if (w > ww) {
        update(2 * ss);
        update(2 * ss + 1);
        if (w == ww + 1) publish(j + 1, d[2 * ss], d[2 * ss + 1]);
      }
      if (ss < 3) {
        update(2 * ss + 2);
        update(2 * ss + 3);
        if (ww == 3 && w == 0) publish(j + 1, d[2 * ss + 2], d[2 * ss + 3]);
      }
#pragma unroll
      for (int t = 2 * ss + 4; t < 8; ++t) update(t);
    }
  }
  __syncthreads();
  // 2 x 2 Cholesky factors of the pivots: [1 / i1, 0; l2, 1 / i2]
  if (tid < 16) {
    const double p11 = pv[2 * tid], r1 = rsqrt(p11), p2 = pv[2 * tid + 1] * r1 * r1;
    i1[tid] = r1;
    l2[tid] *= r1;
    i2[tid] = rsqrt(p2);
    pv[2 * tid + 1] = p2;
    if (blockIdx.x == 0) {
      a.piv[a.k0 + 2 * tid] = p11;
      a.piv[a.k0 + 2 * tid + 1] = p2;
      if (!(p11 > 0.0) || !(p2 > 0.0) || !isfinite(p11) || !isfinite(p2)) atomicExch(a.bad, 1);
    }
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < 8; t += 2) {
    const int j = w + 2 * t, r = 2 * j;
    const double x0 = lane <= r ? d[t] * i1[j] : 0.0;
    X[r][lane] = x0;
    X[r + 1][lane] = lane <= r + 1 ? fma(-l2[j], x0, d[t + 1]) * i2[j] : 0.0;
  }
  __syncthreads();
  pdl_launch();
  for (; g < ng; g += gridDim.x) {
    const int r = g * 16 + row;
    const bool below = g > gk + 1, left = g < gk;
    double x[4];
    if (below || left) {
      // x L_kk' = v by forward substitution, a pivot pair at a time
#pragma unroll
      for (int m = 0; m < 4; ++m) x[m] = pre[m];
      if (g + (int)gridDim.x < ng) fetch(g + gridDim.x);
#pragma unroll
      for (int ss = 0; ss < 4; ++ss) {
#pragma unroll 1
        for (int ww = 0; ww < 4; ++ww) {
          const int j = 4 * ss + ww, src = (lane & 24) + 2 * ww;
          const double f1 = __shfl_sync(~0u, x[ss], src), f2 = __shfl_sync(~0u, x[ss], src + 1);
          const double f = fma(-lp[j], f1, f2);
          if (ww < 3) {
            const double t = fma(-f, pb[j][c + 8 * ss], fma(-f1, pa[j][c + 8 * ss], x[ss]));
            x[ss] = c > 2 * ww + 1 ? t : x[ss];
          }
          if (c == 2 * ww + 1) x[ss] = f;
#pragma unroll
          for (int m = ss + 1; m < 4; ++m) x[m] = fma(-f, pb[j][c + 8 * m], fma(-f1, pa[j][c + 8 * m], x[m]));
        }
      }
#pragma unroll
      for (int m = 0; m < 4; ++m) x[m] *= (c & 1) ? i2[(c >> 1) + 4 * m] : i1[(c >> 1) + 4 * m];
    } else {
#pragma unroll
      for (int m = 0; m < 4; ++m) x[m] = X[c + 8 * m][r - a.k0];
      if (g + (int)gridDim.x < ng) fetch(g + gridDim.x);
    }
    int e = EX_MIN;
    __syncwarp();  // V's last readers
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      V[w][c + 8 * m][lane >> 3] = x[m];
      if (x[m] != 0.0) e = max(e, expo(x[m]));
      if (below) {
        a.P[(int64_t)r * a.B + (a.k0 - a.K0) + c + 8 * m] = x[m];
        a.W[(int64_t)r * np + a.k0 + c + 8 * m] = a.inverse ? 0.0 : x[m];
      } else if (left) {
        a.W[(int64_t)(a.k0 + c + 8 * m) * np + r] = x[m];
      }
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) e = max(e, __shfl_xor_sync(~0u, e, o));
    if (c == 0) {
      a.ex[r] = e;
      a.exo[r] = (a.k0 == a.K0 || !(below || left)) ? e : max(e, a.exo[r]);
      if (a.inverse && !below) a.exm[r] = left ? max(e, a.exm[r]) : e;
    }
    __syncwarp();
    double v4[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v4[i] = V[w][c * 4 + i][lane >> 3];
    put_digits(v4, e, a.dig + (size_t)(r / 128) * BLK, r & 127, c);
    if (!below && !left) {
      for (int i = 0; i < 4; ++i) {
        const int l = g * 16 + 4 * w + i - a.k0, j = lane >> 1;
        double y = X[l][lane];
        if (!a.inverse) {
          if ((l >> 1) == j) y = (l & 1) == 0 ? pv[l] * i1[j] : (lane & 1) ? pv[l] * i2[j] : l2[j];
          else if (lane < l) y = (lane & 1) ? rw[j][l] * i2[j] : ra[j][l] * i1[j];
        }
        a.D[(a.k0 + l) * 32 + lane] = lane <= l ? y : 0.0;
      }
    }
  }
}

// element (i, j), i >= j, of the finished triangle
__device__ __forceinline__ double lower(const double* W, const double* D, int64_t np, int64_t i, int64_t j) {
  return (i >> 5) == (j >> 5) ? D[i * 32 + (j & 31)] : W[i * np + j];
}

// Digits of the outer panel: rows below it from P, columns left of its end (rows of
// M') from W.  Blocks (row tile, K step of the panel).
__global__ void __launch_bounds__(128) k_panel_digits(const __grid_constant__ Panel a, uint8_t* __restrict__ dig,
                                                      int rt0) {
  const int rt = rt0 + blockIdx.x, r = rt * 128 + threadIdx.x, kb = blockIdx.y * 32;
  uint8_t* blk = dig + ((size_t)rt * (a.B / 32) + blockIdx.y) * BLK;
  const int e = a.exo[r];
#pragma unroll
  for (int kg = 0; kg < 4; ++kg) {
    double v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int k = kb + kg * 8 + i;
      if (r >= a.K1) v[i] = a.K0 + k < a.K1 ? a.P[(int64_t)r * a.B + k] : 0.0;
      else v[i] = a.K0 + k < r ? 0.0 : lower(a.W, a.D, a.np, a.K0 + k, r);
    }
    put_digits(v, e, blk, threadIdx.x, kg);
  }
}
// Digits of M' (row j = column j of M = L^-1): all row tiles, each from its own K step on
// (group 0), or `group` row tiles from rt0 on, all of K step ks0 on (zeros left of the diagonal)
__global__ void __launch_bounds__(128) k_minv_digits(const double* __restrict__ W, const double* __restrict__ D, int64_t np,
                                                     int n, int ks, int rt0, int ks0, int group,
                                                     const int32_t* __restrict__ ex, const int32_t* __restrict__ sc,
                                                     int32_t* __restrict__ exd, uint8_t* __restrict__ dig) {
  const int rt = rt0 + blockIdx.x, k0 = ks0 + blockIdx.y;
  if (!group && k0 < 4 * rt) return;
  const int r = rt * 128 + threadIdx.x;
  // A^-1 = D (M'M) D: the scaling goes into the product's exponents
  if (k0 == 4 * rt) exd[r] = r < n ? ex[r] - sc[r] : EX_MIN;
  uint8_t* blk = dig + (group ? (size_t)blockIdx.x * (ks - ks0) + blockIdx.y : blk_of(rt, k0, ks, 1)) * BLK;
  const int e = r < n ? ex[r] : EX_MIN;
#pragma unroll
  for (int kg = 0; kg < 4; ++kg) {
    double v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int k = k0 * 32 + kg * 8 + i;
      v[i] = (k >= r && k < n && r < n) ? lower(W, D, np, k, r) : 0.0;
    }
    put_digits(v, e, blk, threadIdx.x, kg);
  }
}
// sum of log pivots of A, in a fixed order
__global__ void __launch_bounds__(256) k_logsum(const double* __restrict__ piv, const int32_t* __restrict__ sc, int n,
                                                double* __restrict__ out) {
  __shared__ double red[256];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += 256) s += log(piv[i]) + sc[i] * (2.0 * 0.69314718055994530942);
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = red[0];
}
// U = L' (column-major upper = row-major lower), zeros elsewhere
__global__ void k_store_factor(const double* __restrict__ W, const double* __restrict__ D, int64_t np, int64_t n,
                               const int32_t* __restrict__ sc, double* __restrict__ out) {
  const int64_t total = n * n;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / n, c = i % n;
    out[i] = c <= r ? lower(W, D, np, r, c) * pow2d(sc[r]) : 0.0;
  }
}

// Scratch of the factorizations, kept by the handle between calls of up to
// kKeepBytes (a GBLUP of a few thousand animals); larger ones are freed on return,
// where an allocation costs little beside the work.
constexpr size_t kKeepBytes = (size_t)1 << 30;
struct Scratch {
  DevBuf<double> W, P, D, piv;
  DevBuf<uint8_t> din, dout, dm, dm2;
  DevBuf<int32_t> ex, exo, exm, sc;
  DevBuf<int> bad;
  size_t bytes() const { return W.n * 8 + P.n * 8 + din.n + dout.n + dm.n + dm2.n; }
};
template <typename T>
static void at_least(DevBuf<T>& b, size_t n) {
  if (b.n < n) b.resize(n);
}
// at_least for digits, or false where they do not fit
static bool try_at_least(cbx_handle* h, DevBuf<uint8_t>& b, size_t n) {
  if (h->fx_limit && n > h->fx_limit) return false;
  return b.n >= n || b.try_resize(n);
}
// Row tiles of a group, where digits go by groups: 16 (2,048 rows, 512 output tiles of 64 columns a pair of
// groups, 3.4 waves), fewer under a limit
static int group_tiles(cbx_handle* h, int rt, int ks) {
  const size_t row = (size_t)ks * BLK;
  return (int)std::min<size_t>(rt, h->fx_limit ? std::max<size_t>(1, std::min<size_t>(16, h->fx_limit / row)) : 16);
}
static Scratch& scratch(cbx_handle* h) {
  if (!h->fx_slot) h->fx_slot = std::make_shared<Scratch>();
  return *static_cast<Scratch*>(h->fx_slot.get());
}

template <typename K, typename... A>
static void launch_pdl(cbx_handle* h, K kern, dim3 grid, int threads, int smem, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = h->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  CBX_CUDA(cudaLaunchKernelEx(&cfg, kern, args...));
}
// Segments count 32-column tiles; pairs of them make the 64-wide ones.  A 32-wide tile costs
// about 0.6 of a 64-wide one (the same A digits for half the columns): narrow tiles where
// they fill SMs that wide ones leave idle in the last wave.
template <int NT>
static void launch_tiles(cbx_handle* h, Job J) {
  for (Seg& s : J.seg) {
    s.ca /= NT / 32;
    s.cb = (s.cb + NT / 32 - 1) / (NT / 32);
  }
  J.tiles = (J.seg[0].count(128 / NT) + J.seg[1].count(128 / NT)) * std::max(1, J.nz);
  ensure_smem((const void*)k_fx64<NT>, Tile<NT>::SMEM, h->device);
  launch_pdl(h, k_fx64<NT>, dim3(std::min(J.tiles, h->num_sms)), Tile<NT>::THREADS, Tile<NT>::SMEM, J, h->status.p);
  h->launched("k_fx64");
}
static void launch(cbx_handle* h, const Job& J) {
  const int64_t t32 = (int64_t)J.seg[0].count(4) + J.seg[1].count(4), sms = h->num_sms;
  if (t32 <= 0 || J.ks1 <= 0) return;
  if (6 * ((t32 + sms - 1) / sms) < 10 * ((t32 / 2 + sms - 1) / sms)) launch_tiles<32>(h, J);
  else launch_tiles<64>(h, J);
}

__global__ void k_selftest_totals(const int64_t* __restrict__ hi, const int64_t* __restrict__ lo,
                                  const int32_t* __restrict__ e, int64_t n, double* __restrict__ y) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    y[i] = __longlong_as_double((long long)from_totals(hi[i], lo[i], e[i]));
}

}  // namespace fx

void fx64_selftest_totals(cbx_handle* h, const int64_t* hi, const int64_t* lo, const int32_t* e, int64_t n, double* y) {
  fx::k_selftest_totals<<<128, 256, 0, h->stream>>>(hi, lo, e, n, y);
}

static size_t panel_bytes(int64_t rows, int64_t k) {
  CBX_REQUIRE(rows > 0 && k > 0 && rows < (1 << 24) && k < (1 << 24), CBX_ERR_ARG, "bad operand shape");
  return (size_t)((rows + 127) / 128) * ((k + 31) / 32) * fx::BLK;
}

void fx64_digits(cbx_handle* h, FxPanel& P, const double* src, int64_t ld, int64_t rows, int64_t k, bool trans) {
  fx::at_least(P.dig, panel_bytes(rows, k));
  P.rt = (int)((rows + 127) / 128);
  P.ks = (int)((k + 31) / 32);
  fx::at_least(P.ex, (size_t)P.rt * 128);
  cudaStream_t s = h->stream;
  if (trans) fx::k_rowexp_t<<<P.rt * 4, 256, 0, s>>>(src, ld, rows, k, P.ex.p);
  else fx::k_rowexp<<<P.rt * 16, 256, 0, s>>>(src, ld, rows, k, P.ex.p);
  h->launched("k_rowexp");
  for (int y = 0; y < P.ks; y += 65535) {  // grid.y limit
    const int cnt = std::min(65535, P.ks - y);
    fx::k_digits<<<dim3(P.rt, cnt), 128, 0, s>>>(src + (trans ? (int64_t)y * 32 * ld : (int64_t)y * 32), ld, rows,
                                                 k - (int64_t)y * 32, trans, P.ks, P.ex.p,
                                                 P.dig.p + (size_t)y * fx::BLK);
    h->launched("k_digits");
  }
}

bool fx64_try_digits(cbx_handle* h, FxPanel& P, const double* src, int64_t ld, int64_t rows, int64_t k) {
  if (!fx::try_at_least(h, P.dig, panel_bytes(rows, k))) return false;
  fx64_digits(h, P, src, ld, rows, k, false);
  return true;
}

void fx64_gemm(cbx_handle* h, const FxPanel& A, const FxPanel& B, int64_t m, int64_t n, double* C, int64_t ldc) {
  CBX_REQUIRE(A.ks == B.ks && m <= (int64_t)A.rt * 128 && n <= (int64_t)B.rt * 128, CBX_ERR_ARG, "operand shapes differ");
  fx::Job J{};
  J.A = A.dig.p;
  J.B = B.dig.p;
  J.ea = A.ex.p;
  J.eb = B.ex.p;
  J.ka = J.kb = J.ks1 = A.ks;
  J.seg[0] = {0, A.rt, 0, (int)((n + 31) / 32), 0, 0};
  J.mode = 1;
  J.m = (int)m;
  J.n = (int)n;
  J.C = C;
  J.ldc = ldc;
  fx::launch(h, J);
}

bool fx64_matmul(cbx_handle* h, const double* A, FxPanel& Ad, const double* B, FxPanel& Bd, bool has_b, int64_t n,
                 double* C) {
  if ((has_b || fx64_try_digits(h, Bd, B, n, n, n)) && fx64_try_digits(h, Ad, A, n, n, n)) {
    fx64_gemm(h, Ad, Bd, n, n, C, n);
    return true;
  }
  Ad = FxPanel{};
  Bd = FxPanel{};
  const int64_t rows = 128ll * fx::group_tiles(h, (int)((n + 127) / 128), (int)((n + 31) / 32));
  for (int64_t i = 0; i < n; i += rows) {
    const int64_t mi = std::min(rows, n - i);
    fx64_digits(h, Ad, A + i * n, n, mi, n, false);
    for (int64_t j = 0; j < n; j += rows) {
      const int64_t mj = std::min(rows, n - j);
      fx64_digits(h, Bd, B + j * n, n, mj, n, false);
      fx64_gemm(h, Ad, Bd, mi, mj, C + i * n + j, n);
    }
  }
  return false;
}

void fx64_product(cbx_handle* h, const FxPanel& Q, FxPanel& V, DevBuf<double>& part, const double* X, int xs, int64_t p,
                  const int32_t* gmap, int64_t ng, int ncols, double* out, int os, int oc, const int* active,
                  const std::function<bool()>& before) {
  CBX_REQUIRE(ncols >= 1 && ncols <= 64 && ng <= (int64_t)Q.rt * 128, CBX_ERR_ARG, "bad block product");
  cudaStream_t s = h->stream;
  const int nt = ncols <= 32 ? 32 : 64;
  if (V.dig.n < (size_t)Q.ks * fx::BLK) {  // rows past the columns hold finite digits
    V.dig.resize((size_t)Q.ks * fx::BLK);
    V.dig.zero(s);
  }
  fx::at_least(V.ex, 128);
  V.rt = 1;
  V.ks = Q.ks;
  fx::k_colexp<<<nt, 256, 0, s>>>(X, xs, p, gmap, ng, ncols, V.ex.p, active);
  h->launched("k_colexp");
  const int64_t work = (int64_t)Q.ks * ncols * 4;
  fx::k_coldigits<<<(unsigned)std::min<int64_t>((work + 127) / 128, 8 * h->num_sms), 128, 0, s>>>(
      X, xs, p, gmap, ng, ncols, Q.ks, V.ex.p, V.dig.p, active);
  h->launched("k_coldigits");
  // K slices: as many as leave the last wave of row tiles x slices fullest, 8 K steps or more each
  int nz = 1;
  double best = 1e30;
  for (int z = 1; z <= 32 && 8 * z <= std::max(8, Q.ks); ++z) {
    const int64_t waves = ((int64_t)Q.rt * z + h->num_sms - 1) / h->num_sms;
    const double cost = (double)waves / z + 0.01 * z;
    if (cost < best) {
      best = cost;
      nz = z;
    }
  }
  fx::Job J{};
  J.kper = ((Q.ks + nz - 1) / nz + 3) / 4 * 4;
  J.nz = (Q.ks + J.kper - 1) / J.kper;
  J.cz = (int64_t)ng * nt;
  fx::at_least(part, (size_t)J.nz * J.cz);
  J.A = Q.dig.p;
  J.B = V.dig.p;
  J.ea = Q.ex.p;
  J.eb = V.ex.p;
  J.ka = J.kb = J.ks1 = Q.ks;
  J.seg[0] = {0, Q.rt, 0, nt / 32, 0, 0};
  J.mode = 1;
  J.m = (int)ng;
  J.n = ncols;
  J.C = part.p;
  J.ldc = nt;
  J.active = active;
  if (before) J.late = before() ? 1 : 0;
  if (nt == 32) fx::launch_tiles<32>(h, J);
  else fx::launch_tiles<64>(h, J);
  fx::k_slices<<<(unsigned)std::min<int64_t>((ng * oc + 255) / 256, 8 * h->num_sms), 256, 0, s>>>(
      part.p, J.nz, J.cz, nt, ng, ncols, out, os, oc, active);
  h->launched("k_slices");
}

// out = M'M by pairs of row groups: the digits of two groups at a time, from the first group's
// first K step on.  Every total is the same integer as with all digits at once.
static void minv_product_groups(cbx_handle* h, fx::Scratch& S, int64_t np, int64_t n, double* out) {
  cudaStream_t s = h->stream;
  const int rt = (int)(np / 128), ks = (int)(np / 32), gt = fx::group_tiles(h, rt, ks);
  const size_t most = (size_t)gt * ks * fx::BLK;
  S.dm.release();
  S.dm2.release();
  S.dm.resize(most);
  if (gt < rt) S.dm2.resize(most);
  for (int ra = 0; ra < rt; ra += gt) {
    const int na = std::min(gt, rt - ra), ks0 = 4 * ra;
    auto digits = [&](int r0, int cnt, uint8_t* dst) {
      fx::k_minv_digits<<<dim3(cnt, ks - ks0), 128, 0, s>>>(S.W.p, S.D.p, np, (int)n, ks, r0, ks0, cnt, S.exm.p, S.sc.p,
                                                           S.ex.p, dst);
      h->launched("k_minv_digits");
    };
    digits(ra, na, S.dm.p);
    for (int ca = 0; ca <= ra; ca += gt) {
      if (ca < ra) digits(ca, gt, S.dm2.p);
      fx::Job M{};
      // the kernel's block (row tile, K step) is at row tile x (ks - ks0) + K step
      auto base = [&](const uint8_t* p, int r0) {
        return reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(p) -
                                                ((uintptr_t)r0 * (ks - ks0) + ks0) * fx::BLK);
      };
      M.A = base(S.dm.p, ra);
      M.B = ca < ra ? base(S.dm2.p, ca) : M.A;
      M.ea = M.eb = S.ex.p;
      M.ka = M.kb = ks - ks0;
      M.ks0 = ks0;
      M.ks1 = ks;
      M.seg[0] = {ra, ra + na, 4 * ca, 4 * (ca + gt), ca == ra ? 1 : 0, 0};
      M.mode = 2;
      M.m = M.n = (int)n;
      M.C = out;
      M.ldc = n;
      fx::launch(h, M);
    }
  }
}

bool fx64_cholesky(cbx_handle* h, const double* A, int64_t n, bool inverse, double* out, double* logdet, FxAdd add) {
  CBX_REQUIRE(n > 0 && n <= 130000, CBX_ERR_ARG, "matrix order out of range");
  cudaStream_t s = h->stream;
  fx::Scratch& S = fx::scratch(h);
  const int64_t np = (n + 127) / 128 * 128;
  // panel width, inverse / factor in ms: n = 1,000 1.25 / 1.19 with 128, 1.22 / 1.16 with 256;
  // 2,000 2.82 / 2.47, 2.67 / 2.35 (512: 2.88 / 2.36); 8,000 38.3 / 19.9, 34.8 / 18.1 (512: 35.4 /
  // 18.0); 10,000 with 256 61.5 / 29.7, with 512 61.2 / 29.4 (1,024: 67.0 / 32.3); 14,000 132 / 61.9,
  // 129 / 59.8.  A wider panel updates more by K = 32 inside it, a narrower one more often from outside
  const int rt = (int)(np / 128), B0 = n < 10000 ? 256 : 512;
  const int B = (int)std::min<int64_t>(B0, np);
  fx::at_least(S.W, (size_t)np * np);
  fx::at_least(S.P, (size_t)np * B);
  fx::at_least(S.D, (size_t)np * 32);
  fx::at_least(S.piv, (size_t)np + 1);
  fx::at_least(S.din, (size_t)rt * fx::BLK);
  fx::at_least(S.dout, (size_t)rt * (B / 32) * fx::BLK);
  fx::at_least(S.ex, (size_t)np);
  fx::at_least(S.exo, (size_t)np);
  fx::at_least(S.exm, (size_t)np);
  fx::at_least(S.sc, (size_t)np);
  fx::at_least(S.bad, 1);
  CBX_CUDA(cudaMemsetAsync(S.bad.p, 0, sizeof(int), s));
  fx::k_scales<<<(unsigned)(np / 128), 128, 0, s>>>(A, n, np, add, S.sc.p);
  h->launched("k_scales");
  fx::k_load_lower<<<dim3((unsigned)(np / 32), (unsigned)(np / 32)), 256, 0, s>>>(A, n, np, add, S.sc.p, S.W.p);
  h->launched("k_load_lower");
  fx::Panel a{S.W.p, np, 0, 0, 0, B, inverse ? 1 : 0, S.din.p, S.ex.p, S.exo.p, S.exm.p, S.P.p, S.D.p, S.piv.p,
              S.bad.p};
  fx::Job J{};
  J.C = S.W.p;
  J.ldc = np;
  for (int64_t K0 = 0; K0 < n; K0 += B) {
    a.K0 = (int)K0;
    a.K1 = (int)std::min<int64_t>(K0 + B, np);
    const int tp = a.K1 / 128;
    for (int k0 = a.K0; k0 < a.K1 && k0 < n; k0 += 32) {
      a.k0 = k0;
      const int groups = (int)(np / 16) - (inverse ? 0 : k0 / 16);
      fx::k_panel<<<std::min(groups, h->num_sms), 128, 0, s>>>(a);
      h->launched("k_panel");
      const int next = k0 + 32;
      if (next >= a.K1 || next >= n) continue;
      // within the panel: its remaining columns below, and its remaining rows of R
      J.A = J.B = S.din.p;
      J.ea = J.eb = S.ex.p;
      J.ka = J.kb = J.ks1 = 1;
      J.rmin = next;
      J.seg[0] = {next / 128, tp, inverse ? 0 : next / 32, 0, 1, inverse ? 0 : next};
      J.seg[1] = {tp, rt, next / 32, 4 * tp, 0, next};
      fx::launch(h, J);
    }
    if (a.K1 >= n) break;
    const int first = inverse ? 0 : tp;
    fx::k_panel_digits<<<dim3(rt - first, B / 32), 128, 0, s>>>(a, S.dout.p, first);
    h->launched("k_panel_digits");
    J.A = J.B = S.dout.p;
    J.ea = J.eb = S.exo.p;
    J.ka = J.kb = J.ks1 = B / 32;
    J.rmin = a.K1;
    J.seg[0] = {tp, rt, inverse ? 0 : 4 * tp, 0, 1, 0};
    J.seg[1] = {0, 0, 0, 0, 0, 0};
    fx::launch(h, J);
  }
  double ld = 0.0;
  int bad = 0;
  if (logdet) {
    fx::k_logsum<<<1, 256, 0, s>>>(S.piv.p, S.sc.p, (int)n, S.piv.p + np);
    h->launched("k_logsum");
    CBX_CUDA(cudaMemcpyAsync(&ld, S.piv.p + np, sizeof(double), cudaMemcpyDeviceToHost, s));
  }
  CBX_CUDA(cudaMemcpyAsync(&bad, S.bad.p, sizeof(int), cudaMemcpyDeviceToHost, s));
  CBX_CUDA(cudaStreamSynchronize(s));
  h->check_status("FP64 factorization");
  const int ks = (int)(np / 32);
  if (!bad && inverse && !fx::try_at_least(h, S.dm, ((size_t)rt * ks - 2 * (size_t)rt * (rt - 1)) * fx::BLK)) {
    minv_product_groups(h, S, np, n, out);
  } else if (!bad && inverse) {
    fx::k_minv_digits<<<dim3(rt, ks), 128, 0, s>>>(S.W.p, S.D.p, np, (int)n, ks, 0, 0, 0, S.exm.p, S.sc.p, S.ex.p,
                                                   S.dm.p);
    h->launched("k_minv_digits");
    fx::Job M{};
    M.A = M.B = S.dm.p;
    M.ea = M.eb = S.ex.p;
    M.ka = M.kb = M.ks1 = ks;
    M.ktri = 1;
    M.seg[0] = {0, rt, 0, 0, 1, 0};
    M.mode = 2;
    M.m = M.n = (int)n;
    M.C = out;
    M.ldc = n;
    fx::launch(h, M);
  } else if (!bad && out) {
    fx::k_store_factor<<<(unsigned)std::min<int64_t>((n * n + 255) / 256, 8 * h->num_sms), 256, 0, s>>>(
        S.W.p, S.D.p, np, n, S.sc.p, out);
    h->launched("k_store_factor");
  }
  if (logdet) *logdet = ld;
  if (S.bytes() > fx::kKeepBytes) {
    CBX_CUDA(cudaStreamSynchronize(s));
    h->fx_slot.reset();
  }
  return bad == 0;
}

}  // namespace cbx
