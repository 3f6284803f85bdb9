// Genotype matrix-free products from PLINK BED on the device.
//
// Replaces PlinkReader's RHE / PCG support (reference src/core/plink_reader.cpp):
//   computeStats  (:186-237)  per-SNP mean of the observed calls, p = mean / 2,
//                             var = 2p(1-p), inv_std = 1/sqrt(var), or 0 when
//                             var < 1e-9 or no call is observed;
//   multiply_Z_v  (:239-293)  y = Z v, every term (x - mean_j) v_j inv_std_j rounded
//                             to float first, as the reference's per-SNP val_map is;
//   multiply_Zt_v (:341-392)  y_j = (sum_obs x_ij v_i - mean_j sum_obs v_i) inv_std_j;
// and the SNP-effect back-solve of the result writer (src/solve/result_writer.cpp:
// 565-623, the --bfile branch): q = G^-1 u_g, effect_j = ((Z^T q)_j / inv_std_j) /
// total_2pq with total_2pq = the sum of var over SNPs with var >= 1e-9.
//
// The sums are exact.  The FP64 input vector is scaled by a power of two 2^s, chosen
// so that the sum of its magnitudes stays below 2^61, and rounded to int64.  The
// device adds int64 values modulo 2^64, so neither the order of the additions nor
// that of the atomics changes a bit of the result, and partial sums may wrap; the
// totals fit and are scaled back once.  The only rounding is the conversion of each
// input, at most 2^-(s+1) per term: the total error is below n 2^-62 sum|v|, far
// below that of the reference's sequential FP64 sums.
//
// Codes (2 bits, first sample in the low bits): 00 -> x = 2, 01 -> missing,
// 10 -> x = 1, 11 -> x = 0.  With lo / hi the two bits and k = lo + hi, every
// observed call has x = 2 - k (a missing call has k = 1).  So one SNP needs a single
// dense sum S = sum_i k_i v_i plus M = the sum of v over its missing calls, taken
// from a sparse list built once:
//   sum_obs x v = 2T - S - M,   sum_obs v = T - M,
// with T the sum of v over all samples.  Z v needs, per SNP j, w0_j for every
// sample, k (w2_j - w0_j) and, where both bits are set, w3_j - 2 w2_j + w0_j (w_c =
// the float term of code c, which is not linear in x); a missing call then receives
// w2_j, which the sample-major missing list takes back out.  Missing calls are rare
// in genotype data: the sparse passes cost one gather per missing call.
//
// The k-weighted sums run on the tensor cores as sums of six balanced base-2048 digits of
// the fixed-point values (k_geno_zt, k_geno_z).
//
// Layout: the payload is copied once into rows of `pitch` bytes (a multiple of 16,
// the padding bytes zero).  Samples at or beyond n get v = 0 (Z^T v) or are dropped
// (Z v), so the padding codes never reach a result; the missing lists hold calls of
// samples below n only.
#include <algorithm>
#include <cmath>
#include <vector>
#include <cublas_v2.h>
#include <cuda_fp16.h>
#include "dense.h"
#include "handle.h"
#include "pcg.h"
#include "tune.h"

namespace cbx {
namespace geno {

constexpr int ZT_THREADS = 256;   // 32 SNP rows per warp
constexpr int Z_THREADS = 256;    // 256 samples per warp
constexpr int Z_MAX_ROWS = 4096;  // SNP rows per CTA
constexpr int PREP_THREADS = 1024;

// Deterministic block sum of a double (fixed shuffle tree, then warp 0 over the warps).
__device__ double block_sum_f64(double a, double* red) {
  for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) red[w] = a;
  __syncthreads();
  double r = 0.0;
  if (w == 0) {
    r = l < (int)(blockDim.x >> 5) ? red[l] : 0.0;
    for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
  }
  __syncthreads();
  return r;  // valid in thread 0
}

__device__ unsigned long long block_sum_u64(unsigned long long a, unsigned long long* red) {
  for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) red[w] = a;
  __syncthreads();
  unsigned long long r = 0;
  if (w == 0) {
    r = l < (int)(blockDim.x >> 5) ? red[l] : 0ull;
    for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
  }
  __syncthreads();
  return r;  // valid in thread 0
}

// Scale exponent for a sum of magnitudes S: S 2^s < 2^61.
__device__ int fix_exponent(double S) {
  if (!(S > 0.0)) return 0;
  int e = 0;
  frexp(S, &e);  // S = f 2^e, 0.5 <= f < 1
  return 61 - e;
}

// computeStats for one SNP row per block (plink_reader.cpp:192-236).
// Also counts the SNP's missing calls (miss_cnt) for the sparse missing lists.
__global__ void k_geno_stats(const uint8_t* __restrict__ bed, int64_t pitch, int64_t n, int64_t m,
                             double* __restrict__ mean, double* __restrict__ inv_std,
                             double* __restrict__ var2pq, int32_t* __restrict__ miss_cnt) {
  const int64_t j = blockIdx.x;
  if (j >= m) return;
  const uint32_t* row = reinterpret_cast<const uint32_t*>(bed + j * pitch);
  const int64_t nw = (n + 15) / 16;
  int hom1 = 0, het = 0, hom2 = 0, miss = 0;
  for (int64_t t = threadIdx.x; t < nw; t += blockDim.x) {
    const uint32_t v = row[t];
    const int64_t valid = n - 16 * t;  // >= 1
    const uint32_t mask = valid >= 16 ? 0x55555555u : (0x55555555u >> (2 * (16 - valid)));
    const uint32_t lo = v & 0x55555555u, hi = (v >> 1) & 0x55555555u;
    hom1 += __popc(~lo & ~hi & mask);
    het += __popc(~lo & hi & mask);
    hom2 += __popc(lo & hi & mask);
    miss += __popc(lo & ~hi & mask);
  }
  for (int o = 16; o > 0; o >>= 1) {
    hom1 += __shfl_down_sync(0xffffffffu, hom1, o);
    het += __shfl_down_sync(0xffffffffu, het, o);
    hom2 += __shfl_down_sync(0xffffffffu, hom2, o);
    miss += __shfl_down_sync(0xffffffffu, miss, o);
  }
  __shared__ int red[4][32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) { red[0][w] = hom1; red[1][w] = het; red[2][w] = hom2; red[3][w] = miss; }
  __syncthreads();
  if (threadIdx.x != 0) return;
  int a = 0, b = 0, c = 0, d = 0;
  for (int i = 0; i < (int)(blockDim.x >> 5); ++i) {
    a += red[0][i]; b += red[1][i]; c += red[2][i]; d += red[3][i];
  }
  miss_cnt[j] = d;
  const int count = a + b + c;
  double mu = 0.0, is = 0.0, v2 = 0.0;
  if (count > 0) {
    // the reference sums the float codes 2, 1, 0 in double: an exact integer
    mu = __ddiv_rn((double)(2 * a + b), (double)count);
    const double p = __ddiv_rn(mu, 2.0);
    const double var = __dmul_rn(__dmul_rn(2.0, p), __dsub_rn(1.0, p));
    if (!(var < 1e-9)) {
      is = __ddiv_rn(1.0, __dsqrt_rn(var));
      v2 = var;
    }
  }
  mean[j] = mu;
  inv_std[j] = is;
  var2pq[j] = v2;
}

// total_2pq of the back-solve (result_writer.cpp:604-609): one block, fixed order.
__global__ void __launch_bounds__(PREP_THREADS) k_geno_total(const double* __restrict__ var2pq, int64_t m,
                                                            double* __restrict__ out) {
  __shared__ double red[32];
  double a = 0.0;
  for (int64_t j = threadIdx.x; j < m; j += blockDim.x) a += var2pq[j];
  a = block_sum_f64(a, red);
  if (threadIdx.x == 0) *out = a;
}

// Exclusive prefix sum of len int32 counts into ptr[0..len] (one block, fixed order).
__global__ void __launch_bounds__(PREP_THREADS) k_geno_scan(const int32_t* __restrict__ cnt, int64_t len,
                                                           int64_t* __restrict__ ptr) {
  __shared__ long long part[PREP_THREADS];
  const int t = threadIdx.x;
  const int64_t seg = (len + PREP_THREADS - 1) / PREP_THREADS;
  const int64_t lo = std::min<int64_t>(len, t * seg), hi = std::min<int64_t>(len, lo + seg);
  long long sum = 0;
  for (int64_t i = lo; i < hi; ++i) sum += cnt[i];
  part[t] = sum;
  __syncthreads();
  if (t == 0) {
    long long run = 0;
    for (int i = 0; i < PREP_THREADS; ++i) {
      const long long x = part[i];
      part[i] = run;
      run += x;
    }
    ptr[len] = run;
  }
  __syncthreads();
  long long run = part[t];
  for (int64_t i = lo; i < hi; ++i) {
    ptr[i] = run;
    run += cnt[i];
  }
}

// SNP-major missing list: one warp per SNP writes the sample indices of its missing
// calls (increasing) at snp_list[ptr[j]..] and counts them per sample.
__global__ void k_geno_miss_fill(const uint8_t* __restrict__ bed, int64_t pitch, int64_t n, int64_t m,
                                 const int64_t* __restrict__ ptr, int32_t* __restrict__ snp_list,
                                 int32_t* __restrict__ samp_cnt) {
  const int lane = threadIdx.x & 31;
  const int64_t j = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (j >= m) return;
  const uint32_t* row = reinterpret_cast<const uint32_t*>(bed + j * pitch);
  const int64_t nw = (n + 15) / 16;
  int64_t base = ptr[j];
  for (int64_t w0 = 0; w0 < nw; w0 += 32) {
    const int64_t t = w0 + lane;
    uint32_t bits = 0;
    if (t < nw) {
      const uint32_t v = row[t];
      const int64_t valid = n - 16 * t;
      const uint32_t mask = valid >= 16 ? 0x55555555u : (0x55555555u >> (2 * (16 - valid)));
      bits = v & ~(v >> 1) & mask;  // code 01
    }
    const int c = __popc(bits);
    int incl = c;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    int64_t pos = base + incl - c;
    while (bits) {
      const int b = __ffs(bits) - 1;
      const int32_t i = (int32_t)(16 * t + (b >> 1));
      snp_list[pos++] = i;
      atomicAdd(samp_cnt + i, 1);
      bits &= bits - 1;
    }
    base += __shfl_sync(0xffffffffu, incl, 31);
  }
}

// Sample-major copy of the missing list (the order within a sample is free: the
// corrections it feeds are exact integer sums).
__global__ void k_geno_miss_transpose(const int64_t* __restrict__ ptr, const int32_t* __restrict__ snp_list,
                                      int64_t m, const int64_t* __restrict__ samp_ptr,
                                      int32_t* __restrict__ samp_fill, int32_t* __restrict__ samp_list) {
  const int lane = threadIdx.x & 31;
  const int64_t j = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (j >= m) return;
  for (int64_t k = ptr[j] + lane; k < ptr[j + 1]; k += 32) {
    const int32_t i = snp_list[k];
    const int pos = atomicAdd(samp_fill + i, 1);
    samp_list[samp_ptr[i] + pos] = (int32_t)j;
  }
}

// This lane's share of the sum of x[list[k]], lo <= k < hi: eight gathers in flight.
__device__ __forceinline__ unsigned long long gather_sum(const int32_t* __restrict__ list, int64_t lo, int64_t hi,
                                                         const long long* __restrict__ x, int lane) {
  unsigned long long s[8] = {};
  int64_t k = lo + lane;
  for (; k + 7 * 32 < hi; k += 8 * 32) {
    int32_t e[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) e[u] = list[k + 32 * u];
#pragma unroll
    for (int u = 0; u < 8; ++u) s[u] += (unsigned long long)x[e[u]];
  }
  for (; k < hi; k += 32) s[0] += (unsigned long long)x[list[k]];
  return ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
}

// M_j = sum of V over SNP j's missing calls, into acc[m + j] (one warp per SNP).
__global__ void k_geno_miss_zt(const int64_t* __restrict__ ptr, const int32_t* __restrict__ snp_list, int64_t m,
                               const long long* __restrict__ V, unsigned long long* __restrict__ acc) {
  const int lane = threadIdx.x & 31;
  const int64_t j = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (j >= m) return;
  unsigned long long s = gather_sum(snp_list, ptr[j], ptr[j + 1], V, lane);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) acc[m + j] = s;
}

// Takes the missing calls' spurious terms back out of Z v: acc[i] -= sum of W2[j] over the SNPs j where sample i is missing (one warp per sample).
__global__ void k_geno_miss_z(const int64_t* __restrict__ samp_ptr, const int32_t* __restrict__ samp_list,
                              int64_t n, const long long* __restrict__ W2, unsigned long long* __restrict__ acc) {
  const int lane = threadIdx.x & 31;
  const int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= n) return;
  unsigned long long s = gather_sum(samp_list, samp_ptr[i], samp_ptr[i + 1], W2, lane);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) acc[i] -= s;
}

// Blocks of the two-pass preparations: partial sums of one per block, added in block order.
constexpr int PREP_BLOCKS = 128;
constexpr int PREP_NT = 256;

__device__ double sum_parts(const double* part, double* red) {
  return block_sum_f64(threadIdx.x < PREP_BLOCKS ? part[threadIdx.x] : 0.0, red);
}
// sum of the blocks' integer partials, in every thread
__device__ unsigned long long all_sum_u64(const unsigned long long* part) {
  __shared__ unsigned long long red[32], tot;
  const unsigned long long t = block_sum_u64(threadIdx.x < PREP_BLOCKS ? part[threadIdx.x] : 0ull, red);
  if (threadIdx.x == 0) tot = t;
  __syncthreads();
  return tot;
}

// Sums of |v| per block.
__global__ void __launch_bounds__(PREP_NT) k_geno_vsum(const double* __restrict__ v, int64_t n,
                                                      double* __restrict__ part) {
  __shared__ double red[32];
  double a = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)PREP_NT + threadIdx.x; i < n; i += PREP_BLOCKS * (int64_t)PREP_NT)
    a += fabs(v[i]);
  a = block_sum_f64(a, red);
  if (threadIdx.x == 0) part[blockIdx.x] = a;
}
// The scale exponent of the sum of the partials; a non-finite one sets the status.
__device__ int scale_of(const double* part, long long* meta, int* status) {
  __shared__ double red[32];
  __shared__ int s_sh;
  const double a = sum_parts(part, red);
  if (threadIdx.x == 0) {
    const bool ok = isfinite(a);
    s_sh = ok ? fix_exponent(a) : 0;
    if (blockIdx.x == 0) {
      if (!ok) atomicExch(status, DEV_NONFINITE);
      meta[0] = s_sh;
    }
  }
  __syncthreads();
  return s_sh;
}
// v (n, FP64) -> V (n_pad, int64 at scale 2^s, zero past n) and their sums per block;
// meta[0] = s.
__global__ void __launch_bounds__(PREP_NT) k_geno_vprep(const double* __restrict__ v, int64_t n, int64_t n_pad,
                                                       const double* __restrict__ part, long long* __restrict__ V,
                                                       unsigned long long* __restrict__ tpart,
                                                       long long* __restrict__ meta, int* status) {
  __shared__ unsigned long long redu[32];
  const int s = scale_of(part, meta, status);
  unsigned long long t = 0;
  for (int64_t i = blockIdx.x * (int64_t)PREP_NT + threadIdx.x; i < n_pad; i += PREP_BLOCKS * (int64_t)PREP_NT) {
    const long long x = i < n ? __double2ll_rn(ldexp(v[i], s)) : 0ll;
    V[i] = x;
    t += (unsigned long long)x;
  }
  t = block_sum_u64(t, redu);
  if (threadIdx.x == 0) tpart[blockIdx.x] = t;
}

// Float terms of multiply_Z_v per SNP (plink_reader.cpp:258-270), w[3j..], and the sums of
// their largest magnitudes per block.
__global__ void __launch_bounds__(PREP_NT) k_geno_zterms(const double* __restrict__ v, const double* __restrict__ mean,
                                                        const double* __restrict__ inv_std, int64_t m,
                                                        float* __restrict__ w, double* __restrict__ part) {
  __shared__ double red[32];
  double a = 0.0;
  for (int64_t j = blockIdx.x * (int64_t)PREP_NT + threadIdx.x; j < m; j += PREP_BLOCKS * (int64_t)PREP_NT) {
    float w0 = 0.f, w2 = 0.f, w3 = 0.f;
    const double is = inv_std[j];
    if (is != 0.0) {
      const double mu = mean[j];
      const double weight = __dmul_rn(v[j], is);
      w0 = __double2float_rn(__dmul_rn(__dsub_rn(2.0, mu), weight));
      w2 = __double2float_rn(__dmul_rn(__dsub_rn(1.0, mu), weight));
      w3 = __double2float_rn(__dmul_rn(__dsub_rn(0.0, mu), weight));
    }
    w[3 * j] = w0;
    w[3 * j + 1] = w2;
    w[3 * j + 2] = w3;
    a += (double)fmaxf(fabsf(w0), fmaxf(fabsf(w2), fabsf(w3)));
  }
  a = block_sum_f64(a, red);
  if (threadIdx.x == 0) part[blockIdx.x] = a;
}
// Their int64 values at scale 2^s: D[2j], D[2j + 1] = W2 - W0 per unit of k, W3 - 2 W2 + W0
// where both bits are set; D[2m + j] = W2, the spurious term of a missing call; meta[0] = s,
// and the sums of W0 (added to every sample) per block.
__global__ void __launch_bounds__(PREP_NT) k_geno_zprep(const float* __restrict__ w, int64_t m,
                                                       const double* __restrict__ part, long long* __restrict__ D,
                                                       unsigned long long* __restrict__ cpart,
                                                       long long* __restrict__ meta, int* status) {
  __shared__ unsigned long long redu[32];
  const int s = scale_of(part, meta, status);
  unsigned long long c = 0;
  for (int64_t j = blockIdx.x * (int64_t)PREP_NT + threadIdx.x; j < m; j += PREP_BLOCKS * (int64_t)PREP_NT) {
    const long long W0 = __double2ll_rn(ldexp((double)w[3 * j], s));
    const long long W2 = __double2ll_rn(ldexp((double)w[3 * j + 1], s));
    const long long W3 = __double2ll_rn(ldexp((double)w[3 * j + 2], s));
    D[2 * j] = W2 - W0;
    D[2 * j + 1] = W3 - 2 * W2 + W0;
    D[2 * m + j] = W2;
    c += (unsigned long long)W0;
  }
  c = block_sum_u64(c, redu);
  if (threadIdx.x == 0) cpart[blockIdx.x] = c;
}

// ---- products on the tensor cores ---------------------------------------------
// A fixed-point value is cut into six balanced base-2048 digits (|d| <= 1024, exact in
// f16; the top one holds the sign).  A 2-bit field is an f16 as it stands: the bit patterns
// 0, 1, 2, 3 are the subnormals 0, 1, 2, 3 times 2^-24.  So codes become operands of
// mma.m16n8k16 (f16, FP32 accumulation) with one shift and one mask for two of them, the six
// digits are columns of the other operand, and the accumulators are exact integers times
// 2^-24 while a chunk's sum of magnitudes stays below 2^24: 5,461 terms of at most 3,072.
// Each chunk's digits are put together modulo 2^64 and added to the totals, so results do
// not depend on the order.  The codes are decoded in registers and used in place, which a
// tile staged in shared memory for tcgen05 would write and read twice.
constexpr int NDIG = 6;

__device__ __forceinline__ int digit_of(long long x, int j) {
  constexpr unsigned long long bias = 1024ull * (1ull + (1ull << 11) + (1ull << 22) + (1ull << 33) + (1ull << 44));
  const unsigned long long g = (unsigned long long)x + bias;
  return j < 5 ? (int)((g >> (11 * j)) & 2047) - 1024 : j == 5 ? (int)((long long)g >> 55) : 0;
}
__device__ __forceinline__ uint32_t digit_pair(long long lo, long long hi, int j) {
  return (uint32_t)__half_as_ushort(__int2half_rn(digit_of(lo, j))) |
         (uint32_t)__half_as_ushort(__int2half_rn(digit_of(hi, j))) << 16;
}
__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the digits of two columns of one row, as one integer; summed over the quad's columns
__device__ __forceinline__ unsigned long long total_of(float c0, float c1, int t) {
  unsigned long long s = 0;
  if (t < 3)
    s = ((unsigned long long)(long long)__float2int_rn(c0 * 0x1p24f) << (22 * t)) +
        ((unsigned long long)(long long)__float2int_rn(c1 * 0x1p24f) << (22 * t + 11));
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  return s;
}

// Digits of V as the second operand of Z^T v: entry ((seg 4 + q) 4 + i) 32 + lane holds
// column lane / 4 of samples base + {2i, 2i + 8} and base + {2i + 1, 2i + 9}, base = 256 seg +
// 64 (lane % 4) + 16 q: the order in which k_geno_zt meets them.
__global__ void __launch_bounds__(256) k_geno_vdig(const long long* __restrict__ V, int64_t n_pad, int64_t total,
                                                   uint2* __restrict__ B) {
  for (int64_t e = blockIdx.x * 256ll + threadIdx.x; e < total; e += gridDim.x * 256ll) {
    const int lane = (int)(e & 31), i = (int)(e >> 5 & 3), q = (int)(e >> 7 & 3), j = lane >> 2;
    const int64_t base = (e >> 9) * 256 + 64 * (lane & 3) + 16 * q + 2 * i;
    uint2 o = make_uint2(0u, 0u);
    if (j < NDIG && base < n_pad) {
      o.x = digit_pair(V[base], V[base + 8], j);
      o.y = digit_pair(V[base + 1], V[base + 9], j);
    }
    B[e] = o;
  }
}

// Z^T v: a warp takes 32 SNP rows and a chunk of samples, 256 at a time: each lane loads
// 64 samples (16 bytes) of four rows, and 16 MMAs a row pair use them.  acc[row] += sum of
// k V (64-bit atomics).  Bound by the latency of the loads at its few warps, with mma.sync busy a
// quarter of the time (profiled): at n = 20,000, m = 50,000 0.097 ms (0.20 ms as two integer
// multiply-adds a code).
constexpr int ZT_ROWS = 32 * (ZT_THREADS / 32);
__global__ void __launch_bounds__(ZT_THREADS) k_geno_zt(const uint8_t* __restrict__ bed, int64_t pitch, int64_t m,
                                                       int segs_per_cta, const uint2* __restrict__ B,
                                                       unsigned long long* __restrict__ acc) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int64_t row0 = (int64_t)blockIdx.x * ZT_ROWS + (threadIdx.x >> 5) * 32;
  if (row0 >= m) return;
  const int64_t segs = (pitch + 63) / 64;
  const int64_t s0 = (int64_t)blockIdx.y * segs_per_cta, s1 = std::min<int64_t>(segs, s0 + segs_per_cta);
  float c[2][4] = {};
  for (int64_t sg = s0; sg < s1; ++sg) {
    const int64_t off = sg * 64 + 16 * t;
    uint4 w[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int64_t row = row0 + g + 8 * r;
      w[r] = make_uint4(0u, 0u, 0u, 0u);
      if (row < m && off < pitch) w[r] = __ldg(reinterpret_cast<const uint4*>(bed + row * pitch + off));
    }
    const uint2* bp = B + sg * 512 + lane;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t kw[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const uint32_t x = q == 0 ? w[r].x : q == 1 ? w[r].y : q == 2 ? w[r].z : w[r].w;
        kw[r] = (x & 0x55555555u) + ((x >> 1) & 0x55555555u);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint2 b = __ldg(bp + (q * 4 + i) * 32);
#pragma unroll
        for (int h = 0; h < 2; ++h)
          mma_f16(c[h], (kw[2 * h] >> (4 * i)) & 0x00030003u, (kw[2 * h + 1] >> (4 * i)) & 0x00030003u,
                  (kw[2 * h] >> (4 * i + 2)) & 0x00030003u, (kw[2 * h + 1] >> (4 * i + 2)) & 0x00030003u, b.x, b.y);
      }
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const unsigned long long s = total_of(c[h][2 * k], c[h][2 * k + 1], t);
      const int64_t row = row0 + 16 * h + 8 * k + g;
      if (t == 0 && row < m) atomicAdd(acc + row, s);
    }
}

// Digits of D as the second operand of Z v: entry blk 32 + lane holds column lane / 4 of
// the SNPs 16 blk + {2t, 2t + 1} and {2t + 8, 2t + 9} (t = lane % 4), of D[2j] and then of
// D[2j + 1].
__global__ void __launch_bounds__(256) k_geno_zdig(const long long* __restrict__ D, int64_t m, int64_t total,
                                                   uint4* __restrict__ B) {
  for (int64_t e = blockIdx.x * 256ll + threadIdx.x; e < total; e += gridDim.x * 256ll) {
    const int lane = (int)(e & 31), j = lane >> 2;
    const int64_t r = (e >> 5) * 16 + 2 * (lane & 3);
    auto d = [&](int64_t row, int k) { return row < m ? D[2 * row + k] : 0ll; };
    uint4 o = make_uint4(0u, 0u, 0u, 0u);
    if (j < NDIG) {
      o.x = digit_pair(d(r, 0), d(r + 1, 0), j);
      o.y = digit_pair(d(r + 8, 0), d(r + 9, 0), j);
      o.z = digit_pair(d(r, 1), d(r + 1, 1), j);
      o.w = digit_pair(d(r + 8, 1), d(r + 9, 1), j);
    }
    B[e] = o;
  }
}

// Z v: a warp takes 256 samples (two words of 16 per lane group) and a chunk of SNPs, 16
// at a time: lane (g, t) holds the words of SNPs 2t, 2t + 1, 2t + 8, 2t + 9, whose halves
// pair up to samples 0-7 and 8-15 of two SNPs; MMA i multiplies samples i and i + 8 of
// eight words.  A second MMA adds the term of codes with both bits set.  acc[i] += the
// sum (64-bit atomics).  Bound by the issue of the decoding, four instructions an MMA, and the
// MMAs' latency (their pipe is busy a quarter of the time): at n = 20,000, m = 50,000 0.20 ms
// (0.52 ms as integer multiply-adds).
constexpr int Z_SAMPLES = 256 * (Z_THREADS / 32);
__global__ void __launch_bounds__(Z_THREADS) k_geno_z(const uint8_t* __restrict__ bed, int64_t pitch, int64_t m,
                                                     int blks_per_cta, const uint4* __restrict__ B,
                                                     unsigned long long* __restrict__ acc) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int64_t off = (int64_t)blockIdx.x * (Z_SAMPLES / 4) + (threadIdx.x >> 5) * 64 + 8 * g;
  const int64_t blks = (m + 15) / 16;
  const int64_t b0 = (int64_t)blockIdx.y * blks_per_cta, b1 = std::min<int64_t>(blks, b0 + blks_per_cta);
  if (off - 8 * g >= pitch) return;
  float c[2][8][4] = {};
  for (int64_t blk = b0; blk < b1; ++blk) {
    uint2 w[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int64_t row = blk * 16 + 2 * t + (r & 1) + 8 * (r >> 1);
      w[r] = make_uint2(0u, 0u);
      if (row < m && off < pitch) w[r] = __ldg(reinterpret_cast<const uint2*>(bed + row * pitch + off));
    }
    const uint4 b = __ldg(B + blk * 32 + lane);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      uint32_t kw[4], bo[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const uint32_t x = q == 0 ? w[r].x : w[r].y;
        kw[r] = (x & 0x55555555u) + ((x >> 1) & 0x55555555u);
        bo[r] = x & (x >> 1) & 0x55555555u;
      }
      const uint32_t k0 = __byte_perm(kw[0], kw[1], 0x5410), k1 = __byte_perm(kw[0], kw[1], 0x7632);
      const uint32_t k2 = __byte_perm(kw[2], kw[3], 0x5410), k3 = __byte_perm(kw[2], kw[3], 0x7632);
      const uint32_t o0 = __byte_perm(bo[0], bo[1], 0x5410), o1 = __byte_perm(bo[0], bo[1], 0x7632);
      const uint32_t o2 = __byte_perm(bo[2], bo[3], 0x5410), o3 = __byte_perm(bo[2], bo[3], 0x7632);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        mma_f16(c[q][i], (k0 >> (2 * i)) & 0x00030003u, (k1 >> (2 * i)) & 0x00030003u, (k2 >> (2 * i)) & 0x00030003u,
                (k3 >> (2 * i)) & 0x00030003u, b.x, b.y);
        mma_f16(c[q][i], (o0 >> (2 * i)) & 0x00010001u, (o1 >> (2 * i)) & 0x00010001u, (o2 >> (2 * i)) & 0x00010001u,
                (o3 >> (2 * i)) & 0x00010001u, b.z, b.w);
      }
    }
  }
  const int64_t i0 = off * 4;  // first sample of this lane group's two words
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const unsigned long long lo = total_of(c[q][i][0], c[q][i][1], t), hi = total_of(c[q][i][2], c[q][i][3], t);
      if (off < pitch && t == (i & 3)) {
        atomicAdd(acc + i0 + 16 * q + i, lo);
        atomicAdd(acc + i0 + 16 * q + i + 8, hi);
      }
    }
}

// multiply_Zt_v's last step (plink_reader.cpp:387) and, when effect != null, the
// back-solve's effect / frequency (result_writer.cpp:614-620).
__global__ void k_geno_zt_fin(const unsigned long long* __restrict__ acc, const long long* __restrict__ meta,
                              const unsigned long long* __restrict__ tpart,
                              const double* __restrict__ mean, const double* __restrict__ inv_std,
                              int64_t m, const double* __restrict__ total_2pq, double* __restrict__ y,
                              double* __restrict__ effect, double* __restrict__ freq) {
  const int s = (int)meta[0];
  const unsigned long long T = all_sum_u64(tpart);
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < m;
       j += (int64_t)gridDim.x * blockDim.x) {
    const unsigned long long S = acc[j], miss = acc[m + j];
    const long long A = (long long)(2ull * T - S - miss);
    const long long B = (long long)(T - miss);
    const double is = inv_std[j];
    double r = 0.0;
    if (is != 0.0) {
      const double sum_xv = ldexp(__ll2double_rn(A), -s);
      const double sum_v_obs = ldexp(__ll2double_rn(B), -s);
      r = __dmul_rn(__dsub_rn(sum_xv, __dmul_rn(mean[j], sum_v_obs)), is);
    }
    if (y) y[j] = r;
    if (effect) {
      const double t2 = *total_2pq;
      effect[j] = (is > 0.0 && t2 > 0.0) ? __ddiv_rn(__ddiv_rn(r, is), t2) : 0.0;
      freq[j] = __ddiv_rn(mean[j], 2.0);
    }
  }
}

__global__ void k_geno_z_fin(const unsigned long long* __restrict__ acc, const long long* __restrict__ meta,
                             const unsigned long long* __restrict__ cpart, int64_t n, double* __restrict__ y) {
  const int s = (int)meta[0];
  const unsigned long long C = all_sum_u64(cpart);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    y[i] = ldexp(__ll2double_rn((long long)(C + acc[i])), -s);
}

struct State {
  DevBuf<uint8_t> bed;      // m x pitch
  int64_t n = 0, m = 0, pitch = 0;
  DevBuf<double> stats;     // mean (m), inv_std (m), var2pq (m), total_2pq (1)
  DevBuf<long long> fixv;   // fixed-point V (n_pad) or per-SNP values (3m)
  DevBuf<uint4> dig;        // their digits, in the products' order
  DevBuf<double> part;      // partial sums of the preparations
  DevBuf<unsigned long long> tpart;
  DevBuf<float> wterm;      // float terms of Z v (3m)
  DevBuf<long long> meta;   // s, T or C
  DevBuf<unsigned long long> acc;
  DevBuf<double> vin, vout, q;
  // missing calls: SNP-major (miss_ptr m + 1, miss_snp) and sample-major (samp_ptr
  // n + 1, miss_samp) lists of the other index
  int64_t nmiss = 0;
  DevBuf<int64_t> miss_ptr, samp_ptr;
  DevBuf<int32_t> miss_snp, miss_samp;
  double* mean() const { return stats.p; }
  double* inv_std() const { return stats.p + m; }
  double* var2pq() const { return stats.p + 2 * m; }
  double* total() const { return stats.p + 3 * m; }
  int64_t n_pad() const { return 4 * pitch; }
};

State& state(cbx_handle* h) {
  CBX_REQUIRE(h->geno_slot, CBX_ERR_STATE, "call cbx_geno_attach first");
  return *static_cast<State*>(h->geno_slot.get());
}

template <typename F>
void timed(cbx_handle* h, int bucket, double bytes, F&& launch) {
  cbx_handle::ProfRec pr{};
  if (h->prof_on) {
    CBX_CUDA(cudaEventCreate(&pr.a));
    CBX_CUDA(cudaEventCreate(&pr.b));
    CBX_CUDA(cudaEventRecord(pr.a, h->stream));
  }
  launch();
  if (h->prof_on) {
    CBX_CUDA(cudaEventRecord(pr.b, h->stream));
    pr.bucket = bucket;
    pr.bytes = bytes;
    h->prof.push_back(pr);
  }
}

// Buffers of both products, made at the first and kept with the payload.
void scratch(State& g) {
  const int64_t segs = (g.pitch + 63) / 64, blks = (g.m + 15) / 16;
  g.fixv.resize(std::max<int64_t>(g.n_pad(), 3 * g.m));
  g.wterm.resize(3 * g.m);
  g.dig.resize(std::max<int64_t>(segs * 256, blks * 32));
  g.part.resize(PREP_BLOCKS);
  g.tpart.resize(PREP_BLOCKS);
  g.meta.resize(2);
  g.acc.resize(std::max<int64_t>(2 * g.m, g.n_pad()));
}

// y (m) = Z^T v for a device vector v (n).  With effect != null also the
// back-solve's effect and frequency columns.
void zt_device(cbx_handle* h, State& g, const double* v, double* y, double* effect, double* freq) {
  cudaStream_t s = h->stream;
  scratch(g);
  CBX_CUDA(cudaMemsetAsync(g.acc.p + g.m, 0, g.m * sizeof(unsigned long long), s));
  long long* V = g.fixv.p;
  uint2* B = reinterpret_cast<uint2*>(g.dig.p);
  k_geno_vsum<<<PREP_BLOCKS, PREP_NT, 0, s>>>(v, g.n, g.part.p);
  h->launched("k_geno_vsum");
  k_geno_vprep<<<PREP_BLOCKS, PREP_NT, 0, s>>>(v, g.n, g.n_pad(), g.part.p, V, g.tpart.p, g.meta.p, h->status.p);
  h->launched("k_geno_vprep");
  const int64_t segs = (g.pitch + 63) / 64;
  k_geno_vdig<<<gridn(segs * 512, 256, 8 * h->num_sms), 256, 0, s>>>(V, g.n_pad(), segs * 512, B);
  h->launched("k_geno_vdig");
  // algorithmic bytes: the payload once, v once per SNP block of the grid, one row result
  const double bytes = (double)g.m * (double)((g.n + 3) / 4) + 8.0 * (double)g.n + 8.0 * (double)g.m;
  const unsigned gx = (unsigned)((g.m + ZT_ROWS - 1) / ZT_ROWS);
  // 256-sample segments per CTA: 16 (default), 8 or 4 -- at most 4,096 samples, so that the
  // FP32 sums stay exact; exact integer totals, so every shape gives the same bits (the
  // accumulator is zeroed before each run)
  auto zt = [&](int c) {
    CBX_CUDA(cudaMemsetAsync(g.acc.p, 0, g.m * sizeof(unsigned long long), s));
    const int per = c == 1 ? 8 : (c == 2 ? 4 : 16);
    const int64_t gy = (segs + per - 1) / per;
    CBX_REQUIRE(gy <= 65535, CBX_ERR_ARG, "too many samples for the Z'v grid");
    k_geno_zt<<<dim3(gx, (unsigned)gy), ZT_THREADS, 0, s>>>(g.bed.p, g.pitch, g.m, per, B, g.acc.p);
    h->launched("k_geno_zt");
  };
  const int choice = tune::choose(h, tune::GENO_ZT, tune::size_class(g.n), tune::size_class(g.m), 1, 3, zt);
  timed(h, 3, bytes, [&] { zt(choice); });
  if (g.nmiss > 0) {
    k_geno_miss_zt<<<(unsigned)((g.m + 7) / 8), 256, 0, s>>>(g.miss_ptr.p, g.miss_snp.p, g.m, V, g.acc.p);
    h->launched("k_geno_miss_zt");
  }
  k_geno_zt_fin<<<gridn(g.m, 256, 4 * h->num_sms), 256, 0, s>>>(g.acc.p, g.meta.p, g.tpart.p, g.mean(),
                                                                g.inv_std(), g.m, g.total(), y, effect, freq);
  h->launched("k_geno_zt_fin");
}

// y (n) = Z v for a device vector v (m).
void z_device(cbx_handle* h, State& g, const double* v, double* y) {
  cudaStream_t s = h->stream;
  scratch(g);
  const int64_t n_pad = g.n_pad(), blks = (g.m + 15) / 16;
  k_geno_zterms<<<PREP_BLOCKS, PREP_NT, 0, s>>>(v, g.mean(), g.inv_std(), g.m, g.wterm.p, g.part.p);
  h->launched("k_geno_zterms");
  k_geno_zprep<<<PREP_BLOCKS, PREP_NT, 0, s>>>(g.wterm.p, g.m, g.part.p, g.fixv.p, g.tpart.p, g.meta.p, h->status.p);
  h->launched("k_geno_zprep");
  k_geno_zdig<<<gridn(blks * 32, 256, 8 * h->num_sms), 256, 0, s>>>(g.fixv.p, g.m, blks * 32, g.dig.p);
  h->launched("k_geno_zdig");
  const int gx = (int)((g.pitch + Z_SAMPLES / 4 - 1) / (Z_SAMPLES / 4));
  const double bytes = (double)g.m * (double)((g.n + 3) / 4) + 8.0 * (double)g.m + 8.0 * (double)g.n;
  // about 4 (default), 2 or 8 CTAs per SM, at most Z_MAX_ROWS SNPs each, so that the FP32
  // sums stay exact; exact integer totals, so every shape gives the same bits (the
  // accumulator is zeroed before each run)
  auto zk = [&](int c) {
    CBX_CUDA(cudaMemsetAsync(g.acc.p, 0, n_pad * sizeof(unsigned long long), s));
    const int per_sm = c == 1 ? 2 : (c == 2 ? 8 : 4);
    int64_t gy = std::max<int64_t>(1, (per_sm * (int64_t)h->num_sms + gx - 1) / gx);
    const int64_t per = std::min<int64_t>((blks + gy - 1) / gy, Z_MAX_ROWS / 16);
    gy = (blks + per - 1) / per;
    CBX_REQUIRE(gy <= 65535, CBX_ERR_ARG, "too many SNPs for the Z v grid");
    k_geno_z<<<dim3((unsigned)gx, (unsigned)gy), Z_THREADS, 0, s>>>(g.bed.p, g.pitch, g.m, (int)per, g.dig.p, g.acc.p);
    h->launched("k_geno_z");
  };
  const int choice = tune::choose(h, tune::GENO_Z, tune::size_class(g.n), tune::size_class(g.m), 1, 3, zk);
  timed(h, 4, bytes, [&] { zk(choice); });
  if (g.nmiss > 0) {
    k_geno_miss_z<<<(unsigned)((g.n + 7) / 8), 256, 0, s>>>(g.samp_ptr.p, g.miss_samp.p, g.n, g.fixv.p + 2 * g.m, g.acc.p);
    h->launched("k_geno_miss_z");
  }
  k_geno_z_fin<<<gridn(g.n, 256, 4 * h->num_sms), 256, 0, s>>>(g.acc.p, g.meta.p, g.tpart.p, g.n, y);
  h->launched("k_geno_z_fin");
}

}  // namespace geno
}  // namespace cbx

using namespace cbx;

extern "C" int cbx_geno_attach(cbx_handle* h, const uint8_t* bed, int64_t bed_bytes, int64_t n, int64_t m,
                               double* means, double* inv_stds) {
  return cbx_guard(h, [&] {
    CBX_REQUIRE(bed != nullptr, CBX_ERR_ARG, "bed is null");
    CBX_REQUIRE(n > 0 && m > 0, CBX_ERR_ARG, "empty genotype matrix");
    CBX_REQUIRE(n < (int64_t(1) << 31) && m < (int64_t(1) << 31), CBX_ERR_ARG, "n or m too large");
    CBX_REQUIRE(bed_bytes >= 3, CBX_ERR_FORMAT, "Invalid .bed file (too small)");
    CBX_REQUIRE(bed[0] == 0x6C && bed[1] == 0x1B, CBX_ERR_FORMAT, "Invalid .bed file magic number");
    CBX_REQUIRE(bed[2] == 0x01, CBX_ERR_FORMAT, "Only SNP-major mode (0x01) .bed files are supported");
    const int64_t bps = (n + 3) / 4;
    CBX_REQUIRE(bed_bytes >= 3 + m * bps, CBX_ERR_FORMAT,
                ".bed file is truncated: " + std::to_string(bed_bytes) + " < " + std::to_string(3 + m * bps) +
                    " bytes");
    CBX_CUDA(cudaSetDevice(h->device));
    cudaStream_t s = h->stream;
    auto g = std::make_shared<geno::State>();
    g->n = n;
    g->m = m;
    g->pitch = (bps + 15) / 16 * 16;
    g->bed.resize(m * g->pitch);
    g->bed.zero(s);
    CBX_CUDA(cudaMemcpy2DAsync(g->bed.p, g->pitch, bed + 3, bps, bps, m, cudaMemcpyHostToDevice, s));
    g->stats.resize(3 * m + 1);
    DevBuf<int32_t> cnt;
    cnt.resize(std::max(m, n));
    geno::k_geno_stats<<<(unsigned)m, 128, 0, s>>>(g->bed.p, g->pitch, n, m, g->mean(), g->inv_std(),
                                                    g->var2pq(), cnt.p);
    h->launched("k_geno_stats");
    geno::k_geno_total<<<1, geno::PREP_THREADS, 0, s>>>(g->var2pq(), m, g->total());
    h->launched("k_geno_total");
    // sparse missing lists
    g->miss_ptr.resize(m + 1);
    geno::k_geno_scan<<<1, geno::PREP_THREADS, 0, s>>>(cnt.p, m, g->miss_ptr.p);
    h->launched("k_geno_scan");
    CBX_CUDA(cudaMemcpyAsync(&g->nmiss, g->miss_ptr.p + m, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    CBX_CUDA(cudaStreamSynchronize(s));
    if (g->nmiss > 0) {
      g->miss_snp.resize(g->nmiss);
      g->miss_samp.resize(g->nmiss);
      g->samp_ptr.resize(n + 1);
      CBX_CUDA(cudaMemsetAsync(cnt.p, 0, n * sizeof(int32_t), s));
      geno::k_geno_miss_fill<<<(unsigned)((m + 7) / 8), 256, 0, s>>>(g->bed.p, g->pitch, n, m, g->miss_ptr.p,
                                                                     g->miss_snp.p, cnt.p);
      h->launched("k_geno_miss_fill");
      geno::k_geno_scan<<<1, geno::PREP_THREADS, 0, s>>>(cnt.p, n, g->samp_ptr.p);
      h->launched("k_geno_scan");
      CBX_CUDA(cudaMemsetAsync(cnt.p, 0, n * sizeof(int32_t), s));
      geno::k_geno_miss_transpose<<<(unsigned)((m + 7) / 8), 256, 0, s>>>(g->miss_ptr.p, g->miss_snp.p, m,
                                                                          g->samp_ptr.p, cnt.p, g->miss_samp.p);
      h->launched("k_geno_miss_transpose");
    }
    if (means) CBX_CUDA(cudaMemcpyAsync(means, g->mean(), m * sizeof(double), cudaMemcpyDeviceToHost, s));
    if (inv_stds)
      CBX_CUDA(cudaMemcpyAsync(inv_stds, g->inv_std(), m * sizeof(double), cudaMemcpyDeviceToHost, s));
    CBX_CUDA(cudaStreamSynchronize(s));
    h->geno_slot = g;
  });
}

extern "C" int cbx_geno_zt_v(cbx_handle* h, int32_t nvec, const double* v, double* y) {
  return cbx_guard(h, [&] {
    geno::State& g = geno::state(h);
    CBX_REQUIRE(nvec > 0 && v && y, CBX_ERR_ARG, "bad vectors");
    CBX_CUDA(cudaSetDevice(h->device));
    cudaStream_t s = h->stream;
    g.vin.resize(g.n);
    g.vout.resize(g.m);
    for (int c = 0; c < nvec; ++c) {
      CBX_CUDA(cudaMemcpyAsync(g.vin.p, v + (int64_t)c * g.n, g.n * sizeof(double), cudaMemcpyHostToDevice, s));
      geno::zt_device(h, g, g.vin.p, g.vout.p, nullptr, nullptr);
      CBX_CUDA(cudaMemcpyAsync(y + (int64_t)c * g.m, g.vout.p, g.m * sizeof(double), cudaMemcpyDeviceToHost, s));
    }
    h->check_status("cbx_geno_zt_v");
  });
}

extern "C" int cbx_geno_z_v(cbx_handle* h, int32_t nvec, const double* v, double* y) {
  return cbx_guard(h, [&] {
    geno::State& g = geno::state(h);
    CBX_REQUIRE(nvec > 0 && v && y, CBX_ERR_ARG, "bad vectors");
    CBX_CUDA(cudaSetDevice(h->device));
    cudaStream_t s = h->stream;
    g.vin.resize(g.m);
    g.vout.resize(g.n);
    for (int c = 0; c < nvec; ++c) {
      CBX_CUDA(cudaMemcpyAsync(g.vin.p, v + (int64_t)c * g.m, g.m * sizeof(double), cudaMemcpyHostToDevice, s));
      geno::z_device(h, g, g.vin.p, g.vout.p);
      CBX_CUDA(cudaMemcpyAsync(y + (int64_t)c * g.n, g.vout.p, g.n * sizeof(double), cudaMemcpyDeviceToHost, s));
    }
    h->check_status("cbx_geno_z_v");
  });
}

extern "C" int cbx_snp_effects(cbx_handle* h, const double* u_g, int64_t n_g, const double* Ginv,
                               double* effect, double* freq, double* total_2pq) {
  return cbx_guard(h, [&] {
    geno::State& g = geno::state(h);
    CBX_REQUIRE(u_g && effect, CBX_ERR_ARG, "bad vectors");
    CBX_REQUIRE(n_g == g.n, CBX_ERR_ARG,
                "u_g has " + std::to_string(n_g) + " entries; the genotypes have " + std::to_string(g.n) +
                    " samples");
    CBX_CUDA(cudaSetDevice(h->device));
    cudaStream_t s = h->stream;
    g.vin.resize(n_g);
    g.q.resize(n_g);
    g.vout.resize(2 * g.m);
    CBX_CUDA(cudaMemcpyAsync(g.vin.p, u_g, n_g * sizeof(double), cudaMemcpyHostToDevice, s));
    // q = G^-1 u_g (DenseMatrixAdapter::operator*, FP64)
    DevBuf<double> gtmp;
    const double* gd = nullptr;
    if (Ginv) {
      gtmp.resize((size_t)n_g * n_g);
      CBX_CUDA(cudaMemcpyAsync(gtmp.p, Ginv, (size_t)n_g * n_g * sizeof(double), cudaMemcpyHostToDevice, s));
      gd = gtmp.p;
    } else if (h->Ginv.p && h->Ginv_n == n_g) {
      gd = h->Ginv.p;
    }
    if (gd) {
      Libs& L = libs(h);
      const double one = 1.0, zero = 0.0;
      CBX_BLAS(cublasDgemv(L.blas, CUBLAS_OP_T, (int)n_g, (int)n_g, &one, gd, (int)n_g, g.vin.p, 1, &zero,
                           g.q.p, 1));
    } else {
      CBX_REQUIRE(h->mme && h->mme->has_dense && !h->mme->has_sparse && h->mme->q == n_g, CBX_ERR_STATE,
                  "Could not locate Ginv for back-solving (pass Ginv, or call cbx_invert_psd / "
                  "cbx_mme_set_qinv_dense with a dense inverse of order n)");
      qinv_apply(h, 1, g.vin.p, g.q.p);
    }
    geno::zt_device(h, g, g.q.p, nullptr, g.vout.p, g.vout.p + g.m);
    CBX_CUDA(cudaMemcpyAsync(effect, g.vout.p, g.m * sizeof(double), cudaMemcpyDeviceToHost, s));
    if (freq) CBX_CUDA(cudaMemcpyAsync(freq, g.vout.p + g.m, g.m * sizeof(double), cudaMemcpyDeviceToHost, s));
    if (total_2pq) CBX_CUDA(cudaMemcpyAsync(total_2pq, g.total(), sizeof(double), cudaMemcpyDeviceToHost, s));
    h->check_status("cbx_snp_effects");
  });
}
