// Ozaki-scheme DGEMM / ZGEMM on the INT8 tensor pipe (tcgen05 kind::i8).
//
// No reference counterpart: an FP64 GEMM (dgemm.rs:107 semantics, zgemm.rs:123
// through the 4M mapping) emulated with exact integer products.
//
//   1. Scaling: each row i of op(A) gets e_i with max_l |a_il| * 2^-e_i < 1, each
//      column j of op(B) gets f_j likewise (frexp exponents, reduced with
//      atomicMax -- exact and order independent).
//   2. Slicing: v = a * 2^-e_i (exact) is cut into S signed 7-bit slices,
//      v = sum_p A_p 2^-7p + r with A_p = trunc(2^7 r_{p-1}) in [-127, 127]
//      and |r| < 2^-7S: every step is exact in FP64.  Slices are stored
//      K-major, int8, [S][rows][kp] (kp = k rounded up to 16 bytes).
//   3. GEMM: for a 128 x 64 or 128 x 128 tile of C, the products A_p B_q^T with
//      p + q <= S+1 (S(S+1)/2 of them; the rest are below 2^-7(S+1)) are
//      accumulated in INT32 in TMEM, one accumulator per anti-diagonal d = p + q,
//      exactly as long as (#products on d) * 127^2 * kchunk < 2^30 -- K is cut into
//      chunks that satisfy it.  After each pass the epilogue warps combine the
//      diagonals in 64-bit integers (exact) and add them to FP64 registers, one
//      rounding per pass.
//   4. Epilogue: C = alpha * 2^(e_i + f_j) * acc + beta * C in FP64 (beta == 0
//      does not read C, as f64_edge / f32_edge.rs:37-58 do).
// Complex operands (ZGEMM) use the same 4M folding as the split-BF16 CGEMM:
// A'' = [Re A | Im A], B'' rows (2j, 2j+1) = ([Re B_j | -Im B_j], [Im B_j | Re B_j]);
// or, with the handle's complex mapping set to 3M, three real Ozaki GEMMs
// combined as Re = T1 - T2, Im = T3 - T1 - T2 (zgemm_ozaki_3m).
//
// Pipeline: warp 0 lane 0 = TMA producer (two K slabs of 64 bytes in four slots,
// 64-byte swizzle, 3-D maps over the slices); warp 1 = MMA issuer (kind::i8, M=128,
// N=64 or 128, K=32 per instruction), converged so that descriptors stay in
// uniform registers; warps 2-9 = epilogue.  All waits are bounded and report
// through the handle's status word.
//
// Bound: the int8 tensor pipe under the power cap.  DGEMM NN 4096^3: 1.97 -> 1.37 ms
// a call, the GEMM kernel 1.56 -> 1.18 ms (tensor pipe 56 -> 84% busy at 1.63 GHz);
// the same with one barrier per slab, 128-column tiles and one lane issuing 1.20.
#include "common.cuh"
#include "tc_common.cuh"

#include <climits>

namespace coral {
namespace {

constexpr int kOzBM = 128, kOzBK = 64;  // BK in int8 elements (64 bytes)
constexpr int kOzEpiWarps = 8;
constexpr int kOzThreads = 64 + 32 * kOzEpiWarps;

// ---- 1. exponents ---------------------------------------------------------------
// e[r] = max over l of the exponent of |op(X)(r, l)| (frexp: |v| 2^-e < 1),
// combined across column chunks with atomicMax, which is exact in any order.
// Complex: magnitude max(|re|, |im|) covers every real entry the 4M folding
// makes. Column-major rows (element (r, l) at X[r + l ld]): a thread owns a
// row and streams kExpChunkN columns with 8 loads in flight, so a warp reads
// 32 consecutive elements per column. K-major rows (element (r, l) at
// X[l + r ld]): a warp owns a row and streams kExpChunkK contiguous columns.
constexpr int kExpChunkN = 64, kExpChunkK = 256;

template <typename T>
__device__ __forceinline__ double mag(const T& a) {
  if constexpr (sizeof(T) == 16)
    return fmax(fabs(reinterpret_cast<const double2&>(a).x), fabs(reinterpret_cast<const double2&>(a).y));
  else
    return fabs(reinterpret_cast<const double&>(a));
}

template <typename T, bool kKMajorSrc>
__global__ void __launch_bounds__(256)
k_row_exponent(const T* __restrict__ X, size_t ld, int R, int Kd, int* __restrict__ e) {
  double m = 0.0;
  int r;
  if constexpr (!kKMajorSrc) {
    r = blockIdx.y * 256 + threadIdx.x;
    if (r >= R) return;
    const int l0 = blockIdx.x * kExpChunkN, l1 = min(Kd, l0 + kExpChunkN);
    const T* p = X + r;
    int l = l0;
    for (; l + 8 <= l1; l += 8) {
      T a[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) a[u] = __ldg(p + (size_t)(l + u) * ld);
#pragma unroll
      for (int u = 0; u < 8; ++u) m = fmax(m, mag(a[u]));
    }
    for (; l < l1; ++l) m = fmax(m, mag(__ldg(p + (size_t)l * ld)));
  } else {
    const int lane = threadIdx.x & 31;
    r = blockIdx.y * 8 + (threadIdx.x >> 5);
    if (r >= R) return;
    const int l0 = blockIdx.x * kExpChunkK;
    const T* p = X + (size_t)r * ld;
    T a[kExpChunkK / 32];
#pragma unroll
    for (int u = 0; u < kExpChunkK / 32; ++u) {
      const int l = l0 + lane + 32 * u;
      a[u] = l < Kd ? __ldg(p + l) : T{};
    }
#pragma unroll
    for (int u = 0; u < kExpChunkK / 32; ++u) m = fmax(m, mag(a[u]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane != 0) return;
  }
  if (m > 0.0) {
    int ex;
    frexp(m, &ex);  // m = f 2^ex, f in [0.5, 1) -> m 2^-ex < 1
    atomicMax(e + r, ex);
  }
}

// Launches k_row_exponent over R rows of Kd columns (e must hold INT_MIN-like
// starting values).
template <typename T>
coral_status_t launch_row_exponent(Handle* h, const T* X, size_t ld, int R, int Kd, bool kmajor, int* e) {
  if (kmajor) {
    const dim3 g((unsigned)((Kd + kExpChunkK - 1) / kExpChunkK), (unsigned)((R + 7) / 8));
    if (g.y > 65535) return CORAL_ERR_NOT_SUPPORTED;
    k_row_exponent<T, true><<<g, 256, 0, h->stream>>>(X, ld, R, Kd, e);
  } else {
    const dim3 g((unsigned)((Kd + kExpChunkN - 1) / kExpChunkN), (unsigned)((R + 255) / 256));
    if (g.y > 65535) return CORAL_ERR_NOT_SUPPORTED;
    k_row_exponent<T, false><<<g, 256, 0, h->stream>>>(X, ld, R, Kd, e);
  }
  return launch_status(h);
}

// ---- 2. slicing ----------------------------------------------------------------
// The digits of |a| 2^-ex to the base 128 are 7-bit fields of its mantissa,
// shifted: taking them with integer operations gives what the loop
// "r *= 128, t = trunc(r), r -= t" gives, without its 4 fp64 operations and
// conversions per slice.  `low`: the lowest 28 bits (slices 4-7), `high`: the
// 21 above (slices 1-3); the sign applies to every slice.
struct SliceBits {
  uint32_t high, low;
  bool neg;
};
__device__ __forceinline__ SliceBits slice_bits(double a, int ex) {
  long long bits = __double_as_longlong(a);
  int field = (int)((bits >> 52) & 0x7ff);
  SliceBits s{0u, 0u, bits < 0};
  if (field == 0x7ff) {  // NaN slices to 0; an infinity as trunc and the int conversion leave it
    if ((bits & 0xfffffffffffffll) == 0 && !s.neg) {
      s.high = 1u << 14;
      s.neg = true;
    }
    return s;
  }
  int e = field - 1022;  // frexp: |a| in [2^(e-1), 2^e)
  if (field == 0) {      // zero or subnormal: scaled up exactly
    bits = __double_as_longlong(a * 0x1p64);
    field = (int)((bits >> 52) & 0x7ff);
    if (field == 0) return s;
    e = field - 1022 - 64;
  }
  const unsigned long long mant = ((unsigned long long)bits & 0xfffffffffffffull) | 0x10000000000000ull;
  const int shift = min(max(4 + ex - e, 4), 63);  // ex >= e: the row's largest exponent
  const unsigned long long m = mant >> shift;
  s.high = (uint32_t)(m >> 28);
  s.low = (uint32_t)m & 0xfffffffu;
  return s;
}
__device__ __forceinline__ uint32_t slice_digit(const SliceBits& s, int p) {  // p = 0..6
  return p < 3 ? (s.high >> (14 - 7 * p)) & 127u : (s.low >> (42 - 7 * p)) & 127u;
}
template <int S>
__device__ __forceinline__ void slice_value(double a, int ex, int8_t (&out)[S]) {
  static_assert(S == 7, "seven 7-bit slices of a 49-bit fixed-point value");
  const SliceBits b = slice_bits(a, ex);
#pragma unroll
  for (int p = 0; p < S; ++p) {
    const int d = (int)slice_digit(b, p);
    out[p] = (int8_t)(b.neg ? -d : d);
  }
}

// Real: dst[p][row][l] for op(X) rows (K contiguous).  A CTA slices 32 rows x kDepth
// K values through shared memory, all of a thread's kDepth / 8 loads in flight; a
// thread writes kDepth / 8 K values of a row, as many bytes per slice (rows of kp
// bytes, a multiple of 16).  Bound: HBM (8 B read, 7 B written per element); 4096^2:
// 70 -> 50 us against the fp64 loop with byte stores (64 with words).  With 128 K
// values a matrix of few CTAs waits for 16 values one after the other: 32 there (see
// launch_slices).
template <int S, bool kKMajorSrc, int kDepth>
__global__ void __launch_bounds__(256)
k_slice_real(const double* __restrict__ X, size_t ld, int R, int Kd, const int* __restrict__ e,
             int8_t* __restrict__ dst, size_t kp, size_t piece) {
  // element (r, l) at r * kPitch + l + l / kPer: no bank conflicts either way
  constexpr int kRows = 32, kPer = kRows * kDepth / 256, kPitch = kDepth + 9, kWords = kPer / 4;
  __shared__ double tile[kRows * kPitch];
  const int r0 = blockIdx.y * kRows, l0 = blockIdx.x * kDepth;
  const int g = threadIdx.x & 7, row = threadIdx.x >> 3, r_out = r0 + row, l_out = l0 + kPer * g;
  const int ex = r_out < R ? e[r_out] : 0;
  double v[kPer];
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int i = threadIdx.x + 256 * q;
    const int r = r0 + (kKMajorSrc ? i / kDepth : i % kRows), l = l0 + (kKMajorSrc ? i % kDepth : i / kRows);
    v[q] = r < R && l < Kd ? __ldg(kKMajorSrc ? X + l + (size_t)r * ld : X + r + (size_t)l * ld) : 0.0;
  }
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int i = threadIdx.x + 256 * q, l = kKMajorSrc ? i % kDepth : i / kRows;
    tile[(kKMajorSrc ? i / kDepth : i % kRows) * kPitch + l + l / kPer] = v[q];
  }
  __syncthreads();
  if (r_out >= R || l_out >= (int)kp) return;
  uint32_t w[S][kWords];
#pragma unroll
  for (int a = 0; a < kWords; ++a) {
    uint32_t negs = 0u;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const SliceBits s = slice_bits(tile[row * kPitch + (kPer + 1) * g + 4 * a + b], ex);
#pragma unroll
      for (int p = 0; p < S; ++p) w[p][a] = (b ? w[p][a] : 0u) | slice_digit(s, p) << (8 * b);
      if (s.neg) negs |= 0xffu << (8 * b);
    }
#pragma unroll
    for (int p = 0; p < S; ++p) {  // bytes are 0..127: 0x80 - d, top bit flipped, is -d
      const uint32_t minus = (0x80808080u - w[p][a]) ^ 0x80808080u;
      w[p][a] = (w[p][a] & ~negs) | (minus & negs);
    }
  }
  int8_t* o = dst + (size_t)r_out * kp + l_out;
#pragma unroll
  for (int p = 0; p < S; ++p) {
    if constexpr (kWords == 4)
      *reinterpret_cast<uint4*>(o + p * piece) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
    else
      *reinterpret_cast<uint32_t*>(o + p * piece) = w[p][0];
  }
}

// 128 K values per CTA once there is a CTA of them for every SM.
template <int S>
coral_status_t launch_slices(Handle* h, const double* X, size_t ld, int R, int Kd, bool kmajor, const int* e,
                             int8_t* dst, size_t kp, size_t piece) {
  const unsigned rows = (unsigned)((R + 31) / 32);
  const dim3 deep((unsigned)((kp + 127) / 128), rows), flat((unsigned)((kp + 31) / 32), rows);
  const bool many = (size_t)deep.x * rows >= (size_t)h->sm_count;
  if (many && kmajor) k_slice_real<S, true, 128><<<deep, 256, 0, h->stream>>>(X, ld, R, Kd, e, dst, kp, piece);
  else if (many) k_slice_real<S, false, 128><<<deep, 256, 0, h->stream>>>(X, ld, R, Kd, e, dst, kp, piece);
  else if (kmajor) k_slice_real<S, true, 32><<<flat, 256, 0, h->stream>>>(X, ld, R, Kd, e, dst, kp, piece);
  else k_slice_real<S, false, 32><<<flat, 256, 0, h->stream>>>(X, ld, R, Kd, e, dst, kp, piece);
  return launch_status(h);
}

// Complex, 4M layout (see k_split_cplx in gemm_split.cu): A rows [Re | Im];
// B rows 2r = [Re | -Im], 2r+1 = [Im | Re].  Exponent per source row r.
template <int S, bool kKMajorSrc, bool kIsB>
__global__ void __launch_bounds__(256)
k_slice_cplx(const double2* __restrict__ X, size_t ld, int R, int Kd, bool conj,
             const int* __restrict__ e, int8_t* __restrict__ dst, size_t kp, size_t piece) {
  __shared__ double2 tile[32][33];
  const int r0 = blockIdx.y * 32, l0 = blockIdx.x * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (kKMajorSrc) {
      int r = r0 + ty + 8 * q, l = l0 + tx;
      tile[ty + 8 * q][tx] = (r < R && l < Kd) ? __ldg(X + l + (size_t)r * ld) : make_double2(0.0, 0.0);
    } else {
      int l = l0 + ty + 8 * q, r = r0 + tx;
      tile[tx][ty + 8 * q] = (r < R && l < Kd) ? __ldg(X + r + (size_t)l * ld) : make_double2(0.0, 0.0);
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int r = r0 + ty + 8 * q, l = l0 + tx;
    if (r >= R || l >= Kd) continue;
    double2 v = tile[ty + 8 * q][tx];
    if (conj) v.y = -v.y;
    int8_t sr[S], si[S], sn[S];
    slice_value<S>(v.x, e[r], sr);
    slice_value<S>(v.y, e[r], si);
#pragma unroll
    for (int p = 0; p < S; ++p) sn[p] = (int8_t)(-si[p]);
    if (!kIsB) {
      const size_t o = (size_t)r * kp;
#pragma unroll
      for (int p = 0; p < S; ++p) {
        dst[p * piece + o + l] = sr[p];
        dst[p * piece + o + Kd + l] = si[p];
      }
    } else {
      const size_t o0 = (size_t)(2 * r) * kp, o1 = o0 + kp;
#pragma unroll
      for (int p = 0; p < S; ++p) {
        dst[p * piece + o0 + l] = sr[p];
        dst[p * piece + o0 + Kd + l] = sn[p];
        dst[p * piece + o1 + l] = si[p];
        dst[p * piece + o1 + Kd + l] = sr[p];
      }
    }
  }
}

// ---- 3./4. integer GEMM and FP64 recombination -----------------------------------
struct OzMaps {
  CUtensorMap a[2];  // boxes of 3 and of 4 slices
  CUtensorMap b[2];
};

struct OzEpi {
  double* C;
  size_t ldc;
  int m, n;               // logical C (complex: n complex columns)
  const int* ea;          // row exponents of op(A) (length m)
  const int* eb;          // row exponents of B-rows (length n, or 2n complex)
  double alpha_re, alpha_im, beta_re, beta_im;
  int complex_out;
};

__device__ __forceinline__ void oz_tile_coords(int tile, int m_tiles, int n_tiles, int& mt, int& nt) {
  const int group = 16;
  const int per_group = group * n_tiles;
  const int g = tile / per_group;
  const int gm0 = g * group;
  const int gsz = min(group, m_tiles - gm0);
  const int within = tile - g * per_group;
  mt = gm0 + within % gsz;
  nt = within / gsz;
}

// How a tile of BN columns goes through the diagonals d = p + q = 2..8, with one
// BN-column accumulator each in the 512 TMEM columns: BN = 64 takes all seven in
// one pass over K; BN = 128 takes d = 5..8 (22 of the 28 products, all slices),
// then d = 2..4 (6 products, slices 1-3).  An int8 product of 128 x 64 x 32 reads
// as many bytes of shared memory per cycle as there are (48 cycles, 36 with A
// kept in the collector, 32 at the tensor core's peak); one of 128 x 128 x 32 runs
// at its peak of 64.  The wide tile takes more time to drain and write, and half
// as many tiles fill the last wave worse, so run_ozaki_gemm weighs both.
//
// The ring holds two K slabs, each in two slots: "high" (A_4..A_7, B_1..B_4) and
// "low" (A_1..A_3, B_5..B_7).  The products of a slab run as high x high, low A x
// high B, low x low, so a slab starts when its high slot has arrived, the low
// one is needed 10 products later, and the high one is free again 6 (BN = 64:
// 12) before the end: each load has more time than with one barrier per slab
// (80% of the tensor peak).  One barrier per slice had more still, but its
// single issuing lane could not keep up (76%).  In the second pass of BN = 128 a
// slot holds slices 1-3 of a whole slab.  A 3-D tensor map loads a slot's slices
// of one operand at once.
enum OzPart { kOzHighHigh, kOzLowHigh, kOzLowLow, kOzSecondPass };
template <int BN>
struct OzPlan {
  static constexpr int kPasses = BN == 64 ? 1 : 2;
  static constexpr int kLo = BN == 64 ? 2 : 5;       // first pass: d = kLo..8
  static constexpr int kSlabCycles = 56 * (BN == 64 ? 36 : 64);           // a K slab's 2 x 28 products
  static constexpr int kTileCycles = BN == 64 ? 16000 : 40000;            // drain and epilogue of a tile
  static constexpr uint32_t kATile = kOzBM * kOzBK, kBTile = BN * kOzBK;  // bytes per slice
  static constexpr uint32_t kHigh = 4 * (kATile + kBTile), kLow = 3 * (kATile + kBTile);
  static constexpr int kSlots = 4;                                        // high, low, high, low
  __device__ static constexpr uint32_t offset(int slot) { return (slot >> 1) * (kHigh + kLow) + (slot & 1) * kHigh; }
};

// The products of one part of a slab: A_p at a + (p - 1 from the part's first) etc.,
// as low descriptor words.  `first`: the slab starts the accumulators.
template <int BN, int kPart>
__device__ __forceinline__ void oz_issue(uint32_t a, uint32_t b, uint32_t hi, uint32_t tmem, bool first) {
  using P = OzPlan<BN>;
  constexpr uint32_t kIdesc = tc::idesc_s8_s32(kOzBM, BN);
  constexpr int lo = kPart == kOzSecondPass ? 2 : P::kLo, top = kPart == kOzSecondPass ? 4 : 8;
  constexpr int p0 = kPart == kOzHighHigh ? 4 : 1, p1 = kPart == kOzHighHigh ? 7 : 3;
  constexpr int b0 = kPart == kOzLowLow ? 5 : 1, b1 = kPart == kOzLowLow ? 7 : kPart == kOzSecondPass ? 3 : 4;
#pragma unroll
  for (int p = p0; p <= p1; ++p) {
    const int q0 = lo - p > b0 ? lo - p : b0, q1 = top - p < b1 ? top - p : b1;
#pragma unroll
    for (int kk = 0; kk < kOzBK / 32; ++kk) {
      const uint32_t ad = a + (uint32_t)(p - p0) * (P::kATile >> 4) + kk * 2;
#pragma unroll
      for (int q = q0; q <= q1; ++q) {
        const uint32_t acc = tmem + (p + q - lo) * BN;
        const uint32_t bd = b + (uint32_t)(q - b0) * (P::kBTile >> 4) + kk * 2;
        // which products meet their diagonal first: A_4's (d = 5..8), then A_1's (d = 2..4)
        const bool opens = kk == 0 && (kPart == kOzHighHigh ? p == 4 : kPart == kOzLowLow ? false : p == 1 && p + q <= 4);
        const uint32_t accum = opens && first ? 0u : 1u;
        // A_p stays in the collector over its products
        if (q0 == q1) tc::mma_i8_ca<tc::kCollectNone>(acc, ad, bd, hi, kIdesc, accum);
        else if (q == q0) tc::mma_i8_ca<tc::kCollectFill>(acc, ad, bd, hi, kIdesc, accum);
        else if (q == q1) tc::mma_i8_ca<tc::kCollectLastUse>(acc, ad, bd, hi, kIdesc, accum);
        else tc::mma_i8_ca<tc::kCollectUse>(acc, ad, bd, hi, kIdesc, accum);
      }
    }
  }
}

// sum[j] += 2^(-7 hi) * (diagonals lo..hi of column j, each 2^7 below the last):
// the integer combination is exact in 64 bits (below 2^51, see oz_chunk_slabs),
// so a pass costs one fp64 conversion -- an addition to 1.5 * 2^52 -- and one
// multiply-add per element, where converting each diagonal took seven.
template <int kLo, int kHi, int BN, int kCols>
__device__ __forceinline__ void oz_drain(uint32_t acc, double (&sum)[kCols]) {
  constexpr int kD = kHi - kLo + 1;
  constexpr double kScale = 1.0 / (double)(1ull << (7 * kHi));
#pragma unroll
  for (int c0 = 0; c0 < kCols; c0 += 8) {
    uint32_t r[kD][8];
#pragma unroll
    for (int d = 0; d < kD; ++d) tc::tmem_ld8(acc + d * BN + c0, r[d]);
    tc::tmem_wait_ld();
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      long long x = (int)r[0][j];
#pragma unroll
      for (int d = 1; d < kD; ++d) x = x * 128 + (int)r[d][j];
      const double v = __longlong_as_double(x + 0x4338000000000000ll) - 6755399441055744.0;
      sum[c0 + j] = fma(v, kScale, sum[c0 + j]);
    }
  }
}

// Eight accumulator columns from col0 (complex: four columns of C) of one row, for the
// kernel of single tiles: what is read of C and of the column exponents, then, apart
// from it, the results.  (The other kernels' epilogue through these is 8% slower at
// 2048^3: laid out at once the compiler moves the loads of all groups.)
struct OzGroup {
  double c[8];
  int e[8];
};
__device__ __forceinline__ void oz_load(const OzEpi& ep, int row, int col0, OzGroup& g) {
  const bool read_c = !(ep.beta_re == 0.0 && ep.beta_im == 0.0);
  if (!ep.complex_out) {
    const double* crow = ep.C + row;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int col = col0 + j;
      g.c[j] = (read_c && col < ep.n) ? crow[(size_t)col * ep.ldc] : 0.0;
      g.e[j] = col < ep.n ? max(ep.eb[col], -4000) : 0;
    }
  } else {
    const double2* crow = reinterpret_cast<const double2*>(ep.C) + row;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int col = col0 / 2 + j;
      const double2 c = (read_c && col < ep.n) ? crow[(size_t)col * ep.ldc] : make_double2(0.0, 0.0);
      g.c[2 * j] = c.x;
      g.c[2 * j + 1] = c.y;
      g.e[2 * j] = col < ep.n ? max(ep.eb[2 * col], -4000) : 0;
      g.e[2 * j + 1] = col < ep.n ? max(ep.eb[2 * col + 1], -4000) : 0;
    }
  }
}
__device__ __forceinline__ void oz_store(const OzEpi& ep, int row, int col0, int ei, const OzGroup& g,
                                         const double* sum) {
  const bool beta0 = ep.beta_re == 0.0 && ep.beta_im == 0.0;
  const bool beta1 = ep.beta_re == 1.0 && ep.beta_im == 0.0;
  if (!ep.complex_out) {
    double* crow = ep.C + row;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int col = col0 + j;
      if (col >= ep.n) continue;
      const double v = ep.alpha_re * ldexp(sum[j], ei + g.e[j]);
      crow[(size_t)col * ep.ldc] = beta0 ? v : beta1 ? g.c[j] + v : ep.beta_re * g.c[j] + v;
    }
  } else {
    double2* crow = reinterpret_cast<double2*>(ep.C) + row;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int col = col0 / 2 + j;
      if (col >= ep.n) continue;
      const double ar = ldexp(sum[2 * j], ei + g.e[2 * j]), ai = ldexp(sum[2 * j + 1], ei + g.e[2 * j + 1]);
      double2 v = make_double2(ep.alpha_re * ar - ep.alpha_im * ai, ep.alpha_re * ai + ep.alpha_im * ar);
      if (!beta0) {
        const double2 cv = make_double2(g.c[2 * j], g.c[2 * j + 1]);
        if (beta1) { v.x += cv.x; v.y += cv.y; }
        else {
          v.x += ep.beta_re * cv.x - ep.beta_im * cv.y;
          v.y += ep.beta_re * cv.y + ep.beta_im * cv.x;
        }
      }
      crow[(size_t)col * ep.ldc] = v;
    }
  }
}

// kOnce: one tile per CTA and one chunk of K (BN = 64 only).  The epilogue then goes from
// TMEM to C eight columns at a time, in a loop; laid out over all columns of a thread,
// the code runs once and what it costs is fetching it (DGEMM calls, us, with the small
// slicing tiles: 16^3 24.4 -> 18.4, 128^3 29.1 -> 25.0, 512^3 38.9 -> 34.8).
template <int S, int BN, bool kOnce>
__global__ void __launch_bounds__(kOzThreads, 1)
k_gemm_ozaki(const __grid_constant__ OzMaps maps, int kdim, int m_tiles, int n_tiles,
             int chunk_kb, OzEpi ep, unsigned* status, uint64_t limit_ns) {
  static_assert(S == 7, "the passes are laid out for seven slices");
  static_assert(!kOnce || BN == 64, "one pass");
  using P = OzPlan<BN>;
  constexpr uint32_t kATile = P::kATile, kBTile = P::kBTile;
  constexpr int kSlots = P::kSlots;
  constexpr int kCols = BN / 2;  // columns per epilogue thread

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = tc::align1024_shared(smem_raw);
  __shared__ __align__(8) uint64_t full_bar[kSlots], empty_bar[kSlots];
  __shared__ __align__(8) uint64_t acc_full, acc_empty, drain_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nk = (kdim + kOzBK - 1) / kOzBK;
  const int total_tiles = m_tiles * n_tiles;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kSlots; ++s) {
      tc::mbar_init(&full_bar[s], 1);
      tc::mbar_init(&empty_bar[s], 1);
    }
    tc::mbar_init(&acc_full, 1);
    tc::mbar_init(&acc_empty, kOzEpiWarps);
    tc::mbar_init(&drain_bar, 1);
    abort_flag = 0;
    tc::fence_mbar_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(&tmem_slot, 512);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;  // slots filled
      bool stop = false;
      // Waits for the next slot and announces `bytes`; its barrier and address.
      auto next_slot = [&](uint32_t bytes, uint64_t*& bar) -> uint8_t* {
        const int slot = it % kSlots;
        if ((it >= kSlots && !tc::mbar_wait(&empty_bar[slot], ((it / kSlots) - 1) & 1, limit_ns))) {
          atomicOr(status, kStatusTimeout);
          atomicExch(&abort_flag, 1);
          return nullptr;
        }
        if (*(volatile int*)&abort_flag) return nullptr;
        bar = &full_bar[slot];
        if (bytes) tc::mbar_expect_tx(bar, bytes);
        else tc::mbar_arrive(bar);
        ++it;
        return smem + P::offset(slot);
      };
      for (int tile = blockIdx.x; tile < total_tiles && !stop; tile += gridDim.x) {
        int mt, nt;
        oz_tile_coords(tile, m_tiles, n_tiles, mt, nt);
        const int m0 = mt * kOzBM, n0 = nt * BN;
        for (int c0 = 0; c0 < nk && !stop; c0 += chunk_kb) {
          const int c1 = min(nk, c0 + chunk_kb);
          uint64_t* bar;
          uint8_t* st;
          for (int kb = c0; kb < c1 && !stop; ++kb) {
            if (!(st = next_slot(P::kHigh, bar))) { stop = true; break; }
            tc::tma_load_3d(st, &maps.a[1], bar, kb * kOzBK, m0, 3);
            tc::tma_load_3d(st + 4 * kATile, &maps.b[1], bar, kb * kOzBK, n0, 0);
            if (!(st = next_slot(P::kLow, bar))) { stop = true; break; }
            tc::tma_load_3d(st, &maps.a[0], bar, kb * kOzBK, m0, 0);
            tc::tma_load_3d(st + 3 * kATile, &maps.b[0], bar, kb * kOzBK, n0, 4);
          }
          if (P::kPasses == 2) {
            for (int kb = c0; kb < c1 && !stop; ++kb) {
              if (!(st = next_slot(P::kLow, bar))) { stop = true; break; }
              tc::tma_load_3d(st, &maps.a[0], bar, kb * kOzBK, m0, 0);
              tc::tma_load_3d(st + 3 * kATile, &maps.b[0], bar, kb * kOzBK, n0, 0);
            }
            // an odd number of slabs leaves a low slot before the next high one
            if (((c1 - c0) & 1) && !stop && !next_slot(0, bar)) stop = true;
          }
        }
      }
      // every issued load lands before the CTA may exit
      for (int j = (it > kSlots ? it - kSlots : 0); j < it; ++j)
        tc::mbar_wait(&full_bar[j % kSlots], (j / kSlots) & 1, tc::kDrainNs);
    }
  } else if (warp == 1) {
    // ---- MMA issuer: the warp stays converged, one lane issues ----
    const bool lead = tc::elect_one();
    int it = 0, gc = 0;
    bool stop = false;
    const uint64_t ring = tc::desc_k_sw64(tc::smem_u32(smem));
    const uint32_t ring_lo = (uint32_t)ring, hi = (uint32_t)(ring >> 32);
    auto wait_all = [&](uint64_t* bar, uint32_t parity) {
      if (tc::mbar_wait_warp(bar, parity, limit_ns)) return true;
      if (lead) {
        atomicOr(status, kStatusTimeout);
        atomicExch(&abort_flag, 1);
      }
      stop = true;
      return false;
    };
    auto take_slot = [&](int& slot) {
      slot = it % kSlots;
      const bool ok = wait_all(&full_bar[slot], (it / kSlots) & 1);
      tc::tc_fence_after();
      ++it;
      return ok;
    };
    auto at = [&](int slot) { return ring_lo + (P::offset(slot) >> 4); };
    for (int tile = blockIdx.x; tile < total_tiles && !stop; tile += gridDim.x) {
      for (int c0 = 0; c0 < nk && !stop; c0 += chunk_kb) {
        const int c1 = min(nk, c0 + chunk_kb);
        // the epilogue must have drained the previous pass
        if (gc >= 1 && !wait_all(&acc_empty, (gc - 1) & 1)) break;
        tc::tc_fence_after();
        for (int kb = c0; kb < c1; ++kb) {
          int high, low;
          if (!take_slot(high)) break;
          const uint32_t ha = at(high), hb = ha + (4 * kATile >> 4);
          if (lead) oz_issue<BN, kOzHighHigh>(ha, hb, hi, tmem, kb == c0);
          if (!take_slot(low)) break;
          const uint32_t la = at(low), lb = la + (3 * kATile >> 4);
          if (lead) {
            oz_issue<BN, kOzLowHigh>(la, hb, hi, tmem, kb == c0);
            tc::mma_commit(&empty_bar[high]);
            oz_issue<BN, kOzLowLow>(la, lb, hi, tmem, kb == c0);
            tc::mma_commit(&empty_bar[low]);
          }
        }
        if (lead) tc::mma_commit(&acc_full);
        ++gc;
        if (P::kPasses == 2 && !stop) {
          if (!wait_all(&acc_empty, (gc - 1) & 1)) break;
          tc::tc_fence_after();
          int slot;
          for (int kb = c0; kb < c1; ++kb) {
            if (!take_slot(slot)) break;
            if (lead) {
              oz_issue<BN, kOzSecondPass>(at(slot), at(slot) + (3 * kATile >> 4), hi, tmem, kb == c0);
              tc::mma_commit(&empty_bar[slot]);
            }
          }
          if (((c1 - c0) & 1) && !stop && take_slot(slot) && lead) tc::mma_commit(&empty_bar[slot]);
          if (lead) tc::mma_commit(&acc_full);
          ++gc;
        }
      }
    }
    if (lead) {  // every product issued completes before TMEM is released
      tc::mma_commit(&drain_bar);
      tc::mbar_wait(&drain_bar, 0, tc::kDrainNs);
    }
    __syncwarp();
  } else {
    const int ew = warp - 2;
    const int quad = warp & 3;
    const int half = ew >> 2;
    const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
    const bool beta0 = ep.beta_re == 0.0 && ep.beta_im == 0.0;
    const bool beta1 = ep.beta_re == 1.0 && ep.beta_im == 0.0;
    int gc = 0;
    bool stop = false;
    if constexpr (kOnce) {
      int mt, nt;
      oz_tile_coords(blockIdx.x, m_tiles, n_tiles, mt, nt);
      const int row = mt * kOzBM + quad * 32 + lane, col0 = nt * BN + half * kCols;
      const bool in = row < ep.m;
      const int ei = in ? max(ep.ea[row], -4000) : 0;
      OzGroup g;
      if (in) oz_load(ep, row, col0, g);   // on its way while the products run
      if (!tc::mbar_wait_warp(&acc_full, 0, limit_ns)) {
        atomicOr(status, kStatusTimeout);
        stop = true;
      }
      tc::tc_fence_after();
      stop = stop || tc::flag_warp(&abort_flag);
      const uint32_t acc = tmem + half * kCols + lane_base;
#pragma unroll 1
      for (int c = 0; c < kCols && !stop; c += 8) {
        double sum[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        oz_drain<5, 8, BN>(acc + 3 * BN + c, sum);
        oz_drain<2, 4, BN>(acc + c, sum);
        if (in) {
          const OzGroup now = g;
          if (c + 8 < kCols) oz_load(ep, row, col0 + c + 8, g);
          oz_store(ep, row, col0 + c, ei, now, sum);
        }
        __syncwarp();
      }
      stop = true;
    }
    for (int tile = blockIdx.x; tile < total_tiles && !stop; tile += gridDim.x) {
      int mt, nt;
      oz_tile_coords(tile, m_tiles, n_tiles, mt, nt);
      double sum[kCols];
#pragma unroll
      for (int j = 0; j < kCols; ++j) sum[j] = 0.0;
      // C into L2 while the products run (a warp's 32 rows are two or four lines a column)
      if (!beta0) {
        const int prow = mt * kOzBM + quad * 32 + lane, width = ep.complex_out ? 2 : 1;
        const int pcol = (nt * BN + half * kCols) / width, pcols = kCols / width;
        if (prow < ep.m && (lane & (16 / width - 1)) == 0)
          for (int j = 0; j < pcols && pcol + j < ep.n; ++j)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(ep.C + ((size_t)prow + (size_t)(pcol + j) * ep.ldc) * width));
      }
      for (int c0 = 0; c0 < nk && !stop; c0 += chunk_kb) {
#pragma unroll
        for (int pass = 0; pass < P::kPasses; ++pass, ++gc) {
          if (stop || !tc::mbar_wait_warp(&acc_full, gc & 1, limit_ns)) {
            atomicOr(status, kStatusTimeout);
            stop = true;
            break;
          }
          tc::tc_fence_after();
          const uint32_t acc = tmem + half * kCols + lane_base;
          if (BN == 64) {
            oz_drain<5, 8, BN>(acc + 3 * BN, sum);
            oz_drain<2, 4, BN>(acc, sum);
          } else if (pass == 0) {
            oz_drain<5, 8, BN>(acc, sum);
          } else {
            oz_drain<2, 4, BN>(acc, sum);
          }
          tc::tc_fence_before();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&acc_empty);
        }
      }
      if (stop || tc::flag_warp(&abort_flag)) break;
      const int row = mt * kOzBM + quad * 32 + lane;
      if (row >= ep.m) continue;
      const int ei = max(ep.ea[row], -4000);  // all-zero rows keep the INT_MIN-like fill
      const int col0 = nt * BN + half * kCols;
      // All C loads (and column exponents) of the tile row before any store:
      // a store followed by a load the compiler cannot prove disjoint would
      // cost a memory round trip per column.
      constexpr int G = 8;  // columns per group of loads
      if (!ep.complex_out) {
        double* crow = ep.C + row;
#pragma unroll
        for (int g = 0; g < kCols; g += G) {
          double cv[G];
          int ej[G];
#pragma unroll
          for (int j = 0; j < G; ++j) {
            const int col = col0 + g + j;
            cv[j] = (!beta0 && col < ep.n) ? crow[(size_t)col * ep.ldc] : 0.0;
            ej[j] = col < ep.n ? max(ep.eb[col], -4000) : 0;
          }
#pragma unroll
          for (int j = 0; j < G; ++j) {
            const int col = col0 + g + j;
            if (col >= ep.n) continue;
            const double v = ep.alpha_re * ldexp(sum[g + j], ei + ej[j]);
            crow[(size_t)col * ep.ldc] = beta0 ? v : beta1 ? cv[j] + v : ep.beta_re * cv[j] + v;
          }
        }
      } else {
        double2* crow = reinterpret_cast<double2*>(ep.C) + row;
#pragma unroll
        for (int g = 0; g < kCols / 2; g += G / 2) {
        double2 cvs[G / 2];
#pragma unroll
        for (int j0 = 0; j0 < G / 2; ++j0) {
          const int col = col0 / 2 + g + j0;
          cvs[j0] = (!beta0 && col < ep.n) ? crow[(size_t)col * ep.ldc] : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int j0 = 0; j0 < G / 2; ++j0) {
          const int j = g + j0;
          const int col = col0 / 2 + j;
          if (col >= ep.n) continue;
          const double ar = ldexp(sum[2 * j], ei + max(ep.eb[2 * col], -4000));
          const double ai = ldexp(sum[2 * j + 1], ei + max(ep.eb[2 * col + 1], -4000));
          double2 v = make_double2(ep.alpha_re * ar - ep.alpha_im * ai, ep.alpha_re * ai + ep.alpha_im * ar);
          if (!beta0) {
            const double2 cv = cvs[j0];
            if (beta1) { v.x += cv.x; v.y += cv.y; }
            else {
              v.x += ep.beta_re * cv.x - ep.beta_im * cv.y;
              v.y += ep.beta_re * cv.y + ep.beta_im * cv.x;
            }
          }
          crow[(size_t)col * ep.ldc] = v;
        }
        }
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 1) tc::tmem_dealloc(tmem, 512);
}

// K slabs per exact chunk: (products on the fullest diagonal) * 127^2 * k < 2^30, so
// that a diagonal fits INT32 and four of them, 2^7 apart, stay below 2^51.
template <int S>
int oz_chunk_slabs() {
  const long long kmax = (long long)(1 << 30) / (127LL * 127LL * S);
  return (int)(kmax / kOzBK);
}

template <int S, int BN, bool kOnce>
coral_status_t launch_ozaki(Handle* h, const OzMaps& maps, int mr, int nr, int kd, const OzEpi& ep) {
  const size_t smem = 2 * ((size_t)OzPlan<BN>::kHigh + OzPlan<BN>::kLow) + 1024;
  static uint64_t attr_devices = 0;  // bit d: attribute set on device d
  const uint64_t bit = h->device < 64 ? (1ull << h->device) : 0;
  if (!(attr_devices & bit) || !bit) {
    CORAL_CUDA(h, cudaFuncSetAttribute(k_gemm_ozaki<S, BN, kOnce>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_devices |= bit;
  }
  const int m_tiles = (mr + kOzBM - 1) / kOzBM, n_tiles = (nr + BN - 1) / BN;
  const int tiles = m_tiles * n_tiles;
  const int grid = tiles < h->sm_count ? tiles : h->sm_count;
  timed_begin(h);
  k_gemm_ozaki<S, BN, kOnce><<<grid, kOzThreads, smem, h->stream>>>(maps, kd, m_tiles, n_tiles, oz_chunk_slabs<S>(), ep,
                                                             &h->words->status, h->wait_limit * 32ull);
  coral_status_t s = launch_status(h);
  timed_end(h);
  return s;
}

template <int S>
coral_status_t run_ozaki_gemm(Handle* h, const int8_t* ap, size_t a_piece, int mr, const int8_t* bp,
                              size_t b_piece, int nr, int kd, size_t kp, const OzEpi& ep) {
  // Waves of tiles times a tile's cycles.  Both sides measured (us, 64 / 128 wide):
  // 4096^3 1321 / 1175, 2048^3 198 / 185, 1000^3 42 / 73, 4096 x 512 x 64 25 / 32.
  const long long slabs = (kd + kOzBK - 1) / kOzBK;
  auto cost = [&](int bn, int slab_cycles, int tile_cycles) {
    const long long tiles = (long long)((mr + kOzBM - 1) / kOzBM) * ((nr + bn - 1) / bn);
    return (tiles + h->sm_count - 1) / h->sm_count * (slabs * slab_cycles + tile_cycles);
  };
  const int bn = cost(128, OzPlan<128>::kSlabCycles, OzPlan<128>::kTileCycles) <=
                         cost(64, OzPlan<64>::kSlabCycles, OzPlan<64>::kTileCycles)
                     ? 128
                     : 64;
  OzMaps maps;
  std::memset(&maps, 0, sizeof(maps));
  for (int i = 0; i < 2; ++i) {
    if (!encode_slices_map(&maps.a[i], ap, kd, mr, S, kp, a_piece, kOzBK, kOzBM, 3 + i) ||
        !encode_slices_map(&maps.b[i], bp, kd, nr, S, kp, b_piece, kOzBK, bn, 3 + i))
      return CORAL_ERR_NOT_SUPPORTED;
  }
  if (bn == 128) return launch_ozaki<S, 128, false>(h, maps, mr, nr, kd, ep);
  const long long tiles = (long long)((mr + kOzBM - 1) / kOzBM) * ((nr + 63) / 64);
  if (tiles <= h->sm_count && slabs <= oz_chunk_slabs<S>()) return launch_ozaki<S, 64, true>(h, maps, mr, nr, kd, ep);
  return launch_ozaki<S, 64, false>(h, maps, mr, nr, kd, ep);
}

constexpr int kOzSlices = 7;

// Row pitch of the slices in bytes: a multiple of 16 (TMA's strides), and of 128
// where K is deep enough for that to cost little memory, so that a slab's 64-byte
// row never straddles two lines.
size_t slice_pitch(size_t k) {
  return k >= 1024 ? (k + 127) & ~size_t(127) : (k + 15) & ~size_t(15);
}

// Device bytes the real Ozaki GEMM needs for its slices and exponents.
size_t dgemm_ozaki_bytes(size_t m, size_t n, size_t k) {
  constexpr int S = kOzSlices;
  const size_t kp = slice_pitch(k);
  const size_t a_bytes = (S * m * kp + 1023) & ~size_t(1023);
  const size_t b_bytes = (S * n * kp + 1023) & ~size_t(1023);
  const size_t e_bytes = ((m + n) * sizeof(int) + 255) & ~size_t(255);
  return a_bytes + b_bytes + e_bytes;
}

// The real Ozaki GEMM with its slices and exponents in `sc`
// (dgemm_ozaki_bytes(m, n, k) bytes, 1024-byte aligned).
coral_status_t dgemm_ozaki_core(Handle* h, char* sc, int op_a, int op_b, size_t m, size_t n, size_t k,
                                double alpha, const double* A, size_t lda, const double* B,
                                size_t ldb, double beta, double* C, size_t ldc) {
  constexpr int S = kOzSlices;
  const size_t kp = slice_pitch(k);
  const size_t a_piece = m * kp, b_piece = n * kp;
  const size_t a_bytes = (S * a_piece + 1023) & ~size_t(1023);
  const size_t b_bytes = (S * b_piece + 1023) & ~size_t(1023);
  int8_t* ap = reinterpret_cast<int8_t*>(sc);
  int8_t* bp = reinterpret_cast<int8_t*>(sc + a_bytes);
  int* ea = reinterpret_cast<int*>(sc + a_bytes + b_bytes);
  int* eb = ea + m;
  CORAL_CUDA(h, cudaMemsetAsync(ea, 0x80, (m + n) * sizeof(int), h->stream));  // INT_MIN-ish
  const bool a_km = op_a != CORAL_NO_TRANSPOSE, b_km = op_b == CORAL_NO_TRANSPOSE;
  coral_status_t s = launch_row_exponent(h, A, lda, (int)m, (int)k, a_km, ea);
  if (s != CORAL_OK) return s;
  if ((s = launch_row_exponent(h, B, ldb, (int)n, (int)k, b_km, eb)) != CORAL_OK) return s;
  if ((s = launch_slices<S>(h, A, lda, (int)m, (int)k, a_km, ea, ap, kp, a_piece)) != CORAL_OK) return s;
  if ((s = launch_slices<S>(h, B, ldb, (int)n, (int)k, b_km, eb, bp, kp, b_piece)) != CORAL_OK) return s;
  OzEpi ep{C, ldc, (int)m, (int)n, ea, eb, alpha, 0.0, beta, 0.0, 0};
  return run_ozaki_gemm<S>(h, ap, a_piece, (int)m, bp, b_piece, (int)n, (int)k, kp, ep);
}

coral_status_t dgemm_ozaki_impl(Handle* h, int op_a, int op_b, size_t m, size_t n, size_t k,
                                double alpha, const double* A, size_t lda, const double* B,
                                size_t ldb, double beta, double* C, size_t ldc) {
  char* sc = static_cast<char*>(scratch(h, dgemm_ozaki_bytes(m, n, k)));
  if (!sc) return CORAL_ERR_ALLOC;
  return dgemm_ozaki_core(h, sc, op_a, op_b, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
}

// 3M operands: the real matrices Re, Im and Re + Im of op(X) (conjugated when
// `conj`), R x L, column-major with leading dimension R.  Element (r, l) of
// op(X) is X[r + l * ld] (trans == false) or X[l + r * ld]; 32 x 32 tiles
// through shared memory so both the loads and the stores are coalesced.
__global__ void __launch_bounds__(256)
k_cplx_parts(const double2* __restrict__ X, size_t ld, bool trans, bool conj, int R, int L,
             double* __restrict__ re, double* __restrict__ im, double* __restrict__ sum) {
  __shared__ double2 tile[32][33];
  const int r0 = blockIdx.y * 32, l0 = blockIdx.x * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (trans) {  // contiguous along l
      const int r = r0 + ty + 8 * q, l = l0 + tx;
      if (r < R && l < L) tile[ty + 8 * q][tx] = X[l + (size_t)r * ld];
    } else {      // contiguous along r
      const int l = l0 + ty + 8 * q, r = r0 + tx;
      if (r < R && l < L) tile[tx][ty + 8 * q] = X[r + (size_t)l * ld];
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int l = l0 + ty + 8 * q, r = r0 + tx;
    if (r < R && l < L) {
      double2 v = tile[tx][ty + 8 * q];
      if (conj) v.y = -v.y;
      const size_t o = r + (size_t)l * R;
      re[o] = v.x;
      im[o] = v.y;
      sum[o] = v.x + v.y;
    }
  }
}

// C = alpha (T1 - T2 + i (T3 - T1 - T2)) + beta C, T* m x n with ld m.
__global__ void k_combine_3m_z(const double* __restrict__ t1, const double* __restrict__ t2,
                               const double* __restrict__ t3, int m, int n, double2 alpha, double2 beta,
                               double2* __restrict__ C, size_t ldc) {
  const size_t total = (size_t)m * n;
  const bool beta0 = beta.x == 0.0 && beta.y == 0.0;
  const bool beta1 = beta.x == 1.0 && beta.y == 0.0;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (size_t)gridDim.x * blockDim.x) {
    const double a = t1[t], b = t2[t], c3 = t3[t];
    const double re = a - b, im = c3 - a - b;
    double2 v = make_double2(alpha.x * re - alpha.y * im, alpha.x * im + alpha.y * re);
    double2* cp = C + t % m + (t / m) * ldc;
    if (!beta0) {
      const double2 cv = *cp;
      if (beta1) { v.x += cv.x; v.y += cv.y; }
      else {
        v.x += beta.x * cv.x - beta.y * cv.y;
        v.y += beta.x * cv.y + beta.y * cv.x;
      }
    }
    *cp = v;
  }
}

// ZGEMM by the 3M mapping: three real Ozaki GEMMs of m x n x k (Re A Re B,
// Im A Im B, (Re A + Im A)(Re B + Im B)) into fp64 workspace, then the
// combine.  Three quarters of the 4M work; Im C = T3 - T1 - T2, whose error is
// bounded by (|Re A| + |Im A|)(|Re B| + |Im B|) instead of |A| |B| per term.
coral_status_t zgemm_ozaki_3m(Handle* h, int op_a, int op_b, size_t m, size_t n, size_t k,
                              double2 alpha, const double2* A, size_t lda, const double2* B,
                              size_t ldb, double2 beta, double2* C, size_t ldc) {
  auto up = [](size_t b) { return (b + 1023) & ~size_t(1023); };
  const size_t pa = up(m * k * sizeof(double)), pb = up(k * n * sizeof(double));
  const size_t pt = up(m * n * sizeof(double));
  const size_t oz = dgemm_ozaki_bytes(m, n, k);
  char* sc = static_cast<char*>(scratch(h, 3 * pa + 3 * pb + 3 * pt + oz));
  if (!sc) return CORAL_ERR_ALLOC;
  double* ar[3];
  double* br[3];
  double* t[3];
  for (int i = 0; i < 3; ++i) {
    ar[i] = reinterpret_cast<double*>(sc + i * pa);
    br[i] = reinterpret_cast<double*>(sc + 3 * pa + i * pb);
    t[i] = reinterpret_cast<double*>(sc + 3 * pa + 3 * pb + i * pt);
  }
  char* ozs = sc + 3 * pa + 3 * pb + 3 * pt;
  // op(A): m x k; op(B): k x n
  const dim3 ga((unsigned)((k + 31) / 32), (unsigned)((m + 31) / 32));
  k_cplx_parts<<<ga, 256, 0, h->stream>>>(A, lda, op_a != CORAL_NO_TRANSPOSE, op_a == CORAL_CONJ_TRANSPOSE,
                                          (int)m, (int)k, ar[0], ar[1], ar[2]);
  coral_status_t s = launch_status(h);
  if (s != CORAL_OK) return s;
  const dim3 gb((unsigned)((n + 31) / 32), (unsigned)((k + 31) / 32));
  k_cplx_parts<<<gb, 256, 0, h->stream>>>(B, ldb, op_b != CORAL_NO_TRANSPOSE, op_b == CORAL_CONJ_TRANSPOSE,
                                          (int)k, (int)n, br[0], br[1], br[2]);
  if ((s = launch_status(h)) != CORAL_OK) return s;
  for (int i = 0; i < 3; ++i) {
    s = dgemm_ozaki_core(h, ozs, CORAL_NO_TRANSPOSE, CORAL_NO_TRANSPOSE, m, n, k, 1.0, ar[i], m, br[i], k,
                         0.0, t[i], m);
    if (s != CORAL_OK) return s;
  }
  const unsigned g = stream_grid(m * n, 256 * 4, h->sm_count, 8);
  k_combine_3m_z<<<g, 256, 0, h->stream>>>(t[0], t[1], t[2], (int)m, (int)n, alpha, beta, C, ldc);
  return launch_status(h);
}

coral_status_t zgemm_ozaki_impl(Handle* h, int op_a, int op_b, size_t m, size_t n, size_t k,
                                double2 alpha, const double2* A, size_t lda, const double2* B,
                                size_t ldb, double2 beta, double2* C, size_t ldc) {
  constexpr int S = kOzSlices;
  const size_t k2 = 2 * k;
  const size_t kp = slice_pitch(k2);
  const size_t a_piece = m * kp, b_piece = 2 * n * kp;
  const size_t a_bytes = (S * a_piece + 1023) & ~size_t(1023);
  const size_t b_bytes = (S * b_piece + 1023) & ~size_t(1023);
  const size_t e_bytes = ((m + 2 * n + n) * sizeof(int) + 255) & ~size_t(255);
  char* sc = static_cast<char*>(scratch(h, a_bytes + b_bytes + e_bytes));
  if (!sc) return CORAL_ERR_ALLOC;
  int8_t* ap = reinterpret_cast<int8_t*>(sc);
  int8_t* bp = reinterpret_cast<int8_t*>(sc + a_bytes);
  int* ea = reinterpret_cast<int*>(sc + a_bytes + b_bytes);
  int* ebs = ea + m;          // per source column j of op(B) (length n)
  int* eb2 = ebs + n;         // per B'' row (length 2n)
  CORAL_CUDA(h, cudaMemsetAsync(ea, 0x80, (m + n) * sizeof(int), h->stream));
  const bool a_km = op_a != CORAL_NO_TRANSPOSE, b_km = op_b == CORAL_NO_TRANSPOSE;
  coral_status_t s = launch_row_exponent(h, A, lda, (int)m, (int)k, a_km, ea);
  if (s != CORAL_OK) return s;
  if ((s = launch_row_exponent(h, B, ldb, (int)n, (int)k, b_km, ebs)) != CORAL_OK) return s;
  // B'' rows 2j and 2j+1 share column j's exponent.
  CORAL_CUDA(h, cudaMemcpy2DAsync(eb2, 2 * sizeof(int), ebs, sizeof(int), sizeof(int), n,
                                  cudaMemcpyDeviceToDevice, h->stream));
  CORAL_CUDA(h, cudaMemcpy2DAsync(eb2 + 1, 2 * sizeof(int), ebs, sizeof(int), sizeof(int), n,
                                  cudaMemcpyDeviceToDevice, h->stream));
  // (row tails past k2 stay undefined: the tensor maps end at k2 and fill zeros)
  const bool ca = op_a == CORAL_CONJ_TRANSPOSE, cbj = op_b == CORAL_CONJ_TRANSPOSE;
  const dim3 ga((unsigned)((k + 31) / 32), (unsigned)((m + 31) / 32));  // 32 x 32 slicing tiles
  const dim3 gb((unsigned)((k + 31) / 32), (unsigned)((n + 31) / 32));
  if (a_km) k_slice_cplx<S, true, false><<<ga, 256, 0, h->stream>>>(A, lda, (int)m, (int)k, ca, ea, ap, kp, a_piece);
  else k_slice_cplx<S, false, false><<<ga, 256, 0, h->stream>>>(A, lda, (int)m, (int)k, ca, ea, ap, kp, a_piece);
  if ((s = launch_status(h)) != CORAL_OK) return s;
  if (b_km) k_slice_cplx<S, true, true><<<gb, 256, 0, h->stream>>>(B, ldb, (int)n, (int)k, cbj, ebs, bp, kp, b_piece);
  else k_slice_cplx<S, false, true><<<gb, 256, 0, h->stream>>>(B, ldb, (int)n, (int)k, cbj, ebs, bp, kp, b_piece);
  if ((s = launch_status(h)) != CORAL_OK) return s;
  OzEpi ep{reinterpret_cast<double*>(C), ldc, (int)m, (int)n, ea, eb2,
           alpha.x, alpha.y, beta.x, beta.y, 1};
  return run_ozaki_gemm<S>(h, ap, a_piece, (int)m, bp, b_piece, (int)(2 * n), (int)k2, kp, ep);
}

}  // namespace

coral_status_t enqueue_dgemm_ozaki(Handle* h, int op_a, int op_b, size_t m, size_t n, size_t k,
                                   double alpha, const double* A, size_t lda, const double* B,
                                   size_t ldb, double beta, double* C, size_t ldc) {
  if (m > (size_t)INT32_MAX / 2 || n > (size_t)INT32_MAX / 2 || k > (size_t)INT32_MAX / 2)
    return CORAL_ERR_NOT_SUPPORTED;
  return dgemm_ozaki_impl(h, op_a, op_b, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
}

coral_status_t enqueue_zgemm_ozaki(Handle* h, int op_a, int op_b, size_t m, size_t n, size_t k,
                                   double2 alpha, const double2* A, size_t lda, const double2* B,
                                   size_t ldb, double2 beta, double2* C, size_t ldc) {
  if (m > (size_t)INT32_MAX / 4 || n > (size_t)INT32_MAX / 4 || k > (size_t)INT32_MAX / 4)
    return CORAL_ERR_NOT_SUPPORTED;
  if (h->complex_mapping == CORAL_COMPLEX_3M)
    return zgemm_ozaki_3m(h, op_a, op_b, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
  return zgemm_ozaki_impl(h, op_a, op_b, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
}

}  // namespace coral
