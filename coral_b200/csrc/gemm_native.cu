// Native-precision GEMM: C <- alpha * op(A) op(B) + beta * C, column-major, for
// float, double, complex64 and complex128.
//
// Replaces CORAL's packing + macro/micro-kernel subsystem
// (coral-aarch64/src/level3/*_packers.rs, *_macro_kernel.rs, microkernel/).
// A CTA computes a 64 x 64 tile of C (large fp32: 128 x 128).  Slabs of op(A) and
// op(B) stream into a shared-memory ring with cp.async -- 16 bytes at a time
// where base and leading dimension allow, one element at a time otherwise, so
// odd leading dimensions take the same kernel and the same order of summation
// as aligned ones.  fp32 and complex64 multiply on the FMA pipe with packed
// pairs (fma.rn.f32x2), fp64 and complex128 on the fp64 tensor path (8 x 8 x 4
// products; the measured peak, 37.0 TFLOP/s, is the DFMA pipe's 36.6, at a
// sixteenth of the instructions and a quarter of the shared-memory reads).
// Conjugation is a sign, applied to fragments or at the end.
//
// Where the tiles of C leave SMs idle, K is split over the 2, 4 or 8 CTAs of a
// cluster; each CTA then sums its share of the tile from its peers' shared
// memory in rank order (the result does not depend on timing) and writes it.
//
// Bound: the FMA / fp64 pipe.  One B200, graph replay, against the kernels this
// one replaced (128 x 128 TMA-fed and 64 x 64 register-staged tiles, whole K):
//   SGEMM NN  512^3  63 -> 13.3 us    2048^3 418 -> 372 us   4096^3 2.81 -> 2.47 ms (55.7 TFLOP/s)
//   SGEMM TN  513 x 511 x 517 102 -> 16 us
//   DGEMM TN  777 x 1001 x 1501 238 -> 94 us; NN 4096^3 5.36 -> 4.07 ms (33.8 TFLOP/s, 91% of the pipe)
//   CGEMM NN  2048^3 2.55 -> 1.25 ms; ZGEMM CC 2048^3 4.37 -> 2.07 ms (33.2 TFLOP/s)
//
// Epilogue follows f32_edge.rs:37-58: beta == 0 writes alpha*acc without
// reading C, beta == 1 accumulates, else beta*C + alpha*acc.  alpha == 0 or
// k == 0 only scales C (sgemm_nn.rs:29-45, cgemm_nn.rs scale-only path).
#include "common.cuh"
#include "tc_common.cuh"

#include <climits>
#include <cmath>
#include <type_traits>

namespace coral {
namespace {

// ---- asynchronous staging -----------------------------------------------------
// Copies kBytes to shared memory, or writes zeros when !ok (src stays valid).
template <int kBytes>
__device__ __forceinline__ void cp_async(uint32_t dst, const void* src, bool ok) {
  const int n = ok ? kBytes : 0;
  if constexpr (kBytes == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(kBytes), "r"(n)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kLeft>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(kLeft) : "memory");
}

// ---- arithmetic -----------------------------------------------------------------
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
// D (8 x 8) += A (8 x 4) B (4 x 8): lane l holds A[l / 4][l % 4], B[l % 4][l / 4]
// and D[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}
__device__ __forceinline__ double flip(double a, long long sign) {
  return __longlong_as_double(__double_as_longlong(a) ^ sign);
}

template <typename T> struct Ops;
template <> struct Ops<float> {
  static __host__ __device__ bool zero(float a) { return a == 0.f; }
  static __host__ __device__ bool one(float a) { return a == 1.f; }
  static __device__ float mul(float a, float b) { return a * b; }
  static __device__ float add(float a, float b) { return a + b; }
};
template <> struct Ops<double> {
  static __host__ __device__ bool zero(double a) { return a == 0.0; }
  static __host__ __device__ bool one(double a) { return a == 1.0; }
  static __device__ double mul(double a, double b) { return a * b; }
  static __device__ double add(double a, double b) { return a + b; }
};
template <> struct Ops<float2> {
  static __host__ __device__ bool zero(float2 a) { return a.x == 0.f && a.y == 0.f; }
  static __host__ __device__ bool one(float2 a) { return a.x == 1.f && a.y == 0.f; }
  static __device__ float2 mul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
  }
  static __device__ float2 add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
};
template <> struct Ops<double2> {
  static __host__ __device__ bool zero(double2 a) { return a.x == 0.0 && a.y == 0.0; }
  static __host__ __device__ bool one(double2 a) { return a.x == 1.0 && a.y == 0.0; }
  static __device__ double2 mul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
  }
  static __device__ double2 add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
};

// A value of another CTA of the cluster, by its cluster shared address.
template <typename T>
__device__ __forceinline__ T ld_cluster(uint32_t addr) {
  T v;
  if constexpr (std::is_same<T, float>::value)
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  else if constexpr (std::is_same<T, double>::value)
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
  else if constexpr (std::is_same<T, float2>::value)
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  else
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(addr) : "memory");
  return v;
}

// ---- tile shapes ------------------------------------------------------------------
// BM x BN tile of C per CTA, WM x WN warps, K slabs of BK in a ring of kStages,
// kCtas resident CTAs per SM.  fp32: TM x TN outputs per thread on LM x 32 / LM
// lanes.  The 64 x 64 tile runs at 50 cycles per K value and SM (32 at the pipe's
// peak), the 128 x 128 one, with 16 x 8 outputs per thread, at 41 per 64 x 64.
template <typename T, bool kBig> struct Shape;
// Cycles on one SM, fitted to 90 timed shapes (within 15%, the best split chosen or
// within 5% of it): kLone per K value for a CTA alone, kShared per K value and CTA
// when they share the SM, kFixed per CTA and K part for the ring's start, the
// cluster barriers and the sum.
struct CostModel { int lone, shared, fixed; };
template <typename T> constexpr CostModel kCost = {0, 0, 0};
template <> constexpr CostModel kCost<float> = {64, 50, 400};
template <> constexpr CostModel kCost<double> = {108, 68, 800};
template <> constexpr CostModel kCost<float2> = {178, 167, 900};
template <> constexpr CostModel kCost<double2> = {303, 277, 1500};
constexpr CostModel kCostBig = {193, 165, 400};  // float, 128 x 128
template <> struct Shape<float, false> {
  static constexpr int BM = 64, BN = 64, WM = 2, WN = 2, BK = 16, kStages = 4, kCtas = 4, TM = 8, TN = 4, LM = 4;
};
template <> struct Shape<float, true> {
  static constexpr int BM = 128, BN = 128, WM = 2, WN = 2, BK = 16, kStages = 4, kCtas = 2, TM = 16, TN = 8, LM = 4;
};
template <> struct Shape<float2, false> {
  static constexpr int BM = 64, BN = 64, WM = 4, WN = 2, BK = 8, kStages = 4, kCtas = 2;
};
template <> struct Shape<double, false> {
  static constexpr int BM = 64, BN = 64, WM = 2, WN = 2, BK = 16, kStages = 3, kCtas = 3;
};
template <> struct Shape<double2, false> {
  static constexpr int BM = 64, BN = 64, WM = 4, WN = 2, BK = 8, kStages = 3, kCtas = 2;
};

template <typename T> constexpr bool kIsF64 = std::is_same<T, double>::value || std::is_same<T, double2>::value;

// Shared layout of one operand's slab, ROWS rows of op(X) by BK:
//   fp64 kinds, stored along K:  [ROWS][BK + 4]  (as stored)
//   otherwise:                   [BK][ROWS + pad]
// The pads make the fragment reads of a warp free of bank conflicts.
template <typename T, int ROWS, int BK, bool kKMajor>
struct Slab {
  static constexpr bool kRowMajor = kKMajor && kIsF64<T>;
  static constexpr int kPad = kRowMajor ? 4 : std::is_same<T, float>::value ? 4 : std::is_same<T, double>::value ? 4 : 2;
  static constexpr int kLd = (kRowMajor ? BK : ROWS) + kPad;
  static constexpr int kElems = (kRowMajor ? ROWS : BK) * kLd;
  static __device__ __forceinline__ int at(int r, int kk) { return kRowMajor ? r * kLd + kk : kk * kLd + r; }
};

// One thread's share of an operand's slabs.  Rows past the matrix are read from
// its last row (they only reach rows or columns of C that are not stored), so a
// full slab takes no bounds test; the last slab's K tail is zero-filled.
template <typename T, int ROWS, int BK, bool kKMajor, int kThreads>
struct Loader {
  using L = Slab<T, ROWS, BK, kKMajor>;
  static constexpr int V = 16 / (int)sizeof(T);
  static constexpr int ES = (int)sizeof(T);
  // runs of kRun threads walk the contiguous direction (8 K values per run
  // where the slab is transposed on the way: no bank conflicts)
  static constexpr int kVecRun = (kKMajor ? BK : ROWS) / V;
  static constexpr int kRun = !kKMajor ? ROWS : L::kRowMajor ? BK / V : 8;
  static constexpr int kSlots = kKMajor ? ROWS * kRun / kThreads : 1;   // rows per thread
  const T* p[kSlots];
  long long ld;
  uint32_t dst;      // byte offset in the slab
  int kk0;           // first K value of this thread
  int bytes;         // source bytes of a vector along M / N
  bool vec;

  __device__ __forceinline__ void init(const T* __restrict__ X, size_t ld_, bool vec_, int r0, int rows, int k0) {
    const int t = threadIdx.x;
    ld = (long long)ld_;
    vec = vec_;
    if constexpr (!kKMajor) {
      int r;
      if (V > 1 && vec) {
        r = (t % kVecRun) * V;
        kk0 = t / kVecRun;
        const int left = rows - (r0 + r);
        bytes = left >= V ? 16 : left > 0 ? left * ES : 0;
        p[0] = X + (bytes ? r0 + r : 0) + (size_t)(k0 + kk0) * ld_;
      } else {
        r = t % kRun;
        kk0 = t / kRun;
        p[0] = X + min(r0 + r, rows - 1) + (size_t)(k0 + kk0) * ld_;
      }
      dst = (uint32_t)L::at(r, kk0) * ES;
    } else {
      kk0 = (t % kRun) * (L::kRowMajor ? V : 1);
      const int r = t / kRun;
#pragma unroll
      for (int e = 0; e < kSlots; ++e)
        p[e] = X + (size_t)min(r0 + r + e * (kThreads / kRun), rows - 1) * ld_ + k0 + kk0;
      dst = (uint32_t)L::at(r, kk0) * ES;
    }
  }
  // Stages the next slab at shared address `st`; `left` K values remain.
  __device__ __forceinline__ void slab(uint32_t st, int left) {
    const uint32_t d = st + dst;
    const bool full = left >= BK;
    if constexpr (!kKMajor) {
      if (V > 1 && vec) {
        constexpr int kStep = kThreads / kVecRun, kN = BK / kStep;
#pragma unroll
        for (int e = 0; e < kN; ++e) {
          const bool ok = full || kk0 + e * kStep < left;
          copy(d + (uint32_t)(L::at(0, e * kStep) * ES), ok ? p[0] + e * kStep * ld : p[0] - kk0 * ld, ok ? bytes : 0);
        }
      } else {
        constexpr int kStep = kThreads / kRun, kN = BK / kStep;
        if (full) {
#pragma unroll
          for (int e = 0; e < kN; ++e)
            cp_async<ES>(d + (uint32_t)(L::at(0, e * kStep) * ES), p[0] + e * kStep * ld, true);
        } else {
#pragma unroll
          for (int e = 0; e < kN; ++e) {
            const bool ok = kk0 + e * kStep < left;
            cp_async<ES>(d + (uint32_t)(L::at(0, e * kStep) * ES), ok ? p[0] + e * kStep * ld : p[0] - kk0 * ld, ok);
          }
        }
      }
      p[0] += (long long)BK * ld;
    } else if constexpr (L::kRowMajor) {
      constexpr int kStep = kThreads / kRun;
#pragma unroll
      for (int e = 0; e < kSlots; ++e) {
        const uint32_t de = d + (uint32_t)(L::at(e * kStep, 0) * ES);
        if (V == 1 || vec) {
          const int n = full ? V : min(max(left - kk0, 0), V);
          copy(de, n ? p[e] : p[e] - kk0, n * ES);
        } else {
#pragma unroll
          for (int v = 0; v < V; ++v) {
            const bool ok = full || kk0 + v < left;
            cp_async<(V == 1 ? 16 : ES)>(de + v * ES, ok ? p[e] + v : p[e] - kk0, ok);
          }
        }
        p[e] += BK;
      }
    } else {
      constexpr int kStep = kThreads / kRun;
#pragma unroll
      for (int e = 0; e < kSlots; ++e) {
#pragma unroll
        for (int h = 0; h < BK; h += 8) {
          const uint32_t de = d + (uint32_t)(L::at(e * kStep, h) * ES);
          if (full) {
            cp_async<ES>(de, p[e] + h, true);
          } else {
            const bool ok = kk0 + h < left;
            cp_async<ES>(de, ok ? p[e] + h : p[e] - kk0, ok);
          }
        }
        p[e] += BK;
      }
    }
  }
  static __device__ __forceinline__ void copy(uint32_t d, const T* src, int n) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
  }
};

// ---- warp tiles: accumulate one slab, then write the tile to Cs[n][m] -----------
template <typename T, typename S, bool AK, bool BKM> struct WarpTile;

// Lane grid of the FMA kinds, LM rows x 32 / LM columns: rows from lane bits 1
// up, columns from bit 0 and the top bits, so that lanes l and l ^ 1 read the
// same A vector and l and l ^ 2 the same B vector.  A 16-byte shared load whose
// lanes agree in one of these ways takes 2 cycles, in any other grid 4
// (measured), and the fragment loads would bound the kernel.
template <int LM>
__device__ __forceinline__ int lane_m(int lane) { return (lane >> 1) & (LM - 1); }
template <int LM>
__device__ __forceinline__ int lane_n(int lane) { return (lane & 1) | ((lane / (2 * LM)) << 1); }

// fp32: thread tile TM x TN in groups of 4 rows / columns, packed along m.
template <typename S, bool AK, bool BKM>
struct WarpTile<float, S, AK, BKM> {
  static constexpr int LM = S::LM, LN = 32 / LM, TM = S::TM, TN = S::TN, WTM = LM * TM, WTN = LN * TN;
  static_assert(WTM * S::WM == S::BM && WTN * S::WN == S::BN, "warp tiles cover the CTA tile");
  using SA = Slab<float, S::BM, S::BK, AK>;
  using SB = Slab<float, S::BN, S::BK, BKM>;
  uint64_t acc[TM / 2][TN];
  int m0, n0;
  __device__ __forceinline__ void init(int warp, int lane, bool, bool) {
    m0 = (warp % S::WM) * WTM + lane_m<LM>(lane) * 4;
    n0 = (warp / S::WM) * WTN + lane_n<LM>(lane) * 4;
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] = 0;
  }
  __device__ __forceinline__ void slab(const float* a, const float* b) {
    const float* ap = a + SA::at(m0, 0);
    const float* bp = b + SB::at(n0, 0);
#pragma unroll
    for (int kk = 0; kk < S::BK; ++kk) {
      uint64_t av[TM / 2];
      float bv[TN];
#pragma unroll
      for (int g = 0; g < TM / 4; ++g) {
        const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(ap + SA::at(g * 4 * LM, kk));
        av[2 * g] = u.x;
        av[2 * g + 1] = u.y;
      }
#pragma unroll
      for (int g = 0; g < TN / 4; ++g) {
        const float4 u = *reinterpret_cast<const float4*>(bp + SB::at(g * 4 * LN, kk));
        bv[4 * g] = u.x;
        bv[4 * g + 1] = u.y;
        bv[4 * g + 2] = u.z;
        bv[4 * g + 3] = u.w;
      }
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const uint64_t bb = pack2(bv[j], bv[j]);
#pragma unroll
        for (int i = 0; i < TM / 2; ++i) fma2(acc[i][j], av[i], bb);
      }
    }
  }
  template <int kLdC>
  __device__ __forceinline__ void put(float* cs) {
#pragma unroll
    for (int j = 0; j < TN; ++j)
#pragma unroll
      for (int g = 0; g < TM / 4; ++g) {
        float* p = cs + (n0 + (j / 4) * 4 * LN + j % 4) * kLdC + m0 + g * 4 * LM;
        *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(acc[2 * g][j], acc[2 * g + 1][j]);
      }
  }
};

// complex64: thread tile 4 x 4 in groups of 2; re(a) b and im(a) b accumulate
// apart (two packed multiply-adds per product, no swap), the signs of the
// conjugations and of i^2 come in once, at the end.
template <typename S, bool AK, bool BKM>
struct WarpTile<float2, S, AK, BKM> {
  static constexpr int LM = 4, LN = 8, TM = 4, TN = 4;
  static constexpr int WTM = LM * TM, WTN = LN * TN;
  static_assert(WTM * S::WM == S::BM && WTN * S::WN == S::BN, "warp tiles cover the CTA tile");
  using SA = Slab<float2, S::BM, S::BK, AK>;
  using SB = Slab<float2, S::BN, S::BK, BKM>;
  uint64_t ar[TM][TN], ai[TM][TN];
  int m0, n0;
  float sa, sb;
  __device__ __forceinline__ void init(int warp, int lane, bool conj_a, bool conj_b) {
    m0 = (warp % S::WM) * WTM + lane_m<LM>(lane) * 2;
    n0 = (warp / S::WM) * WTN + lane_n<LM>(lane) * 2;
    sa = conj_a ? -1.f : 1.f;
    sb = conj_b ? -1.f : 1.f;
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) ar[i][j] = ai[i][j] = 0;
  }
  __device__ __forceinline__ void slab(const float2* a, const float2* b) {
#pragma unroll
    for (int kk = 0; kk < S::BK; ++kk) {
      uint64_t re[TM], im[TM], bv[TN];
#pragma unroll
      for (int g = 0; g < TM / 2; ++g) {
        const float4 u = *reinterpret_cast<const float4*>(a + SA::at(m0 + g * 2 * LM, kk));
        re[2 * g] = pack2(u.x, u.x);
        im[2 * g] = pack2(u.y, u.y);
        re[2 * g + 1] = pack2(u.z, u.z);
        im[2 * g + 1] = pack2(u.w, u.w);
      }
#pragma unroll
      for (int g = 0; g < TN / 2; ++g) {
        const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(b + SB::at(n0 + g * 2 * LN, kk));
        bv[2 * g] = u.x;
        bv[2 * g + 1] = u.y;
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          fma2(ar[i][j], re[i], bv[j]);
          fma2(ai[i][j], im[i], bv[j]);
        }
    }
  }
  template <int kLdC>
  __device__ __forceinline__ void put(float2* cs) {
#pragma unroll
    for (int j = 0; j < TN; ++j)
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const float2 r = unpack2(ar[i][j]), q = unpack2(ai[i][j]);
        cs[(n0 + (j / 2) * 2 * LN + j % 2) * kLdC + m0 + (i / 2) * 2 * LM + i % 2] =
            make_float2(r.x - sa * sb * q.y, sb * r.y + sa * q.x);
      }
  }
};

// fp64: 8 x 8 x 4 tensor-core products.
template <typename S, bool AK, bool BKM>
struct WarpTile<double, S, AK, BKM> {
  static constexpr int WTM = S::BM / S::WM, WTN = S::BN / S::WN, NM = WTM / 8, NN = WTN / 8;
  using SA = Slab<double, S::BM, S::BK, AK>;
  using SB = Slab<double, S::BN, S::BK, BKM>;
  double acc[NM][NN][2];
  int m0, n0, g, t;
  __device__ __forceinline__ void init(int warp, int lane, bool, bool) {
    m0 = (warp % S::WM) * WTM;
    n0 = (warp / S::WM) * WTN;
    g = lane >> 2;
    t = lane & 3;
#pragma unroll
    for (int i = 0; i < NM; ++i)
#pragma unroll
      for (int j = 0; j < NN; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  }
  __device__ __forceinline__ void slab(const double* a, const double* b) {
#pragma unroll
    for (int kk = 0; kk < S::BK; kk += 4) {
      double av[NM], bv[NN];
#pragma unroll
      for (int i = 0; i < NM; ++i) av[i] = a[SA::at(m0 + 8 * i + g, kk + t)];
#pragma unroll
      for (int j = 0; j < NN; ++j) bv[j] = b[SB::at(n0 + 8 * j + g, kk + t)];
#pragma unroll
      for (int i = 0; i < NM; ++i)
#pragma unroll
        for (int j = 0; j < NN; ++j) dmma(acc[i][j], av[i], bv[j]);
    }
  }
  template <int kLdC>
  __device__ __forceinline__ void put(double* cs) {
#pragma unroll
    for (int j = 0; j < NN; ++j)
#pragma unroll
      for (int i = 0; i < NM; ++i)
#pragma unroll
        for (int c = 0; c < 2; ++c) cs[(n0 + 8 * j + 2 * t + c) * kLdC + m0 + 8 * i + g] = acc[i][j][c];
  }
};

// complex128: four real tensor-core products per complex one.
template <typename S, bool AK, bool BKM>
struct WarpTile<double2, S, AK, BKM> {
  static constexpr int WTM = S::BM / S::WM, WTN = S::BN / S::WN, NM = WTM / 8, NN = WTN / 8;
  using SA = Slab<double2, S::BM, S::BK, AK>;
  using SB = Slab<double2, S::BN, S::BK, BKM>;
  double re[NM][NN][2], im[NM][NN][2];
  int m0, n0, g, t;
  long long fa, fb;
  __device__ __forceinline__ void init(int warp, int lane, bool conj_a, bool conj_b) {
    m0 = (warp % S::WM) * WTM;
    n0 = (warp / S::WM) * WTN;
    g = lane >> 2;
    t = lane & 3;
    fa = conj_a ? (1ll << 63) : 0;
    fb = conj_b ? (1ll << 63) : 0;
#pragma unroll
    for (int i = 0; i < NM; ++i)
#pragma unroll
      for (int j = 0; j < NN; ++j) re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0.0;
  }
  __device__ __forceinline__ void slab(const double2* a, const double2* b) {
#pragma unroll
    for (int kk = 0; kk < S::BK; kk += 4) {
      double2 av[NM], bv[NN];
#pragma unroll
      for (int i = 0; i < NM; ++i) {
        av[i] = a[SA::at(m0 + 8 * i + g, kk + t)];
        av[i].y = flip(av[i].y, fa);
      }
#pragma unroll
      for (int j = 0; j < NN; ++j) {
        bv[j] = b[SB::at(n0 + 8 * j + g, kk + t)];
        bv[j].y = flip(bv[j].y, fb);
      }
#pragma unroll
      for (int i = 0; i < NM; ++i) {
        const double neg = flip(av[i].y, 1ll << 63);
#pragma unroll
        for (int j = 0; j < NN; ++j) {
          dmma(re[i][j], av[i].x, bv[j].x);
          dmma(im[i][j], av[i].x, bv[j].y);
        }
#pragma unroll
        for (int j = 0; j < NN; ++j) {
          dmma(re[i][j], neg, bv[j].y);
          dmma(im[i][j], av[i].y, bv[j].x);
        }
      }
    }
  }
  template <int kLdC>
  __device__ __forceinline__ void put(double2* cs) {
#pragma unroll
    for (int j = 0; j < NN; ++j)
#pragma unroll
      for (int i = 0; i < NM; ++i)
#pragma unroll
        for (int c = 0; c < 2; ++c)
          cs[(n0 + 8 * j + 2 * t + c) * kLdC + m0 + 8 * i + g] = make_double2(re[i][j][c], im[i][j][c]);
  }
};

template <typename T, typename S, bool AK, bool BKM>
struct Smem {
  static constexpr int kA = Slab<T, S::BM, S::BK, AK>::kElems, kB = Slab<T, S::BN, S::BK, BKM>::kElems;
  static constexpr int kLdC = S::BM + (sizeof(T) == 16 ? 1 : sizeof(T) == 4 ? 4 : 2);
  static constexpr size_t kRing = (size_t)S::kStages * (kA + kB) * sizeof(T);
  static constexpr size_t kTile = (size_t)S::BN * kLdC * sizeof(T);
  static constexpr size_t kBytes = kRing > kTile ? kRing : kTile;
};

constexpr int kRaster = 16;  // M-tiles per raster group

// blockIdx.x = output tile, blockIdx.z = K part = rank in the cluster
template <typename T, bool kBig, bool AK, bool BKM>
__global__ void __launch_bounds__(32 * Shape<T, kBig>::WM * Shape<T, kBig>::WN, Shape<T, kBig>::kCtas)
k_gemm_native(int m, int n, int k, int k_part, T alpha, const T* __restrict__ A, size_t lda, const T* __restrict__ B,
              size_t ldb, T beta, T* __restrict__ C, size_t ldc, int flags) {
  using S = Shape<T, kBig>;
  using M = Smem<T, S, AK, BKM>;
  constexpr int kThreads = 32 * S::WM * S::WN, BK = S::BK, kStages = S::kStages;
  extern __shared__ __align__(16) unsigned char native_smem[];
  T* ring = reinterpret_cast<T*>(native_smem);
  const uint32_t ring_addr = tc::smem_u32(native_smem);
  const bool vec_a = flags & 1, vec_b = flags & 2;

  const int m_tiles = (int)(((unsigned)m + S::BM - 1) / S::BM), n_tiles = (int)(((unsigned)n + S::BN - 1) / S::BN);
  const int grp = (int)blockIdx.x / (kRaster * n_tiles), in = (int)blockIdx.x - grp * kRaster * n_tiles;
  const int gsz = min(kRaster, m_tiles - grp * kRaster);
  const int m0 = (grp * kRaster + in % gsz) * S::BM, n0 = (in / gsz) * S::BN;
  const int k_lo = (int)min((long long)k, (long long)blockIdx.z * k_part);
  const int k_len = min(k - k_lo, k_part);
  const int nk = (int)(((unsigned)k_len + BK - 1) / BK);

  Loader<T, S::BM, BK, AK, kThreads> la;
  Loader<T, S::BN, BK, BKM, kThreads> lb;
  la.init(A, lda, vec_a, m0, m, k_lo);
  lb.init(B, ldb, vec_b, n0, n, k_lo);
  auto load = [&](int kt) {
    if (kt < nk) {
      const uint32_t st = ring_addr + (uint32_t)((kt % kStages) * (M::kA + M::kB) * (int)sizeof(T));
      const int left = k_len - kt * BK;
      la.slab(st, left);
      lb.slab(st + M::kA * (int)sizeof(T), left);
    }
    cp_async_commit();
  };

  WarpTile<T, S, AK, BKM> w;
  w.init(threadIdx.x >> 5, threadIdx.x & 31, (flags & 4) != 0, (flags & 8) != 0);
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) load(s);
  for (int kt = 0; kt < nk; ++kt) {
    cp_async_wait<kStages - 2>();
    __syncthreads();  // slab kt has landed; every warp is done with slab kt - 1
    load(kt + kStages - 1);
    const T* a = ring + (size_t)(kt % kStages) * (M::kA + M::kB);
    w.slab(a, a + M::kA);
  }
  cp_async_wait<0>();
  __syncthreads();

  // tile to shared memory, then C in whole columns (a warp: 32 rows)
  w.template put<M::kLdC>(ring);
  const int parts = gridDim.z, rank = blockIdx.z;
  if (parts > 1) tc::cluster_sync(); else __syncthreads();
  const bool beta0 = Ops<T>::zero(beta), beta1 = Ops<T>::one(beta);
  const int total = S::BM * S::BN / parts;
  constexpr int U = 8;  // C loads in flight per thread
  for (int e0 = threadIdx.x; e0 < total; e0 += U * kThreads) {
    T cv[U], acc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = e0 + u * kThreads + rank * total;
      const int gr = m0 + i % S::BM, gc = n0 + i / S::BM;
      if (!beta0 && gr < m && gc < n && e0 + u * kThreads < total) cv[u] = C[gr + (size_t)gc * ldc];
    }
    if (parts == 1) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = e0 + u * kThreads;
        acc[u] = ring[(i / S::BM) * M::kLdC + i % S::BM];
      }
    } else {
      for (int p = 0; p < parts; ++p) {
        const uint32_t base = tc::mapa_shared(ring_addr, p);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int i = e0 + u * kThreads + rank * total;
          if (e0 + u * kThreads < total) {
            const T v = ld_cluster<T>(base + (uint32_t)((i / S::BM) * M::kLdC + i % S::BM) * (uint32_t)sizeof(T));
            acc[u] = p == 0 ? v : Ops<T>::add(acc[u], v);
          }
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = e0 + u * kThreads + rank * total;
      const int gr = m0 + i % S::BM, gc = n0 + i / S::BM;
      if (gr < m && gc < n && e0 + u * kThreads < total) {
        const T v = Ops<T>::mul(alpha, acc[u]);
        C[gr + (size_t)gc * ldc] =
            beta0 ? v : beta1 ? Ops<T>::add(cv[u], v) : Ops<T>::add(Ops<T>::mul(beta, cv[u]), v);
      }
    }
  }
  if (parts > 1) tc::cluster_sync();  // peers may still read this CTA's tile
}

template <typename T, bool kBig, bool AK, bool BKM>
coral_status_t launch(Handle* h, int m, int n, int k, int splits, T alpha, const T* A, size_t lda, const T* B,
                      size_t ldb, T beta, T* C, size_t ldc, int flags) {
  using S = Shape<T, kBig>;
  using M = Smem<T, S, AK, BKM>;
  static uint64_t attr_devices = 0;  // bit d: attribute set on device d
  const uint64_t bit = h->device < 64 ? (1ull << h->device) : 0;
  if (!(attr_devices & bit) || !bit) {
    CORAL_CUDA(h, cudaFuncSetAttribute(k_gemm_native<T, kBig, AK, BKM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)M::kBytes));
    attr_devices |= bit;
  }
  const size_t tiles = (((size_t)m + S::BM - 1) / S::BM) * (((size_t)n + S::BN - 1) / S::BN);
  if (tiles > 0x7fffffffu) return CORAL_ERR_NOT_SUPPORTED;
  // whole slabs per K part; past INT_MAX only for a part that covers all of K
  const size_t slabs = ((size_t)k + S::BK - 1) / S::BK;
  const size_t part = (slabs + splits - 1) / splits * S::BK;
  const int k_part = (int)(part < (size_t)INT_MAX ? part : (size_t)INT_MAX);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)tiles, 1, (unsigned)splits);
  cfg.blockDim = dim3(32 * S::WM * S::WN);
  cfg.dynamicSmemBytes = M::kBytes;
  cfg.stream = h->stream;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = 1;
  at.val.clusterDim.y = 1;
  at.val.clusterDim.z = (unsigned)splits;
  cfg.attrs = &at;
  cfg.numAttrs = splits > 1 ? 1 : 0;
  timed_begin(h);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_gemm_native<T, kBig, AK, BKM>, m, n, k, k_part, alpha, A, lda, B,
                                           ldb, beta, C, ldc, flags);
  coral_status_t s = e == cudaSuccess ? launch_status(h) : cuda_status(h, e);
  timed_end(h);
  return s;
}

template <typename T, bool kBig>
coral_status_t launch_ops(Handle* h, bool ak, bool bk, int m, int n, int k, int splits, T alpha, const T* A,
                          size_t lda, const T* B, size_t ldb, T beta, T* C, size_t ldc, int flags) {
  if (ak && bk) return launch<T, kBig, true, true>(h, m, n, k, splits, alpha, A, lda, B, ldb, beta, C, ldc, flags);
  if (ak) return launch<T, kBig, true, false>(h, m, n, k, splits, alpha, A, lda, B, ldb, beta, C, ldc, flags);
  if (bk) return launch<T, kBig, false, true>(h, m, n, k, splits, alpha, A, lda, B, ldb, beta, C, ldc, flags);
  return launch<T, kBig, false, false>(h, m, n, k, splits, alpha, A, lda, B, ldb, beta, C, ldc, flags);
}

// K parts (and, for fp32, the large tile) with the least time on the busiest SM by
// the cost model.  Depends on sizes and type alone: aligned and unaligned
// operands sum in the same order.
template <typename T>
void choose_split(size_t m, size_t n, size_t k, int sms, int& splits, bool& big) {
  using S = Shape<T, false>;
  const double tiles = (double)((m + S::BM - 1) / S::BM) * (double)((n + S::BN - 1) / S::BN);
  const CostModel c = kCost<T>;
  double best = 0.0;
  splits = 1;
  big = false;
  for (int s = 1; s <= 8; s *= 2) {
    const double kp = (double)((k + s - 1) / s), ctas = ceil(tiles * s / sms);
    if (s > 1 && kp < S::BK) break;
    const double t = kp * fmax(c.lone, c.shared * ctas) + ctas * c.fixed * s;
    if (s == 1 || t < best) {
      best = t;
      splits = s;
    }
  }
  if constexpr (std::is_same<T, float>::value) {
    using B = Shape<float, true>;
    const double bt = (double)((m + B::BM - 1) / B::BM) * (double)((n + B::BN - 1) / B::BN), ctas = ceil(bt / sms);
    if ((double)k * fmax(kCostBig.lone, kCostBig.shared * ctas) + ctas * kCostBig.fixed < best) {
      splits = 1;
      big = true;
    }
  }
}

// C <- beta * C (beta == 0 writes zeros without reading C).
template <typename T>
__global__ void k_scale_c(int m, int n, T beta, T* __restrict__ C, size_t ldc) {
  const bool beta0 = Ops<T>::zero(beta);
  size_t total = (size_t)m * n;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (size_t)gridDim.x * blockDim.x) {
    size_t i = t % m, j = t / m;
    T* cp = C + i + j * ldc;
    *cp = beta0 ? T{} : Ops<T>::mul(beta, *cp);
  }
}

}  // namespace

// Validates the GEMM arguments the way the reference's debug_asserts do
// (sgemm_nn.rs:24-27) and reports the 1-based position of the first bad one.
int gemm_bad_arg(int op_a, int op_b, size_t m, size_t n, size_t k, const void* a, size_t lda,
                 const void* b, size_t ldb, const void* c, size_t ldc, bool complex_ops) {
  const int maxop = complex_ops ? CORAL_CONJ_TRANSPOSE : CORAL_CONJ_TRANSPOSE;
  if (op_a < 0 || op_a > maxop) return 1;
  if (op_b < 0 || op_b > maxop) return 2;
  const size_t a_rows = op_a == CORAL_NO_TRANSPOSE ? m : k;
  const size_t b_rows = op_b == CORAL_NO_TRANSPOSE ? k : n;
  if (m && n && !c) return 12;
  if (ldc < (m ? m : 1)) return 13;
  if (m && n && k) {
    if (!a) return 7;
    if (lda < (a_rows ? a_rows : 1)) return 8;
    if (!b) return 9;
    if (ldb < (b_rows ? b_rows : 1)) return 10;
  }
  if (m > INT32_MAX || n > INT32_MAX || k > INT32_MAX) return -1;
  return 0;
}

template <typename T>
coral_status_t enqueue_gemm_native(Handle* h, int op_a, int op_b, size_t m, size_t n, size_t k, T alpha, const T* A,
                                   size_t lda, const T* B, size_t ldb, T beta, T* C, size_t ldc) {
  if (m == 0 || n == 0) return CORAL_OK;
  if (Ops<T>::zero(alpha) || k == 0) {
    if (Ops<T>::one(beta)) return CORAL_OK;
    unsigned g = stream_grid(m * n, 256 * 4, h->sm_count, 8);
    k_scale_c<T><<<g, 256, 0, h->stream>>>((int)m, (int)n, beta, C, ldc);
    return launch_status(h);
  }
  // The widest C that is accepted.  The grid below would carry more; the limit stays so
  // that a size is refused or not as it always was.
  constexpr size_t kMaxCols = 65535u * (std::is_same<T, float>::value ? 128u : sizeof(T) == 16 ? 32u : 64u);
  if (n > kMaxCols) return CORAL_ERR_NOT_SUPPORTED;
  // ConjugateTranspose on a real type means Transpose (sgemm.rs:97-103).
  const bool ak = op_a != CORAL_NO_TRANSPOSE, bk = op_b == CORAL_NO_TRANSPOSE;
  constexpr bool kCplx = std::is_same<T, float2>::value || std::is_same<T, double2>::value;
  auto vec = [](const T* p, size_t ld) { return aligned16(p) && (ld * sizeof(T)) % 16 == 0; };
  const int flags = (vec(A, lda) ? 1 : 0) | (vec(B, ldb) ? 2 : 0) |
                    (kCplx && op_a == CORAL_CONJ_TRANSPOSE ? 4 : 0) | (kCplx && op_b == CORAL_CONJ_TRANSPOSE ? 8 : 0);
  const int mi = (int)m, ni = (int)n, ki = (int)k;
  int splits;
  bool big;
  choose_split<T>(m, n, k, h->sm_count, splits, big);
  if constexpr (std::is_same<T, float>::value)
    if (big) return launch_ops<T, true>(h, ak, bk, mi, ni, ki, 1, alpha, A, lda, B, ldb, beta, C, ldc, flags);
  return launch_ops<T, false>(h, ak, bk, mi, ni, ki, splits, alpha, A, lda, B, ldb, beta, C, ldc, flags);
}

#define CORAL_NATIVE(T)                                                                                          \
  template coral_status_t enqueue_gemm_native<T>(Handle*, int, int, size_t, size_t, size_t, T, const T*, size_t, \
                                                 const T*, size_t, T, T*, size_t)
CORAL_NATIVE(float);
CORAL_NATIVE(double);
CORAL_NATIVE(float2);
CORAL_NATIVE(double2);

}  // namespace coral
