// Grouped (batched, uneven) SGEMM and batched STRSV.
//
// No reference counterpart: each instance has exactly the semantics of
// coral_sgemm (sgemm.rs:106-130, epilogue f32_edge.rs:37-58) or coral_strsv
// (strsv.rs:60-74); the batch is described by an array of descriptors in
// DEVICE memory, so a call enqueues a fixed number of kernels with no host
// work per instance and can be captured in a CUDA graph (size the handle's
// scratch with one uncaptured call first).
//
// Grouped GEMM on the tensor cores (bf16 inputs, or fp32 inputs in
// split-BF16x3 mode): grouped_tc.cu.  The FP32 FMA form below serves fp32
// inputs in the NATIVE and SPLIT_BF16X6 modes.
//
// Grouped GEMM (FMA form): k_tile_prefix (one CTA) turns the descriptors into an
// exclusive prefix sum of 64 x 64 output tiles; k_gemm_grouped (persistent,
// 4 CTAs per SM) walks the global tile index space with a grid stride, finds
// each tile's instance by binary search over the prefix array and computes
// the tile on the FP32 FMA pipes: 256 threads, 4 x 4 outputs per thread,
// 16-deep K slabs double-buffered through shared memory.  The bf16-input
// variant reads bf16 operands and accumulates in fp32.
//
// Batched TRSV: one CTA per instance (a warp up to 32 rows), blocked right-looking
// substitution over 64-row diagonal blocks.  One warp runs the chain (take the
// previous block off the next 64 rows, solve their diagonal block, divide by the
// diagonal as strlsv.rs:66-140 does) while the other seven take that previous block
// off all rows further down (coalesced column streaming, 48 loads in flight per
// thread) and copy the next diagonal block and the block below it to shared
// memory, so the chain waits for memory at its start only.  What bounds it: the
// chain of the largest instance (3.5 us per 64 rows alone on the GPU, twice that
// beside a second CTA and 3 TB/s of others), then HBM.  Sizes log-uniform in
// [32, 1024], 1024 instances, 330 MB: 372 -> 107 us (3.1 TB/s); one instance of 1024
// rows: 261 -> 53 us.  Of that, starting the longest instances first gave 40 us;
// asking for the next panel through L2 prefetches cost 10 us (more instructions
// than it saved) and is not done; two rows per thread took 136 us,
// four the same as three.  Transposed operators read the same memory by rows,
// backward solves walk it from its end.
#include "common.cuh"

#include <cuda_bf16.h>

namespace coral {
namespace {

struct GemmProblem {
  int32_t op_a, op_b, m, n, k;
  float alpha, beta;
  int32_t reserved;
  const void* a;
  const void* b;
  float* c;
  int64_t lda, ldb, ldc;
};
static_assert(sizeof(GemmProblem) == sizeof(coral_sgemm_problem_t), "descriptor layout");

struct TrsvProblem {
  int32_t uplo, trans, diag, n;
  const float* a;
  float* x;
  int64_t lda, incx;
};
static_assert(sizeof(TrsvProblem) == sizeof(coral_strsv_problem_t), "descriptor layout");

constexpr int kGT = 64;       // output tile edge
constexpr int kGK = 16;       // K slab
constexpr int kGThreads = 256;

__global__ void k_tile_prefix(const GemmProblem* __restrict__ probs, int count, int* __restrict__ prefix) {
  __shared__ int warp_tot[32];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < count; base += blockDim.x) {
    const int i = base + threadIdx.x;
    int t = 0;
    if (i < count) {
      const GemmProblem p = probs[i];
      t = (p.m > 0 && p.n > 0) ? ((p.m + kGT - 1) / kGT) * ((p.n + kGT - 1) / kGT) : 0;
    }
    // block-wide exclusive scan
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int v = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    if (lane == 31) warp_tot[w] = v;
    __syncthreads();
    if (w == 0) {
      int s = lane < (int)(blockDim.x >> 5) ? warp_tot[lane] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int u = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += u;
      }
      warp_tot[lane] = s;  // inclusive warp totals
    }
    __syncthreads();
    const int excl = carry + (w ? warp_tot[w - 1] : 0) + v - t;
    if (i < count) prefix[i] = excl;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = excl + t;
    __syncthreads();
  }
  if (threadIdx.x == 0) prefix[count] = carry;
}

template <typename TIn>
__device__ __forceinline__ float ld_in(const TIn* p);
template <> __device__ __forceinline__ float ld_in<float>(const float* p) { return __ldg(p); }
template <> __device__ __forceinline__ float ld_in<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __bfloat162float(*p);
}

template <typename TIn>
__global__ void __launch_bounds__(kGThreads)
k_gemm_grouped(const GemmProblem* __restrict__ probs, int count, const int* __restrict__ prefix) {
  __shared__ __align__(16) float As[2][kGK][kGT + 4];
  __shared__ __align__(16) float Bs[2][kGK][kGT + 4];
  const int total = prefix[count];
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  for (int t = blockIdx.x; t < total; t += gridDim.x) {
    // instance holding tile t: last i with prefix[i] <= t
    int lo = 0, hi = count - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (prefix[mid] <= t) lo = mid; else hi = mid - 1;
    }
    const GemmProblem p = probs[lo];
    const int local = t - prefix[lo];
    const int mt = (p.m + kGT - 1) / kGT;
    const int m0 = (local % mt) * kGT, n0 = (local / mt) * kGT;
    const TIn* A = static_cast<const TIn*>(p.a);
    const TIn* B = static_cast<const TIn*>(p.b);
    const bool a_km = p.op_a != CORAL_NO_TRANSPOSE, b_km = p.op_b == CORAL_NO_TRANSPOSE;

    float ra[4], rb[4];
    auto load = [&](int k0) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int idx = threadIdx.x + e * kGThreads;
        int r, kk;
        if (a_km) { kk = idx % kGK; r = idx / kGK; } else { r = idx % kGT; kk = idx / kGT; }
        const int gr = m0 + r, gk = k0 + kk;
        ra[e] = (gr < p.m && gk < p.k) ? ld_in<TIn>(a_km ? A + gk + (size_t)gr * p.lda : A + gr + (size_t)gk * p.lda) : 0.f;
        int c;
        if (b_km) { kk = idx % kGK; c = idx / kGK; } else { c = idx % kGT; kk = idx / kGT; }
        const int gc = n0 + c, gk2 = k0 + kk;
        rb[e] = (gc < p.n && gk2 < p.k) ? ld_in<TIn>(b_km ? B + gk2 + (size_t)gc * p.ldb : B + gc + (size_t)gk2 * p.ldb) : 0.f;
      }
    };
    auto store = [&](int buf) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int idx = threadIdx.x + e * kGThreads;
        int r, kk;
        if (a_km) { kk = idx % kGK; r = idx / kGK; } else { r = idx % kGT; kk = idx / kGT; }
        As[buf][kk][r] = ra[e];
        int c;
        if (b_km) { kk = idx % kGK; c = idx / kGK; } else { c = idx % kGT; kk = idx / kGT; }
        Bs[buf][kk][c] = rb[e];
      }
    };
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    const int ks = (p.k + kGK - 1) / kGK;
    __syncthreads();  // previous tile's readers are done with the buffers
    if (ks > 0) {
      load(0);
      store(0);
    }
    __syncthreads();
    for (int s = 0; s < ks; ++s) {
      const int cur = s & 1;
      if (s + 1 < ks) load((s + 1) * kGK);
#pragma unroll
      for (int kk = 0; kk < kGK; ++kk) {
        const float4 a4 = *reinterpret_cast<const float4*>(&As[cur][kk][ty * 4]);
        const float4 b4 = *reinterpret_cast<const float4*>(&Bs[cur][kk][tx * 4]);
        const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
      }
      if (s + 1 < ks) store(cur ^ 1);
      __syncthreads();
    }
    const bool beta0 = p.beta == 0.f, beta1 = p.beta == 1.f;
    const bool scale_only = p.alpha == 0.f || p.k == 0;  // sgemm_nn.rs:29-45
    // the four C loads of a column before its stores (no round trip per element)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gc = n0 + tx * 4 + j;
      if (gc >= p.n) continue;
      if (scale_only && beta1) continue;
      float cv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int gr = m0 + ty * 4 + i;
        cv[i] = (!beta0 && gr < p.m) ? p.c[gr + (size_t)gc * p.ldc] : 0.f;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int gr = m0 + ty * 4 + i;
        if (gr >= p.m) continue;
        float* cp = p.c + gr + (size_t)gc * p.ldc;
        if (scale_only) {
          *cp = beta0 ? 0.f : cv[i] * p.beta;
        } else {
          const float v = p.alpha * acc[i][j];
          *cp = beta0 ? v : beta1 ? cv[i] + v : p.beta * cv[i] + v;
        }
      }
    }
  }
}

// ---- batched TRSV --------------------------------------------------------------
constexpr int kBT = 64;
constexpr int kBTThreads = 256;
constexpr int kBTBulk = kBTThreads - 32;   // threads of the warps beside the solving one
constexpr int kBTLd = 68;                  // column pitch of the diagonal block (16-byte multiple)
constexpr int kBTLs = 65;                  // and of the block below it
constexpr int kRows = 3;                   // rows per thread of the update
constexpr int kBTMaxX = 1024;              // right-hand sides up to here stay in shared memory
constexpr int kBTWindow = 1024;            // instances ordered together

// The window a CTA draws from.
struct TrsvWindow {
  TrsvProblem cur;               // the system at `drawn`, for the CTA as a whole
  unsigned short ord[kBTWindow];
  int w, local, big, units, first;
  int drawn, next;
};

struct TrsvSmem {
  float D[2][kBT][kBTLd];   // [column][row]
  float S[2][kBT][kBTLs];   // [column][row]
  float xb[2][kBT];
  float part[4][kBT];
  float inv[kBT];
  float x[kBTMaxX];
  TrsvWindow win;
};
extern __shared__ __align__(16) unsigned char trsv_smem[];

// The system in solve order: always lower triangular, element (i, j) of op(A)
// at a[i * rs + j * cs], right-hand side i at x[i * xs].  A backward solve
// walks the same memory from its end.
struct TrsvView {
  const float* a;
  float* x;
  long long rs, cs, xs;
  int n;
};

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// Starts the copy of diagonal block b (lower half) and of the block below the
// previous diagonal (rows of block b, columns of block b - 1); warp w of
// `warps`, lanes along the stored direction.
__device__ __forceinline__ void trsv_fetch(const TrsvView& v, int b, bool below, TrsvSmem& sm, int w, int warps,
                                           bool rows_first) {
  const int b0 = b * kBT, bn = min(kBT, v.n - b0), lane = threadIdx.x & 31;
  const float* diag = v.a + b0 * (v.rs + v.cs);
  const float* left = diag - kBT * v.cs;
  float(*D)[kBTLd] = sm.D[b & 1];
  float(*S)[kBTLs] = sm.S[(b - 1) & 1];
  if (rows_first) {
    const bool in0 = lane < bn, in1 = lane + 32 < bn;
    diag += lane * v.rs;
    left += lane * v.rs;
    for (int c = w; c < kBT; c += warps) {
      const long long o = c * v.cs;
      if (in0 && c <= lane) cp_async4(&D[c][lane], diag + o);
      if (in1 && c <= lane + 32) cp_async4(&D[c][lane + 32], diag + o + 32 * v.rs);
      if (below) {
        if (in0) cp_async4(&S[c][lane], left + o);
        if (in1) cp_async4(&S[c][lane + 32], left + o + 32 * v.rs);
      }
    }
  } else {
    diag += lane * v.cs;
    left += lane * v.cs;
    for (int r = w; r < bn; r += warps) {
      const long long o = r * v.rs;
      if (lane <= r) cp_async4(&D[lane][r], diag + o);
      if (lane + 32 <= r) cp_async4(&D[lane + 32][r], diag + o + 32 * v.cs);
      if (below) {
        cp_async4(&S[lane][r], left + o);
        cp_async4(&S[lane + 32][r], left + o + 32 * v.cs);
      }
    }
  }
}

// Zeros what the copies of a last, short block b leave untouched: rows past the
// system then solve to 0 and take nothing from the others.
__device__ __forceinline__ void trsv_pad(TrsvSmem& sm, int b, int bn) {
  float(*D)[kBTLd] = sm.D[b & 1];
  float(*S)[kBTLs] = sm.S[(b - 1) & 1];
  for (int e = threadIdx.x; e < kBT * kBT; e += kBTThreads) {
    const int r = e % kBT, c = e / kBT;
    if (r >= bn) {
      if (c <= r) D[c][r] = r == c ? 1.f : 0.f;
      S[c][r] = 0.f;
    }
  }
}

// Reciprocal of the diagonal entry of row r (one thread per row), 1 for a unit
// diagonal; returns whether the product with it can stand for the division.
__device__ __forceinline__ bool trsv_recip(TrsvSmem& sm, int b, int r, bool unit) {
  float(*D)[kBTLd] = sm.D[b & 1];
  if (unit) D[r][r] = 1.f;
  const float d = unit ? 1.f : D[r][r];
  sm.inv[r] = 1.f / d;
  return fabsf(d) > 0x1p-60f && fabsf(d) < 0x1p60f;
}

// One warp: solves diagonal block b for the right-hand sides rh[h] of rows
// lane + 32 h, 8 rows at a time.  Every lane solves the 8 x 8 corner (no
// exchange inside its chain), then takes its 8 products off its own rows.
// x / d is x * (1 / d) with one residual correction.  Where that could round
// differently -- a diagonal far from 1 (!fast), or a result that is not finite,
// which reaches every later row -- the block is solved again with divisions.
__device__ __forceinline__ void trsv_solve(TrsvSmem& sm, int b, bool fast, const float (&rhs)[2]) {
  const int lane = threadIdx.x & 31;
  const float(*D)[kBTLd] = sm.D[b & 1];
  float rh[2] = {rhs[0], rhs[1]}, last = 0.f;
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    float q[8], xs[8], l[8][8], iv[8], o[2][8];  // corner: right-hand sides, solution; own rows
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (j < 4) *reinterpret_cast<float4*>(l[j]) = *reinterpret_cast<const float4*>(&D[8 * s + j][8 * s]);
      *reinterpret_cast<float4*>(l[j] + 4) = *reinterpret_cast<const float4*>(&D[8 * s + j][8 * s + 4]);
    }
    *reinterpret_cast<float4*>(iv) = *reinterpret_cast<const float4*>(&sm.inv[8 * s]);
    *reinterpret_cast<float4*>(iv + 4) = *reinterpret_cast<const float4*>(&sm.inv[8 * s + 4]);
#pragma unroll
    for (int h = s / 4; h < 2; ++h)
#pragma unroll
      for (int j = 0; j < 8; ++j) o[h][j] = D[8 * s + j][lane + 32 * h];
#pragma unroll
    for (int j = 0; j < 8; ++j) q[j] = __shfl_sync(0xffffffffu, rh[s / 4], (8 * s + j) & 31);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float t = q[j] * iv[j];
      xs[j] = fmaf(fmaf(-t, l[j][j], q[j]), iv[j], t);
#pragma unroll
      for (int i = j + 1; i < 8; ++i) q[i] = fmaf(-l[j][i], xs[j], q[i]);
    }
    last = xs[7];
    float mine = xs[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) mine = (lane & 7) == j ? xs[j] : mine;
#pragma unroll
    for (int h = s / 4; h < 2; ++h) {
      float a = rh[h], c = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        a = fmaf(-o[h][j], xs[j], a);
        c = fmaf(-o[h][4 + j], xs[4 + j], c);
      }
      if (lane + 32 * h >= 8 * s + 8) rh[h] = a + c;
    }
    if ((lane >> 3) == (s & 3)) rh[s / 4] = mine;
  }
  if (!(fast && fabsf(last) < INFINITY)) {
    rh[0] = rhs[0];
    rh[1] = rhs[1];
#pragma unroll 1
    for (int j = 0; j < kBT; ++j) {
      const float x = __shfl_sync(0xffffffffu, j < 32 ? rh[0] : rh[1], j & 31) / D[j][j];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = lane + 32 * h;
        if (r == j) rh[h] = x;
        if (r > j) rh[h] = fmaf(-D[j][r], x, rh[h]);
      }
    }
  }
  float* xb = sm.xb[b & 1];
  xb[lane] = rh[0];
  xb[lane + 32] = rh[1];
  __syncwarp();
}

// Order of the solves: within each window of kBTWindow instances by decreasing size
// class (quarters of an octave), so the longest start first.  A CTA sorts a window
// by itself -- no plan pass, no memory beyond its own -- and then draws positions of
// it from the window's ticket; with more windows than one it goes on to the next
// that has any left.  Systems of up to kBTSmall rows come last in a window, a warp
// each and eight to a ticket: with a CTA and a ticket each they cost the 74 KB and
// the barriers of a large one (us: 1000 systems of 8 rows 20.5 -> 5.6, 100000 of 4
// 1640 -> 86, 20000 of 32 331 -> 67).
constexpr int kBTClasses = 128, kBTSmall = 32, kBTSmallClasses = 20;
constexpr int kBTWarps = kBTThreads / 32;
constexpr unsigned kBTSpent = 1u << 31;   // a ticket's mark: the window has no position left
__device__ __forceinline__ int trsv_class(int n) {
  const int v = n - 1;
  if (v <= 0) return 0;
  const int lg = 31 - __clz(v);
  return lg * 4 + (lg >= 2 ? (v >> (lg - 2)) & 3 : 0);
}
// threadIdx.x read anew: what is derived from it here is not kept over the solves,
// which leave no register for it (200 bytes of spills against 32).
__device__ __forceinline__ int tid_now() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}
// Fills ord with the window's instances (from its first) in order, input order inside
// a class: every CTA that sorts a window has to find the same.  Returns how many have
// more than kBTSmall rows.  Called and left by all threads together; the buffers of
// the diagonal blocks are free then.
__device__ __forceinline__ int trsv_order(const TrsvProblem* __restrict__ probs, int count, int base, TrsvSmem& sm) {
  constexpr int kPer = kBTWindow / kBTThreads, kRuns = kBTWindow / 32;   // a run: 32 instances
  static_assert(sizeof(int) * kRuns * kBTClasses <= sizeof(sm.D), "the table lies over the diagonal blocks");
  int(*table)[kBTClasses] = reinterpret_cast<int(*)[kBTClasses]>(&sm.D[0][0][0]);   // of a run: class -> count, place
  __shared__ int start[kBTClasses], big;
  const int t = tid_now(), lane = t & 31, warp = t >> 5;
  int key[kPer];
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int i = base + q * kBTThreads + t;
    key[q] = i < count ? trsv_class(probs[i].n) : -1;
  }
#pragma unroll
  for (int e = 0; e < kRuns * kBTClasses / kBTThreads; ++e) (&table[0][0])[e * kBTThreads + t] = 0;
  __syncthreads();
  int rank[kPer];
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const unsigned peers = __match_any_sync(0xffffffffu, key[q]);
    rank[q] = __popc(peers & ((1u << lane) - 1u));
    if (key[q] >= 0 && rank[q] == 0) table[q * kBTWarps + warp][key[q]] = __popc(peers);
  }
  __syncthreads();
  if (t < kBTClasses) {
    int run = 0;
#pragma unroll 8
    for (int r = 0; r < kRuns; ++r) {
      const int c = table[r][t];
      table[r][t] = run;
      run += c;
    }
    start[t] = run;
  }
  __syncthreads();
  if (warp == 0) {  // first position of each class: 4 classes a lane, from the top
    int h[4], sum = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) sum += h[q] = start[kBTClasses - 1 - (lane * 4 + q)];
    int before = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, before, o);
      if (lane >= o) before += u;
    }
    before -= sum;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = kBTClasses - 1 - (lane * 4 + q);
      start[c] = before;
      before += h[q];
      if (c == kBTSmallClasses) big = before;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kPer; ++q)
    if (key[q] >= 0)
      sm.win.ord[start[key[q]] + table[q * kBTWarps + warp][key[q]] + rank[q]] = (unsigned short)(q * kBTThreads + t);
  __syncthreads();
  return big;
}

// The system in solve order (see TrsvView).
__device__ __forceinline__ TrsvView trsv_view(const TrsvProblem& p) {
  const bool t = p.trans != CORAL_NO_TRANSPOSE;
  TrsvView v;
  v.n = p.n;
  v.rs = t ? p.lda : 1;
  v.cs = t ? 1 : p.lda;
  v.xs = p.incx;
  v.a = p.a;
  v.x = p.x;
  if ((p.uplo == CORAL_LOWER) == t) {
    v.a += (long long)(p.n - 1) * (1 + p.lda);
    v.x += (long long)(p.n - 1) * p.incx;
    v.rs = -v.rs;
    v.cs = -v.cs;
    v.xs = -v.xs;
  }
  return v;
}

// One warp: a system of at most kBTSmall rows, lane = row, every load in flight.  As
// in trsv_solve a product with the reciprocal and one correction stand for the
// division, and divisions proper where they could round differently (a division per
// row in the chain: 8 us for 32 rows).
__device__ __noinline__ void trsv_small(const TrsvProblem& p) {
  if (p.n <= 0) return;
  const TrsvView v = trsv_view(p);
  const int lane = threadIdx.x & 31, n = v.n;
  const float* row = v.a + lane * v.rs;
  const bool in = lane < n;
  float a[kBTSmall];
#pragma unroll
  for (int g = 0; g < kBTSmall; g += 8)
    if (g < n)
#pragma unroll
      for (int c = g; c < g + 8; ++c) a[c] = in && c < lane ? row[c * v.cs] : 0.f;
  const float d = in && p.diag != CORAL_UNIT ? row[lane * v.cs] : 1.f;
  const float rhs = in ? v.x[lane * v.xs] : 0.f;
  const float inv = 1.f / d;
  float r = rhs;
#pragma unroll
  for (int g = 0; g < kBTSmall; g += 8)
    if (g < n)
#pragma unroll
      for (int c = g; c < g + 8; ++c) {
        const float t = r * inv, x = fmaf(fmaf(-t, d, r), inv, t);
        const float xc = __shfl_sync(0xffffffffu, x, c);
        r = lane > c ? fmaf(-a[c], xc, r) : lane == c ? x : r;
      }
  if (!__all_sync(0xffffffffu, fabsf(d) > 0x1p-60f && fabsf(d) < 0x1p60f && fabsf(r) < INFINITY)) {
    r = rhs;
#pragma unroll 1
    for (int c = 0; c < n; ++c) {
      const float x = __shfl_sync(0xffffffffu, r, c) / __shfl_sync(0xffffffffu, d, c);
      if (lane == c) r = x;
      if (in && lane > c) r = fmaf(-row[c * v.cs], x, r);
    }
  }
  if (in) v.x[lane * v.xs] = r;
}

// First CTA that starts in window w, of `grid` CTAs over nwin windows.
__device__ __forceinline__ int trsv_first_cta(int w, int nwin, int grid) { return (w * grid + nwin - 1) / nwin; }
// One thread: the next position of the window, or -1.  Every CTA draws one position too
// many.  With one window the CTA that draws the last of those returns the ticket to
// zero; with more, a window without positions is marked.
__device__ __noinline__ void trsv_draw(TrsvWindow& win, const TrsvProblem* __restrict__ probs, unsigned* tickets,
                                       int nwin, int own) {
  const unsigned units = win.units;
  const unsigned d = own < (int)units ? (unsigned)own : win.first + atomicAdd(&tickets[win.w], 1u);
  if (d >= units) {
    if (nwin > 1) atomicOr(&tickets[win.w], kBTSpent);
    else if (d - units == gridDim.x - 1) tickets[0] = 0u;
  }
  win.drawn = d < units ? (int)d : -1;
  if (d < (unsigned)win.big) win.cur = probs[win.w * kBTWindow + win.ord[d]];
}

// One CTA: a system of any size.
__device__ __forceinline__ void trsv_solve_cta(const TrsvProblem& pr, TrsvSmem& sm) {
  const TrsvProblem p = pr;
  if (p.n <= 0) return;
  const bool t = p.trans != CORAL_NO_TRANSPOSE, unit = p.diag == CORAL_UNIT;
  const TrsvView v = trsv_view(p);
  const int n = v.n, nblk = (n + kBT - 1) / kBT;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool in_smem = n <= kBTMaxX;

  trsv_fetch(v, 0, false, sm, warp, kBTThreads / 32, !t);
  if (nblk > 1) trsv_fetch(v, 1, true, sm, warp, kBTThreads / 32, !t);
  if (in_smem)
    for (int i = threadIdx.x; i < n; i += kBTThreads) sm.x[i] = v.x[i * v.xs];
  auto rhs = [&](int i) { return i >= n ? 0.f : in_smem ? sm.x[i] : v.x[i * v.xs]; };
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (n < kBT) trsv_pad(sm, 0, n);
  else if (nblk == 2 && n < 2 * kBT) trsv_pad(sm, 1, n - kBT);
  __syncthreads();
  bool ok = true;
  if (threadIdx.x < kBT) ok = trsv_recip(sm, 0, threadIdx.x, unit);
  bool fast = __syncthreads_and(ok);
  if (warp == 0) {
    const float r2[2] = {rhs(lane), rhs(lane + 32)};
    trsv_solve(sm, 0, fast, r2);
    if (lane < n) v.x[lane * v.xs] = sm.xb[0][lane];
    if (lane + 32 < n) v.x[(lane + 32) * v.xs] = sm.xb[0][lane + 32];
  }
  __syncthreads();
  for (int b = 0; b + 1 < nblk; ++b) {
    const float* xb = sm.xb[b & 1];
    // Rows of block b + 1: everything up to block b - 1 is already off them;
    // take block b off (4 threads a row, every warp), then one warp solves.
    const int b1 = (b + 1) * kBT;
    {
      const float(*S)[kBTLs] = sm.S[b & 1];
      const int row = threadIdx.x % kBT, part = threadIdx.x / kBT;  // a warp: 32 rows, 16 columns
      float a0 = 0.f, a1 = 0.f;
#pragma unroll
      for (int c = 0; c < 16; c += 4) {
        const float4 x4 = *reinterpret_cast<const float4*>(xb + part * 16 + c);
        a0 = fmaf(S[part * 16 + c][row], x4.x, a0);
        a1 = fmaf(S[part * 16 + c + 1][row], x4.y, a1);
        a0 = fmaf(S[part * 16 + c + 2][row], x4.z, a0);
        a1 = fmaf(S[part * 16 + c + 3][row], x4.w, a1);
      }
      sm.part[part][row] = a0 + a1;
      ok = part != 3 || trsv_recip(sm, b + 1, row, unit);
    }
    fast = __syncthreads_and(ok);
    if (warp == 0) {
      float r2[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = lane + 32 * h;
        r2[h] = rhs(b1 + r) - ((sm.part[0][r] + sm.part[1][r]) + (sm.part[2][r] + sm.part[3][r]));
      }
      trsv_solve(sm, b + 1, fast, r2);
      const float* xn = sm.xb[(b + 1) & 1];
      if (b1 + lane < n) v.x[(b1 + lane) * v.xs] = xn[lane];
      if (b1 + lane + 32 < n) v.x[(b1 + lane + 32) * v.xs] = xn[lane + 32];
    } else {
      const int tb = threadIdx.x - 32;
      if (b + 2 < nblk) trsv_fetch(v, b + 2, true, sm, warp - 1, kBTBulk / 32, !t);
      const int lo = (b + 2) * kBT;
      const float* col = v.a + (long long)b * kBT * v.cs;
      if (!t) {
        // kRows rows per thread, 16 loads per row before their sums
        for (int i = lo + tb; i < n; i += kRows * kBTBulk) {
          const float* pr[kRows];
#pragma unroll
          for (int q = 0; q < kRows; ++q) pr[q] = col + min(i + q * kBTBulk, n - 1) * v.rs;
          const int rows = min(kRows, (n - i + kBTBulk - 1) / kBTBulk);
          float sum[kRows][2] = {};
#pragma unroll 1
          for (int c0 = 0; c0 < kBT; c0 += 16) {
            float a[kRows][16];
#pragma unroll
            for (int q = 0; q < kRows; ++q)
              if (q < rows)
#pragma unroll
                for (int c = 0; c < 16; ++c) a[q][c] = pr[q][(c0 + c) * v.cs];
#pragma unroll
            for (int c = 0; c < 16; c += 4) {
              const float4 x4 = *reinterpret_cast<const float4*>(xb + c0 + c);
#pragma unroll
              for (int q = 0; q < kRows; ++q)
                if (q < rows) {
                  sum[q][0] = fmaf(a[q][c], x4.x, sum[q][0]);
                  sum[q][1] = fmaf(a[q][c + 1], x4.y, sum[q][1]);
                  sum[q][0] = fmaf(a[q][c + 2], x4.z, sum[q][0]);
                  sum[q][1] = fmaf(a[q][c + 3], x4.w, sum[q][1]);
                }
            }
          }
#pragma unroll
          for (int q = 0; q < kRows; ++q)
            if (q < rows) {
              const int k = i + q * kBTBulk;
              if (in_smem) sm.x[k] -= sum[q][0] + sum[q][1];
              else v.x[k * v.xs] -= sum[q][0] + sum[q][1];
            }
        }
      } else {
        // stored along the row: a warp reads 8 rows, lanes along the columns
        const float x0 = xb[lane], x1 = xb[lane + 32];
        for (int i = lo + (warp - 1) * 8; i < n; i += (kBTBulk / 32) * 8) {
          float a[8], d[8];
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            const float* pr = col + min(i + r, n - 1) * v.rs;
            a[r] = pr[lane * v.cs];
            d[r] = pr[(lane + 32) * v.cs];
          }
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            float sum = fmaf(d[r], x1, a[r] * x0);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            a[r] = sum;
          }
          float mine = a[0];
#pragma unroll
          for (int r = 1; r < 8; ++r) mine = lane == r ? a[r] : mine;
          if (lane < 8 && i + lane < n) {
            if (in_smem) sm.x[i + lane] -= mine;
            else v.x[(i + lane) * v.xs] -= mine;
          }
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
    // (the last block's copies were waited for by the threads that made them)
    __syncthreads();
    if (b + 3 == nblk && n < nblk * kBT) {
      trsv_pad(sm, nblk - 1, n - (nblk - 1) * kBT);
      __syncthreads();
    }
  }
}

// Without tickets a CTA takes the instance of its index.  With them (one per window,
// then the number of CTAs that have finished; all zero before and after) the CTAs
// stay and draw.  Against a CTA per position, each of which looked its instance up (3
// us): batches of many small systems gain most, 300 of 900 to 1300 rows 206 -> 201,
// and where the longest system decides the end costs 1 us (1024 in [32, 1024] 106.4
// -> 107.2).  Drawing while the last block is solved does not take that back.
__global__ void __launch_bounds__(kBTThreads, 2)
k_trsv_batched(const TrsvProblem* __restrict__ probs, int count, unsigned* tickets) {
  TrsvSmem& sm = *reinterpret_cast<TrsvSmem*>(trsv_smem);
  TrsvWindow& win = sm.win;   // (no register holds it over a solve)
  const int nwin = (int)(((unsigned)count + kBTWindow - 1) / kBTWindow);
  if (!tickets) {
    if (tid_now() == 0) win.cur = probs[blockIdx.x];
  } else if (tid_now() == 0) {
    win.w = (int)(blockIdx.x * (unsigned)nwin / gridDim.x);
    win.units = 0;   // nothing sorted yet
    win.first = -1;  // nothing drawn yet
  }
  __syncthreads();
  for (;;) {
    if (tickets) {
      if (win.units == 0) {
        const int b = trsv_order(probs, count, win.w * kBTWindow, sm);
        if (tid_now() == 0) {
          win.local = min(kBTWindow, count - win.w * kBTWindow);
          win.big = b;
          win.units = b + (win.local - b + kBTWarps - 1) / kBTWarps;
          const int f = trsv_first_cta(win.w, nwin, gridDim.x);
          // first positions: the second half backwards, so that the CTA that shares an SM
          // with the longest system starts on the shortest of this wave
          int own = win.units;
          if (win.first < 0) {
            const int c = trsv_first_cta(win.w + 1, nwin, gridDim.x) - f, h = c / 2;
            own = (int)blockIdx.x - f;
            if (own >= h) own = h + (c - 1 - own);
          }
          win.first = min(win.units, trsv_first_cta(win.w + 1, nwin, gridDim.x) - f);
          trsv_draw(win, probs, tickets, nwin, own);
        }
        __syncthreads();
      }
      const int u = win.drawn;
      if (u < 0) {
        // on to the next window that has a position left, if any
        if (nwin == 1) break;
        __syncthreads();
        if (tid_now() == 0) win.next = nwin;
        __syncthreads();
        for (int i = 1 + tid_now(); i < nwin; i += kBTThreads)
          if (!(*(volatile unsigned*)&tickets[(win.w + i) % nwin] & kBTSpent)) {
            atomicMin(&win.next, i);
            break;
          }
        __syncthreads();
        if (win.next == nwin) break;
        __syncthreads();
        if (tid_now() == 0) {
          win.w = (win.w + win.next) % nwin;
          win.units = 0;
        }
        __syncthreads();
        continue;
      }
      if (u >= win.big) {
        __syncthreads();   // `drawn` is read
        if (tid_now() == 0) trsv_draw(win, probs, tickets, nwin, win.units);
        const int pos = win.big + (u - win.big) * kBTWarps + (tid_now() >> 5);
        if (pos < win.local) trsv_small(probs[win.w * kBTWindow + win.ord[pos]]);
        __syncthreads();
        continue;
      }
    }
    trsv_solve_cta(win.cur, sm);
    if (!tickets) return;
    __syncthreads();
    if (tid_now() == 0) trsv_draw(win, probs, tickets, nwin, win.units);
    __syncthreads();   // before the buffers are written again
  }
  // with more windows than one, the last CTA to come here returns the tickets to zero
  if (nwin > 1 && tid_now() == 0) {
    __threadfence();
    if (atomicAdd(&tickets[nwin], 1u) == gridDim.x - 1)
      for (int i = 0; i <= nwin; ++i) tickets[i] = 0u;
  }
}

// The tickets of one call, zero before and after it; null: there are none to be had,
// the solves go in input order.  Calls that may run at the same time have tickets of
// their own.  The calls on streams take theirs in turn from a ring; a captured call
// may run again beside any other, so it keeps its own (a word up to 1024 systems).
unsigned* trsv_tickets(Handle* h, size_t nwin) {
  const size_t need = nwin > 1 ? nwin + 1 : 1, ring = kTicketKept - kTrsvFlagBase;
  if (capture_of(h->stream)) {
    if (need > kCounterPool - kTicketKept - h->tickets_kept) return nullptr;
    h->tickets_kept += need;
    return h->counters + kTicketKept + h->tickets_kept - need;
  }
  if (need > ring) return nullptr;
  own_state(h);   // the ring comes round
  if (need > ring - h->ticket_next) h->ticket_next = 0;
  h->ticket_next += need;
  return h->counters + kTrsvFlagBase + h->ticket_next - need;
}

}  // namespace
}  // namespace coral

using namespace coral;

extern "C" {

coral_status_t coral_sgemm_grouped(coral_handle_t hh, int input_type, size_t count,
                                   const coral_sgemm_problem_t* problems) {
  CORAL_HANDLE(hh);
  if (input_type != CORAL_INPUT_F32 && input_type != CORAL_INPUT_BF16) return bad_arg(H, 1);
  if (count == 0) return CORAL_OK;
  if (!problems) return bad_arg(H, 3);
  if (count > (size_t)INT32_MAX / 2) return CORAL_ERR_NOT_SUPPORTED;
  // Tensor cores for bf16 inputs and for fp32 inputs in split-BF16x3 mode;
  // exact FP32 FMA tiles otherwise (NATIVE, and SPLIT_BF16X6, whose error
  // bound the two-piece split does not meet).
  if (input_type == CORAL_INPUT_BF16 || H->gemm_mode == CORAL_GEMM_SPLIT_BF16X3)
    return enqueue_grouped_tc(H, input_type == CORAL_INPUT_BF16, count, problems);
  int* prefix = static_cast<int*>(scratch(H, (count + 1) * sizeof(int)));
  if (!prefix) return CORAL_ERR_ALLOC;
  const GemmProblem* pr = reinterpret_cast<const GemmProblem*>(problems);
  k_tile_prefix<<<1, 1024, 0, H->stream>>>(pr, (int)count, prefix);
  coral_status_t s = launch_status(H);
  if (s != CORAL_OK) return s;
  const unsigned grid = (unsigned)H->sm_count * 4;
  timed_begin(H);
  if (input_type == CORAL_INPUT_F32)
    k_gemm_grouped<float><<<grid, kGThreads, 0, H->stream>>>(pr, (int)count, prefix);
  else
    k_gemm_grouped<__nv_bfloat16><<<grid, kGThreads, 0, H->stream>>>(pr, (int)count, prefix);
  s = launch_status(H);
  timed_end(H);
  return s;
}

coral_status_t coral_set_grouped_config(coral_handle_t hh, const int tile_n[4]) {
  CORAL_HANDLE(hh);
  if (!tile_n) {
    H->grouped_policy = GroupedPolicy{{64, 128, 128, 256}};
    return CORAL_OK;
  }
  for (int i = 0; i < 4; ++i)
    if (tile_n[i] != 64 && tile_n[i] != 128 && tile_n[i] != 256) return bad_arg(H, 1);
  for (int i = 0; i < 4; ++i) H->grouped_policy.bn[i] = tile_n[i];
  return CORAL_OK;
}

coral_status_t coral_get_grouped_config(coral_handle_t hh, int tile_n[4]) {
  CORAL_HANDLE(hh);
  if (!tile_n) return bad_arg(H, 1);
  for (int i = 0; i < 4; ++i) tile_n[i] = H->grouped_policy.bn[i];
  return CORAL_OK;
}

coral_status_t coral_strsv_batched(coral_handle_t hh, size_t count,
                                   const coral_strsv_problem_t* problems) {
  CORAL_HANDLE(hh);
  if (count == 0) return CORAL_OK;
  if (!problems) return bad_arg(H, 2);
  if (count > (size_t)INT32_MAX) return CORAL_ERR_NOT_SUPPORTED;
  static uint64_t attr_devices = 0;  // bit d: attribute set on device d
  const uint64_t bit = H->device < 64 ? (1ull << H->device) : 0;
  if (!(attr_devices & bit) || !bit) {
    CORAL_CUDA(H, cudaFuncSetAttribute(k_trsv_batched, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(TrsvSmem)));
    attr_devices |= bit;
  }
  // Past two CTAs per SM the order of the solves matters: fixed CTAs that draw.
  const size_t slots = (size_t)H->sm_count * 2;
  unsigned* tickets = count > slots ? trsv_tickets(H, (count + kBTWindow - 1) / kBTWindow) : nullptr;
  timed_begin(H);
  k_trsv_batched<<<(unsigned)(tickets ? slots : count), kBTThreads, sizeof(TrsvSmem), H->stream>>>(
      reinterpret_cast<const TrsvProblem*>(problems), (int)count, tickets);
  coral_status_t s = launch_status(H);
  timed_end(H);
  return s;
}

}  // extern "C"
