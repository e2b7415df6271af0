// DTRSV, CTRSV, ZTRSV: solve op(A) x = b in place, A triangular, op in
// {N, T, C} (dtrsv.rs, ctrsv.rs, ztrsv.rs -> the *trlsv / *trusv files).
// Complex data is interleaved (re, im) with lda / incx in complex units.
//
// One launch, one 64-row block of the solve per CTA, in clusters of 16 CTAs
// (8 where 16 cannot be placed).  Rank 0 of each cluster takes a ticket, so
// the cluster with ticket t solves blocks 16 t .. 16 t + 15 in solve order and
// only waits for clusters that started earlier -- no deadlock whatever the
// scheduling.  A CTA
//   1. stages its diagonal block of op(A) in shared memory (unstored triangle
//      masked, unit diagonal applied, conjugated for op C), forms the
//      reciprocals of its diagonal and scales each row by its reciprocal
//      (negated, ready for the updates), and reads its right-hand side;
//   2. for every earlier block k in solve order: holds its panel tile of
//      op(A) in registers (loaded while block k - 1 was waited for), reads x_k
//      from block k's published slots and accumulates op(A)(b, k) x_k -- four
//      threads per row, 16 columns each;
//   3. solves the row-scaled system by forward (backward) substitution in
//      one warp, fully unrolled (the diagonal block is never inverted: FP64
//      substitution as the reference does, dtrlsv.rs), and pushes the result
//      from its registers into the shared memory of the next CTA;
//   4. writes x_b over b, pushes it to the cluster's other later CTAs and
//      publishes it in its slots for later clusters: within a cluster a block's
//      solution reaches the next one through distributed shared memory instead
//      of an L2 round trip.
// Bound: the chain of n / 64 hops (the 67 MB of DTRSV's n = 4096 triangle would
// stream in 10 us).  A hop's cycles in DTRSV, before and after this form: last
// tile's products and reduction 1250 -> 630 (pairs of x_k by 16-byte loads that
// neighbouring lanes share, on padded banks), substitution 2640 -> 1600 (see
// substitute()), hand-over about 700.  n = 4096, op N: DTRSV 153 -> 105 us,
// CTRSV 172 -> 124, ZTRSV 262 -> 184; n = 16384: 797 -> 610, 827 -> 645,
// 1464 -> 1046; n = 64 (the reciprocals of the diagonal in one division per lane,
// the loads all in flight): 8.6 -> 5.2, 9.6 -> 5.9, 10.5 -> 7.3.
// Slots: every 32-bit word of a block's solution is published as one 64-bit
// slot (epoch << 32) | word, so a single load delivers both the readiness of
// that word and its value (aligned 64-bit accesses are single-copy atomic):
// a consumer's poll is its data load.  The last CTA resets the ticket counter
// and publishes the call's epoch, so no reset pass is needed.  Waits give up
// after the handle's wait limit and set the status word.
#include "common.cuh"
#include "field.cuh"
#include "tc_common.cuh"

#include <type_traits>

namespace coral {
namespace {

// Block edge: 64 rows for every element type, four threads per block row.
// 128-row blocks halve the serial hand-offs but double each block's
// substitution chain; at n = 4096 they measured slower (dtrsv 253 against
// 200 us, ctrsv 250 against 187 us), and a complex128 block of 128 rows
// would not fit in shared memory.
template <typename T> constexpr int kTBOf = 64;
// Rows solved together (see substitute()).
template <typename T> constexpr int kCornerOf = std::is_same<T, double>::value ? 8 : 4;
// Row pitch of the diagonal block in shared memory: 16-byte aligned pairs of
// columns, and lanes on consecutive rows on different banks.
template <typename T> constexpr int kPitchOf = kTBOf<T> + (sizeof(T) == 16 ? 1 : 2);
template <typename T> struct alignas(16) Two { T x, y; };

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// Cluster shared-memory accesses: a 32-bit load from another CTA's shared
// memory, a 64-bit store into it, and a 64-bit load of this CTA's shared
// memory that observes those stores.
__device__ __forceinline__ unsigned ld_cluster_u32(uint32_t addr) {
  unsigned v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster_u64(uint32_t addr, unsigned long long v) {
  asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_local_tag(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.cluster.shared::cta.u64 %0, [%1];" : "=l"(v) : "r"(tc::smem_u32(p)) : "memory");
  return v;
}
constexpr int kDczClMax = 16;  // CTAs per cluster: 16, or 8 where 16 cannot be placed

// 32-bit words per element (slots per element).
template <typename T> constexpr int kWords = (int)(sizeof(T) / 4);

// Substitution on the row-scaled diagonal block in one warp, fully unrolled, by
// corners of B rows.  D (in solve order) holds -op(A)(i, j) / op(A)(i, i) below
// the diagonal and v the scaled right-hand side of rows lane + 32 h, so every
// x_i is its row's final v_i.  The lanes that own the next B rows hand them to
// all (xs, two halves in turn); every lane solves their B x B corner -- the same
// products in every lane, but one multiply-add per row on the chain and no
// exchange -- while it takes the products off its own later rows.  Cycles of the
// 64 rows, one warp alone, double: 1540 (B = 8), 1800 (B = 4), 2290 by one
// broadcast per row; a wider product makes the 28 of an 8 x 8 corner the bound,
// so complex takes B = 4 (complex64 3260 -> 1950, complex128 4400 -> 3150).
template <typename T, int TB, int B, int P>
__device__ __forceinline__ void substitute(const T* D, T* xs, T (&v)[TB / 32], int lane) {
  using F = Fld<T>;
  using T2 = Two<T>;
  constexpr int H = TB / 32, C = 32 / B;
#pragma unroll
  for (int s = 0; s < TB / B; ++s) {
    T2 co[B][B / 2], ro[H][B / 2];
#pragma unroll
    for (int j = 0; j < B / 2; ++j) {
#pragma unroll
      for (int i = 2 * j + 1; i < B; ++i)
        co[i][j] = *reinterpret_cast<const T2*>(D + (B * s + i) * P + B * s + 2 * j);
    }
    T* xb = xs + B * (s & 1);
    if (lane / B == s % C) xb[lane % B] = v[s / C];
    __syncwarp();
    T q[B];
#pragma unroll
    for (int j = 0; j < B; j += 2) {
      const T2 t = *reinterpret_cast<const T2*>(xb + j);
      q[j] = t.x;
      q[j + 1] = t.y;
    }
#pragma unroll
    for (int j = 0; j < B / 2; ++j)
#pragma unroll
      for (int h = 0; h < H; ++h)
        if (32 * (h + 1) > B * (s + 1))
          ro[h][j] = *reinterpret_cast<const T2*>(D + (lane + 32 * h) * P + B * s + 2 * j);
    T w[H];
#pragma unroll
    for (int h = 0; h < H; ++h) w[h] = v[h];
#pragma unroll
    for (int j = 0; j < B; ++j) {
#pragma unroll
      for (int i = j + 1; i < B; ++i) F::mac(q[i], j & 1 ? co[i][j / 2].y : co[i][j / 2].x, q[j]);
#pragma unroll
      for (int h = 0; h < H; ++h)
        if (32 * (h + 1) > B * (s + 1)) F::mac(w[h], j & 1 ? ro[h][j / 2].y : ro[h][j / 2].x, q[j]);
    }
    T own[B];  // q[lane % B], by bits (indexing q would put it in local memory)
#pragma unroll
    for (int j = 0; j < B; ++j) own[j] = q[j];
#pragma unroll
    for (int m = B / 2; m > 0; m /= 2)
#pragma unroll
      for (int j = 0; j < m; ++j) own[j] = lane & m ? own[j + m] : own[j];
#pragma unroll
    for (int h = 0; h < H; ++h)
      if (lane + 32 * h >= B * (s + 1)) v[h] = w[h];
    if (lane / B == s % C) v[s / C] = own[0];
  }
}
__device__ __forceinline__ uint64_t gtime() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

template <typename T, bool kConj, int kTB = kTBOf<T>, int kTThr = 4 * kTBOf<T>>
// Two CTAs per SM where the registers allow it: past 148 blocks the CTAs that
// wait no longer keep later ones out (DTRSV n = 16384: 820 us with one, 610 with
// two; n = 4096, all resident either way, 106 against 110).  complex128 keeps
// one: its two tiles take 128 registers.
__global__ void __launch_bounds__(kTThr, sizeof(T) == 16 ? 1 : 2)
k_trsv_g(int n, const T* __restrict__ A, size_t lda, T* x, size_t incx, bool lower_eff, bool trans,
         bool unit, unsigned long long* slots, unsigned* ticket, unsigned* done, unsigned* epoch_word,
         unsigned* status, uint64_t limit_ns) {
  using F = Fld<T>;
  constexpr int W = kWords<T>;
  constexpr int kSlotWords = kTB * W;   // slots per block (<= kTThr)
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int kP = kPitchOf<T>;
  T* D = reinterpret_cast<T*>(smem);   // diagonal block of op(A), in solve order
  // solutions pushed by the earlier CTAs of the cluster: xin[rank][word]
  unsigned long long(*xin)[kSlotWords] =
      reinterpret_cast<unsigned long long(*)[kSlotWords]>(smem + sizeof(T) * kTB * kP);
  __shared__ __align__(16) T xk[2][kTB + 2 * 4];  // solution of the block being applied (even, odd)
  __shared__ T rv[kTB];        // right-hand side, then this block's solution
  __shared__ __align__(16) T xs[2 * kCornerOf<T>];
  __shared__ T rdiag[kTB];     // reciprocals of the diagonal
  __shared__ int gave_up[2];   // a wait of the even / odd block ran out
  __shared__ unsigned sticket, sepoch, my_ticket, my_epoch;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nblk = (n + kTB - 1) / kTB;
  const unsigned rank = tc::cluster_ctarank();
  unsigned ncl_u;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(ncl_u));
  const int ncl = (int)ncl_u;
  for (int i = tid; i < ncl * kSlotWords; i += kTThr) (&xin[0][0])[i] = 0ull;
  if (tid == 0) {
    gave_up[0] = gave_up[1] = 0;
    if (rank == 0) {
      // one ticket per cluster: the cluster takes the next ncl blocks in solve
      // order, so it only ever waits for clusters that started earlier
      sticket = atomicAdd(ticket, 1u);
      const unsigned e = *(volatile unsigned*)epoch_word + 1u;
      sepoch = e ? e : 1u;   // slots start at 0: never a live epoch
    }
  }
  tc::cluster_sync();
  if (tid == 0) {
    my_ticket = ld_cluster_u32(tc::mapa_shared(tc::smem_u32(&sticket), 0));
    my_epoch = ld_cluster_u32(tc::mapa_shared(tc::smem_u32(&sepoch), 0));
  }
  __syncthreads();
  const unsigned epoch = my_epoch;
  const int s_first = (int)my_ticket * ncl;   // solve index of this cluster's rank 0
  const int s = s_first + (int)rank;          // this CTA's solve index
  const bool active = s < nblk;
  auto blk_of = [&](int sp) { return lower_eff ? sp : nblk - 1 - sp; };
  const int blk = active ? blk_of(s) : 0;
  const int b0 = blk * kTB;
  // row or column of the block <-> its place in the order of the solve
  auto order_of = [&](int i) { return lower_eff ? i : kTB - 1 - i; };
  auto opv = [](T v) { return kConj ? F::conj(v) : v; };

  if (active) {
  // ---- 1. diagonal block, its reciprocals, the row scaling; right-hand side ----
  constexpr int kQ = kTB / 4;           // columns per thread of a panel tile
  static_assert(kSlotWords <= kTThr && kTThr == 4 * kTB, "one slot per thread, four threads per row");
  const int r = (tid >> 3) * 2 + (tid & 1), q = (tid >> 1) & 3;
  T a[kQ];                              // panel tile, loaded ahead; the diagonal block first
#pragma unroll
  for (int u = 0; u < kQ; ++u) {
    const int rr = tid % kTB, cc = tid / kTB + 4 * u;  // stored element (b0 + rr, b0 + cc)
    const int gr = b0 + rr, gc = b0 + cc;
    a[u] = (gr < n && gc < n) ? A[gr + (size_t)gc * lda] : F::zero();
  }
  const T rhs = b0 + r < n ? x[(size_t)(b0 + r) * incx] : F::zero();
  if (tid < kTB) {   // one division per lane; the element comes again from L1
    const size_t gd = b0 + tid;
    rdiag[tid] = F::div(F::one(), unit || gd >= (size_t)n ? F::one() : opv(A[gd + gd * lda]));
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kQ; ++u) {
    const int rr = tid % kTB, cc = tid / kTB + 4 * u;
    const int ir = trans ? cc : rr, ic = trans ? rr : cc;   // op(A)(ir, ic)
    const bool in_tri = lower_eff ? ir > ic : ir < ic;
    if (ir != ic) D[order_of(ir) * kP + order_of(ic)] = F::neg(F::mul(in_tri ? opv(a[u]) : F::zero(), rdiag[ir]));
  }

  // Panel tile of the block of solve index idx.  Thread (r, q) takes columns
  // q * kQ + j of the tile when A is read as stored (lanes of a warp on 8
  // consecutive rows of 4 column runs), and the pairs at 2 q + 8 j when it is
  // read transposed, where the 4 threads of a row then read 8 consecutive
  // elements of one stored column (with 16 in a run instead DTRSV T took 1.6
  // times as long at n = 4096).  The tile is held as stored; the conjugation of
  // op C is applied where an element is used.
  auto load_tile = [&](int idx, T (&t)[kQ]) {
    const int k0 = blk_of(idx) * kTB;
#pragma unroll
    for (int j = 0; j < kQ; ++j) {
      const int gr = b0 + r, gc = k0 + (trans ? 2 * q + 8 * (j / 2) + j % 2 : q * kQ + j);   // op(A)(gr, gc)
      const bool in = gr < n && gc < n;
      t[j] = in ? (trans ? A[gc + (size_t)gr * lda] : A[gr + (size_t)gc * lda]) : F::zero();
    }
  };

  bool aborted = false;
  // ---- 2. panel: sum over earlier blocks k of op(A)(b, k) x_k in solve
  // order; a block of this cluster is read from the copy its CTA pushed into
  // this CTA's shared memory, an earlier cluster's from its slots ----
  T acc[4] = {F::zero(), F::zero(), F::zero(), F::zero()};
  if (s > 0) load_tile(0, a);
  for (int idx = 0; idx < s; ++idx) {
    T ahead[kQ];
    if (idx + 1 < s) load_tile(idx + 1, ahead);
    if (tid < kSlotWords) {
      const bool local = idx >= s_first;
      const unsigned long long* sp =
          local ? &xin[idx - s_first][tid] : slots + (size_t)blk_of(idx) * kSlotWords + tid;
      unsigned long long w = local ? ld_local_tag(sp) : ld_relaxed_u64(sp);
      if ((unsigned)(w >> 32) != epoch) {
        const uint64_t t0 = gtime();
        for (unsigned spins = 1;; ++spins) {
          w = local ? ld_local_tag(sp) : ld_relaxed_u64(sp);
          if ((unsigned)(w >> 32) == epoch) break;
          const uint64_t el = gtime() - t0;
          if (el > limit_ns || ((spins & 15u) == 0 && el > 20000ull && *(volatile unsigned*)status != 0)) {
            atomicOr(status, kStatusTimeout);
            gave_up[idx & 1] = 1;
            break;
          }
        }
      }
      reinterpret_cast<uint32_t*>(xk[idx & 1])[tid + 2 * W * (tid / (kQ * W))] = (uint32_t)w;
    }
    __syncthreads();  // (the other half of xk is free: every thread passed here after using it)
    if (gave_up[idx & 1]) {  // (not written again before every thread is past here)
      aborted = true;
      break;
    }
#pragma unroll
    for (int j = 0; j < kQ; j += 2) {
      const Two<T> t = *reinterpret_cast<const Two<T>*>(
          &xk[idx & 1][trans ? 2 * q + 8 * (j / 2) + 2 * (j / 4) : q * (kQ + 2) + j]);
      F::mac(acc[j & 3], opv(a[j]), t.x);
      F::mac(acc[(j & 3) + 1], opv(a[j + 1]), t.y);
    }
#pragma unroll
    for (int j = 0; j < kQ; ++j) a[j] = ahead[j];
  }
  T sum = F::add(F::add(acc[0], acc[1]), F::add(acc[2], acc[3]));
  sum = F::add(sum, F::shfl_xor(sum, 2));
  sum = F::add(sum, F::shfl_xor(sum, 4));
  if (q == 0) rv[r] = F::mul(F::sub(rhs, sum), rdiag[r]);
  __syncthreads();

  // ---- 3. substitution on the row-scaled diagonal block (one warp), its
  // solution straight into the shared memory of the next CTA ----
  if (warp == 0) {
    T v[kTB / 32];
    int row[kTB / 32];
#pragma unroll
    for (int m = 0; m < kTB / 32; ++m) {
      row[m] = order_of(lane + 32 * m);
      v[m] = rv[row[m]];
    }
    substitute<T, kTB, kCornerOf<T>, kP>(D, xs, v, lane);
    const bool push = !aborted && (int)rank + 1 < ncl && s + 1 < nblk;
#pragma unroll
    for (int m = 0; m < kTB / 32; ++m) {
      if (push) {
        const uint32_t* words = reinterpret_cast<const uint32_t*>(&v[m]);
        const uint32_t next = tc::mapa_shared(tc::smem_u32(&xin[rank][row[m] * W]), rank + 1);
#pragma unroll
        for (int w = 0; w < W; ++w) st_cluster_u64(next + 8 * w, ((unsigned long long)epoch << 32) | words[w]);
      }
      rv[row[m]] = v[m];
    }
  }
  __syncthreads();

  // ---- 4. publish: x_b over b, every word of it into the shared memory of
  // the CTAs of the cluster after the next one and into the block's slots for
  // later clusters ----
  if (!aborted) {
    if (tid < kTB && b0 + tid < n) x[(size_t)(b0 + tid) * incx] = rv[tid];
    if (tid < kSlotWords) {
      const unsigned long long val =
          ((unsigned long long)epoch << 32) | reinterpret_cast<const uint32_t*>(rv)[tid];
      const uint32_t mine = tc::smem_u32(&xin[rank][tid]);
      st_relaxed_u64(slots + (size_t)blk * kSlotWords + tid, val);
      for (int d = (int)rank + 2; d < ncl && s_first + d < nblk; ++d)
        st_cluster_u64(tc::mapa_shared(mine, (uint32_t)d), val);
    }
  }
  }  // active
  // No CTA leaves while a CTA of its cluster may still push into it.
  __syncthreads();
  tc::cluster_sync();
  // The last CTA to finish (aborted or not) resets the ticket counter and
  // publishes this call's epoch for the next call.
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(done, 1u) == gridDim.x - 1) {
      *ticket = 0u;
      *done = 0u;
      __threadfence();
      atomicExch(epoch_word, epoch);
    }
  }
}

template <typename T>
coral_status_t trsv_g(Handle* H, int uplo, int trans, int diag, size_t n, const void* matrix, size_t lda,
                      void* x, size_t incx, size_t align) {
  if (uplo != CORAL_UPPER && uplo != CORAL_LOWER) return bad_arg(H, 1);
  if (trans < CORAL_NO_TRANSPOSE || trans > CORAL_CONJ_TRANSPOSE) return bad_arg(H, 2);
  if (diag != CORAL_UNIT && diag != CORAL_NON_UNIT) return bad_arg(H, 3);
  if (n == 0) return CORAL_OK;
  if (!matrix) return bad_arg(H, 5);
  if (lda < n) return bad_arg(H, 6);
  if (!x) return bad_arg(H, 7);
  if (incx == 0) return bad_arg(H, 8);
  if (((uintptr_t)matrix | (uintptr_t)x) & (align - 1)) return bad_arg(H, 5);
  if (n > (size_t)INT32_MAX) return CORAL_ERR_NOT_SUPPORTED;
  constexpr int kTB = kTBOf<T>, kTThr = 4 * kTBOf<T>;
  const size_t nblk = (n + kTB - 1) / kTB;
  const size_t nslots = nblk * kTB * kWords<T>;   // one slot per 32-bit word of x
  own_state(H);
  if (H->trsv_slots_len < nslots) {
    if (H->trsv_slots) {
      CORAL_CUDA(H, cudaStreamSynchronize(H->stream));
      cudaFree(H->trsv_slots);
      H->trsv_slots = nullptr;
      H->trsv_slots_len = 0;
    }
    const size_t len = ((nslots + 65535) / 65536) * 65536;
    CORAL_CUDA(H, cudaMalloc(&H->trsv_slots, len * sizeof(unsigned long long)));
    CORAL_CUDA(H, cudaMemsetAsync(H->trsv_slots, 0, len * sizeof(unsigned long long), H->stream));
    H->trsv_slots_len = len;
  }
  const bool t = trans != CORAL_NO_TRANSPOSE;
  const bool cj = trans == CORAL_CONJ_TRANSPOSE && !std::is_same<T, double>::value;
  const bool lower_eff = (uplo == CORAL_LOWER) != t;
  const size_t smem = (size_t)kTB * kPitchOf<T> * sizeof(T) + (size_t)kDczClMax * kTB * kWords<T> * 8;
  // per device and kernel form: the attributes are set, and the cluster size
  // (16 where the hardware places it, else 8) is chosen, on the first call
  static int cluster_size[2][64] = {{0}};
  int& cl = cluster_size[cj][H->device < 64 ? H->device : 63];
  auto kern = cj ? k_trsv_g<T, true> : k_trsv_g<T, false>;
  if (cl == 0) {
    CORAL_CUDA(H, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int c = 8;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
      cudaLaunchConfig_t q = {};
      cudaLaunchAttribute qa[1];
      qa[0].id = cudaLaunchAttributeClusterDimension;
      qa[0].val.clusterDim.x = 16;
      qa[0].val.clusterDim.y = qa[0].val.clusterDim.z = 1;
      q.gridDim = dim3(16);
      q.blockDim = dim3(kTThr);
      q.dynamicSmemBytes = smem;
      q.attrs = qa;
      q.numAttrs = 1;
      int activec = 0;
      if (cudaOccupancyMaxActiveClusters(&activec, kern, &q) == cudaSuccess && activec >= 1) c = 16;
    }
    cudaGetLastError();  // a refused query leaves the size at 8, not an error
    cl = c;
  }
  T* X = static_cast<T*>(x);
  const T* Am = static_cast<const T*>(matrix);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)cl;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(((nblk + cl - 1) / cl) * cl));
  cfg.blockDim = dim3(kTThr);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = H->stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  timed_begin(H);
  const cudaError_t le = cudaLaunchKernelEx(&cfg, kern, (int)n, Am, lda, X, incx, lower_eff, t, diag == CORAL_UNIT,
                                            H->trsv_slots, &H->words->trsv_ticket, &H->words->trsv_done,
                                            &H->words->trsv_epoch, &H->words->status, H->wait_limit * 32ull);
  if (le != cudaSuccess) {
    timed_end(H);
    count_launch();
    cudaGetLastError();
    return cuda_status(H, le);
  }
  coral_status_t s = launch_status(H);
  timed_end(H);
  return s;
}

}  // namespace
}  // namespace coral

using namespace coral;

extern "C" {

coral_status_t coral_dtrsv(coral_handle_t hh, int uplo, int trans, int diag, size_t n, const double* matrix,
                           size_t lda, double* x, size_t incx) {
  CORAL_HANDLE(hh);
  return trsv_g<double>(H, uplo, trans, diag, n, matrix, lda, x, incx, 8);
}

coral_status_t coral_ctrsv(coral_handle_t hh, int uplo, int trans, int diag, size_t n, const float* matrix,
                           size_t lda, float* x, size_t incx) {
  CORAL_HANDLE(hh);
  return trsv_g<float2>(H, uplo, trans, diag, n, matrix, lda, x, incx, 8);
}

coral_status_t coral_ztrsv(coral_handle_t hh, int uplo, int trans, int diag, size_t n, const double* matrix,
                           size_t lda, double* x, size_t incx) {
  CORAL_HANDLE(hh);
  return trsv_g<double2>(H, uplo, trans, diag, n, matrix, lda, x, incx, 16);
}

}  // extern "C"
