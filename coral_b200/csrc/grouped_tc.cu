// Grouped (uneven) SGEMM on the 5th-generation tensor cores (tcgen05 + TMEM).
//
// No reference counterpart: each instance has the semantics of coral_sgemm
// (sgemm.rs:106-130; quick returns sgemm_nn.rs:29-45; epilogue
// f32_edge.rs:37-58).  Two arithmetic forms share one kernel:
//   - bf16 inputs, fp32 accumulation: one tcgen05 product per K step;
//   - fp32 inputs as split-BF16x3: each value split into two bf16 pieces
//     (a = a0 + a1 + r, |r| <= 2^-18 |a|) and A0 B0 + A0 B1 + A1 B0 summed in
//     the fp32 TMEM accumulator, as the single split GEMM does.
//
// The instances' operands have arbitrary leading dimensions and alignments,
// which tensor maps cannot describe without per-instance host work, so the
// operands are staged by producer warps instead of TMA: blocks of 32 rows x 32
// K values, read in runs of consecutive elements whichever way the operand is
// stored, converted to bf16 pieces in registers and written into the K-major
// 64-byte-swizzled layout that a TMA CU_TENSOR_MAP_SWIZZLE_64B load would write,
// so the MMA descriptors are the same as the TMA-fed kernels'.
//
// Plan (k_grouped_plan, one CTA): every instance gets a tile width BN from the
// handle's per-class policy (classes by n: <= 64, <= 128, <= 256, > 256;
// BN in {64, 128, 256}; a descriptor's `reserved` field of 64/128/256
// overrides it), instances are ordered by decreasing K bucket (longest tiles
// first), and the exclusive prefix sum of 128 x BN output tiles is formed.
//
// GEMM (k_gemm_grouped_tc, persistent, one CTA per SM, 26 warps):
//   warp 0      scheduler: takes up to 4 tile indices at once from a global
//               atomic counter (dynamic load balance), finds their instances
//               with 8 lanes each, and publishes tile and descriptor through
//               a 16-deep shared queue (one tile at a time by one lane took
//               5 us a tile and bound the kernel at 310 us);
//   warps 1-16  producers, four groups: A of even slabs, A of odd ones, B of
//               even, B of odd, into a ring of shared-memory stages (4 for fp32
//               pieces, 8 for bf16); they also ask for the tile's C in L2;
//   warp 17     MMA issuer (lane 0): tcgen05.mma M=128, N=BN, K=16 into one of
//               two TMEM accumulators of 256 columns, in chunks of at most
//               32 slabs (1024 K) per accumulation;
//   warps 18-25 epilogue: tcgen05.ld the accumulator (thread = row, the two
//               warps of a quadrant on alternate 16 columns), apply alpha / beta
//               to C with coalesced column accesses, the C loads of the next 16
//               columns ahead of this group's stores; chunks after the first
//               add alpha * partial into C.
// Bound: issue slots (55% busy, a quarter of the stalls on instruction fetch)
// and the latency of the slabs; 4096 instances with sizes log-uniform in
// [16, 512] (1.34 GB, a floor of 208 us): fp32 810 -> 478 us, bf16 807 -> 450.
// 2000 of 128^3: fp32 197 -> 111 us, bf16 186 -> 98.  Timed apart (the other
// side's work left out): producers 350 us, epilogue 295, control alone 190.
// Few large instances whose operands both lie along K are what the 16-byte
// loads of the earlier form did better: 16 of 1024^3 transposed fp32 221 -> 250
// us, one 4096^3 in bf16 653 -> 725; their other orders gain (fp32 337 -> 224,
// bf16 1351 -> 562).  Wide loads here cost the batch above a fifth or more.
// Every wait is bounded: a wait that gives up sets the handle's status word
// (reported by coral_sync) and the CTA winds down.
#include "common.cuh"
#include "tc_common.cuh"

#include <cuda_bf16.h>

#include <type_traits>

namespace coral {
namespace {

constexpr int kTM = 128;          // tile rows (TMEM lanes)
constexpr int kTK = 32;           // K slab: one 64-byte swizzled row of bf16
constexpr int kMaxBN = 256;
constexpr int kProdWarps = 16;
constexpr int kEpiWarps = 8;
constexpr int kMmaWarp = 1 + kProdWarps;
constexpr int kEpiWarp0 = kMmaWarp + 1;
constexpr int kTcThreads = 32 * (kEpiWarp0 + kEpiWarps);  // 832
constexpr int kQueue = 16;
constexpr int kBatch = 4;   // tiles the scheduler looks up at once
constexpr int kChunkSlabs = 32;
constexpr uint32_t kAPieceBytes = kTM * kTK * 2;       // 8 KiB
constexpr uint32_t kBPieceBytes = kMaxBN * kTK * 2;    // 16 KiB

template <int NPC> struct TcCfg;
template <> struct TcCfg<2> {
  static constexpr int kStages = 4, kProducts = 3;
  // (A piece, B piece) per product, smallest terms first: A1 B0, A0 B1, A0 B0;
  // A0 stays in the tensor core's A collector between its two products
  __device__ static constexpr int a(int q) { return q == 0 ? 1 : 0; }
  __device__ static constexpr int b(int q) { return q == 1 ? 1 : 0; }
  __device__ static constexpr int collect(int q) {
    return q == 1 ? tc::kCollectFill : q == 2 ? tc::kCollectLastUse : tc::kCollectNone;
  }
};
template <> struct TcCfg<1> {
  static constexpr int kStages = 8, kProducts = 1;
  __device__ static constexpr int a(int) { return 0; }
  __device__ static constexpr int b(int) { return 0; }
  __device__ static constexpr int collect(int) { return tc::kCollectNone; }
};

template <int NPC>
constexpr uint32_t tc_stage_bytes() { return NPC * (kAPieceBytes + kBPieceBytes); }
template <int NPC>
constexpr size_t tc_smem_bytes() { return (size_t)TcCfg<NPC>::kStages * tc_stage_bytes<NPC>() + 1024; }

struct TileInfo {
  int more;    // 0: no more tiles
  int m0, n0, bn;
  int nslabs;  // K slabs; 0: scale-only tile (alpha == 0 or k == 0)
  coral_sgemm_problem_t p;  // the instance
};

__device__ __forceinline__ int policy_bn(const GroupedPolicy& pol, const coral_sgemm_problem_t& p) {
  if (p.reserved == 64 || p.reserved == 128 || p.reserved == 256) return p.reserved;
  const int cls = p.n <= 64 ? 0 : p.n <= 128 ? 1 : p.n <= 256 ? 2 : 3;
  return pol.bn[cls];
}

// One CTA.  order[pos] = instance, bn_pos[pos] = its tile width, prefix[pos] =
// tiles before position pos (prefix[count] = total).  Positions follow
// decreasing K bucket, so the longest tiles are handed out first.  K falls in a
// few buckets, so the shared counters are taken once per bucket and warp, not
// once per lane, and the prefix sum is one scan over per-thread runs (4096
// instances: 18 us with a counter access per lane and a scan per 1024).
__global__ void __launch_bounds__(1024, 1)
k_grouped_plan(const coral_sgemm_problem_t* __restrict__ probs, int count, GroupedPolicy pol,
               int* __restrict__ order, int* __restrict__ bn_pos, long long* __restrict__ prefix) {
  __shared__ int hist[32], cursor[32];
  __shared__ long long warp_tot[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x < 32) hist[threadIdx.x] = 0;
  __syncthreads();
  // what the plan needs of instance i, in two 16-byte loads where they are aligned
  struct Entry { int key, bn; long long tiles; };
  const bool vec = (reinterpret_cast<uintptr_t>(probs) & 15) == 0;
  auto fetch = [&](int i) -> Entry {
    if (i >= count) return {-1, 0, 0};
    coral_sgemm_problem_t p;
    int4 w[2];
    const int4* src = reinterpret_cast<const int4*>(probs + i);
    if (vec) {
      w[0] = src[0];
      w[1] = src[1];
    } else {
      const int2* s2 = reinterpret_cast<const int2*>(src);
      const int2 a = s2[0], b = s2[1], c = s2[2], d = s2[3];
      w[0] = make_int4(a.x, a.y, b.x, b.y);
      w[1] = make_int4(c.x, c.y, d.x, d.y);
    }
    p.m = w[0].z;
    p.n = w[0].w;
    p.k = w[1].x;
    p.alpha = __int_as_float(w[1].y);
    p.reserved = w[1].w;
    Entry e;
    e.key = p.m <= 0 || p.n <= 0 || p.k <= 0 || p.alpha == 0.f ? 0 : 31 - __clz(p.k);
    e.bn = policy_bn(pol, p);
    e.tiles = p.m > 0 && p.n > 0 ? (((long long)p.m + kTM - 1) / kTM) * (((long long)p.n + e.bn - 1) / e.bn) : 0;
    return e;
  };
  auto count_key = [&](int key) {
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    if (key >= 0 && lane == __ffs(peers) - 1) atomicAdd(&hist[key], __popc(peers));
  };
  auto place = [&](int i, const Entry& e) {
    const unsigned peers = __match_any_sync(0xffffffffu, e.key);
    const int leader = __ffs(peers) - 1;
    int pos = 0;
    if (e.key >= 0 && lane == leader) pos = atomicAdd(&cursor[e.key], __popc(peers));
    pos = __shfl_sync(0xffffffffu, pos, leader) + __popc(peers & ((1u << lane) - 1u));
    if (e.key >= 0) {
      order[pos] = i;
      bn_pos[pos] = e.bn;
      prefix[pos] = e.tiles;  // replaced by the sum below
    }
  };
  // up to 4096 instances stay in registers between the two passes
  constexpr int kKept = 4;
  const int rounds = (count + 1023) / 1024;
  Entry kept[kKept];
#pragma unroll
  for (int q = 0; q < kKept; ++q) kept[q] = fetch(q * 1024 + threadIdx.x);
#pragma unroll
  for (int q = 0; q < kKept; ++q)
    if (q < rounds) count_key(kept[q].key);
  for (int q = kKept; q < rounds; ++q) count_key(fetch(q * 1024 + threadIdx.x).key);
  __syncthreads();
  if (w == 0) {  // first position of each bucket, the deepest first
    int before = hist[31 - lane];
    const int own = before;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, before, o);
      if (lane >= o) before += u;
    }
    cursor[31 - lane] = before - own;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kKept; ++q)
    if (q < rounds) place(q * 1024 + threadIdx.x, kept[q]);
  for (int q = kKept; q < rounds; ++q) place(q * 1024 + threadIdx.x, fetch(q * 1024 + threadIdx.x));
  __syncthreads();
  const int per = (count + 1023) / 1024, lo = threadIdx.x * per, hi = min(count, lo + per);
  long long own = 0;
  for (int pos = lo; pos < hi; ++pos) own += prefix[pos];
  long long v = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  if (lane == 31) warp_tot[w] = v;
  __syncthreads();
  if (w == 0) {
    long long t = warp_tot[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long u = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += u;
    }
    warp_tot[lane] = t;
  }
  __syncthreads();
  long long run = (w ? warp_tot[w - 1] : 0) + v - own;
  for (int pos = lo; pos < hi; ++pos) {
    const long long t = prefix[pos];
    prefix[pos] = run;
    run += t;
  }
  if (threadIdx.x == 1023) prefix[count] = run;
}

// ---- producers' staging -------------------------------------------------------
// A group of 4 warps stages one operand of every other slab, 32 rows at a time
// (a "block"): each thread takes 8 values of a block, and the loads of
// kInFlight blocks are issued before any value is converted.  How the 8 values
// lie follows the operand's storage, so that every warp load reads one or two
// runs of consecutive elements:
//   along the rows:  one row (lane), 8 consecutive K values (one chunk per warp);
//   along K:         4 rows (2 apart), 2 consecutive K values (16 lanes a row).
// Either way value j lies (j >> 1) * s1 + (j & 1) * s0 from the first, so one
// piece of code loads both, and everything else is fixed per tile or moves by
// a fixed step from slab to slab: with the kernel bound by issue slots, not by
// memory, what a block costs is the instructions around its 8 loads.
constexpr int kGroups = 4, kGroupWarps = kProdWarps / kGroups;
constexpr int kInFlight = 4;
static_assert(kGroupWarps == 4, "the blocks below are laid out for 128 threads");

template <typename TIn>
__device__ __forceinline__ uint32_t ld_bits(const TIn* p) {
  if constexpr (sizeof(TIn) == 4) return __ldg(reinterpret_cast<const unsigned int*>(p));
  else return __ldg(reinterpret_cast<const unsigned short*>(p));
}

// One operand of a tile as a producer thread sees it.
template <typename TIn>
struct Operand {
  const TIn* p;        // this thread's first value of block 0 of the slab at hand
  long long s0, s1;    // from value 2i to 2i + 1, from 2i to 2i + 2
  long long block;     // from a block to the next
  int rows;            // rows of the tile inside the operand
  uint32_t dst;        // byte offset of this thread's part of block 0 in the stage
  bool along_k;

  __device__ __forceinline__ void init(const void* x, long long ld, bool along_k_, int row0, int rows_, int tid) {
    const int w = tid >> 5, lane = tid & 31;
    along_k = along_k_;
    rows = rows_;
    const TIn* base = static_cast<const TIn*>(x);
    if (along_k) {
      const int kp = lane & 15;
      p = base + (size_t)(row0 + 8 * w + (lane >> 4)) * ld + 2 * kp;
      s0 = 1;
      block = 32 * ld;
      dst = (uint32_t)(w * 512 + (lane >> 4) * 64 + (kp & 3) * 4 + ((kp >> 2) << 4));
    } else {
      p = base + row0 + lane + (size_t)(8 * w) * ld;
      s0 = ld;
      block = 32;
      dst = (uint32_t)((lane >> 3) * 512 + (lane & 7) * 64 + ((w ^ ((lane >> 1) & 3)) << 4));
    }
    s1 = 2 * ld;
  }
  // Values of block b that are inside: bit j for value j, `left` K values remain.
  __device__ __forceinline__ unsigned inside(int b, int left, int tid) const {
    const int w = tid >> 5, lane = tid & 31;
    if (along_k) {
      const int dr = rows - (32 * b + 8 * w + (lane >> 4)), dk = left - 2 * (lane & 15);
      const unsigned in_rows = dr <= 0 ? 0u : dr >= 7 ? 0xffu : (1u << (((dr + 1) >> 1) * 2)) - 1u;
      return in_rows & (dk >= 2 ? 0xffu : dk == 1 ? 0x55u : 0u);
    }
    const int dk = left - 8 * w;
    return 32 * b + lane >= rows || dk <= 0 ? 0u : dk >= 8 ? 0xffu : (1u << dk) - 1u;
  }
  // Loads the thread's 8 values (bits) of block b; zeros outside the operand.
  __device__ __forceinline__ void load(int b, int left, int tid, uint32_t (&v)[8]) const {
    const TIn* q = p + b * block;
    if (left >= kTK && 32 * b + 32 <= rows) {
#pragma unroll
      for (int j = 0; j < 8; j += 2, q += s1) {
        v[j] = ld_bits(q);
        v[j + 1] = ld_bits(q + s0);
      }
    } else {
      const unsigned ok = inside(b, left, tid);
#pragma unroll
      for (int j = 0; j < 8; j += 2, q += s1) {
        v[j] = v[j + 1] = 0u;
        if (ok & (1u << j)) v[j] = ld_bits(q);
        if (ok & (2u << j)) v[j + 1] = ld_bits(q + s0);
      }
    }
  }
};

// Two values as packed bf16 pieces (fp32: a = a0 + a1 + r; bf16: their bits).
template <typename TIn, int NPC>
__device__ __forceinline__ void pieces(uint32_t a, uint32_t b, uint32_t (&q)[NPC]) {
  if constexpr (sizeof(TIn) == 2) {
    q[0] = a | (b << 16);
  } else {
    const float fa = __uint_as_float(a), fb = __uint_as_float(b);
    const __nv_bfloat162 h = __floats2bfloat162_rn(fa, fb);
    q[0] = *reinterpret_cast<const uint32_t*>(&h);
    const __nv_bfloat162 l =
        __floats2bfloat162_rn(fa - __uint_as_float(q[0] << 16), fb - __uint_as_float(q[0] & 0xffff0000u));
    q[NPC - 1] = *reinterpret_cast<const uint32_t*>(&l);
  }
}

// Writes a block's values into the 64-byte-swizzled K-major tile (rows of 32
// bf16, 8-row / 512-byte atoms, 16-byte chunk c of row r at chunk c ^ ((r >> 1)
// & 3)); d: the thread's place in the block, piece i at d + i * piece_bytes.
template <typename TIn, int NPC>
__device__ __forceinline__ void store_block(bool along_k, uint8_t* d, uint32_t piece_bytes, const uint32_t (&v)[8]) {
  uint32_t q[4][NPC];
#pragma unroll
  for (int h = 0; h < 4; ++h) pieces<TIn, NPC>(v[2 * h], v[2 * h + 1], q[h]);
  if (along_k) {  // rows 2 apart: 128 bytes on, the chunk's low bits flipped
    const uint32_t chunk = tc::smem_u32(d) & 0x30u;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      uint8_t* da = d + (int)((chunk ^ (a << 4)) - chunk) + a * 128;
#pragma unroll
      for (int i = 0; i < NPC; ++i) *reinterpret_cast<uint32_t*>(da + i * piece_bytes) = q[a][i];
    }
  } else {
#pragma unroll
    for (int i = 0; i < NPC; ++i)
      *reinterpret_cast<uint4*>(d + i * piece_bytes) = make_uint4(q[0][i], q[1][i], q[2][i], q[3][i]);
  }
}

template <typename TIn, int NPC>
__global__ void __launch_bounds__(kTcThreads, 1)
k_gemm_grouped_tc(const coral_sgemm_problem_t* __restrict__ probs, int count,
                  const int* __restrict__ order, const int* __restrict__ bn_pos,
                  const long long* __restrict__ prefix, unsigned long long* tile_counter,
                  unsigned* status, uint64_t limit_ns) {
  using Cfg = TcCfg<NPC>;
  constexpr int S = Cfg::kStages;
  constexpr uint32_t kStage = tc_stage_bytes<NPC>();

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = tc::align1024_shared(smem_raw);
  __shared__ __align__(8) uint64_t full_bar[S], empty_bar[S];
  __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2];
  __shared__ __align__(8) uint64_t tq_full[kQueue], tq_empty[kQueue];
  __shared__ __align__(8) uint64_t drain_bar;
  __shared__ TileInfo tq[kQueue];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      tc::mbar_init(&full_bar[s], 2 * kGroupWarps);
      tc::mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&acc_full[b], 1);
      tc::mbar_init(&acc_empty[b], kEpiWarps);
    }
    for (int q = 0; q < kQueue; ++q) {
      tc::mbar_init(&tq_full[q], 1);
      tc::mbar_init(&tq_empty[q], kProdWarps + 1 + kEpiWarps);
    }
    tc::mbar_init(&drain_bar, 1);
    abort_flag = 0;
    tc::fence_mbar_init();
  }
  if (warp == kMmaWarp) {
    tc::tmem_alloc(&tmem_slot, 2 * kMaxBN);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = tmem_slot;

  auto give_up = [&]() {
    atomicOr(status, kStatusTimeout);
    atomicExch(&abort_flag, 1);
  };
  // Consumer side of the tile queue: the j-th tile of this CTA, which stays valid
  // until release_tile(j) (one arrival per consumer warp).  A whole warp calls it,
  // all of its lanes with the same answer, or one lane.  It is the only place where
  // the producers and the epilogue leave: their waits inside a tile may give up lane
  // by lane, so the tile is finished all the same, its slots not waited for and
  // nothing of it stored.  On the batch above, fp32 and bf16: 478 us and 450, as with
  // lanes that leave one by one and the rest at a full-warp barrier (480 and 448);
  // with a vote here 494 and 460, with one at each wait too 501 and 463.
  auto next_tile = [&](int j, bool whole_warp) -> const TileInfo* {
    const int q = j % kQueue;
    if (!tc::mbar_wait(&tq_full[q], (j / kQueue) & 1, limit_ns)) give_up();
    if (whole_warp) {
      __syncwarp();   // a lane that gave up has set the flag, and lane 0 reads it for all
      const int stop = *(volatile int*)&abort_flag;
      return __shfl_sync(0xffffffffu, stop, 0) == 0 && tq[q].more ? &tq[q] : nullptr;
    }
    return !*(volatile int*)&abort_flag && tq[q].more ? &tq[q] : nullptr;
  };
  auto release_tile = [&](int j) { tc::mbar_arrive(&tq_empty[j % kQueue]); };

  if (warp == 0) {
    // ---- scheduler: kBatch tiles at a time, 8 lanes each ----
    const long long total = prefix[count];
    // fewer at a time where each CTA gets a few only, down to one
    const int batch = (int)max(1ll, min((long long)kBatch, total / (4 * (long long)gridDim.x)));
    const int g = lane >> 3, sub = lane & 7;
    for (int j0 = 0;; j0 += batch) {
      const int j = j0 + g, q = j % kQueue;
      bool ok = true;
      if (sub == 0 && j >= kQueue && g < batch) ok = tc::mbar_wait(&tq_empty[q], ((j / kQueue) - 1) & 1, limit_ns);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) give_up();
        break;
      }
      long long t = 0;
      if (lane == 0) t = *(volatile int*)&abort_flag ? total : (long long)atomicAdd(tile_counter, (unsigned long long)batch);
      t = __shfl_sync(0xffffffffu, t, 0) + g;
      // last position with prefix <= t, an 8-way step at a time
      int lo = 0, hi = t < total ? count - 1 : 0;
      while (__any_sync(0xffffffffu, lo < hi)) {
        const int step = (hi - lo + 8) / 8, at = lo + (sub + 1) * step;
        const bool le = at <= hi && prefix[at] <= t;
        const int c = __popc((__ballot_sync(0xffffffffu, le) >> (8 * g)) & 0xffu);
        lo += c * step;
        hi = min(hi, lo + step - 1);
      }
      if (sub == 0 && g < batch) {
        TileInfo ti{};
        if (t < total) {
          ti.p = probs[order[lo]];
          ti.more = 1;
          ti.bn = bn_pos[lo];
          const long long local = t - prefix[lo];
          const int mt = (ti.p.m + kTM - 1) / kTM;
          ti.m0 = (int)(local % mt) * kTM;
          ti.n0 = (int)(local / mt) * ti.bn;
          ti.nslabs = (ti.p.alpha == 0.f || ti.p.k <= 0) ? 0 : (ti.p.k + kTK - 1) / kTK;
        }
        tq[q] = ti;
        tc::mbar_arrive(&tq_full[q]);
      }
      if (__shfl_sync(0xffffffffu, t, 8 * (batch - 1)) >= total) break;  // the batch held an end mark
    }
  } else if (warp < kMmaWarp) {
    // ---- producers: groups 0 and 1 stage A, 2 and 3 stage B, of even and odd slabs ----
    const int ptid = threadIdx.x - 32, group = ptid / (32 * kGroupWarps), tid = ptid % (32 * kGroupWarps);
    const bool is_a = group < 2;
    const uint32_t piece_bytes = is_a ? kAPieceBytes : kBPieceBytes;
    int it0 = 0;  // running number of the tile's first slab
    const TileInfo* tp;
    for (int j = 0; (tp = next_tile(j, true)); ++j) {
      const TileInfo& ti = *tp;
      const coral_sgemm_problem_t& p = ti.p;
      // C is read in the epilogue, a column at a time: bring it into L2 now
      if (p.beta != 0.f && !(p.beta == 1.f && ti.nslabs == 0)) {
        const int cols = min(ti.bn, p.n - ti.n0), row = ti.m0 + (ptid & 3) * 32;
        if (row < p.m)
          for (int c = ptid >> 2; c < cols; c += 8 * kProdWarps)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(p.c + row + (size_t)(ti.n0 + c) * p.ldc));
      }
      const int nslabs = ti.nslabs, kd = p.k;
      if (nslabs) {
        Operand<TIn> o;
        if (is_a)
          o.init(p.a, p.lda, p.op_a != CORAL_NO_TRANSPOSE, ti.m0, min(kTM, p.m - ti.m0), tid);
        else
          o.init(p.b, p.ldb, p.op_b == CORAL_NO_TRANSPOSE, ti.n0, min(ti.bn, p.n - ti.n0), tid);
        const long long slab = o.along_k ? kTK : kTK * (o.s1 >> 1);
        const int nb = (o.rows + 31) >> 5;
        int kb = (group ^ it0) & 1;
        o.p += kb * slab;
        for (; kb < nslabs; kb += 2, o.p += 2 * slab) {
          const int it = it0 + kb, s = it % S, left = kd - kb * kTK;
          uint8_t* st = smem + (size_t)s * kStage + (is_a ? 0 : NPC * kAPieceBytes) + o.dst;
          for (int b0 = 0; b0 < nb; b0 += kInFlight) {
            uint32_t v[kInFlight][8];
#pragma unroll
            for (int u = 0; u < kInFlight; ++u)
              if (b0 + u < nb) o.load(b0 + u, left, tid, v[u]);
            // no way out from here: the lanes go on together, see next_tile
            if (b0 == 0 && it >= S && !tc::mbar_wait_or(&empty_bar[s], ((it / S) - 1) & 1, limit_ns, &abort_flag))
              give_up();
#pragma unroll
            for (int u = 0; u < kInFlight; ++u)
              if (b0 + u < nb) store_block<TIn, NPC>(o.along_k, st + (b0 + u) * 2048, piece_bytes, v[u]);
          }
          tc::fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&full_bar[s]);
        }
        it0 += nslabs;
      }
      __syncwarp();
      if (lane == 0) release_tile(j);
    }
  } else if (warp == kMmaWarp) {
    if (lane == 0) {
      // ---- MMA issuer ----
      int it = 0, gc = 0;
      bool stop = false;
      const TileInfo* tp;
      for (int j = 0; !stop && (tp = next_tile(j, false)); ++j) {
        const int nslabs = tp->nslabs;
        const uint32_t idesc = tc::idesc_bf16_f32(kTM, tp->bn);
        release_tile(j);
        const int chunks = (nslabs + kChunkSlabs - 1) / kChunkSlabs;
        for (int c = 0; c < chunks && !stop; ++c, ++gc) {
          const int b = gc & 1;
          if (gc >= 2 && !tc::mbar_wait(&acc_empty[b], ((gc >> 1) - 1) & 1, limit_ns)) {
            give_up();
            stop = true;
            break;
          }
          tc::tc_fence_after();
          const uint32_t acc = tmem + b * kMaxBN;
          const int kb0 = c * kChunkSlabs, kb1 = min(nslabs, kb0 + kChunkSlabs);
          for (int kb = kb0; kb < kb1; ++kb, ++it) {
            const int s = it % S;
            if (!tc::mbar_wait(&full_bar[s], (it / S) & 1, limit_ns)) {
              give_up();
              stop = true;
              break;
            }
            tc::tc_fence_after();
            const uint32_t sa = tc::smem_u32(smem + (size_t)s * kStage);
            const uint32_t sb = sa + NPC * kAPieceBytes;
#pragma unroll
            for (int kk = 0; kk < kTK / 16; ++kk) {
#pragma unroll
              for (int q = 0; q < Cfg::kProducts; ++q) {
                const uint64_t ad = tc::desc_k_sw64(sa + Cfg::a(q) * kAPieceBytes + kk * 32);
                const uint64_t bd = tc::desc_k_sw64(sb + Cfg::b(q) * kBPieceBytes + kk * 32);
                const uint32_t accum = ((kb - kb0) | kk | q) != 0;
                switch (Cfg::collect(q)) {
                  case tc::kCollectFill: tc::mma_f16_ca<tc::kCollectFill>(acc, ad, bd, idesc, accum); break;
                  case tc::kCollectLastUse:
                    tc::mma_f16_ca<tc::kCollectLastUse>(acc, ad, bd, idesc, accum);
                    break;
                  default: tc::mma_f16(acc, ad, bd, idesc, accum); break;
                }
              }
            }
            tc::mma_commit(&empty_bar[s]);
          }
          if (!stop) tc::mma_commit(&acc_full[b]);
        }
      }
      // every MMA issued by this thread completes before TMEM is released
      tc::mma_commit(&drain_bar);
      tc::mbar_wait(&drain_bar, 0, tc::kDrainNs);
    }
  } else {
    // ---- epilogue ----
    const int quad = warp & 3, half = (warp - kEpiWarp0) >> 2;  // rows; every other group of 16 columns
    const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
    int gc = 0;
    const TileInfo* tp;
    for (int j = 0; (tp = next_tile(j, true)); ++j) {
      const int m0 = tp->m0, n0 = tp->n0, nslabs = tp->nslabs, m = tp->p.m;
      const int row = m0 + quad * 32 + lane;
      const int ncols = min(tp->bn, tp->p.n - n0);
      const float alpha = tp->p.alpha, beta = tp->p.beta;
      const bool beta0 = beta == 0.f, beta1 = beta == 1.f;
      const long long ldc = tp->p.ldc;
      float* const crow = tp->p.c + row + (size_t)n0 * ldc;
      __syncwarp();
      if (lane == 0) release_tile(j);
      if (nslabs == 0) {  // scale-only (sgemm_nn.rs:29-45), 16 C loads before their stores
        if (!beta1 && row < m)
          for (int g = 16 * half; g < ncols; g += 32) {
            float cv[16];
#pragma unroll
            for (int jj = 0; jj < 16; ++jj)
              cv[jj] = (!beta0 && g + jj < ncols) ? crow[(size_t)(g + jj) * ldc] : 0.f;
#pragma unroll
            for (int jj = 0; jj < 16; ++jj)
              if (g + jj < ncols) crow[(size_t)(g + jj) * ldc] = beta0 ? 0.f : beta * cv[jj];
          }
        continue;
      }
      const int chunks = (nslabs + kChunkSlabs - 1) / kChunkSlabs;
      for (int c = 0; c < chunks; ++c, ++gc) {
        const int b = gc & 1;
        const bool in = row < m, read_c = (c > 0 || !beta0) && in;
        const float keep = c > 0 ? 1.f : beta;  // factor of what C holds
        float cv[16];
        float* q = crow + (size_t)(16 * half) * ldc;
        auto load_c = [&](const float* from, int cols) {  // up to 16 columns
          if (!read_c) return;
          if (cols >= 16) {
#pragma unroll
            for (int jj = 0; jj < 16; ++jj, from += ldc) cv[jj] = *from;
          } else {
#pragma unroll
            for (int jj = 0; jj < 16; ++jj, from += ldc)
              if (jj < cols) cv[jj] = *from;
          }
        };
        // the first 16 columns of C on their way while the products finish
        load_c(q, ncols - 16 * half);
        const bool ok = tc::mbar_wait_or(&acc_full[b], (gc >> 1) & 1, limit_ns, &abort_flag);
        if (!ok) give_up();
        tc::tc_fence_after();
        for (int col0 = 16 * half; col0 < ncols; col0 += 32) {
          uint32_t r[16];
          tc::tmem_ld16(tmem + b * kMaxBN + col0 + lane_base, r);
          tc::tmem_wait_ld();
          float out[16];
#pragma unroll
          for (int jj = 0; jj < 16; ++jj) {
            const float v = alpha * __uint_as_float(r[jj]);
            out[jj] = keep == 1.f ? cv[jj] + v : keep == 0.f ? v : keep * cv[jj] + v;
          }
          // the next group's C before this group's stores
          load_c(q + 32 * ldc, ncols - col0 - 32);
          if (in && ok) {
            float* to = q;
            if (ncols - col0 >= 16) {
#pragma unroll
              for (int jj = 0; jj < 16; ++jj, to += ldc) *to = out[jj];
            } else {
#pragma unroll
              for (int jj = 0; jj < 16; ++jj, to += ldc)
                if (col0 + jj < ncols) *to = out[jj];
            }
          }
          q += 32 * ldc;
        }
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&acc_empty[b]);
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) tc::tmem_dealloc(tmem, 2 * kMaxBN);
}

template <typename TIn, int NPC>
coral_status_t launch_grouped_tc(Handle* h, int count, const coral_sgemm_problem_t* probs, const int* order,
                                 const int* bn_pos, const long long* prefix, unsigned long long* counter) {
  const size_t smem = tc_smem_bytes<NPC>();
  static uint64_t attr_devices = 0;  // bit d: attribute set on device d
  const uint64_t bit = h->device < 64 ? (1ull << h->device) : 0;
  if (!(attr_devices & bit) || !bit) {
    CORAL_CUDA(h, cudaFuncSetAttribute(k_gemm_grouped_tc<TIn, NPC>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_devices |= bit;
  }
  const uint64_t limit_ns = h->wait_limit * 32ull;
  timed_begin(h);
  k_gemm_grouped_tc<TIn, NPC><<<h->sm_count, kTcThreads, smem, h->stream>>>(
      probs, count, order, bn_pos, prefix, counter, &h->words->status, limit_ns);
  coral_status_t s = launch_status(h);
  timed_end(h);
  return s;
}

}  // namespace

// Enqueues the plan and the tensor-core grouped GEMM: bf16 inputs (npc 1) or
// fp32 inputs as split-BF16x3 (npc 2).
coral_status_t enqueue_grouped_tc(Handle* h, bool bf16_inputs, size_t count,
                                  const coral_sgemm_problem_t* probs) {
  auto up = [](size_t b) { return (b + 255) & ~size_t(255); };
  const size_t o_order = 0, o_bn = up(count * 4), o_prefix = o_bn + up(count * 4);
  const size_t o_ctr = o_prefix + up((count + 1) * 8);
  char* sc = static_cast<char*>(scratch(h, o_ctr + 256));
  if (!sc) return CORAL_ERR_ALLOC;
  int* order = reinterpret_cast<int*>(sc + o_order);
  int* bn_pos = reinterpret_cast<int*>(sc + o_bn);
  long long* prefix = reinterpret_cast<long long*>(sc + o_prefix);
  unsigned long long* counter = reinterpret_cast<unsigned long long*>(sc + o_ctr);
  CORAL_CUDA(h, cudaMemsetAsync(counter, 0, sizeof(unsigned long long), h->stream));
  k_grouped_plan<<<1, 1024, 0, h->stream>>>(probs, (int)count, h->grouped_policy, order, bn_pos, prefix);
  coral_status_t s = launch_status(h);
  if (s != CORAL_OK) return s;
  return bf16_inputs
             ? launch_grouped_tc<__nv_bfloat16, 1>(h, (int)count, probs, order, bn_pos, prefix, counter)
             : launch_grouped_tc<float, 2>(h, (int)count, probs, order, bn_pos, prefix, counter);
}

}  // namespace coral
