// GEMM on CTA pairs: tcgen05.mma.cta_group::2, one 256 x 256 tile of D per pair; INT8 (kind::i8),
// f32 as 3xTF32 (kind::tf32 on hi/lo planes) and f32 as three f16 products (kind::f16 on hi/lo planes
// of block-scaled values: the same 22 bits per operand at twice the rate and half the bytes).
//
// Why a pair: with one CTA per 128 x 256 tile every SM has to land 48 KB of operands in
// shared memory per 512 tensor-core cycles while the MMA reads 96 B/clk from the same
// shared memory, and the tensor pipe idles waiting for data.  A pair shares the B operand:
// each CTA loads its own 128 rows of A and HALF of the 256 B rows (32 KB per stage), the MMA
// of the leader CTA reads both halves, and each CTA ends up with its own 128 x 256 slice of
// D in its tensor memory.
//
// Roles per CTA (320 threads) as in gemm_tc.cuh: warp 0 TMA producer, warp 1 MMA issuer
// (only in the leader CTA) and tensor-memory owner, warps 2..9 epilogue.  Cross-CTA
// signalling:
//   full[s]    lives in the leader; both CTAs' TMA loads complete their bytes on it
//   empty[s]   one per CTA; the leader's tcgen05.commit multicasts the arrive to both (f16 planes: lo[s] too,
//              for the lo planes alone)
//   tfull[a]   one per CTA; commit multicast
//   tempty[a]  lives in the leader; the 16 epilogue warps of the pair arrive on it
// No TMA multicast is used: every CTA issues plain loads into its own shared memory.
// All waits are bounded (see gemm_tc.cuh); the two cluster barriers are reached by every
// thread on every path.
#pragma once
#include "gemm_tc.cuh"

namespace gemm2 {

using gemm::BM;
using gemm::NUM_THREADS;
using gemm::ROW_BYTES;
using gemm::WAIT_LIMIT_NS;

constexpr int BN2 = 256;      // columns of D per pair tile
#ifndef VTLB_PAIR_STAGES
#define VTLB_PAIR_STAGES 6  // shared-memory ring depth of the INT8 pair kernel (tuning knob)
#endif

template <int KIND>
struct Cfg {
  static constexpr int NOP = gemm::Traits<KIND>::NOP;                 // operand planes per side
  static constexpr int STAGES = KIND == gemm::KIND_I8 ? VTLB_PAIR_STAGES : 3;
  static constexpr uint32_t A_TILE = BM * ROW_BYTES;                  // this CTA's 128 rows of A
  static constexpr uint32_t B_HALF = (BN2 / 2) * ROW_BYTES;           // this CTA's 128 rows of B
  static constexpr uint32_t STAGE = NOP * (A_TILE + B_HALF);          // 32 KB (INT8) / 64 KB (TF32x3)
  static constexpr uint32_t TILES = STAGES * STAGE;
  static constexpr uint32_t BARS_OFF = TILES + gemm::STAGING;         // epilogue staging tiles in between
  // full, empty, two each of tfull and tempty, and for f16 planes: lo planes empty
  static constexpr int NUM_BARS = 2 * STAGES + 4 + (KIND == gemm::KIND_F16X3 ? STAGES : 0);
  static constexpr uint32_t SMEM_TOTAL = BARS_OFF + 8 * NUM_BARS + 16 + 1024;
  // TF32x3 closes its accumulator every CHUNK_KB stages (the f32 accumulate of tcgen05 truncates;
  // see gemm_tc.cuh).  With 256 columns per accumulator and two buffers there is no room in tensor
  // memory for a separate accumulator of the small cross terms: here they share the main one, which
  // costs three truncations per K step instead of one, still two orders inside the error bound.
  // The f16 planes close it every 2 stages = 128 elements (a stage holds twice the K): sums of 4096 uniform products are
  // off by 4.7e-7 of 64-bit ones, of normal ones by 2.3e-7, where 3xTF32 leaves 1.08e-6 and 9.2e-7.  (6.8e-7 and 4.9e-7
  // with the cross terms among the hi.hi ones; so ordered, 4 stages left 1.58e-6 of uniform ones.)
  static constexpr int CHUNK_KB = KIND == gemm::KIND_I8 ? 0 : KIND == gemm::KIND_F16X3 ? 2 : 4;
  static constexpr int SCALE_KB = gemm::kHalfBlock * 2 / (int)ROW_BYTES;  // stages that share a scale (f16 planes)
  static_assert(KIND != gemm::KIND_F16X3 || SCALE_KB % CHUNK_KB == 0, "an accumulator has one scale");
};
constexpr uint32_t TMEM_COLS = 2 * BN2;

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of `addr` (a shared::cta address of this CTA) in CTA `rank`
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA load into this CTA's shared memory whose byte count completes on an mbarrier that may
// live in the peer CTA (cluster address).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* tmap, int x, int y,
                                                 uint32_t bar_cluster_addr) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 "
      "[%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
      "l"(tmap), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* tmap, int x, int y, int z,
                                                 uint32_t bar_cluster_addr) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 "
      "[%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
      "l"(tmap), "r"(bar_cluster_addr), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc2(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish2() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// arrive on the mbarrier at this shared-memory offset in both CTAs of the pair once every
// tcgen05 operation issued so far has completed
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  const uint16_t mask = 3;
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"(mask)
      : "memory");
}
__device__ __forceinline__ void umma_tf32_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                               uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D = D / 2^kHalfShift + A.B
__device__ __forceinline__ void umma_f16_pair_shift(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.eq.b32 p, 0, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p, %4;\n"
      "}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "n"(gemm::kHalfShift)
      : "memory");
}
__device__ __forceinline__ void umma_i8_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Scratch of the K-split tiles (see the kernel): flags first, then the parked accumulators.
constexpr int KSPLIT_MAX_TILES = 64;  // at most half of the CTA pairs of a device
constexpr int KSPLIT_FLAG_WORDS = KSPLIT_MAX_TILES * 2 * gemm::EPI_WARPS;  // [tile][rank][warp]
constexpr size_t KSPLIT_BYTES = (size_t)KSPLIT_FLAG_WORDS * 4 + (size_t)KSPLIT_MAX_TILES * 2 * BM * BN2 * 4;
static_assert(KSPLIT_MAX_TILES == vtlb_ctx::kKsplitTiles && KSPLIT_FLAG_WORDS * 4 == vtlb_ctx::kKsplitFlagBytes &&
                  KSPLIT_BYTES == vtlb_ctx::kKsplitBytes,
              "the context allocates the K-split buffer with these sizes");

__device__ __forceinline__ void flag_release(uint32_t* flag, uint32_t value) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(flag), "r"(value) : "memory");
}
// Spins until *flag == value; gives up after limit_ns or when the CTA's abort flag is raised
// (and raises it), like the mbarrier waits.
__device__ __forceinline__ bool flag_wait_bounded(const uint32_t* flag, uint32_t value,
                                                  volatile uint32_t* abort_flag, uint64_t limit_ns) {
  uint64_t t0 = 0;
  for (uint32_t spins = 0;; ++spins) {
    uint32_t seen;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(flag) : "memory");
    if (seen == value) return true;
    if ((spins & 63u) == 63u) {
      if (*abort_flag) return false;
      uint64_t now;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
      if (t0 == 0) t0 = now;
      else if (now - t0 > limit_ns) {
        *abort_flag = 1;
        return false;
      }
      __nanosleep(64);
    }
  }
}

// Bits of the rows (0 .. 31, bit 8 * (row / 4) + row % 4) of a group of 32 that have elements listed in a block.
__device__ __forceinline__ uint64_t rest_flags(const gemm::HalfSide& s, int blk, int row) {
  return __ldg(reinterpret_cast<const unsigned long long*>(s.flags + ((size_t)blk * s.rp + row) / 4)) &
         0x0f0f0f0f0f0f0f0full;
}
__device__ __forceinline__ float half_kept(const gemm::HalfSide& s, int ld, int row, int k, float scale) {
  const size_t at = (size_t)row * ld + k;
  return __fmaf_rn(__half2float(__ldg(s.lo + at)), 1.0f / (1 << gemm::kHalfShift), __half2float(__ldg(s.hi + at))) * scale;
}
// The products of the elements that the f16 planes do not hold (gemm::HalfSide::rest): to this warp's 32 rows x four
// chunks of 32 columns (64 apart, the first at col0), rest(a) * b with all of b, and what is held of a * rest(b).  The
// sums start with them, so the loads run beside the tile's first MMAs.  Each costs a round of loads and an addition,
// predicated, per value.  A fixed order, so results repeat.
__device__ __forceinline__ void add_rests(float (&sum)[BN2 / 2], const gemm::HalfOperands& o, int row0, int col0,
                                          int lane, int M, int N, int K) {
  constexpr int NC = BN2 / 64, G = gemm::kHalfGroup;
  const int blocks = (K + gemm::kHalfBlock - 1) / gemm::kHalfBlock;
  const int my_bit = lane / 4 * 8 + lane % 4;
  for (int b0 = 0; b0 < blocks; b0 += 32) {  // a lane looks one block over
    const int mine = b0 + lane < blocks ? b0 + lane : b0;
    uint64_t any = rest_flags(o.a, mine, row0);
#pragma unroll
    for (int cc = 0; cc < NC; ++cc) any |= rest_flags(o.b, mine, col0 + cc * 64);
    uint32_t todo = __ballot_sync(0xffffffffu, b0 + lane < blocks && any != 0);
    while (todo) {
      const int blk = b0 + __ffs(todo) - 1;
      todo &= todo - 1;
      // what lies behind the last row or column was never written
      const int row = row0 + lane;
      const uint32_t rows = __ballot_sync(0xffffffffu, row < M && (rest_flags(o.a, blk, row0) >> my_bit & 1));
      if (rows) {
        const int2* list = o.a.rest + ((size_t)blk * o.a.rp + row) * gemm::kHalfRest;
#pragma unroll 1
        for (int e = 0; e < gemm::kHalfRest; ++e) {  // a lane its own row's
          const int2 it = rows >> lane & 1u ? __ldg(list + e) : make_int2(-1, 0);
          uint32_t have = __ballot_sync(0xffffffffu, it.x >= 0);
          if (!have) break;
#pragma unroll 1
          for (; have; have &= have - 1) {
            const int r = __ffs(have) - 1, k = __shfl_sync(0xffffffffu, it.x, r);
            const float rest = __int_as_float(__shfl_sync(0xffffffffu, it.y, r));
            float b[NC];
            bool more = false;
#pragma unroll
            for (int cc = 0; cc < NC; ++cc) {  // the loads of all four chunks together
              const int n = col0 + cc * 64 + lane, at = n < N ? n : N - 1;
              b[cc] = half_kept(o.b, o.ld, at, k, __ldg(o.b.scale + ((size_t)blk * o.b.rp + at) / G));
              more = more || (n < N && (rest_flags(o.b, blk, col0 + cc * 64) >> my_bit & 1));
            }
            if (__any_sync(0xffffffffu, more)) {  // the column may have a rest at the same k
#pragma unroll
              for (int cc = 0; cc < NC; ++cc) {
                const int n = col0 + cc * 64 + lane;
                if (n >= N || !(rest_flags(o.b, blk, col0 + cc * 64) >> my_bit & 1)) continue;
                const int2* lb = o.b.rest + ((size_t)blk * o.b.rp + n) * gemm::kHalfRest;
                for (int i = 0; i < gemm::kHalfRest; ++i) {
                  const int2 jt = __ldg(lb + i);
                  if (jt.x < 0) break;
                  if (jt.x == k) b[cc] += __int_as_float(jt.y);
                }
              }
            }
#pragma unroll
            for (int cc = 0; cc < NC; ++cc) {
              const float p = b[cc] * rest;
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                const float t = __shfl_sync(0xffffffffu, p, j);
                if (lane == r) sum[cc * 32 + j] += t;
              }
            }
          }
        }
      }
#pragma unroll
      for (int cc = 0; cc < NC; ++cc) {
        const int n = col0 + cc * 64 + lane;
        const uint32_t cols =
            __ballot_sync(0xffffffffu, n < N && (rest_flags(o.b, blk, col0 + cc * 64) >> my_bit & 1));
        if (!cols) continue;
        const int2* list = o.b.rest + ((size_t)blk * o.b.rp + n) * gemm::kHalfRest;
#pragma unroll 1
        for (int e = 0; e < gemm::kHalfRest; ++e) {  // a lane its own column's
          const int2 it = cols >> lane & 1u ? __ldg(list + e) : make_int2(-1, 0);
          uint32_t have = __ballot_sync(0xffffffffu, it.x >= 0);
          if (!have) break;
#pragma unroll 1
          for (; have; have &= have - 1) {
            const int c = __ffs(have) - 1, k = __shfl_sync(0xffffffffu, it.x, c);
            float p = __int_as_float(__shfl_sync(0xffffffffu, it.y, c));
            p *= row < M ? half_kept(o.a, o.ld, row, k, __ldg(o.a.scale + (size_t)blk * o.a.rp + row)) : 0.0f;
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (c == j) sum[cc * 32 + j] += p;
          }
        }
      }
    }
  }
}

template <int KIND, class Epi>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ gemm::TmapSet tm, const Epi epi, int M, int N, int K,
                 int group_m, int a_chunk_k, int split_tiles, uint32_t* ksplit_buf, uint32_t ksplit_epoch,
                 uint32_t* status, const gemm::HalfOperands ho) {
  using T = gemm::Traits<KIND>;
  using C = Cfg<KIND>;
  constexpr int NOP = C::NOP, STAGES = C::STAGES;
  constexpr int BK = ROW_BYTES / T::ELEM;  // elements of K per stage
  constexpr int XSTEP = KIND == gemm::KIND_F16X3 ? (int)ROW_BYTES : BK;  // ... in tensor-map coordinates (f16: bytes)
  constexpr int KSTEPS = ROW_BYTES / 32;
  constexpr uint32_t IDESC = ptx::umma_idesc(T::CFMT, T::ABFMT, 2 * BM, BN2);

  // one of the two kernels launched for a product on f16 planes leaves at once; both CTAs of a pair read the same
  // (those launches do not start early, so the word may be read before the wait below)
  if (KIND != gemm::KIND_I8 && ho.unfit != nullptr && (*ho.unfit == ho.epoch) != (KIND == gemm::KIND_TF32X3)) return;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const uint32_t bars = base + C::BARS_OFF;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
  auto tfull_bar = [&](int a) { return bars + 8u * (2 * STAGES + a); };
  auto tempty_bar = [&](int a) { return bars + 8u * (2 * STAGES + 2 + a); };
  auto lo_empty_bar = [&](int s) { return bars + 8u * (2 * STAGES + 4 + s); };  // f16 planes only
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_raw + (bars - raw) + 8u * C::NUM_BARS);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();  // 0 = leader
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const int tiles_m = (M + 2 * BM - 1) / (2 * BM), tiles_n = (N + BN2 - 1) / BN2;
  const int num_tiles = tiles_m * tiles_n;
  const int num_kb = (K + BK - 1) / BK;
  const int chunk_kb = C::CHUNK_KB ? C::CHUNK_KB : num_kb;
  // Work units.  When the tiles do not fill the last wave of CTA pairs, `split_tiles` tiles (the
  // first ones) are cut along K into two units each, which evens out the work per pair (4096^3:
  // 256 tiles on 74 pairs = 3.46 waves; with 34 tiles cut, 68 pairs run 3.5 tiles' worth and 6
  // pairs run 3).  Pair 2s runs the first K half of cut tile s as its FIRST unit, parks the raw
  // int32 accumulators in `ksplit_buf` and publishes one flag per epilogue warp; pair 2s+1 runs
  // the second half as its SECOND unit (after a full tile), adds the parked values to its own and
  // does the epilogue proper.  By then the parked half has long landed, and the slower epilogue of
  // that one unit hides behind the MMAs of the next.  Integer addition keeps the result
  // bit-identical.  INT8 only.  The first-half unit never waits for anybody and has the lower CTA
  // numbers, which are dispatched first: the second-half unit's (bounded) wait cannot deadlock.
  //
  // Unit `it` of this pair: false when the pair has run out of work.  Full tiles fill every
  // position that is not a half unit, in order of (it, pair).
  auto decode_unit = [&](int it, int& tmi, int& tni, int& k_half, int& slot) -> bool {
    const int S = split_tiles, P = num_pairs, p = pair;
    const bool cut = p < 2 * S;
    k_half = -1;
    slot = 0;
    int f;  // index among the full tiles
    if (it == 0) {
      if (cut && (p & 1) == 0) {
        k_half = 0;
        slot = p >> 1;
      }
      f = cut ? (p >> 1) : p - S;
    } else if (it == 1) {
      if (cut && (p & 1) == 1) {
        k_half = 1;
        slot = p >> 1;
      }
      f = (P - S) + (cut ? (p >> 1) : p - S);
    } else {
      f = 2 * (P - S) + (it - 2) * P + p;
    }
    int tile = slot;
    if (k_half < 0) {
      if (f >= num_tiles - S) return false;
      tile = S + f;
    }
    gemm::decode_tile(tile, tiles_m, tiles_n, group_m, tmi, tni);
    return true;
  };
  auto k_range = [&](int k_half, int& kb_begin, int& kb_end) {
    kb_begin = k_half == 1 ? num_kb / 2 : 0;
    kb_end = k_half == 0 ? num_kb / 2 : num_kb;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      ptx::mbar_init(full_bar(s), 1);   // the leader's expect_tx arrive; bytes from both CTAs
      ptx::mbar_init(empty_bar(s), 1);  // one multicast commit
      if (KIND == gemm::KIND_F16X3) ptx::mbar_init(lo_empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(tfull_bar(a), 1);
      ptx::mbar_init(tempty_bar(a), 2 * gemm::EPI_WARPS);  // the epilogue warps of both CTAs
    }
    *abort_flag = 0;
    ptx::fence_barrier_init();
    ptx::fence_proxy_async();
    for (int i = 0; i < NOP; ++i) {
      ptx::prefetch_tmap(&tm.a[i]);
      ptx::prefetch_tmap(&tm.b[i]);
    }
  }
  if (warp == 1) {
    tmem_alloc2(ptx::smem_u32(tmem_slot), TMEM_COLS);
    tmem_relinquish2();
  }
  ptx::tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // barriers of both CTAs are initialised before anyone signals them
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // a single wave is launched early: the set-up above overlapped the kernel in front, which is done from here on
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    if (lane == 0) {
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (int it = 0; ok; ++it) {
        int tmi, tni, kh, slot, kb_begin, kb_end;
        if (!decode_unit(it, tmi, tni, kh, slot)) break;
        k_range(kh, kb_begin, kb_end);
        const int m0 = tmi * 2 * BM + (int)rank * BM;
        const int n0 = tni * BN2 + (int)rank * (BN2 / 2);
        for (int kb = kb_begin; kb < kb_end; ++kb) {
          if (!ptx::mbar_wait_bounded(KIND == gemm::KIND_F16X3 ? lo_empty_bar(stage) : empty_bar(stage), phase ^ 1u,
                                      abort_flag, WAIT_LIMIT_NS)) {
            ok = false;
            break;
          }
          const uint32_t leader_full = mapa(full_bar(stage), 0);
          if (rank == 0) ptx::mbar_arrive_expect_tx(full_bar(stage), 2 * C::STAGE);
          const uint32_t sa = base + stage * C::STAGE;
          const uint32_t sb = sa + NOP * C::A_TILE;
          if constexpr (KIND == gemm::KIND_F16X3) {
            // the lo planes of a stage are free two thirds of a chunk before its hi planes (see the MMA warp)
            tma_load_2d_pair(sa + C::A_TILE, &tm.a[1], kb * XSTEP, m0, leader_full);
            tma_load_2d_pair(sb + C::B_HALF, &tm.b[1], kb * XSTEP, n0, leader_full);
            if (!ptx::mbar_wait_bounded(empty_bar(stage), phase ^ 1u, abort_flag, WAIT_LIMIT_NS)) {
              ok = false;
              break;
            }
            tma_load_2d_pair(sa, &tm.a[0], kb * XSTEP, m0, leader_full);
            tma_load_2d_pair(sb, &tm.b[0], kb * XSTEP, n0, leader_full);
          } else {
#pragma unroll
            for (int i = 0; i < NOP; ++i) {
              if (a_chunk_k)  // A stored as [chunk][M][a_chunk_k] (gathered column shards)
                tma_load_3d_pair(sa + i * C::A_TILE, &tm.a[i], (kb * BK) % a_chunk_k, m0, (kb * BK) / a_chunk_k,
                                 leader_full);
              else
                tma_load_2d_pair(sa + i * C::A_TILE, &tm.a[i], kb * XSTEP, m0, leader_full);
            }
#pragma unroll
            for (int i = 0; i < NOP; ++i)
              tma_load_2d_pair(sb + i * C::B_HALF, &tm.b[i], kb * XSTEP, n0, leader_full);
          }
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader only)
    if (lane == 0 && rank == 0) {
      uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
      bool ok = true;
      for (int it = 0; ok; ++it) {
        int tmi, tni, kh, slot, kb_begin, kb_end;
        if (!decode_unit(it, tmi, tni, kh, slot)) break;
        k_range(kh, kb_begin, kb_end);
        for (int kb0 = kb_begin; kb0 < kb_end && ok; kb0 += chunk_kb) {
          const int kb1 = kb0 + chunk_kb < kb_end ? kb0 + chunk_kb : kb_end;
          if (!ptx::mbar_wait_bounded(tempty_bar(acc), acc_phase ^ 1u, abort_flag, WAIT_LIMIT_NS)) {
            ok = false;
            break;
          }
          ptx::tc_fence_after();
          const uint32_t d_tmem = tmem_base + acc * BN2;
          // f16 planes: first the cross terms of the whole chunk, which are 2^12 times too large, then hi.hi, whose
          // first MMA takes the factor back.  A stage's lo planes are free after its cross terms, its hi planes after
          // hi.hi: with three stages, chunks of two and one barrier for both the loads came 1.5 to 2 % late.
          const uint32_t first_stage = stage;
          for (int kb = kb0; kb < kb1; ++kb) {
            if (!ptx::mbar_wait_bounded(full_bar(stage), phase, abort_flag, WAIT_LIMIT_NS)) {
              ok = false;
              break;
            }
            ptx::tc_fence_after();
            const uint32_t sa = base + stage * C::STAGE;
            const uint32_t sb = sa + NOP * C::A_TILE;
#pragma unroll
            for (int kk = 0; kk < KSTEPS; ++kk) {
              const uint32_t first = (kb == kb0 && kk == 0) ? 0u : 1u;
              if constexpr (KIND == gemm::KIND_I8) {
                const uint64_t da = ptx::umma_desc_k_sw128(sa) + 2u * kk;
                const uint64_t db = ptx::umma_desc_k_sw128(sb) + 2u * kk;
                umma_i8_pair(d_tmem, da, db, IDESC, first);
              } else {
                const uint64_t a_hi = ptx::umma_desc_k_sw128(sa) + 2u * kk;
                const uint64_t a_lo = ptx::umma_desc_k_sw128(sa + C::A_TILE) + 2u * kk;
                const uint64_t b_hi = ptx::umma_desc_k_sw128(sb) + 2u * kk;
                const uint64_t b_lo = ptx::umma_desc_k_sw128(sb + C::B_HALF) + 2u * kk;
                if constexpr (KIND == gemm::KIND_F16X3) {
                  umma_f16_pair(d_tmem, a_lo, b_hi, IDESC, first);
                  umma_f16_pair(d_tmem, a_hi, b_lo, IDESC, 1);
                } else {
                  umma_tf32_pair(d_tmem, a_lo, b_hi, IDESC, first);  // small terms first
                  umma_tf32_pair(d_tmem, a_hi, b_lo, IDESC, 1);
                  umma_tf32_pair(d_tmem, a_hi, b_hi, IDESC, 1);
                }
              }
            }
            umma_commit_pair(KIND == gemm::KIND_F16X3 ? lo_empty_bar(stage) : empty_bar(stage));
            if (++stage == STAGES) {
              stage = 0;
              phase ^= 1u;
            }
          }
          if constexpr (KIND == gemm::KIND_F16X3) {
            uint32_t st = first_stage;
            for (int kb = kb0; kb < kb1 && ok; ++kb) {
              const uint32_t sa = base + st * C::STAGE;
              const uint32_t sb = sa + NOP * C::A_TILE;
#pragma unroll
              for (int kk = 0; kk < KSTEPS; ++kk) {
                const uint64_t a_hi = ptx::umma_desc_k_sw128(sa) + 2u * kk;
                const uint64_t b_hi = ptx::umma_desc_k_sw128(sb) + 2u * kk;
                if (kb == kb0 && kk == 0) umma_f16_pair_shift(d_tmem, a_hi, b_hi, IDESC);
                else umma_f16_pair(d_tmem, a_hi, b_hi, IDESC, 1);
              }
              umma_commit_pair(empty_bar(st));
              if (++st == STAGES) st = 0;
            }
          }
          if (!ok) break;
          umma_commit_pair(tfull_bar(acc));
          acc ^= 1u;
          if (acc == 0) acc_phase ^= 1u;
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (both CTAs)
    const int q = warp & 3;
    const int half = (warp - 2) >> 2;  // even or odd 32-column chunks
    const uint32_t stg = base + C::TILES + (uint32_t)(warp - 2) * gemm::STAGING_PER_WARP;
    const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16);
    uint32_t acc = 0, acc_phase = 0;
    bool ok = true;
    const bool listed = KIND == gemm::KIND_F16X3 && *ho.listed == ho.epoch;
    for (int it = 0; ok; ++it) {
      int tmi, tni, kh, slot;
      if (!decode_unit(it, tmi, tni, kh, slot)) break;
      const int m0 = tmi * 2 * BM + (int)rank * BM;
      const int n0 = tni * BN2;
      const int row0 = m0 + q * 32;
      if constexpr (KIND == gemm::KIND_I8) {
        // Per-row and per-column operands of the epilogue (scales, bias) are fetched before the
        // wait for the accumulator, one column per lane, and handed round by shuffles later:
        // their latency would otherwise sit in front of every 32-column chunk.
        const typename Epi::Pre pre = epi.prefetch(row0 + lane, n0 + half * 32 + lane, M, N);
        ok = ptx::mbar_wait_bounded(tfull_bar(acc), acc_phase, abort_flag, WAIT_LIMIT_NS);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        ptx::tc_fence_after();
        // K-split tile: the unit of the first K half parks its accumulators,
        // [slot][rank][warp][chunk][value][lane], and the unit of the second half adds them to its own.
        const int wslot = (slot * 2 + (int)rank) * gemm::EPI_WARPS + (warp - 2);
        uint32_t* park = ksplit_buf + KSPLIT_FLAG_WORDS + (size_t)wslot * (BN2 / 64) * 1024;
        if (kh == 1) {  // wait for the first K half of this tile
          if (lane == 0) ok = flag_wait_bounded(ksplit_buf + wslot, ksplit_epoch, abort_flag, WAIT_LIMIT_NS);
          ok = __all_sync(0xffffffffu, __shfl_sync(0xffffffffu, (int)ok, 0) != 0);
          if (!ok) break;
        }
        float row_amax = 0.0f;
        auto do_chunk = [&](int cc, bool tma) {
          const int c = 2 * cc + half;
          uint32_t v[32];
          ptx::tmem_ld_32x32(lane_base + acc * BN2 + c * 32, v);
          ptx::tmem_wait_ld();
          uint32_t* pc = park + cc * 1024 + lane;
          if (kh == 0) {
#pragma unroll
            for (int j = 0; j < 32; ++j) __stcg(pc + j * 32, v[j]);
          } else {
            if (kh == 1) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] += __ldcg(pc + j * 32);
            }
            epi.transform_pre(pre, cc, v);
            row_amax = fmaxf(row_amax, epi.chunk_amax(n0 + c * 32, v, N));  // one atomic per warp and tile
            if (tma) gemm::stage_and_store(stg, &tm.out[0], lane, row0, n0 + c * 32, v, M, N);
            else gemm::stage_and_store_rows(stg, epi.out_words(), epi.out_pitch(), lane, row0, n0 + c * 32, v, M, N);
          }
          __syncwarp();
        };
        if (epi.tma != 0) {
#pragma unroll
          for (int cc = 0; cc < BN2 / 64; ++cc) do_chunk(cc, true);
        } else {
#pragma unroll
          for (int cc = 0; cc < BN2 / 64; ++cc) do_chunk(cc, false);
        }
        if (kh != 0) epi.commit_amax(row0 + lane, M, row_amax);
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa(tempty_bar(acc), 0));
        if (kh == 0) {  // publish: every lane's stores, then the flag
          __threadfence();
          __syncwarp();
          if (lane == 0) flag_release(ksplit_buf + wslot, ksplit_epoch);
        }
        acc ^= 1u;
        if (acc == 0) acc_phase ^= 1u;
      } else {
        float sum[BN2 / 2];  // this warp's four 32-column chunks
#pragma unroll
        for (int j = 0; j < BN2 / 2; ++j) sum[j] = 0.0f;
        if constexpr (KIND == gemm::KIND_F16X3)
          if (listed) add_rests(sum, ho, row0, n0 + half * 32, lane, M, N, K);
        // ReLU-backward mask of the tile's outputs, fetched now as one bit per value
        uint32_t mask_bits[BN2 / 64];
        if constexpr (gemm::EpiHasPlanes<Epi>::value) {
#pragma unroll
          for (int cc = 0; cc < BN2 / 64; ++cc) {
            mask_bits[cc] = epi.load_mask_bits(row0 + lane, n0 + (2 * cc + half) * 32, M, N);
            asm volatile("" ::: "memory");  // one chunk's eight loads at a time: the running sums own the registers
          }
        }
        for (int kb0 = 0; kb0 < num_kb; kb0 += chunk_kb) {
          // f16 planes: this row's factors for the warp's four chunks, fetched before the wait (the arrays are
          // padded to whole tiles: no bounds to check).  Powers of two, and so are their products: the split passes
          // left operands whose factors could leave the f32 range to the other kernel.
          float f[BN2 / 64];
          if constexpr (KIND == gemm::KIND_F16X3) {
            const int blk = kb0 / C::SCALE_KB;
            const float fa = __ldg(ho.a.scale + (size_t)blk * ho.a.rp + row0 + lane);
#pragma unroll
            for (int cc = 0; cc < BN2 / 64; ++cc)
              f[cc] = __fmul_rn(fa, __ldg(ho.b.scale + ((size_t)blk * ho.b.rp + n0) / gemm::kHalfGroup + 2 * cc + half));
          }
          ok = ptx::mbar_wait_bounded(tfull_bar(acc), acc_phase, abort_flag, WAIT_LIMIT_NS);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          ptx::tc_fence_after();
#pragma unroll
          for (int cc = 0; cc < BN2 / 32; ++cc) {  // 16 columns at a time: the running sums own the registers
            uint32_t v[16];
            ptx::tmem_ld_32x16(lane_base + acc * BN2 + (2 * (cc / 2) + half) * 32 + (cc & 1) * 16, v);
            ptx::tmem_wait_ld();
            if constexpr (KIND == gemm::KIND_F16X3) {
              // sum += acc * factor, two columns an instruction; the product is exact, only the sum rounds
              const uint64_t f2 = ptx::f2_pack(f[cc / 2], f[cc / 2]);
#pragma unroll
              for (int j = 0; j < 16; j += 2) {
                float& s0 = sum[cc * 16 + j];
                float& s1 = sum[cc * 16 + j + 1];
                const uint64_t a2 = ptx::f2_pack(__uint_as_float(v[j]), __uint_as_float(v[j + 1]));
                ptx::f2_unpack(ptx::f2_fma(a2, f2, ptx::f2_pack(s0, s1)), s0, s1);
              }
            } else {
#pragma unroll
              for (int j = 0; j < 16; ++j) sum[cc * 16 + j] = __fadd_rn(sum[cc * 16 + j], __uint_as_float(v[j]));
            }
          }
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(mapa(tempty_bar(acc), 0));
          acc ^= 1u;
          if (acc == 0) acc_phase ^= 1u;
        }
        if (!ok) break;
#pragma unroll
        for (int cc = 0; cc < BN2 / 64; ++cc) {
          uint32_t v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(sum[cc * 32 + j]);
          if constexpr (gemm::EpiHasPlanes<Epi>::value) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (mask_bits[cc] >> j & 1u) v[j] = 0u;
          }
          gemm::epilogue_chunk(epi, tm, stg, lane, row0, n0 + (2 * cc + half) * 32, v, M, N, 0, true);
          __syncwarp();
        }
      }
    }
  }

  // ------------------------------------------------------------ teardown
  if (warp >= 2 && lane == 0) ptx::bulk_wait_read_all();  // staged TMA stores have left shared memory
  ptx::tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0) atomicOr(status, VTLB_ST_GEMM_TIMEOUT);
    for (int i = 0; i < 100; ++i) __nanosleep(1000);
  }
  cluster_sync_all();  // the peer may still signal this CTA's barriers until it gets here
  ptx::tc_fence_after();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc2(tmem_base, TMEM_COLS);
  }
}

// True when the problem has enough 256 x 256 tiles for the CTA pairs to pay off.
inline bool pair_worthwhile(vtlb_ctx* ctx, int M, int N) {
  const int tiles = ((M + 255) / 256) * ((N + 255) / 256);
  return M >= 512 && N >= 256 && tiles >= ctx->sm_count / 4;
}

template <int KIND, class Epi>
int launch_pair(vtlb_ctx* ctx, const gemm::TmapSet& tm, const Epi& epi, int M, int N, int K,
                int a_chunk_k = 0, bool k_split = false, const gemm::HalfOperands& ho = gemm::HalfOperands()) {
  using C = Cfg<KIND>;
  static_assert(C::SMEM_TOTAL <= 232448, "shared memory budget");
  auto kern = gemm_pair_kernel<KIND, Epi>;
  static std::atomic<uint64_t> configured{0};
  if (!(configured.load(std::memory_order_relaxed) >> (ctx->device & 63) & 1)) {
    VTLB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM_TOTAL));
    configured.fetch_or(1ull << (ctx->device & 63), std::memory_order_relaxed);
  }
  const int tiles = ((M + 2 * BM - 1) / (2 * BM)) * ((N + BN2 - 1) / BN2);
  int pairs = ctx->sm_count / 2;
  if (tiles < pairs) pairs = tiles;
  // A product on f16 planes is two launches, of which one does the work: they are timed as one.
  const bool timed = ctx->prof_on && ctx->prof_ev && ctx->prof_n < vtlb_ctx::kProfSlots;
  const bool opens = KIND != gemm::KIND_TF32X3 || !ho.unfit, closes = KIND != gemm::KIND_F16X3;
  if (timed && opens) cudaEventRecord(ctx->prof_ev[2 * ctx->prof_n], ctx->stream);
  const int group_m = gemm::pick_group_m((M + 2 * BM - 1) / (2 * BM),
                                         (size_t)2 * BM * K * gemm::Traits<KIND>::ELEM * C::NOP);
  // When the final wave would fill at most half of the pairs, cut that many tiles into two half-K
  // units each (INT8 only: integer partial sums add up exactly); they all fit in the first wave.
  int split_tiles = 0;
  if (KIND == gemm::KIND_I8 && k_split) {
    const int rem = tiles % pairs;
    const int num_kb = (K + 127) / 128;
    if (tiles > pairs && rem > 0 && 2 * rem <= pairs && rem <= KSPLIT_MAX_TILES && num_kb >= 8) split_tiles = rem;
  }
  if (split_tiles && ++ctx->ksplit_epoch == 0) ctx->ksplit_epoch = 1;  // flags hold the epoch of their launch
  // One wave of tiles starts early behind the kernel in front, as a rule the one that quantises or splits its rows
  // (999 x 3001 x 2047 with its quantisation: 24.7 -> 19.8 us, a part of it from the quantisation); more gain nothing (4096^3: neutral to 1.5 % slower).
  if (tiles <= pairs && KIND == gemm::KIND_I8)
    VTLB_CUDA(ctx, vtlb_launch_early(kern, dim3(2 * pairs), dim3(NUM_THREADS), C::SMEM_TOTAL, ctx->stream, tm, epi, M, N, K,
                                     group_m, a_chunk_k, split_tiles, (uint32_t*)ctx->ksplit_buf, ctx->ksplit_epoch,
                                     ctx->d_status, ho));
  else
    kern<<<2 * pairs, NUM_THREADS, C::SMEM_TOTAL, ctx->stream>>>(tm, epi, M, N, K, group_m, a_chunk_k, split_tiles,
                                                                 (uint32_t*)ctx->ksplit_buf, ctx->ksplit_epoch,
                                                                 ctx->d_status, ho);
  if (timed && closes) {
    cudaEventRecord(ctx->prof_ev[2 * ctx->prof_n + 1], ctx->stream);
    ctx->prof_n++;
    ctx->prof_flops += 2.0 * M * N * K;
  }
  VTLB_LAUNCHED(ctx);
  return VTLB_OK;
}

}  // namespace gemm2
