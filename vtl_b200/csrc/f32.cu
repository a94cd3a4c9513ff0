// f32 dense contraction: la.matmul / Linear forward and backward of the
// reference (la/la.v:38-55, nn/layers/linear_forward_f32.v:16-18,
// nn/gates/layers/linear.v:69-79) on tcgen05 tensor cores.
//
// The reference multiplies in f64 and rounds once.  Here every f32 operand x is
// split into hi and lo by a memory-bound pass that also lays the operand out
// K-major (transposing when the caller's layout is the other way round), and the
// GEMM issues three MMAs per K step (lo.hi + hi.lo + hi.hi).  hi and lo are TF32
// numbers, or, where the product fills 256 x 256 tiles on CTA pairs, f16 numbers
// of block-scaled values (struct HalfPlanes), at twice the tensor rate.  The
// dropped lo.lo term and the rounding of lo are ~2^-22 relative per product, well
// inside the 1e-5*sqrt(K)*max|A|*max|B| bound.  Small products run on CUDA cores
// (small_product).
#include "f32_common.cuh"

namespace {

using f32::split1;

// src [R, C] row-major (C % 4 == 0, 16-byte aligned) -> hi/lo [R, C].  12 bytes/element.
__device__ __forceinline__ void split_rows_vec(const float4* __restrict__ src, float4* __restrict__ hi,
                                               float4* __restrict__ lo, size_t n4) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n4;
       i += (size_t)gridDim.x * blockDim.x) {
    float4 x = src[i], h, l;
    split1(x.x, h.x, l.x);
    split1(x.y, h.y, l.y);
    split1(x.z, h.z, l.z);
    split1(x.w, h.w, l.w);
    hi[i] = h;
    lo[i] = l;
  }
}
// General case: src [R, C] -> hi/lo [R, ldo], ldo >= C.
__device__ __forceinline__ void split_rows(const float* __restrict__ src, int R, int C, int ldo, float* __restrict__ hi,
                                           float* __restrict__ lo) {
  const size_t n = (size_t)R * C;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const size_t r = i / C, c = i - r * C;
    float h, l;
    split1(src[i], h, l);
    hi[r * ldo + c] = h;
    lo[r * ldo + c] = l;
  }
}
// src [R, C] row-major -> hi/lo [C, ldo] (the transpose), ldo >= R.  32x32 tiles
// through shared memory so that both the reads and the writes are coalesced.
__device__ __forceinline__ void split_transpose(const float* __restrict__ src, int R, int C, int ldo,
                                                float* __restrict__ hi, float* __restrict__ lo, float (&tile)[32][33]) {
  const int tiles_c = (C + 31) / 32, tiles_r = (R + 31) / 32;
  const long long ntiles = (long long)tiles_c * tiles_r;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
  for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int r0 = (int)(t / tiles_c) * 32, c0 = (int)(t % tiles_c) * 32;
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
      const int r = r0 + ty + j, c = c0 + tx;
      tile[ty + j][tx] = (r < R && c < C) ? src[(size_t)r * C + c] : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
      const int c = c0 + ty + j, r = r0 + tx;
      if (c < C && r < R) {
        float h, l;
        split1(tile[tx][ty + j], h, l);
        hi[(size_t)c * ldo + r] = h;
        lo[(size_t)c * ldo + r] = l;
      }
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) split_rows_vec_kernel(const float4* __restrict__ src, float4* __restrict__ hi,
                                                             float4* __restrict__ lo, size_t n4) {
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched early (vtlb_launch_early): the kernel in front is done
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  split_rows_vec(src, hi, lo, n4);
}
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ src, int R, int C, int ldo,
                                                         float* __restrict__ hi, float* __restrict__ lo) {
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched early (vtlb_launch_early): the kernel in front is done
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  split_rows(src, R, C, ldo, hi, lo);
}
__global__ void __launch_bounds__(256) split_transpose_kernel(const float* __restrict__ src, int R, int C, int ldo,
                                                              float* __restrict__ hi, float* __restrict__ lo) {
  __shared__ float tile[32][33];
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched early (vtlb_launch_early): the kernel in front is done
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  split_transpose(src, R, C, ldo, hi, lo, tile);
}

// The multiplier 2^e that brings a block's largest magnitude into [2^14, 2^15), and 2^-e.  e is kept where both
// are normal numbers; a block of zeros (or of NaNs) gets 1.
__device__ __forceinline__ void block_scale(float amax, float& mul, float& inv) {
  const int ex = (int)(__float_as_uint(amax) >> 23);  // biased exponent; 255 for an infinity
  const int e = amax > 0.0f ? min(126, 14 + 127 - ex) : 0;
  mul = __uint_as_float((uint32_t)(127 + e) << 23);
  inv = __uint_as_float((uint32_t)(127 - e) << 23);
}
__device__ __forceinline__ float warp_amax(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// Largest of the eight warps' values; everybody gets it.
__device__ __forceinline__ float block_amax(float v, float (&part)[8]) {
  v = warp_amax(v);
  __syncthreads();  // the previous use of part is over
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  v = part[0];
#pragma unroll
  for (int w = 1; w < 8; ++w) v = fmaxf(v, part[w]);
  return v;
}
// Where a split pass puts the planes of an operand and what belongs to them (gemm::HalfSide), and how it says that f16
// cannot hold the operand: elements listed so far and how many may be, the word and the product's epoch.
struct HalfOut {
  __half *hi, *lo;
  float* scale;
  uint8_t* flags;
  int2* rest;
  int ld, rp;
  uint32_t *count, *unfit, *listed;
  uint32_t limit, epoch;
};
// True in every thread once the product is known to be unfit: nothing is left to do then.
__device__ __forceinline__ bool known_unfit(const HalfOut& o) {
  return __syncthreads_or(threadIdx.x == 0 && *(volatile const uint32_t*)o.unfit == o.epoch);
}
// One scale of a block: so extreme that the product of two such would leave the f32 range (an infinity in the block
// among them)?
__device__ __forceinline__ void note_scale(float mul, const HalfOut& o) {
  if (mul > 0x1p74f || mul < 0x1p-63f) *o.unfit = o.epoch;
}
constexpr float kHalfUp = (float)(1 << gemm::kHalfShift), kHalfDown = 1.0f / kHalfUp;
// x in two halves of the scaled value; true if they do not hold it to 22 bits.  hi + lo / 2^12 is exact in f32 (a
// multiple of the scaled value's last bit and no longer than it), and so is what is left of x.
__device__ __forceinline__ float half_rest(float x, float inv, __half hi, __half lo) {
  return __fmaf_rn(-__fmaf_rn(__half2float(lo), kHalfDown, __half2float(hi)), inv, x);
}
__device__ __forceinline__ bool split_half(float x, float mul, float inv, __half& hi, __half& lo) {
  const float v = x * mul;
  hi = __float2half_rn(v);
  lo = __float2half_rn((v - __half2float(hi)) * kHalfUp);
  return fabsf(half_rest(x, inv, hi, lo)) > 0x1p-22f * fabsf(x);
}
// Lists what the halves of one row's block leave, eight elements per lane: bit j of `bad` (of some lane) says that
// element j, at k_of(j), is not held.  In the order of the lanes, so that a run repeats itself.
template <class KOf>
__device__ __forceinline__ void list_rests(uint32_t bad, const float (&x)[8], float mul, float inv, KOf k_of, int kb,
                                           int row, const HalfOut& o) {
  const int lane = threadIdx.x & 31;
  int at = __popc(bad);
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int before = __shfl_up_sync(0xffffffffu, at, d);
    if (lane >= d) at += before;
  }
  const int n = __shfl_sync(0xffffffffu, at, 31);
  at -= __popc(bad);
  int2* list = o.rest + ((size_t)kb * o.rp + row) * gemm::kHalfRest;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (bad >> j & 1u) {
      __half hi, lo;
      split_half(x[j], mul, inv, hi, lo);
      if (at < gemm::kHalfRest) list[at] = make_int2(k_of(j), __float_as_int(half_rest(x[j], inv, hi, lo)));
      ++at;
    }
  }
  if (lane >= n && lane < gemm::kHalfRest) list[lane] = make_int2(-1, 0);
  if (lane == 0) {
    *o.listed = o.epoch;
    if (n > gemm::kHalfRest || atomicAdd(o.count, (uint32_t)n) + n > o.limit) *o.unfit = o.epoch;
  }
}

// src [R, C] row-major -> scaled f16 planes [R, ld] and what belongs to them.  A CTA takes 32 rows x 256 values, a warp
// four of the rows, eight values per lane.  GROUP: one scale for the 32 rows (operand B), else one per row.
// Bound by HBM, 8 bytes per element: 8192 x 4096 in 43 us (6.2 TB/s); the TF32 planes, 12 bytes, took 70 us.
template <bool VEC, bool GROUP>
__global__ void __launch_bounds__(256) split_rows_half_kernel(const float* __restrict__ src, int R, int C,
                                                              const HalfOut o) {
  __shared__ float part[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int blocks = (C + gemm::kHalfBlock - 1) / gemm::kHalfBlock;
  const long long n = (long long)((R + 31) / 32) * blocks;
  for (long long t = blockIdx.x; t < n; t += gridDim.x) {
    const int grp = (int)(t / blocks), kb = (int)(t - (long long)grp * blocks);
    const int c = kb * gemm::kHalfBlock + lane * 8, r0 = grp * 32 + warp * 4;
    float v[4][8], m[4], all = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float* a = src + (size_t)(r0 + q) * C + c;
      const bool row = r0 + q < R;
      if (VEC) {
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 u0 = row && c < C ? __ldg(reinterpret_cast<const float4*>(a)) : z;  // C % 4 == 0
        const float4 u1 = row && c + 4 < C ? __ldg(reinterpret_cast<const float4*>(a) + 1) : z;
        v[q][0] = u0.x; v[q][1] = u0.y; v[q][2] = u0.z; v[q][3] = u0.w;
        v[q][4] = u1.x; v[q][5] = u1.y; v[q][6] = u1.z; v[q][7] = u1.w;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[q][j] = row && c + j < C ? __ldg(a + j) : 0.0f;
      }
    }
    if (known_unfit(o)) return;  // asked behind the loads, which take as long
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      m[q] = 0.0f;
#pragma unroll
      for (int j = 0; j < 8; ++j) m[q] = fmaxf(m[q], fabsf(v[q][j]));
      all = fmaxf(all, m[q]);
    }
    if (GROUP) all = block_amax(all, part);
    uint32_t bad = 0;  // bit 8 q + j: element j of row q is not held
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float mul, inv;
      block_scale(GROUP ? all : warp_amax(m[q]), mul, inv);
      if (r0 + q >= R) break;
      if (lane == 0 && (!GROUP || q == 0)) note_scale(mul, o);
      union { __half h[8]; uint4 u; } ph, pl;
#pragma unroll
      for (int j = 0; j < 8; ++j) bad |= split_half(v[q][j], mul, inv, ph.h[j], pl.h[j]) ? 1u << (8 * q + j) : 0u;
      if (c < o.ld) {  // ld is C rounded up to 8
        *reinterpret_cast<uint4*>(o.hi + (size_t)(r0 + q) * o.ld + c) = ph.u;
        *reinterpret_cast<uint4*>(o.lo + (size_t)(r0 + q) * o.ld + c) = pl.u;
      }
      if (!GROUP && lane == 0) o.scale[(size_t)kb * o.rp + r0 + q] = inv;
      if (GROUP && threadIdx.x == 0 && q == 0) o.scale[(size_t)kb * (o.rp / gemm::kHalfGroup) + grp] = inv;
    }
    uint32_t flags = 0;
    if (__any_sync(0xffffffffu, bad != 0)) {  // seldom: the row is read again, which leaves the registers to the rest
#pragma unroll 1
      for (int q = 0; q < 4; ++q) {
        const uint32_t b = bad >> (8 * q) & 0xffu;
        if (!__any_sync(0xffffffffu, b != 0)) continue;
        float x[8], mx = 0.0f, mul, inv;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          x[j] = c + j < C ? __ldg(src + (size_t)(r0 + q) * C + c + j) : 0.0f;
          mx = fmaxf(mx, fabsf(x[j]));
        }
        block_scale(GROUP ? all : warp_amax(mx), mul, inv);
        list_rests(b, x, mul, inv, [&](int j) { return c + j; }, kb, r0 + q, o);
        flags |= 1u << q;
      }
    }
    if (lane == 0) o.flags[(size_t)kb * (o.rp / 4) + r0 / 4] = (uint8_t)flags;
  }
}

// src [R, C] row-major -> planes of the transpose, [C, ld >= R], and what belongs to them; where `colsum` is given, also
// the f64 column sums of each block, colsum[block][C] (the bias gradient's partial sums: a pass of its own over the
// gradient took 71 us per 8192 x 4096).  A CTA turns 256 rows x 32 columns through shared memory: 128-byte rows in, and
// a warp writes 128 contiguous bytes of a plane per instruction.  8192 x 4096: 57 us (73 us for TF32 planes).
template <bool GROUP>
__global__ void __launch_bounds__(256) split_transpose_half_kernel(const float* __restrict__ src, int R, int C,
                                                                   double* __restrict__ colsum, const HalfOut o) {
  __shared__ float tile[gemm::kHalfBlock][33];
  __shared__ float part[8];
  const int tiles_c = (C + 31) / 32, tiles_r = (R + gemm::kHalfBlock - 1) / gemm::kHalfBlock;
  const long long ntiles = (long long)tiles_c * tiles_r;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int kb = (int)(t / tiles_c), r0 = kb * gemm::kHalfBlock, c0 = (int)(t - (long long)kb * tiles_c) * 32;
    const int c = c0 + lane;
    float all = 0.0f;
    __syncthreads();  // the previous tile has been read
#pragma unroll 16
    for (int j = 0; j < gemm::kHalfBlock; j += 8) {
      const int r = r0 + warp + j;
      const float x = (r < R && c < C) ? __ldg(src + (size_t)r * C + c) : 0.0f;
      tile[warp + j][lane] = x;
      if (GROUP) all = fmaxf(all, fabsf(x));
    }
    if (known_unfit(o) && !colsum) return;  // also waits for the tile; the column sums are wanted all the same
    if (GROUP) all = block_amax(all, part);
    uint32_t bad = 0;  // bit 8 q + j: element j of column q is not held
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int col = warp * 4 + q, cg = c0 + col;
      if (cg >= C) break;
      float v[8];
      float m = 0.0f, mul, inv;
#pragma unroll
      for (int i = 0; i < 4; ++i) {  // rows i * 64 + lane * 2 + {0, 1}
        v[2 * i] = tile[i * 64 + lane * 2][col];
        v[2 * i + 1] = tile[i * 64 + lane * 2 + 1][col];
        m = fmaxf(m, fmaxf(fabsf(v[2 * i]), fabsf(v[2 * i + 1])));
      }
      block_scale(GROUP ? all : warp_amax(m), mul, inv);
      if (lane == 0 && (!GROUP || q == 0)) note_scale(mul, o);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = r0 + i * 64 + lane * 2;
        __half2 h, l;
        bad |= split_half(v[2 * i], mul, inv, h.x, l.x) ? 1u << (8 * q + 2 * i) : 0u;
        bad |= split_half(v[2 * i + 1], mul, inv, h.y, l.y) ? 2u << (8 * q + 2 * i) : 0u;
        if (r < o.ld) {  // ld is R rounded up to 8
          *reinterpret_cast<__half2*>(o.hi + (size_t)cg * o.ld + r) = h;
          *reinterpret_cast<__half2*>(o.lo + (size_t)cg * o.ld + r) = l;
        }
      }
      if (!GROUP && lane == 0) o.scale[(size_t)kb * o.rp + cg] = inv;
      if (GROUP && threadIdx.x == 0 && q == 0) o.scale[(size_t)kb * (o.rp / gemm::kHalfGroup) + c0 / 32] = inv;
      if (colsum) {
        double s = 0.0;
#pragma unroll
        for (int i = 0; i < 8; ++i) s = __dadd_rn(s, (double)v[i]);
#pragma unroll
        for (int o2 = 16; o2 > 0; o2 >>= 1) s = __dadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o2));
        if (lane == 0) colsum[(size_t)kb * C + cg] = s;
      }
    }
    uint32_t flags = 0;
    if (__any_sync(0xffffffffu, bad != 0)) {  // seldom
#pragma unroll 1
      for (int q = 0; q < 4; ++q) {
        const uint32_t b = bad >> (8 * q) & 0xffu;
        if (!__any_sync(0xffffffffu, b != 0)) continue;
        float x[8], mx = 0.0f, mul, inv;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          x[j] = tile[(j >> 1) * 64 + lane * 2 + (j & 1)][warp * 4 + q];
          mx = fmaxf(mx, fabsf(x[j]));
        }
        block_scale(GROUP ? all : warp_amax(mx), mul, inv);
        list_rests(b, x, mul, inv, [&](int j) { return r0 + (j >> 1) * 64 + lane * 2 + (j & 1); }, kb, c0 + warp * 4 + q, o);
        flags |= 1u << q;
      }
    }
    if (lane == 0) o.flags[(size_t)kb * (o.rp / 4) + c0 / 4 + warp] = (uint8_t)flags;
  }
}

// TF32 planes of both operands of a product whose operands do not fit f16 planes; returns at once for all others.
struct SplitSource {
  const float* src;
  float *hi, *lo;
  int rows, kdim, ld, transposed;  // transposed: stored [kdim, rows]
};
__global__ void __launch_bounds__(256) split_unfit_kernel(SplitSource a, SplitSource b, const uint32_t* unfit,
                                                          uint32_t epoch, uint32_t* counts) {
  __shared__ float tile[32][33];
  if (blockIdx.x == 0 && threadIdx.x < 2) counts[threadIdx.x] = 0;  // listed elements: the next product counts again
  if (*unfit != epoch) return;
  for (int o = 0; o < 2; ++o) {
    const SplitSource& s = o ? b : a;
    if (s.transposed)
      split_transpose(s.src, s.kdim, s.rows, s.ld, s.hi, s.lo, tile);
    else if (s.ld == s.kdim && ((uintptr_t)s.src & 15) == 0)
      split_rows_vec((const float4*)s.src, (float4*)s.hi, (float4*)s.lo, (size_t)s.rows * s.kdim / 4);
    else
      split_rows(s.src, s.rows, s.kdim, s.ld, s.hi, s.lo);
  }
}

// Column sums of G[M,N] in f64: partial[s][n] = sum over rows r == s (mod S).
__global__ void __launch_bounds__(128) colsum_partial_kernel(const float* __restrict__ G, int M,
                                                             int N, double* __restrict__ partial) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  double s = 0.0;
  for (int r = blockIdx.y; r < M; r += gridDim.y) s += (double)G[(size_t)r * N + n];
  partial[(size_t)blockIdx.y * N + n] = s;
}
__global__ void __launch_bounds__(128) colsum_final_kernel(const double* __restrict__ partial,
                                                           int S, int N, float* __restrict__ out) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  double s = 0.0;
  for (int i = 0; i < S; ++i) s += partial[(size_t)i * N + n];
  out[n] = (float)s;
}

// Column sums for short matrices in one launch: 32 columns per CTA, 8 row slices summed in f64
// and combined through shared memory in a fixed order.
__global__ void __launch_bounds__(256) colsum_short_kernel(const float* __restrict__ G, int M, int N,
                                                           float* __restrict__ out) {
  __shared__ double part[8][33];
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched early (vtlb_launch_early): the kernel in front is done
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int n = blockIdx.x * 32 + tx;
  double s = 0.0;
  if (n < N)
    for (int r = ty; r < M; r += 8) s += (double)G[(size_t)r * N + n];
  part[ty][tx] = s;
  __syncthreads();
  if (ty == 0 && n < N) {
    double t = 0.0;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += part[i][tx];
    out[n] = (float)t;
  }
}

// out[i] = sum over splits of partial[k][i].  One element per thread; eight running sums per
// element keep eight loads in flight (the order of the additions is fixed: split k goes to sum
// k mod 8, the eight sums are combined pairwise at the end).
__global__ void __launch_bounds__(256) reduce_splits_kernel(const float* __restrict__ partial,
                                                            int splits, size_t n,
                                                            float* __restrict__ out) {
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched early (vtlb_launch_early): the kernel in front is done from here on
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    float s[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) s[j] = 0.0f;
    int k = 0;
    for (; k + 8 <= splits; k += 8) {
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = partial[(size_t)(k + j) * n + i];
#pragma unroll
      for (int j = 0; j < 8; ++j) s[j] = __fadd_rn(s[j], v[j]);
    }
    for (int j = 0; k < splits; ++k, ++j) s[j] = __fadd_rn(s[j], partial[(size_t)k * n + i]);
    const float a = __fadd_rn(__fadd_rn(s[0], s[1]), __fadd_rn(s[2], s[3]));
    const float b = __fadd_rn(__fadd_rn(s[4], s[5]), __fadd_rn(s[6], s[7]));
    out[i] = __fadd_rn(a, b);
  }
}

}  // namespace

// Writes op(src) as K-major hi/lo [rows, ld] where rows x kdim is the logical
// operand.  `transposed` says src is stored [kdim, rows].
int f32::split_operand(vtlb_ctx* ctx, const float* src, int rows, int kdim, bool transposed, int ld,
                  float* hi, float* lo) {
  vtlb_prof_scope prof(ctx, VTLB_PHASE_SPLIT);
  if (!transposed) {
    if ((kdim & 3) == 0 && ld == kdim && vtlb_aligned16(src)) {
      const size_t n4 = (size_t)rows * kdim / 4;
      VTLB_CUDA(ctx, vtlb_launch_early(split_rows_vec_kernel, dim3(f32::grid_for(ctx, n4, 256 * 4)), dim3(256), 0,
                                       ctx->stream, (const float4*)src, (float4*)hi, (float4*)lo, n4));
    } else {
      VTLB_CUDA(ctx, vtlb_launch_early(split_rows_kernel, dim3(f32::grid_for(ctx, (size_t)rows * kdim, 256 * 4)), dim3(256),
                                       0, ctx->stream, src, rows, kdim, ld, hi, lo));
    }
  } else {
    const size_t tiles = (size_t)((rows + 31) / 32) * ((kdim + 31) / 32);
    VTLB_CUDA(ctx, vtlb_launch_early(split_transpose_kernel, dim3(f32::grid_for(ctx, tiles, 1)), dim3(256), 0, ctx->stream,
                                     src, kdim, rows, ld, hi, lo));
  }
  VTLB_LAUNCHED(ctx);
  return VTLB_OK;
}

namespace {

using f32::split_operand;

// Optional extras of a product (all null / zero by default):
//   a_planes / b_planes   the operand already split into K-major TF32 planes [rows, ld(K)] by whoever
//                         produced it (then no split pass runs for it)
//   mask                  ReLU backward on the result: C = mask < 0 ? 0 : C, mask laid out like C
//   out_rows / out_cols   receive the TF32 planes of C ([M, ld(N)]) and of C transposed ([N, ld(M)])
// The tensor-core kernels do mask and planes in their epilogue; where they cannot (CUDA-core route,
// unaligned pointers) the same results come from separate passes over the stored C.
struct GemmExtras {
  const vtlb_planes* a_planes = nullptr;
  const vtlb_planes* b_planes = nullptr;
  const float* mask = nullptr;
  const vtlb_planes* out_rows = nullptr;
  const vtlb_planes* out_cols = nullptr;
  // column sums of A as stored ([K, M], transA): the bias gradient, from the pass that transposes A; *colsum_done
  // says whether that pass ran
  float* a_colsum = nullptr;
  bool* colsum_done = nullptr;
};

// Splits one operand into f16 planes; `transposed` says src is stored [kdim, rows], `group` that 32 rows share a
// scale (operand B).
int split_operand_half(vtlb_ctx* ctx, const float* src, int kdim, bool transposed, bool group, int ld,
                       const f32::HalfPlanes::Side& p, double* colsum, uint32_t epoch) {
  vtlb_prof_scope prof(ctx, VTLB_PHASE_SPLIT);
  HalfOut o{p.hi, p.lo, p.scale, p.flags, p.rest, ld, p.rp};
  o.count = ctx->d_status + vtlb_ctx::kRestWord + (group ? 1 : 0);
  o.unfit = ctx->d_status + vtlb_ctx::kUnfitWord;
  o.listed = ctx->d_status + vtlb_ctx::kListedWord;
  o.limit = 4u + (uint32_t)((unsigned long long)p.rows * kdim >> 19);
  o.epoch = epoch;
  const int grid = f32::grid_for(ctx, (size_t)((p.rows + 31) / 32) * ((kdim + gemm::kHalfBlock - 1) / gemm::kHalfBlock), 1);
  if (transposed) {
    auto kern = group ? split_transpose_half_kernel<true> : split_transpose_half_kernel<false>;
    kern<<<grid, 256, 0, ctx->stream>>>(src, kdim, p.rows, colsum, o);
  } else {
    const bool vec = (kdim & 3) == 0 && vtlb_aligned16(src);
    auto kern = group ? (vec ? split_rows_half_kernel<true, true> : split_rows_half_kernel<false, true>)
                      : (vec ? split_rows_half_kernel<true, false> : split_rows_half_kernel<false, false>);
    kern<<<grid, 256, 0, ctx->stream>>>(src, p.rows, kdim, o);
  }
  VTLB_LAUNCHED(ctx);
  return VTLB_OK;
}

int relu_mask_inplace(vtlb_ctx* ctx, float* C, const float* mask, size_t n) {
  return vtlb_relu_bwd_f32(ctx, C, mask, C, n);
}

// Which products run on CUDA cores.  Up to the limit all; beyond it, unless the caller has set one, those whose long K
// a tensor-core tile would walk alone: that kernel takes 14 us and 16 us per 1000 of K with its split passes, the
// CUDA-core one 5.5 us and 85 us per GFLOP as long as its K ranges stay at 256 or less (256 x 512 x 600: 20.5 against
// 24.8 us, 256 x 256 x 2048: 26 against 47, 512 x 64 x 4096: 28 against 80; 512 x 512 x 512: 27 against 23).
bool ranges_short(vtlb_ctx* ctx, int M, int N, int K) {
  return (double)((M + 31) / 32) * ((N + 63) / 64) * ((K + 255) / 256) <= 4.0 * ctx->sm_count;
}
bool small_product(vtlb_ctx* ctx, int M, int N, int K) {
  const double flops = 2.0 * M * N * K;
  if (flops <= ctx->small_gemm_flops) return true;
  return ctx->small_gemm_default && K >= 512 && flops <= 1.0e8 + 1.9e5 * K && ranges_short(ctx, M, N, K);
}
// Both products of a Linear backward (contractions of N and M), which share a launch there.
bool small_backward(vtlb_ctx* ctx, int M, int N, int K) {
  const double flops = 2.0 * M * N * K;
  if (flops <= ctx->small_gemm_flops) return true;
  return ctx->small_gemm_default && flops <= 1.2e8 + 0.95e5 * ((double)M + N) && ranges_short(ctx, M, K, N) &&
         ranges_short(ctx, N, K, M);
}

int gemm_f32_impl(vtlb_ctx* ctx, int transA, int transB, int M, int N, int K, const float* A,
                  const float* B, float* C, const float* bias, int relu, float* pre,
                  const GemmExtras& ex = GemmExtras()) {
  if (!vtlb_aligned16(C) || (pre && !vtlb_aligned16(pre)) || (bias && !vtlb_aligned16(bias)))
    return vtlb_fail(ctx, VTLB_EINVAL, "f32 GEMM: output and bias pointers must be 16-byte aligned");
  const int ld_rows = vtlb_plane_ld(N), ld_cols = vtlb_plane_ld(M);
  int rc, fused = 0;
  const bool planes_in_or_out = ex.a_planes || ex.b_planes || ex.out_rows || ex.out_cols;
  bool small = small_product(ctx, M, N, K);
  if (small && 2.0 * M * N * K > ctx->small_gemm_flops) {
    // CUDA cores read the operands while C is written.  Above the limit a result may lie over an operand: the
    // tensor-core routes have copied both before they write.
    auto over = [&](const float* out) {
      return vtlb_overlap(out, (size_t)M * N, A, (size_t)M * K) || vtlb_overlap(out, (size_t)M * N, B, (size_t)N * K);
    };
    small = !over(C) && !(pre && over(pre));
  }
  if (!small && !planes_in_or_out && f32::pair_product(ctx, M, N)) {
    // Large products: f16 planes on CTA pairs, twice the tensor rate of TF32 planes and half their bytes.  Planes
    // that come in or go out are TF32 ones, so products with those keep the 3xTF32 kernel.
    const int blocks = (K + gemm::kHalfBlock - 1) / gemm::kHalfBlock;
    const bool sums = ex.a_colsum && transA;
    f32::HalfPlanes p;
    if ((rc = f32::alloc_half_planes(ctx, M, N, K, sums ? (size_t)blocks * M * sizeof(double) : 0, &p))) return rc;
    double* partial = sums ? (double*)p.extra : nullptr;
    if (++ctx->half_epoch == 0) ctx->half_epoch = 1;
    const uint32_t epoch = ctx->half_epoch;
    if ((rc = split_operand_half(ctx, A, K, transA != 0, false, p.ld, p.a, partial, epoch))) return rc;
    if ((rc = split_operand_half(ctx, B, K, transB == 0, true, p.ld, p.b, nullptr, epoch))) return rc;
    {
      const SplitSource sa{A, p.tf32.a_hi, p.tf32.a_lo, M, K, p.tf32.ld, transA != 0};
      const SplitSource sb{B, p.tf32.b_hi, p.tf32.b_lo, N, K, p.tf32.ld, transB == 0};
      split_unfit_kernel<<<ctx->sm_count * 8, 256, 0, ctx->stream>>>(sa, sb, ctx->d_status + vtlb_ctx::kUnfitWord, epoch,
                                                                     ctx->d_status + vtlb_ctx::kRestWord);
      VTLB_LAUNCHED(ctx);
    }
    f32::EpiBiasRelu epi{C, bias, pre, N, relu};
    epi.mask = ex.mask;
    if ((rc = f32::launch_f16x3(ctx, p, M, N, K, epi, epoch, &fused))) return rc;
    if (sums) {  // written last, as by a pass of its own
      colsum_final_kernel<<<(M + 127) / 128, 128, 0, ctx->stream>>>(partial, blocks, M, ex.a_colsum);
      VTLB_LAUNCHED(ctx);
      *ex.colsum_done = true;
    }
  } else if (small) {  // launch-latency-bound sizes: CUDA cores, no split passes
    if ((rc = f32::sgemm_small(ctx, transA, transB, M, N, K, A, B, C, bias, relu, pre, nullptr, nullptr, ex.mask)))
      return rc;
    if (ex.mask) fused |= 2;  // the mask is part of that kernel's epilogue
  } else {
    f32::Planes p;
    if ((rc = f32::alloc_planes(ctx, ex.a_planes ? 0 : M, ex.b_planes ? 0 : N, K, 0, &p))) return rc;
    // op(A) is [M,K]: stored [K,M] when transA.  The B operand of the kernel is
    // [N,K] K-major: B stored [K,N] (transB == 0) must be transposed.
    if (ex.a_planes) {
      p.a_hi = (float*)ex.a_planes->hi;
      p.a_lo = (float*)ex.a_planes->lo;
    } else if ((rc = split_operand(ctx, A, M, K, transA != 0, p.ld, p.a_hi, p.a_lo))) {
      return rc;
    }
    if (ex.b_planes) {
      p.b_hi = (float*)ex.b_planes->hi;
      p.b_lo = (float*)ex.b_planes->lo;
    } else if ((rc = split_operand(ctx, B, N, K, transB == 0, p.ld, p.b_hi, p.b_lo))) {
      return rc;
    }
    f32::EpiBiasRelu epi{C, bias, pre, N, relu};
    epi.mask = ex.mask;
    epi.planes = (ex.out_rows ? 1 : 0) | (ex.out_cols ? 2 : 0);
    if (ex.out_rows) {
      epi.rows_hi = (float*)ex.out_rows->hi;
      epi.rows_lo = (float*)ex.out_rows->lo;
      epi.ld_rows = ld_rows;
    }
    if (ex.out_cols) {
      epi.cols_hi = (float*)ex.out_cols->hi;
      epi.cols_lo = (float*)ex.out_cols->lo;
      epi.ld_cols = ld_cols;
    }
    if ((rc = f32::launch_tf32x3(ctx, p, M, N, K, epi, 1, &fused))) return rc;
  }
  if (ex.mask && !(fused & 2) && (rc = relu_mask_inplace(ctx, C, ex.mask, (size_t)M * N))) return rc;
  // planes written by the epilogue are those of the masked result only when it also masked
  const bool planes_ok = (fused & 1) && (!ex.mask || (fused & 2));
  if (!planes_ok) {
    if (ex.out_rows && (rc = split_operand(ctx, C, M, N, false, ld_rows, (float*)ex.out_rows->hi, (float*)ex.out_rows->lo)))
      return rc;
    if (ex.out_cols && (rc = split_operand(ctx, C, N, M, true, ld_cols, (float*)ex.out_cols->hi, (float*)ex.out_cols->lo)))
      return rc;
  }
  return VTLB_OK;
}

int colsum(vtlb_ctx* ctx, const float* G, int M, int N, float* out) {
  vtlb_prof_scope prof(ctx, VTLB_PHASE_ELEMENTWISE);
  if (M <= 1024) {
    VTLB_CUDA(ctx, vtlb_launch_early(colsum_short_kernel, dim3((N + 31) / 32), dim3(256), 0, ctx->stream, G, M, N, out));
    VTLB_LAUNCHED(ctx);
    return VTLB_OK;
  }
  int S = (M + 63) / 64;
  if (S > 64) S = 64;
  if (S < 1) S = 1;
  void* scr = nullptr;
  int rc = vtlb_scratch(ctx, (size_t)S * N * sizeof(double), &scr);
  if (rc) return rc;
  dim3 grid((N + 127) / 128, S);
  colsum_partial_kernel<<<grid, 128, 0, ctx->stream>>>(G, M, N, (double*)scr);
  VTLB_LAUNCHED(ctx);
  colsum_final_kernel<<<(N + 127) / 128, 128, 0, ctx->stream>>>((const double*)scr, S, N, out);
  VTLB_LAUNCHED(ctx);
  return VTLB_OK;
}

int check_f32(vtlb_ctx* ctx, const char* fn, int M, int N, int K) {
  if (M < 0 || N < 0 || K <= 0)
    return vtlb_fail(ctx, VTLB_EINVAL, "%s: bad shape M=%d N=%d K=%d (K must be > 0)", fn, M, N, K);
  return VTLB_OK;
}

}  // namespace

int f32::reduce_splits(vtlb_ctx* ctx, const float* partial, int splits, size_t n, float* out) {
  VTLB_CUDA(ctx, vtlb_launch_early(reduce_splits_kernel, dim3(f32::grid_for(ctx, n, 256)), dim3(256), 0, ctx->stream, partial,
                                   splits, n, out));
  VTLB_LAUNCHED(ctx);
  return VTLB_OK;
}

VTLB_API int vtlb_gemm_f32(vtlb_ctx* ctx, int transA, int transB, int M, int N, int K,
                           const void* d_A, const void* d_B, void* d_C,
                           const void* d_bias_or_null, int relu) {
  VTLB_ENTER(ctx);
  int rc = check_f32(ctx, "vtlb_gemm_f32", M, N, K);
  if (rc) return rc;
  if (M == 0 || N == 0) return VTLB_OK;
  if (!d_A || !d_B || !d_C) return vtlb_fail(ctx, VTLB_EINVAL, "vtlb_gemm_f32: null pointer");
  return gemm_f32_impl(ctx, transA, transB, M, N, K, (const float*)d_A, (const float*)d_B,
                       (float*)d_C, (const float*)d_bias_or_null, relu, nullptr);
}

namespace {

int check_planes(vtlb_ctx* ctx, const char* fn, const char* what, const vtlb_planes* p) {
  if (p && (!p->hi || !p->lo || !vtlb_aligned16(p->hi) || !vtlb_aligned16(p->lo)))
    return vtlb_fail(ctx, VTLB_EINVAL, "%s: %s planes need two 16-byte-aligned arrays", fn, what);
  return VTLB_OK;
}

int linear_fwd_impl(vtlb_ctx* ctx, const char* fn, const void* d_X, const void* d_W, const void* d_b_or_null,
                    void* d_Y, int M, int N, int K, int relu, void* d_pre_or_null, const vtlb_planes* x_rows,
                    const vtlb_planes* y_rows, const vtlb_planes* y_cols) {
  int rc = check_f32(ctx, fn, M, N, K);
  if (rc) return rc;
  if (M == 0 || N == 0) return VTLB_OK;
  if (!d_X || !d_W || !d_Y) return vtlb_fail(ctx, VTLB_EINVAL, "%s: null pointer", fn);
  if ((rc = check_planes(ctx, fn, "input", x_rows)) || (rc = check_planes(ctx, fn, "output", y_rows)) ||
      (rc = check_planes(ctx, fn, "transposed output", y_cols)))
    return rc;
  if (!x_rows && !y_rows && !y_cols && 2.0 * M * N * K <= ctx->small_gemm_flops &&
      f32::narrow_linear_ok(M, N, K, d_X, d_W, d_X))
    return f32::narrow_linear_fwd(ctx, (const float*)d_X, (const float*)d_W, (const float*)d_b_or_null, (float*)d_Y, M, N,
                                  K, relu, (float*)d_pre_or_null);
  GemmExtras ex;
  ex.a_planes = x_rows;
  ex.out_rows = y_rows;
  ex.out_cols = y_cols;
  return gemm_f32_impl(ctx, 0, 1, M, N, K, (const float*)d_X, (const float*)d_W, (float*)d_Y,
                       (const float*)d_b_or_null, relu, (float*)d_pre_or_null, ex);
}

int linear_bwd_impl(vtlb_ctx* ctx, const char* fn, const void* d_G, const void* d_X, const void* d_W,
                    void* d_dX_or_null, void* d_dW_or_null, void* d_db_or_null, int M, int N, int K,
                    const vtlb_planes* g_rows, const vtlb_planes* g_cols, const vtlb_planes* x_cols,
                    const void* d_relu_mask_src_or_null, const vtlb_planes* dx_rows, const vtlb_planes* dx_cols) {
  if (M <= 0 || N <= 0 || K <= 0) return vtlb_fail(ctx, VTLB_EINVAL, "%s: bad shape M=%d N=%d K=%d", fn, M, N, K);
  if (!d_G) return vtlb_fail(ctx, VTLB_EINVAL, "%s: null gradient", fn);
  int rc;
  if ((rc = check_planes(ctx, fn, "gradient", g_rows)) || (rc = check_planes(ctx, fn, "transposed gradient", g_cols)) ||
      (rc = check_planes(ctx, fn, "transposed input", x_cols)) || (rc = check_planes(ctx, fn, "dX", dx_rows)) ||
      (rc = check_planes(ctx, fn, "transposed dX", dx_cols)))
    return rc;
  if (!d_dX_or_null && (d_relu_mask_src_or_null || dx_rows || dx_cols))
    return vtlb_fail(ctx, VTLB_EINVAL, "%s: a mask or dX planes were given without a dX output", fn);
  // a layer with few output features and many inputs: memory-bound kernels that stream X / dX once
  const bool any_planes = g_rows || g_cols || x_cols || dx_rows || dx_cols;
  const bool narrow = !any_planes && 2.0 * M * N * K <= ctx->small_gemm_flops;
  if (narrow && d_dX_or_null && d_W && f32::narrow_linear_ok(M, N, K, d_dX_or_null, d_W, d_W)) {
    if ((rc = f32::narrow_linear_dx(ctx, (const float*)d_G, (const float*)d_W, (float*)d_dX_or_null, M, N, K))) return rc;
    if (d_relu_mask_src_or_null &&
        (rc = relu_mask_inplace(ctx, (float*)d_dX_or_null, (const float*)d_relu_mask_src_or_null, (size_t)M * K)))
      return rc;
    d_dX_or_null = nullptr;
  }
  if (narrow && d_dW_or_null && d_X && f32::narrow_linear_ok(M, N, K, d_X, d_dW_or_null, d_X)) {
    if ((rc = f32::narrow_linear_dw(ctx, (const float*)d_G, (const float*)d_X, (float*)d_dW_or_null,
                                    (float*)d_db_or_null, M, N, K)))
      return rc;
    d_dW_or_null = nullptr;
    d_db_or_null = nullptr;
  }
  bool db_done = false;
  // a small layer: both products in one launch, where no result lies over another or over what is read (the mask may be
  // dX itself: each value is read by the thread that writes it)
  const void *outs[3] = {d_dX_or_null, d_dW_or_null, d_db_or_null};
  const size_t out_n[3] = {(size_t)M * K, (size_t)N * K, (size_t)N};
  auto apart = [&] {
    const void* ins[4] = {d_G, d_X, d_W, d_relu_mask_src_or_null};
    const size_t in_n[4] = {(size_t)M * N, (size_t)M * K, (size_t)N * K, (size_t)M * K};
    for (int o = 0; o < 3; ++o) {
      for (int i = 0; i < 4; ++i)
        if (outs[o] && ins[i] && !(o == 0 && i == 3 && outs[o] == ins[i]) && vtlb_overlap(outs[o], out_n[o], ins[i], in_n[i]))
          return false;
      for (int p = 0; p < o; ++p)
        if (outs[o] && outs[p] && vtlb_overlap(outs[o], out_n[o], outs[p], out_n[p])) return false;
    }
    return true;
  };
  if (!any_planes && small_backward(ctx, M, N, K) && d_dX_or_null && d_dW_or_null && d_W && d_X &&
      vtlb_aligned16(d_dX_or_null) && vtlb_aligned16(d_dW_or_null) && apart()) {
    bool done = false;
    if ((rc = f32::sgemm_small_linear_bwd(ctx, (const float*)d_G, (const float*)d_X, (const float*)d_W,
                                          (float*)d_dX_or_null, (float*)d_dW_or_null, (float*)d_db_or_null, M, N, K,
                                          (const float*)d_relu_mask_src_or_null, &done, &db_done)))
      return rc;
    if (done) d_dX_or_null = d_dW_or_null = nullptr;
  }
  if (d_dX_or_null) {  // dX[M,K] = G[M,N] . W[N,K]   (then, optionally, ReLU backward of the layer below)
    if (!d_W) return vtlb_fail(ctx, VTLB_EINVAL, "%s: dX needs W", fn);
    GemmExtras ex;
    ex.a_planes = g_rows;
    ex.mask = (const float*)d_relu_mask_src_or_null;
    ex.out_rows = dx_rows;
    ex.out_cols = dx_cols;
    if ((rc = gemm_f32_impl(ctx, 0, 0, M, K, N, (const float*)d_G, (const float*)d_W, (float*)d_dX_or_null, nullptr,
                            0, nullptr, ex)))
      return rc;
  }
  if (d_dW_or_null) {  // dW[N,K] = G^T[N,M] . X[M,K]
    if (!d_X) return vtlb_fail(ctx, VTLB_EINVAL, "%s: dW needs X", fn);
    if (d_db_or_null && 2.0 * M * N * K <= ctx->small_gemm_flops && vtlb_aligned16(d_dW_or_null)) {
      // small product: the CUDA-core kernel sums the rows of G^T (= the bias gradient) on the way
      if ((rc = f32::sgemm_small(ctx, 1, 0, N, K, M, (const float*)d_G, (const float*)d_X, (float*)d_dW_or_null,
                                 nullptr, 0, nullptr, (float*)d_db_or_null, &db_done)))
        return rc;
    } else {
      GemmExtras ex;
      ex.a_planes = g_cols;
      ex.b_planes = x_cols;
      ex.a_colsum = (float*)d_db_or_null;
      ex.colsum_done = &db_done;
      if ((rc = gemm_f32_impl(ctx, 1, 0, N, K, M, (const float*)d_G, (const float*)d_X, (float*)d_dW_or_null,
                              nullptr, 0, nullptr, ex)))
        return rc;
    }
  }
  if (d_db_or_null && !db_done) {
    if ((rc = colsum(ctx, (const float*)d_G, M, N, (float*)d_db_or_null))) return rc;
  }
  return VTLB_OK;
}

}  // namespace

VTLB_API int vtlb_plane_ld(int kdim) { return kdim <= 0 ? 0 : (int)vtlb_round_up((size_t)kdim, 4); }

VTLB_API int vtlb_f32_planes_worthwhile(vtlb_ctx* ctx, int M, int N, int K) {
  // products the CUDA-core route takes never read operand planes
  return ctx && M > 0 && N > 0 && K > 0 && !small_product(ctx, M, N, K);
}

VTLB_API int vtlb_linear_fwd_f32(vtlb_ctx* ctx, const void* d_X, const void* d_W,
                                 const void* d_b_or_null, void* d_Y, int M, int N, int K, int relu,
                                 void* d_pre_or_null) {
  VTLB_ENTER(ctx);
  return linear_fwd_impl(ctx, "vtlb_linear_fwd_f32", d_X, d_W, d_b_or_null, d_Y, M, N, K, relu, d_pre_or_null,
                         nullptr, nullptr, nullptr);
}

VTLB_API int vtlb_linear_fwd_f32_planes(vtlb_ctx* ctx, const void* d_X, const void* d_W, const void* d_b_or_null,
                                        void* d_Y, int M, int N, int K, int relu, void* d_pre_or_null,
                                        const vtlb_planes* x_rows_or_null, const vtlb_planes* y_rows_or_null,
                                        const vtlb_planes* y_cols_or_null) {
  VTLB_ENTER(ctx);
  return linear_fwd_impl(ctx, "vtlb_linear_fwd_f32_planes", d_X, d_W, d_b_or_null, d_Y, M, N, K, relu,
                         d_pre_or_null, x_rows_or_null, y_rows_or_null, y_cols_or_null);
}

VTLB_API int vtlb_linear_bwd_f32(vtlb_ctx* ctx, const void* d_G, const void* d_X, const void* d_W,
                                 void* d_dX_or_null, void* d_dW_or_null, void* d_db_or_null, int M,
                                 int N, int K) {
  VTLB_ENTER(ctx);
  return linear_bwd_impl(ctx, "vtlb_linear_bwd_f32", d_G, d_X, d_W, d_dX_or_null, d_dW_or_null, d_db_or_null, M, N,
                         K, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr);
}

VTLB_API int vtlb_linear_bwd_f32_planes(vtlb_ctx* ctx, const void* d_G, const void* d_X, const void* d_W,
                                        void* d_dX_or_null, void* d_dW_or_null, void* d_db_or_null, int M, int N,
                                        int K, const vtlb_planes* g_rows_or_null, const vtlb_planes* g_cols_or_null,
                                        const vtlb_planes* x_cols_or_null, const void* d_relu_mask_src_or_null,
                                        const vtlb_planes* dx_rows_or_null, const vtlb_planes* dx_cols_or_null) {
  VTLB_ENTER(ctx);
  return linear_bwd_impl(ctx, "vtlb_linear_bwd_f32_planes", d_G, d_X, d_W, d_dX_or_null, d_dW_or_null, d_db_or_null,
                         M, N, K, g_rows_or_null, g_cols_or_null, x_cols_or_null, d_relu_mask_src_or_null,
                         dx_rows_or_null, dx_cols_or_null);
}

VTLB_API int vtlb_split_planes_f32(vtlb_ctx* ctx, const void* d_src, int R, int C, const vtlb_planes* rows_or_null,
                                   const vtlb_planes* cols_or_null) {
  VTLB_ENTER(ctx);
  if (R <= 0 || C <= 0 || !d_src) return vtlb_fail(ctx, VTLB_EINVAL, "vtlb_split_planes_f32: bad arguments");
  int rc;
  if ((rc = check_planes(ctx, "vtlb_split_planes_f32", "row", rows_or_null)) ||
      (rc = check_planes(ctx, "vtlb_split_planes_f32", "column", cols_or_null)))
    return rc;
  if (rows_or_null && (rc = split_operand(ctx, (const float*)d_src, R, C, false, vtlb_plane_ld(C),
                                          (float*)rows_or_null->hi, (float*)rows_or_null->lo)))
    return rc;
  if (cols_or_null && (rc = split_operand(ctx, (const float*)d_src, C, R, true, vtlb_plane_ld(R),
                                          (float*)cols_or_null->hi, (float*)cols_or_null->lo)))
    return rc;
  return VTLB_OK;
}

// ---------------------------------------------------------------- bias gradient without allocation
// Some hosts cannot let this library allocate device memory while they run: a
// serving process that handed every byte of HBM to its own pools at start-up
// (so a cudaMalloc here would simply fail), or a control loop with a latency
// budget that the implicit synchronisation of an allocation would break.  For
// them the bias gradient (column sums of G) is offered with its partial-sum
// scratch in a fixed array that is part of the library image: every GPU that
// loads the library holds these 2 MiB until the process exits.
constexpr int kNoAllocMaxN = 4096;  // widest G supported by the fixed scratch
constexpr int kNoAllocMaxS = 64;    // row slices (same cap as the allocating path)
static __device__ __align__(256) double g_bias_grad_scratch[(size_t)kNoAllocMaxS * kNoAllocMaxN];

// In host code the array's name is only a handle; the device address has to be
// asked for, once per device, with that device current.
// (Atomic: two host threads may make their first calls on different contexts at the same time;
// both would resolve the same address, so the order of the stores does not matter.)
static std::atomic<double*> g_bias_grad_scratch_addr[64];

VTLB_API int vtlb_bias_grad_f32_noalloc(vtlb_ctx* ctx, const void* d_G, int M, int N, void* d_db) {
  VTLB_ENTER(ctx);
  if (M <= 0 || N <= 0)
    return vtlb_fail(ctx, VTLB_EINVAL, "vtlb_bias_grad_f32_noalloc: bad shape M=%d N=%d", M, N);
  if (N > kNoAllocMaxN)
    return vtlb_fail(ctx, VTLB_EINVAL,
                     "vtlb_bias_grad_f32_noalloc: N=%d exceeds the fixed scratch (at most %d "
                     "columns); use vtlb_linear_bwd_f32, which allocates",
                     N, kNoAllocMaxN);
  if (!d_G || !d_db) return vtlb_fail(ctx, VTLB_EINVAL, "vtlb_bias_grad_f32_noalloc: null pointer");
  if (ctx->device < 0 || ctx->device >= 64)
    return vtlb_fail(ctx, VTLB_EINVAL, "vtlb_bias_grad_f32_noalloc: device index %d not supported", ctx->device);
  double* scratch = g_bias_grad_scratch_addr[ctx->device].load(std::memory_order_relaxed);
  if (!scratch) {  // first call on this device: resolve the array's device address
    void* p = nullptr;
    VTLB_CUDA(ctx, cudaGetSymbolAddress(&p, g_bias_grad_scratch));
    scratch = (double*)p;
    g_bias_grad_scratch_addr[ctx->device].store(scratch, std::memory_order_relaxed);
  }
  int S = (M + 63) / 64;
  if (S > kNoAllocMaxS) S = kNoAllocMaxS;
  // every partial[s][n] with s < S, n < N is written by the first kernel before the second
  // reads it, so nothing left over from an earlier call is ever used and nothing needs clearing
  dim3 grid((N + 127) / 128, S);
  colsum_partial_kernel<<<grid, 128, 0, ctx->stream>>>((const float*)d_G, M, N, scratch);
  VTLB_LAUNCHED(ctx);
  colsum_final_kernel<<<(N + 127) / 128, 128, 0, ctx->stream>>>(scratch, S, N, (float*)d_db);
  VTLB_LAUNCHED(ctx);
  return VTLB_OK;
}
