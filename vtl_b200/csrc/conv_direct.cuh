// Convolution on CUDA cores, for the products the tensor-core kernels are bad at: first layers (3 source channels
// padded to a K block of 32, or 3 output columns to a tile of 64) and small batches (a handful of 128-pixel tiles,
// each walking a long K alone).  Nothing is lowered, regrouped or split into planes: full f32 products and sums.
//   conv_direct_kernel  dst[b][cd][y][x] = sum over (cs, a, b') of src[b][cs][y + oy + a][x + ox + b'] * w
//                       forward, and the input gradient of a unit stride (weights mirrored)
//   wgrad_direct_kernel dW[o][c][a][b'] = sum over pixels of g[o][y][x] * x[c][y*sh - ph + a][x*sw - pw + b']
#pragma once
#include <math.h>

#include "conv_igemm.cuh"
#include "conv_slab.cuh"
#include "f32_common.cuh"
#include "ptx.cuh"

namespace cdirect {

constexpr int PX = 4;            // neighbouring pixels of a thread
constexpr int kThreads = 256;
constexpr int kStageBytes = 40 * 1024;

struct Params {
  const float* src;
  const float* w;
  const float* bias;  // may be null
  float* dst;
  float* pre;         // may be null: the values before the ReLU
  int B, Cs, Hs, Ws, Cd, Hd, Wd;
  int oy, ox;         // source position of output (0, 0) at tap (0, 0)
  int mirror;         // 0: w is [cd][cs][K][K]; 1: w is [cs][cd][K][K], taps reversed
  int relu, vec;      // vec: rows of dst may be written 16 bytes at a time
  int TH, W4, CG, Z;  // a CTA: TH rows x W4 pixel groups, CG groups of CT channels, Z slices of the source channels
  int CS, pitch;      // source channels per stage, row pitch of the staged source
  int tiles_y;
};

// One f32 from global to shared memory without a register in between; zero where `in` is false (nothing is read).
__device__ __forceinline__ void copy_f32(float* dst, const float* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(ptx::smem_u32(dst)), "l"(src), "r"(in ? 4 : 0)
               : "memory");
}

// A thread keeps CT channels x 4 pixels; per source row it reads 4 + K - 1 values (16-byte loads, neighbouring lanes
// 16 bytes apart) and K x CT weights (one address per warp as a rule) from shared memory for 4 * K * CT products.
// Bound by FFMA issue; two products an instruction, paired over channels.
template <int K, int CT>
__global__ void __launch_bounds__(kThreads, 3) conv_direct_kernel(const Params p) {
  extern __shared__ __align__(16) float smem[];
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched early: the kernel in front is done from here on
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  constexpr int KK = K * K, NV = (PX + K - 1 + 3) / 4;
  const int CB = p.CG * CT, rows = p.TH + K - 1, PG = p.TH * p.W4;
  float* ssrc = smem;                              // [CS][rows][pitch]
  float* sw = smem + p.CS * rows * p.pitch;        // [CS][K*K][CB]
  const int img = blockIdx.x / p.tiles_y, y0 = (blockIdx.x - img * p.tiles_y) * p.TH;
  const int cd0 = blockIdx.y * CB;
  const int pg = threadIdx.x % PG, rest = threadIdx.x / PG;
  const int cg = rest % p.CG, z = rest / p.CG;
  const bool active = z < p.Z;
  const int yl = pg / p.W4, x0 = (pg - yl * p.W4) * PX;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t acc[PX][CT / 2];
#pragma unroll
  for (int i = 0; i < PX; ++i)
#pragma unroll
    for (int c = 0; c < CT / 2; ++c) acc[i][c] = 0ull;

  for (int cs0 = 0; cs0 < p.Cs; cs0 += p.CS) {
    const int nc = min(p.CS, p.Cs - cs0);
    if (cs0) __syncthreads();
    for (int r = warp; r < nc * rows; r += kThreads / 32) {
      const int c = r / rows, y = y0 + r - c * rows + p.oy;
      const bool row = y >= 0 && y < p.Hs;
      const float* s = p.src + ((size_t)(img * p.Cs + cs0 + c) * p.Hs + (row ? y : 0)) * p.Ws;
      for (int x = lane; x < p.pitch; x += 32) {
        const int gx = x + p.ox;
        const bool in = row && gx >= 0 && gx < p.Ws;
        copy_f32(ssrc + r * p.pitch + x, in ? s + gx : p.src, in);
      }
    }
    const int n = nc * KK * CB;  // contiguous runs of the weights in the order of their storage
    for (int i = threadIdx.x; i < n; i += kThreads) {
      int c, cd, t;
      size_t at;
      if (p.mirror) {
        c = i / (CB * KK);
        const int r = i - c * CB * KK;
        cd = r / KK;
        t = KK - 1 - (r - cd * KK);
        at = ((size_t)(cs0 + c) * p.Cd + cd0 + cd) * KK + (KK - 1 - t);
      } else {
        cd = i / (nc * KK);
        const int r = i - cd * nc * KK;
        c = r / KK;
        t = r - c * KK;
        at = ((size_t)(cd0 + cd) * p.Cs + cs0 + c) * KK + t;
      }
      const bool in = cd0 + cd < p.Cd;
      copy_f32(sw + (c * KK + t) * CB + cd, in ? p.w + at : p.w, in);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (active) {
      for (int c = z; c < nc; c += p.Z) {
#pragma unroll
        for (int a = 0; a < K; ++a) {
          const float4* row = reinterpret_cast<const float4*>(ssrc + (c * rows + yl + a) * p.pitch + x0);
          uint64_t s2[4 * NV];
#pragma unroll
          for (int v = 0; v < NV; ++v) {
            const float4 q = row[v];
            s2[4 * v] = ptx::f2_pack(q.x, q.x);
            s2[4 * v + 1] = ptx::f2_pack(q.y, q.y);
            s2[4 * v + 2] = ptx::f2_pack(q.z, q.z);
            s2[4 * v + 3] = ptx::f2_pack(q.w, q.w);
          }
#pragma unroll
          for (int b = 0; b < K; ++b) {
            const ulonglong2* wp = reinterpret_cast<const ulonglong2*>(sw + (c * KK + a * K + b) * CB + cg * CT);
#pragma unroll
            for (int h = 0; h < CT / 4; ++h) {
              const ulonglong2 w4 = wp[h];
#pragma unroll
              for (int i = 0; i < PX; ++i) {
                acc[i][2 * h] = ptx::f2_fma(w4.x, s2[b + i], acc[i][2 * h]);
                acc[i][2 * h + 1] = ptx::f2_fma(w4.y, s2[b + i], acc[i][2 * h + 1]);
              }
            }
          }
        }
      }
    }
  }

  // the slices' sums, added in order by slice 0
  float out[CT][PX];
#pragma unroll
  for (int c = 0; c < CT / 2; ++c)
#pragma unroll
    for (int i = 0; i < PX; ++i) ptx::f2_unpack(acc[i][c], out[2 * c][i], out[2 * c + 1][i]);
  if (p.Z > 1) {
    const int slots = PG * p.CG, slot = cg * PG + pg;
    __syncthreads();
    float4* park = reinterpret_cast<float4*>(smem);  // [Z - 1][CT][slots]
    if (active && z > 0) {
#pragma unroll
      for (int c = 0; c < CT; ++c)
        park[((z - 1) * CT + c) * slots + slot] = make_float4(out[c][0], out[c][1], out[c][2], out[c][3]);
    }
    __syncthreads();
    if (z > 0) return;
    for (int k = 0; k + 1 < p.Z; ++k) {
#pragma unroll
      for (int c = 0; c < CT; ++c) {
        const float4 v = park[(k * CT + c) * slots + slot];
        out[c][0] = __fadd_rn(out[c][0], v.x);
        out[c][1] = __fadd_rn(out[c][1], v.y);
        out[c][2] = __fadd_rn(out[c][2], v.z);
        out[c][3] = __fadd_rn(out[c][3], v.w);
      }
    }
  }
  const int y = y0 + yl;
  if (!active || y >= p.Hd || x0 >= p.Wd) return;
#pragma unroll
  for (int c = 0; c < CT; ++c) {
    const int cd = cd0 + cg * CT + c;
    if (cd >= p.Cd) break;
    const size_t o = ((size_t)(img * p.Cd + cd) * p.Hd + y) * p.Wd + x0;
    const float bias = p.bias ? __ldg(p.bias + cd) : 0.0f;
    float v[PX];
#pragma unroll
    for (int i = 0; i < PX; ++i) v[i] = p.bias ? __fadd_rn(out[c][i], bias) : out[c][i];
    if (p.vec) {
      if (p.pre) *reinterpret_cast<float4*>(p.pre + o) = make_float4(v[0], v[1], v[2], v[3]);
      if (p.relu) {
#pragma unroll
        for (int i = 0; i < PX; ++i) v[i] = v[i] < 0.0f ? 0.0f : v[i];
      }
      *reinterpret_cast<float4*>(p.dst + o) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int i = 0; i < PX; ++i)
        if (x0 + i < p.Wd) {
          if (p.pre) p.pre[o + i] = v[i];
          p.dst[o + i] = p.relu && v[i] < 0.0f ? 0.0f : v[i];
        }
    }
  }
}

// Lanes run over pixels; a warp keeps OT output channels x one input channel x K*K taps, and its lanes' sums are
// folded by halving (each step sends half of the values, so 32 lanes cost about as many shuffles as there are
// values).  The eight warps of a CTA share its pixels, and the CTAs of blockIdx.x share all of them.
template <int K, int OT>
__global__ void __launch_bounds__(kThreads) wgrad_direct_kernel(const float* __restrict__ g, const float* __restrict__ x,
                                                                int C, int H, int W, int O, int Ho, int Wo, int ph,
                                                                int pw, int sh, int sw, int pixels, int per_cta,
                                                                float* __restrict__ partial) {
  constexpr int KK = K * K, N = OT * KK, NP = (N + 31) / 32 * 32;
  __shared__ float fold[kThreads / 32][NP];
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched early: the kernel in front is done from here on
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.y, o0 = blockIdx.z * OT, P = Ho * Wo;
  const int p0 = blockIdx.x * per_cta, p1 = pixels - p0 < per_cta ? pixels : p0 + per_cta;
  float acc[NP];
#pragma unroll
  for (int i = 0; i < NP; ++i) acc[i] = 0.0f;
  int p = p0 + threadIdx.x;
  int b = p / P, r = p - b * P, py = r / Wo, px = r - py * Wo;
  const int step_y = kThreads / Wo, step_x = kThreads - step_y * Wo;
  const int last_o = O - 1 - o0;
  for (; p < p1; p += kThreads) {
    const float* gp = g + ((size_t)b * O + o0) * P + py * Wo + px;
    const int iy = py * sh - ph, ix = px * sw - pw;
    const float* xp = x + ((ptrdiff_t)((size_t)b * C + c) * H + iy) * W + ix;
    float gv[OT], xv[KK];
#pragma unroll
    for (int o = 0; o < OT; ++o) gv[o] = __ldg(gp + (size_t)min(o, last_o) * P);  // past the last: not written
#pragma unroll
    for (int a = 0; a < K; ++a)
#pragma unroll
      for (int t = 0; t < K; ++t)
        xv[a * K + t] = iy + a >= 0 && iy + a < H && ix + t >= 0 && ix + t < W ? __ldg(xp + a * W + t) : 0.0f;
#pragma unroll
    for (int o = 0; o < OT; ++o)
#pragma unroll
      for (int t = 0; t < KK; ++t) acc[o * KK + t] = __fmaf_rn(gv[o], xv[t], acc[o * KK + t]);
    px += step_x;
    py += step_y;
    if (px >= Wo) {
      px -= Wo;
      ++py;
    }
    while (py >= Ho) {
      py -= Ho;
      ++b;
    }
  }
  // fold the lanes: after the step over lane bit m, a lane keeps the upper or the lower half of its values
  int idx = 0;
#pragma unroll
  for (int m = 16, n = NP; m >= 1; m >>= 1) {
    n >>= 1;
    const bool up = lane & m;
    idx += up ? n : 0;
#pragma unroll
    for (int i = 0; i < NP / 2; ++i) {
      if (i >= n) break;
      const float send = up ? acc[i] : acc[i + n], keep = up ? acc[i + n] : acc[i];
      acc[i] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, m));
    }
  }
#pragma unroll
  for (int i = 0; i < NP / 32; ++i) fold[warp][idx + i] = acc[i];
  __syncthreads();
  for (int i = threadIdx.x; i < N; i += kThreads) {
    float s = fold[0][i];
#pragma unroll
    for (int w = 1; w < kThreads / 32; ++w) s = __fadd_rn(s, fold[w][i]);
    const int o = i / KK, t = i - o * KK;
    if (o <= last_o) partial[(((size_t)blockIdx.x * O + o0 + o) * C + c) * KK + t] = s;
  }
}

// ---------------------------------------------------------------- host side
inline int mode() {
  static int env = -1;
  if (env < 0) {
    const char* e = getenv("VTLB_CONV_DIRECT");
    env = e ? atoi(e) : 1;
  }
  return env;
}
inline bool window_ok(int kh, int kw) { return kh == kw && (kh == 1 || kh == 3 || kh == 5); }

// Eight channels a thread, or four where eight would leave a third or more of them idle.
inline bool wide(int Cd) { return (Cd + 7) / 8 * 8 * 2 < (Cd + 3) / 4 * 4 * 3; }
inline int tile_rows(int Hd, int Wd) {
  const int th = 64 / ((Wd + PX - 1) / PX);
  return th < 1 ? 1 : th > Hd ? Hd : th;
}
constexpr int kMaxW = 128;        // output columns: a row of pixel groups fits a CTA, and the stage shared memory
constexpr int kMaxTerms = 1600;   // terms of a sum up to which its error stays below the tensor-core kernels'

// The launch of a product: fills in the tiling fields of `p`; returns the bytes of shared memory.
struct Launch {
  long long tiles;   // of rows
  int groups, CT;    // channel groups of CT
  size_t smem;
};
inline Launch plan(vtlb_ctx* ctx, Params& p, int K) {
  const int CT = wide(p.Cd) ? 8 : 4;
  Launch l = {0, (p.Cd + CT - 1) / CT, CT, 0};
  p.W4 = (p.Wd + PX - 1) / PX;
  p.TH = tile_rows(p.Hd, p.Wd);
  p.tiles_y = (p.Hd + p.TH - 1) / p.TH;
  const int PG = p.TH * p.W4;
  l.tiles = (long long)p.B * p.tiles_y;
  p.CG = kThreads / PG < l.groups ? kThreads / PG : l.groups;
  while (p.CG > 1 && l.tiles * ((l.groups + p.CG - 1) / p.CG) < 2 * ctx->sm_count) p.CG = (p.CG + 1) / 2;
  p.pitch = (p.W4 * PX + K - 1 + 3) / 4 * 4;
  // One source channel has to fit the stage.  On a tiny plane a CTA could hold the weights of hundreds of channels
  // (256 groups of 8 on one pixel group); a single group takes 4 KB at most.
  auto channel_bytes = [&] { return ((p.TH + K - 1) * p.pitch + K * K * p.CG * CT) * 4; };
  while (p.CG > 1 && channel_bytes() > kStageBytes) p.CG = (p.CG + 1) / 2;
  const int per_channel = channel_bytes();
  p.Z = kThreads / (PG * p.CG);
  if (p.Z > p.Cs) p.Z = p.Cs;
  if (p.Z > 8) p.Z = 8;
  p.CS = kStageBytes / per_channel;
  if (p.CS > p.Cs) p.CS = p.Cs;
  if (p.CS > p.Z) p.CS = p.CS / p.Z * p.Z;
  l.smem = (size_t)p.CS * per_channel;
  const size_t park = (size_t)(p.Z - 1) * PG * p.CG * CT * PX * 4;
  if (park > l.smem) l.smem = park;
  return l;
}

// Microseconds.  3 x 3 and 5 x 5: fitted to 116 measured products (forward and input gradient, batches 16 to 256, 1 to 64
// channels, 10 to 32 pixels; mean error 17 %): products padded to whole threads, and the chain of stages.  Of 234 more
// (1 to 1024 images, 1 to 255 channels, 1 to 128 pixels) the rule below sent 2 to the slower kernel, by 16 and 30 %.
// 1 x 1: fitted to 436 products over the wide range (16 %).  A window of one does so little with what it stages that
// staging binds it: products of the threads that are there, the chain of source channels, what a CTA stages in each wave
// of three per SM, and CTAs started.
inline double direct_us(vtlb_ctx* ctx, int B, int Cs, int Cd, int Hd, int Wd, int k) {
  if (k != 1) {
    const int th = tile_rows(Hd, Wd), ct = wide(Cd) ? 8 : 4;
    const double pixels = (double)B * ((Hd + th - 1) / th) * th * ((Wd + PX - 1) / PX) * PX;
    return 5.7 + 0.0356e-6 * 2.0 * pixels * ((Cd + ct - 1) / ct * ct) * Cs * k * k + 0.13 * Cs * k;
  }
  Params p = {};
  p.B = B, p.Cs = Cs, p.Cd = Cd, p.Hd = Hd, p.Wd = Wd;
  const Launch l = plan(ctx, p, 1);
  const double ctas = (double)l.tiles * ((l.groups + p.CG - 1) / p.CG);
  const double products = ctas * p.TH * p.W4 * PX * p.CG * l.CT * Cs, staged = (double)Cs * (p.TH * p.pitch + p.CG * l.CT);
  return 5.27 + 0.0954e-6 * products + 0.0371 * Cs + 0.767e-3 * ceil(ctas / (3 * ctx->sm_count)) * staged +
         0.451 * ctas / ctx->sm_count;
}
// The tensor-core kernels' (7 % mean error, 1 x 1 11 %): waves of tiles of 128 pixels x 64 channels, each walking its K
// blocks of 32; the gathered kernel stores planes of a size that is no multiple of 32 pixels value by value.
inline double tensor_us(vtlb_ctx* ctx, const igemm::Geometry& g, const cslab::Tiling* slab, int Cd) {
  const double blocks_k = (g.K + 31) / 32, cols = (Cd + 63) / 64;
  const double tiles = cols * (slab ? (double)g.B * slab->tiles_per_img
                                    : (double)(((long long)g.B * g.Ho * g.Wo + 127) / 128));
  const double waves = ceil(tiles / ctx->sm_count), ragged = g.Ho * g.Wo % 32 ? Cd * tiles / ctx->sm_count : 0.0;
  if (slab) return 8.6 + waves * (2.8 + 0.273 * blocks_k);
  if (g.kh == 1) return 6.9 + waves * (3.57 + 0.922 * blocks_k) + 0.0272 * ragged;
  return 9.8 + waves * (1.94 + 0.763 * blocks_k) + 0.126 * ragged;
}
// Of the 436 products with a 1 x 1 window 323 run here, 10 of them slower than on tensor cores, by 42 % at most; the sum of
// all is 10.3 ms, 28.4 on tensor cores alone, 10.1 with the better kernel each time.  With the 3 x 3 estimates it was
// 11.6: they sent 50 x 104 x 18 x 18 -> 214 here (137 us, 42 on tensor cores).
// At 256 x 3 x 32 x 32, 32 channels, 3 x 3: forward 24 us (40 on tensor cores), input gradient 55 (103); with 32 -> 64
// channels 342 and 327 (106 and 190), which stay where they are.
inline bool worthwhile(vtlb_ctx* ctx, const igemm::Geometry& g, const cslab::Tiling* slab, int Cd) {
  if (!mode() || !window_ok(g.kh, g.kw) || g.sy != 1 || g.sx != 1 || g.Wo > kMaxW || g.K > kMaxTerms ||
      (Cd + 3) / 4 > 65535)
    return false;
  return mode() == 2 ||
         (g.kh == 1 ? 1.2 : 1.1) * direct_us(ctx, g.B, g.Cs, Cd, g.Ho, g.Wo, g.kh) < tensor_us(ctx, g, slab, Cd);
}
// The weight gradient, likewise: rows of one image per SM on the tensor cores where that kernel applies
// (cwgrad::usable), else the lowered product, bound by the patch matrix it writes.
// At 256 x 3 x 32 x 32, 32 channels, 3 x 3: 50 us (114); 50 x 20 x 12 x 12, 50 channels, 5 x 5: 26 us (33).
inline bool wgrad_worthwhile(vtlb_ctx* ctx, int B, int C, int O, int Ho, int Wo, int kh, int kw, bool pixel_kernel) {
  const double pixels = (double)B * Ho * Wo;
  if (!mode() || !window_ok(kh, kw) || C > 65535 || O > 65535 || pixels > 1e9) return false;
  const int ot = kh == 1 ? 16 : kh == 3 ? 8 : 4;
  const double rate = kh == 1 ? 3.5e6 : kh == 3 ? 12e6 : 10e6;  // products twice, per microsecond
  const double direct = 7.0 + 2.0 * pixels * ((O + ot - 1) / ot * ot) * C * kh * kw / rate;
  const double tensor = pixel_kernel ? 15.0 + 1.75 * B * Ho * ((C + 31) / 32) * ((O + 63) / 64) / ctx->sm_count
                                     : 24.0 + 4.73e-6 * pixels * C * kh * kw;
  return mode() == 2 || 1.1 * direct < tensor;
}

template <int K>
int launch_direct_k(vtlb_ctx* ctx, Params p) {
  const Launch l = plan(ctx, p, K);
  p.vec = p.Wd % 4 == 0 && vtlb_aligned16(p.dst) && (!p.pre || vtlb_aligned16(p.pre));
  const dim3 grid((unsigned)l.tiles, (l.groups + p.CG - 1) / p.CG);
  VTLB_CUDA(ctx, vtlb_launch_early(l.CT == 8 ? conv_direct_kernel<K, 8> : conv_direct_kernel<K, 4>, grid, dim3(kThreads),
                                   l.smem, ctx->stream, p));
  VTLB_LAUNCHED(ctx);
  return VTLB_OK;
}
inline int launch_direct(vtlb_ctx* ctx, const Params& p, int K) {
  return K == 1 ? launch_direct_k<1>(ctx, p) : K == 3 ? launch_direct_k<3>(ctx, p) : launch_direct_k<5>(ctx, p);
}

template <int K, int OT>
int launch_wgrad_t(vtlb_ctx* ctx, const float* g, const float* x, float* dW, int B, int C, int H, int W, int O, int Ho,
                   int Wo, int ph, int pw, int sh, int sw) {
  const int og = (O + OT - 1) / OT, pixels = B * Ho * Wo;
  // CTAs for four waves of two per SM, each with at least eight steps of its lanes
  int parts = (8 * ctx->sm_count + og * C - 1) / (og * C);
  const int most = (pixels + 8 * kThreads - 1) / (8 * kThreads);
  if (parts > most) parts = most;
  const int per = (int)vtlb_round_up((pixels + parts - 1) / parts, kThreads);
  parts = (pixels + per - 1) / per;
  const size_t n = (size_t)O * C * K * K;
  void* scr = nullptr;
  if (int rc = vtlb_scratch(ctx, (size_t)parts * n * sizeof(float), &scr)) return rc;
  // a dW over x or g is written when both have been read, as by the kernels that this one stands in for
  const bool by_scratch = parts > 1 || vtlb_overlap(dW, n, x, (size_t)B * C * H * W) || vtlb_overlap(dW, n, g, (size_t)B * O * Ho * Wo);
  VTLB_CUDA(ctx, vtlb_launch_early(wgrad_direct_kernel<K, OT>, dim3(parts, C, og), dim3(kThreads), 0, ctx->stream, g, x, C,
                                   H, W, O, Ho, Wo, ph, pw, sh, sw, pixels, per, by_scratch ? (float*)scr : dW));
  VTLB_LAUNCHED(ctx);
  return by_scratch ? f32::reduce_splits(ctx, (const float*)scr, parts, n, dW) : VTLB_OK;
}
inline int launch_wgrad(vtlb_ctx* ctx, const float* g, const float* x, float* dW, int B, int C, int H, int W, int O,
                        int Ho, int Wo, int K, int ph, int pw, int sh, int sw) {
  if (K == 1) return launch_wgrad_t<1, 16>(ctx, g, x, dW, B, C, H, W, O, Ho, Wo, ph, pw, sh, sw);
  if (K == 3) return launch_wgrad_t<3, 8>(ctx, g, x, dW, B, C, H, W, O, Ho, Wo, ph, pw, sh, sw);
  return launch_wgrad_t<5, 4>(ctx, g, x, dW, B, C, H, W, O, Ho, Wo, ph, pw, sh, sw);
}

}  // namespace cdirect
