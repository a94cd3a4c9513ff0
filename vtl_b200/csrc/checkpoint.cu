// Checkpoint tensor payloads on the device.  The reference stores every tensor as text:
// each element widened to f64, its 8 bytes most significant first, the byte string in
// standard base64 with '=' padding (encode_tensor / decode_tensor,
// nn/models/serialization.v:421-473).  Encoding and decoding 134 M parameters this way is
// 0.5 GB in and 1.4 GB out of pure byte shuffling, bound by HBM: it runs here, next to the
// parameters, and only the text crosses PCIe.
//
// Work split: 3 elements = 24 bytes = 32 base64 characters per thread, so every thread writes
// (reads, when decoding) two aligned 16-byte pieces of text and no base64 group straddles two
// threads.  Only the last thread sees a short group and the padding.
#include "common.cuh"

namespace {

__host__ __device__ inline size_t b64_len(size_t n) { return (n * 8 + 2) / 3 * 4; }

// Four 6-bit values, one per byte -> their four characters of the standard alphabet, all bytes at
// once.  (v + 128 - k) has bit 7 set exactly when v >= k, so the range tests cost one add each;
// 'A'+v for v < 26, 'a'+v-26 (= v+71) below 52, '0'+v-52 (= v-4) below 62, then '+' and '/'.
// No byte ever carries or borrows: v + 65 + 6 <= 134, and what is subtracted never exceeds it.
__device__ __forceinline__ uint32_t b64_chars4(uint32_t v4) {
  const uint32_t ge26 = ((v4 + 0x66666666u) >> 7) & 0x01010101u;
  const uint32_t ge52 = ((v4 + 0x4c4c4c4cu) >> 7) & 0x01010101u;
  const uint32_t ge62 = ((v4 + 0x42424242u) >> 7) & 0x01010101u;
  const uint32_t ge63 = ((v4 + 0x41414141u) >> 7) & 0x01010101u;
  return (v4 + 0x41414141u + ge26 * 6u) - (ge52 * 75u + ge62 * 15u - ge63 * 3u);
}
// Byte i of the result = byte sel_i (0..7) of the table {hi, lo}, four look-ups in one instruction.
__device__ __forceinline__ uint32_t lookup4(uint32_t lo, uint32_t hi, uint32_t sel) { return __byte_perm(lo, hi, sel); }

// Four characters, one per byte -> their four 6-bit values, all bytes at once; *bad gets a bit of 0x9b in the byte
// of a character outside the alphabet.  The high digit of a character (its bits 4..6) picks, by one byte permutation
// each for all four:
//   off   what turns the character into its value modulo 64: digits +4, 'A'..'Z' -65 = +63, 'a'..'z' -71 = +57,
//         '+' +19 (and '/' three less); the sum stays below 256, so no byte carries into the next
//   low   what carries the low digit into bit 4 when it is not one of the alphabet under that high digit: 2x takes
//         11..15, 3x 0..9, 4x and 6x 1..15, 5x and 7x 0..10, 0x and 1x none
//   both  bits that have to be set: 2x only has '+' (2b) and '/' (2f), which leaves out 2c..2e
// Testing each of the five ranges of the alphabet took twice the instructions, and they bound the decoder.
__device__ __forceinline__ uint32_t b64_vals4(uint32_t c4, uint32_t* bad) {
  const uint32_t digit = (c4 >> 4) & 0x07070707u;
  const uint32_t two = digit | (digit >> 4);           // nibbles 0, 1 in byte 0 and 2, 3 in byte 2
  const uint32_t sel = __byte_perm(two, 0u, 0x4420u);  // one selector nibble per character
  const uint32_t off = lookup4(0x04130000u, 0x39393f3fu, sel);
  const uint32_t low = lookup4(0x06151010u, 0x051f051fu, sel);
  const uint32_t both = lookup4(0x00030000u, 0x00000000u, sel);
  *bad |= (((c4 & 0x0f0f0f0fu) + low) & 0x10101010u) | (~c4 & both) | (c4 & 0x80808080u);
  const uint32_t slash = (c4 >> 2) & both & 0x01010101u;  // '/' has bit 2, '+' has not
  return (c4 + off - slash * 3u) & 0x3f3f3f3fu;
}
// Four 6-bit values, the first in the low byte -> 24 bits, the first on top.
__device__ __forceinline__ uint32_t b64_bits24(uint32_t v4) {
  const uint32_t top = __dp4a(v4, 0x00000140u, 0u);  // v0 * 64 + v1
  return __dp4a(v4, 0x01400000u, top << 12);         // ... + v2 * 64 + v3
}
// Eight such groups -> three f64, most significant byte first.
__device__ __forceinline__ void b64_doubles(const uint32_t (&t)[8], double (&out)[3]) {
  // 24-bit pieces abc, def, ghi, ... : word 0 = abcd, word 1 = efgh, word 2 = ijkl and so on
  out[0] = __hiloint2double((int)__byte_perm(t[0], t[1], 0x2106u), (int)__byte_perm(t[1], t[2], 0x1065u));
  out[1] = __hiloint2double((int)__byte_perm(t[2], t[3], 0x0654u), (int)__byte_perm(t[4], t[5], 0x2106u));
  out[2] = __hiloint2double((int)__byte_perm(t[5], t[6], 0x1065u), (int)__byte_perm(t[6], t[7], 0x0654u));
}

// The 32 characters of three f64 bit patterns (most significant byte first), packed four to a word
// in memory order (first character in the low byte).
__device__ __forceinline__ void encode3(const unsigned long long (&bits)[3], uint32_t (&out)[8]) {
  // the 192 bits as six 32-bit words, big-endian order
  const uint32_t w[6] = {(uint32_t)(bits[0] >> 32), (uint32_t)bits[0], (uint32_t)(bits[1] >> 32),
                         (uint32_t)bits[1],         (uint32_t)(bits[2] >> 32), (uint32_t)bits[2]};
#pragma unroll
  for (int g = 0; g < 8; ++g) {  // characters 4g .. 4g+3 = bits 24g .. 24g+23
    const int bit0 = 24 * g, wi = bit0 >> 5, sh = bit0 & 31;
    // 24 bits starting at bit `sh` of word wi (bit 0 = most significant)
    const unsigned long long two = ((unsigned long long)w[wi] << 32) | (wi + 1 < 6 ? w[wi + 1] : 0u);
    const uint32_t t = (uint32_t)(two >> (40 - sh)) & 0xffffffu;
    out[g] = b64_chars4((t >> 18) | (((t >> 12) & 63u) << 8) | (((t >> 6) & 63u) << 16) | ((t & 63u) << 24));
  }
}

__global__ void __launch_bounds__(256) ckpt_encode_kernel(const float* __restrict__ src, size_t n,
                                                          unsigned char* __restrict__ out) {
  const size_t groups = (n + 2) / 3;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < groups;
       t += (size_t)gridDim.x * blockDim.x) {
    const size_t e0 = t * 3;
    const int have = n - e0 >= 3 ? 3 : (int)(n - e0);
    unsigned long long bits[3] = {0ull, 0ull, 0ull};
#pragma unroll
    for (int j = 0; j < 3; ++j)
      if (j < have) bits[j] = (unsigned long long)__double_as_longlong((double)src[e0 + j]);
    uint32_t ch[8];
    encode3(bits, ch);
    unsigned char* dst = out + t * 32;
    if (have == 3) {
      reinterpret_cast<uint4*>(dst)[0] = make_uint4(ch[0], ch[1], ch[2], ch[3]);
      reinterpret_cast<uint4*>(dst)[1] = make_uint4(ch[4], ch[5], ch[6], ch[7]);
    } else {
      // 8 bytes -> 11 characters + "=", 16 bytes -> 22 characters + "=="
      const int nchar = have == 1 ? 11 : 22, total = have == 1 ? 12 : 24;
      for (int i = 0; i < total; ++i)
        dst[i] = i < nchar ? (unsigned char)(ch[i >> 2] >> (8 * (i & 3))) : (unsigned char)'=';
    }
  }
}

// flags: bit 0 = a character outside the alphabet, bit 1 = malformed padding
// A warp's 96 values leave through shared memory: a lane writing its three next to one another makes three
// partial writes of every 32-byte sector.  16.8 M values: 95 us before, 83 us with the look-ups and this, 66 us with the
// bits put together by dp4a and byte permutations (246 MB, 37 us at the measured copy rate; integer issue bounds it).
__global__ void __launch_bounds__(256) ckpt_decode_kernel(const unsigned char* __restrict__ text, size_t n,
                                                          float* __restrict__ dst, uint32_t* __restrict__ flags) {
  __shared__ float turn[8][96];
  const size_t groups = (n + 2) / 3;
  const int lane = threadIdx.x & 31;
  float* mine = turn[threadIdx.x >> 5];
  for (size_t t0 = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) / 32 * 32; t0 < groups;
       t0 += (size_t)gridDim.x * blockDim.x) {
    const size_t t = t0 + lane, e0 = t * 3;
    const int have = e0 >= n ? 0 : n - e0 >= 3 ? 3 : (int)(n - e0);
    const unsigned char* srcp = text + t * 32;
    uint32_t bad = 0, t24[8];
    if (have == 3) {
      const uint4 a = reinterpret_cast<const uint4*>(srcp)[0], b = reinterpret_cast<const uint4*>(srcp)[1];
      const uint32_t ch[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
      for (int g = 0; g < 8; ++g) t24[g] = b64_bits24(b64_vals4(ch[g], &bad));
    } else {  // the last group of a text, or none: 'A' (value 0) where there is no character
      const int nchar = have == 0 ? 0 : have == 1 ? 11 : 22, total = have == 0 ? 0 : have == 1 ? 12 : 24;
      uint32_t ch[8], pad = 0;  // every character is on its way before the first is looked at
#pragma unroll
      for (int g = 0; g < 8; ++g) {
        ch[g] = 0;
#pragma unroll
        for (int i = 4 * g; i < 4 * g + 4; ++i) {
          const uint32_t c = i < total ? srcp[i] : '=';
          if (i >= nchar) pad |= c ^ '=';
          ch[g] |= (i < nchar ? c : 'A') << (8 * (i & 3));
        }
      }
#pragma unroll
      for (int g = 0; g < 8; ++g) t24[g] = b64_bits24(b64_vals4(ch[g], &bad));
      if (pad) atomicOr(flags, 2u);
    }
    double v[3];
    b64_doubles(t24, v);
    if (bad) atomicOr(flags, 1u);
    __syncwarp();  // the previous round's values have been read
#pragma unroll
    for (int j = 0; j < 3; ++j)
      mine[lane * 3 + j] = (float)v[j];  // vtl.cast[T]: plain conversion
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 3; ++j)
      if (t0 * 3 + j * 32 + lane < n) dst[t0 * 3 + j * 32 + lane] = mine[j * 32 + lane];
  }
}

int ckpt_grid(vtlb_ctx* ctx, size_t groups) {
  size_t b = (groups + 255) / 256;
  const size_t cap = (size_t)ctx->sm_count * 16;
  if (b > cap) b = cap;
  return b < 1 ? 1 : (int)b;
}

}  // namespace

VTLB_API size_t vtlb_ckpt_text_len(size_t n) { return b64_len(n); }

VTLB_API int vtlb_ckpt_encode_f32(vtlb_ctx* ctx, const void* d_src, size_t n, void* d_text) {
  VTLB_ENTER(ctx);
  if (n == 0) return VTLB_OK;
  if (!d_src || !d_text) return vtlb_fail(ctx, VTLB_EINVAL, "vtlb_ckpt_encode_f32: null pointer");
  if (!vtlb_aligned16(d_text)) return vtlb_fail(ctx, VTLB_EINVAL, "vtlb_ckpt_encode_f32: text buffer not 16-byte aligned");
  ckpt_encode_kernel<<<ckpt_grid(ctx, (n + 2) / 3), 256, 0, ctx->stream>>>((const float*)d_src, n,
                                                                          (unsigned char*)d_text);
  VTLB_LAUNCHED(ctx);
  return VTLB_OK;
}

VTLB_API int vtlb_ckpt_decode_f32(vtlb_ctx* ctx, const void* d_text, size_t text_len, void* d_dst, size_t n) {
  VTLB_ENTER(ctx);
  if (text_len != b64_len(n))
    return vtlb_fail(ctx, VTLB_EINVAL, "vtlb_ckpt_decode_f32: %zu characters cannot hold %zu values (%zu expected)",
                     text_len, n, b64_len(n));
  if (n == 0) return VTLB_OK;
  if (!d_text || !d_dst) return vtlb_fail(ctx, VTLB_EINVAL, "vtlb_ckpt_decode_f32: null pointer");
  if (!vtlb_aligned16(d_text)) return vtlb_fail(ctx, VTLB_EINVAL, "vtlb_ckpt_decode_f32: text buffer not 16-byte aligned");
  void* scr = nullptr;
  int rc = vtlb_scratch(ctx, 256, &scr);
  if (rc) return rc;
  uint32_t* d_flags = (uint32_t*)scr;
  VTLB_CUDA(ctx, cudaMemsetAsync(d_flags, 0, sizeof(uint32_t), ctx->stream));
  ckpt_decode_kernel<<<ckpt_grid(ctx, (n + 2) / 3), 256, 0, ctx->stream>>>((const unsigned char*)d_text, n,
                                                                          (float*)d_dst, d_flags);
  VTLB_LAUNCHED(ctx);
  uint32_t flags = 0;
  VTLB_CUDA(ctx, cudaMemcpyAsync(&flags, d_flags, sizeof(flags), cudaMemcpyDeviceToHost, ctx->stream));
  VTLB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (flags & 1u) return vtlb_fail(ctx, VTLB_EINVAL, "vtlb_ckpt_decode_f32: character outside the base64 alphabet");
  if (flags & 2u) return vtlb_fail(ctx, VTLB_EINVAL, "vtlb_ckpt_decode_f32: malformed base64 padding");
  return VTLB_OK;
}
