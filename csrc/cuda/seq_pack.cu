// Moving the real tokens of a padded [B, L] batch into packed rows and back, for the jagged attention kernels.
//
//   src[r]  = token of packed row r (-1 behind the last real token)
//   dest[t] = packed row of token t (-1 for padding)
//
// Everything here is bound by memory.  One gather serves both directions (rows without a source are zeroed in the same
// pass), and q | k | v travel as one row of 3 D columns.  The SASRec step at [512, 200], 256 columns (half of the tokens
// real), two layers: training 9.9 -> 6.9 ms, evaluation 4.10 -> 2.16 ms on a B200, against one zero-filled index_copy
// per operand and its index_add / gather backward.
#include "common.cuh"

namespace recml {
namespace pack {

constexpr int kWarps = 8;

__global__ void __launch_bounds__(256) count_kernel(const unsigned char* __restrict__ mask, int B, int L, int* __restrict__ counts) {
  const int b = blockIdx.x * kWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (b >= B) return;
  const unsigned char* row = mask + static_cast<long long>(b) * L;
  int n = 0;
  for (int i = lane; i < L; i += 32) n += row[i] != 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  if (lane == 0) counts[b] = n;
}

// A block's eight warps take one sample each; the block adds up the counts before its first sample itself, so no scan
// kernel stands between the two.  Rows of `src` behind the last real token are filled by the whole grid.
__global__ void __launch_bounds__(256) index_kernel(const unsigned char* __restrict__ mask, const int* __restrict__ counts, int B,
                                                    int L, int* __restrict__ offsets, int* __restrict__ src,
                                                    int* __restrict__ dest) {
  __shared__ int part[2][kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b0 = blockIdx.x * kWarps;
  int before = 0, rest = 0;                       // real tokens of samples [0, b0) and [b0, B)
  for (int i = threadIdx.x; i < B; i += 256) { const int c = counts[i]; if (i < b0) before += c; else rest += c; }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    before += __shfl_xor_sync(0xffffffffu, before, o);
    rest += __shfl_xor_sync(0xffffffffu, rest, o);
  }
  if (lane == 0) { part[0][warp] = before; part[1][warp] = rest; }
  __syncthreads();
  int base = 0, total = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) { base += part[0][w]; total += part[0][w] + part[1][w]; }
  const int b = b0 + warp;
  for (int i = b0; i < min(b, B); ++i) base += counts[i];
  if (b < B) {
    if (lane == 0) offsets[b] = base;
    const unsigned char* row = mask + static_cast<long long>(b) * L;
    for (int i0 = 0; i0 < L; i0 += 32) {
      const int i = i0 + lane;
      const bool on = i < L && row[i] != 0;
      const unsigned int m = __ballot_sync(0xffffffffu, on);
      const int t = b * L + i;
      const int r = base + __popc(m & ((1u << lane) - 1));
      if (i < L) dest[t] = on ? r : -1;
      if (on) src[r] = t;
      base += __popc(m);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) offsets[B] = total;
  for (long long r = total + blockIdx.x * 256LL + threadIdx.x; r < static_cast<long long>(B) * L; r += gridDim.x * 256LL) src[r] = -1;
}

// out[r, :] = idx[r] >= 0 ? in[idx[r], :] : 0 for rows of 16-byte chunks; a thread takes four chunks of a block's 1024.
// I: the type that holds a chunk's number (a 32-bit division by the row length is far cheaper than a 64-bit one).
template <typename I>
__global__ void __launch_bounds__(256) gather_kernel(const uint4* __restrict__ in, unsigned int ld_in, const int* __restrict__ idx,
                                                     uint4* __restrict__ out, unsigned int chunks, I total) {
  const I i0 = static_cast<I>(blockIdx.x) * 1024 + threadIdx.x;
  uint4 v[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const I i = i0 + u * 256;
    v[u] = make_uint4(0, 0, 0, 0);
    if (i < total) {
      const I r = i / chunks;
      const int s = __ldg(idx + r);
      if (s >= 0) v[u] = __ldg(in + static_cast<long long>(s) * ld_in + (i - r * chunks));
    }
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const I i = i0 + u * 256;
    if (i < total) out[i] = v[u];
  }
}

// out[t, :] = (dq | dk | dv)[dest[t], :] in bf16 (zeros for padding); dq is fp32, `dest` null means row t itself.
template <typename I>
__global__ void __launch_bounds__(256) gather_qkv_grad_kernel(const float* __restrict__ dq, const __nv_bfloat16* __restrict__ dk,
                                                              const __nv_bfloat16* __restrict__ dv, const int* __restrict__ dest,
                                                              uint4* __restrict__ out, int D, I total) {
  const I i0 = static_cast<I>(blockIdx.x) * 512 + threadIdx.x;
  const unsigned int chunks = 3u * D / 8;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const I i = i0 + u * 256;
    if (i >= total) return;
    const I t = i / chunks;
    const int c = static_cast<int>(i - t * chunks) * 8;
    const long long s = dest != nullptr ? __ldg(dest + t) : static_cast<long long>(t);
    uint4 v = make_uint4(0, 0, 0, 0);
    if (s >= 0) {
      if (c < D) {
        const float4* p = reinterpret_cast<const float4*>(dq + s * D + c);
        const float4 a = __ldg(p), b = __ldg(p + 1);
        v = make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
      } else {
        v = __ldg(reinterpret_cast<const uint4*>(c < 2 * D ? dk + s * D + (c - D) : dv + s * D + (c - 2 * D)));
      }
    }
    out[i] = v;
  }
}

// out[t, h] = sum_d a[t, h, d] * b[t, h, d] (fp32 products and sums); LPH lanes of eight columns per head.
template <int LPH>
__global__ void __launch_bounds__(256) head_dot_kernel(const __nv_bfloat16* __restrict__ a, long long lda,
                                                       const __nv_bfloat16* __restrict__ b, long long ldb, int H,
                                                       float* __restrict__ out, long long items) {
  const long long i = blockIdx.x * 256LL + threadIdx.x;          // (t, h, lane)
  const long long th = i / LPH;
  const int l = static_cast<int>(i % LPH);
  float s = 0.f;
  if (th < items) {
    const long long t = th / H;
    const int c = static_cast<int>(th - t * H) * (LPH * 8) + l * 8;
    const uint4 x = __ldg(reinterpret_cast<const uint4*>(a + t * lda + c)), y = __ldg(reinterpret_cast<const uint4*>(b + t * ldb + c));
    const uint32_t xw[4] = {x.x, x.y, x.z, x.w}, yw[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) s = fmaf(bf16_hi(xw[j]), bf16_hi(yw[j]), fmaf(bf16_lo(xw[j]), bf16_lo(yw[j]), s));
  }
#pragma unroll
  for (int o = LPH / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (l == 0 && th < items) out[th] = s;
}

static bool off16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; }

}  // namespace pack
}  // namespace recml

using namespace recml::pack;

// mask: [B, L] bytes; counts [B], offsets [B + 1], src / dest [B * L] int32.
extern "C" int recml_pack_index(const void* mask, int B, int L, int* counts, int* offsets, int* src, int* dest, cudaStream_t stream) {
  if (B <= 0 || L <= 0) return 0;
  if (static_cast<long long>(B) * L > 0x7fffffffLL) return -10;
  const int blocks = (B + kWarps - 1) / kWarps;
  count_kernel<<<blocks, 256, 0, stream>>>(static_cast<const unsigned char*>(mask), B, L, counts);
  index_kernel<<<blocks, 256, 0, stream>>>(static_cast<const unsigned char*>(mask), counts, B, L, offsets, src, dest);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// Rows of `width` bf16 columns, width and ld_in multiples of 8, 16-byte aligned bases.
extern "C" int recml_gather_rows(const void* in, long long ld_in, const int* idx, void* out, long long rows, int width,
                                 cudaStream_t stream) {
  if (rows <= 0 || width <= 0) return 0;
  if (width % 8 || ld_in % 8 || ld_in / 8 > 0xffffffffLL || off16(in) || off16(out)) return -10;
  const long long total = rows * (width / 8);
  const unsigned blocks = static_cast<unsigned>((total + 1023) / 1024);
  const uint4* i4 = static_cast<const uint4*>(in);
  uint4* o4 = static_cast<uint4*>(out);
  if (total < (1LL << 31)) gather_kernel<unsigned int><<<blocks, 256, 0, stream>>>(i4, ld_in / 8, idx, o4, width / 8, total);
  else gather_kernel<long long><<<blocks, 256, 0, stream>>>(i4, ld_in / 8, idx, o4, width / 8, total);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// out [rows, 3 D] bf16 contiguous; dq fp32, dk / dv bf16, all [*, D] contiguous.
extern "C" int recml_gather_qkv_grad(const float* dq, const void* dk, const void* dv, const int* dest, void* out, long long rows,
                                     int D, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (D % 8 || off16(dq) || off16(dk) || off16(dv) || off16(out)) return -10;
  const long long total = rows * (3LL * D / 8);
  const unsigned blocks = static_cast<unsigned>((total + 511) / 512);
  const __nv_bfloat16 *k = static_cast<const __nv_bfloat16*>(dk), *v = static_cast<const __nv_bfloat16*>(dv);
  uint4* o4 = static_cast<uint4*>(out);
  if (total < (1LL << 31)) gather_qkv_grad_kernel<unsigned int><<<blocks, 256, 0, stream>>>(dq, k, v, dest, o4, D, total);
  else gather_qkv_grad_kernel<long long><<<blocks, 256, 0, stream>>>(dq, k, v, dest, o4, D, total);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// a, b: [T, H, Dh] bf16 with row pitches lda / ldb (multiples of 8), Dh 64 or 128; out [T, H] fp32.
extern "C" int recml_head_dot(const void* a, long long lda, const void* b, long long ldb, long long T, int H, int Dh, float* out,
                              cudaStream_t stream) {
  if (T <= 0 || H <= 0) return 0;
  if ((Dh != 64 && Dh != 128) || lda % 8 || ldb % 8 || off16(a) || off16(b)) return -10;
  using bf = __nv_bfloat16;
  const long long items = T * H;
  const unsigned blocks = static_cast<unsigned>((items * (Dh / 8) + 255) / 256);
  if (Dh == 64) head_dot_kernel<8><<<blocks, 256, 0, stream>>>(static_cast<const bf*>(a), lda, static_cast<const bf*>(b), ldb, H, out, items);
  else head_dot_kernel<16><<<blocks, 256, 0, stream>>>(static_cast<const bf*>(a), lda, static_cast<const bf*>(b), ldb, H, out, items);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
