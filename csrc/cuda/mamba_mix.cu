// What surrounds the scan of a Mamba2 mixer, forward and backward, in one pass over each activation:
//
//   dt = softplus(dt_raw + dt_bias),  cum = log2(e) * prefix sums of a dt over a sequence,  xs = x dt     (before)
//   y  = rms_norm(v silu(z)) w + b                                                                       (behind)
//
// xbc [T, H P + 2 N] holds x | b | c of a token (bf16); the scan reads b and c where they are.  Everything here is bound
// by memory; the arithmetic is fp32 and each result is rounded to bf16 once.  Two Mamba2 blocks at [256, 200, 256], forward
// and backward: 6.05 -> 3.82 ms on a B200, against casts, splits, products and prefix sums as separate fp32 passes.
#include "common.cuh"

namespace recml {
namespace mix {

constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ float wsum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
__device__ __forceinline__ void unpack8(const uint4& t, float (&v)[8]) {
  const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) { v[2 * j] = bf16_lo(w[j]); v[2 * j + 1] = bf16_hi(w[j]); }
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
  return make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
}
template <typename T> __device__ __forceinline__ float ldf(const T* p);
template <> __device__ __forceinline__ float ldf<float>(const float* p) { return __ldg(p); }
template <> __device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
template <typename T> __device__ __forceinline__ void stf(T* p, float v);
template <> __device__ __forceinline__ void stf<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void stf<__nv_bfloat16>(__nv_bfloat16* p, float v) { *p = __float2bfloat16(v); }

// ---- before the scan ---------------------------------------------------------------------------------------------
// One warp per (sample, head): 32 steps at a time, the carry in a register.  cum is [H, pitch]; its columns from T on
// are zeroed by the warps of the last sample.
template <typename TD>
__global__ void __launch_bounds__(256) dt_scan_kernel(const TD* __restrict__ raw, const float* __restrict__ bias,
                                                      const float* __restrict__ a, int B, int L, int H, float* __restrict__ dt,
                                                      float* __restrict__ cum, long long pitch) {
  const long long wid = (blockIdx.x * 256LL + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const long long T = static_cast<long long>(B) * L;
  if (wid >= static_cast<long long>(B) * H) return;
  const int h = static_cast<int>(wid % H);
  const long long b = wid / H;
  const float ah = __ldg(a + h), bh = __ldg(bias + h);
  float carry = 0.f;
  for (int l0 = 0; l0 < L; l0 += 32) {
    const int l = l0 + lane;
    const long long t = b * L + l;
    float d = 0.f;
    if (l < L) {
      const float u = ldf<TD>(raw + t * H + h) + bh;
      d = u > 20.f ? u : log1pf(expf(u));
      dt[t * H + h] = d;
    }
    float s = ah * d;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float v = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += v;
    }
    s += carry;
    if (l < L) cum[h * pitch + t] = s * kLog2e;
    carry = __shfl_sync(0xffffffffu, s, 31);
  }
  if (b == B - 1)
    for (long long t = T + lane; t < pitch; t += 32) cum[h * pitch + t] = 0.f;
}

// xs[t, h, :] = x[t, h, :] * dt[t, h], eight columns per thread and step.
__global__ void __launch_bounds__(256) scale_kernel(const __nv_bfloat16* __restrict__ xbc, int C, const float* __restrict__ dt,
                                                    int H, int P, __nv_bfloat16* __restrict__ xs, long long T) {
  const unsigned int per_row = static_cast<unsigned int>(H) * P / 8;
  const long long t = blockIdx.x * static_cast<long long>(blockDim.y) + threadIdx.y;
  if (t >= T) return;
  for (unsigned int c = threadIdx.x; c < per_row; c += blockDim.x) {
    float v[8];
    unpack8(__ldg(reinterpret_cast<const uint4*>(xbc + t * C + c * 8)), v);
    const float d = __ldg(dt + t * H + c * 8 / P);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] *= d;
    *reinterpret_cast<uint4*>(xs + t * H * P + c * 8) = pack8(v);
  }
}

// ---- and its backward --------------------------------------------------------------------------------------------
// dxbc = (dxs dt | db | dc) in bf16 and dots[t, h] = dxs . x; P / 8 neighbouring lanes share a head.
template <int LPH>
__global__ void __launch_bounds__(256) scale_bwd_kernel(const __nv_bfloat16* __restrict__ dxs, const __nv_bfloat16* __restrict__ xbc,
                                                        const float* __restrict__ dt, const float* __restrict__ db,
                                                        const float* __restrict__ dc, int H, __nv_bfloat16* __restrict__ dxbc,
                                                        float* __restrict__ dots, long long T) {
  constexpr int P = LPH * 8;                       // = N, the state size
  const int per_row = (H + 2) * LPH, C = (H + 2) * P;
  const long long i = blockIdx.x * 256LL + threadIdx.x;
  const long long t = i / per_row;
  const int k = static_cast<int>(i - t * per_row), h = k / LPH;
  const bool on = t < T;
  float s = 0.f;
  if (on) {
    float o[8];
    if (h < H) {
      float x[8];
      unpack8(__ldg(reinterpret_cast<const uint4*>(dxs + t * H * P + k * 8)), o);
      unpack8(__ldg(reinterpret_cast<const uint4*>(xbc + t * C + k * 8)), x);
      const float d = __ldg(dt + t * H + h);
#pragma unroll
      for (int j = 0; j < 8; ++j) { s = fmaf(o[j], x[j], s); o[j] *= d; }
    } else {
      const float4* g = reinterpret_cast<const float4*>((h == H ? db : dc) + t * P + (k - h * LPH) * 8);
      const float4 u = __ldg(g), v = __ldg(g + 1);
      o[0] = u.x; o[1] = u.y; o[2] = u.z; o[3] = u.w; o[4] = v.x; o[5] = v.y; o[6] = v.z; o[7] = v.w;
    }
    *reinterpret_cast<uint4*>(dxbc + t * C + k * 8) = pack8(o);
  }
#pragma unroll
  for (int o = LPH / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (on && h < H && k % LPH == 0) dots[t * H + h] = s;
}

// One warp per (sample, head), from the end of the sequence: da = suffix sums of dcum, ddt = a da + dots; the gradient of
// the raw step sizes, and the sums for a and dt_bias (pre-zeroed, one atomic per warp).
template <typename TD>
__global__ void __launch_bounds__(256) dt_scan_bwd_kernel(const float* __restrict__ dcum, long long pitch,
                                                          const float* __restrict__ dots, const float* __restrict__ dt,
                                                          const TD* __restrict__ raw, const float* __restrict__ bias,
                                                          const float* __restrict__ a, int B, int L, int H, TD* __restrict__ draw,
                                                          float* __restrict__ da_sum, float* __restrict__ dbias_sum) {
  const long long wid = (blockIdx.x * 256LL + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= static_cast<long long>(B) * H) return;
  const int h = static_cast<int>(wid % H);
  const long long b = wid / H;
  const float ah = __ldg(a + h), bh = __ldg(bias + h);
  float carry = 0.f, sa = 0.f, sb = 0.f;
  for (int l0 = (L - 1) / 32 * 32; l0 >= 0; l0 -= 32) {
    const int l = l0 + lane;
    const long long t = b * L + l;
    float s = l < L ? __ldg(dcum + h * pitch + t) : 0.f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float v = __shfl_down_sync(0xffffffffu, s, o);
      if (lane + o < 32) s += v;
    }
    s += carry;
    carry = __shfl_sync(0xffffffffu, s, 0);
    if (l < L) {
      const float u = ldf<TD>(raw + t * H + h) + bh;
      const float sig = u > 20.f ? 1.f : 1.f / (1.f + expf(-u));
      const float g = fmaf(ah, s, __ldg(dots + t * H + h)) * sig;
      stf<TD>(draw + t * H + h, g);
      sa = fmaf(s, __ldg(dt + t * H + h), sa);
      sb += g;
    }
  }
  sa = wsum(sa); sb = wsum(sb);
  if (lane == 0) { atomicAdd(da_sum + h, sa); atomicAdd(dbias_sum + h, sb); }
}

// ---- behind the scan: rms_norm(v silu(z)) w + b ------------------------------------------------------------------
// A warp holds whole rows in registers, lane l columns [c * 256 + 8 l, + 8) of chunk c; the gated value is rounded to
// bf16 first (what the norm sees), so the backward recomputes it from v and z and nothing else is kept but 1 / rms.
template <int NCH>
__global__ void __launch_bounds__(256) gated_rms_fwd_kernel(const __nv_bfloat16* __restrict__ v, const __nv_bfloat16* __restrict__ z,
                                                            const float* __restrict__ w, const float* __restrict__ bias,
                                                            __nv_bfloat16* __restrict__ y, float* __restrict__ rstd_out, long long M,
                                                            int D, float eps) {
  const long long row = (blockIdx.x * 256LL + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= M) return;
  float g[NCH][8];
  float ss = 0.f;
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int col = c * 256 + lane * 8;
    if (col < D) {
      float a[8], b[8];
      unpack8(__ldg(reinterpret_cast<const uint4*>(v + row * D + col)), a);
      unpack8(__ldg(reinterpret_cast<const uint4*>(z + row * D + col)), b);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        g[c][j] = __bfloat162float(__float2bfloat16(a[j] * (b[j] / (1.f + __expf(-b[j])))));
        ss = fmaf(g[c][j], g[c][j], ss);
      }
    }
  }
  const float rstd = rsqrtf(wsum(ss) / D + eps);
  if (lane == 0) rstd_out[row] = rstd;
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int col = c * 256 + lane * 8;
    if (col < D) {
      float o[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = fmaf(g[c][j] * rstd, __ldg(w + col + j), bias != nullptr ? __ldg(bias + col + j) : 0.f);
      *reinterpret_cast<uint4*>(y + row * D + col) = pack8(o);
    }
  }
}

template <int NCH>
__global__ void __launch_bounds__(256) gated_rms_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ v,
                                                            const __nv_bfloat16* __restrict__ z, const float* __restrict__ w,
                                                            const float* __restrict__ rstd_in, __nv_bfloat16* __restrict__ dv,
                                                            __nv_bfloat16* __restrict__ dz, float* __restrict__ dw,
                                                            float* __restrict__ db, long long M, int D, int rows_per_warp) {
  __shared__ float red[8][NCH * 256];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const long long r0 = ((blockIdx.x * 256LL + threadIdx.x) >> 5) * rows_per_warp, r1 = min(M, r0 + rows_per_warp);
  float aw[NCH][8], ab[NCH][8];
#pragma unroll
  for (int c = 0; c < NCH; ++c)
#pragma unroll
    for (int j = 0; j < 8; ++j) { aw[c][j] = 0.f; ab[c][j] = 0.f; }
  for (long long row = r0; row < r1; ++row) {
    const float rstd = __ldg(rstd_in + row);
    uint4 tv[NCH], tz[NCH], td[NCH];
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const int col = c * 256 + lane * 8;
      if (col < D) {
        tv[c] = __ldg(reinterpret_cast<const uint4*>(v + row * D + col));
        tz[c] = __ldg(reinterpret_cast<const uint4*>(z + row * D + col));
        td[c] = __ldg(reinterpret_cast<const uint4*>(dy + row * D + col));
      }
    }
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const int col = c * 256 + lane * 8;
      if (col < D) {
        float a[8], b[8], d[8];
        unpack8(tv[c], a); unpack8(tz[c], b); unpack8(td[c], d);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xh = __bfloat162float(__float2bfloat16(a[j] * (b[j] / (1.f + __expf(-b[j]))))) * rstd;
          aw[c][j] = fmaf(d[j], xh, aw[c][j]);
          ab[c][j] += d[j];
          s = fmaf(d[j] * __ldg(w + col + j), xh, s);
        }
      }
    }
    s = wsum(s) / D;
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const int col = c * 256 + lane * 8;
      if (col < D) {
        float a[8], b[8], d[8], o[8];
        unpack8(tv[c], a); unpack8(tz[c], b); unpack8(td[c], d);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float e = 1.f + __expf(-b[j]), sg = 1.f / e, si = b[j] * sg;
          const float xh = __bfloat162float(__float2bfloat16(a[j] * (b[j] / e))) * rstd;     // as in the forward
          const float dg = rstd * (d[j] * __ldg(w + col + j) - xh * s);
          o[j] = dg * si;
          d[j] = dg * a[j] * fmaf(si, 1.f - sg, sg);
        }
        *reinterpret_cast<uint4*>(dv + row * D + col) = pack8(o);
        *reinterpret_cast<uint4*>(dz + row * D + col) = pack8(d);
      }
    }
  }
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
    for (int c = 0; c < NCH; ++c)
#pragma unroll
      for (int j = 0; j < 8; ++j) red[wib][c * 256 + lane * 8 + j] = pass == 0 ? aw[c][j] : ab[c][j];
    __syncthreads();
    for (int i = threadIdx.x; i < D; i += 256) {
      float t = 0.f;
#pragma unroll
      for (int q = 0; q < 8; ++q) t += red[q][i];
      atomicAdd((pass == 0 ? dw : db) + i, t);
    }
    __syncthreads();
  }
}

static bool off16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; }

}  // namespace mix
}  // namespace recml

using namespace recml::mix;

// xbc [T, H P + 2 N] bf16 (P = N in {64, 128}), raw [T, H] bf16 or fp32, a / bias [H] fp32 -> dt [T, H] fp32,
// cum [H, pitch] fp32 (zero behind T), xs [T, H P] bf16.  T = B L.
extern "C" int recml_mamba_pre_fwd(const void* xbc, const void* raw, int raw_bf16, const float* bias, const float* a, int B, int L,
                                   int H, int P, float* dt, float* cum, long long pitch, void* xs, cudaStream_t stream) {
  if (B <= 0 || L <= 0 || H <= 0) return 0;
  if ((P != 64 && P != 128) || off16(xbc) || off16(xs) || pitch < static_cast<long long>(B) * L) return -10;
  using bf = __nv_bfloat16;
  const long long T = static_cast<long long>(B) * L;
  const unsigned blocks = static_cast<unsigned>((static_cast<long long>(B) * H + 7) / 8);
  if (raw_bf16) dt_scan_kernel<<<blocks, 256, 0, stream>>>(static_cast<const bf*>(raw), bias, a, B, L, H, dt, cum, pitch);
  else dt_scan_kernel<<<blocks, 256, 0, stream>>>(static_cast<const float*>(raw), bias, a, B, L, H, dt, cum, pitch);
  scale_kernel<<<static_cast<unsigned>((T + 3) / 4), dim3(64, 4), 0, stream>>>(static_cast<const bf*>(xbc), (H + 2) * P, dt, H, P,
                                                                               static_cast<bf*>(xs), T);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// dots [T, H] is scratch; da and dbias [H] are zero on entry.
extern "C" int recml_mamba_pre_bwd(const void* dxs, const float* db, const float* dc, const float* dcum, long long pitch,
                                   const void* xbc, const float* dt, const void* raw, int raw_bf16, const float* bias,
                                   const float* a, int B, int L, int H, int P, float* dots, void* dxbc, void* draw, float* da,
                                   float* dbias, cudaStream_t stream) {
  if (B <= 0 || L <= 0 || H <= 0) return 0;
  if ((P != 64 && P != 128) || off16(xbc) || off16(dxs) || off16(dxbc) || off16(db) || off16(dc)) return -10;
  using bf = __nv_bfloat16;
  const long long T = static_cast<long long>(B) * L, items = T * (H + 2) * (P / 8);
  const unsigned sb = static_cast<unsigned>((items + 255) / 256);
  if (P == 64) scale_bwd_kernel<8><<<sb, 256, 0, stream>>>(static_cast<const bf*>(dxs), static_cast<const bf*>(xbc), dt, db, dc, H,
                                                           static_cast<bf*>(dxbc), dots, T);
  else scale_bwd_kernel<16><<<sb, 256, 0, stream>>>(static_cast<const bf*>(dxs), static_cast<const bf*>(xbc), dt, db, dc, H,
                                                    static_cast<bf*>(dxbc), dots, T);
  const unsigned blocks = static_cast<unsigned>((static_cast<long long>(B) * H + 7) / 8);
  if (raw_bf16)
    dt_scan_bwd_kernel<<<blocks, 256, 0, stream>>>(dcum, pitch, dots, dt, static_cast<const bf*>(raw), bias, a, B, L, H,
                                                   static_cast<bf*>(draw), da, dbias);
  else
    dt_scan_bwd_kernel<<<blocks, 256, 0, stream>>>(dcum, pitch, dots, dt, static_cast<const float*>(raw), bias, a, B, L, H,
                                                   static_cast<float*>(draw), da, dbias);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// v, z, y: [M, D] bf16 contiguous, D % 8 == 0, D <= 1024, 16-byte aligned; w [D], bias [D] or null, rstd [M].
extern "C" int recml_gated_rms_fwd(const void* v, const void* z, const float* w, const float* bias, void* y, float* rstd, long long M,
                                   int D, float eps, cudaStream_t stream) {
  if (M <= 0) return 0;
  if (D <= 0 || D % 8 || D > 1024 || off16(v) || off16(z) || off16(y)) return -10;
  using bf = __nv_bfloat16;
  const unsigned blocks = static_cast<unsigned>((M + 7) / 8);
#define RECML_GR(N) gated_rms_fwd_kernel<N><<<blocks, 256, 0, stream>>>(static_cast<const bf*>(v), static_cast<const bf*>(z), w, bias, \
                                                                        static_cast<bf*>(y), rstd, M, D, eps)
  if (D <= 256) RECML_GR(1);
  else if (D <= 512) RECML_GR(2);
  else RECML_GR(4);
#undef RECML_GR
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// dw, db [D] fp32, zero on entry.
extern "C" int recml_gated_rms_bwd(const void* dy, const void* v, const void* z, const float* w, const float* rstd, void* dv, void* dz,
                                   float* dw, float* db, long long M, int D, cudaStream_t stream) {
  if (M <= 0) return 0;
  if (D <= 0 || D % 8 || D > 1024 || off16(dy) || off16(v) || off16(z) || off16(dv) || off16(dz)) return -10;
  using bf = __nv_bfloat16;
  // enough rows per warp that the column sums at a block's end do not count, enough blocks for six on every SM
  long long rpw = (M + 148LL * 6 * 8 - 1) / (148LL * 6 * 8);
  rpw = rpw < 1 ? 1 : rpw > 16 ? 16 : rpw;
  const unsigned blocks = static_cast<unsigned>((M + 8 * rpw - 1) / (8 * rpw));
#define RECML_GR(N) gated_rms_bwd_kernel<N><<<blocks, 256, 0, stream>>>(static_cast<const bf*>(dy), static_cast<const bf*>(v), \
      static_cast<const bf*>(z), w, rstd, static_cast<bf*>(dv), static_cast<bf*>(dz), dw, db, M, D, static_cast<int>(rpw))
  if (D <= 256) RECML_GR(1);
  else if (D <= 512) RECML_GR(2);
  else RECML_GR(4);
#undef RECML_GR
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
