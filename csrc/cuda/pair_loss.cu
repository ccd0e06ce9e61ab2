// Binary cross-entropy of one positive and one negative item per position, forward and backward:
//
//   pos = h . p, neg = h . n (per row of D columns);   loss = sum w (softplus(-pos) + softplus(neg))
//
// Bound by memory: three bf16 rows come in per position and, backward, three go out.  A warp takes whole rows in
// 16-byte loads, products and sums are fp32, and the sums over the rows are kept in double (one atomic per block), so
// the loss is as exact for a million positions as for one.  SASRec training at [512, 200, 256]: 5.39 -> 4.58 ms on a
// B200 against casts to fp32, broadcast products and their backwards.
#include "common.cuh"

namespace recml {
namespace pairloss {

struct Rows { const __nv_bfloat16* h; const __nv_bfloat16* p; const __nv_bfloat16* n; long long ldh, ldp, ldn; };

__device__ __forceinline__ void unpack8(const uint4& t, float (&v)[8]) {
  const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) { v[2 * j] = bf16_lo(w[j]); v[2 * j + 1] = bf16_hi(w[j]); }
}
__device__ __forceinline__ uint4 ld8(const __nv_bfloat16* p) { return __ldg(reinterpret_cast<const uint4*>(p)); }
// log(1 + e^x) without overflow
__device__ __forceinline__ float softplus(float x) { return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))); }
__device__ __forceinline__ float sigmoid(float x) { return 1.f / (1.f + expf(-x)); }

// coef[t] = (d loss / d pos, d loss / d neg); sums = (sum of losses, sum of weights), pre-zeroed.
__global__ void __launch_bounds__(256) fwd_kernel(const Rows r, const float* __restrict__ w, long long T, int D,
                                                  float2* __restrict__ coef, double* __restrict__ sums) {
  __shared__ double part[2][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double sl = 0.0, sw = 0.0;
  for (long long t = blockIdx.x * 8LL + warp; t < T; t += gridDim.x * 8LL) {
    float a = 0.f, b = 0.f;
    for (int c = lane * 8; c < D; c += 256) {
      float h[8], p[8], n[8];
      const uint4 hv = ld8(r.h + t * r.ldh + c), pv = ld8(r.p + t * r.ldp + c), nv = ld8(r.n + t * r.ldn + c);
      unpack8(hv, h); unpack8(pv, p); unpack8(nv, n);
#pragma unroll
      for (int j = 0; j < 8; ++j) { a = fmaf(h[j], p[j], a); b = fmaf(h[j], n[j], b); }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { a += __shfl_xor_sync(0xffffffffu, a, o); b += __shfl_xor_sync(0xffffffffu, b, o); }
    if (lane == 0) {
      const float wt = w[t];
      coef[t] = make_float2(-sigmoid(-a) * wt, sigmoid(b) * wt);
      sl += static_cast<double>((softplus(-a) + softplus(b)) * wt);
      sw += static_cast<double>(wt);
    }
  }
  if (lane == 0) { part[0][warp] = sl; part[1][warp] = sw; }
  __syncthreads();
  if (threadIdx.x < 2) {
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) s += part[threadIdx.x][q];
    atomicAdd(sums + threadIdx.x, s);
  }
}

// out[0] = sums[0] / max(sums[1], 1), out[1] = 1 / max(sums[1], 1)
__global__ void mean_kernel(const double* __restrict__ sums, float* __restrict__ out) {
  const double d = sums[1] > 1.0 ? sums[1] : 1.0;
  out[0] = static_cast<float>(sums[0] / d);
  out[1] = static_cast<float>(1.0 / d);
}

// dh, dp, dn [T, D] contiguous.  The gradient of the mean loss is *grad (fp32) and mean[1] = 1 / denominator.
__global__ void __launch_bounds__(256) bwd_kernel(const Rows r, const float2* __restrict__ coef, const float* __restrict__ mean,
                                                  const float* __restrict__ grad, long long T, int D, __nv_bfloat16* __restrict__ dh,
                                                  __nv_bfloat16* __restrict__ dp, __nv_bfloat16* __restrict__ dn) {
  const int lane = threadIdx.x & 31;
  const long long t = blockIdx.x * 8LL + (threadIdx.x >> 5);
  if (t >= T) return;
  const float scale = __ldg(grad) * __ldg(mean + 1);
  const float2 k = __ldg(coef + t);
  const float ca = k.x * scale, cb = k.y * scale;
  for (int c = lane * 8; c < D; c += 256) {
    float h[8], p[8], n[8];
    const uint4 hv = ld8(r.h + t * r.ldh + c), pv = ld8(r.p + t * r.ldp + c), nv = ld8(r.n + t * r.ldn + c);
    unpack8(hv, h); unpack8(pv, p); unpack8(nv, n);
    uint32_t x[4], y[4], z[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      x[j] = pack_bf16(fmaf(ca, p[2 * j], cb * n[2 * j]), fmaf(ca, p[2 * j + 1], cb * n[2 * j + 1]));
      y[j] = pack_bf16(ca * h[2 * j], ca * h[2 * j + 1]);
      z[j] = pack_bf16(cb * h[2 * j], cb * h[2 * j + 1]);
    }
    *reinterpret_cast<uint4*>(dh + t * D + c) = make_uint4(x[0], x[1], x[2], x[3]);
    *reinterpret_cast<uint4*>(dp + t * D + c) = make_uint4(y[0], y[1], y[2], y[3]);
    *reinterpret_cast<uint4*>(dn + t * D + c) = make_uint4(z[0], z[1], z[2], z[3]);
  }
}

static bool bad(const void* p, long long ld) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0 || ld % 8 != 0; }

}  // namespace pairloss
}  // namespace recml

using namespace recml::pairloss;

// h, pos, neg: [T, D] bf16 with row pitches (multiples of 8; D too), 16-byte aligned; w [T]; sums [2] double, zero on
// entry; coef [T, 2]; mean [2] receives the mean loss and the reciprocal of its denominator.
extern "C" int recml_pair_bce_fwd(const void* h, long long ldh, const void* pos, long long ldp, const void* neg, long long ldn,
                                  const float* w, long long T, int D, void* coef, double* sums, float* mean, cudaStream_t stream) {
  if (D <= 0 || D % 8 || bad(h, ldh) || bad(pos, ldp) || bad(neg, ldn)) return -10;
  const Rows r{static_cast<const __nv_bfloat16*>(h), static_cast<const __nv_bfloat16*>(pos), static_cast<const __nv_bfloat16*>(neg),
               ldh, ldp, ldn};
  if (T > 0) {
    const long long want = (T + 7) / 8;
    const int blocks = static_cast<int>(want < 148 * 8 ? want : 148 * 8);
    fwd_kernel<<<blocks, 256, 0, stream>>>(r, w, T, D, static_cast<float2*>(coef), sums);
  }
  mean_kernel<<<1, 1, 0, stream>>>(sums, mean);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

extern "C" int recml_pair_bce_bwd(const void* h, long long ldh, const void* pos, long long ldp, const void* neg, long long ldn,
                                  const void* coef, const float* mean, const float* grad, long long T, int D, void* dh, void* dpos,
                                  void* dneg, cudaStream_t stream) {
  if (D <= 0 || D % 8 || bad(h, ldh) || bad(pos, ldp) || bad(neg, ldn) || bad(dh, 0) || bad(dpos, 0) || bad(dneg, 0)) return -10;
  if (T <= 0) return 0;
  const Rows r{static_cast<const __nv_bfloat16*>(h), static_cast<const __nv_bfloat16*>(pos), static_cast<const __nv_bfloat16*>(neg),
               ldh, ldp, ldn};
  bwd_kernel<<<static_cast<unsigned>((T + 7) / 8), 256, 0, stream>>>(
      r, static_cast<const float2*>(coef), mean, grad, T, D, static_cast<__nv_bfloat16*>(dh), static_cast<__nv_bfloat16*>(dpos),
      static_cast<__nv_bfloat16*>(dneg));
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
