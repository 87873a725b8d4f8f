// Fused post-expert RMSNorm + score-weighted top-k reduction, forward and backward.
//
//   y[t,k,:]  = cast_norm( g * h3[t,k,:] * rstd[t,k] ),  rstd = rsqrt(mean_d((g*h3)^2) + eps)
//   out[t,:]  = cast_out( sum_k s[t,k] * y[t,k,:] )                      (routes with id < 0 skipped)
// g = gamma + gain_center when an input-scale gamma is given (inference), else 1.
// Same composition as the reference's standalone RMSNorm followed by scale_and_sum
// (dist_moe/kernels/norm/fused_rmsnorm_combine.py:427-466); the backward is its autograd:
//   grad_s[t,k]    = <y[t,k,:], go[t,:]>
//   grad_h3[t,k,:] = rstd * s * (go - y * <go, y> / D)
// HBM bound: forward reads h3 once (a token's K rows stay in shared memory, or hit L1 in the second pass where they do not
// fit), backward reads h3 and go once and writes grad_h3 in place.
#include <type_traits>

#include "common.cuh"
#include "../../include/dist_moe_b200.h"

namespace dm {

constexpr int kNormMaxK = 32;
constexpr int kNormBlocks = 4;                // resident blocks of the staged form, at most
constexpr int64_t kNormStaged = 216 * 1024;  // rows in the shared memory of an SM

__device__ __forceinline__ void up8(const uint4& v, float (&f)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

// Compensated accumulation of the sum of squares (dist_moe/_postprocess.py:44-46 `use_kahan`): every thread keeps a
// running compensation term, and partial sums are merged with an error-free two-sum, so the result is the fp32
// rounding of a nearly exact sum whatever the order.
__device__ __forceinline__ void kahan_add(float& s, float& c, float x) {
  const float y = __fsub_rn(x, c);
  const float t = __fadd_rn(s, y);
  c = __fsub_rn(__fsub_rn(t, s), y);
  s = t;
}
__device__ __forceinline__ void two_sum_merge(float& s, float& c, float s2, float c2) {
  const float t = __fadd_rn(s, s2);
  const float bp = __fsub_rn(t, s);
  const float err = __fadd_rn(__fsub_rn(s, __fsub_rn(t, bp)), __fsub_rn(s2, bp));
  c = __fsub_rn(__fadd_rn(c, c2), err);  // c follows kahan_add's sign: it holds minus the lost low part
  s = t;
}
__device__ __forceinline__ void warp_reduce_sumsq(float& ss, float& cc, int kahan) {
  if (kahan) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      const float s2 = __shfl_xor_sync(0xffffffffu, ss, d), c2 = __shfl_xor_sync(0xffffffffu, cc, d);
      two_sum_merge(ss, cc, s2, c2);
    }
  } else {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
  }
}

// A block's tokens from `first` on, their rows read from memory.
template <typename IdT>
__device__ __forceinline__ void norm_tokens(int64_t first, const uint4* __restrict__ h3, const void* scores, int scores_bf16,
                                            const IdT* __restrict__ ids, const uint4* __restrict__ gamma, float gain_center, float eps,
                                            int norm_bf16, uint4* __restrict__ out, float* __restrict__ rstd_out, int64_t T, int K,
                                            int vec, uint4* save_dst, int kahan, float (*part)[8], float (*partc)[8], float* rs) {
  const bool save = save_dst != nullptr;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float inv_d = 1.0f / static_cast<float>(vec * 8);
  for (int64_t t = first; t < T; t += gridDim.x) {
    for (int k = 0; k < K; ++k) {
      const int64_t route = t * K + k;
      float ss = 0.f, cc = 0.f;
      for (int v = threadIdx.x; v < vec; v += 256) {
        const uint4 raw = h3[route * vec + v];
        if (save) save_dst[route * vec + v] = raw;
        float h[8];
        up8(raw, h);
        if (gamma != nullptr) {
          float g[8];
          up8(gamma[v], g);
#pragma unroll
          for (int j = 0; j < 8; ++j) h[j] *= (g[j] + gain_center);
        }
        if (kahan) {
#pragma unroll
          for (int j = 0; j < 8; ++j) kahan_add(ss, cc, __fmul_rn(h[j], h[j]));
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) ss += h[j] * h[j];
        }
      }
      warp_reduce_sumsq(ss, cc, kahan);
      if (lane == 0) {
        part[k][warp] = ss;
        partc[k][warp] = cc;
      }
    }
    __syncthreads();
    if (threadIdx.x < K) {
      float ss = 0.f;
      if (kahan) {
        float cc = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) two_sum_merge(ss, cc, part[threadIdx.x][w], partc[threadIdx.x][w]);
        ss = __fsub_rn(ss, cc);
      } else {
#pragma unroll
        for (int w = 0; w < 8; ++w) ss += part[threadIdx.x][w];
      }
      const int64_t route = t * K + threadIdx.x;
      const float r = ids[route] >= 0 ? rsqrtf(ss * inv_d + eps) : 0.f;
      rs[threadIdx.x] = r;
      if (rstd_out != nullptr) rstd_out[route] = r;
    }
    __syncthreads();
    for (int v = threadIdx.x; v < vec; v += 256) {
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      float g[8];
      if (gamma != nullptr) {
        up8(gamma[v], g);
#pragma unroll
        for (int j = 0; j < 8; ++j) g[j] += gain_center;
      }
      for (int k = 0; k < K; ++k) {
        const int64_t route = t * K + k;
        if (ids[route] < 0) continue;
        const float w = scores_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(scores)[route])
                                    : static_cast<const float*>(scores)[route];
        const float r = rs[k];
        float h[8];
        up8(h3[route * vec + v], h);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float y = (gamma != nullptr ? h[j] * g[j] : h[j]) * r;
          if (norm_bf16) y = round_bf16(y);
          acc[j] += y * w;
        }
      }
      out[t * vec + v] = make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]),
                                    pack_bf16x2(acc[4], acc[5]), pack_bf16x2(acc[6], acc[7]));
    }
    __syncthreads();
  }
}
// The same out of line: what the staged form below falls back on costs its registers and its code nothing.
template <typename IdT>
__device__ __noinline__ void norm_tokens_late(int64_t first, const uint4* h3, const void* scores, int scores_bf16, const IdT* ids,
                                              const uint4* gamma, float gain_center, float eps, int norm_bf16, uint4* out,
                                              float* rstd_out, int64_t T, int K, int vec, uint4* save_dst, int kahan,
                                              float (*part)[8], float (*partc)[8], float* rs) {
  norm_tokens<IdT>(first, h3, scores, scores_bf16, ids, gamma, gain_center, eps, norm_bf16, out, rstd_out, T, K, vec, save_dst, kahan,
                   part, partc, rs);
}

template <typename IdT>
__global__ void __launch_bounds__(256) rmsnorm_combine_fwd_kernel(
    const uint4* __restrict__ h3, const void* scores, int scores_bf16, const IdT* __restrict__ ids,
    const uint4* __restrict__ gamma, float gain_center, float eps, int norm_bf16, uint4* __restrict__ out,
    float* __restrict__ rstd_out, int64_t T, int K, int vec, uint8_t* save_base, const int64_t* save_offset,
    const int* save_cond, int save_expect, int kahan, int*) {
  __shared__ float part[kNormMaxK][8];
  __shared__ float partc[kNormMaxK][8];
  __shared__ float rs[kNormMaxK];
  bool save = save_base != nullptr;
  if (save && save_cond != nullptr) save = ((*save_cond != 0) == (save_expect != 0));
  if (save && save_offset != nullptr) save = *save_offset >= 0;
  uint4* save_dst = save ? reinterpret_cast<uint4*>(save_base + (save_offset ? *save_offset : 0)) : nullptr;
  norm_tokens<IdT>(blockIdx.x, h3, scores, scores_bf16, ids, gamma, gain_center, eps, norm_bf16, out, rstd_out, T, K, vec, save_dst,
                   kahan, part, partc, rs);
}

// The same sums in the same order with a token's K rows, which are contiguous, in shared memory: one bulk copy per token, the next
// token's on its way while this one is worked on.  The kernel above has two loads of a thread in flight, reads every row twice and
// looks at its options for every element (17 instructions each; issue-bound once the loads overlap: 41 us in the first example
// below); here they are template parameters, and four rows are summed and reduced side by side.  One B200, us: T = 4096, K = 4, D =
// 2816 59 -> 27; K = 8: D = 1024 57 -> 25, 3456 116 -> 54, 7168 229 -> 157 (one block per SM); T = 16, K = 4, D = 2816 5.5 -> 3.1.
// Bound: HBM (92 MB in 27 us, 0.6 of the copy rate) and the three barriers of a token.  What the loop keeps for a copy that does not
// come in time costs 0.3 us of the first example and under 0.1 at T = 16; asking all threads at a barrier (__syncthreads_or) cost
// 2.0, copies by the threads that read them (cp.async), which need no such thing, 5.7.
template <typename IdT, bool kGamma, bool kNorm16, bool kKahan>
__global__ void __launch_bounds__(256, kNormBlocks) rmsnorm_combine_fwd_staged_kernel(
    const uint4* __restrict__ h3, const void* scores, int scores_bf16, const IdT* __restrict__ ids,
    const uint4* __restrict__ gamma, float gain_center, float eps, int, uint4* __restrict__ out,
    float* __restrict__ rstd_out, int64_t T, int K, int vec, uint8_t* save_base, const int64_t* save_offset,
    const int* save_cond, int save_expect, int, int* status, int buffers) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ uint64_t full[2];
  __shared__ int abort_flag;
  __shared__ float part[kNormMaxK][8];
  __shared__ float partc[kNormMaxK][8];
  __shared__ float rs[kNormMaxK];
  __shared__ float ws[kNormMaxK];
  bool save = save_base != nullptr;
  if (save && save_cond != nullptr) save = ((*save_cond != 0) == (save_expect != 0));
  if (save && save_offset != nullptr) save = *save_offset >= 0;
  uint4* save_dst = save ? reinterpret_cast<uint4*>(save_base + (save_offset ? *save_offset : 0)) : nullptr;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float inv_d = 1.0f / static_cast<float>(vec * 8);
  const int rows = K * vec;  // vectors of a token
  const uint32_t bytes = static_cast<uint32_t>(rows) * 16;
  int issued = 0;  // copies that thread 0 has started
  auto fetch = [&](int64_t t, int b) {
    ++issued;
    mbar_arrive_expect_tx(&full[b], bytes);
    bulk_load(smem + b * bytes, h3 + t * rows, bytes, &full[b]);
  };
  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    mbar_fence_init();
    fence_proxy_async_smem();
    if (blockIdx.x < T) fetch(blockIdx.x, 0);
  }
  __syncthreads();
  int b = 0, it = 0;
  for (int64_t t = blockIdx.x; t < T; t += gridDim.x, ++it) {
    const int64_t ahead = t + gridDim.x;
    if (buffers == 2 && threadIdx.x == 0 && ahead < T) fetch(ahead, b ^ 1);  // every thread has left that buffer
    if (threadIdx.x < K) {
      const int64_t route = t * K + threadIdx.x;
      ws[threadIdx.x] = scores_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(scores)[route])
                                    : static_cast<const float*>(scores)[route];
    }
    const bool valid = threadIdx.x < K && ids[t * K + threadIdx.x] >= 0;
    const uint32_t parity = buffers == 2 ? (it >> 1) & 1 : it & 1;
    uint4* src = reinterpret_cast<uint4*>(smem + b * bytes);
    // A copy that did not come in time (none is known): a thread fetches the rows' pieces that it reads itself.  The copy may still
    // land, with the same bytes; the block leaves this loop before anything else takes their place.
    if (!mbar_wait(&full[b], parity, &abort_flag))
      for (int k = 0; k < K; ++k)
        for (int v = threadIdx.x; v < vec; v += 256) src[k * vec + v] = h3[t * rows + k * vec + v];
    // four rows at a time: their loads, sums and reductions overlap
    for (int k0 = 0; k0 < K; k0 += 4) {
      float ss[4] = {0.f, 0.f, 0.f, 0.f}, cc[4] = {0.f, 0.f, 0.f, 0.f};
      for (int v = threadIdx.x; v < vec; v += 256) {
        uint4 raw[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) raw[q] = k0 + q < K ? src[(k0 + q) * vec + v] : make_uint4(0, 0, 0, 0);
        float g[8];
        if (kGamma) {
          up8(gamma[v], g);
#pragma unroll
          for (int j = 0; j < 8; ++j) g[j] += gain_center;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (save && k0 + q < K) save_dst[t * rows + (k0 + q) * vec + v] = raw[q];
          float h[8];
          up8(raw[q], h);
          if (kGamma) {
#pragma unroll
            for (int j = 0; j < 8; ++j) h[j] *= g[j];
          }
          if (kKahan) {
#pragma unroll
            for (int j = 0; j < 8; ++j) kahan_add(ss[q], cc[q], __fmul_rn(h[j], h[j]));
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) ss[q] += h[j] * h[j];
          }
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) warp_reduce_sumsq(ss[q], cc[q], kKahan);
      if (lane == 0) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (k0 + q < K) {
            part[k0 + q][warp] = ss[q];
            partc[k0 + q][warp] = cc[q];
          }
      }
    }
    __syncthreads();
    if (threadIdx.x < K) {
      float ss = 0.f;
      if (kKahan) {
        float cc = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) two_sum_merge(ss, cc, part[threadIdx.x][w], partc[threadIdx.x][w]);
        ss = __fsub_rn(ss, cc);
      } else {
#pragma unroll
        for (int w = 0; w < 8; ++w) ss += part[threadIdx.x][w];
      }
      const float r = valid ? rsqrtf(ss * inv_d + eps) : 0.f;
      rs[threadIdx.x] = valid ? r : -1.0f;  // rsqrtf is never negative: a route that is left out
      if (rstd_out != nullptr) rstd_out[t * K + threadIdx.x] = r;
    }
    __syncthreads();
    // raised before the barriers above, or by a wait for the next token: the same for all threads
    const bool stop = *const_cast<volatile int*>(&abort_flag) != 0;
    for (int v = threadIdx.x; v < vec; v += 256) {
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      float g[8];
      if (kGamma) {
        up8(gamma[v], g);
#pragma unroll
        for (int j = 0; j < 8; ++j) g[j] += gain_center;
      }
#pragma unroll 4
      for (int k = 0; k < K; ++k) {
        const float r = rs[k], w = ws[k];
        if (r < 0.0f) continue;
        float h[8];
        up8(src[k * vec + v], h);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float y = (kGamma ? h[j] * g[j] : h[j]) * r;
          if (kNorm16) y = round_bf16(y);
          acc[j] += y * w;
        }
      }
      out[t * vec + v] = make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]),
                                    pack_bf16x2(acc[4], acc[5]), pack_bf16x2(acc[6], acc[7]));
    }
    __syncthreads();
    if (stop) {  // no further copies; the rest of the block's tokens with their rows in memory, and the copies under way to their end
      norm_tokens_late<IdT>(ahead, h3, scores, scores_bf16, ids, gamma, gain_center, eps, kNorm16, out, rstd_out, T, K, vec, save_dst,
                            kKahan, part, partc, rs);
      if (threadIdx.x == 0) {
        set_status(status, kPipelineTimeout, 5, blockIdx.x);
        const uint64_t t0 = globaltimer_ns();
        for (; it < issued; ++it)
          while (!mbar_try_wait(&full[buffers == 2 ? it & 1 : 0], buffers == 2 ? (it >> 1) & 1 : it & 1) &&
                 globaltimer_ns() - t0 < 1000000000ull) {
          }
      }
      return;
    }
    if (buffers == 2)
      b ^= 1;
    else if (threadIdx.x == 0 && ahead < T)
      fetch(ahead, 0);
  }
}

// One warp per route.  h3 may alias grad_h3 (each lane reads a chunk before it writes it).
template <typename IdT>
__global__ void __launch_bounds__(256) rmsnorm_combine_bwd_kernel(
    const uint4* __restrict__ grad_out, const void* scores, int scores_bf16, const IdT* __restrict__ ids,
    const uint8_t* h3_base, const int64_t* h3_offset, const float* __restrict__ rstd_in, float eps, int norm_bf16,
    uint4* grad_h3, float* __restrict__ grad_scores, int64_t T, int K, int vec, int kahan) {
  const uint4* h3 = reinterpret_cast<const uint4*>(h3_base + (h3_offset ? *h3_offset : 0));
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  const float inv_d = 1.0f / static_cast<float>(vec * 8);
  const int64_t routes = T * K;
  for (int64_t route = blockIdx.x * static_cast<int64_t>(wpb) + (threadIdx.x >> 5); route < routes;
       route += static_cast<int64_t>(gridDim.x) * wpb) {
    const int64_t t = route / K;
    const bool valid = ids[route] >= 0;
    if (!valid) {
      for (int v = lane; v < vec; v += 32) grad_h3[route * vec + v] = make_uint4(0, 0, 0, 0);
      if (lane == 0 && grad_scores != nullptr) grad_scores[route] = 0.f;
      continue;
    }
    const float w = scores_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(scores)[route])
                                : static_cast<const float*>(scores)[route];
    float ss = 0.f, cc = 0.f, hg = 0.f;
    for (int v = lane; v < vec; v += 32) {
      float h[8], g[8];
      up8(h3[route * vec + v], h);
      up8(grad_out[t * vec + v], g);
      if (kahan) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          kahan_add(ss, cc, __fmul_rn(h[j], h[j]));
          hg += h[j] * g[j];
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          ss += h[j] * h[j];
          hg += h[j] * g[j];
        }
      }
    }
    if (kahan) {
      warp_reduce_sumsq(ss, cc, 1);
      ss = __fsub_rn(ss, cc);
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) hg += __shfl_xor_sync(0xffffffffu, hg, d);
    } else {
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) {
        ss += __shfl_xor_sync(0xffffffffu, ss, d);
        hg += __shfl_xor_sync(0xffffffffu, hg, d);
      }
    }
    const float r = rstd_in != nullptr ? rstd_in[route] : rsqrtf(ss * inv_d + eps);
    // <go, y> with y = h * r (the rounding of y to bf16 is ignored inside this inner product)
    const float gy = hg * r;
    float dot_y = 0.f;
    const float c = gy * inv_d;
    for (int v = lane; v < vec; v += 32) {
      float h[8], g[8], o[8];
      up8(h3[route * vec + v], h);
      up8(grad_out[t * vec + v], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float y = h[j] * r;
        if (norm_bf16) y = round_bf16(y);
        dot_y += y * g[j];
        o[j] = r * w * (g[j] - (h[j] * r) * c);
      }
      grad_h3[route * vec + v] = make_uint4(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]),
                                            pack_bf16x2(o[4], o[5]), pack_bf16x2(o[6], o[7]));
    }
    if (grad_scores != nullptr) {
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) dot_y += __shfl_xor_sync(0xffffffffu, dot_y, d);
      if (lane == 0) grad_scores[route] = dot_y;
    }
  }
}

}  // namespace dm

using namespace dm;

extern "C" int dm_rmsnorm_combine_fwd_status(const void* h3, const void* scores, int scores_are_bf16, const void* ids,
                                             int ids_are_int64, const void* gamma, float gain_center, float eps,
                                             int norm_is_bf16, int use_kahan, void* out, float* rstd_out, int64_t T, int K,
                                             int64_t D, void* save_base, const int64_t* save_offset, const int* save_cond,
                                             int save_expect, int* status, void* stream) {
  if (!h3 || !scores || !ids || !out || T <= 0 || K <= 0 || K > kNormMaxK || D <= 0 || (D % 8) != 0) return kRcBadArg;
  const int vec = static_cast<int>(D / 8);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto run = [&](auto kernel, auto* typed_ids, int per_sm, size_t smem, auto... more) {
    const int blocks = static_cast<int>(T < grid_cap(per_sm) ? T : grid_cap(per_sm));
    kernel<<<blocks, 256, smem, st>>>(static_cast<const uint4*>(h3), scores, scores_are_bf16, typed_ids,
                                      static_cast<const uint4*>(gamma), gain_center, eps, norm_is_bf16, static_cast<uint4*>(out),
                                      rstd_out, T, K, vec, static_cast<uint8_t*>(save_base), save_offset, save_cond, save_expect,
                                      use_kahan ? 1 : 0, status, more...);
    return static_cast<int>(cudaGetLastError());
  };
  auto choose = [&](auto* typed_ids) {
    using IdT = std::remove_const_t<std::remove_pointer_t<decltype(typed_ids)>>;
    const int64_t bytes = K * D * 2;
    // One short row has nothing to overlap with: 4,096 tokens of K = 1, rows in memory | staged, D = 256 9.9 | 12.0 us, 1024 11.0 | 13.4,
    // 2048 15.3 | 16.4, 2816 20.8 | 18.9, 7168 39.1 | 31.1.  Two rows: D = 128 13.7 | 12.5, 1024 19.0 | 14.8.
    if (bytes > kNormStaged || (K == 1 && D <= 2048)) return run(rmsnorm_combine_fwd_kernel<IdT>, typed_ids, 8, 0);
    // Resident blocks with so many buffers each; a block's tables take under 4 KiB.  Two buffers only where two blocks of them fit: with
    // one such block an SM (K x D from 27,137 to 27,648) 4,096 tokens of K = 4, D = 6912 took 85 us, with three blocks of one
    // buffer 52; K = 6, D = 4608 101 | 59, K = 8, D = 3456 90 | 54.
    auto resident = [&](int buffers) { return (kNormStaged + 4096) / (buffers * bytes + 4096); };
    const int buffers = resident(2) >= 2 ? 2 : 1;
    const int64_t fit = resident(buffers);
    auto staged = [&](auto gamma_tag, auto norm_tag, auto kahan_tag) {
      constexpr auto kernel =
          rmsnorm_combine_fwd_staged_kernel<IdT, decltype(gamma_tag)::value, decltype(norm_tag)::value, decltype(kahan_tag)::value>;
      static PerDeviceOnce attr_set;
      const int rc = once_per_device(attr_set, [] {
        return static_cast<int>(
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kNormStaged)));
      });
      if (rc != 0) return rc;
      return run(kernel, typed_ids, static_cast<int>(fit < kNormBlocks ? fit : kNormBlocks),
                 static_cast<size_t>(buffers * bytes), buffers);
    };
    // The options are template parameters: looked at for every element they made the kernel issue-bound.
    auto with_kahan = [&](auto g, auto n) { return use_kahan ? staged(g, n, std::true_type{}) : staged(g, n, std::false_type{}); };
    auto with_norm = [&](auto g) { return norm_is_bf16 ? with_kahan(g, std::true_type{}) : with_kahan(g, std::false_type{}); };
    return gamma ? with_norm(std::true_type{}) : with_norm(std::false_type{});
  };
  return ids_are_int64 ? choose(static_cast<const int64_t*>(ids)) : choose(static_cast<const int32_t*>(ids));
}

extern "C" int dm_rmsnorm_combine_fwd(const void* h3, const void* scores, int scores_are_bf16, const void* ids,
                                      int ids_are_int64, const void* gamma, float gain_center, float eps,
                                      int norm_is_bf16, int use_kahan, void* out, float* rstd_out, int64_t T, int K,
                                      int64_t D, void* save_base, const int64_t* save_offset, const int* save_cond,
                                      int save_expect, void* stream) {
  return dm_rmsnorm_combine_fwd_status(h3, scores, scores_are_bf16, ids, ids_are_int64, gamma, gain_center, eps, norm_is_bf16,
                                       use_kahan, out, rstd_out, T, K, D, save_base, save_offset, save_cond, save_expect, nullptr,
                                       stream);
}

extern "C" int dm_rmsnorm_combine_bwd(const void* grad_out, const void* scores, int scores_are_bf16, const void* ids,
                                      int ids_are_int64, const void* h3_base, const int64_t* h3_offset,
                                      const float* rstd, float eps, int norm_is_bf16, int use_kahan, void* grad_h3,
                                      float* grad_scores, int64_t T, int K, int64_t D, void* stream) {
  if (!grad_out || !scores || !ids || !h3_base || !grad_h3 || T <= 0 || K <= 0 || D <= 0 || (D % 8) != 0)
    return kRcBadArg;
  const int vec = static_cast<int>(D / 8);
  int64_t blocks = (T * K + 7) / 8;
  if (blocks > grid_cap(16)) blocks = grid_cap(16);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (ids_are_int64)
    rmsnorm_combine_bwd_kernel<int64_t><<<static_cast<int>(blocks), 256, 0, st>>>(
        static_cast<const uint4*>(grad_out), scores, scores_are_bf16, static_cast<const int64_t*>(ids),
        static_cast<const uint8_t*>(h3_base), h3_offset, rstd, eps, norm_is_bf16, static_cast<uint4*>(grad_h3),
        grad_scores, T, K, vec, use_kahan ? 1 : 0);
  else
    rmsnorm_combine_bwd_kernel<int32_t><<<static_cast<int>(blocks), 256, 0, st>>>(
        static_cast<const uint4*>(grad_out), scores, scores_are_bf16, static_cast<const int32_t*>(ids),
        static_cast<const uint8_t*>(h3_base), h3_offset, rstd, eps, norm_is_bf16, static_cast<uint4*>(grad_h3),
        grad_scores, T, K, vec, use_kahan ? 1 : 0);
  return static_cast<int>(cudaGetLastError());
}
