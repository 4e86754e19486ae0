// The end of a layer and of a token step as single launches. A decode step of few sequences is a chain of small kernels of which each
// costs 1.5 - 2 us whatever it does: the sum of residual, routed and gated shared expert with the norm that follows took nine
// (cast, gate product, cast, sigmoid, cast, product, two sums, norm), the expert bookkeeping three (clear, count, clear), the greedy
// choice two.
#include "layer_tail.cuh"

#include "common.cuh"

namespace b200 {

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int kWarps>
__device__ __forceinline__ float block_sum(float v, float* scratch) {
  v = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < kWarps; ++i) s += scratch[i];
  return s;
}

__device__ __forceinline__ void unpack8(uint4 u, float (&f)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 p = unpack_bf16x2(w[e]);
    f[2 * e] = p.x;
    f[2 * e + 1] = p.y;
  }
}

// One block of 256 threads per row; a thread holds NV pieces of eight features, so a row is read once. Bound by bytes for many rows,
// by latency for few.
template <int NV>
__global__ void __launch_bounds__(256) layer_tail_kernel(const LayerTailArgs a) {
  let_dependents_start();
  __shared__ float scratch[8];
  const int64_t row = blockIdx.x, base = row * a.D;
  const int n8 = a.D / 8;
  float gate = 1.f;
  if (a.gate_w != nullptr) {
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = threadIdx.x + i * 256;
      if (c < n8) {
        float h[8], w[8];
        unpack8(reinterpret_cast<const uint4*>(a.h + base)[c], h);
        unpack8(reinterpret_cast<const uint4*>(a.gate_w)[c], w);
#pragma unroll
        for (int e = 0; e < 8; ++e) dot = fmaf(h[e], w[e], dot);
      }
    }
    gate = 1.f / (1.f + __expf(-block_sum<8>(dot, scratch)));
  }
  float v[NV][8], sq = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = threadIdx.x + i * 256;
    if (c >= n8) continue;
    float t[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[i][e] = 0.f;
    if (a.x != nullptr) unpack8(reinterpret_cast<const uint4*>(a.x + base)[c], v[i]);
    if (a.routed != nullptr) {
      const float4* r = reinterpret_cast<const float4*>(a.routed + base) + 2 * c;
      const float4 r0 = r[0], r1 = r[1];
      v[i][0] += r0.x; v[i][1] += r0.y; v[i][2] += r0.z; v[i][3] += r0.w;
      v[i][4] += r1.x; v[i][5] += r1.y; v[i][6] += r1.z; v[i][7] += r1.w;
    }
    if (a.shared != nullptr) {
      unpack8(reinterpret_cast<const uint4*>(a.shared + base)[c], t);
#pragma unroll
      for (int e = 0; e < 8; ++e) v[i][e] = fmaf(t[e], gate, v[i][e]);
    }
    const uint4 out = make_uint4(pack_bf16x2(v[i][0], v[i][1]), pack_bf16x2(v[i][2], v[i][3]), pack_bf16x2(v[i][4], v[i][5]),
                                 pack_bf16x2(v[i][6], v[i][7]));
    reinterpret_cast<uint4*>(a.x_out + base)[c] = out;
    unpack8(out, v[i]);       // the norm is of the rounded row
#pragma unroll
    for (int e = 0; e < 8; ++e) sq = fmaf(v[i][e], v[i][e], sq);
  }
  if (a.norm_w == nullptr) return;
  const float rstd = rsqrtf(block_sum<8>(sq, scratch) / a.D + a.eps), one = a.one_plus ? 1.f : 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = threadIdx.x + i * 256;
    if (c >= n8) continue;
    float w[8], y[8];
    unpack8(reinterpret_cast<const uint4*>(a.norm_w)[c], w);
#pragma unroll
    for (int e = 0; e < 8; ++e) y[e] = v[i][e] * rstd * (one + w[e]);
    reinterpret_cast<uint4*>(a.h_out + base)[c] =
        make_uint4(pack_bf16x2(y[0], y[1]), pack_bf16x2(y[2], y[3]), pack_bf16x2(y[4], y[5]), pack_bf16x2(y[6], y[7]));
  }
}

// Block 0 counts in shared memory, the others clear the output.
__global__ void __launch_bounds__(512)
moe_prepare_zero_kernel(const int* __restrict__ idx, int n_pairs, int n_experts, int* __restrict__ counts, int* __restrict__ pos,
                        float4* __restrict__ out, int64_t n_out4, int* __restrict__ order, int* __restrict__ flags, int n_flags) {
  __shared__ int cnt[kPrepareMaxExperts], sums[16];
  if (blockIdx.x > 0) {
    const int64_t step = static_cast<int64_t>(gridDim.x - 1) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x - 1) * blockDim.x + threadIdx.x; i < n_out4; i += step)
      out[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    return;
  }
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  cnt[t] = 0;
  __syncthreads();
  for (int p = t; p < n_pairs; p += 512) {
    const int e = idx[p];
    pos[p] = e >= 0 && e < n_experts ? atomicAdd(&cnt[e], 1) : 0;
  }
  if (order != nullptr)
    for (int i = t; i < n_flags; i += 512) flags[i] = 0;
  __syncthreads();
  const int mine = cnt[t];
  if (t < n_experts) counts[t] = mine;
  if (order == nullptr) return;
  int incl = mine;              // first place of every expert
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int n = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += n;
  }
  if (lane == 31) sums[warp] = incl;
  __syncthreads();
  int first = incl - mine;
  for (int w = 0; w < warp; ++w) first += sums[w];
  cnt[t] = first;
  __syncthreads();
  for (int p = t; p < n_pairs; p += 512) {
    const int e = idx[p];
    if (e >= 0 && e < n_experts) order[cnt[e] + pos[p]] = p;
  }
}

__global__ void __launch_bounds__(256)
silu_mul_kernel(const __nv_bfloat16* __restrict__ g, int64_t ldg, const __nv_bfloat16* __restrict__ u, int64_t ldu,
                __nv_bfloat16* __restrict__ out, int64_t n8, int i8) {
  let_dependents_start();
  const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n8; i += step) {
    const int64_t row = i / i8, c = i - row * i8;
    float x[8], y[8];
    unpack8(reinterpret_cast<const uint4*>(g + row * ldg)[c], x);
    unpack8(reinterpret_cast<const uint4*>(u + row * ldu)[c], y);
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
      w[e] = pack_bf16x2(x[2 * e] / (1.f + __expf(-x[2 * e])) * y[2 * e], x[2 * e + 1] / (1.f + __expf(-x[2 * e + 1])) * y[2 * e + 1]);
    reinterpret_cast<uint4*>(out)[i] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

__device__ __forceinline__ uint32_t order_key(uint32_t bf16_bits) {   // larger key, larger value; +0 and -0 alike, NaN on top
  const uint32_t mag = bf16_bits & 0x7fffu;
  if (mag > 0x7f80u) return 0xffffu;
  if (mag == 0) return 0x8000u;
  return (bf16_bits & 0x8000u) ? 0x8000u - mag : 0x8000u + mag;
}

// A cluster of kArgBlocks blocks per row (one block reads a row of 152 thousand in 16.6 us, eight in 6.5): a thread keeps the
// best (value, place) of its pieces of eight as one 64-bit key, the place inverted so that the larger key is the earlier one.
constexpr int kArgBlocks = 8, kArgThreads = 512;

__global__ void __cluster_dims__(kArgBlocks, 1, 1) __launch_bounds__(kArgThreads)
argmax_rows_kernel(const __nv_bfloat16* __restrict__ x, int64_t ldx, int N, int64_t* __restrict__ ids) {
  __shared__ unsigned long long warp_best[kArgThreads / 32], block_best;
  const int part = blockIdx.x % kArgBlocks, first = part * kArgThreads + threadIdx.x;
  constexpr int kStride = kArgBlocks * kArgThreads;
  const __nv_bfloat16* row = x + (blockIdx.x / kArgBlocks) * ldx;
  const uint4* row8 = reinterpret_cast<const uint4*>(row);
  const int n8 = (reinterpret_cast<uintptr_t>(row) & 15) == 0 ? N / 8 : 0;
  uint32_t key = 0;
  int at = 0x7fffffff;
  auto take = [&](uint32_t bits, int i) {
    const uint32_t k = order_key(bits);
    if (k > key || (k == key && i < at)) {
      key = k;
      at = i;
    }
  };
#pragma unroll 4
  for (int c = first; c < n8; c += kStride) {
    const uint4 u = __ldg(row8 + c);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      take(w[e] & 0xffffu, 8 * c + 2 * e);
      take(w[e] >> 16, 8 * c + 2 * e + 1);
    }
  }
  const uint16_t* row1 = reinterpret_cast<const uint16_t*>(row);
  for (int i = 8 * n8 + first; i < N; i += kStride) take(row1[i], i);
  unsigned long long best = (static_cast<unsigned long long>(key) << 32) | (0x7fffffffu - static_cast<uint32_t>(at));
  auto larger = [](unsigned long long v, int width) {
    for (int o = width / 2; o > 0; o >>= 1) {
      const unsigned long long n = __shfl_xor_sync(0xffffffffu, v, o);
      v = n > v ? n : v;
    }
    return v;
  };
  best = larger(best, 32);
  if ((threadIdx.x & 31) == 0) warp_best[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x < 32) {
    best = larger(threadIdx.x < kArgThreads / 32 ? warp_best[threadIdx.x] : 0ull, 32);
    if (threadIdx.x == 0) block_best = best;
  }
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
  if (part == 0 && threadIdx.x < 32) {
    best = 0;
    if (threadIdx.x < kArgBlocks) {
      uint32_t peer;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(smem_u32(&block_best)), "r"(threadIdx.x));
      asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(best) : "r"(peer) : "memory");
    }
    best = larger(best, 32);
    if (threadIdx.x == 0) ids[blockIdx.x / kArgBlocks] = 0x7fffffffu - static_cast<uint32_t>(best);
  }
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");   // its shared memory was being read
}

}  // namespace

cudaError_t launch_layer_tail(const LayerTailArgs& a, cudaStream_t st) {
  if (a.D < 8 || a.D % 8 != 0 || a.D > kTailMaxWidth || a.x_out == nullptr || (a.gate_w != nullptr && a.h == nullptr) ||
      (a.norm_w != nullptr && a.h_out == nullptr))
    return cudaErrorInvalidValue;
  if (a.rows <= 0) return cudaSuccess;
  if (a.D <= 2048) layer_tail_kernel<1><<<a.rows, 256, 0, st>>>(a);
  else if (a.D <= 4096) layer_tail_kernel<2><<<a.rows, 256, 0, st>>>(a);
  else layer_tail_kernel<4><<<a.rows, 256, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_moe_prepare_zero(const int* idx, int n_pairs, int n_experts, int* counts, int* pos, float* out, int64_t n_out,
                                    int* order, int* flags, int n_flags, cudaStream_t st) {
  if ((order != nullptr && flags == nullptr) || n_pairs < 0 || n_pairs > kPrepareMaxPairs || n_experts < 1 || n_experts > kPrepareMaxExperts || n_out % 4 != 0)
    return cudaErrorInvalidValue;
  const int64_t want = (n_out / 4 + 2047) / 2048;       // four stores a thread
  moe_prepare_zero_kernel<<<1 + static_cast<int>(want < 1184 ? want : 1184), 512, 0, st>>>(idx, n_pairs, n_experts, counts, pos,
                                                                                       reinterpret_cast<float4*>(out), n_out / 4, order,
                                                                                       flags, n_flags);
  return cudaGetLastError();
}

cudaError_t launch_silu_mul(const __nv_bfloat16* g, int64_t ldg, const __nv_bfloat16* u, int64_t ldu, __nv_bfloat16* out, int64_t rows,
                            int I, cudaStream_t st) {
  if (I < 8 || I % 8 != 0 || ldg % 8 != 0 || ldu % 8 != 0) return cudaErrorInvalidValue;
  const int64_t n8 = rows * (I / 8), want = (n8 + 511) / 512;     // two pieces a thread
  if (n8 <= 0) return cudaSuccess;
  silu_mul_kernel<<<static_cast<int>(want < 4736 ? want : 4736), 256, 0, st>>>(g, ldg, u, ldu, out, n8, I / 8);
  return cudaGetLastError();
}

cudaError_t launch_argmax_rows(const __nv_bfloat16* x, int64_t ldx, int rows, int N, int64_t* ids, cudaStream_t st) {
  if (N < 1 || rows < 0) return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  argmax_rows_kernel<<<rows * kArgBlocks, kArgThreads, 0, st>>>(x, ldx, N, ids);
  return cudaGetLastError();
}

}  // namespace b200
