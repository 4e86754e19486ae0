// Gated-DeltaNet prefill: everything of the chunked gated delta rule that does NOT depend on the running state,
// forward and backward, as one kernel each (matrix instructions around an fp32 inverse, no library call).
//
// Per chunk of 64 tokens and per value head the chunked algorithm needs (jax_gpt/models/qwen35/deltanet.py:214-300,
// which computes them with batched einsums and a triangular solve):
//     beta = sigmoid(b)            g = -exp(A_log) softplus(a + dt_bias)        G = cumsum(g) inside the chunk
//     q^ = l2norm(q) dk^-1/2       k^ = l2norm(k)
//     A     = strict_lower(beta_i (k^_i . k^_j) exp(G_i - G_j))
//     X     = (I + A)^-1 [beta v | beta exp(G) k^]            ->  v_eff (64 x 128), k_cum (64 x 128)
//     intra = lower(q^_i . k^_j exp(G_i - G_j))               k_dec = k^ exp(G_end - G)      q_e = q^ exp(G)
// and the inter-chunk scan (gdn_kernels.cu) consumes [k_cum ; q_e], intra, k_dec, v_eff, exp(G_end).
//
// One CTA owns one (batch, q/k head, chunk) and loops over the value heads that share the q/k head. The raw bf16 rows of q, k and
// v lie in shared memory as they are; every product with them is exact in its operands, their L2 norms scale fp32 sums or factors.
//
// The backward kernel recomputes the forward quantities from the same inputs and pushes the gradients through the solve, the
// decays, the gates, the Gram matrices and the two L2 norms down to d(mixed), d(b), d(a), d(A_log) and d(dt_bias). Gradients of q
// and k are summed over the value heads in registers, so the kernel has no global atomics except the two per-head scalars.
#include "seq_kernels.cuh"

#include "common.cuh"

namespace b200 {

namespace {

constexpr int kC = 64;            // chunk length
constexpr int kD = 128;           // dk = dv
constexpr int kThreads = 256;
constexpr float kQScale = 0.08838834764831845f;   // 128^-1/2

struct PrepGeom {
  int T, N, Hqk, Hv, conv_dim;
};

__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.f / (1.f + expf(-x)); }
__device__ __forceinline__ float bf2f(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ float2 bf2f2(const __nv_bfloat16* p) {
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
}
struct PrepFwdArgs {
  const __nv_bfloat16* mixed;   // [B, T, conv_dim]: q | k | v after conv + SiLU
  const __nv_bfloat16* b_in;    // [B, T, Hv]
  const __nv_bfloat16* a_in;    // [B, T, Hv]
  const float* A_log;           // [Hv]
  const float* dt_bias;         // [Hv]
  __nv_bfloat16* kq;            // [B*Hv, N, 128, 128]
  __nv_bfloat16* intra;         // [B*Hv, N, 64, 64]
  __nv_bfloat16* kdec;          // [B*Hv, N, 64, 128]
  __nv_bfloat16* veff;          // [B*Hv, N, 64, 128]
  float* e;                     // [B*Hv, N]
  PrepGeom gm;
};

// ---- forward -----------------------------------------------------------------------------------------------------------
// Bound by instruction issue, not by bytes (0.2 GB for 4096 tokens and 32 heads): with a right-hand side column per thread and the
// substitution unrolled over 64 registers the kernel ran at a fifth of the issue rate, its 43 KB of straight-line code and the
// chain through every row of the substitution exposed at two CTAs per SM. The products are matrix instructions here:
//   - the Gram matrices from the raw bf16 rows, whose products are exact; the norms scale the fp32 sums;
//   - T = (I + A)^-1 in fp32: the four 16 x 16 blocks on the diagonal by substitution, a column per thread, then two doublings
//     T21 = -T22 (A21 T11), each two small products over the whole block;
//   - X = (T diag(beta)) V and (T diag(beta exp(G) / |k|)) K: again raw bf16 rows on the right; the fp32 factor on the left is cut
//     into three bf16 parts (24 bits), so nothing is rounded that was not before.
// 4096 tokens, 32 value heads: 349 -> 131 us; against 64 bits the outputs are off by the same 1.66e-3 (their rounding to bf16).
constexpr int kRawLd = kD + 8;    // row stride (bf16) of the raw tiles: eight rows of 16 bytes fall into different banks
constexpr int kALd = kC + 4;      // row stride (floats) of A
constexpr int kTLd = kC + 8;      // and of T, which is read as pairs of floats of eight rows
constexpr int kULd = 32 + 4;

struct PrepFwdSmem {
  __nv_bfloat16 q[kC * kRawLd], k[kC * kRawLd], v[kC * kRawLd];
  float A[kC * kALd], T[kC * kTLd], U[32 * kULd];
  float beta[kC], G[kC], eg[kC], ed[kC], rq[kC], rk[kC], kscale[kC];
  float warp0_sum;
};

__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)) : "memory");
}

// 64 rows of 128 features from column `col` of the projections, zeros from row T on.
template <int NT>
__device__ __forceinline__ void load_raw_tile(const __nv_bfloat16* mixed_b, const PrepGeom& gm, int n, int col, __nv_bfloat16* dst) {
#pragma unroll
  for (int i = threadIdx.x; i < kC * (kD / 8); i += NT) {
    const int r = i >> 4, c8 = i & 15, t = n * kC + r;
    uint4 u = make_uint4(0, 0, 0, 0);
    if (t < gm.T) u = *reinterpret_cast<const uint4*>(mixed_b + static_cast<size_t>(t) * gm.conv_dim + col + c8 * 8);
    *reinterpret_cast<uint4*>(dst + r * kRawLd + c8 * 8) = u;
  }
}

// out (rows x cols) = sign * a (rows x inner) b (inner x cols), fp32 in shared memory, a thread per output, rows * cols a multiple
// of the block; `blocks` such products, the operands a step apart.
template <int NT, int kRows, int kCols, int kInner>
__device__ __forceinline__ void small_product(float* out, int ldo, const float* a, int lda, const float* b, int ldb, float sign,
                                              int blocks, int out_step, int a_step, int b_step) {
  const int per = kRows * kCols;
  for (int o = threadIdx.x; o < blocks * per; o += NT) {
    const int blk = o / per, r = (o % per) / kCols, c = o % kCols;
    const float* ar = a + blk * a_step + r * lda;
    const float* bc = b + blk * b_step + c;
    float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
    for (int m = 0; m < kInner; m += 4) {
      const float4 x = *reinterpret_cast<const float4*>(ar + m);
      s0 = fmaf(x.x, bc[m * ldb], s0);
      s1 = fmaf(x.y, bc[(m + 1) * ldb], s1);
      s2 = fmaf(x.z, bc[(m + 2) * ldb], s2);
      s3 = fmaf(x.w, bc[(m + 3) * ldb], s3);
    }
    out[blk * out_step + r * ldo + c] = sign * ((s0 + s1) + (s2 + s3));
  }
}

// T = (I + A)^-1 of the strictly lower triangular A; blocks of T above the diagonal that a product reads are cleared.
template <int NT>
__device__ __forceinline__ void unit_lower_inverse(const float* A, float* T, float* U) {
  const int tid = threadIdx.x;
  if (tid < kC) {
    const int b0 = tid & ~15, j = tid & 15;
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float acc[4] = {i == j ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int m = 0; m < i; ++m) acc[m & 3] = fmaf(-A[(b0 + i) * kALd + b0 + m], x[m], acc[m & 3]);
      x[i] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
      T[(b0 + i) * kTLd + tid] = x[i];
    }
  } else if (tid >= 128) {
    for (int i = tid - 128; i < 512; i += NT - 128) {   // the blocks right of the first and of the third on the diagonal
      const int r = (i >> 8) * 32 + ((i >> 4) & 15), c = (i >> 8) * 32 + 16 + (i & 15);
      T[r * kTLd + c] = 0.f;
    }
  }
  __syncthreads();
  small_product<NT, 16, 16, 16>(U, kULd, A + 16 * kALd, kALd, T, kTLd, 1.f, 2, 16 * kULd, 32 * kALd + 32, 32 * kTLd + 32);
  __syncthreads();
  small_product<NT, 16, 16, 16>(T + 16 * kTLd, kTLd, T + 16 * kTLd + 16, kTLd, U, kULd, -1.f, 2, 32 * kTLd + 32, 32 * kTLd + 32, 16 * kULd);
  __syncthreads();
  small_product<NT, 32, 32, 32>(U, kULd, A + 32 * kALd, kALd, T, kTLd, 1.f, 1, 0, 0, 0);
  __syncthreads();
  small_product<NT, 32, 32, 32>(T + 32 * kTLd, kTLd, T + 32 * kTLd + 32, kTLd, U, kULd, -1.f, 1, 0, 0, 0);
  __syncthreads();
}

__global__ void __launch_bounds__(kThreads, 2) gdn_chunk_prep_fwd_kernel(const PrepFwdArgs p) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  PrepFwdSmem& sm = *reinterpret_cast<PrepFwdSmem*>(smem_raw);
  const PrepGeom gm = p.gm;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const int n = blockIdx.x, hq = blockIdx.y, batch = blockIdx.z;
  const int rep = gm.Hv / gm.Hqk;
  const __nv_bfloat16* mixed_b = p.mixed + static_cast<size_t>(batch) * gm.T * gm.conv_dim;
  load_raw_tile<kThreads>(mixed_b, gm, n, hq * kD, sm.q);
  load_raw_tile<kThreads>(mixed_b, gm, n, gm.Hqk * kD + hq * kD, sm.k);
  __syncthreads();
  {
    // reciprocal norms, four threads per row
    const int i = tid >> 2, qd = tid & 3;
    float ssq = 0.f, ssk = 0.f;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const uint4 a = *reinterpret_cast<const uint4*>(sm.q + i * kRawLd + (qd + 4 * m) * 8);
      const uint4 b = *reinterpret_cast<const uint4*>(sm.k + i * kRawLd + (qd + 4 * m) * 8);
      const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 x = unpack_bf16x2(aw[e]), y = unpack_bf16x2(bw[e]);
        ssq += x.x * x.x + x.y * x.y;
        ssk += y.x * y.x + y.y * y.y;
      }
    }
    ssq += __shfl_xor_sync(0xffffffffu, ssq, 1);
    ssq += __shfl_xor_sync(0xffffffffu, ssq, 2);
    ssk += __shfl_xor_sync(0xffffffffu, ssk, 1);
    ssk += __shfl_xor_sync(0xffffffffu, ssk, 2);
    if (qd == 0) {
      sm.rq[i] = rsqrtf(ssq + 1e-6f) * kQScale;
      sm.rk[i] = rsqrtf(ssk + 1e-6f);
    }
  }
  __syncthreads();
  // Gram matrices: warps 0-3 the row tiles of k^ k^T, warps 4-7 those of q^ k^T; entries above the diagonal are not computed
  const int mt = warp & 3, row_lo = mt * 16 + g, row_hi = row_lo + 8;
  const bool of_q = warp >= 4;
  float gram[8][4];
#pragma unroll
  for (int j = 0; j < 8; ++j) gram[j][0] = gram[j][1] = gram[j][2] = gram[j][3] = 0.f;
  {
    const __nv_bfloat16* left = of_q ? sm.q : sm.k;
#pragma unroll
    for (int ks = 0; ks < kD / 16; ++ks) {
      uint32_t a[4];
      ldsm4(a, left + (mt * 16 + (lane & 15)) * kRawLd + ks * 16 + (lane >> 4) * 8);
#pragma unroll
      for (int j2 = 0; j2 < 4; ++j2) {
        if (j2 > mt) continue;
        uint32_t b[4];
        ldsm4(b, sm.k + (j2 * 16 + (lane >> 4) * 8 + (lane & 7)) * kRawLd + ks * 16 + ((lane >> 3) & 1) * 8);
        mma_16816(gram[2 * j2], a, b[0], b[1]);
        mma_16816(gram[2 * j2 + 1], a, b[2], b[3]);
      }
    }
    const float* rl = of_q ? sm.rq : sm.rk;
    const float lo = rl[row_lo], hi = rl[row_hi];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float c0 = sm.rk[j * 8 + 2 * t4], c1 = sm.rk[j * 8 + 2 * t4 + 1];
      gram[j][0] *= lo * c0;
      gram[j][1] *= lo * c1;
      gram[j][2] *= hi * c0;
      gram[j][3] *= hi * c1;
    }
  }

  for (int r = 0; r < rep; ++r) {
    const int hv = hq * rep + r;
    const size_t chunk = (static_cast<size_t>(batch) * gm.Hv + hv) * gm.N + n;
    load_raw_tile<kThreads>(mixed_b, gm, n, 2 * gm.Hqk * kD + hv * kD, sm.v);
    // gates, the cumulative sum by two warps; rows at or beyond T have beta = g = 0
    float beta = 0.f, G = 0.f;
    if (tid < kC) {
      const int t = n * kC + tid;
      if (t < gm.T) {
        const size_t off = (static_cast<size_t>(batch) * gm.T + t) * gm.Hv + hv;
        beta = sigmoid_f(bf2f(p.b_in + off));
        G = -expf(p.A_log[hv]) * softplus_f(bf2f(p.a_in + off) + p.dt_bias[hv]);
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, G, o);
        if (lane >= o) G += up;
      }
      if (tid == 31) sm.warp0_sum = G;
    }
    __syncthreads();
    if (tid < kC) {
      if (tid >= 32) G += sm.warp0_sum;
      const float eg = expf(G);
      sm.beta[tid] = beta;
      sm.G[tid] = G;
      sm.eg[tid] = eg;
      sm.kscale[tid] = beta * eg * sm.rk[tid];
    }
    __syncthreads();
    if (tid < kC) sm.ed[tid] = expf(sm.G[kC - 1] - sm.G[tid]);
    {
      const float G_lo = sm.G[row_lo], G_hi = sm.G[row_hi], b_lo = sm.beta[row_lo], b_hi = sm.beta[row_hi];
      __nv_bfloat16* intra = p.intra + chunk * kC * kC;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int c0 = j * 8 + 2 * t4, c1 = c0 + 1;
        const float2 Gc = *reinterpret_cast<const float2*>(sm.G + c0);
        if (of_q) {
          const float w00 = c0 <= row_lo ? gram[j][0] * expf(G_lo - Gc.x) : 0.f, w01 = c1 <= row_lo ? gram[j][1] * expf(G_lo - Gc.y) : 0.f;
          const float w10 = c0 <= row_hi ? gram[j][2] * expf(G_hi - Gc.x) : 0.f, w11 = c1 <= row_hi ? gram[j][3] * expf(G_hi - Gc.y) : 0.f;
          *reinterpret_cast<uint32_t*>(intra + row_lo * kC + c0) = pack_bf16x2(w00, w01);
          *reinterpret_cast<uint32_t*>(intra + row_hi * kC + c0) = pack_bf16x2(w10, w11);
        } else {
          const float a00 = c0 < row_lo ? b_lo * gram[j][0] * expf(G_lo - Gc.x) : 0.f, a01 = c1 < row_lo ? b_lo * gram[j][1] * expf(G_lo - Gc.y) : 0.f;
          const float a10 = c0 < row_hi ? b_hi * gram[j][2] * expf(G_hi - Gc.x) : 0.f, a11 = c1 < row_hi ? b_hi * gram[j][3] * expf(G_hi - Gc.y) : 0.f;
          *reinterpret_cast<float2*>(sm.A + row_lo * kALd + c0) = make_float2(a00, a01);
          *reinterpret_cast<float2*>(sm.A + row_hi * kALd + c0) = make_float2(a10, a11);
        }
      }
    }
    __syncthreads();
    unit_lower_inverse<kThreads>(sm.A, sm.T, sm.U);
    {
      // X = (T diag(s)) R: warps 0-3 the value columns (s = beta), warps 4-7 the key columns (s = beta exp(G) / |k|), 32 columns each
      const __nv_bfloat16* right = (of_q ? sm.k : sm.v) + mt * 32;
      const float* scale = of_q ? sm.kscale : sm.beta;
      __nv_bfloat16* out = (of_q ? p.kq + chunk * 2 * kC * kD : p.veff + chunk * kC * kD) + mt * 32;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        float acc[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          if (ks > m) continue;
          uint32_t part[3][4];
#pragma unroll
          for (int f = 0; f < 4; ++f) {     // fragment registers: rows g, g + 8, columns 2 t4 and 8 further
            const int row = m * 16 + g + (f & 1) * 8, col = ks * 16 + 2 * t4 + (f >> 1) * 8;
            float2 x = *reinterpret_cast<const float2*>(sm.T + row * kTLd + col);
            const float2 s = *reinterpret_cast<const float2*>(scale + col);
            x.x *= s.x;
            x.y *= s.y;
#pragma unroll
            for (int e = 0; e < 3; ++e) {
              part[e][f] = pack_bf16x2(x.x, x.y);
              const float2 h = unpack_bf16x2(part[e][f]);
              x.x -= h.x;
              x.y -= h.y;
            }
          }
#pragma unroll
          for (int j2 = 0; j2 < 2; ++j2) {
            uint32_t b[4];
            ldsm4_t(b, right + (ks * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * kRawLd + j2 * 16 + (lane >> 4) * 8);
#pragma unroll
            for (int e = 2; e >= 0; --e) {  // the small parts first
              mma_16816(acc[2 * j2], part[e], b[0], b[1]);
              mma_16816(acc[2 * j2 + 1], part[e], b[2], b[3]);
            }
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          *reinterpret_cast<uint32_t*>(out + (m * 16 + g) * kD + j * 8 + 2 * t4) = pack_bf16x2(acc[j][0], acc[j][1]);
          *reinterpret_cast<uint32_t*>(out + (m * 16 + g + 8) * kD + j * 8 + 2 * t4) = pack_bf16x2(acc[j][2], acc[j][3]);
        }
      }
    }
    for (int idx = tid; idx < kC * (kD / 8); idx += kThreads) {
      const int i = idx >> 4, c8 = idx & 15;
      const uint4 q8 = *reinterpret_cast<const uint4*>(sm.q + i * kRawLd + c8 * 8);
      const uint4 k8 = *reinterpret_cast<const uint4*>(sm.k + i * kRawLd + c8 * 8);
      const float rq = sm.rq[i], rk = sm.rk[i], eg = sm.eg[i], ed = sm.ed[i];
      const uint32_t qw[4] = {q8.x, q8.y, q8.z, q8.w}, kw[4] = {k8.x, k8.y, k8.z, k8.w};
      uint32_t qo[4], ko[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 x = unpack_bf16x2(qw[e]), y = unpack_bf16x2(kw[e]);
        qo[e] = pack_bf16x2(x.x * rq * eg, x.y * rq * eg);
        ko[e] = pack_bf16x2(y.x * rk * ed, y.y * rk * ed);
      }
      *reinterpret_cast<uint4*>(p.kq + (chunk * 2 * kC + kC + i) * kD + c8 * 8) = make_uint4(qo[0], qo[1], qo[2], qo[3]);
      *reinterpret_cast<uint4*>(p.kdec + (chunk * kC + i) * kD + c8 * 8) = make_uint4(ko[0], ko[1], ko[2], ko[3]);
    }
    if (tid == 0) p.e[chunk] = sm.eg[kC - 1];
    __syncthreads();
  }
}

struct PrepBwdArgs {
  const __nv_bfloat16* mixed;
  const __nv_bfloat16* b_in;
  const __nv_bfloat16* a_in;
  const float* A_log;
  const float* dt_bias;
  const __nv_bfloat16* d_kq;      // [B*Hv, N, 128, 128]: rows 0-63 d k_cum, rows 64-127 d q_e
  const __nv_bfloat16* d_intra;   // [B*Hv, N, 64, 64]
  const __nv_bfloat16* d_kdec;    // [B*Hv, N, 64, 128]
  const __nv_bfloat16* d_veff;    // [B*Hv, N, 64, 128]
  const float* d_e;               // [B*Hv, N]
  __nv_bfloat16* d_mixed;         // [B, T, conv_dim]
  float* d_b;                     // [B, T, Hv]
  float* d_a;                     // [B, T, Hv]
  float* d_A_log;                 // [Hv], accumulated
  float* d_dt_bias;               // [Hv], accumulated
  PrepGeom gm;
};

// ---- backward ----------------------------------------------------------------------------------------------------------
// With T = (I + A)^-1, X = T R and the incoming dX: Y = T^T dX is the gradient of the right-hand sides R, and that of A is
// -strict_lower(Y X^T) = -strict_lower(T^T (dX R^T) T^T), so X itself is not needed. dX and the raw rows of R are bf16, products with
// them are matrix instructions with an fp32 factor in three bf16 parts as in the forward kernel; the two 64 x 64 x 64 products with T
// on both sides are fp32. One CTA of 16 warps: the 64 x 128 sums of dQ and dK over the value heads stay in registers (warps 0-7 dQ, 8-15
// dK, a row tile and 64 columns each).
//
// The kernel before solved the two triangular systems with a column of 64 registers per thread and formed Y X^T and three products with
// dS, dW, dW^T on the CUDA cores, 800 us for 2048 tokens and 32 value heads; here 249 us. The terms
// of dG (the gates' cumulative sums) largely cancel: they are added up in 64 bits, which halves to quarters the error of d(A_log), d(dt_bias).
constexpr int kBwdThreads = 512;

struct PrepBwdSmem {
  __nv_bfloat16 q[kC * kRawLd], k[kC * kRawLd], v[kC * kRawLd], dxv[kC * kRawLd], dxk[kC * kRawLd];
  float A[kC * kALd], M0[kC * kALd], N[kC * kALd];     // M0: k^ k^T with the decays, strictly lower; A = beta M0; N = dX R^T
  float T[kC * kTLd], P[kC * kTLd], S[kC * kTLd], W[kC * kTLd], U[32 * kULd];   // P = N T^T; S = dS + dS^T; W = dW
  float beta[kC], g[kC], G[kC], eg[kC], ed[kC], asig[kC], rq[kC], rk[kC], kscale[kC];
  double dG[kC];                     // its terms largely cancel in the sums from a row to the end
  float dbeta[kC], dotq[kC], dotk[kC];
  float warp0_sum;
};
static_assert(sizeof(PrepBwdSmem) <= 227 * 1024, "shared memory");

__device__ __forceinline__ void load_chunk_tile(const __nv_bfloat16* src, __nv_bfloat16* dst) {   // 64 x 128, contiguous
  for (int i = threadIdx.x; i < kC * (kD / 8); i += kBwdThreads)
    *reinterpret_cast<uint4*>(dst + (i >> 4) * kRawLd + (i & 15) * 8) = reinterpret_cast<const uint4*>(src)[i];
}
template <class F>
__device__ __forceinline__ F quad_sum(F v) {     // over the four lanes that share a fragment's row
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}
__device__ __forceinline__ double column_sum(double v) {   // over the eight lanes that share a fragment's column
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  v += __shfl_xor_sync(0xffffffffu, v, 8);
  return v + __shfl_xor_sync(0xffffffffu, v, 16);
}

// The matrix unit cuts its sums off instead of rounding them: every step of 16 starts at zero and is added on with rounding.
__device__ __forceinline__ void add4(float (&acc)[4], const float (&x)[4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) acc[e] += x[e];
}
__device__ __forceinline__ void mma_add(float (&acc)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  float x[4] = {};
  mma_16816(x, a, b0, b1);
  add4(acc, x);
}

// acc (16 rows x 8 * NT columns of fragments) += left (16 x 16 per step, fp32 by `load(row, col)` = columns col, col + 1) right, over
// the steps [k0, k1) of 16; `right` points at the first of the columns in a raw tile.
template <int NT, class Load>
__device__ __forceinline__ void split_product(float (&acc)[NT][4], const Load& load, int k0, int k1, const __nv_bfloat16* right) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
#pragma unroll 1
  for (int ks = k0; ks < k1; ++ks) {
    uint32_t part[3][4];
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      float2 x = load(g + (f & 1) * 8, ks * 16 + 2 * t4 + (f >> 1) * 8);
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        part[e][f] = pack_bf16x2(x.x, x.y);
        const float2 h = unpack_bf16x2(part[e][f]);
        x.x -= h.x;
        x.y -= h.y;
      }
    }
#pragma unroll
    for (int j2 = 0; j2 < NT / 2; ++j2) {
      uint32_t b[4];
      ldsm4_t(b, right + (ks * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * kRawLd + j2 * 16 + (lane >> 4) * 8);
      float lo[4] = {}, hi[4] = {};
#pragma unroll
      for (int e = 2; e >= 0; --e) {  // the small parts first
        mma_16816(lo, part[e], b[0], b[1]);
        mma_16816(hi, part[e], b[2], b[3]);
      }
      add4(acc[2 * j2], lo);
      add4(acc[2 * j2 + 1], hi);
    }
  }
}

__global__ void __launch_bounds__(kBwdThreads, 1) gdn_chunk_prep_bwd_kernel(const PrepBwdArgs p) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  PrepBwdSmem& sm = *reinterpret_cast<PrepBwdSmem*>(smem_raw);
  const PrepGeom gm = p.gm;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const int n = blockIdx.x, hq = blockIdx.y, batch = blockIdx.z;
  const int rep = gm.Hv / gm.Hqk;
  const size_t tok0 = static_cast<size_t>(batch) * gm.T;
  const __nv_bfloat16* mixed_b = p.mixed + tok0 * gm.conv_dim;
  __nv_bfloat16* d_mixed_b = p.d_mixed + tok0 * gm.conv_dim;
  load_raw_tile<kBwdThreads>(mixed_b, gm, n, hq * kD, sm.q);
  load_raw_tile<kBwdThreads>(mixed_b, gm, n, gm.Hqk * kD + hq * kD, sm.k);
  __syncthreads();
  {
    // reciprocal norms, eight threads per row
    const int i = tid >> 3, qd = tid & 7;
    float ssq = 0.f, ssk = 0.f;
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const uint4 a = *reinterpret_cast<const uint4*>(sm.q + i * kRawLd + (qd + 8 * m) * 8);
      const uint4 b = *reinterpret_cast<const uint4*>(sm.k + i * kRawLd + (qd + 8 * m) * 8);
      const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 x = unpack_bf16x2(aw[e]), y = unpack_bf16x2(bw[e]);
        ssq += x.x * x.x + x.y * x.y;
        ssk += y.x * y.x + y.y * y.y;
      }
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      ssq += __shfl_xor_sync(0xffffffffu, ssq, o);
      ssk += __shfl_xor_sync(0xffffffffu, ssk, o);
    }
    if (qd == 0) {
      sm.rq[i] = rsqrtf(ssq + 1e-6f) * kQScale;
      sm.rk[i] = rsqrtf(ssk + 1e-6f);
    }
  }
  for (int i = tid; i < kC; i += kBwdThreads) sm.dotq[i] = sm.dotk[i] = 0.f;
  __syncthreads();
  const int mt = warp & 3, row_lo = mt * 16 + g, row_hi = row_lo + 8, part = (warp >> 2) & 1;
  const bool second = warp >= 8;     // Gram matrix of q^, key columns, dK; the first eight warps: of k^, value columns, dQ
  // Gram matrices (32 columns per warp, nothing above the diagonal)
  float gram[4][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) gram[j][0] = gram[j][1] = gram[j][2] = gram[j][3] = 0.f;
  {
    const __nv_bfloat16* left = second ? sm.q : sm.k;
#pragma unroll
    for (int ks = 0; ks < kD / 16; ++ks) {
      uint32_t a[4];
      ldsm4(a, left + (mt * 16 + (lane & 15)) * kRawLd + ks * 16 + (lane >> 4) * 8);
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        const int cb = part * 2 + jj;
        if (cb > mt) continue;
        uint32_t b[4];
        ldsm4(b, sm.k + (cb * 16 + (lane >> 4) * 8 + (lane & 7)) * kRawLd + ks * 16 + ((lane >> 3) & 1) * 8);
        mma_add(gram[2 * jj], a, b[0], b[1]);
        mma_add(gram[2 * jj + 1], a, b[2], b[3]);
      }
    }
    const float* rl = second ? sm.rq : sm.rk;
    const float lo = rl[row_lo], hi = rl[row_hi];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float c0 = sm.rk[part * 32 + j * 8 + 2 * t4], c1 = sm.rk[part * 32 + j * 8 + 2 * t4 + 1];
      gram[j][0] *= lo * c0;
      gram[j][1] *= lo * c1;
      gram[j][2] *= hi * c0;
      gram[j][3] *= hi * c1;
    }
  }
  float acc[8][4];                   // dQ (of the scaled q^) or dK: rows row_lo, row_hi, columns part * 64 + 8 j + 2 t4 (+ 1)
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;

  for (int r = 0; r < rep; ++r) {
    const int hv = hq * rep + r;
    const size_t chunk = (static_cast<size_t>(batch) * gm.Hv + hv) * gm.N + n;
    load_raw_tile<kBwdThreads>(mixed_b, gm, n, 2 * gm.Hqk * kD + hv * kD, sm.v);
    load_chunk_tile(p.d_veff + chunk * kC * kD, sm.dxv);
    load_chunk_tile(p.d_kq + chunk * 2 * kC * kD, sm.dxk);
    const float a_neg = -expf(p.A_log[hv]);
    float beta = 0.f, G = 0.f;
    if (tid < kC) {
      const int t = n * kC + tid;
      float asig = 0.f;
      if (t < gm.T) {
        const size_t off = (tok0 + t) * gm.Hv + hv;
        const float x = bf2f(p.a_in + off) + p.dt_bias[hv];
        beta = sigmoid_f(bf2f(p.b_in + off));
        G = a_neg * softplus_f(x);
        asig = sigmoid_f(x);
      }
      sm.g[tid] = G;
      sm.asig[tid] = asig;
      sm.dG[tid] = 0.;
      sm.dbeta[tid] = 0.f;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, G, o);
        if (lane >= o) G += up;
      }
      if (tid == 31) sm.warp0_sum = G;
    }
    __syncthreads();
    if (tid < kC) {
      if (tid >= 32) G += sm.warp0_sum;
      const float eg = expf(G);
      sm.beta[tid] = beta;
      sm.G[tid] = G;
      sm.eg[tid] = eg;
      sm.kscale[tid] = beta * eg * sm.rk[tid];
    }
    __syncthreads();
    if (tid < kC) sm.ed[tid] = expf(sm.G[kC - 1] - sm.G[tid]);
    {
      const float G_lo = sm.G[row_lo], G_hi = sm.G[row_hi], b_lo = sm.beta[row_lo], b_hi = sm.beta[row_hi];
      double e_lo = 0., e_hi = 0.;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c0 = part * 32 + j * 8 + 2 * t4, c1 = c0 + 1;
        const float2 Gc = *reinterpret_cast<const float2*>(sm.G + c0);
        // decays, zero above the diagonal
        const float d00 = c0 <= row_lo ? expf(G_lo - Gc.x) : 0.f, d01 = c1 <= row_lo ? expf(G_lo - Gc.y) : 0.f;
        const float d10 = c0 <= row_hi ? expf(G_hi - Gc.x) : 0.f, d11 = c1 <= row_hi ? expf(G_hi - Gc.y) : 0.f;
        if (second) {
          // W = q^ k^T D: dW = d_intra D, and d_intra W feeds dG (row sums minus column sums)
          const __nv_bfloat16* di = p.d_intra + chunk * kC * kC + c0;
          const float2 i0 = bf2f2(di + row_lo * kC), i1 = bf2f2(di + row_hi * kC);
          const float w00 = i0.x * d00, w01 = i0.y * d01, w10 = i1.x * d10, w11 = i1.y * d11;
          *reinterpret_cast<float2*>(sm.W + row_lo * kTLd + c0) = make_float2(w00, w01);
          *reinterpret_cast<float2*>(sm.W + row_hi * kTLd + c0) = make_float2(w10, w11);
          const double x00 = w00 * gram[j][0], x01 = w01 * gram[j][1], x10 = w10 * gram[j][2], x11 = w11 * gram[j][3];
          e_lo += x00 + x01;
          e_hi += x10 + x11;
          const double s0 = column_sum(x00 + x10), s1 = column_sum(x01 + x11);
          if (g == 0) {
            atomicAdd(sm.dG + c0, -s0);
            atomicAdd(sm.dG + c1, -s1);
          }
        } else {
          const float m00 = c0 < row_lo ? gram[j][0] * d00 : 0.f, m01 = c1 < row_lo ? gram[j][1] * d01 : 0.f;
          const float m10 = c0 < row_hi ? gram[j][2] * d10 : 0.f, m11 = c1 < row_hi ? gram[j][3] * d11 : 0.f;
          *reinterpret_cast<float2*>(sm.M0 + row_lo * kALd + c0) = make_float2(m00, m01);
          *reinterpret_cast<float2*>(sm.M0 + row_hi * kALd + c0) = make_float2(m10, m11);
          *reinterpret_cast<float2*>(sm.A + row_lo * kALd + c0) = make_float2(b_lo * m00, b_lo * m01);
          *reinterpret_cast<float2*>(sm.A + row_hi * kALd + c0) = make_float2(b_hi * m10, b_hi * m11);
        }
      }
      if (second) {
        e_lo = quad_sum(e_lo);
        e_hi = quad_sum(e_hi);
        if (t4 == 0) {
          atomicAdd(sm.dG + row_lo, e_lo);
          atomicAdd(sm.dG + row_hi, e_hi);
        }
      }
    }
    __syncthreads();
    unit_lower_inverse<kBwdThreads>(sm.A, sm.T, sm.U);
    {
      // N = dX_v V^T diag(beta) + dX_k K^T diag(beta exp(G) / |k|): 16 columns per warp
      const int c16 = (warp >> 2) * 16;
      float nv[2][4], nk[2][4];
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) nv[j][e] = nk[j][e] = 0.f;
#pragma unroll
      for (int ks = 0; ks < kD / 16; ++ks) {
        const int ao = (mt * 16 + (lane & 15)) * kRawLd + ks * 16 + (lane >> 4) * 8;
        const int bo = (c16 + (lane >> 4) * 8 + (lane & 7)) * kRawLd + ks * 16 + ((lane >> 3) & 1) * 8;
        uint32_t a[4], b[4];
        ldsm4(a, sm.dxv + ao);
        ldsm4(b, sm.v + bo);
        mma_add(nv[0], a, b[0], b[1]);
        mma_add(nv[1], a, b[2], b[3]);
        ldsm4(a, sm.dxk + ao);
        ldsm4(b, sm.k + bo);
        mma_add(nk[0], a, b[0], b[1]);
        mma_add(nk[1], a, b[2], b[3]);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int c0 = c16 + j * 8 + 2 * t4;
        const float2 sv = *reinterpret_cast<const float2*>(sm.beta + c0), sk = *reinterpret_cast<const float2*>(sm.kscale + c0);
        *reinterpret_cast<float2*>(sm.N + row_lo * kALd + c0) =
            make_float2(nv[j][0] * sv.x + nk[j][0] * sk.x, nv[j][1] * sv.y + nk[j][1] * sk.y);
        *reinterpret_cast<float2*>(sm.N + row_hi * kALd + c0) =
            make_float2(nv[j][2] * sv.x + nk[j][2] * sk.x, nv[j][3] * sv.y + nk[j][3] * sk.y);
      }
    }
    {
      // Y = T^T dX, 64 columns per warp in two halves. Values: dV = beta Y; keys: dK += beta exp(G) Y. The rows' products with the
      // right-hand sides' own factors (v, k^) go to the gates.
      auto t_transposed = [&](int row, int l) {
        const float* t = sm.T + l * kTLd + mt * 16 + row;
        return make_float2(t[0], t[kTLd]);
      };
      const float b_lo = sm.beta[row_lo], b_hi = sm.beta[row_hi], eb_lo = b_lo * sm.eg[row_lo], eb_hi = b_hi * sm.eg[row_hi];
      float u_lo = 0.f, u_hi = 0.f;
      const __nv_bfloat16* raw = second ? sm.k : sm.v;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int col = part * 64 + h * 32;
        float y[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) y[j][0] = y[j][1] = y[j][2] = y[j][3] = 0.f;
        split_product<4>(y, t_transposed, mt, 4, (second ? sm.dxk : sm.dxv) + col);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int c = col + j * 8 + 2 * t4;
          const float2 x0 = bf2f2(raw + row_lo * kRawLd + c), x1 = bf2f2(raw + row_hi * kRawLd + c);
          u_lo += y[j][0] * x0.x + y[j][1] * x0.y;
          u_hi += y[j][2] * x1.x + y[j][3] * x1.y;
          if (second) {
            acc[4 * h + j][0] += eb_lo * y[j][0];
            acc[4 * h + j][1] += eb_lo * y[j][1];
            acc[4 * h + j][2] += eb_hi * y[j][2];
            acc[4 * h + j][3] += eb_hi * y[j][3];
          } else {
            __nv_bfloat16* dv = d_mixed_b + 2 * gm.Hqk * kD + hv * kD + c;
            const int t = n * kC + row_lo;
            if (t < gm.T) *reinterpret_cast<uint32_t*>(dv + static_cast<size_t>(t) * gm.conv_dim) = pack_bf16x2(b_lo * y[j][0], b_lo * y[j][1]);
            if (t + 8 < gm.T) *reinterpret_cast<uint32_t*>(dv + static_cast<size_t>(t + 8) * gm.conv_dim) = pack_bf16x2(b_hi * y[j][2], b_hi * y[j][3]);
          }
        }
      }
      u_lo = quad_sum(u_lo);
      u_hi = quad_sum(u_hi);
      if (t4 == 0) {
        if (second) {
          const float k_lo = u_lo * sm.rk[row_lo], k_hi = u_hi * sm.rk[row_hi];
          atomicAdd(sm.dbeta + row_lo, sm.eg[row_lo] * k_lo);
          atomicAdd(sm.dbeta + row_hi, sm.eg[row_hi] * k_hi);
          atomicAdd(sm.dG + row_lo, static_cast<double>(eb_lo * k_lo));
          atomicAdd(sm.dG + row_hi, static_cast<double>(eb_hi * k_hi));
        } else {
          atomicAdd(sm.dbeta + row_lo, u_lo);
          atomicAdd(sm.dbeta + row_hi, u_hi);
        }
      }
    }
    __syncthreads();
    // dA = -strict_lower(T^T N T^T): thread (ti, tj) owns rows ti, ti + 32 and columns tj + 16 b
    const int ti = tid >> 4, tj = tid & 15;
    {
      float pr[2][4];
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) pr[a][b] = 0.f;
#pragma unroll
      for (int lb = 0; lb < 4; ++lb)
#pragma unroll
        for (int l = lb * 16; l < lb * 16 + 16; l += 4) {   // T_jl = 0 for l > j
          const float4 n0 = *reinterpret_cast<const float4*>(sm.N + ti * kALd + l), n1 = *reinterpret_cast<const float4*>(sm.N + (ti + 32) * kALd + l);
#pragma unroll
          for (int b = lb; b < 4; ++b) {
            const float4 t = *reinterpret_cast<const float4*>(sm.T + (tj + 16 * b) * kTLd + l);
            pr[0][b] += n0.x * t.x + n0.y * t.y + n0.z * t.z + n0.w * t.w;
            pr[1][b] += n1.x * t.x + n1.y * t.y + n1.z * t.z + n1.w * t.w;
          }
        }
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        sm.P[ti * kTLd + tj + 16 * b] = pr[0][b];
        sm.P[(ti + 32) * kTLd + tj + 16 * b] = pr[1][b];
      }
    }
    __syncthreads();
    {
      float da[2][4];
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) da[a][b] = 0.f;
#pragma unroll 4
      for (int l = warp * 2; l < 32; ++l) {                 // T_li = 0 for i > l; rows ti < 32 have no columns from 32 on
        const float t0 = sm.T[l * kTLd + ti];
#pragma unroll
        for (int b = 0; b < 2; ++b) da[0][b] = fmaf(-t0, sm.P[l * kTLd + tj + 16 * b], da[0][b]);
      }
#pragma unroll 4
      for (int l = 32; l < kC; ++l) {
        const float t0 = sm.T[l * kTLd + ti], t1 = sm.T[l * kTLd + ti + 32];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const float x = sm.P[l * kTLd + tj + 16 * b];
          if (b < 2) da[0][b] = fmaf(-t0, x, da[0][b]);
          da[1][b] = fmaf(-t1, x, da[1][b]);
        }
      }
      // dA A feeds dG (row sums minus column sums), dA M0 dbeta, dS = dA beta D the Gram matrix of k^
#pragma unroll
      for (int a = 0; a < 2; ++a) {
        const int i = ti + 32 * a;
        const float b_i = sm.beta[i], G_i = sm.G[i];
        double row_e = 0.;
        float row_b = 0.f;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int j = tj + 16 * b;
          const bool low = j < i;
          const float dA = low ? da[a][b] : 0.f, m0 = low ? sm.M0[i * kALd + j] : 0.f;
          const float x = dA * m0;
          const double E = x * b_i;
          row_e += E;
          row_b += x;
          const double col = E + __shfl_xor_sync(0xffffffffu, E, 16);   // the two rows of the warp
          if (lane < 16) atomicAdd(sm.dG + j, -col);
          const float dS = low ? dA * b_i * expf(G_i - sm.G[j]) : 0.f;
          if (j <= i) sm.S[i * kTLd + j] = dS;
          if (low) sm.S[j * kTLd + i] = dS;
        }
#pragma unroll
        for (int o = 8; o >= 1; o >>= 1) {
          row_e += __shfl_xor_sync(0xffffffffu, row_e, o);
          row_b += __shfl_xor_sync(0xffffffffu, row_b, o);
        }
        if (tj == 0) {
          atomicAdd(sm.dG + i, row_e);
          atomicAdd(sm.dbeta + i, row_b);
        }
      }
    }
    __syncthreads();
    {
      // dQ += dW K^ + exp(G) dq_e;  dK += (dS + dS^T) K^ + dW^T Q^ + exp(G_end - G) dk_dec; the raw rows' norms scale the left side
      const int col = part * 64;
      if (second) {
        auto s_left = [&](int row, int j) {
          const float2 s = *reinterpret_cast<const float2*>(sm.S + (mt * 16 + row) * kTLd + j), rk = *reinterpret_cast<const float2*>(sm.rk + j);
          return make_float2(s.x * rk.x, s.y * rk.y);
        };
        auto w_transposed = [&](int row, int j) {
          const float* w = sm.W + j * kTLd + mt * 16 + row;
          const float2 rq = *reinterpret_cast<const float2*>(sm.rq + j);
          return make_float2(w[0] * rq.x, w[kTLd] * rq.y);
        };
        split_product<8>(acc, s_left, 0, 4, sm.k + col);
        split_product<8>(acc, w_transposed, mt, 4, sm.q + col);
      } else {
        auto w_left = [&](int row, int j) {
          const float2 w = *reinterpret_cast<const float2*>(sm.W + (mt * 16 + row) * kTLd + j), rk = *reinterpret_cast<const float2*>(sm.rk + j);
          return make_float2(w.x * rk.x, w.y * rk.y);
        };
        split_product<8>(acc, w_left, 0, mt + 1, sm.k + col);
      }
      const __nv_bfloat16* grad = second ? p.d_kdec + chunk * kC * kD : p.d_kq + (chunk * 2 * kC + kC) * kD;
      const __nv_bfloat16* raw = second ? sm.k : sm.q;
      const float* dec = second ? sm.ed : sm.eg;
      const float d_lo = dec[row_lo], d_hi = dec[row_hi];
      float s_lo = 0.f, s_hi = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int c = col + j * 8 + 2 * t4;
        const float2 g0 = bf2f2(grad + row_lo * kD + c), g1 = bf2f2(grad + row_hi * kD + c);
        const float2 x0 = bf2f2(raw + row_lo * kRawLd + c), x1 = bf2f2(raw + row_hi * kRawLd + c);
        s_lo += g0.x * x0.x + g0.y * x0.y;
        s_hi += g1.x * x1.x + g1.y * x1.y;
        acc[j][0] += d_lo * g0.x;
        acc[j][1] += d_lo * g0.y;
        acc[j][2] += d_hi * g1.x;
        acc[j][3] += d_hi * g1.y;
      }
      const float* norm = second ? sm.rk : sm.rq;
      s_lo = quad_sum(s_lo) * norm[row_lo] * d_lo;
      s_hi = quad_sum(s_hi) * norm[row_hi] * d_hi;
      if (t4 == 0) {
        atomicAdd(sm.dG + row_lo, static_cast<double>(second ? -s_lo : s_lo));
        atomicAdd(sm.dG + row_hi, static_cast<double>(second ? -s_hi : s_hi));
        if (second) atomicAdd(sm.dG + kC - 1, static_cast<double>(s_lo) + s_hi);
      }
      if (tid == 0) atomicAdd(sm.dG + kC - 1, static_cast<double>(p.d_e[chunk] * sm.eg[kC - 1]));
    }
    __syncthreads();
    // gates: dg = reverse cumulative sum of dG; g = -exp(A_log) softplus(a + dt_bias); beta = sigmoid(b)
    if (tid < kC) {
      double dg_sum = 0.;
      for (int m = tid; m < kC; ++m) dg_sum += sm.dG[m];
      const float dg = static_cast<float>(dg_sum);
      const int t = n * kC + tid;
      float d_alog = 0.f, d_dtb = 0.f;
      if (t < gm.T) {
        const size_t off = (tok0 + t) * gm.Hv + hv;
        const float d_a = dg * a_neg * sm.asig[tid], be = sm.beta[tid];
        p.d_a[off] = d_a;
        p.d_b[off] = sm.dbeta[tid] * be * (1.f - be);
        d_alog = dg * sm.g[tid];
        d_dtb = d_a;
      }
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) {
        d_alog += __shfl_xor_sync(0xffffffffu, d_alog, o);
        d_dtb += __shfl_xor_sync(0xffffffffu, d_dtb, o);
      }
      if ((tid & 31) == 0) {
        atomicAdd(p.d_A_log + hv, d_alog);
        atomicAdd(p.d_dt_bias + hv, d_dtb);
      }
    }
    __syncthreads();
  }

  // through the L2 norms: y = s x r, r = rsqrt(sum x^2 + eps), s = dk^-1/2 for q and 1 for k  =>  dx = s r dy - x r^2 (y . dy)
  {
    const __nv_bfloat16* raw = second ? sm.k : sm.q;
    const float* norm = second ? sm.rk : sm.rq;
    float* dots = second ? sm.dotk : sm.dotq;
    float s_lo = 0.f, s_hi = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int c = part * 64 + j * 8 + 2 * t4;
      const float2 x0 = bf2f2(raw + row_lo * kRawLd + c), x1 = bf2f2(raw + row_hi * kRawLd + c);
      s_lo += acc[j][0] * x0.x + acc[j][1] * x0.y;
      s_hi += acc[j][2] * x1.x + acc[j][3] * x1.y;
    }
    s_lo = quad_sum(s_lo);
    s_hi = quad_sum(s_hi);
    if (t4 == 0) {
      atomicAdd(dots + row_lo, s_lo);
      atomicAdd(dots + row_hi, s_hi);
    }
    __syncthreads();
    // r = norm / s: r^2 (y . dy) = norm^3 / s^2 (x . dy)
    const float inv_s2 = second ? 1.f : 1.f / (kQScale * kQScale);
    const float n_lo = norm[row_lo], n_hi = norm[row_hi];
    const float f_lo = n_lo * n_lo * n_lo * inv_s2 * dots[row_lo], f_hi = n_hi * n_hi * n_hi * inv_s2 * dots[row_hi];
    const int t = n * kC + row_lo;
    __nv_bfloat16* out = d_mixed_b + static_cast<size_t>(t) * gm.conv_dim + (second ? gm.Hqk * kD : 0) + hq * kD;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int c = part * 64 + j * 8 + 2 * t4;
      const float2 x0 = bf2f2(raw + row_lo * kRawLd + c), x1 = bf2f2(raw + row_hi * kRawLd + c);
      if (t < gm.T) *reinterpret_cast<uint32_t*>(out + c) = pack_bf16x2(n_lo * acc[j][0] - x0.x * f_lo, n_lo * acc[j][1] - x0.y * f_lo);
      if (t + 8 < gm.T)
        *reinterpret_cast<uint32_t*>(out + 8 * static_cast<size_t>(gm.conv_dim) + c) =
            pack_bf16x2(n_hi * acc[j][2] - x1.x * f_hi, n_hi * acc[j][3] - x1.y * f_hi);
    }
  }
}

bool prep_geom_ok(int B, int T, int Hqk, int Hv) { return B >= 1 && T >= 1 && Hqk >= 1 && Hv >= Hqk && Hv % Hqk == 0; }

}  // namespace

cudaError_t launch_gdn_chunk_prep(const __nv_bfloat16* mixed, const __nv_bfloat16* b_in, const __nv_bfloat16* a_in,
                                  const float* A_log, const float* dt_bias, __nv_bfloat16* kq, __nv_bfloat16* intra,
                                  __nv_bfloat16* kdec, __nv_bfloat16* veff, float* e, int B, int T, int Hqk, int Hv,
                                  cudaStream_t stream) {
  if (!prep_geom_ok(B, T, Hqk, Hv)) return cudaErrorInvalidValue;
  const int N = (T + kC - 1) / kC;
  constexpr int smem = sizeof(PrepFwdSmem);
  static bool configured = false;
  if (!configured) {
    cudaError_t err = cudaFuncSetAttribute(gdn_chunk_prep_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (err != cudaSuccess) return err;
    configured = true;
  }
  PrepFwdArgs args{mixed, b_in, a_in, A_log, dt_bias, kq, intra, kdec, veff, e, {T, N, Hqk, Hv, (2 * Hqk + Hv) * kD}};
  gdn_chunk_prep_fwd_kernel<<<dim3(N, Hqk, B), kThreads, smem, stream>>>(args);
  return cudaGetLastError();
}

cudaError_t launch_gdn_chunk_prep_bwd(const __nv_bfloat16* mixed, const __nv_bfloat16* b_in, const __nv_bfloat16* a_in,
                                      const float* A_log, const float* dt_bias, const __nv_bfloat16* d_kq,
                                      const __nv_bfloat16* d_intra, const __nv_bfloat16* d_kdec,
                                      const __nv_bfloat16* d_veff, const float* d_e, __nv_bfloat16* d_mixed, float* d_b,
                                      float* d_a, float* d_A_log, float* d_dt_bias, int B, int T, int Hqk, int Hv,
                                      cudaStream_t stream) {
  if (!prep_geom_ok(B, T, Hqk, Hv)) return cudaErrorInvalidValue;
  const int N = (T + kC - 1) / kC;
  constexpr int smem = sizeof(PrepBwdSmem);
  static bool configured = false;
  if (!configured) {
    cudaError_t err = cudaFuncSetAttribute(gdn_chunk_prep_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (err != cudaSuccess) return err;
    configured = true;
  }
  PrepBwdArgs args{mixed, b_in, a_in, A_log, dt_bias, d_kq, d_intra, d_kdec, d_veff, d_e,
                   d_mixed, d_b, d_a, d_A_log, d_dt_bias, {T, N, Hqk, Hv, (2 * Hqk + Hv) * kD}};
  gdn_chunk_prep_bwd_kernel<<<dim3(N, Hqk, B), kBwdThreads, smem, stream>>>(args);
  return cudaGetLastError();
}

}  // namespace b200
