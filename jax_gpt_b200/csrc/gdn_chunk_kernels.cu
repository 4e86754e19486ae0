// Gated-DeltaNet prefill: everything of the chunked gated delta rule that does NOT depend on the running state,
// forward and backward, as one kernel each (fp32 on the CUDA cores, no library call).
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
// One CTA of 256 threads owns one (batch, q/k head, chunk) and loops over the value heads that share the q/k head:
// the normalised q and k tiles stay in shared memory as fp32, the 64 x 64 Gram matrices are computed by a 16 x 16
// thread grid (4 x 4 interleaved entries each), and the unit-lower-triangular solve is a forward substitution with
// one right-hand-side COLUMN per thread held in 64 registers (256 columns = 256 threads), so it needs no barriers.
//
// The backward kernel recomputes the forward quantities from the same inputs, solves the transposed system
// Y = (I + A)^-T dX by backward substitution (again one column per thread), forms dA = -strict_lower(Y X^T), and
// pushes the gradients through the decays, the gates, the Gram matrices and the two L2 norms down to d(mixed),
// d(b), d(a), d(A_log) and d(dt_bias). Gradients of q and k are summed over the value heads on chip, so the kernel
// has no global atomics except the two per-head scalars. Those 2 x 64 x 128 fp32 sums are thread-private (64 values
// per thread) but must survive the substitution phases, which need every register for the 64-entry columns; shared
// memory is full, so they are parked in tensor memory (tcgen05.st / tcgen05.ld, 128 columns) between the phases.
#include "seq_kernels.cuh"

#include "common.cuh"

namespace b200 {

namespace {

constexpr int kC = 64;            // chunk length
constexpr int kD = 128;           // dk = dv
constexpr int kLd = kD + 4;       // row stride (floats) of the 64 x 128 fp32 tiles in shared memory
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
__device__ __forceinline__ float dot4(const float4& a, const float4& b) { return a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w; }

// Loads the chunk's q and k rows (bf16, 128 wide each) as fp32 into sq / sk, L2-normalises every row (q is also
// scaled by dk^-1/2) and leaves the reciprocal norms in s_rq / s_rk. Rows at or beyond T become zero.
__device__ void load_qk_normalised(const __nv_bfloat16* mixed_b, const PrepGeom& gm, int n, int hq, float* sq, float* sk,
                                   float* s_rq, float* s_rk) {
  const int tid = threadIdx.x;
  for (int idx = tid; idx < 2 * kC * 16; idx += kThreads) {
    const int which = idx / (kC * 16), rem = idx % (kC * 16);
    const int i = rem / 16, v8 = rem % 16;
    const int t = n * kC + i;
    float* dst = (which ? sk : sq) + i * kLd + v8 * 8;
    if (t < gm.T) {
      const uint4 raw = *reinterpret_cast<const uint4*>(mixed_b + static_cast<size_t>(t) * gm.conv_dim +
                                                        which * gm.Hqk * kD + hq * kD + v8 * 8);
      const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = __bfloat1622float2(p[e]);
        dst[2 * e] = f.x;
        dst[2 * e + 1] = f.y;
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) dst[e] = 0.f;
    }
  }
  __syncthreads();
  const int i = tid >> 2, qd = tid & 3;
  float ssq = 0.f, ssk = 0.f;
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    const float2 a = *reinterpret_cast<const float2*>(sq + i * kLd + 2 * (qd + 4 * m));
    const float2 b = *reinterpret_cast<const float2*>(sk + i * kLd + 2 * (qd + 4 * m));
    ssq += a.x * a.x + a.y * a.y;
    ssk += b.x * b.x + b.y * b.y;
  }
  ssq += __shfl_xor_sync(0xffffffffu, ssq, 1);
  ssq += __shfl_xor_sync(0xffffffffu, ssq, 2);
  ssk += __shfl_xor_sync(0xffffffffu, ssk, 1);
  ssk += __shfl_xor_sync(0xffffffffu, ssk, 2);
  const float rq = rsqrtf(ssq + 1e-6f), rk = rsqrtf(ssk + 1e-6f);
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    float2* a = reinterpret_cast<float2*>(sq + i * kLd + 2 * (qd + 4 * m));
    float2* b = reinterpret_cast<float2*>(sk + i * kLd + 2 * (qd + 4 * m));
    a->x *= rq * kQScale;
    a->y *= rq * kQScale;
    b->x *= rk;
    b->y *= rk;
  }
  if (qd == 0) {
    s_rq[i] = rq;
    s_rk[i] = rk;
  }
  __syncthreads();
}

// Thread (ti, tj) of the 16 x 16 grid owns entries (ti + 16 a, tj + 16 b): s = k^ k^T, w = q^ k^T. Entries above
// the diagonal are never used, so block columns b > a are skipped.
__device__ __forceinline__ void gram_blocks(const float* sq, const float* sk, int ti, int tj, float (&s)[4][4],
                                            float (&w)[4][4]) {
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) s[a][b] = w[a][b] = 0.f;
#pragma unroll 2
  for (int c = 0; c < kD; c += 4) {
    float4 ki[4], qi[4], kj[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      ki[a] = *reinterpret_cast<const float4*>(sk + (ti + 16 * a) * kLd + c);
      qi[a] = *reinterpret_cast<const float4*>(sq + (ti + 16 * a) * kLd + c);
      kj[a] = *reinterpret_cast<const float4*>(sk + (tj + 16 * a) * kLd + c);
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b)
        if (b <= a) {
          s[a][b] += dot4(ki[a], kj[b]);
          w[a][b] += dot4(qi[a], kj[b]);
        }
  }
}

// Gates of one value head for the 64 rows of the chunk (threads 0..63 compute, everybody leaves synchronised):
// s_beta, s_g (raw log-decay), s_G (inclusive cumulative sum), s_eg = exp(G), s_ed = exp(G_end - G), s_asig =
// sigmoid(a + dt_bias) (the derivative of the softplus). Rows at or beyond T have beta = g = 0.
__device__ void chunk_gates(const __nv_bfloat16* b_in, const __nv_bfloat16* a_in, float a_neg, float dtb,
                            const PrepGeom& gm, int batch, int n, int hv, float* s_beta, float* s_g, float* s_G,
                            float* s_eg, float* s_ed, float* s_asig) {
  const int tid = threadIdx.x;
  if (tid < kC) {
    const int t = n * kC + tid;
    float beta = 0.f, g = 0.f, asig = 0.f;
    if (t < gm.T) {
      const size_t off = (static_cast<size_t>(batch) * gm.T + t) * gm.Hv + hv;
      beta = sigmoid_f(bf2f(b_in + off));
      const float x = bf2f(a_in + off) + dtb;
      g = a_neg * softplus_f(x);
      asig = sigmoid_f(x);
    }
    s_beta[tid] = beta;
    s_g[tid] = g;
    s_asig[tid] = asig;
  }
  __syncthreads();
  if (tid < kC) {
    float G = 0.f;
    for (int j = 0; j <= tid; ++j) G += s_g[j];
    s_G[tid] = G;
  }
  __syncthreads();
  if (tid < kC) {
    s_eg[tid] = expf(s_G[tid]);
    s_ed[tid] = expf(s_G[kC - 1] - s_G[tid]);
  }
  __syncthreads();
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
__device__ __forceinline__ void load_raw_tile(const __nv_bfloat16* mixed_b, const PrepGeom& gm, int n, int col, __nv_bfloat16* dst) {
#pragma unroll
  for (int i = threadIdx.x; i < kC * (kD / 8); i += kThreads) {
    const int r = i >> 4, c8 = i & 15, t = n * kC + r;
    uint4 u = make_uint4(0, 0, 0, 0);
    if (t < gm.T) u = *reinterpret_cast<const uint4*>(mixed_b + static_cast<size_t>(t) * gm.conv_dim + col + c8 * 8);
    *reinterpret_cast<uint4*>(dst + r * kRawLd + c8 * 8) = u;
  }
}

// out (rows x cols) = sign * a (rows x inner) b (inner x cols), fp32 in shared memory, a thread per output, rows * cols a multiple
// of the block; `blocks` such products, the operands a step apart.
template <int kRows, int kCols, int kInner>
__device__ __forceinline__ void small_product(float* out, int ldo, const float* a, int lda, const float* b, int ldb, float sign,
                                              int blocks, int out_step, int a_step, int b_step) {
  const int per = kRows * kCols;
  for (int o = threadIdx.x; o < blocks * per; o += kThreads) {
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
    for (int i = tid - 128; i < 512; i += 128) {   // the blocks right of the first and of the third on the diagonal
      const int r = (i >> 8) * 32 + ((i >> 4) & 15), c = (i >> 8) * 32 + 16 + (i & 15);
      T[r * kTLd + c] = 0.f;
    }
  }
  __syncthreads();
  small_product<16, 16, 16>(U, kULd, A + 16 * kALd, kALd, T, kTLd, 1.f, 2, 16 * kULd, 32 * kALd + 32, 32 * kTLd + 32);
  __syncthreads();
  small_product<16, 16, 16>(T + 16 * kTLd, kTLd, T + 16 * kTLd + 16, kTLd, U, kULd, -1.f, 2, 32 * kTLd + 32, 32 * kTLd + 32, 16 * kULd);
  __syncthreads();
  small_product<32, 32, 32>(U, kULd, A + 32 * kALd, kALd, T, kTLd, 1.f, 1, 0, 0, 0);
  __syncthreads();
  small_product<32, 32, 32>(T + 32 * kTLd, kTLd, T + 32 * kTLd + 32, kTLd, U, kULd, -1.f, 1, 0, 0, 0);
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
  load_raw_tile(mixed_b, gm, n, hq * kD, sm.q);
  load_raw_tile(mixed_b, gm, n, gm.Hqk * kD + hq * kD, sm.k);
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
    load_raw_tile(mixed_b, gm, n, 2 * gm.Hqk * kD + hv * kD, sm.v);
    // gates (see chunk_gates), the cumulative sum by two warps
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
    unit_lower_inverse(sm.A, sm.T, sm.U);
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

constexpr int kBwdSmemFloats = 4 * kC * kLd + 3 * kC * kC + 10 * kC + 4;

__global__ void __launch_bounds__(kThreads, 1) gdn_chunk_prep_bwd_kernel(const PrepBwdArgs p) {
  extern __shared__ __align__(16) float smem[];
  float* sq = smem;
  float* sk = sq + kC * kLd;
  float* sX = sk + kC * kLd;
  float* sY = sX + kC * kLd;
  float* sM0 = sY + kC * kLd;        // k^ k^T * decay (strict lower), later dS + dS^T
  float* sM1 = sM0 + kC * kC;        // q^ k^T * decay (lower), later dW
  float* sM2 = sM1 + kC * kC;        // dW^T
  float* s_beta = sM2 + kC * kC;
  float* s_g = s_beta + kC;
  float* s_G = s_g + kC;
  float* s_eg = s_G + kC;
  float* s_ed = s_eg + kC;
  float* s_asig = s_ed + kC;
  float* s_rq = s_asig + kC;
  float* s_rk = s_rq + kC;
  float* s_dG = s_rk + kC;
  float* s_dbeta = s_dG + kC;
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(s_dbeta + kC);
  const PrepGeom gm = p.gm;
  const int tid = threadIdx.x, n = blockIdx.x, hq = blockIdx.y, batch = blockIdx.z;
  const int rep = gm.Hv / gm.Hqk;
  const size_t tok0 = static_cast<size_t>(batch) * gm.T;
  const __nv_bfloat16* mixed_b = p.mixed + tok0 * gm.conv_dim;
  __nv_bfloat16* d_mixed_b = p.d_mixed + tok0 * gm.conv_dim;
  load_qk_normalised(mixed_b, gm, n, hq, sq, sk, s_rq, s_rk);
  const int ti = tid >> 4, tj = tid & 15;     // Gram-matrix mapping
  const int ri = tid >> 2, rqd = tid & 3;     // row mapping: row ri, column pairs rqd + 4 m
  const int cc = tid & 127, hb = tid >> 7;    // column mapping: column cc, rows 2 m + hb
  // gradients of the scaled q^ and of k^, summed over the value heads: parked in tensor memory, this thread's lane
  // (warp % 4 selects the lane quadrant) and 64 columns (dq: 0-31, dk: 32-63 of the warp's column group)
  if (tid < 32) {
    tmem_alloc(s_tmem, 128);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t park = *s_tmem + ((static_cast<uint32_t>((tid >> 5) & 3) * 32u) << 16) + static_cast<uint32_t>(tid >> 7) * 64u;
  {
    uint32_t z[32];
#pragma unroll
    for (int m = 0; m < 32; ++m) z[m] = 0u;
    tmem_st_32x32(park, z);
    tmem_st_32x32(park + 32, z);
    tmem_st_wait();
  }

  for (int r = 0; r < rep; ++r) {
    const int hv = hq * rep + r;
    const size_t chunk = (static_cast<size_t>(batch) * gm.Hv + hv) * gm.N + n;
    const float a_neg = -expf(p.A_log[hv]);
    chunk_gates(p.b_in, p.a_in, a_neg, p.dt_bias[hv], gm, batch, n, hv, s_beta, s_g, s_G, s_eg, s_ed, s_asig);
    if (tid < kC) s_dG[tid] = s_dbeta[tid] = 0.f;
    {
      float s[4][4], w[4][4];
      gram_blocks(sq, sk, ti, tj, s, w);
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int i = ti + 16 * a, j = tj + 16 * b;
          const float D = j <= i ? expf(s_G[i] - s_G[j]) : 0.f;
          sM0[i * kC + j] = j < i ? s[a][b] * D : 0.f;
          sM1[i * kC + j] = j <= i ? w[a][b] * D : 0.f;
        }
    }
    __syncthreads();

    float da[4][4];                            // dA of this thread's Gram entries
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) da[a][b] = 0.f;

#pragma unroll 1
    for (int h = 0; h < 2; ++h) {              // h = 0: the value columns, h = 1: the key columns of the solve
      // The two substitutions of a pass are independent (X needs the right-hand side, Y the incoming gradient):
      // threads 0-127 solve the columns of X while threads 128-255 solve the columns of Y.
      if (tid < 128) {
        const int c = tid;
        float x[kC];
        if (h == 0) {
          const __nv_bfloat16* vp = mixed_b + 2 * gm.Hqk * kD + hv * kD + c;
#pragma unroll
          for (int i = 0; i < kC; ++i) {
            const int t = n * kC + i;
            x[i] = t < gm.T ? s_beta[i] * bf2f(vp + static_cast<size_t>(t) * gm.conv_dim) : 0.f;
          }
        } else {
#pragma unroll
          for (int i = 0; i < kC; ++i) x[i] = s_beta[i] * s_eg[i] * sk[i * kLd + c];
        }
        // X = (I + A)^-1 R with A_ij = beta_i M0_ij
#pragma unroll
        for (int i = 1; i < kC; ++i) {
          float acc = 0.f;
#pragma unroll
          for (int j4 = 0; j4 * 4 < i; ++j4) {
            const float4 m = *reinterpret_cast<const float4*>(sM0 + i * kC + 4 * j4);
            acc += m.x * x[4 * j4] + m.y * x[4 * j4 + 1] + m.z * x[4 * j4 + 2] + m.w * x[4 * j4 + 3];
          }
          x[i] -= s_beta[i] * acc;
        }
#pragma unroll
        for (int i = 0; i < kC; ++i) sX[i * kLd + c] = x[i];
      } else {
        const int c = tid - 128;
        float x[kC];
        // Y = (I + A)^-T dX, right-looking: once y_j is final, y_i -= A_ji y_j for every i < j
        const __nv_bfloat16* dxp = h == 0 ? p.d_veff + chunk * kC * kD + c : p.d_kq + chunk * 2 * kC * kD + c;
#pragma unroll
        for (int i = 0; i < kC; ++i) x[i] = bf2f(dxp + i * kD);
#pragma unroll
        for (int j = kC - 1; j >= 1; --j) {
          const float t = s_beta[j] * x[j];
#pragma unroll
          for (int i4 = 0; i4 * 4 < j; ++i4) {
            const float4 m = *reinterpret_cast<const float4*>(sM0 + j * kC + 4 * i4);
            x[4 * i4] -= m.x * t;
            x[4 * i4 + 1] -= m.y * t;
            x[4 * i4 + 2] -= m.z * t;
            x[4 * i4 + 3] -= m.w * t;
          }
        }
#pragma unroll
        for (int i = 0; i < kC; ++i) sY[i * kLd + c] = x[i];
        if (h == 0) {
          __nv_bfloat16* dvp = d_mixed_b + 2 * gm.Hqk * kD + hv * kD + c;
#pragma unroll
          for (int i = 0; i < kC; ++i) {
            const int t = n * kC + i;
            if (t < gm.T) dvp[static_cast<size_t>(t) * gm.conv_dim] = __float2bfloat16(s_beta[i] * x[i]);
          }
        }
      }
      __syncthreads();
      // dA -= Y X^T on this thread's entries
#pragma unroll 2
      for (int c = 0; c < kD; c += 4) {
        float4 yi[4], xj[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          yi[a] = *reinterpret_cast<const float4*>(sY + (ti + 16 * a) * kLd + c);
          xj[a] = *reinterpret_cast<const float4*>(sX + (tj + 16 * a) * kLd + c);
        }
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b)
            if (b <= a) da[a][b] -= dot4(yi[a], xj[b]);
      }
      // per-row dot products of Y with the right-hand side's own factor (v, or k^)
      {
        float u = 0.f;
        const int t = n * kC + ri;
        if (h == 0) {
          if (t < gm.T) {
            const __nv_bfloat16* vp = mixed_b + static_cast<size_t>(t) * gm.conv_dim + 2 * gm.Hqk * kD + hv * kD;
#pragma unroll
            for (int m = 0; m < 16; ++m) {
              const float2 y2 = *reinterpret_cast<const float2*>(sY + ri * kLd + 2 * (rqd + 4 * m));
              const float2 v2 = bf2f2(vp + 2 * (rqd + 4 * m));
              u += y2.x * v2.x + y2.y * v2.y;
            }
          }
        } else {
#pragma unroll
          for (int m = 0; m < 16; ++m) {
            const float2 y2 = *reinterpret_cast<const float2*>(sY + ri * kLd + 2 * (rqd + 4 * m));
            const float2 k2 = *reinterpret_cast<const float2*>(sk + ri * kLd + 2 * (rqd + 4 * m));
            u += y2.x * k2.x + y2.y * k2.y;
          }
        }
        u += __shfl_xor_sync(0xffffffffu, u, 1);
        u += __shfl_xor_sync(0xffffffffu, u, 2);
        if (rqd == 0) {
          if (h == 0) {
            atomicAdd(s_dbeta + ri, u);
          } else {
            atomicAdd(s_dbeta + ri, s_eg[ri] * u);
            atomicAdd(s_dG + ri, s_beta[ri] * s_eg[ri] * u);
          }
        }
      }
      __syncthreads();
    }

    // through the decayed Gram matrices: E = dA * A + d_intra * intra feeds dG (row sums minus column sums);
    // dS = dA beta D and dW = d_intra D go to q^ and k^ through three 64 x 64 x 128 products
    {
      float m0[4][4], m1[4][4], di[4][4];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int i = ti + 16 * a, j = tj + 16 * b;
          m0[a][b] = sM0[i * kC + j];
          m1[a][b] = sM1[i * kC + j];
          di[a][b] = j <= i ? bf2f(p.d_intra + (chunk * kC + i) * kC + j) : 0.f;
        }
      __syncthreads();      // every entry is in registers before the mirrored writes start
      float row_e[4], row_b[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        row_e[a] = row_b[a] = 0.f;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int i = ti + 16 * a, j = tj + 16 * b;
          if (j > i) continue;               // the mirror entry's owner writes this position
          const float D = expf(s_G[i] - s_G[j]);
          const float dA = j < i ? da[a][b] : 0.f;
          const float E = dA * s_beta[i] * m0[a][b] + di[a][b] * m1[a][b];
          row_e[a] += E;
          atomicAdd(s_dG + j, -E);
          row_b[a] += dA * m0[a][b];
          const float dS = dA * s_beta[i] * D;
          const float dW = di[a][b] * D;
          sM0[i * kC + j] = dS;
          sM0[j * kC + i] = dS;
          sM1[i * kC + j] = dW;
          sM2[j * kC + i] = dW;
          if (j < i) {
            sM1[j * kC + i] = 0.f;
            sM2[i * kC + j] = 0.f;
          }
        }
      }
#pragma unroll
      for (int a = 0; a < 4; ++a) {
#pragma unroll
        for (int o = 8; o >= 1; o >>= 1) {
          row_e[a] += __shfl_xor_sync(0xffffffffu, row_e[a], o);
          row_b[a] += __shfl_xor_sync(0xffffffffu, row_b[a], o);
        }
        if (tj == 0) {
          atomicAdd(s_dG + ti + 16 * a, row_e[a]);
          atomicAdd(s_dbeta + ti + 16 * a, row_b[a]);
        }
      }
    }
    __syncthreads();
    float dq[32], dk[32];
    {
      uint32_t v[32];
      tmem_ld_32x32(park, v);
      tmem_ld_wait();
#pragma unroll
      for (int m = 0; m < 32; ++m) dq[m] = __uint_as_float(v[m]);
      tmem_ld_32x32(park + 32, v);
      tmem_ld_wait();
#pragma unroll
      for (int m = 0; m < 32; ++m) {
        const int i = 2 * m + hb;
        dk[m] = __uint_as_float(v[m]) + s_beta[i] * s_eg[i] * sY[i * kLd + cc];   // sY: the key half of Y
      }
    }
    {
      float col[kC];
#pragma unroll
      for (int j = 0; j < kC; ++j) col[j] = sk[j * kLd + cc];
#pragma unroll
      for (int m = 0; m < 32; ++m) {
        const int i = 2 * m + hb;
        float a0 = 0.f, a1 = 0.f;
#pragma unroll
        for (int j4 = 0; j4 < 16; ++j4) {
          const float4 s4 = *reinterpret_cast<const float4*>(sM0 + i * kC + 4 * j4);
          const float4 w4 = *reinterpret_cast<const float4*>(sM1 + i * kC + 4 * j4);
          a0 += s4.x * col[4 * j4] + s4.y * col[4 * j4 + 1] + s4.z * col[4 * j4 + 2] + s4.w * col[4 * j4 + 3];
          a1 += w4.x * col[4 * j4] + w4.y * col[4 * j4 + 1] + w4.z * col[4 * j4 + 2] + w4.w * col[4 * j4 + 3];
        }
        dk[m] += a0;
        dq[m] += a1;
      }
#pragma unroll
      for (int j = 0; j < kC; ++j) col[j] = sq[j * kLd + cc];
#pragma unroll
      for (int m = 0; m < 32; ++m) {
        const int i = 2 * m + hb;
        float a0 = 0.f;
#pragma unroll
        for (int j4 = 0; j4 < 16; ++j4) {
          const float4 t4 = *reinterpret_cast<const float4*>(sM2 + i * kC + 4 * j4);
          a0 += t4.x * col[4 * j4] + t4.y * col[4 * j4 + 1] + t4.z * col[4 * j4 + 2] + t4.w * col[4 * j4 + 3];
        }
        dk[m] += a0;
      }
    }
    // q_e = q^ exp(G), k_dec = k^ exp(G_end - G), e = exp(G_end)
    {
      const __nv_bfloat16* dqe = p.d_kq + (chunk * 2 * kC + kC) * kD;
      const __nv_bfloat16* dkd = p.d_kdec + chunk * kC * kD;
      float s1 = 0.f, s2 = 0.f;
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        const int c2 = 2 * (rqd + 4 * m);
        const float2 g1 = bf2f2(dqe + ri * kD + c2), g2 = bf2f2(dkd + ri * kD + c2);
        const float2 q2 = *reinterpret_cast<const float2*>(sq + ri * kLd + c2);
        const float2 k2 = *reinterpret_cast<const float2*>(sk + ri * kLd + c2);
        s1 += g1.x * q2.x + g1.y * q2.y;
        s2 += g2.x * k2.x + g2.y * k2.y;
      }
      s1 += __shfl_xor_sync(0xffffffffu, s1, 1);
      s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
      s2 += __shfl_xor_sync(0xffffffffu, s2, 1);
      s2 += __shfl_xor_sync(0xffffffffu, s2, 2);
      if (rqd == 0) {
        const float t = s_ed[ri] * s2;
        atomicAdd(s_dG + ri, s_eg[ri] * s1 - t);
        atomicAdd(s_dG + kC - 1, t);
      }
      if (tid == 0) atomicAdd(s_dG + kC - 1, p.d_e[chunk] * s_eg[kC - 1]);
#pragma unroll
      for (int m = 0; m < 32; ++m) {
        const int i = 2 * m + hb;
        dq[m] += s_eg[i] * bf2f(dqe + i * kD + cc);
        dk[m] += s_ed[i] * bf2f(dkd + i * kD + cc);
      }
    }
    if (r + 1 < rep) {
      uint32_t v[32];
#pragma unroll
      for (int m = 0; m < 32; ++m) v[m] = __float_as_uint(dq[m]);
      tmem_st_32x32(park, v);
#pragma unroll
      for (int m = 0; m < 32; ++m) v[m] = __float_as_uint(dk[m]);
      tmem_st_32x32(park + 32, v);
      tmem_st_wait();
    } else {
      // last value head: straight to shared memory for the L2-norm backward (sX is free; sY still feeds nothing)
#pragma unroll
      for (int m = 0; m < 32; ++m) sX[(2 * m + hb) * kLd + cc] = dq[m];
      __syncthreads();      // every thread has read the key half of Y out of sY
#pragma unroll
      for (int m = 0; m < 32; ++m) sY[(2 * m + hb) * kLd + cc] = dk[m];
    }
    __syncthreads();
    // gates: dg = reverse cumulative sum of dG; g = -exp(A_log) softplus(a + dt_bias); beta = sigmoid(b)
    if (tid < kC) {
      float dg = 0.f;
      for (int m = tid; m < kC; ++m) dg += s_dG[m];
      const int t = n * kC + tid;
      float d_alog = 0.f, d_dtb = 0.f;
      if (t < gm.T) {
        const size_t off = (tok0 + t) * gm.Hv + hv;
        const float d_a = dg * a_neg * s_asig[tid];
        const float beta = s_beta[tid];
        p.d_a[off] = d_a;
        p.d_b[off] = s_dbeta[tid] * beta * (1.f - beta);
        d_alog = dg * s_g[tid];
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

  // through the L2 norms: y = x r, r = rsqrt(sum x^2 + eps)  =>  dx = r (dy - y (y . dy))
  {
    float dotq = 0.f, dotk = 0.f;
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int c2 = 2 * (rqd + 4 * m);
      const float2 gq = *reinterpret_cast<const float2*>(sX + ri * kLd + c2);
      const float2 gk = *reinterpret_cast<const float2*>(sY + ri * kLd + c2);
      const float2 q2 = *reinterpret_cast<const float2*>(sq + ri * kLd + c2);
      const float2 k2 = *reinterpret_cast<const float2*>(sk + ri * kLd + c2);
      dotq += gq.x * q2.x + gq.y * q2.y;
      dotk += gk.x * k2.x + gk.y * k2.y;
    }
    dotq += __shfl_xor_sync(0xffffffffu, dotq, 1);
    dotq += __shfl_xor_sync(0xffffffffu, dotq, 2);
    dotk += __shfl_xor_sync(0xffffffffu, dotk, 1);
    dotk += __shfl_xor_sync(0xffffffffu, dotk, 2);
    const int t = n * kC + ri;
    if (t < gm.T) {
      const float rq = s_rq[ri], rk = s_rk[ri];
      __nv_bfloat16* oq = d_mixed_b + static_cast<size_t>(t) * gm.conv_dim + hq * kD;
      __nv_bfloat16* ok = oq + gm.Hqk * kD;
      // sq holds q^ s (s = dk^-1/2): d q^ = s dQ, q^ (q^ . d q^) = sq (sq . dQ) / s
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        const int c2 = 2 * (rqd + 4 * m);
        const float2 gq = *reinterpret_cast<const float2*>(sX + ri * kLd + c2);
        const float2 gk = *reinterpret_cast<const float2*>(sY + ri * kLd + c2);
        const float2 q2 = *reinterpret_cast<const float2*>(sq + ri * kLd + c2);
        const float2 k2 = *reinterpret_cast<const float2*>(sk + ri * kLd + c2);
        *reinterpret_cast<__nv_bfloat162*>(oq + c2) = __floats2bfloat162_rn(
            rq * (kQScale * gq.x - q2.x * dotq / kQScale), rq * (kQScale * gq.y - q2.y * dotq / kQScale));
        *reinterpret_cast<__nv_bfloat162*>(ok + c2) =
            __floats2bfloat162_rn(rk * (gk.x - k2.x * dotk), rk * (gk.y - k2.y * dotk));
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid < 32) tmem_dealloc(*s_tmem, 128);
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
  constexpr int smem = kBwdSmemFloats * 4;
  static bool configured = false;
  if (!configured) {
    cudaError_t err = cudaFuncSetAttribute(gdn_chunk_prep_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (err != cudaSuccess) return err;
    configured = true;
  }
  PrepBwdArgs args{mixed, b_in, a_in, A_log, dt_bias, d_kq, d_intra, d_kdec, d_veff, d_e,
                   d_mixed, d_b, d_a, d_A_log, d_dt_bias, {T, N, Hqk, Hv, (2 * Hqk + Hv) * kD}};
  gdn_chunk_prep_bwd_kernel<<<dim3(N, Hqk, B), kThreads, smem, stream>>>(args);
  return cudaGetLastError();
}

}  // namespace b200
