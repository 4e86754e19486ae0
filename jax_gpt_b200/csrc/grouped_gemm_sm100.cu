// Grouped GEMM of gated experts for sm_100a: rows sorted by expert, weights (experts, out, in), the group ends on the device.
//
//   kGlu: act[r, c] = glu(w_row[r] (W_e xs[r])[c], w_row[r] (W_e xs[r])[I + c])       W_e (2 I, K), gate rows first
//   else: out[r, c] = (W_e xs[r])[c]                                                  W_e (C, K)
//
// The WEIGHTS are the 256 rows of the matrix instruction's tile and the tokens its columns, as many as the expert has (at most 256, in
// steps of 32): with the tokens as rows an expert of 351 rows on average would pay for 512. A pair of CTAs shares a tile, each
// stages 128 weight rows and half of the tokens. For the GLU the weight rows of a tile are taken as eight of the gate, the eight of the up
// projection that go with them, and so on (one 5-D tensor map reads them in that order): both operands of the activation lie in one
// warp, lane and lane ^ 8, and gate and up are never written out.
//
// Bound by the tensor pipe for many rows per expert, by the stream of the weights for few. 64 experts, width 2048, inner 1024, against the
// library's grouped GEMM (whose up projection leaves the activation to another 35 us kernel): 352 rows each 181 + 96 us (library 197 + 105),
// 512 rows 212 + 115 (215 + 114), 8 rows 86 + 46 (110 + 65; the weights alone take 83 + 41 us).
//
//   warp 0: TMA loads in both CTAs; warp 1: matrix instructions (leader) and tensor memory; warps 2 .. 9: epilogue (transposed through
//   shared memory so that a token's columns are stored together). Barriers as in the CTA-pair GEMM; every wait is bounded.
#include "common.cuh"
#include "cta_pair.cuh"
#include "gemm_sm100.cuh"
#include "serve_common.cuh"
#include "serve_kernels.cuh"
#include "tma_host.h"

namespace b200 {

namespace {

constexpr int kRows = 128;                 // weight rows per CTA
constexpr int kTokens = 256;               // token columns of a tile, at most
constexpr int kStep = 32;                  // ... in steps of this (two CTAs, 16 each)
constexpr int BK = 64;
constexpr int kStages = 6;
constexpr int kABytes = kRows * BK * 2, kBBytes = kTokens / 2 * BK * 2, kStageBytes = kABytes + kBBytes;
constexpr int kEpiWarps = 8, kEpiBytes = 32 * 64;   // per warp: 32 tokens of up to 32 columns
constexpr int kThreads = 64 + 32 * kEpiWarps;
constexpr int kMaxExperts = 1024;          // per launch

struct GroupedBars {
  uint64_t full[kStages], empty[kStages], tmem_full[2], tmem_empty[2];
  uint32_t tmem_base;
  int abort_flag, sums[kThreads / 32];
  int tile0[kMaxExperts + 1], row0[kMaxExperts + 1];   // first tile and first row of each expert
};
constexpr int kSmemBytes = kStages * kStageBytes + kEpiWarps * kEpiBytes + static_cast<int>(sizeof(GroupedBars)) + 1024;
static_assert(kSmemBytes <= 227 * 1024, "shared memory");

struct GroupedMaps {
  CUtensorMap w, x64, x16;                 // weights; token rows in boxes of 64 and of 16
};

// Token columns per tile of an expert with `rows` rows: as few tiles as there can be, of equal size.
__device__ __forceinline__ int tile_tokens(int rows, int nt) { return ((rows + nt - 1) / nt + kStep - 1) / kStep * kStep; }

struct GroupedTile {
  int e, m, n0, valid, n;                  // expert, weight block, first token row, its rows, columns of the instruction
};
__device__ __forceinline__ GroupedTile grouped_tile(const GroupedBars* bars, const GroupedArgs& a, int t) {
  int lo = 0, hi = a.experts - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (bars->tile0[mid + 1] > t) hi = mid;
    else lo = mid + 1;
  }
  const int start = bars->row0[lo], rows = bars->row0[lo + 1] - start;
  const int nt = (rows + kTokens - 1) / kTokens, r = t - bars->tile0[lo], step = tile_tokens(rows, nt), at = (r % nt) * step;
  const int valid = min(step, rows - at);
  return {a.expert0 + lo, r / nt, start + at, valid, (valid + kStep - 1) / kStep * kStep};
}

template <bool kGlu>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
grouped_gemm_kernel(const __grid_constant__ GroupedMaps tm, const __grid_constant__ GroupedArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* epi = smem + kStages * kStageBytes;
  GroupedBars* bars = reinterpret_cast<GroupedBars*>(epi + kEpiWarps * kEpiBytes);
  volatile int* abort_flag = &bars->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank()), pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->tmem_full[i], 1);
      mbar_init(&bars->tmem_empty[i], 2 * kEpiWarps);
    }
    bars->abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(&bars->tmem_base, 2 * kTokens);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers are initialised before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  let_dependents_start();
  wait_for_stream();

  // tiles per expert, summed up by the block: each thread a run of experts
  const int m_blocks = (a.cols + (kGlu ? kRows : 2 * kRows) - 1) / (kGlu ? kRows : 2 * kRows);
  {
    const int per = (a.experts + kThreads - 1) / kThreads, e0 = min(a.experts, static_cast<int>(threadIdx.x) * per), e1 = min(a.experts, e0 + per);
    auto end_of = [&](int e) { return a.expert0 + e >= 0 ? __ldg(a.ends + a.expert0 + e) : 0; };
    auto tiles_of = [&](int from, int to) { return (to - from + kTokens - 1) / kTokens * m_blocks; };
    int own = 0, from = end_of(e0 - 1);
    if (threadIdx.x == 0) bars->row0[0] = from;
    for (int e = e0; e < e1; ++e) {
      const int to = end_of(e);
      bars->row0[e + 1] = to;
      own += tiles_of(from, to);
      from = to;
    }
    int sum = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += up;
    }
    if (lane == 31) bars->sums[warp] = sum;
    __syncthreads();
    int at = sum - own, total = 0;
    for (int w = 0; w < kThreads / 32; ++w) {
      if (w < warp) at += bars->sums[w];
      total += bars->sums[w];
    }
    for (int e = e0; e < e1; ++e) {     // the rows' ends lie in shared memory since the barrier
      bars->tile0[e] = at;
      at += tiles_of(bars->row0[e], bars->row0[e + 1]);
    }
    if (threadIdx.x == 0) bars->tile0[a.experts] = total;
    __syncthreads();
  }
  const int num_tiles = bars->tile0[a.experts], total_kb = (a.K + BK - 1) / BK;

  if (warp == 0) {
    if (elect_one()) {
      const uint32_t full_leader = mapa_u32(smem_u32(&bars->full[0]), 0);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = pair; t < num_tiles && ok; t += n_pairs) {
        const GroupedTile tl = grouped_tile(bars, a, t);
        const int half = tl.n / 2, row0 = tl.n0 + rank * half;   // half: a multiple of 16, at most 128
        for (int kb = 0; kb < total_kb; ++kb) {
          if (!mbar_wait(&bars->empty[stage], phase ^ 1, abort_flag)) {
            report_status(a.status, kWaitEmptyTimeout, blockIdx.x, t, kb);
            ok = false;
            break;
          }
          uint8_t* sa = smem + stage * kStageBytes;
          uint8_t* sb = sa + kABytes;
          if (rank == 0) mbar_arrive_expect_tx(&bars->full[stage], 2 * (kABytes + half * BK * 2));
          const uint32_t fb = full_leader + stage * 8;
          if (kGlu) tma_load_5d_pair(sa, &tm.w, fb, kb * BK, 0, 0, tl.m * (kRows / 8) + rank * (kRows / 16), tl.e);
          else tma_load_3d_pair(sa, &tm.w, fb, kb * BK, tl.m * 2 * kRows + rank * kRows, tl.e);
          int r = 0;
          for (; r + 64 <= half; r += 64) tma_load_2d_pair(sb + r * BK * 2, &tm.x64, fb, kb * BK, row0 + r);
          for (; r < half; r += 16) tma_load_2d_pair(sb + r * BK * 2, &tm.x16, fb, kb * BK, row0 + r);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if ((!ok || *abort_flag) && rank == 0) {
        // unwinding: the copies of both CTAs still in flight get a bounded time to land before the pair meets at the exit
        for (int s = 0; s < kStages; ++s) {
          const uint32_t armed = (s < stage) ? phase : (phase ^ 1);
          const uint64_t t0 = globaltimer_ns();
          while (!mbar_try_wait(&bars->full[s], armed)) {
            if (globaltimer_ns() - t0 > 2000000ull) break;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {   // one thread waits and issues
      int stage = 0, iter = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = pair; t < num_tiles && ok; t += n_pairs, ++iter) {
        const GroupedTile tl = grouped_tile(bars, a, t);
        const uint32_t idesc = make_idesc(2 * kRows, tl.n, 0, 0, 1);
        const int acc = iter & 1;
        if (!mbar_wait(&bars->tmem_empty[acc], ((iter >> 1) & 1) ^ 1, abort_flag)) {
          report_status(a.status, kWaitTmemEmptyTimeout, blockIdx.x, t, iter);
          break;
        }
        tc_fence_after();
        for (int kb = 0; kb < total_kb; ++kb) {
          if (!mbar_wait(&bars->full[stage], phase, abort_flag)) {
            report_status(a.status, kWaitFullTimeout, blockIdx.x, t, kb);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * kStageBytes), sb = sa + kABytes;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma_bf16_pair(tmem_base + acc * kTokens, make_smem_desc(sa + k * 32, 16, 1024), make_smem_desc(sb + k * 32, 16, 1024), idesc,
                           (kb > 0 || k > 0) ? 1u : 0u);
          tc_commit_pair(&bars->empty[stage]);  // frees the stage in both CTAs
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) tc_commit_pair(&bars->tmem_full[acc]);
      }
    }
  } else {
    const int q = warp & 3;            // TMEM lane quarter this warp may read
    const int half = (warp - 2) >> 2;  // every other group of 32 tokens
    uint8_t* stg = epi + (warp - 2) * kEpiBytes;
    const uint32_t empty_leader = mapa_u32(smem_u32(&bars->tmem_empty[0]), 0);
    int iter = 0;
    for (int t = pair; t < num_tiles; t += n_pairs, ++iter) {
      const GroupedTile tl = grouped_tile(bars, a, t);
      const int acc = iter & 1;
      if (!mbar_wait(&bars->tmem_full[acc], (iter >> 1) & 1, abort_flag)) {
        if (lane == 0) report_status(a.status, kWaitTmemFullTimeout, blockIdx.x, t, iter);
        break;
      }
      __syncwarp();
      tc_fence_after();
      const uint32_t tacc = tmem_base + acc * kTokens + (static_cast<uint32_t>(q * 32) << 16);
      for (int c = half * 32; c < tl.valid; c += 64) {
        uint32_t v[32];
        tmem_ld_32x32(tacc + c, v);
        tmem_ld_wait();
        __nv_bfloat16* dst = a.out + static_cast<int64_t>(tl.n0 + c) * a.cols;
        if (kGlu) {
          // lanes 0-7 and 16-23 hold eight gate rows each, lane ^ 8 the up rows that go with them; the former finish the first 16 tokens, the
          // latter the other 16. A token's 16 columns are 32 bytes; the second half of the tokens lies 32 bytes further (other banks).
          const bool up = (lane & 8) != 0;
          const float w = (a.w_row != nullptr && c + lane < tl.valid) ? __ldg(a.w_row + tl.n0 + c + lane) : 1.f;
          const int col = (lane >> 4) * 8 + (lane & 7);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float mine = __uint_as_float(up ? v[16 + j] : v[j]);
            const float other = __shfl_xor_sync(0xffffffffu, __uint_as_float(up ? v[j] : v[16 + j]), 8);
            const int token = (up ? 16 : 0) + j;
            const float wt = __shfl_sync(0xffffffffu, w, token);
            const float h = clamped_glu(wt * (up ? other : mine), wt * (up ? mine : other), a.glu);
            *reinterpret_cast<__nv_bfloat16*>(stg + token * 32 + (up ? 32 : 0) + col * 2) = __float2bfloat16(h);
          }
          __syncwarp();
          const int col0 = tl.m * kRows + rank * (kRows / 2) + q * 16;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int token = i * 16 + (lane >> 1), cc = col0 + (lane & 1) * 8;
            if (c + token < tl.valid && cc < a.cols)
              *reinterpret_cast<uint4*>(dst + static_cast<int64_t>(token) * a.cols + cc) =
                  *reinterpret_cast<const uint4*>(stg + token * 32 + i * 32 + (lane & 1) * 16);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) *reinterpret_cast<__nv_bfloat16*>(stg + j * 64 + lane * 2) = __float2bfloat16(__uint_as_float(v[j]));
          __syncwarp();
          const int col0 = tl.m * 2 * kRows + rank * kRows + q * 32 + (lane & 3) * 8;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int token = i * 8 + (lane >> 2);
            if (c + token < tl.valid && col0 < a.cols)
              *reinterpret_cast<uint4*>(dst + static_cast<int64_t>(token) * a.cols + col0) =
                  *reinterpret_cast<const uint4*>(stg + token * 64 + (lane & 3) * 16);
          }
        }
        __syncwarp();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(empty_leader + acc * 8);
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // neither CTA leaves (or frees TMEM) while the other may still read its memory
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 2 * kTokens);
  }
}

}  // namespace

cudaError_t launch_grouped_gemm(const __nv_bfloat16* xs, const __nv_bfloat16* w, int64_t w_row_stride, int64_t w_expert_stride,
                                const GroupedArgs& args_in, bool glu, int rows, int n_experts, cudaStream_t st) {
  GroupedArgs a = args_in;
  if (rows < 0 || n_experts < 1 || a.K < 1 || a.cols < 1 || a.K % 8 != 0 || a.cols % 8 != 0) return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  GroupedMaps tm;
  cudaError_t err;
  const uint64_t K = a.K, ld = w_row_stride * 2ull, le = w_expert_stride * 2ull, C = a.cols;
  if (glu) err = encode_tma_5d(&tm.w, w, 2, {K, 8, 2, C / 8, static_cast<uint64_t>(n_experts)}, {ld, C * ld, 8 * ld, le}, {BK, 8, 2, kRows / 16, 1});
  else err = encode_tma_3d(&tm.w, w, 2, K, C, n_experts, ld, le, BK, kRows, 1);
  if (err != cudaSuccess) return err;
  if ((err = encode_tma_2d(&tm.x64, xs, 2, K, rows, K * 2, BK, 64)) != cudaSuccess) return err;
  if ((err = encode_tma_2d(&tm.x16, xs, 2, K, rows, K * 2, BK, 16)) != cudaSuccess) return err;
  auto kernel = glu ? grouped_gemm_kernel<true> : grouped_gemm_kernel<false>;
  static bool configured[2] = {false, false};
  if (!configured[glu]) {
    if ((err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes)) != cudaSuccess) return err;
    configured[glu] = true;
  }
  const int m_blocks = (a.cols + (glu ? kRows : 2 * kRows) - 1) / (glu ? kRows : 2 * kRows);
  for (a.expert0 = 0; a.expert0 < n_experts; a.expert0 += kMaxExperts) {
    a.experts = n_experts - a.expert0 < kMaxExperts ? n_experts - a.expert0 : kMaxExperts;
    const int64_t tiles = static_cast<int64_t>(m_blocks) * (rows / kTokens + (rows < a.experts ? rows : a.experts));   // at most
    const int max_pairs = gemm_sm_count() / 2;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2 * static_cast<unsigned>(tiles < max_pairs ? tiles : max_pairs));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr = dependent_launch();
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if ((err = cudaLaunchKernelEx(&cfg, kernel, tm, a)) != cudaSuccess) return err;
  }
  return cudaGetLastError();
}

}  // namespace b200
