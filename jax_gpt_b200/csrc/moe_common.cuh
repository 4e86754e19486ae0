// Pieces shared by the expert-parallel MoE kernels (moe_kernels.cu, moe_fp8_kernels.cu): the
// shared-memory routing tables built from the all-gathered pair counts, the static tile order,
// bounded counter waits and the release/acquire helpers of the arrival protocol.
#pragma once
#include "common.cuh"
#include "moe_kernels.cuh"

namespace b200 {

namespace {

constexpr int kMoeBM = 128, kMoeBN = 256;

struct MoeTables {
  int send_off[kMoeMaxExperts];      // first row of MY pairs for global expert e in its destination buffer
  int rows[kMoeMaxLocalExperts];     // rows received per local expert
  int base[kMoeMaxLocalExperts];     // first row of the local expert in this rank's receive buffer
  // Static tile order, cut into n_slots = EL + lag slots; tile0[s] is the first tile of slot s. Forward: slot s
  // holds the GEMM1 (gate|up) tiles of expert s followed by the GEMM2 (down) tiles of expert s - lag. Backward:
  // slot s holds the dAct and dW_down tiles of expert s followed by the dX and dW_gate|up tiles of expert s - lag
  // (the ones that wait for that expert's dAct tiles). The lag keeps about two rounds of tiles between producer
  // and consumer tiles, so that CTAs working side by side in the order do not stall on one another.
  int tile0[2 * kMoeMaxLocalExperts + 1];
  int lag, n_slots;
  int mt0[kMoeMaxLocalExperts + 1];    // first m-tile index of the local expert
  int scan[32];                        // scratch of block_scan; while the tables are built, a word per rank
  int overflow;                      // some rank would receive more rows than cap_rows
};


__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

__device__ __forceinline__ unsigned ld_acquire_gpu_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned ld_acquire_sys_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_sys_add_u32(unsigned* p, unsigned v) {
  asm volatile("red.release.sys.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void red_relaxed_sys_add_u32(unsigned* p, unsigned v) {
  asm volatile("red.relaxed.sys.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Bounded wait until *p (cumulative counter) has reached `target` (wrap-safe signed difference).
template <bool kSystem>
__device__ __forceinline__ bool wait_counter_ge(const unsigned* p, unsigned target, uint64_t budget_ns,
                                                volatile int* abort_flag) {
  const uint64_t t0 = globaltimer_ns();
  while (true) {
    const unsigned v = kSystem ? ld_acquire_sys_u32(p) : ld_acquire_gpu_u32(p);
    if (static_cast<int>(v - target) >= 0) return true;
    if (*abort_flag) return false;
    if (globaltimer_ns() - t0 > budget_ns) {
      *abort_flag = 1;
      return false;
    }
    __nanosleep(32);
  }
}


// ---- the static tile order, from tb->rows: the pieces that the host and the device build it from ----

__host__ __device__ __forceinline__ int pad_rows(int rows, int pad) { return (rows + pad - 1) / pad * pad; }
__host__ __device__ __forceinline__ int m_tiles(int rows) { return (rows + kMoeBM - 1) / kMoeBM; }

// Tiles that an expert with `mt` m-tiles puts into its own slot (front) and into the slot `lag` later (back).
template <class Args>
__host__ __device__ __forceinline__ int front_tiles(const Args& a, int mt, bool backward) {
  if (!backward) return mt * (a.inter / 128);
  return mt > 0 ? mt * (a.inter / kMoeBN) + (a.inter / kMoeBM) * (a.d_model / kMoeBN) : 0;
}
template <class Args>
__host__ __device__ __forceinline__ int back_tiles(const Args& a, int mt, bool backward) {
  const int n2 = a.d_model / kMoeBN;
  if (!backward) return mt * n2;
  return mt > 0 ? mt * n2 + (a.d_model / kMoeBM) * (2 * a.inter / kMoeBN) : 0;
}

// Lag in experts: while one producer tile runs, the grid claims about grid_ctas * (its cost / average cost) tiles; three
// times that, plus the tiles the CTAs claim ahead of their load warps, at the average number of tiles per expert. The cost
// of a tile is in 64-deep K blocks, plus a few blocks' worth of epilogue: the tiles other tiles wait for (GEMM1 / dAct,
// full-depth K) take longer than the average tile, and the lag has to cover their duration. `mt`, `padded`, `active`:
// m-tiles, padded rows and experts with rows, over all experts.
template <class Args>
__host__ __device__ __forceinline__ int order_lag(const Args& a, int mt, int padded, int active, bool backward, int claim_ahead,
                                                  int grid_ctas) {
  const int EL = a.e_local, n1 = a.inter / 128, n2 = a.d_model / kMoeBN;
  const int over = 6, prod = a.d_model / 64 + over + (backward ? 4 : 0);
  int64_t t, cost;
  if (!backward) {
    t = static_cast<int64_t>(mt) * (n1 + n2);
    cost = static_cast<int64_t>(mt) * (n1 * prod + n2 * (a.inter / 64 + over));
  } else {
    // dAct tiles, dX tiles, dW_down and dW_gate|up tiles
    const int q0 = a.inter / kMoeBN, q23 = (a.inter / kMoeBM) * n2 + (a.d_model / kMoeBM) * (2 * a.inter / kMoeBN);
    t = static_cast<int64_t>(mt) * (q0 + n2) + static_cast<int64_t>(active) * q23;
    cost = static_cast<int64_t>(mt) * (q0 * prod + n2 * (2 * a.inter / 64 + over)) +
           static_cast<int64_t>(q23) * (padded / 64 + static_cast<int64_t>(active) * over);
  }
  int lag = 1;
  if (t > 0) {
    const float lag_tiles = static_cast<float>(grid_ctas) * (3.f * prod * static_cast<float>(t) / static_cast<float>(cost) + claim_ahead);
    lag = static_cast<int>(lag_tiles * EL / static_cast<float>(t)) + 1;
  }
  return lag < 1 ? 1 : (lag > EL ? EL : lag);
}

template <class Args>
__host__ __device__ __forceinline__ int slot_tiles(const Args& a, const int* rows, int sl, int lag, bool backward) {
  return (sl < a.e_local ? front_tiles(a, m_tiles(rows[sl]), backward) : 0) +
         (sl >= lag ? back_tiles(a, m_tiles(rows[sl - lag]), backward) : 0);
}

// The regions of the local experts in the receive buffer (base), their m-tile numbering (mt0) and the order itself (lag,
// n_slots, tile0), on the host: the tests walk it and compare build_tile_order_block with it.
template <class Args>
inline void build_tile_order(const Args& a, MoeTables* tb, bool backward, int pad, int claim_ahead, int grid_ctas) {
  const int EL = a.e_local;
  int padded = 0, mt = 0, active = 0;
  for (int el = 0; el < EL; ++el) {
    tb->base[el] = padded;
    tb->mt0[el] = mt;
    padded += pad_rows(tb->rows[el], pad);
    mt += m_tiles(tb->rows[el]);
    active += tb->rows[el] > 0;
  }
  tb->mt0[EL] = mt;
  tb->lag = order_lag(a, mt, padded, active, backward, claim_ahead, grid_ctas);
  tb->n_slots = EL + tb->lag;
  int u = 0;
  for (int sl = 0; sl < tb->n_slots; ++sl) {
    tb->tile0[sl] = u;
    u += slot_tiles(a, tb->rows, sl, tb->lag, backward);
  }
  tb->tile0[tb->n_slots] = u;
}

// Sum of `v` over the threads before this one; *total: over all. Every thread of the block calls it; `warp_sums` holds 32.
__device__ __forceinline__ int block_scan(int v, int* warp_sums, int* total) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = (blockDim.x + 31) >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int n = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += n;
  }
  __syncthreads();   // the sums of the scan before have been read
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  int before = 0, all = 0;
  for (int w = 0; w < warps; ++w) {
    const int n = warp_sums[w];
    before += w < warp ? n : 0;
    all += n;
  }
  *total = all;
  return before + incl - v;
}

// build_tile_order by a whole block (of whole warps): a few experts and slots a thread, sums over the block by scans. One
// thread walking them took 40 us of every launch with 512 experts (one token 111 -> 67 us, 32 tokens 331 -> 294 us).
template <class Args>
__device__ void build_tile_order_block(const Args& a, MoeTables* tb, bool backward, int pad, int claim_ahead, int grid_ctas) {
  const int EL = a.e_local, t = threadIdx.x, nt = blockDim.x;
  const int per = (EL + nt - 1) / nt, e0 = min(EL, t * per), e1 = min(EL, e0 + per);
  int p = 0, m = 0, act = 0, padded, mt, active;
  for (int el = e0; el < e1; ++el) {
    p += pad_rows(tb->rows[el], pad);
    m += m_tiles(tb->rows[el]);
    act += tb->rows[el] > 0;
  }
  p = block_scan(p, tb->scan, &padded);
  m = block_scan(m, tb->scan, &mt);
  block_scan(act, tb->scan, &active);
  for (int el = e0; el < e1; ++el) {
    tb->base[el] = p;
    tb->mt0[el] = m;
    p += pad_rows(tb->rows[el], pad);
    m += m_tiles(tb->rows[el]);
  }
  const int lag = order_lag(a, mt, padded, active, backward, claim_ahead, grid_ctas), n_slots = EL + lag;
  const int pers = (n_slots + nt - 1) / nt, s0 = min(n_slots, t * pers), s1 = min(n_slots, s0 + pers);
  int u = 0, tiles;
  for (int sl = s0; sl < s1; ++sl) u += slot_tiles(a, tb->rows, sl, lag, backward);
  u = block_scan(u, tb->scan, &tiles);
  for (int sl = s0; sl < s1; ++sl) {
    tb->tile0[sl] = u;
    u += slot_tiles(a, tb->rows, sl, lag, backward);
  }
  if (t == 0) {
    tb->mt0[EL] = mt;
    tb->tile0[n_slots] = tiles;
    tb->lag = lag;
    tb->n_slots = n_slots;
  }
}

// Fills the shared-memory tables from the all-gathered count matrix counts[src][e].
template <class Args>
__device__ void build_tables(const Args& a, const int* counts_all, MoeTables* tb, bool backward = false, int pad = 64,
                             int claim_ahead = 0) {
  const int W = a.world, EL = a.e_local, ET = W * EL, t = threadIdx.x, nt = blockDim.x;
  if (t == 0) tb->overflow = 0;
  // Padded totals per global expert (every expert's region starts on a `pad`-row boundary; ragged-K weight gradients read whole
  // blocks and the padding rows are kept zero), scanned over all experts; less the sum before its destination's first expert and
  // plus the rows of the sources placed before this rank that is where this rank's rows of the expert go.
  const int per = (ET + nt - 1) / nt, e0 = min(ET, t * per), e1 = min(ET, e0 + per);
  int run = 0, total;
  for (int e = e0; e < e1; ++e) {
    int n = 0;
    for (int s = 0; s < W; ++s) n += __ldcg(counts_all + s * ET + e);
    const int el = e - a.rank * EL;
    if (el >= 0 && el < EL) tb->rows[el] = n;
    run += pad_rows(n, pad);
  }
  run = block_scan(run, tb->scan, &total);
  for (int e = e0; e < e1; ++e) {
    tb->send_off[e] = run;
    int n = 0;
    for (int s = 0; s < W; ++s) n += __ldcg(counts_all + s * ET + e);
    run += pad_rows(n, pad);
  }
  __syncthreads();
  int first = 0;
  if (t < W) {
    first = tb->send_off[t * EL];
    if ((t + 1 < W ? tb->send_off[(t + 1) * EL] : total) - first > a.cap_rows) tb->overflow = 1;
    tb->scan[t] = first;     // one word per destination rank
  }
  __syncthreads();
  for (int e = e0; e < e1; ++e) {
    int before = -tb->scan[e / EL];
    for (int s = 0; s < a.rank; ++s) before += __ldcg(counts_all + s * ET + e);
    tb->send_off[e] += before;
  }
  build_tile_order_block(a, tb, backward, pad, claim_ahead, static_cast<int>(gridDim.x));
  __syncthreads();
}

struct TileInfo {
  int el, m, n, phase;  // phase 0: GEMM1 (gate|up), 1: GEMM2 (down)
};

template <class Args>
__host__ __device__ __forceinline__ TileInfo decode_tile(const Args& a, const MoeTables* tb, int t) {
  const int n1 = a.inter / 128, n2 = a.d_model / kMoeBN;
  // first slot whose tile range ends after t (slots without tiles have empty ranges): binary search
  int sl = 0, hi = tb->n_slots - 1;
  while (sl < hi) {
    const int mid = (sl + hi) >> 1;
    if (tb->tile0[mid + 1] > t) hi = mid;
    else sl = mid + 1;
  }
  int r = t - tb->tile0[sl];
  const int g1 = (sl < a.e_local) ? ((tb->rows[sl] + kMoeBM - 1) / kMoeBM) * n1 : 0;
  TileInfo ti;
  if (r < g1) {
    const int mt = (tb->rows[sl] + kMoeBM - 1) / kMoeBM;
    ti.el = sl;
    ti.phase = 0;
    ti.m = r % mt;
    ti.n = r / mt;
  } else {
    r -= g1;
    ti.el = sl - tb->lag;
    const int mt = (tb->rows[ti.el] + kMoeBM - 1) / kMoeBM;
    ti.phase = 1;
    ti.m = r % mt;
    ti.n = r / mt;
  }
  return ti;
}


}  // namespace

}  // namespace b200
