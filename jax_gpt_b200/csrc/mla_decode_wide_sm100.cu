// Paged MLA decode for many heads (65 and more): the heads are the M side of both products.
//
// A CTA owns 128 heads of one sequence, a range of its pages and HALF of the 512 latent columns of the output:
//     S [128 heads x 64 tokens]   = Q[128 x 576] . C^T            (both halves compute it)
//     O [128 heads x 256 latents] += P[128 x 64] . C[:, half]     (accumulator stays in TMEM)
// One page is one tile. Nine 64-column chunks of it: the four of the CTA's own half serve as K and as V and are held until the
// output product is done (three slots of 32 KB), the other five (other half, rotary part) are released chunk by chunk as soon as
// the score product has read them (six slots of 8 KB). Tensor memory: O 256 columns, two score buffers of 64 (the probabilities
// overwrite their scores), and the own half of Q, 128 columns, as the A operand; the other five chunks of Q lie in shared memory.
// A lane of the softmax warps owns a head, so the row maximum and sum need no exchange; O is rescaled only where the maximum
// grew by more than 2^8 since the last time.
//
// What bounds it: the score product, computed by both halves (36 + 16 tcgen05 steps a tile, about 1660 cycles at 128 x 64), with
// the loads of one tile and the softmax of the next behind it. The transposed kernel of mla_decode_sm100.cu keeps O in registers
// and has 32 heads a CTA: its chain load -> scores -> softmax over lanes -> output is exposed for every tile and 128 heads read
// each page four times.
// 64 sequences of 2048 tokens, 128 heads: 328 us there and 10 us of merge, 54 us here without one.
#include "mla_decode_sm100.cuh"

#include <math.h>

#include "common.cuh"
#include "tma_host.h"

namespace b200 {

namespace {

constexpr int kTok = kMlaPage;                   // tokens per tile
constexpr int kHeadRows = 128;
constexpr int kThreads = 192;                    // producer, MMA issuer, four softmax warps
constexpr int kChunkBytes = kTok * 128;          // 64 tokens x 64 bf16
constexpr int kQChunkBytes = kHeadRows * 128;
constexpr int kFreeChunks = 5;                   // chunks that only the score product reads
constexpr int kHeldChunks = 4;                   // own half: K and V
constexpr int kFreeSlots = 6, kHeldSlots = 3;
constexpr int kHeldBytes = kHeldChunks * kChunkBytes;
constexpr int kColO = 0, kColS = 256, kColQ = 384, kTmemCols = 512;
constexpr float kRescale = 8.f;                  // log2 growth of the maximum that the accumulator tolerates

struct WideSmem {
  uint64_t free_full[kFreeSlots], free_empty[kFreeSlots], held_full[kHeldSlots], held_empty[kHeldSlots];
  uint64_t s_full[2], p_ready[2], pv_done, q_full, q_tmem;
  uint32_t tmem_base;
  int abort_flag;
};

constexpr int kSmemBytes =
    1024 + kFreeChunks * kQChunkBytes + kHeldSlots * kHeldBytes + kFreeSlots * kChunkBytes + static_cast<int>(sizeof(WideSmem));
static_assert(kSmemBytes <= 227 * 1024, "shared memory");

// chunk i of Q and of a page that only the score product reads: the other half's four, then the rotary part
__device__ __forceinline__ int free_chunk(int i, int half) { return i < 4 ? (half ^ 1) * 4 + i : 8; }

__global__ void __launch_bounds__(kThreads, 1)
mla_decode_wide_kernel(const __grid_constant__ CUtensorMap t_pool, const __grid_constant__ CUtensorMap t_q,
                       const __nv_bfloat16* __restrict__ q_rows, const __grid_constant__ MlaDecodeArgs a,
                       __nv_bfloat16* __restrict__ out) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* qs = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* held = qs + kFreeChunks * kQChunkBytes;
  uint8_t* fre = held + kHeldSlots * kHeldBytes;
  WideSmem* sh = reinterpret_cast<WideSmem*>(fre + kFreeSlots * kChunkBytes);
  volatile int* abort_flag = &sh->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = blockIdx.x & 1, split = blockIdx.x >> 1, n_parts = gridDim.x >> 1;
  const int hb = blockIdx.y, b = blockIdx.z;
  const int sid = a.seq_ids[b];
  const int len = a.seq_lens[sid];
  const int first = a.window > 0 ? max(0, len - a.window) : 0;   // first token seen
  const int tile0 = first / kTok, n_tiles = (len + kTok - 1) / kTok - tile0;
  const int t0 = tile0 + static_cast<int>(static_cast<int64_t>(n_tiles) * split / n_parts);
  const int t1 = tile0 + static_cast<int>(static_cast<int64_t>(n_tiles) * (split + 1) / n_parts);
  const int n_it = t1 - t0;
  const int h0 = hb * kHeadRows;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kFreeSlots; ++i) {
      mbar_init(&sh->free_full[i], 1);
      mbar_init(&sh->free_empty[i], 1);
    }
    for (int i = 0; i < kHeldSlots; ++i) {
      mbar_init(&sh->held_full[i], 1);
      mbar_init(&sh->held_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sh->s_full[i], 1);
      mbar_init(&sh->p_ready[i], 128);
    }
    mbar_init(&sh->pv_done, 1);
    mbar_init(&sh->q_full, 1);
    mbar_init(&sh->q_tmem, 128);
    sh->abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(&sh->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh->tmem_base;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (n_it > 0 && elect_one()) {
      const int* bt = a.block_table + static_cast<int64_t>(sid) * a.max_pages;
      auto page_of = [&](int it) { return it < n_it && t0 + it < a.max_pages ? bt[t0 + it] : -1; };
      int page = page_of(0);
      mbar_arrive_expect_tx(&sh->q_full, kFreeChunks * kQChunkBytes);
      for (int i = 0; i < kFreeChunks; ++i)
        tma_load_2d(qs + i * kQChunkBytes, &t_q, &sh->q_full, free_chunk(i, half) * 64, b * a.heads + h0);
      int n_free = 0, n_held = 0;     // fills so far
      int slot = 0, use = 0;          // of the free ring
      bool ok = true;
      for (int it = 0; it < n_it && ok; ++it) {
        if (page < 0 || !bounds_ok(page, a.n_pages, a.status, 222)) {  // a sequence longer than its page list: give up cleanly
          report_status(a.status, kBadArgument, 71, b, t0 + it);
          *abort_flag = 1;
          ok = false;
          break;
        }
        const int next = page_of(it + 1);
        for (int i = 0; i < kFreeChunks; ++i) {
          if (use > 0 && !mbar_wait(&sh->free_empty[slot], (use - 1) & 1, abort_flag)) {
            report_status(a.status, kWaitEmptyTimeout, 78, b, it);
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(&sh->free_full[slot], kChunkBytes);
          tma_load_2d(fre + slot * kChunkBytes, &t_pool, &sh->free_full[slot], free_chunk(i, half) * 64, page * kMlaPage);
          ++n_free;
          if (++slot == kFreeSlots) {
            slot = 0;
            ++use;
          }
        }
        if (!ok) break;
        const int hs = it % kHeldSlots, hu = it / kHeldSlots;
        if (hu > 0 && !mbar_wait(&sh->held_empty[hs], (hu - 1) & 1, abort_flag)) {
          report_status(a.status, kWaitEmptyTimeout, 79, b, it);
          ok = false;
          break;
        }
        mbar_arrive_expect_tx(&sh->held_full[hs], kHeldBytes);
        for (int i = 0; i < kHeldChunks; ++i)
          tma_load_2d(held + hs * kHeldBytes + i * kChunkBytes, &t_pool, &sh->held_full[hs], (half * 4 + i) * 64, page * kMlaPage);
        ++n_held;
        page = next;
      }
      if (!ok || *abort_flag) {
        // leave no bulk copy in flight: the last fill of each slot completes its barrier when the bytes land
        const uint64_t tw = globaltimer_ns();
        auto drain = [&](uint64_t* bar, int fills) {
          if (fills > 0)
            while (!mbar_try_wait(bar, (fills - 1) & 1) && globaltimer_ns() - tw < 2000000ull) {
            }
        };
        drain(&sh->q_full, 1);
        for (int i = 0; i < kFreeSlots; ++i) drain(&sh->free_full[i], (n_free + kFreeSlots - 1 - i) / kFreeSlots);
        for (int i = 0; i < kHeldSlots; ++i) drain(&sh->held_full[i], (n_held + kHeldSlots - 1 - i) / kHeldSlots);
      }
    }
  } else if (warp == 1) {
    if (n_it > 0 && elect_one()) {   // one thread waits and issues
      constexpr uint32_t idesc_s = make_idesc(kHeadRows, kTok, 0, 0, 1);
      constexpr uint32_t idesc_pv = make_idesc(kHeadRows, 256, 0, 1, 1);
      const uint64_t d_q = make_smem_desc(smem_u32(qs), 16, 1024);
      const uint64_t d_free = make_smem_desc(smem_u32(fre), 16, 1024);
      const uint64_t d_hk = make_smem_desc(smem_u32(held), 16, 1024);
      const uint64_t d_hv = make_smem_desc(smem_u32(held), kChunkBytes, 1024);
      bool ok = mbar_wait(&sh->q_full, 0, abort_flag) && mbar_wait(&sh->q_tmem, 0, abort_flag);
      if (!ok) report_status(a.status, kWaitFullTimeout, 72, b, 0);
      tc_fence_after();
      int slot = 0, use = 0;
      auto scores = [&](int it) {
        const uint32_t d = tmem + kColS + (it & 1) * kTok;
        for (int i = 0; i < kFreeChunks; ++i) {
          if (!mbar_wait(&sh->free_full[slot], use & 1, abort_flag)) return false;
          tc_fence_after();
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_bf16(d, d_q + ((i * kQChunkBytes + k * 32) >> 4), d_free + ((slot * kChunkBytes + k * 32) >> 4), idesc_s,
                      (i > 0 || k > 0) ? 1u : 0u);
          tc_commit(&sh->free_empty[slot]);
          if (++slot == kFreeSlots) {
            slot = 0;
            ++use;
          }
        }
        const int hs = it % kHeldSlots;
        if (!mbar_wait(&sh->held_full[hs], (it / kHeldSlots) & 1, abort_flag)) return false;
        tc_fence_after();
#pragma unroll
        for (int i = 0; i < kHeldChunks; ++i)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_bf16_ts(d, tmem + kColQ + i * 32 + k * 8, d_hk + ((hs * kHeldBytes + i * kChunkBytes + k * 32) >> 4), idesc_s, 1u);
        tc_commit(&sh->s_full[it & 1]);
        return true;
      };
      ok = ok && scores(0);
      for (int it = 0; it < n_it && ok; ++it) {
        // the scores of the next tile overwrite the probabilities of the tile before: its output product was issued earlier
        if (it + 1 < n_it && !scores(it + 1)) {
          report_status(a.status, kWaitFullTimeout, 73, b, it);
          break;
        }
        if (!mbar_wait(&sh->p_ready[it & 1], (it >> 1) & 1, abort_flag)) {
          report_status(a.status, kWaitFullTimeout, 74, b, it);
          break;
        }
        tc_fence_after();
        const int hs = it % kHeldSlots;
#pragma unroll
        for (int k = 0; k < kTok / 16; ++k)
          umma_bf16_ts(tmem + kColO, tmem + kColS + (it & 1) * kTok + k * 8, d_hv + ((hs * kHeldBytes + k * 2048) >> 4), idesc_pv,
                       (it > 0 || k > 0) ? 1u : 0u);
        tc_commit(&sh->held_empty[hs]);
        tc_commit(&sh->pv_done);
      }
    }
  } else {
    // ---------------- softmax: one head per lane ----------------
    const int q = warp & 3;
    const int row = q * 32 + lane;
    const uint32_t tl = tmem + (static_cast<uint32_t>(q * 32) << 16);
    const bool live = h0 + row < a.heads;
    const int64_t head = static_cast<int64_t>(b) * a.heads + h0 + row;
    bool ok = true;
    if (n_it > 0) {
      const uint4* src = reinterpret_cast<const uint4*>(q_rows + (live ? head : 0) * kMlaWidth + half * 256);
#pragma unroll 1
      for (int i = 0; i < kHeldChunks; ++i) {
        uint32_t v[32];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint4 w = live ? src[i * 8 + j] : make_uint4(0, 0, 0, 0);
          v[4 * j] = w.x;
          v[4 * j + 1] = w.y;
          v[4 * j + 2] = w.z;
          v[4 * j + 3] = w.w;
        }
        tmem_st_32x32(tl + kColQ + i * 32, v);
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&sh->q_tmem);
    }
    float ref = -INFINITY, l = 0.f;
    for (int it = 0; it < n_it; ++it) {
      if (ok && !mbar_wait(&sh->s_full[it & 1], (it >> 1) & 1, abort_flag)) {
        if (lane == 0) report_status(a.status, kWaitTmemFullTimeout, 75, b, it);
        ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);   // warp-uniform from here on (TMEM loads and stores below)
      if (!ok) break;
      tc_fence_after();
      const uint32_t ts = tl + kColS + (it & 1) * kTok;
      uint32_t v0[32], v1[32];
      tmem_ld_32x32(ts, v0);
      tmem_ld_32x32(ts + 32, v1);
      tmem_ld_wait();
      const int tok = (t0 + it) * kTok;
      float s[kTok];
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        s[j] = __uint_as_float(v0[j]) * a.scale_log2;
        s[32 + j] = __uint_as_float(v1[j]) * a.scale_log2;
      }
      if (tok < first || tok + kTok > len) {
#pragma unroll
        for (int j = 0; j < kTok; ++j)
          if (tok + j < first || tok + j >= len) s[j] = -INFINITY;
      }
      float mx[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
      for (int j = 4; j < kTok; ++j) mx[j & 3] = fmaxf(mx[j & 3], s[j]);
      const float mt = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      if (it == 0) {
        ref = mt;
      } else if (__any_sync(0xffffffffu, mt > ref + kRescale)) {
        // rare: O must hold still, i.e. the output product of the tile before is done (this tile's waits for p_ready)
        if (!mbar_wait(&sh->pv_done, (it - 1) & 1, abort_flag)) ok = false;
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          if (lane == 0) report_status(a.status, kWaitTmemFullTimeout, 76, b, it);
          break;
        }
        tc_fence_after();
        const float nref = fmaxf(ref, mt);
        const float alpha = nref == ref ? 1.f : exp2f(ref - nref);
#pragma unroll 1
        for (int c = 0; c < 256; c += 32) {
          uint32_t o[32];
          tmem_ld_32x32(tl + kColO + c, o);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
          tmem_st_32x32(tl + kColO + c, o);
        }
        l *= alpha;
        ref = nref;
      }
      const float mref = ref == -INFINITY ? 0.f : ref;
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t p[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        p[j] = pack_bf16x2(exp2f(s[2 * j] - mref), exp2f(s[2 * j + 1] - mref));
        const float2 f = unpack_bf16x2(p[j]);   // the denominator sums what the tensor core will use
        sum[j & 3] += f.x + f.y;
      }
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      tmem_st_32x32(ts, p);
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&sh->p_ready[it & 1]);
    }
    if (ok && n_it > 0) {
      if (!mbar_wait(&sh->pv_done, (n_it - 1) & 1, abort_flag)) ok = false;
      ok = __all_sync(0xffffffffu, ok);
      if (!ok && lane == 0) report_status(a.status, kWaitTmemFullTimeout, 77, b, n_it);
      tc_fence_after();
    }
    // ---- the CTA's half of the rows: final with one key range, else a normalised partial and its log2-sum-exp ----
    const bool some = ok && n_it > 0 && l > 0.f;
    const bool whole = n_parts == 1;
    const float sk = whole && a.sink != nullptr && live ? exp2f(a.sink[h0 + row] * 1.4426950408889634f - ref) : 0.f;
    const float inv = some ? 1.f / (l + sk) : 0.f;
    const int64_t part = (static_cast<int64_t>(b) * n_parts + split) * a.heads + h0 + row;
#pragma unroll 1
    for (int c = 0; c < 256; c += 32) {
      uint32_t o[32];
      if (n_it > 0) {
        tmem_ld_32x32(tl + kColO + c, o);
        tmem_ld_wait();
      }
      if (!live) continue;
      if (whole) {
        uint4* dst = reinterpret_cast<uint4*>(out + head * kMlaLatent + half * 256 + c);
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
          uint32_t w[4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            w[e] = some ? pack_bf16x2(__uint_as_float(o[j + 2 * e]) * inv, __uint_as_float(o[j + 2 * e + 1]) * inv) : 0u;
          dst[j / 8] = make_uint4(w[0], w[1], w[2], w[3]);
        }
      } else {
        float4* dst = reinterpret_cast<float4*>(a.part_out + part * kMlaLatent + half * 256 + c);
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          dst[j / 4] = some ? make_float4(__uint_as_float(o[j]) * inv, __uint_as_float(o[j + 1]) * inv,
                                          __uint_as_float(o[j + 2]) * inv, __uint_as_float(o[j + 3]) * inv)
                            : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    if (!whole && half == 0 && live) a.part_lse[part] = some ? ref + log2f(l) : -INFINITY;
    tc_fence_before();
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
}

}  // namespace

cudaError_t launch_mla_decode_wide(const __nv_bfloat16* q, const __nv_bfloat16* pool, const MlaDecodeArgs& args, int n_parts,
                                   __nv_bfloat16* out, cudaStream_t stream) {
  CUtensorMap t_pool, t_q;
  cudaError_t e;
  if ((e = encode_tma_2d(&t_pool, pool, 2, kMlaWidth, static_cast<uint64_t>(args.n_pages) * kMlaPage, kMlaWidth * 2ull, 64,
                         kMlaPage)) != cudaSuccess)
    return e;
  if ((e = encode_tma_2d(&t_q, q, 2, kMlaWidth, static_cast<uint64_t>(args.batch) * args.heads, kMlaWidth * 2ull, 64,
                         kHeadRows)) != cudaSuccess)
    return e;
  if ((e = cudaFuncSetAttribute(mla_decode_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes)) != cudaSuccess)
    return e;
  const int head_blocks = (args.heads + kHeadRows - 1) / kHeadRows;
  mla_decode_wide_kernel<<<dim3(2 * n_parts, head_blocks, args.batch), kThreads, kSmemBytes, stream>>>(t_pool, t_q, q, args, out);
  return cudaGetLastError();
}

}  // namespace b200
