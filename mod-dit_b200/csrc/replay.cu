// Exact sparsity-map replay for sm_100a: S = round(q*scale) k^T on the tcgen05 tensor pipe, then a
// compare-and-count epilogue straight out of tensor memory.
//
// One persistent CTA per SM.  A CTA walks segments: the pairs of key tiles of one query tile (or a part of them, past
// kSegPairs and among the query tiles left over after whole rounds, whose pairs are dealt out evenly).  No map element
// depends on two segments, so nothing has to be put together.
// One CTA per query tile (each with its own start: barriers, tensor memory, the Q tile, its rounding) spent half of a
// short sweep outside the tensor pipe and left a nearly empty last wave: 744 CTAs of 31 key tiles took 102 us for 41 us
// of tensor work.
//   warp 0      TMA producer: Q tiles through two buffers, K tiles through a 4-stage ring
//   warp 1      MMA issuer: two key tiles per instruction (N = 256), into one of two 256-column accumulators
//   warp 2      tensor-memory allocation / release; with warp 3: scales and rounds the next segment's Q tile
//   warps 4-7   count group 0 (even key tiles = first 128 columns of an accumulator); thread r owns row r
//   warps 8-11  count group 1 (odd key tiles = second 128 columns)
// The Q tile is scaled and rounded to the input dtype in shared memory before its first MMA (the
// reference rounds the scaled query the same way).  Counts of the four 64x64 quarters of every
// 128x128 tile are accumulated in shared memory and a segment's map elements are written once, coalesced.
// Tensor-pipe work: 2*128*128*D flop per tile; memory traffic: one K tile (128*D*2 bytes) per tile,
// served from L2 for all but the first query tile of a head.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "ptx.cuh"
#include "tmap.cuh"

namespace moddit {
namespace {

constexpr int kThreads = 384;
constexpr int kTile = 128;
constexpr int kStages = 4;
constexpr int kPairStages = kStages / 2;

constexpr int kSegPairs = 128;          // pairs of key tiles per segment at most: the size of a count buffer

enum BarrierIndex {
  kQFull0 = 0,                      // 2: the segment's Q tile has landed
  kQReady0 = kQFull0 + 2,           // 2: ... and is scaled and rounded
  kQFree0 = kQReady0 + 2,           // 2: its last product has completed
  kKFull0 = kQFree0 + 2,            // kPairStages: both key tiles of a pair have landed
  kKEmpty0 = kKFull0 + kPairStages, // kPairStages
  kSFull0 = kKEmpty0 + kPairStages, // 2: accumulator b holds the scores of a pair of key tiles
  kSFree0 = kSFull0 + 2,        // 2
  kNumBarriers = kSFree0 + 2
};

struct __align__(8) Control {
  unsigned long long bars[kNumBarriers];
  uint32_t tmem_base;
  int abort_flag;
  int quarter[2][2 * kSegPairs * 4];      // counts of the 64x64 quarters of a segment's key tiles, two segments in turn
};

template <int D>
constexpr size_t smem_bytes() {
  return static_cast<size_t>(2 + kStages) * kTile * D * 2 + 1024 + sizeof(Control);
}

// What one CTA works on, as segments: whole query tiles in rounds over the grid (CTAs that run side by side stay on one
// head, whose K tiles they share through the L2), then its share of the tiles left over after whole rounds.  Left-over
// tiles for four fifths of the grid or more are a round of their own: dealing them out would save a fifth of a tile's
// sweep at most and costs a second segment's Q tile (16 heads of 9 x 9 tiles: 10.3 us, dealt out 12.3).
// 32-bit throughout: the host admits items (heads x query tiles) below 2^31, and fewer than a grid are left over.
// (64-bit divisions at every segment took 1-3 % of a launch.)
struct Segments {
  int pairs, ntk, rounds, r, u;
  int bh, qt, p0, p1;      // current segment: pairs [p0, p1) of query tile qt of head bh
  __device__ __forceinline__ Segments(int BH, int ntk_) : pairs((ntk_ + 1) / 2), ntk(ntk_) {
    const unsigned items = static_cast<unsigned>(BH) * ntk_;
    rounds = static_cast<int>(items / gridDim.x);
    unsigned left = items - rounds * gridDim.x;
    tail0_ = items - left;
    if (5 * left >= 4 * gridDim.x) {
      if (blockIdx.x < left) ++rounds;
      left = 0;
    }
    const unsigned units = left * pairs;
    r = 0;
    u = 0;
    tail_u_ = units * blockIdx.x / gridDim.x;
    tail_end_ = units * (blockIdx.x + 1) / gridDim.x;
  }
  __device__ __forceinline__ bool next() {
    unsigned item;
    if (r < rounds) {
      item = static_cast<unsigned>(r) * gridDim.x + blockIdx.x;
      p0 = u;
      p1 = min(pairs, p0 + kSegPairs);
      u = p1;
      if (u == pairs) { u = 0; ++r; }
    } else {
      if (tail_u_ >= tail_end_) return false;
      const unsigned t = tail_u_ / pairs;
      item = tail0_ + t;
      p0 = static_cast<int>(tail_u_ - t * pairs);
      p1 = min(min(pairs, p0 + kSegPairs), p0 + static_cast<int>(tail_end_ - tail_u_));
      tail_u_ += p1 - p0;
    }
    bh = static_cast<int>(item / ntk);
    qt = static_cast<int>(item - static_cast<unsigned>(bh) * ntk);
    return true;
  }
 private:
  unsigned tail0_, tail_u_, tail_end_;
};

__device__ __forceinline__ void report(int32_t* status, int code, int role, int where) {
  if (atomicCAS(status, 0, code) == 0) {
    status[1] = static_cast<int32_t>(blockIdx.x);
    status[2] = role;
    status[3] = where;
  }
}

template <int D, bool kBF16>
__global__ void __launch_bounds__(kThreads, 1) replay_map_kernel(
    const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
    const float* __restrict__ lse, int BH, int N, int bs, float scale, float log_thr, int q_off, int k_off, int n,
    __half* __restrict__ map, int32_t* __restrict__ status) {
  constexpr int kTileBytes = kTile * D * 2;
  constexpr int kChunks = D / 64;
  constexpr int kChunkBytes = kTile * 128;
  constexpr uint32_t kIdesc256 = ptx::idesc_f16(128, 256, kBF16, false);
  constexpr uint32_t kIdesc128 = ptx::idesc_f16(128, 128, kBF16, false);
  // K ring, chunk-major: [64-column chunk][stage][128 rows x 128 B], so the rows of two consecutive stages are
  // contiguous inside a chunk and one N = 256 operand covers both tiles
  constexpr int kRingChunkBytes = kStages * kChunkBytes;

  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Control* ctl = reinterpret_cast<Control*>(smem + (2 + kStages) * kTileBytes);
  const uint32_t sQ = ptx::smem_u32(smem);
  const uint32_t sK = sQ + 2 * kTileBytes;
  const uint32_t bar0 = ptx::smem_u32(&ctl->bars[0]);
  auto bar = [&](int i) { return bar0 + 8u * static_cast<uint32_t>(i); };
  volatile int* abort_flag = &ctl->abort_flag;

  const int warp = ptx::warp_index();
  const int lane = threadIdx.x % 32;
  const int vtok = n * bs;                                  // video tokens
  const int ntk = (vtok + kTile - 1) / kTile;
  Segments seg(BH, ntk);

  if (threadIdx.x == 0) {
    for (int i = 0; i < kNumBarriers; ++i) {
      uint32_t c = 1;
      if (i >= kQReady0 && i < kQReady0 + 2) c = 64;
      if (i >= kSFree0) c = 256;
      ptx::mbar_init(bar(i), c);
    }
    ctl->abort_flag = 0;
    ptx::fence_barrier_init();
    ptx::prefetch_tensormap(&tm_q);
    ptx::prefetch_tensormap(&tm_k);
  }
  for (int i = threadIdx.x; i < 2 * 2 * kSegPairs * 4; i += kThreads) ctl->quarter[0][i] = 0;
  if (warp == 2) {
    ptx::tmem_alloc(ptx::smem_u32(&ctl->tmem_base), 512);
    ptx::tmem_relinquish();
    ptx::tc_fence_before();
  }
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;

  if (warp == 0) {
    if (ptx::elect_one()) {
      bool ok = true;
      int issued = 0, sn = 0;                               // key pairs and Q tiles requested so far
      // the Q tile of the segment after the current one is requested first: it is scaled while this one is multiplied
      Segments ahead = seg;
      auto load_q = [&](int bh, int qt) -> bool {
        const int b = sn & 1;
        if (!ptx::mbar_wait(bar(kQFree0 + b), ((sn >> 1) & 1) ^ 1, abort_flag)) return false;
        ptx::mbar_expect_tx(bar(kQFull0 + b), kTileBytes);
        for (int c = 0; c < kChunks; ++c)
          ptx::tma_load_3d(sQ + b * kTileBytes + c * kChunkBytes, &tm_q, bar(kQFull0 + b), c * 64, q_off + qt * kTile, bh);
        ++sn;
        return true;
      };
      if (ahead.next()) ok = load_q(ahead.bh, ahead.qt);
      while (ok && seg.next()) {
        // two key tiles (one N = 256 operand) share a barrier pair: the issuing thread pays one wait and one
        // commit per MMA group for its operands
        for (int p = seg.p0; p < seg.p1; ++p) {
          const int j = 2 * p;
          const int ps = issued % kPairStages;
          const bool two = (j + 1) < ntk;
          ok = ptx::mbar_wait(bar(kKEmpty0 + ps), ((issued / kPairStages) & 1) ^ 1, abort_flag);
          if (!ok) { report(status, 1, 0, j); break; }
          ptx::mbar_expect_tx(bar(kKFull0 + ps), (two ? 2u : 1u) * kTileBytes);
          for (int t = 0; t < (two ? 2 : 1); ++t)
            for (int c = 0; c < kChunks; ++c)
              ptx::tma_load_3d(sK + c * kRingChunkBytes + (2 * ps + t) * kChunkBytes, &tm_k, bar(kKFull0 + ps), c * 64,
                               k_off + (j + t) * kTile, seg.bh);
          ++issued;
          // its buffer is free once the segment before this one is through: so is the stage that the second pair went to
          if (p == min(seg.p0 + 1, seg.p1 - 1) && ahead.next()) {
            ok = load_q(ahead.bh, ahead.qt);
            if (!ok) { report(status, 1, 0, j); break; }
          }
        }
      }
      if (!ok) {
        // give copies in flight a bounded time to land (their barriers may never be consumed)
        for (int pj = max(0, issued - kPairStages); pj < issued; ++pj)
          for (int i = 0; i < 4096 && !ptx::mbar_try_wait(bar(kKFull0 + pj % kPairStages), (pj / kPairStages) & 1); ++i) {}
        for (int t = max(0, sn - 2); t < sn; ++t)
          for (int i = 0; i < 4096 && !ptx::mbar_try_wait(bar(kQFull0 + (t & 1)), (t >> 1) & 1); ++i) {}
      }
    }
  } else if (warp == 1) {
    if (ptx::elect_one()) {
      bool ok = true;
      const uint64_t dq0 = ptx::smem_desc_sw128(sQ, 16, 1024);
      const uint64_t dk0 = ptx::smem_desc_sw128(sK, 16, 1024);
      auto advance = [](uint64_t desc, uint32_t bytes) -> uint64_t {
        // the start-address field (units of 16 bytes) never carries out for shared-memory addresses
        return (desc & 0xffffffff00000000ull) | static_cast<uint32_t>(static_cast<uint32_t>(desc) + (bytes >> 4));
      };
      int pj = 0;
      for (int sn = 0; ok && seg.next(); ++sn) {
        ok = ptx::mbar_wait(bar(kQReady0 + (sn & 1)), (sn >> 1) & 1, abort_flag);
        if (!ok) { report(status, 2, 1, -1); break; }
        const uint64_t dq = advance(dq0, static_cast<uint32_t>(sn & 1) * kTileBytes);
        for (int p = seg.p0; p < seg.p1; ++p, ++pj) {
          const int ps = pj % kPairStages;
          const int b = pj & 1;
          ok = ptx::mbar_wait(bar(kKFull0 + ps), (pj / kPairStages) & 1, abort_flag);
          if (ok) ok = ptx::mbar_wait(bar(kSFree0 + b), ((pj >> 1) & 1) ^ 1, abort_flag);
          if (!ok) { report(status, 2, 1, 2 * p); break; }
          ptx::tc_fence_after();
          const uint64_t dk = advance(dk0, static_cast<uint32_t>(2 * ps) * kChunkBytes);
          const uint32_t idesc = (2 * p + 1) < ntk ? kIdesc256 : kIdesc128;
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk)
            ptx::mma_ss(tmem + b * 256, advance(dq, (kk / 4) * kChunkBytes + (kk % 4) * 32),
                        advance(dk, (kk / 4) * kRingChunkBytes + (kk % 4) * 32), idesc, kk > 0 ? 1u : 0u);
          ptx::tc_commit(bar(kSFull0 + b));
          ptx::tc_commit(bar(kKEmpty0 + ps));
        }
        if (ok) ptx::tc_commit(bar(kQFree0 + (sn & 1)));
      }
    }
  } else if (warp < 4) {
    // scale + round each Q tile in place (element-wise, so the swizzled order does not matter).  These warps wait through
    // most of a sweep, beside count warps that bound the kernel: polling without sleep cost 48 heads of 352 x 352 tiles
    // at head dimension 64 5 % (17.0 against 16.2 ms).
    bool ok = true;
    for (int sn = 0; ok && seg.next(); ++sn) {
      ok = ptx::mbar_wait_idle(bar(kQFull0 + (sn & 1)), (sn >> 1) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) { if (lane == 0) report(status, 4, 2, -1); break; }
      uint4* q4 = reinterpret_cast<uint4*>(smem + (sn & 1) * kTileBytes);
#pragma unroll 4
      for (int i = static_cast<int>(threadIdx.x) - 64; i < kTileBytes / 16; i += 64) {
        uint4 w = q4[i];
        uint32_t* p = reinterpret_cast<uint32_t*>(&w);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if constexpr (kBF16) {
            const __nv_bfloat162 h2 = *reinterpret_cast<const __nv_bfloat162*>(&p[u]);
            const __nv_bfloat162 o2 = __halves2bfloat162(__float2bfloat16_rn(__bfloat162float(h2.x) * scale),
                                                         __float2bfloat16_rn(__bfloat162float(h2.y) * scale));
            p[u] = *reinterpret_cast<const uint32_t*>(&o2);
          } else {
            const __half2 h2 = *reinterpret_cast<const __half2*>(&p[u]);
            const __half2 o2 = __halves2half2(__float2half_rn(__half2float(h2.x) * scale),
                                              __float2half_rn(__half2float(h2.y) * scale));
            p[u] = *reinterpret_cast<const uint32_t*>(&o2);
          }
        }
        q4[i] = w;
      }
      ptx::fence_proxy_async_smem();
      ptx::mbar_arrive(bar(kQReady0 + (sn & 1)));
    }
  } else {
    const int g = (warp - 4) / 4;
    const int wq = warp % 4;
    const int r = wq * 32 + lane;
    const int t256 = threadIdx.x - 128;                     // 0..255 over both count groups
    const uint32_t lane_base = static_cast<uint32_t>(wq * 32) << 16;
    const int rh = r >> 6;
    const float inv_area = 1.0f / static_cast<float>(bs * bs);
    bool ok = true;
    int pj = 0;
    // A warp whose wait gave up stays in step at the barriers below (they have no time limit) and does nothing else.
    for (int sn = 0; seg.next(); ++sn) {
      int* quarter = ctl->quarter[sn & 1];
      const int grow = q_off + seg.qt * kTile + r;
      const bool row_ok = (seg.qt * kTile + r) < vtok && grow < N;
      const float line = row_ok ? (lse[static_cast<int64_t>(seg.bh) * N + grow] + log_thr) : -INFINITY;
      for (int p = seg.p0; p < seg.p1 && ok; ++p, ++pj) {
        const int j = 2 * p + g;
        const int b = pj & 1;
        ok = ptx::mbar_wait(bar(kSFull0 + b), (pj >> 1) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) { if (lane == 0) report(status, 5, 2 + g, j); break; }
        ptx::tc_fence_after();
        if (j >= ntk) {                                     // odd number of key tiles: nothing in the second half
          ptx::mbar_arrive(bar(kSFree0 + b));
          continue;
        }
        float v[kTile];
#pragma unroll
        for (int c = 0; c < 4; ++c) ptx::tmem_ld32(tmem + lane_base + b * 256 + g * 128 + c * 32, reinterpret_cast<uint32_t*>(v) + c * 32);
        ptx::tmem_ld_wait();
        ptx::tc_fence_before();
        ptx::mbar_arrive(bar(kSFree0 + b));
        int c_lo = 0, c_hi = 0;
#pragma unroll
        for (int c = 0; c < 64; ++c) c_lo += (v[c] < line) ? 1 : 0;
#pragma unroll
        for (int c = 64; c < 128; ++c) c_hi += (v[c] < line) ? 1 : 0;
        c_lo = __reduce_add_sync(0xffffffffu, c_lo);
        c_hi = __reduce_add_sync(0xffffffffu, c_hi);
        if (lane == 0) {
          atomicAdd(&quarter[(j - 2 * seg.p0) * 4 + rh * 2 + 0], c_lo);
          atomicAdd(&quarter[(j - 2 * seg.p0) * 4 + rh * 2 + 1], c_hi);
        }
      }
      // all 256 counting threads meet; each then writes its map elements and clears their counts, while the others may
      // already add to the other buffer (this one is used again after the next such meeting)
      asm volatile("bar.sync 1, 256;" ::: "memory");
      const bool valid = !*abort_flag;
      const int j0 = 2 * seg.p0, j1 = min(2 * seg.p1, ntk);
      for (int j = j0 + t256; j < j1; j += 256) {
        int* cnt = quarter + (j - j0) * 4;
        const int c00 = cnt[0], c01 = cnt[1], c10 = cnt[2], c11 = cnt[3];
        cnt[0] = cnt[1] = cnt[2] = cnt[3] = 0;
        if (!valid) continue;
        __half* base = map + static_cast<int64_t>(seg.bh) * n * n;
        if (bs == 128) {
          if (seg.qt < n && j < n) base[static_cast<int64_t>(seg.qt) * n + j] = __float2half_rn(static_cast<float>(c00 + c01 + c10 + c11) * inv_area);
        } else {
          const int count[2][2] = {{c00, c01}, {c10, c11}};
#pragma unroll
          for (int h2 = 0; h2 < 2; ++h2)
#pragma unroll
            for (int c2 = 0; c2 < 2; ++c2)
              if (2 * seg.qt + h2 < n && 2 * j + c2 < n)
                base[static_cast<int64_t>(2 * seg.qt + h2) * n + 2 * j + c2] = __float2half_rn(static_cast<float>(count[h2][c2]) * inv_area);
        }
      }
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 512);
  }
}

template <int D, bool kBF16>
int launch(const void* q, const void* k, const float* lse, int dtype, int BH, int N, int bs, float scale,
           float log_thr, int q_off, int k_off, int n, void* map, int32_t* status, cudaStream_t st) {
  CUtensorMap tq, tk;
  if (int rc = make_tmap_rows(&tq, q, dtype, BH, N, D, kTile)) return rc;
  if (int rc = make_tmap_rows(&tk, k, dtype, BH, N, D, kTile)) return rc;
  const int ntk = ceil_div(n * bs, kTile);
  const long long units = static_cast<long long>(BH) * ntk * ((ntk + 1) / 2);
  int sms = 0;
  if (int rc = sm_count(&sms)) return rc;
  const size_t smem = smem_bytes<D>();
  // the entry point's limit (moddit.h); with BH <= 65535 it keeps the item counts of Segments in 32 bits
  if (ntk > (D == 128 ? 4218 : 9338))
    return fail(MODDIT_E_UNSUPPORTED, "replay_map: %d key tiles of 128 exceed the limit of %d", ntk, D == 128 ? 4218 : 9338);
  auto kernel = replay_map_kernel<D, kBF16>;
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem)) return rc;
  kernel<<<static_cast<unsigned>(units < sms ? units : sms), kThreads, smem, st>>>(tq, tk, lse, BH, N, bs, scale, log_thr, q_off, k_off, n,
                                                static_cast<__half*>(map), status);
  MODDIT_CHECK_LAUNCH("replay_map_kernel");
  return MODDIT_OK;
}

}  // namespace
}  // namespace moddit

using namespace moddit;

// The status words live in a small device buffer owned by the library user only for the sparse
// forward; the replay entry point keeps the reference's signature (no status argument), so it uses a
// per-device static word that the kernel only ever writes when a bounded wait expires.
static __device__ int32_t g_replay_status[4];

extern "C" int moddit_replay_map(const void* q, const void* k, const float* lse, int dtype, int BH, int N, int D,
                                 int block_size, float softmax_scale, float log_threshold, int q_video_offset,
                                 int k_video_offset, int video_blocks, void* map_f16, void* stream) {
  clear_error();
  MODDIT_CHECK_ARG(q && k && lse && map_f16, "replay_map: null pointer");
  MODDIT_CHECK_ARG(BH > 0 && BH <= 65535 && N > 0, "replay_map: BH=%d N=%d out of range", BH, N);
  MODDIT_CHECK_ARG(video_blocks > 0, "replay_map: video_blocks must be positive");
  MODDIT_CHECK_ARG(q_video_offset >= 0 && k_video_offset >= 0, "replay_map: video offsets must be non-negative");
  if (block_size != 64 && block_size != 128)
    return fail(MODDIT_E_UNSUPPORTED, "replay_map: block_size must be 64 or 128, got %d", block_size);
  if (D != 64 && D != 128) return fail(MODDIT_E_UNSUPPORTED, "replay_map: head_dim must be 64 or 128, got %d", D);
  if (dtype != MODDIT_BF16 && dtype != MODDIT_FP16) return fail(MODDIT_E_ARG, "replay_map: unknown dtype %d", dtype);
  const long long vt = static_cast<long long>(video_blocks) * block_size;
  MODDIT_CHECK_ARG(q_video_offset + vt <= N, "replay_map: Q video region exceeds sequence length");
  MODDIT_CHECK_ARG(k_video_offset + vt <= N, "replay_map: K video region exceeds sequence length");
  if (!aligned16(q) || !aligned16(k)) return fail(MODDIT_E_ALIGN, "replay_map: q and k must be 16-byte aligned");
  if (int rc = require_sm100()) return rc;
  int32_t* status = nullptr;
  MODDIT_CHECK_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&status), g_replay_status));
  cudaStream_t st = as_stream(stream);
  if (D == 128) {
    return dtype == MODDIT_BF16 ? launch<128, true>(q, k, lse, dtype, BH, N, block_size, softmax_scale, log_threshold,
                                                    q_video_offset, k_video_offset, video_blocks, map_f16, status, st)
                                : launch<128, false>(q, k, lse, dtype, BH, N, block_size, softmax_scale, log_threshold,
                                                     q_video_offset, k_video_offset, video_blocks, map_f16, status, st);
  }
  return dtype == MODDIT_BF16 ? launch<64, true>(q, k, lse, dtype, BH, N, block_size, softmax_scale, log_threshold,
                                                 q_video_offset, k_video_offset, video_blocks, map_f16, status, st)
                              : launch<64, false>(q, k, lse, dtype, BH, N, block_size, softmax_scale, log_threshold,
                                                  q_video_offset, k_video_offset, video_blocks, map_f16, status, st);
}

// Reads (and clears) the replay kernel's status words; non-zero code means a bounded wait expired in
// some earlier replay launch on the current device.  Synchronises `stream`.
extern "C" int moddit_replay_status(int32_t* host_status4, void* stream) {
  clear_error();
  MODDIT_CHECK_ARG(host_status4, "replay_status: null pointer");
  int32_t* status = nullptr;
  MODDIT_CHECK_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&status), g_replay_status));
  cudaStream_t st = as_stream(stream);
  MODDIT_CHECK_CUDA(cudaMemcpyAsync(host_status4, status, 4 * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  MODDIT_CHECK_CUDA(cudaMemsetAsync(status, 0, 4 * sizeof(int32_t), st));
  MODDIT_CHECK_CUDA(cudaStreamSynchronize(st));
  return MODDIT_OK;
}
