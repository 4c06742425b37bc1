// Block-sparse flash-attention forward for sm_100a: tcgen05 MMAs with accumulators in tensor memory,
// K/V tiles fetched by TMA from a compacted work list (a skipped block costs no memory traffic),
// warp-specialised online softmax.
//
// One CTA owns a PAIR of adjacent 128-row query tiles (A, B) of one head and walks the union of
// their key-tile lists, so a K/V tile needed by both is fetched once.  Where a launch has fewer pairs than
// SMs a CTA may own one tile of a pair; it walks the same list and passes over what the tile does not keep.
// Roles (12 warps):
//   warp 0      TMA producer: Q tiles once, then K and V tiles through two 2-stage rings (V of entry e and K
//               of entry e + 1 share their barriers: they are consumed together)
//   warp 1      MMA issuer: S_X = Q_X K^T (SS form), O_X += P_X V (P read from tensor memory)
//   warp 2      tensor-memory allocation / release
//   warps 4-7   softmax of tile A: thread r owns row r (tensor-memory lane r)
//   warps 8-11  softmax of tile B
// Tensor memory (512 columns): S_A [0,128) S_B [128,256) O_A [256,256+D) O_B [256+D,256+2D); P_X
// (16-bit) overwrites the first 64 columns of S_X.  MMAs issued by one thread execute in order, which
// is what makes the aliasing and the "S ready implies the previous P V finished" reasoning valid.
// The issue order of an entry that both tiles keep,  PV(A,e) QK(A,e+1) PV(B,e) QK(B,e+1),  lets the softmax
// of one tile overlap the MMAs of the other.  A tile that does not keep entry e has no P V in it, so its
// QK(e+1) comes first (B's before A's part if need be): the tile's last P V was issued earlier by the same
// thread, and K(e+1) has landed with V(e), which was waited for.
//
// Every wait is bounded (ptx::mbar_wait); on expiry the CTA records a status word, lets its copies
// land, releases tensor memory and returns.
//
// Tensor-pipe work per kept 128x128 tile: 4*128*128*D flop (QK^T and PV); memory traffic per fetched
// key tile: 2*128*D*2 bytes (K and V), shared by both query tiles.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "ptx.cuh"
#include "tmap.cuh"

namespace moddit {
namespace {

constexpr int kThreads = 384;
constexpr int kTile = 128;
constexpr float kRescaleThreshold = 8.0f;   // log2 domain: rescale O only when the row max grew by more than this

enum BarrierIndex {
  kQFull = 0,
  kKFirst,                      // K tile of entry 0
  kFull0, kFull1,               // entry e (index e & 1): V tile of e and K tile of e + 1 have landed
  kEmpty0, kEmpty1,             // entry e: its V stage and the K stage of e + 1 may be overwritten
  kSFullA, kSFullB,
  kPLoA, kPHiA, kPLoB, kPHiB,   // first 96 / last 32 keys of P stored, per query tile
  kOFinal,
  kNumBarriers
};

// Optional destination of the output rows on a multi-GPU run: instead of one local (BH, N, D) tensor the
// rows of sequence shard r (rows [r*rows_per_peer, (r+1)*rows_per_peer)) are stored straight into rank r's
// (total_heads, rows_per_peer, D) buffer at head `head_base + bh` - the output re-shard is fused into the
// epilogue as plain peer stores.
constexpr int kMaxPeers = 8;
struct OutScatter {
  void* peer[kMaxPeers];
  int n_peers;          // 0: write `out` locally
  int rows_per_peer;
  int head_base;
};

struct __align__(8) Control {
  unsigned long long bars[kNumBarriers];
  uint32_t tmem_base;
  int abort_flag;
};

template <int D>
constexpr size_t smem_bytes() {
  // 2 Q tiles + 2 K stages + 2 V stages, 1024-byte alignment slack, control block
  return static_cast<size_t>(6) * kTile * D * 2 + 1024 + sizeof(Control);
}

__device__ __forceinline__ void report(int32_t* status, int code, int role, int where) {
  if (atomicCAS(status, 0, code) == 0) {
    status[1] = static_cast<int32_t>(blockIdx.y * gridDim.x + blockIdx.x);
    status[2] = role;
    status[3] = where;
  }
}

template <bool kBF16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if constexpr (kBF16) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  } else {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
}

// Which work item a block has.  The first 2 * n_single blocks have one query tile each, the two of a pair next to each other;
// the others have a pair.
struct BlockItem {
  int npairs, item;
  int flags;            // bits of its query tiles in a list entry: 0xff, 0x0f (the first only) or 0xf0 (the second only)
  __device__ __forceinline__ BlockItem(int n_single, int Hm, const int32_t* order) {
    const int b = static_cast<int>(blockIdx.x);
    const bool single = b < 2 * n_single;
    const int index = single ? b >> 1 : b - n_single;
    npairs = (static_cast<int>(gridDim.x) - n_single) / Hm;
    item = order ? order[index] : index;
    flags = single ? ((b & 1) ? 0xf0 : 0x0f) : 0xff;
  }
};

// Pairs whose two query tiles run as blocks of their own: as many as there would be idle SMs, the first ones of `order` (the two
// longest lists of every head, then the first head's from the longest on, the second head's, ...; without an order the first
// by index).  A tile by itself has the exponential unit and the tensor pipe to itself; its rows are computed as in a pair, bit
// for bit.  It fetches K and V of the whole list of its pair, also of entries that only the other tile keeps.  Launch alone:
// 132 pairs whose longest list is three times the mean 118 -> 108 us, 32 pairs at head dimension 64 44 -> 38.
// Launches that run at the same time (`pairs_beside`: the others' work items) divide the idle SMs by their work items, because
// a tile by itself needs more than half of its pair's time: two launches of 66 pairs take 74 us together (99 when each was
// split as if it had the chip to itself, 81 without single tiles), three 120 (142, 123).
int single_pairs(int sms, int items, int batches, int pairs_beside) {
  const int64_t idle = max(0, (sms - pairs_beside) / batches - items);
  const int64_t mine = static_cast<int64_t>(items) * batches;
  return min(items, static_cast<int>(idle * mine / (mine + pairs_beside)));
}

template <int D, bool kBF16>
__global__ void __launch_bounds__(kThreads, 1) sparse_attn_fwd_kernel(
    const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
    const __grid_constant__ CUtensorMap tm_v, const int32_t* __restrict__ counts,
    const int32_t* __restrict__ entries, const int32_t* __restrict__ order, int Hm, int ntk, int N, float scale_log2, int q_split, int kvl_lo,
    int kvl_hi, int n_single, void* __restrict__ out_raw, float* __restrict__ lse, int32_t* __restrict__ status,
    const __grid_constant__ OutScatter scatter) {
  constexpr int kTileBytes = kTile * D * 2;       // one Q, K or V tile
  constexpr int kChunks = D / 64;                 // 64-element (128-byte) column chunks per tile
  constexpr int kChunkBytes = kTile * 128;
  constexpr uint32_t kIdescQK = ptx::idesc_f16(128, 128, kBF16, false);
  constexpr uint32_t kIdescPV = ptx::idesc_f16(128, D, kBF16, true);

  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Control* ctl = reinterpret_cast<Control*>(smem + 6 * kTileBytes);
  const uint32_t sQ = ptx::smem_u32(smem);
  const uint32_t sK = sQ + 2 * kTileBytes;
  const uint32_t sV = sQ + 4 * kTileBytes;
  const uint32_t bar0 = ptx::smem_u32(&ctl->bars[0]);
  auto bar = [&](int i) { return bar0 + 8u * static_cast<uint32_t>(i); };
  volatile int* abort_flag = &ctl->abort_flag;

  const int warp = ptx::warp_index();
  const int lane = threadIdx.x % 32;
  // grid: x = work item (mask head, query-tile pair, or one tile of it), y = batch.  Blocks start in increasing blockIdx.x;
  // `order` (from the work-list builder) puts long lists first, otherwise items run head by head.
  const BlockItem blk(n_single, Hm, order);
  const int npairs = blk.npairs, item = blk.item;
  const int mh = item / npairs;
  const int pair = item - mh * npairs;
  const int bh = blockIdx.y * Hm + mh;
  const int ntq = (N + kTile - 1) / kTile;
  if (2 * pair + (blk.flags == 0xf0) >= ntq) return;          // the second query tile of a pair that has one only
  const int cnt = counts[static_cast<int64_t>(mh) * npairs + pair];
  const int32_t* ent = entries + (static_cast<int64_t>(mh) * npairs + pair) * ntk;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kNumBarriers; ++i) ptx::mbar_init(bar(i), (i >= kPLoA && i <= kPHiB) ? 128u : 1u);
    ctl->abort_flag = 0;
    ptx::fence_barrier_init();
    ptx::prefetch_tensormap(&tm_q);
    ptx::prefetch_tensormap(&tm_k);
    ptx::prefetch_tensormap(&tm_v);
  }
  if (warp == 2) {
    ptx::tmem_alloc(ptx::smem_u32(&ctl->tmem_base), 512);
    ptx::tmem_relinquish();
    ptx::tc_fence_before();
  }
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;

  // Register budget: the softmax warpgroups hold a 128-value row per thread, the control warps need little
  // (128 control threads give up what 256 softmax threads take: 168 -> 72 / 216, the split that spills least).
  // The control branch and the softmax branch are disjoint in the control-flow graph so that each gets
  // its own register allocation.
  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (ptx::elect_one()) {
      const int q0 = blk.flags == 0xf0, q1 = blk.flags != 0x0f && 2 * pair + 1 < ntq;      // first and last query tile
      ptx::mbar_expect_tx(bar(kQFull), (q1 - q0 + 1) * kTileBytes);
      for (int x = q0; x <= q1; ++x)
        for (int c = 0; c < kChunks; ++c)
          ptx::tma_load_3d(sQ + x * kTileBytes + c * kChunkBytes, &tm_q, bar(kQFull), c * 64, (2 * pair + x) * kTile,
                           bh);
      // Entry e consumes V(e) and K(e+1) together (P V of e, then Q K^T of e + 1), so the two tiles share one
      // pair of barriers: the MMA-issuing thread pays one wait and one commit per entry for its operands.
      bool ok = true;
      int issued = 0;
      if (cnt > 0) {
        ptx::mbar_expect_tx(bar(kKFirst), kTileBytes);
        for (int c = 0; c < kChunks; ++c)
          ptx::tma_load_3d(sK + c * kChunkBytes, &tm_k, bar(kKFirst), c * 64, (ent[0] >> 8) * kTile, bh);
      }
      for (int e = 0; e < cnt && ok; ++e) {
        const int s = e & 1;
        // kEmpty1 also completes once before the loop (the first K tile's stage), hence the shifted parity
        const uint32_t par = ((e >> 1) & 1) ^ (s ? 0u : 1u);
        const bool next = (e + 1) < cnt;
        ok = ptx::mbar_wait(bar(kEmpty0 + s), par, abort_flag);
        if (!ok) { report(status, 1, 0, e); break; }
        ptx::mbar_expect_tx(bar(kFull0 + s), (next ? 2u : 1u) * kTileBytes);
        const int row0 = (ent[e] >> 8) * kTile;
        for (int c = 0; c < kChunks; ++c)
          ptx::tma_load_3d(sV + s * kTileBytes + c * kChunkBytes, &tm_v, bar(kFull0 + s), c * 64, row0, bh);
        if (next) {
          const int row1 = (ent[e + 1] >> 8) * kTile;
          for (int c = 0; c < kChunks; ++c)
            ptx::tma_load_3d(sK + (s ^ 1) * kTileBytes + c * kChunkBytes, &tm_k, bar(kFull0 + s), c * 64, row1, bh);
        }
        issued = e + 1;
      }
      if (!ok) {
        // give copies in flight a bounded time to land (their barriers may never be consumed)
        for (int i = 0; i < 4096 && cnt > 0 && !ptx::mbar_try_wait(bar(kKFirst), 0); ++i) {}
        for (int e = max(0, issued - 2); e < issued; ++e)
          for (int i = 0; i < 4096 && !ptx::mbar_try_wait(bar(kFull0 + (e & 1)), (e >> 1) & 1); ++i) {}
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (ptx::elect_one()) {
      // Descriptor bases are built once; inside the loops an MMA costs one 32-bit add per operand (the
      // issuing thread shares its scheduler with two busy softmax warps, so every instruction counts).
      auto advance = [](uint64_t desc, uint32_t bytes) -> uint64_t {
        // the start-address field (bits 0-13, units of 16 bytes) never carries out for shared-memory addresses
        return (desc & 0xffffffff00000000ull) | static_cast<uint32_t>(static_cast<uint32_t>(desc) + (bytes >> 4));
      };
      const uint64_t dq0 = ptx::smem_desc_sw128(sQ, 16, 1024), dk0 = advance(dq0, sK - sQ);
      const uint64_t dv0 = ptx::smem_desc_sw128(sV, kChunkBytes, 1024);
      auto issue_qk = [&](int x, int s) {
        const uint64_t a0 = advance(dq0, x * kTileBytes), b0 = advance(dk0, s * kTileBytes);
        const uint32_t d = tmem + x * 128;
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (kk / 4) * kChunkBytes + (kk % 4) * 32;
          ptx::mma_ss(d, advance(a0, off), advance(b0, off), kIdescQK, kk > 0 ? 1u : 0u);
        }
        ptx::tc_commit(bar(kSFullA + x));
      };
      // P*V for the first 96 keys of the tile (part 0) or the last 32
      auto issue_pv_part = [&](int x, int s, int part, uint32_t acc) {
        const uint64_t b0 = advance(dv0, s * kTileBytes);
        const uint32_t d = tmem + 256 + x * D, a = tmem + x * 128;
#pragma unroll
        for (int kq = 0; kq < (part ? 2 : 6); ++kq) {
          const int kk = part * 6 + kq;
          ptx::mma_ts(d, a + kk * 8, advance(b0, kk * 2048), kIdescPV, (acc || kq > 0) ? 1u : 0u);
        }
      };
      // waits for the two parts of P in turn; returns false if a wait gave up
      auto pv_when_ready = [&](int x, int s, uint32_t acc, uint32_t parity) -> bool {
        if (!ptx::mbar_wait(bar(kPLoA + 2 * x), parity, abort_flag)) return false;
        ptx::tc_fence_after();
        issue_pv_part(x, s, 0, acc);
        if (!ptx::mbar_wait(bar(kPHiA + 2 * x), parity, abort_flag)) return false;
        ptx::tc_fence_after();
        issue_pv_part(x, s, 1, 1u);
        return true;
      };
      bool ok = ptx::mbar_wait(bar(kQFull), 0, abort_flag);
      if (!ok) report(status, 2, 1, -1);
      uint32_t tiles = 0;                   // bit x: parity of tile x's P, bit 2 + x: tile x has an accumulator
      if (ok && cnt > 0) {
        ok = ptx::mbar_wait(bar(kKFirst), 0, abort_flag);
        if (!ok) report(status, 2, 1, 0);
        if (ok) {
          ptx::tc_fence_after();
          const int fl = ent[0] & blk.flags;
          if (fl & 0x0f) issue_qk(0, 0);
          if (fl & 0xf0) issue_qk(1, 0);
          ptx::tc_commit(bar(kEmpty1));     // K stage 0 is free for the K tile of entry 2 (loaded with V of entry 1)
        }
      }
      int fl_carry = (cnt > 0) ? (ent[0] & blk.flags) : 0;
      for (int e = 0; e < cnt && ok; ++e) {
        const int s = e & 1;
        const int fl = fl_carry;
        const bool next = (e + 1) < cnt;
        const int fln = next ? (ent[e + 1] & blk.flags) : 0;   // issued here, first used after the P V of tile A
        fl_carry = fln;
        ok = ptx::mbar_wait(bar(kFull0 + s), (e >> 1) & 1, abort_flag);
        if (!ok) { report(status, 2, 1, e); break; }
        // A tile that does not keep this entry starts on the next one before the other tile's P is waited for: where two
        // neighbouring entries are kept by one tile each (a diagonal does that), both tiles work at the same time.  So the
        // slot begins with the second tile where that has no P V; the tile's number is a run-time value, because the copies
        // of the products that constants need cost launches without such entries more than they gain.  Launch, fixed order /
        // one copy for either tile here and a further one for the early scores / this: dense 24 heads x 6,820 tokens 542 /
        // 540 - 549 / 525 us, HunyuanVideo (12 % one-sided) 21.06 / 20.89 / 20.41 ms, Wan (21 %) 15.54 / 15.23 / 14.94,
        // cumulative-mass clip (50 %) 693 / 677 / 669 us; one copy in a loop of two 536, 20.87, 15.31, 677.
        const int first = (fl & 0xf0) ? 0 : 1;
        auto half_slot = [&](int x) -> bool {
          if ((fl >> (4 * x)) & 0xf) {
            if (!pv_when_ready(x, s, tiles & (4u << x), (tiles >> x) & 1u)) return false;
            tiles = (tiles ^ (1u << x)) | (4u << x);
          }
          if ((fln >> (4 * x)) & 0xf) issue_qk(x, s ^ 1);
          return true;
        };
        ok = half_slot(first) && half_slot(first ^ 1);
        if (!ok) { report(status, 3, 1, e); break; }
        ptx::tc_commit(bar(kEmpty0 + s));
      }
      ptx::tc_commit(bar(kOFinal));
    }
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    // ------------------------------------------------------------------ softmax + epilogue
    const int x = (warp - 4) / 4;                 // 0: tile A, 1: tile B
    const int wq = warp % 4;                      // tensor-memory lane quarter of this warp
    const int r = wq * 32 + lane;                 // row inside the tile
    const int tile = 2 * pair + x;
    const int mine = (blk.flags >> (4 * x)) & 0xf;      // 0: this block does not have the tile
    const int grow = tile * kTile + r;            // global query row
    const int kvl = (grow < q_split) ? kvl_lo : kvl_hi;
    const int kvl_min = min(kvl_lo, kvl_hi);
    const uint32_t lane_base = static_cast<uint32_t>(wq * 32) << 16;
    const uint32_t tS = tmem + lane_base + x * 128;
    const uint32_t tO = tmem + lane_base + 256 + x * D;
    const int rh = r >> 6;

    float m = -INFINITY, l = 0.f;
    uint32_t par_s = 0;
    int done = 0;
    bool ok = true;
    for (int e = 0; e < cnt; ++e) {
      const int en = ent[e];
      const int sub = (en >> (4 * x)) & mine;
      if (!sub) continue;
      const int col0 = (en >> 8) * kTile;
      ok = ptx::mbar_wait(bar(kSFullA + x), par_s, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) { if (lane == 0) report(status, 4, 2 + x, e); break; }
      par_s ^= 1;
      ptx::tc_fence_after();

      float v[kTile];
#pragma unroll
      for (int c = 0; c < 4; ++c) ptx::tmem_ld32(tS + c * 32, reinterpret_cast<uint32_t*>(v) + c * 32);
      ptx::tmem_ld_wait();

      if (sub != 0xf || col0 + kTile > kvl_min) {
        const int lim = kvl - col0;               // columns >= lim are beyond the valid keys
        const bool keep_lo = (sub >> (2 * rh)) & 1;
        const bool keep_hi = (sub >> (2 * rh + 1)) & 1;
#pragma unroll
        for (int c = 0; c < kTile; ++c) {
          const bool valid = (c < 64 ? keep_lo : keep_hi) && (c < lim);
          v[c] = valid ? v[c] : -INFINITY;
        }
      }
      // P = exp2(S*scale - ref) for the whole row, packed to 16 bits and stored over the first 64 columns
      // of S; returns the row sum.
      // row maximum: eight independent chains of three-input max
      float mxa[8];
#pragma unroll
      for (int a = 0; a < 8; ++a) mxa[a] = ptx::max3(v[a], v[a + 8], v[a + 16]);
#pragma unroll
      for (int c = 24; c + 16 <= kTile; c += 16)
#pragma unroll
        for (int a = 0; a < 8; ++a) mxa[a] = ptx::max3(mxa[a], v[c + a], v[c + a + 8]);
#pragma unroll
      for (int a = 0; a < 8; ++a) mxa[a] = fmaxf(mxa[a], v[kTile - 8 + a]);
      const float mx = fmaxf(ptx::max3(mxa[0], mxa[1], mxa[2]), ptx::max3(mxa[3], mxa[4], mxa[5]));
      const float m_new = fmaxf(m, ptx::max3(mx, mxa[6], mxa[7]) * scale_log2);
      if (done == 0) {
        m = m_new;
      } else if (__any_sync(0xffffffffu, m_new > m + kRescaleThreshold)) {
        const float alpha = (m == -INFINITY) ? 0.f : ptx::ex2(m - m_new);
        l *= alpha;
        m = m_new;
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          float o[32];
          ptx::tmem_ld32(tO + c * 32, reinterpret_cast<uint32_t*>(o));
          ptx::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] *= alpha;
          ptx::tmem_st32(tO + c * 32, reinterpret_cast<const uint32_t*>(o));
        }
      }
      // P = exp2(S*scale - m), two fp32 lanes per instruction where the hardware has packed forms.  The row is handed to
      // the MMA warp in two parts, P*V of the first running while the second is still being computed: 96 keys, then 32,
      // so that only two of the eight products are left when the row is done (halves left four; both in turn in one
      // process: HunyuanVideo launch 20.76 -> 20.50 ms, Wan 15.35 -> 15.07, four heads over 8,448 tokens 115 -> 111 us).
      const float ref = (m == -INFINITY) ? 0.f : m;
      const uint64_t scale2 = ptx::pack_f32x2(scale_log2, scale_log2);
      const uint64_t nref2 = ptx::pack_f32x2(-ref, -ref);
      uint64_t sum2a = 0, sum2b = 0;    // bit pattern of (0.f, 0.f)
      auto exp_pairs = [&](int c0, int pairs, uint32_t* pk) {
#pragma unroll
        for (int i = 0; i < pairs; ++i) {
          const uint64_t x2 = ptx::fma_f32x2(ptx::pack_f32x2(v[c0 + 2 * i], v[c0 + 2 * i + 1]), scale2, nref2);
          float x0, x1;
          ptx::unpack_f32x2(x2, x0, x1);
          const float p0 = ptx::ex2(x0), p1 = ptx::ex2(x1);
          const uint64_t p2 = ptx::pack_f32x2(p0, p1);
          if (i & 1) sum2b = ptx::add_f32x2(sum2b, p2); else sum2a = ptx::add_f32x2(sum2a, p2);
          pk[i] = pack2<kBF16>(p0, p1);
        }
      };
      auto hand_over = [&](int part) {
        ptx::tmem_st_wait();
        ptx::tc_fence_before();
        ptx::mbar_arrive(bar(kPLoA + 2 * x + part));
      };
      uint32_t pk[32];
      exp_pairs(0, 32, pk);
      ptx::tmem_st32(tS, pk);
      exp_pairs(64, 16, pk);
      ptx::tmem_st16(tS + 32, pk);
      hand_over(0);
      exp_pairs(96, 16, pk);
      ptx::tmem_st16(tS + 48, pk);
      hand_over(1);
      float s0, s1, s2, s3;
      ptx::unpack_f32x2(sum2a, s0, s1);
      ptx::unpack_f32x2(sum2b, s2, s3);
      const float sum = (s0 + s1) + (s2 + s3);
      l += sum;
      ++done;
    }

    if (ok) {
      ok = ptx::mbar_wait(bar(kOFinal), 0, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok && lane == 0) report(status, 5, 2 + x, -1);
    }
    if (ok && mine != 0 && tile < ntq) {
      ptx::tc_fence_after();
      const float inv = (done > 0 && l > 0.f) ? 1.f / l : 0.f;
      uint4* dst;
      if (scatter.n_peers > 0) {
        const int r = min(grow / scatter.rows_per_peer, scatter.n_peers - 1);
        dst = reinterpret_cast<uint4*>(
            static_cast<unsigned char*>(scatter.peer[r]) +
            (static_cast<int64_t>(scatter.head_base + bh) * scatter.rows_per_peer + (grow - r * scatter.rows_per_peer)) * D * 2);
      } else {
        dst = reinterpret_cast<uint4*>(static_cast<unsigned char*>(out_raw) +
                                       (static_cast<int64_t>(bh) * N + grow) * D * 2);
      }
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        float o[32];
        if (done > 0) {
          ptx::tmem_ld32(tO + c * 32, reinterpret_cast<uint32_t*>(o));
          ptx::tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = 0.f;
        }
        if (grow < N) {
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            uint4 w;
            w.x = pack2<kBF16>(o[q4 * 8 + 0] * inv, o[q4 * 8 + 1] * inv);
            w.y = pack2<kBF16>(o[q4 * 8 + 2] * inv, o[q4 * 8 + 3] * inv);
            w.z = pack2<kBF16>(o[q4 * 8 + 4] * inv, o[q4 * 8 + 5] * inv);
            w.w = pack2<kBF16>(o[q4 * 8 + 6] * inv, o[q4 * 8 + 7] * inv);
            dst[c * 4 + q4] = w;
          }
        }
      }
      if (lse != nullptr && grow < N) {
        lse[static_cast<int64_t>(bh) * N + grow] =
            (done > 0 && l > 0.f) ? (m + log2f(l)) * 0.6931471805599453f : -INFINITY;
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

// ====================================================================================================
// Head dimension 64.
//
// At D = 64 a tile carries half the tensor work of the D = 128 tile for the same exponentials, and two softmax warps per
// scheduler do not fill the exponential unit: with one warpgroup per query tile and 128-key rows a slot (two query tiles x
// one key tile) took 3,100 clocks for 2,048 of that unit, both warps busy throughout with latencies of their own.  So every
// query tile has two independent chains, one for either 64-key half of its key tiles: scores, online softmax with a
// reference and a sum of its own, P V into an accumulator of its own - four warpgroups, four warps per scheduler, nothing
// exchanged until the two accumulators of a row are put together at the end.
//   S_c [64 c, 64 c + 64)   O_c [256 + 64 c, 320 + 64 c)   for chain c = 2 * tile + half; P_c (16-bit) overwrites the first
//   32 columns of S_c.
// Each query tile has an issuing thread that takes its two chains in turn, PV(0,e) QK(0,e+1) PV(1,e) QK(1,e+1); a chain that
// entry e does not concern has its QK(e+1) first.  Products of one thread execute in order, which makes the aliasing of P and
// S safe and lets "S ready" imply that the chain's previous P V is done.  A half that neither half of the tile's rows keeps
// costs nothing.
// Measured, launch alone, before -> now, in turn in one process: 48 heads x 45,104 tokens at 12 % of the blocks 4.87 -> 4.19
// ms, 32 heads x 16,640 tokens at 33 % 1.22 -> 1.08, dense 48 heads x 20,624 tokens 7.29 -> 6.17 (7.35 -> 6.65 where the power
// limit holds the clock down after a second of such launches).
// ====================================================================================================
constexpr int kThreads64 = 640;   // 4 control warps, 4 softmax warpgroups
constexpr int kStages64 = 3;      // K and V tiles in flight (16 KB each); four would not fit beside the merge buffer
enum BarrierIndex64 {
  k6QFull = 0,
  k6KFirst,
  k6Full0,                                       // [kStages64] V(e) and K(e + 1) have landed (index e % kStages64)
  k6DoneA0 = k6Full0 + kStages64,                // [kStages64] tile A's issuer has finished all its MMAs of slot e
  k6DoneB0 = k6DoneA0 + kStages64,               // [kStages64] the same for tile B
  k6SFull = k6DoneB0 + kStages64,                // [4] scores of a chain are ready
  k6OFinal = k6SFull + 4,                        // [2] all products of a query tile are done
  k6P = k6OFinal + 2,                            // [4] P of a chain has been stored (128 arrivals)
  k6NumBarriers = k6P + 4
};

struct __align__(8) Control64 {
  unsigned long long bars[k6NumBarriers];
  uint32_t tmem_base;
  int abort_flag;
};

// per query tile: 64 accumulator columns, reference and sum of the second chain's rows
constexpr int kMergeFloats64 = 66 * kTile;

constexpr size_t smem_bytes_d64() {
  return static_cast<size_t>(2 + 2 * kStages64) * kTile * 64 * 2 + 2 * kMergeFloats64 * sizeof(float) + 1024 +
         sizeof(Control64);
}

// Maximum of 64 values: eight independent chains of three-input max.
__device__ __forceinline__ float row_max64(const float* v) {
  float a[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) a[i] = ptx::max3(v[i], v[i + 8], v[i + 16]);
#pragma unroll
  for (int c = 24; c + 16 <= 64; c += 16)
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = ptx::max3(a[i], v[c + i], v[c + i + 8]);
#pragma unroll
  for (int i = 0; i < 8; ++i) a[i] = fmaxf(a[i], v[56 + i]);
  return fmaxf(ptx::max3(a[0], a[1], a[2]), ptx::max3(ptx::max3(a[3], a[4], a[5]), a[6], a[7]));
}

// P = exp2(S * scale - ref) for 2 * kPairs columns of one row: pk = 16-bit pairs; the row sum goes into the packed sums.
template <bool kBF16, int kPairs>
__device__ __forceinline__ void exp_pairs(const float* v, float scale_log2, float ref, uint32_t* pk, uint64_t& sum2a,
                                          uint64_t& sum2b) {
  const uint64_t scale2 = ptx::pack_f32x2(scale_log2, scale_log2);
  const uint64_t nref2 = ptx::pack_f32x2(-ref, -ref);
#pragma unroll
  for (int i = 0; i < kPairs; ++i) {
    const uint64_t x2 = ptx::fma_f32x2(ptx::pack_f32x2(v[2 * i], v[2 * i + 1]), scale2, nref2);
    float x0, x1;
    ptx::unpack_f32x2(x2, x0, x1);
    const float p0 = ptx::ex2(x0), p1 = ptx::ex2(x1);
    const uint64_t p2 = ptx::pack_f32x2(p0, p1);
    if (i & 1) sum2b = ptx::add_f32x2(sum2b, p2); else sum2a = ptx::add_f32x2(sum2a, p2);
    pk[i] = pack2<kBF16>(p0, p1);
  }
}

template <bool kBF16>
__global__ void __launch_bounds__(kThreads64, 1) sparse_attn_fwd_d64_kernel(
    const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
    const __grid_constant__ CUtensorMap tm_v, const int32_t* __restrict__ counts,
    const int32_t* __restrict__ entries, const int32_t* __restrict__ order, int Hm, int ntk, int N, float scale_log2,
    int q_split, int kvl_lo, int kvl_hi, int n_single, void* __restrict__ out_raw, float* __restrict__ lse,
    int32_t* __restrict__ status, const __grid_constant__ OutScatter scatter) {
  constexpr int D = 64;
  constexpr int kTileBytes = kTile * D * 2;       // one Q, K or V tile: 128 rows x 128 bytes
  constexpr uint32_t kIdescQK = ptx::idesc_f16(128, 64, kBF16, false);
  constexpr uint32_t kIdescPV = ptx::idesc_f16(128, D, kBF16, true);

  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* merge = reinterpret_cast<float*>(smem + (2 + 2 * kStages64) * kTileBytes);
  Control64* ctl = reinterpret_cast<Control64*>(merge + 2 * kMergeFloats64);
  const uint32_t sQ = ptx::smem_u32(smem);
  const uint32_t sK = sQ + 2 * kTileBytes;
  const uint32_t sV = sK + kStages64 * kTileBytes;
  const uint32_t bar0 = ptx::smem_u32(&ctl->bars[0]);
  auto bar = [&](int i) { return bar0 + 8u * static_cast<uint32_t>(i); };
  volatile int* abort_flag = &ctl->abort_flag;

  const int warp = ptx::warp_index();
  const int lane = threadIdx.x % 32;
  const BlockItem blk(n_single, Hm, order);
  const int npairs = blk.npairs, item = blk.item;
  const int mh = item / npairs;
  const int pair = item - mh * npairs;
  const int bh = blockIdx.y * Hm + mh;
  const int ntq = (N + kTile - 1) / kTile;
  if (2 * pair + (blk.flags == 0xf0) >= ntq) return;          // the second query tile of a pair that has one only
  const int cnt = counts[static_cast<int64_t>(mh) * npairs + pair];
  const int32_t* ent = entries + (static_cast<int64_t>(mh) * npairs + pair) * ntk;

  if (threadIdx.x == 0) {
    for (int i = 0; i < k6NumBarriers; ++i) ptx::mbar_init(bar(i), i >= k6P ? 128u : 1u);
    ctl->abort_flag = 0;
    ptx::fence_barrier_init();
    ptx::prefetch_tensormap(&tm_q);
    ptx::prefetch_tensormap(&tm_k);
    ptx::prefetch_tensormap(&tm_v);
  }
  if (warp == 2) {
    ptx::tmem_alloc(ptx::smem_u32(&ctl->tmem_base), 512);
    ptx::tmem_relinquish();
    ptx::tc_fence_before();
  }
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;

  // Slot j's completion shows on k6Done_X[j % kStages64].  "Slot -1" is the Q K^T of entry 0, issued before the loop:
  // it shares the last index, whose phases are therefore one ahead of the others'.
  auto done_index = [](int j) -> int { return (j + kStages64) % kStages64; };
  auto done_parity = [](int j) -> uint32_t {
    return static_cast<uint32_t>((((j + kStages64) % kStages64 == kStages64 - 1) ? (j + 1) / kStages64 : j / kStages64) & 1);
  };

  // 640 threads start with 96 registers each, 61,440 in all; of these 128 x 40 + 512 x 104 = 58,368 are kept.
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer
      if (ptx::elect_one()) {
        const int q0 = blk.flags == 0xf0, q1 = blk.flags != 0x0f && 2 * pair + 1 < ntq;      // first and last query tile
        ptx::mbar_expect_tx(bar(k6QFull), (q1 - q0 + 1) * kTileBytes);
        for (int x = q0; x <= q1; ++x)
          ptx::tma_load_3d(sQ + x * kTileBytes, &tm_q, bar(k6QFull), 0, (2 * pair + x) * kTile, bh);
        bool ok = true;
        int issued = 0;
        if (cnt > 0) {
          ptx::mbar_expect_tx(bar(k6KFirst), kTileBytes);
          ptx::tma_load_3d(sK, &tm_k, bar(k6KFirst), 0, (ent[0] >> 8) * kTile, bh);
        }
        // entry e: V(e) into V stage e % kStages64 and K(e + 1) into K stage (e + 1) % kStages64, once slot
        // e - kStages64 has completed in both tiles (it read both stages last)
        for (int e = 0; e < cnt && ok; ++e) {
          const int s = e % kStages64;
          const bool next = (e + 1) < cnt;
          if (e >= kStages64 - 1) {
            const int j = e - kStages64;
            ok = ptx::mbar_wait(bar(k6DoneA0 + done_index(j)), done_parity(j), abort_flag) &&
                 ptx::mbar_wait(bar(k6DoneB0 + done_index(j)), done_parity(j), abort_flag);
            if (!ok) { report(status, 1, 0, e); break; }
          }
          ptx::mbar_expect_tx(bar(k6Full0 + s), (next ? 2u : 1u) * kTileBytes);
          ptx::tma_load_3d(sV + s * kTileBytes, &tm_v, bar(k6Full0 + s), 0, (ent[e] >> 8) * kTile, bh);
          if (next)
            ptx::tma_load_3d(sK + ((e + 1) % kStages64) * kTileBytes, &tm_k, bar(k6Full0 + s), 0, (ent[e + 1] >> 8) * kTile,
                             bh);
          issued = e + 1;
        }
        if (!ok) {
          // give copies in flight a bounded time to land (their barriers may never be consumed)
          for (int i = 0; i < 4096 && cnt > 0 && !ptx::mbar_try_wait(bar(k6KFirst), 0); ++i) {}
          for (int e = max(0, issued - kStages64); e < issued; ++e)
            for (int i = 0; i < 4096 && !ptx::mbar_try_wait(bar(k6Full0 + e % kStages64), (e / kStages64) & 1); ++i) {}
        }
      }
    } else if (warp == 1 || warp == 3) {
      // ------------------------------------------------------------------ MMA issuers, one per query tile
      if (ptx::elect_one()) {
        const int x = warp >> 1;
        const uint64_t dqx = ptx::smem_desc_sw128(sQ + x * kTileBytes, 16, 1024);
        const uint64_t dk0 = ptx::smem_desc_sw128(sK, 16, 1024);
        const uint64_t dv0 = ptx::smem_desc_sw128(sV, kTileBytes, 1024);
        auto advance = [](uint64_t desc, uint32_t bytes) -> uint64_t {
          return (desc & 0xffffffff00000000ull) | static_cast<uint32_t>(static_cast<uint32_t>(desc) + (bytes >> 4));
        };
        // the 64-key halves of an entry that the tile keeps in either half of its rows
        auto halves = [&](int e) -> uint32_t {
          const uint32_t f = static_cast<uint32_t>(ent[e] & blk.flags) >> (4 * x);
          return (f | (f >> 2)) & 3u;
        };
        auto issue_qk = [&](int h, int s) {   // s: K stage
          const uint64_t b0 = advance(dk0, static_cast<uint32_t>(s) * kTileBytes + h * (kTileBytes / 2));
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk)
            ptx::mma_ss(tmem + (2 * x + h) * 64, advance(dqx, kk * 32), advance(b0, kk * 32), kIdescQK, kk > 0 ? 1u : 0u);
          ptx::tc_commit(bar(k6SFull + 2 * x + h));
        };
        bool ok = ptx::mbar_wait(bar(k6QFull), 0, abort_flag);
        if (!ok) report(status, 2, 1 + x, -1);
        // halves of entry e, e + 1 and e + 2: each is loaded two slots before the issuer needs it (a load issued
        // where its value is used would put a trip to the L2 on the issuing thread's path every slot)
        uint32_t sub = (cnt > 0) ? halves(0) : 0u, subn = (cnt > 1) ? halves(1) : 0u;
        if (ok && cnt > 0) {
          ok = ptx::mbar_wait(bar(k6KFirst), 0, abort_flag);
          if (!ok) report(status, 2, 1 + x, 0);
          if (ok) {
            ptx::tc_fence_after();
            if (sub & 1u) issue_qk(0, 0);
            if (sub & 2u) issue_qk(1, 0);
            ptx::tc_commit(bar(k6DoneA0 + kStages64 * x + kStages64 - 1));   // "slot -1": K stage 0 is free again
          }
        }
        uint32_t par_p = 0, acc = 0;          // a bit per chain
        for (int e = 0; e < cnt && ok; ++e) {
          const int s = e % kStages64;
          const uint32_t subnn = (e + 2 < cnt) ? halves(e + 2) : 0u;   // first used in the next slot
          ok = ptx::mbar_wait(bar(k6Full0 + s), (e / kStages64) & 1, abort_flag);
          if (!ok) { report(status, 2, 1 + x, e); break; }
          // a chain that this entry does not concern starts on the next one before the other chain's P is waited for
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if (((subn & ~sub) >> h) & 1u) issue_qk(h, (e + 1) % kStages64);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if ((sub >> h) & 1u) {
              ok = ptx::mbar_wait(bar(k6P + 2 * x + h), (par_p >> h) & 1u, abort_flag);
              if (!ok) { report(status, 3, 1 + x, e); break; }
              ptx::tc_fence_after();
              const uint64_t b0 = advance(dv0, static_cast<uint32_t>(s) * kTileBytes + h * (kTileBytes / 2));
#pragma unroll
              for (int kk = 0; kk < 4; ++kk)
                ptx::mma_ts(tmem + 256 + (2 * x + h) * 64, tmem + (2 * x + h) * 64 + kk * 8, advance(b0, kk * 2048), kIdescPV,
                            (((acc >> h) & 1u) || kk > 0) ? 1u : 0u);
              par_p ^= 1u << h;
              acc |= 1u << h;
              if ((subn >> h) & 1u) issue_qk(h, (e + 1) % kStages64);
            }
          }
          if (!ok) break;
          ptx::tc_commit(bar(k6DoneA0 + kStages64 * x + s));  // this tile's MMAs of slot e are done
          sub = subn;
          subn = subnn;
        }
        ptx::tc_commit(bar(k6OFinal + x));
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    // ------------------------------------------------------------------ softmax + epilogue
    const int chain = (warp - 4) / 4;             // 2 * query tile + key half
    const int x = chain >> 1, h = chain & 1;
    const int wq = warp % 4;                      // tensor-memory lane quarter of this warp
    const int r = wq * 32 + lane;                 // row inside the tile
    const int tile = 2 * pair + x;
    const int grow = tile * kTile + r;            // global query row
    const int kvl = (grow < q_split) ? kvl_lo : kvl_hi;
    const int kvl_min = min(kvl_lo, kvl_hi);
    const uint32_t lane_base = static_cast<uint32_t>(wq * 32) << 16;
    const uint32_t tS = tmem + lane_base + chain * 64;
    const uint32_t tO = tmem + lane_base + 256 + chain * 64;
    const int bit_mine = 4 * x + 2 * (r >> 6) + h;     // flag of this row half (the same for the whole warp)
    const int bits_both = (0x5 << (4 * x + h)) & blk.flags;   // flags of this key half, both row halves

    float m = -INFINITY, l = 0.f;
    uint32_t par_s = 0;
    int done = 0;
    bool ok = true;
    int en_next = (cnt > 0) ? ent[0] : 0;
    for (int e = 0; e < cnt; ++e) {
      const int en = en_next;
      en_next = (e + 1 < cnt) ? ent[e + 1] : 0;   // in flight while this entry is processed
      if (!(en & bits_both)) continue;
      ok = ptx::mbar_wait(bar(k6SFull + chain), par_s, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) { if (lane == 0) report(status, 4, 2 + chain, e); break; }
      par_s ^= 1;
      ptx::tc_fence_after();
      if ((en >> bit_mine) & 1) {
        float v[64];
        ptx::tmem_ld32(tS, reinterpret_cast<uint32_t*>(v));
        ptx::tmem_ld32(tS + 32, reinterpret_cast<uint32_t*>(v) + 32);
        ptx::tmem_ld_wait();
        const int col0 = (en >> 8) * kTile + h * 64;
        if (col0 + 64 > kvl_min) {                // the half reaches past the valid keys of some row
          const int lim = kvl - col0;             // columns >= lim are beyond the valid keys of this row
#pragma unroll
          for (int c = 0; c < 64; ++c) v[c] = (c < lim) ? v[c] : -INFINITY;
        }
        const float m_new = fmaxf(m, row_max64(v) * scale_log2);
        // A new reference rescales O; that is done below, before P is handed over, so that the exponentials follow the
        // row maximum in one piece of straight code.
        const bool rescale = done > 0 && __any_sync(0xffffffffu, m_new > m + kRescaleThreshold);
        const float alpha = (m == -INFINITY) ? 0.f : ptx::ex2(m - m_new);
        if (rescale) l *= alpha;
        if (rescale || done == 0) m = m_new;
        const float ref = (m == -INFINITY) ? 0.f : m;
        uint64_t sum2a = 0, sum2b = 0;    // bit pattern of (0.f, 0.f)
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          uint32_t pk[16];
          exp_pairs<kBF16, 16>(v + 32 * part, scale_log2, ref, pk, sum2a, sum2b);
          ptx::tmem_st16(tS + 16 * part, pk);
        }
        float s0, s1, s2, s3;
        ptx::unpack_f32x2(sum2a, s0, s1);
        ptx::unpack_f32x2(sum2b, s2, s3);
        l += (s0 + s1) + (s2 + s3);
        if (rescale) {
#pragma unroll
          for (int c = 0; c < D / 16; ++c) {
            float o[16];
            ptx::tmem_ld16(tO + c * 16, reinterpret_cast<uint32_t*>(o));
            ptx::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] *= alpha;
            ptx::tmem_st16(tO + c * 16, reinterpret_cast<const uint32_t*>(o));
          }
        }
      } else {
        uint32_t pk[16];                          // a half this row half does not keep: no exponentials at all
#pragma unroll
        for (int i = 0; i < 16; ++i) pk[i] = 0u;
        ptx::tmem_st16(tS, pk);
        ptx::tmem_st16(tS + 16, pk);
      }
      ptx::tmem_st_wait();
      ptx::tc_fence_before();
      ptx::mbar_arrive(bar(k6P + chain));
      ++done;
    }

    if (ok) {
      ok = ptx::mbar_wait(bar(k6OFinal + x), 0, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok && lane == 0) report(status, 5, 2 + chain, -1);
    }
    ptx::tc_fence_after();
    // The second chain hands its rows to the first through shared memory, which puts the two together and stores them.
    float* mg = merge + x * kMergeFloats64;
    if (h == 1) {
#pragma unroll
      for (int c = 0; c < D / 16; ++c) {
        float o[16];
        if (done > 0 && ok) {
          ptx::tmem_ld16(tO + c * 16, reinterpret_cast<uint32_t*>(o));
          ptx::tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = 0.f;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) mg[(c * 16 + i) * kTile + r] = o[i];
      }
      mg[64 * kTile + r] = m;
      mg[65 * kTile + r] = l;
    }
    if (x == 0) asm volatile("bar.sync 1, 256;" ::: "memory");
    else asm volatile("bar.sync 2, 256;" ::: "memory");
    if (h == 0 && ok && bits_both != 0 && tile < ntq) {
      const float m1 = mg[64 * kTile + r], l1 = mg[65 * kTile + r];
      const float mm = fmaxf(m, m1);
      const float w0 = (m == -INFINITY) ? 0.f : ptx::ex2(m - mm);
      const float w1 = (m1 == -INFINITY) ? 0.f : ptx::ex2(m1 - mm);
      const float lt = l * w0 + l1 * w1;
      const float inv = lt > 0.f ? 1.f / lt : 0.f;
      const float f0 = w0 * inv, f1 = w1 * inv;
      uint4* dst;
      if (scatter.n_peers > 0) {
        const int pr = min(grow / scatter.rows_per_peer, scatter.n_peers - 1);
        dst = reinterpret_cast<uint4*>(
            static_cast<unsigned char*>(scatter.peer[pr]) +
            (static_cast<int64_t>(scatter.head_base + bh) * scatter.rows_per_peer + (grow - pr * scatter.rows_per_peer)) * D * 2);
      } else {
        dst = reinterpret_cast<uint4*>(static_cast<unsigned char*>(out_raw) + (static_cast<int64_t>(bh) * N + grow) * D * 2);
      }
#pragma unroll
      for (int c = 0; c < D / 16; ++c) {
        float o[16];
        if (done > 0) {
          ptx::tmem_ld16(tO + c * 16, reinterpret_cast<uint32_t*>(o));
          ptx::tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = 0.f;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) o[i] = o[i] * f0 + mg[(c * 16 + i) * kTile + r] * f1;
        if (grow < N) {
#pragma unroll
          for (int q4 = 0; q4 < 2; ++q4) {
            uint4 w;
            w.x = pack2<kBF16>(o[q4 * 8 + 0], o[q4 * 8 + 1]);
            w.y = pack2<kBF16>(o[q4 * 8 + 2], o[q4 * 8 + 3]);
            w.z = pack2<kBF16>(o[q4 * 8 + 4], o[q4 * 8 + 5]);
            w.w = pack2<kBF16>(o[q4 * 8 + 6], o[q4 * 8 + 7]);
            dst[c * 2 + q4] = w;
          }
        }
      }
      if (lse != nullptr && grow < N) {
        lse[static_cast<int64_t>(bh) * N + grow] = lt > 0.f ? (mm + log2f(lt)) * 0.6931471805599453f : -INFINITY;
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

template <bool kBF16>
int launch_d64(const void* q, const void* k, const void* v, int dtype, int BH, int N, const int32_t* counts,
               const int32_t* entries, const int32_t* order, int Hm, float softmax_scale, int q_split, int kvl_lo,
               int kvl_hi, int pairs_beside, void* out, float* lse, int32_t* status, const OutScatter& scatter, cudaStream_t st) {
  CUtensorMap tq, tk, tv;
  if (int rc = make_tmap_rows(&tq, q, dtype, BH, N, 64, kTile)) return rc;
  if (int rc = make_tmap_rows(&tk, k, dtype, BH, N, 64, kTile)) return rc;
  if (int rc = make_tmap_rows(&tv, v, dtype, BH, N, 64, kTile)) return rc;
  const int ntq = ceil_div(N, kTile);
  const int npairs = (ntq + 1) / 2;
  auto kernel = sparse_attn_fwd_d64_kernel<kBF16>;
  const size_t smem = smem_bytes_d64();
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem)) return rc;
  const float scale_log2 = softmax_scale * 1.4426950408889634f;
  int sms = 0;
  if (int rc = sm_count(&sms)) return rc;
  const int n_single = single_pairs(sms, npairs * Hm, BH / Hm, pairs_beside);
  kernel<<<dim3(npairs * Hm + n_single, BH / Hm), kThreads64, smem, st>>>(tq, tk, tv, counts, entries, order, Hm, ntq, N,
                                                                         scale_log2, q_split, kvl_lo, kvl_hi, n_single, out,
                                                                         lse, status, scatter);
  MODDIT_CHECK_LAUNCH("sparse_attn_fwd_d64_kernel");
  return MODDIT_OK;
}

template <int D, bool kBF16>
int launch(const void* q, const void* k, const void* v, int dtype, int BH, int N, const int32_t* counts,
           const int32_t* entries, const int32_t* order, int Hm, float softmax_scale, int q_split, int kvl_lo, int kvl_hi,
           int pairs_beside, void* out, float* lse, int32_t* status, const OutScatter& scatter, cudaStream_t st) {
  CUtensorMap tq, tk, tv;
  if (int rc = make_tmap_rows(&tq, q, dtype, BH, N, D, kTile)) return rc;
  if (int rc = make_tmap_rows(&tk, k, dtype, BH, N, D, kTile)) return rc;
  if (int rc = make_tmap_rows(&tv, v, dtype, BH, N, D, kTile)) return rc;
  const int ntq = ceil_div(N, kTile);
  const int npairs = (ntq + 1) / 2;
  auto kernel = sparse_attn_fwd_kernel<D, kBF16>;
  const size_t smem = smem_bytes<D>();
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem)) return rc;
  const float scale_log2 = softmax_scale * 1.4426950408889634f;
  int sms = 0;
  if (int rc = sm_count(&sms)) return rc;
  const int n_single = single_pairs(sms, npairs * Hm, BH / Hm, pairs_beside);
  kernel<<<dim3(npairs * Hm + n_single, BH / Hm), kThreads, smem, st>>>(tq, tk, tv, counts, entries, order, Hm, ntq, N,
                                                                       scale_log2, q_split, kvl_lo, kvl_hi, n_single, out,
                                                                       lse, status, scatter);
  MODDIT_CHECK_LAUNCH("sparse_attn_fwd_kernel");
  return MODDIT_OK;
}

}  // namespace
}  // namespace moddit

using namespace moddit;

extern "C" int moddit_sparse_attn_single_pairs(int sms, int pairs, int batches, int pairs_beside) {
  return sms > 0 && pairs > 0 && batches > 0 && pairs_beside >= 0 ? single_pairs(sms, pairs, batches, pairs_beside) : 0;
}

static int sparse_attn_dispatch(const void* q, const void* k, const void* v, int dtype, int BH, int N, int D,
                                const int32_t* counts, const int32_t* entries, const int32_t* order, int Hm,
                                float softmax_scale, int q_split, int kv_len_lo, int kv_len_hi, int pairs_beside, void* out,
                                float* lse, int32_t* status, const OutScatter& scatter, void* stream) {
  MODDIT_CHECK_ARG(q && k && v && counts && entries && status, "sparse_attn_fwd: null pointer");
  MODDIT_CHECK_ARG(out || scatter.n_peers > 0, "sparse_attn_fwd: no output destination");
  MODDIT_CHECK_ARG(BH > 0 && BH <= 65535 && N > 0 && Hm > 0, "sparse_attn_fwd: BH=%d N=%d Hm=%d out of range", BH, N, Hm);
  MODDIT_CHECK_ARG(BH % Hm == 0, "sparse_attn_fwd: BH=%d is not a multiple of the mask heads Hm=%d", BH, Hm);
  MODDIT_CHECK_ARG(softmax_scale > 0.f, "sparse_attn_fwd: softmax_scale must be positive");
  MODDIT_CHECK_ARG(kv_len_lo >= 0 && kv_len_lo <= N && kv_len_hi >= 0 && kv_len_hi <= N,
                   "sparse_attn_fwd: kv_len (%d, %d) outside [0, N=%d]", kv_len_lo, kv_len_hi, N);
  MODDIT_CHECK_ARG(pairs_beside >= 0, "sparse_attn_fwd: pairs_beside=%d must not be negative", pairs_beside);
  if (D != 64 && D != 128) return fail(MODDIT_E_UNSUPPORTED, "sparse_attn_fwd: head_dim must be 64 or 128, got %d", D);
  if (dtype != MODDIT_BF16 && dtype != MODDIT_FP16) return fail(MODDIT_E_ARG, "sparse_attn_fwd: unknown dtype %d", dtype);
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(out))
    return fail(MODDIT_E_ALIGN, "sparse_attn_fwd: q, k, v and out must be 16-byte aligned");
  if (int rc = require_sm100()) return rc;
  cudaStream_t st = as_stream(stream);
  if (D == 128) {
    return dtype == MODDIT_BF16
               ? launch<128, true>(q, k, v, dtype, BH, N, counts, entries, order, Hm, softmax_scale, q_split, kv_len_lo,
                                   kv_len_hi, pairs_beside, out, lse, status, scatter, st)
               : launch<128, false>(q, k, v, dtype, BH, N, counts, entries, order, Hm, softmax_scale, q_split, kv_len_lo,
                                    kv_len_hi, pairs_beside, out, lse, status, scatter, st);
  }
  return dtype == MODDIT_BF16
             ? launch_d64<true>(q, k, v, dtype, BH, N, counts, entries, order, Hm, softmax_scale, q_split, kv_len_lo, kv_len_hi,
                                pairs_beside, out, lse, status, scatter, st)
             : launch_d64<false>(q, k, v, dtype, BH, N, counts, entries, order, Hm, softmax_scale, q_split, kv_len_lo, kv_len_hi,
                                 pairs_beside, out, lse, status, scatter, st);
}

static int scatter_to(OutScatter* sc, void* const* peer_out, int n_peers, int N, int head_base) {
  MODDIT_CHECK_ARG(peer_out, "sparse_attn_fwd_scatter: null peer table");
  MODDIT_CHECK_ARG(n_peers >= 1 && n_peers <= kMaxPeers, "sparse_attn_fwd_scatter: n_peers=%d outside [1, %d]", n_peers,
                   kMaxPeers);
  MODDIT_CHECK_ARG(N % n_peers == 0, "sparse_attn_fwd_scatter: N=%d does not divide over %d peers", N, n_peers);
  MODDIT_CHECK_ARG(head_base >= 0, "sparse_attn_fwd_scatter: head_base must be non-negative");
  for (int i = 0; i < n_peers; ++i) {
    MODDIT_CHECK_ARG(peer_out[i] && aligned16(peer_out[i]), "sparse_attn_fwd_scatter: peer buffer %d null or unaligned", i);
    sc->peer[i] = peer_out[i];
  }
  sc->n_peers = n_peers;
  sc->rows_per_peer = N / n_peers;
  sc->head_base = head_base;
  return MODDIT_OK;
}

extern "C" int moddit_sparse_attn_fwd(const void* q, const void* k, const void* v, int dtype, int BH, int N, int D,
                                      const int32_t* counts, const int32_t* entries, const int32_t* order, int Hm,
                                      float softmax_scale, int q_split, int kv_len_lo, int kv_len_hi, void* out,
                                      float* lse, int32_t* status, void* stream) {
  clear_error();
  MODDIT_CHECK_ARG(out, "sparse_attn_fwd: null output pointer");
  return sparse_attn_dispatch(q, k, v, dtype, BH, N, D, counts, entries, order, Hm, softmax_scale, q_split, kv_len_lo,
                              kv_len_hi, 0, out, lse, status, OutScatter{}, stream);
}

extern "C" int moddit_sparse_attn_fwd_scatter(const void* q, const void* k, const void* v, int dtype, int BH, int N,
                                              int D, const int32_t* counts, const int32_t* entries,
                                              const int32_t* order, int Hm, float softmax_scale, int q_split,
                                              int kv_len_lo, int kv_len_hi, void* const* peer_out, int n_peers,
                                              int head_base, float* lse, int32_t* status, void* stream) {
  clear_error();
  OutScatter sc = {};
  if (int rc = scatter_to(&sc, peer_out, n_peers, N, head_base)) return rc;
  return sparse_attn_dispatch(q, k, v, dtype, BH, N, D, counts, entries, order, Hm, softmax_scale, q_split, kv_len_lo,
                              kv_len_hi, 0, nullptr, lse, status, sc, stream);
}

extern "C" int moddit_sparse_attn_fwd_beside(const void* q, const void* k, const void* v, int dtype, int BH, int N, int D,
                                             const int32_t* counts, const int32_t* entries, const int32_t* order, int Hm,
                                             float softmax_scale, int q_split, int kv_len_lo, int kv_len_hi, int pairs_beside,
                                             void* out, void* const* peer_out, int n_peers, int head_base, float* lse,
                                             int32_t* status, void* stream) {
  clear_error();
  MODDIT_CHECK_ARG((out != nullptr) != (peer_out != nullptr), "sparse_attn_fwd_beside: one output destination, not both or none");
  OutScatter sc = {};
  if (peer_out != nullptr)
    if (int rc = scatter_to(&sc, peer_out, n_peers, N, head_base)) return rc;
  return sparse_attn_dispatch(q, k, v, dtype, BH, N, D, counts, entries, order, Hm, softmax_scale, q_split, kv_len_lo,
                              kv_len_hi, pairs_beside, out, lse, status, sc, stream);
}
