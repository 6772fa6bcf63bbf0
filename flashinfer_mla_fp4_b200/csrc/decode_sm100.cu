// FP4 MLA decode for sm_100a: persistent, warp-specialised, tcgen05 + TMEM + TMA.
//
// One CTA per SM walks a contiguous range of 128-token KV tiles (common.cuh: work partition).
// For a tile of request b and a group of 64 query heads the CTA computes, with tokens on the
// MMA M axis ("swapped" orientation, so 64 heads do not waste half of a 128-row MMA):
//
//   S_lat^T [128 tok, 64 head] = K_lat (E2M1, 128x512)  . Q_lat^T(E4M3)  16 x tcgen05.mma K=32
//   S_rope^T[128 tok, 64 head] = K_rope(E4M3, 128x64)   . Q_rope^T        2 x tcgen05.mma
//   x = (scale_t * S_lat + S_rope) * softmax_scale*log2(e)              per token row, registers
//   P' = exp2(x - m_head) * scale_t, split into E4M3 hi + E4M3 lo       (two terms ~ 8 mantissa bits)
//   O^T[512 dim, 64 head] += V^T (E2M1, MN-major view of the same K_lat tile) . (P'_hi + P'_lo)
//
// The packed E2M1 latent goes from global memory to shared memory by TMA with the 4-bit tensor-map
// type that writes every 16 codes as 8 bytes of data + 8 bytes of padding: the form in which
// tcgen05.mma.kind::f8f6f4 reads 4-bit operands.  A 128-dim block of a tile is then [128 tokens][128 B]
// with the 128-byte swizzle, and the very same bytes serve as the K-major A operand of QK^T and as the
// MN-major A operand of PV: there is no conversion pass and no copy of the tile in any other format.
// RoPE bytes, per-token scales and Q arrive by TMA as well.
//
// What bounds it (measured with one MMA form at a time, operands in shared memory): at N = 64 an MMA reads A (4 KiB) and
// B (2 KiB) at the 128 B/clk of shared memory, 48 clk, and a PV pair that shares A through the collector takes 78: the 18 + 32
// MMAs of a tile measured alone take 863 + 1248 = 2111 clk of tensor pipe, beside 72 KiB of TMA writes (560 clk of the same port).  A
// tile takes 2300 (8x32768 tokens, from a CTA's fifth tile to its last): the pipe also waits for P', whose one buffer is free when the last PV has completed.
// Everything else is arranged to stay under that:
//   * latent blocks are handled in pairs (32 KiB, five pair slots = two and a half tiles in flight): one barrier, one wait
//     and one commit per pair;
//   * QK^T and PV are issued by a warp each: the queue of the tensor pipe is short, so a gap in one warp's issue (a wait, the
//     bookkeeping of a tile) is a gap of the pipe unless the other warp has something queued (one warp for both, in the order
//     PV(t), QK(t+2), measured 106 us where two take 88).  The two take turns all the same: PV(t) follows QK(t+1), and QK(t+2)
//     is let in when PV(t) is half issued.  That way the pipe has QK^T to work on while P(t+1), which may be stored only when
//     PV(t) has completed, is on its way; left alone, the two streams ran side by side and then both waited (92.7 us).
//   * two warps issue the copies of a tile (pair 0 and scales | RoPE and pair 1).  Each issues from one elected lane with
//     page ids fetched 32 at a time.  (With per-lane copies, per-line L2 prefetches and a vote per wait, the one copy warp of
//     an earlier version took 3500 clk per tile and bounded the whole kernel: 51.6 us for the north star, 138 us for B=2,
//     H=128, q_len=2, 131072 tokens.  The TMA unit itself needs 870 clk for a tile that is in L2.)
//
// Warp roles (384 threads): 0 QK^T issue and Q loads, 1 and 3 TMA issue, 2 merge plan and PV issue (issue warps run
// warp-uniform code, one elected lane per instruction), 4-11 softmax / O rescale / epilogue (TMEM lane = token or dim; two
// warps share a lane quarter and split the 64 heads).
//
// Requests that are split across CTAs are merged at the end of the same kernel (tail_merge).  The two-kernel mode leaves the
// merge to the combine kernel instead.
//
// Code that runs once per launch is fetched cold: 1 clk per instruction within 32 KiB of code, 2.6 within 128 KiB, 6 to 11
// beyond (measured with straight-line code).  So the loops are rolled and the one-shot paths small.
//
// Every wait is bounded: when a wait expires the CTA records MLA_FP4_ERR_DEVICE_TIMEOUT in the
// status words, stops issuing work, drains and exits normally.
#include <atomic>

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include "common.cuh"
#include "launch.h"
#include "ptx_sm100.cuh"

namespace mla {

namespace {

constexpr int kWarpQK = 0, kWarpTMA = 1, kWarpPV = 2, kWarpTMA2 = 3;
constexpr int kFetchWarps = 3;         // TMA, PV, TMA2: they fetch the partials to merge
constexpr int kWarpPlan = 11;          // the softmax warp that makes the first plan while the dependency is waited for
constexpr int kWarpSoftmax0 = 4;       // 8 warps; warp & 3 is the TMEM lane quarter the warp may access
constexpr int kThreads = 384;          // 12 warps, three per scheduler
constexpr int kSoftmaxWarps = 8;       // warp w works on TMEM lanes 32*(w%4).. and heads 32*(w/4)..
constexpr int kSoftmaxThreads = 32 * kSoftmaxWarps;
constexpr int kRing = 5;                   // pairs of latent blocks in flight: two and a half tiles
constexpr int kBlocks = 4;                 // 128-dim blocks of the latent
constexpr int kBlockBytes = kTile * 128;   // 16 KiB: [128 tokens][128 B], 128B swizzle
constexpr int kPairBytes = 2 * kBlockBytes;
constexpr int kScaleStages = 4;            // per-token scales; a stage is free when the pair slots of its tile come round (see tma_role)
constexpr int kMaxSeg = 16;                // segments staged per round
constexpr float kPShift = 4.0f;            // P' = 2^(y - M + 4): keeps the E4M3 lo term out of the subnormals
constexpr float kLazyThreshold = 4.75f;    // the references move only when one is beaten by 2^4.75: P' <= 2^8.75 = 430.5, just inside E4M3 (448)
constexpr float kNoteMargin = 2.0f;        // a warp whose best token beats its reference by 2^2 has its say in how they move (note_tops)

// shared memory map (bytes from a 1024-aligned base)
constexpr uint32_t kOffKV = 0;                                            // [5][2][16384]
constexpr uint32_t kOffRope = kOffKV + kRing * kPairBytes;                // [128][64]  64B swizzle
constexpr uint32_t kOffQLat = kOffRope + kTile * 64;                      // [4][64][128]  128B swizzle
constexpr uint32_t kOffQRope = kOffQLat + kBlocks * kGroupHeads * 128;    // [64][64]      64B swizzle
constexpr uint32_t kOffP = kOffQRope + kGroupHeads * 64;                  // [hi,lo][128][64] 64B swizzle (MN-major)
constexpr uint32_t kOffScale = kOffP + 2 * kTile * 64;                    // [4][128] f32
constexpr uint32_t kOffM = kOffScale + kScaleStages * kTile * 4;          // [2][64] f32 NEGATED references -(M - shift): the ones in force, and room for the next
constexpr uint32_t kOffF = kOffM + 2 * kGroupHeads * 4;                   // [64] f32 rescale factor of a moved reference, [64] f32 by how much it moved
constexpr uint32_t kOffNotes = kOffF + 2 * kGroupHeads * 4;               // [tile mod 3][64] s32 notes of beaten references; epilogue: [4][64] f32 row sums
constexpr uint32_t kOffLinv = kOffNotes + 4 * kGroupHeads * 4;             // [64] f32 output factor; tail: 1/sum of the merge weights
constexpr uint32_t kOffLse = kOffLinv + kGroupHeads * 4;                  // [64] f32
constexpr uint32_t kOffScMax = kOffLse + kGroupHeads * 4;                 // [8] f32 per-warp largest token scale
constexpr uint32_t kOffBars = kOffScMax + kSoftmaxWarps * 4;              // mbarriers (8 B each)
// barrier indices
__device__ __forceinline__ constexpr int bar_kv_full(int slot) { return slot; }            // a pair (and, pair 0, the tile's scales) has landed
__device__ __forceinline__ constexpr int bar_kv_empty(int slot) { return kRing + slot; }   // PV has finished with it
__device__ __forceinline__ constexpr int bar_s_full(int s) { return 2 * kRing + s; }       // QK^T of a tile is in TMEM
__device__ __forceinline__ constexpr int bar_s_empty(int s) { return 2 * kRing + 2 + s; }  // ... and has been read
constexpr int kBarRopeFull = 2 * kRing + 4, kBarRopeEmpty = 2 * kRing + 5, kBarPFull = 2 * kRing + 6, kBarPvDone = 2 * kRing + 7,
              kBarQFull = 2 * kRing + 8, kBarQEmpty = 2 * kRing + 9, kBarOFree = 2 * kRing + 10, kBarDrain = 2 * kRing + 11,
              kBarTail = 2 * kRing + 12, kBarQkIssued = 2 * kRing + 13, kBarPvIssued = 2 * kRing + 14,
              kBarScale = 2 * kRing + 15;  // pair kernel: scales of a tile, four stages
constexpr int kNumBars = kBarScale + kScaleStages;
static_assert(kNumBars <= 32, "initialised by one warp, a barrier per lane");
constexpr uint32_t kOffTail = (kOffBars + kNumBars * 8 + 15u) & ~15u;     // merge plan: [148] slot ids
constexpr uint32_t kOffSegs = kOffTail + kMaxCombineSlots * 4;            // Segment[kMaxSeg]
constexpr uint32_t kOffMisc = kOffSegs + kMaxSeg * 24;
constexpr uint32_t kSmemBytes = kOffMisc + 256;
constexpr uint32_t kSmemAlloc = kSmemBytes + 1024;                        // slack for manual 1024-alignment
static_assert(sizeof(Segment) == 24, "segment staging layout");
static_assert(kSmemAlloc <= 232448, "shared memory budget exceeded");
static_assert(kOffBars % 8 == 0 && kOffSegs % 8 == 0 && kOffMisc % 8 == 0 && kOffLinv % 16 == 0, "alignment");

// TMEM columns
constexpr uint32_t kColSLat = 0;     // + 64 * stage
constexpr uint32_t kColSRope = 128;  // + 64 * stage
constexpr uint32_t kColO = 256;      // + 64 * block

constexpr uint32_t kFmtE2M1 = 5u << 7;  // A operand format field of kind::f8f6f4 (E4M3 = 0)
constexpr uint32_t kIdescQKRope = ptx::idesc_e4m3(128, kGroupHeads, false, false);       // E4M3 x E4M3
constexpr uint32_t kIdescQK = ptx::idesc_e4m3(128, kGroupHeads, false, false) | kFmtE2M1;  // E2M1 (K tile) x E4M3 (Q)
constexpr uint32_t kIdescPV = ptx::idesc_e4m3(128, kGroupHeads, true, true) | kFmtE2M1;    // E2M1 (V^T, MN-major) x E4M3 (P)

// A split request this CTA wrote a partial for: [0] the CTA's first segment (even slot), [1] its last (odd slot).
struct MergeReq {
  int b, g;
  flat_t start;   // flat index of the request's first (phantom) tile
  int vtiles;     // its tiles, phantom ones included; 0: no such partial
};
struct Misc {
  int n;              // CTAs that share the work: the first n of the grid
  uint32_t tmem_base;
  volatile int abort;
  uint32_t polls;     // poll budget of a bounded wait
  int32_t* status;
  int nseg, more;     // segments staged for the current round; another round follows
  flat_t next;        // flat position at which the next round starts
  flat_t Tt;          // size of the flat tile space (-1: it does not fit 32 bits)
  MergeReq merge[2];
  // the merge this CTA takes part in (plan_merge)
  MergeReq m;
  int n_slots, n_part, rank;
  int unit0, unit1;   // this CTA's share of every slot: units [unit0, unit1) of 16 bytes
  int mode;           // how the split requests of this step are merged: kMergeShared or kMergeLast
  int32_t gen;        // generation of this decode step, fetched once per CTA
  int last;           // kMergeLast: this CTA is the last writer of the request
  int cta;            // pair kernel: this CTA's place in the partition (cta_in_partition)
};
static_assert(sizeof(Misc) <= 256, "misc area");

__device__ __forceinline__ uint8_t* smem_ptr(uint32_t smem) { return static_cast<uint8_t*>(__cvta_shared_to_generic(smem)); }
__device__ __forceinline__ Misc* misc_of(uint32_t smem) { return reinterpret_cast<Misc*>(smem_ptr(smem) + kOffMisc); }
__device__ __forceinline__ const Segment* segs_of(uint32_t smem) { return reinterpret_cast<const Segment*>(smem_ptr(smem) + kOffSegs); }
__device__ __forceinline__ uint32_t bar_addr(uint32_t smem, int idx) { return smem + kOffBars + 8u * idx; }

// A bounded wait expired: flag the CTA (every role then stops issuing and drains) and leave a record.
__device__ __noinline__ void flag_timeout(uint32_t smem, int idx, uint32_t parity) {
  Misc* m = misc_of(smem);
  m->abort = 1;
  int32_t* status = m->status;
  if (status && atomicCAS(status, 0, MLA_FP4_ERR_DEVICE_TIMEOUT) == 0) {
    status[1] = idx;
    status[2] = blockIdx.x;
    status[3] = threadIdx.x;
    status[4] = int(parity);
  }
}
// Bounded wait of a whole (converged) warp.  Returns false (and flags the CTA) when it expires or the CTA is aborting.
__device__ __noinline__ bool wait_slow(uint32_t smem, int idx, uint32_t parity) {
  Misc* m = misc_of(smem);
  const uint32_t bar = bar_addr(smem, idx), polls = m->polls;
#pragma unroll 1
  for (uint32_t i = 0; i < polls; ++i) {
    if (__all_sync(0xffffffffu, ptx::mbar_try_wait(bar, parity))) return true;  // suspends in hardware for a while: not a hot spin
    if (__any_sync(0xffffffffu, m->abort)) return false;
    if (i > 4096) __nanosleep(128);
  }
  if ((threadIdx.x & 31) == 0) flag_timeout(smem, idx, parity);
  __syncwarp();
  return false;
}
__device__ __forceinline__ bool wait(uint32_t smem, int idx, uint32_t parity) {
  if (__all_sync(0xffffffffu, ptx::mbar_try_wait(bar_addr(smem, idx), parity))) return true;
  return __all_sync(0xffffffffu, wait_slow(smem, idx, parity));  // (already the same in all lanes; the vote says so to the compiler)
}
// Bounded wait that ignores the abort flag: lets in-flight asynchronous work land before exit.  Its bound has a floor (some milliseconds): however
// small a budget the caller gave the other waits, a copy must not land in the shared memory of a CTA that has left.
template <bool kCluster = false>
__device__ __noinline__ void drain_wait(uint32_t smem, int idx, uint32_t parity) {
  const uint32_t bar = bar_addr(smem, idx), polls = misc_of(smem)->polls;
  const uint32_t limit = min(max(polls, 1u << 10), 1u << 20);
#pragma unroll 1
  for (uint32_t i = 0; i < limit; ++i) {
    if (kCluster ? ptx::mbar_try_wait_cluster(bar, parity) : ptx::mbar_try_wait(bar, parity)) return;
    __nanosleep(64);
  }
}

__device__ __forceinline__ int ld_acquire(const int32_t* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ int ld_relaxed(const int32_t* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int32_t* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// The kernel's forms: one head group per CTA, over any CTAs or over as many for each group (shared_grid); two groups on a pair of CTAs.  The
// first carries none of the second's arithmetic, which stands in the prologue of every CTA (4x4096 tokens, 64 heads 13.45 -> 13.50 us).
enum Form { kFormAlone, kFormShared, kFormPair };

// running position of a role across rounds
struct RoleState {
  uint32_t it;         // tiles processed so far by this CTA (selects stages and barrier phases)
  uint32_t seg;        // segments processed so far
  uint32_t m, mod3;    // softmax: which references are in force; it mod 3
  uint32_t slot, lap;  // pair slot of the role's next latent pair, and how many times the ring has been filled before it
  __device__ __forceinline__ void advance(uint32_t n) {
    slot += n;
    if (slot >= uint32_t(kRing)) { slot -= kRing; ++lap; }
  }
};

// ------------------------------------------------------------------------------------------
// partition: the segments of this CTA (one warp; common.cuh has the same walk as a sequential loop)
// ------------------------------------------------------------------------------------------
// Lane i looks at request base + i: a scan gives its place in the flat tile space, the overlap with the CTA's range its
// segment, a ballot the segment's number.  The lengths are kept in shared memory (the latent ring is idle now) for the second
// pass and for start_work, which keeps its own reading in the other half; whole chunks of 32 requests outside the range are skipped with one reduction.  A sequential
// walk by one thread took 2500 clk of every CTA's prologue.
constexpr int kLensMax = int(kRing * kPairBytes / 8);
__device__ __forceinline__ int fresh_len(const DecodeParams& p, int i) {  // from L2: an earlier, speculative read must leave nothing in L1
  const int n = __ldcg(p.seq_lens + i);
  return n < p.seq_cap ? n : p.seq_cap;
}
// How many CTAs share the work when the decode kernel merges by itself.  A CTA more shortens everybody's walk, but every partial of a
// request is one more for all its writers to weigh and sum: with Tt tiles over n CTAs, 1.25 us * Tt / n + 0.05 us * n / pairs,
// which is least at n = 5 sqrt(Tt * pairs).  Then the longest walk k is kept and n lowered as far as k allows: CTAs
// that cannot shorten the longest walk only add partials, and a CTA without work does not hold the step up when it starts late.
// On 148 SMs, 64 heads, the whole grid -> as many as this: 1x16000 tokens 21.3 -> 17.5 us, 1x32768 22.9 -> 19.5, 4x4096 15.1 -> 14.1,
// 2x1024 14.0 -> 12.0; with several requests or head groups the whole grid works beyond five tiles a CTA (8x32768, 128 requests).  4 / 5 / 6 sqrt(Tt * pairs), with today's
// merge: 1x32768 18.45 / 17.2 / 18.2, 1x8192 14.15 / 13.3 / 13.3, 2x32768 19.6 / 18.6 / 18.6, 4x4096 13.2 / 13.2 / 13.55, 2x16000 17.5 /
// 17.4 / 15.8.  Approximate arithmetic will do: every CTA takes the same steps, and any 1 <= n <= Tt is right.  (The host's form of this
// rule, mla_fp4_work_ctas, is exact; the two agree while no walk is longer than a thousand tiles: where the root decides, Tt * pairs is
// below n^2 / 25, so that its argument keeps clear of the squares by more than the 1e-3 allows for.)
// Where the groups share the CTAs evenly (shared_grid) the number is a multiple of them: that many times what one group's tiles, T, need for the same walk.
template <Form F>
__device__ __forceinline__ int work_ctas(flat_t Tt, flat_t T, int groups, int pairs, int n) {
  if (Tt > 5 * n && pairs > 1) return n;  // the whole grid, and next to nothing to gain from the rounding
  const float tiles = float(Tt);
  float best, r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(best) : "f"(25.f * tiles * float(pairs)));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fminf(float(n), best)));
  const float k = float(__float2int_ru(tiles * r - 1e-3f));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(k));
  if (F != kFormAlone) return min(n, groups * max(1, __float2int_ru(float(T) * r - 1e-3f)));
  return min(n, max(1, __float2int_ru(tiles * r - 1e-3f)));
}
// This CTA's place in the partition.  In the pair kernel the two CTAs of a cluster walk the same tiles for two neighbouring head groups.
// There the working CTAs are a multiple of the groups, so that every group is shared by as many, `per`, in ranges of its own tiles that are
// the same for all groups: cluster w takes range w mod per of the groups 2 (w / per) and 2 (w / per) + 1.  (Short requests: `per` is the
// batch.)  The partition is thus the one of the other kernel, on other CTAs.
__device__ __forceinline__ int cta_in_partition(int per, int groups) {
  const int w = int(blockIdx.x >> 1), gp = int(uint32_t(w) / uint32_t(per));
  return 2 * gp < groups ? (2 * gp + int(blockIdx.x & 1)) * per + (w - gp * per) : per * groups;  // (beyond the last: no work)
}
template <bool kPair>
__device__ __forceinline__ int cta_of(const Misc* misc) { return kPair ? misc->cta : int(blockIdx.x); }
template <Form F>
__device__ __noinline__ void stage_segments(const DecodeParams& p, uint32_t smem, int lane, bool first_round, bool report) {
  Misc* misc = misc_of(smem);
  Segment* out = reinterpret_cast<Segment*>(smem_ptr(smem) + kOffSegs);
  int* lens = reinterpret_cast<int*>(smem_ptr(smem) + kOffKV);
  int cta = blockIdx.x;
  int n = gridDim.x;
  auto len_of = [&](int i) { return i < kLensMax ? lens[i] : fresh_len(p, i); };
  unsigned long long acc = 0;
  uint32_t mx = 0;
#pragma unroll 4
  for (int i = lane; i < p.batch; i += 32) {
    const int len = fresh_len(p, i);
    if (i < kLensMax) lens[i] = len;
    const uint32_t v = uint32_t(vtiles_of(len));
    acc += v;
    mx = max(mx, v);
  }
  const unsigned long long T64 = (static_cast<unsigned long long>(__reduce_add_sync(0xffffffffu, uint32_t(acc >> 24))) << 24) +
                                 __reduce_add_sync(0xffffffffu, uint32_t(acc) & 0xffffffu);
  mx = __reduce_max_sync(0xffffffffu, mx);
  int nseg = 0, more = 0;
  flat_t next = 0, Tt = 0;
  if (lane < 2 && first_round) misc->merge[lane].vtiles = 0;
  __syncwarp();
  if (!partition_fits(int64_t(T64) * p.groups, n)) {  // never with real caches: nothing is decoded, the status says why
    Tt = -1;
    if (lane == 0 && p.status && report) atomicCAS(p.status, 0, MLA_FP4_ERR_UNSUPPORTED);
  } else if (whole_requests(mx > 0 ? int(mx) - kPhantom : 0, int64_t(p.batch) * p.groups, n)) {  // CTA v: pair v, whole
    Tt = flat_t(T64) * p.groups;
    if (F == kFormPair) cta = cta_in_partition(p.batch, p.groups);
    if (cta < p.batch * p.groups) {
      const int g = cta / p.batch, b = cta - g * p.batch;
      const int len = len_of(b);
      if (len > 0) {
        if (lane == 0) out[0] = Segment{b, g, 0, tiles_of(len), len, -1};
        nseg = 1;
      }
    }
  } else if (T64 > 0) {
    const flat_t T = flat_t(T64);
    Tt = T * p.groups;
    if (p.fused_merge) n = work_ctas<F>(Tt, T, p.groups, p.batch * p.groups, n);
    if (F == kFormPair) cta = cta_in_partition(n / p.groups, p.groups);
    const flat_t cut = cta_lo(Tt, n, cta + (lane & 1));  // one division for both ends
    const flat_t lo = first_round ? __shfl_sync(0xffffffffu, cut, 0) : misc->next, hi = __shfl_sync(0xffffffffu, cut, 1);
    int g = lo < T ? 0 : int(uint32_t(lo) / uint32_t(T));
#pragma unroll 1
    for (flat_t run = flat_t(g) * T; cta < n && run < hi && !more; ++g) {
#pragma unroll 1
      for (int base = 0; base < p.batch && run < hi && !more; base += 32) {
        const int b = base + lane;
        const int len = b < p.batch ? len_of(b) : 0;
        const flat_t v = vtiles_of(len);
        const flat_t tot = __reduce_add_sync(0xffffffffu, v);
        if (run + tot > lo) {
          flat_t fs = v;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const flat_t u = __shfl_up_sync(0xffffffffu, fs, o);
            if (lane >= o) fs += u;
          }
          fs += run - v;  // the request's first (phantom) tile
          const flat_t from = max(lo, fs), to = min(hi, fs + v);
          const int rb = max(from, fs + kPhantom) - fs - kPhantom, re = to - fs - kPhantom;
          const bool live = v > 0 && from < to && re > rb;
          const uint32_t m = __ballot_sync(0xffffffffu, live);
          const int k = nseg + __popc(m & ((1u << lane) - 1u));
          if (live && k < kMaxSeg) {
            const bool whole = rb == 0 && re == v - kPhantom;
            const bool head = first_round && k == 0;
            out[k] = Segment{b, g, rb, re, len, whole ? -1 : slot_of(cta, head)};
            if (!whole) misc->merge[head ? 0 : 1] = MergeReq{b, g, fs, v};
          }
          nseg += __popc(m);
          if (nseg > kMaxSeg) {  // the rest in another round
            const uint32_t over = __ballot_sync(0xffffffffu, live && k == kMaxSeg);
            next = __shfl_sync(0xffffffffu, from, __ffs(over) - 1);
            nseg = kMaxSeg;
            more = 1;
          }
        }
        run += tot;
      }
    }
  }
  if (lane == 0) {
    misc->nseg = nseg;
    misc->more = more;
    misc->next = next;
    misc->Tt = Tt;
    misc->n = n;
    if (F == kFormPair) misc->cta = cta;
  }
  __syncwarp();
}

// The end of the prologue: from here on the kernel reads what earlier kernels wrote (sequence lengths, q, the cache, the
// workspace), and the plan is known.
// The plan made before the wait stands if the lengths have not changed.  A CTA that starts late, on an SM that the kernel ahead
// held to its end, finds nothing to wait for: there the lengths are read again while the plan is being made (1.8 us of code that
// comes from L2 line by line).
template <Form F>
__device__ __forceinline__ void start_work(const DecodeParams& p, uint32_t smem, int warp, int lane) {
  Misc* misc = misc_of(smem);
  if (p.pdl_wait) asm volatile("griddepcontrol.wait;" ::: "memory");
  // Let a dependent kernel start its launch and prologue early; it still waits for the end of this whole grid.
  if (p.pdl) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (warp == kWarpTMA) {
    bool stands = false;
    if (p.pdl_wait) {
      int* lens = reinterpret_cast<int*>(smem_ptr(smem) + kOffKV);
      const int nb = p.batch <= kLensMax ? p.batch : 0;
#pragma unroll 4
      for (int i = lane; i < nb; i += 32) lens[kLensMax + i] = fresh_len(p, i);
      ptx::bar_sync(8, 64);
      bool same = true;
#pragma unroll 1
      for (int i = lane; i < nb; i += 32) same &= lens[kLensMax + i] == lens[i];
      stands = __all_sync(0xffffffffu, same) && p.batch <= kLensMax && misc->Tt >= 0;
    }
    if (!stands) stage_segments<F>(p, smem, lane, true, true);
    ptx::fence_proxy_async_smem();  // the lengths give way to the first copies
    __threadfence_block();
    asm volatile("bar.arrive 2, %0;" ::"n"(kThreads) : "memory");
  } else {
    ptx::bar_sync(2, kThreads);
  }
}

// ------------------------------------------------------------------------------------------
// role: TMA issue (warp 1: pair 0 and scales of every tile; warp 3: RoPE and pair 1)
// ------------------------------------------------------------------------------------------
// Page ids are fetched 32 at a time, lane i holding the id of page i of the window, the next window's load in flight; an
// id outside the pool is never turned into an address: the tile's barrier then never completes and the bounded wait reports it.
//
// Pair position 2t + w (tile t, pair w) lives in slot (2t + w) mod 5 and is filled once PV of the position five back has
// completed, which lies in tile t-3 or t-2.  So when pair 0 of tile t is issued the softmax of tile t-3 is over, and the scale
// stage t mod 4, last read by tile t-4, is free: it needs no barrier of its own and its bytes count on the pair's barrier.
// page id `at + lane` of a segment, -1 beyond its pages or outside the pool
__device__ __forceinline__ int page_window(const DecodeParams& p, const Segment& g, int at) {
  const int ppt = kTile >> p.page_shift;
  const int lp = g.tile_begin * ppt + at + int(threadIdx.x & 31);
  const int id = lp < min(((g.seq_len - 1) >> p.page_shift) + 1, g.tile_end * ppt) ? __ldcg(p.block_tables + size_t(g.b) * p.block_table_stride + lp) : -1;
  return int64_t(id) < p.num_pages ? id : -1;
}
// entry `i` of a window, in a uniform register
__device__ __forceinline__ int uniform_page(int window, int i) { return __reduce_max_sync(0xffffffffu, int(threadIdx.x & 31) == (i & 31) ? window : -1); }
template <Form F>
__device__ __forceinline__ void tma_role(const DecodeParams& p, uint32_t smem, uint32_t which, const CUtensorMap* map_rope,
                                         const CUtensorMap* map_lat, RoleState& st, bool starting) {
  const Segment* sg = segs_of(smem);
  const int lane = threadIdx.x & 31;
  const int ppt = kTile >> p.page_shift;  // pages per tile
  const uint32_t ps = uint32_t(p.page_size);
  bool ok = true;
  // A kernel's instructions come from L2 line by line when it starts: the first tile's copies were in flight 1.8 us after the plan
  // was known.  So while the plan is made, the code of a tile is gone through once with nothing to copy (`dry`: every copy
  // predicated off, no page, no wait, no position taken).  With the plan made by another warp meanwhile: 16 requests of 200..4000
  // tokens with 128 heads 17.0 -> 16.7 us, 61x300 11.7 -> 11.45, 8x32768 35.05 -> 34.65, 128 requests of 128..32768 88.6 -> 87.8.
  bool dry = starting && p.pdl_wait;
  st.slot = starting ? which : st.slot;
  uint32_t nseg = 0;
  if (!dry) {
    if (starting) start_work<F>(p, smem, which ? kWarpTMA2 : kWarpTMA, lane);
    nseg = ptx::uniform_u32(uint32_t(misc_of(smem)->nseg));
  }
#pragma unroll 1
  for (uint32_t si = 0; dry || (si < nseg && ok);) {
    Segment g{0, 0, 0, 1, 0, -1};
    if (!dry) g = sg[si];
    g.tile_begin = int(ptx::uniform_u32(uint32_t(g.tile_begin)));
    g.tile_end = int(ptx::uniform_u32(uint32_t(g.tile_end)));
    g.seq_len = int(ptx::uniform_u32(uint32_t(g.seq_len)));
    const int total = dry ? ppt : ((g.seq_len - 1) >> p.page_shift) + 1;
    int cur = page_window(p, g, 0), nxt = page_window(p, g, 32), ahead = 64, at = 0;
#pragma unroll 1
    for (int t = g.tile_begin; t < g.tile_end; ++t, ++st.it) {
      const int np = min(ppt, total - t * ppt);
      // the first four pages' ids are in hand before the waits: a slot that has come free is refilled with straight-line copies
      int pg[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) pg[i] = uniform_page(cur, at + i);
      const uint32_t e = ptx::elect_one() && !dry;
      auto for_pages = [&](auto copy) {  // copy(issue, page, index)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i < np) copy(e && pg[i] >= 0 ? 1u : 0u, pg[i], i);
#pragma unroll 1
        for (int i = 4; i < np; ++i) {
          const int page = uniform_page(cur, at + i);
          copy(e && page >= 0 ? 1u : 0u, page, i);
        }
      };
      if (which) {  // RoPE bytes: the one buffer is free once the two RoPE MMAs of the previous tile have completed
        if (st.it >= 1) ok = wait(smem, kBarRopeEmpty, (st.it - 1) & 1);
        if (!ok) break;
        const uint32_t bar = bar_addr(smem, kBarRopeFull);
        if (e) ptx::mbar_arrive_expect_tx(bar, uint32_t(np) * ps * 64u);
        for_pages([&](uint32_t issue, int page, int i) { ptx::tma_load_3d_if(issue, smem + kOffRope + uint32_t(i) * ps * 64u, map_rope, bar, kLatent / 2, 0, page); });
      }
      const uint32_t bar = bar_addr(smem, bar_kv_full(st.slot)), dst = smem + kOffKV + st.slot * kPairBytes;
      if (st.lap >= 1) ok = wait(smem, bar_kv_empty(st.slot), (st.lap - 1) & 1);
      if (!ok) break;
      // the transaction count of a 4-bit copy is in packed bytes: 64 per row and block
      if (e) ptx::mbar_arrive_expect_tx(bar, uint32_t(np) * ps * (which ? 128u : 132u));
      const int c0 = int(256u * which);
      for_pages([&](uint32_t issue, int page, int i) {
        ptx::tma_load_3d_if(issue, dst + uint32_t(i) * ps * 128u, map_lat, bar, c0, 0, page);
        ptx::tma_load_3d_if(issue, dst + uint32_t(i) * ps * 128u + kBlockBytes, map_lat, bar, c0 + 128, 0, page);
      });
      if (!which) {
        const uint32_t dst_sc = smem + kOffScale + (st.it & (kScaleStages - 1)) * (kTile * 4);
        for_pages([&](uint32_t issue, int page, int i) { ptx::bulk_load_if(issue, dst_sc + uint32_t(i) * ps * 4u, p.kv_cache_sf + int64_t(page) * ps, ps * 4u, bar); });
      }
      // The rows of the tile four ahead are brought into L2 (page ids in hand reach 32 to 64 pages: with pages of 8 tokens, sixteen to a
      // tile, that is not four tiles, and nothing is prefetched): the ring holds two and a half tiles, and a pair's slot comes free
      // two tiles before the pair is needed, so a load that comes from DRAM (2000 clk instead of 900) shows in every tile:
      // 2x131072 tokens, H=128, q_len=2: 97.5 -> 92.6 us; 8x32768: 37.6 -> 36.8.
      if (which) {
        const int i = at + 4 * ppt + lane;
        const int in_cur = __shfl_sync(0xffffffffu, cur, i & 31), in_nxt = __shfl_sync(0xffffffffu, nxt, i & 31);
        const int page = i < 32 ? in_cur : (i < 64 ? in_nxt : -1);
        if (lane < ppt && page >= 0)
          asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(static_cast<const uint8_t*>(p.kv_cache) + size_t(page) * ps * kRowBytes),
                       "r"(ps * kRowBytes) : "memory");
      }
      st.advance(2);
      at += ppt;
      if (at == 32) {
        at = 0;
        cur = nxt;
        nxt = page_window(p, g, ahead);
        ahead += 32;
      }
    }
    ++si;
    ++st.seg;
    if (dry) {
      dry = false;
      si = 0;
      st = RoleState{};
      st.slot = which;
      start_work<F>(p, smem, which ? kWarpTMA2 : kWarpTMA, lane);
      nseg = ptx::uniform_u32(uint32_t(misc_of(smem)->nseg));
    }
  }
  if (!ok && lane == 0) {  // let copies that were issued but never consumed land before exit (bounded; a refused page never does)
    const uint32_t armed = st.it;  // this warp's pair positions 2k + which, k < armed
    for (uint32_t k = armed > 5u ? armed - 5u : 0u; k < armed; ++k) {
      const uint32_t pos = 2u * k + which;
      drain_wait(smem, bar_kv_full(pos % kRing), (pos / kRing) & 1);
    }
    if (which && armed >= 1) drain_wait(smem, kBarRopeFull, (armed - 1) & 1);
    if (which) drain_wait(smem, kBarRopeFull, armed & 1);  // armed for a tile whose pair was not
  }
  __syncwarp();
}

// ------------------------------------------------------------------------------------------
// roles: MMA issue.  The whole warp runs this code with uniform control flow and uniform values (ptx::uniform_u32); only the
// tcgen05 instructions are predicated on the elected lane, so their operands stay in uniform registers.
// ------------------------------------------------------------------------------------------
// A shared-memory descriptor as two words.  Only the 14-bit address field (bytes >> 4) in the low word
// changes from one instruction to the next and it cannot carry out (shared memory is smaller than
// 2^18 bytes), so stepping a descriptor is ONE 32-bit add.
struct Desc {
  uint32_t lo, hi;
  __device__ __forceinline__ uint64_t at(uint32_t off16) const { return (uint64_t(hi) << 32) | uint64_t(lo + off16); }
};
__device__ __forceinline__ Desc make_desc(uint32_t addr, uint32_t lbo, uint32_t sbo, uint32_t layout) {
  const uint64_t d = ptx::smem_desc(addr, lbo, sbo, layout);
  return Desc{uint32_t(d), uint32_t(d >> 32)};
}

// role: QK^T issue and Q loads (warp 0).  RoPE first (its commit frees the one RoPE buffer for the next tile), then the two
// pairs.  There is one Q buffer, so Q of a segment is loaded by the warp that needs it, when the last QK^T of the segment
// before has completed.
__device__ __forceinline__ void qk_role(const DecodeParams& p, uint32_t smem, uint32_t tmem, const CUtensorMap* map_q_lat,
                                        const CUtensorMap* map_q_rope, RoleState& st) {
  const uint32_t nseg = ptx::uniform_u32(uint32_t(misc_of(smem)->nseg));
  const Segment* sg = segs_of(smem);
  const Desc rope = make_desc(smem + kOffRope, 16, 512, 4), q_rope = make_desc(smem + kOffQRope, 16, 512, 4);
  const Desc kv = make_desc(smem + kOffKV, 16, 1024, 2), q_lat = make_desc(smem + kOffQLat, 16, 1024, 2);  // K-major, 128B swizzle
  bool ok = true;
#pragma unroll 1
  for (uint32_t si = 0; si < nseg && ok; ++si, ++st.seg) {
    const Segment g = sg[si];
    if (st.seg >= 1 && !wait(smem, kBarQEmpty, (st.seg - 1) & 1)) break;
    int qpos, head0;
    group_coords(g.g, p.num_heads, qpos, head0);
    if (ptx::elect_one()) {
      const uint32_t bar = bar_addr(smem, kBarQFull);
      ptx::mbar_arrive_expect_tx(bar, kGroupHeads * kQDim);
      ptx::tma_load_4d(smem + kOffQRope, map_q_rope, bar, kLatent, head0, qpos, g.b);
#pragma unroll 1
      for (int j = 0; j < kBlocks; ++j)
        ptx::tma_load_4d(smem + kOffQLat + j * kGroupHeads * 128, map_q_lat, bar, 128 * j, head0, qpos, g.b);
    }
    __syncwarp();
    const uint32_t n = ptx::uniform_u32(uint32_t(g.tile_end - g.tile_begin));
    ok = wait(smem, kBarQFull, st.seg & 1);
#pragma unroll 1
    for (uint32_t t = 0; t < n && ok; ++t, ++st.it) {
      const uint32_t it = st.it, s64 = 64u * (it & 1);
      // S of this stage has been read by the softmax of tile it-2; PV of tile it-2, if of this segment, is half issued; the RoPE
      // bytes of this tile have landed.  (The two issue barriers cannot run ahead of the warp that waits for them: inside a
      // segment PV(it-1) waits for this tile's QK^T, and QK^T of it+1 for PV(it-1).  tests/test_issue_order.py tries every interleaving.)
      if (it >= 2) ok = wait(smem, bar_s_empty(it & 1), ((it >> 1) - 1) & 1);
      if (t >= 2) ok = ok && wait(smem, kBarPvIssued, it & 1);
      ok = ok && wait(smem, kBarRopeFull, it & 1);
      if (!ok) break;
      ptx::tc_fence_after();
      const uint32_t e = ptx::elect_one();
#pragma unroll
      for (uint32_t ks = 0; ks < 2; ++ks) ptx::umma_f8(e, tmem + kColSRope + s64, rope.at(2 * ks), q_rope.at(2 * ks), kIdescQKRope, ks);
      if (e) ptx::umma_commit(bar_addr(smem, kBarRopeEmpty));
      __syncwarp();
#pragma unroll 1
      for (uint32_t pr = 0; pr < 2 && ok; ++pr) {
        ok = wait(smem, bar_kv_full(st.slot), st.lap & 1);
        if (!ok) break;
        ptx::tc_fence_after();
        const uint32_t a = st.slot * (kPairBytes >> 4), b = pr * ((2 * kGroupHeads * 128) >> 4);
#pragma unroll
        for (uint32_t j = 0; j < 2; ++j)
#pragma unroll
          for (uint32_t ks = 0; ks < 4; ++ks)
            ptx::umma_f8(e, tmem + kColSLat + s64, kv.at(a + j * (kBlockBytes >> 4) + 2 * ks), q_lat.at(b + j * ((kGroupHeads * 128) >> 4) + 2 * ks),
                         kIdescQK, (pr | j | ks) ? 1u : 0u);
        if (pr && e) {
          ptx::mbar_arrive(bar_addr(smem, kBarQkIssued));  // (first: who has seen what follows from S finds it done)
          ptx::umma_commit(bar_addr(smem, bar_s_full(it & 1)));
        }
        __syncwarp();
        st.advance(1);
      }
    }
    // every QK^T of this segment has been issued: Q may be overwritten once they complete
    if (ptx::elect_one()) ptx::umma_commit(bar_addr(smem, kBarQEmpty));
    __syncwarp();
  }
  if (misc_of(smem)->abort && (threadIdx.x & 31) == 0) {  // a Q load in flight lands (one of the two waits runs to its bound)
    drain_wait(smem, kBarQFull, 0);
    drain_wait(smem, kBarQFull, 1);
  }
  __syncwarp();
}

// role: PV issue (warp 2).  Per block of 128 dims 4 token steps x (hi, lo), which share A through the collector; the commit
// after a pair frees its slot.
__device__ __forceinline__ void pv_role(uint32_t smem, uint32_t tmem, RoleState& st) {
  const uint32_t nseg = ptx::uniform_u32(uint32_t(misc_of(smem)->nseg));
  const Segment* sg = segs_of(smem);
  const Desc kv = make_desc(smem + kOffKV, kBlockBytes, 1024, 2);  // V^T: MN-major, 128B swizzle; 32 tokens per step = 4 groups of 8 rows (4096 B)
  const Desc pd = make_desc(smem + kOffP, 512, 512, 4);            // P^T: MN-major (64 heads contiguous), 64B swizzle; 2048 B per step
#pragma unroll 1
  for (uint32_t si = 0; si < nseg; ++si, ++st.seg) {
    const uint32_t n = ptx::uniform_u32(uint32_t(sg[si].tile_end - sg[si].tile_begin));
    if (st.seg >= 1 && !wait(smem, kBarOFree, (st.seg - 1) & 1)) return;  // O^T of the previous segment has been read out
#pragma unroll 1
    for (uint32_t t = 0; t < n; ++t, ++st.it) {
      // P of this tile, and QK^T of the segment's next tile has been issued (so it lies ahead of this PV in the queue of the tensor
      // pipe).  In this order: P says that QK^T of this tile was reported as issued, so the phase before the one waited for is over and
      // its parity cannot be taken for an older phase's.  (The other way round, tile 0 found the barrier untouched and did not wait.)
      if (!wait(smem, kBarPFull, st.it & 1)) return;
      if (t + 1 < n && !wait(smem, kBarQkIssued, (st.it + 1) & 1)) return;
      ptx::tc_fence_after();
      const uint32_t e = ptx::elect_one(), keep = t ? 1u : 0u;
#pragma unroll 1
      for (uint32_t pr = 0; pr < 2; ++pr) {
        const uint32_t a = st.slot * (kPairBytes >> 4), d = tmem + kColO + 128u * pr;
#pragma unroll
        for (uint32_t j = 0; j < 2; ++j)
#pragma unroll
          for (uint32_t ks = 0; ks < 4; ++ks) {
            const uint64_t ad = kv.at(a + j * (kBlockBytes >> 4) + 256 * ks);
            ptx::umma_f8_a_fill(e, d + 64u * j, ad, pd.at(128 * ks), kIdescPV, ks ? 1u : keep);
            ptx::umma_f8_a_lastuse(e, d + 64u * j, ad, pd.at(((kTile * 64) >> 4) + 128 * ks), kIdescPV, 1u);
            if (j == 0 && ks == 0 && pr && e) ptx::mbar_arrive(bar_addr(smem, kBarPvIssued));
          }
        if (e) {
          ptx::umma_commit(bar_addr(smem, bar_kv_empty(st.slot)));
          if (pr) ptx::umma_commit(bar_addr(smem, kBarPvDone));
        }
        __syncwarp();
        st.advance(1);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------
// role: softmax / rescale / epilogue (warps 4..11, thread = TMEM lane)
// ------------------------------------------------------------------------------------------
// ---- packed FP32 pairs (sm_100 f32x2 arithmetic)
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ uint64_t pack2u(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ void lds_pairs(uint32_t addr, uint64_t& p0, uint64_t& p1) {
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(p0), "=l"(p1) : "r"(addr) : "memory");
}
__device__ __forceinline__ float lds_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint4 lds_u32x4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float4 lds_f32x4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void sts_f32(uint32_t addr, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

// two-term E4M3 split of a pair: hi = e4m3(v), lo = e4m3(v - hi); returns hi (16 bits), lo via reference.
// Five two-wide instructions; the softmax pass is bound by instruction issue (two warps per scheduler), and a
// split on the FMA pipe (Veltkamp) measured slower because it needs one more.
__device__ __forceinline__ uint32_t split_e4m3x2(uint64_t v2, uint32_t& lo) {
  float a, b;
  unpack2(v2, a, b);
  __half2 h = __floats2half2_rn(a, b);
  const __nv_fp8x2_storage_t hi = __nv_cvt_halfraw2_to_fp8x2(*reinterpret_cast<__half2_raw*>(&h), __NV_SATFINITE, __NV_E4M3);
  __half2_raw back = __nv_cvt_fp8x2_to_halfraw2(hi, __NV_E4M3);
  __half2 r = __hsub2(h, *reinterpret_cast<__half2*>(&back));
  lo = __nv_cvt_halfraw2_to_fp8x2(*reinterpret_cast<__half2_raw*>(&r), __NV_SATFINITE, __NV_E4M3);
  return hi;
}

// Sum over the 32 lanes of 32 per-lane values held as 16 pairs; lane L ends with the total of value L.
constexpr int kHalfHeads = kGroupHeads / 2;  // heads per softmax warp
constexpr int kPairs = kHalfHeads / 2;
__device__ __forceinline__ float warp_transpose_sum32(uint64_t (&l2)[kPairs], int lane) {
  float v[kHalfHeads];
#pragma unroll
  for (int i = 0; i < kPairs; ++i) unpack2(l2[i], v[2 * i], v[2 * i + 1]);
#pragma unroll
  for (int o = 16, n = kHalfHeads; o > 0; o >>= 1, n >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      const float keep = up ? v[i + n / 2] : v[i];
      const float send = up ? v[i] : v[i + n / 2];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return v[0];
}

struct SoftmaxTile {
  uint32_t t_lat, t_rope;  // TMEM addresses of this thread's lane, S columns of the stage
  uint32_t negm;           // shared address of the negated references (-m) of this warp's 32 heads
  uint64_t sc2, cs2;       // (scale_t, scale_t), (c, c)
  uint64_t cap2, rcap2;    // soft-cap variant: (cap, cap), (1/cap, 1/cap)
  bool valid;
};
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float tanh_approx(float x) {
  float r;
  asm("tanh.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// First half of a tile's softmax, over the 32 heads this thread owns of its token: the exponents y = x*c - m with the reference
// as it stands; returns the largest for the lazy-reference check.  Nothing has been exponentiated yet, so a reference that turns
// out to be beaten, by however much, costs a subtraction.  The S columns of the second 16 heads are on their way while the
// first are worked on.
// kSoftCap: the raw score x = q.k passes through cap * tanh(x / cap) first (compiled only into the soft-cap kernel).
template <bool kSoftCap>
__device__ __forceinline__ float exponents(const SoftmaxTile& t, uint64_t (&y2)[kPairs]) {
  float mx = -INFINITY;
  uint32_t a[2][16], b[2][16];
  ptx::tmem_ld16(t.t_lat, a[0]);
  ptx::tmem_ld16(t.t_rope, b[0]);
  ptx::tmem_wait_ld();
#pragma unroll
  for (int cidx = 0; cidx < 2; ++cidx) {
    if (cidx == 0) {
      ptx::tmem_ld16(t.t_lat + 16, a[1]);
      ptx::tmem_ld16(t.t_rope + 16, b[1]);
    } else {
      ptx::tmem_wait_ld();
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {  // 4 heads per shared load of the references
      uint64_t nm[2];
      lds_pairs(t.negm + 64 * cidx + 16 * q, nm[0], nm[1]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = 4 * q + 2 * h;
        uint64_t x2 = fma2(pack2u(a[cidx][i], a[cidx][i + 1]), t.sc2, pack2u(b[cidx][i], b[cidx][i + 1]));
        if (kSoftCap) {
          float x0, x1;
          unpack2(mul2(x2, t.rcap2), x0, x1);
          x2 = mul2(pack2(tanh_approx(x0), tanh_approx(x1)), t.cap2);
        }
        const uint64_t y = fma2(x2, t.cs2, nm[h]);
        y2[8 * cidx + 2 * q + h] = y;
        float y0, y1;
        unpack2(y, y0, y1);
        mx = max3(mx, y0, y1);
      }
    }
  }
  if (!t.valid) {  // token beyond seq_len: weight exactly zero, whatever its row holds (its RoPE bytes may decode to NaN)
#pragma unroll
    for (int q = 0; q < kPairs; ++q) y2[q] = pack2(-INFINITY, -INFINITY);
    mx = -INFINITY;
  }
  return mx;
}

// How the references move.  A head's best token should have a P' of exactly 2^kPShift, which has no rounding error: that counts
// where few tokens carry the weight.  So when a token beats a reference by more than the lazy threshold, not its head alone is
// moved, but every head to the top of the tokens that the warps have noted: each warp with a token that beats some reference by
// 2^kNoteMargin, or by the threshold, notes the largest y + log2|scale_t| of each of its heads (as integers that compare like the
// floats) before the vote of the softmax warps.  After it every warp works out the new references and factors of its 32 heads from the
// notes (the four warps of a half write the same values): no barrier but the vote.  The first tile of a segment is the same with
// references of zero and every warp noting.  Notes go round three places: those of tile t-1 are cleared after the vote of tile t,
// when nobody reads them any more, and used again by tile t+2, which no warp reaches before all have voted in tile t+1.
// Error against 64 bits (FP32 output) and time with the beaten heads alone moved -> this: 2x256 tokens, 16 heads, logits eight times as
// large 2.97e-4 -> 1.81e-4, 8.43 -> 8.46 us; 128 requests of 128..32768 tokens with outliers 2.14e-4 -> 1.92e-4, 93.9 -> 95.2 us.  All heads
// by the tokens of all warps that are above a reference: as exact, with those notes before the vote (a margin of 0) 95.9 us
// and 2x131072 tokens, 128 heads, q_len 2 89.8 -> 93 us; behind the vote and another barrier 104.4 us.
// (With heavy-tailed token scales a reference is beaten in every other tile, mostly by more than FP32 exponentials could hold:
// recomputing such tiles from the scores took 1100 clk each.)
constexpr int kNoScore = int(0x80000000u);
__device__ __forceinline__ void note_tops(uint32_t notes, const uint64_t (&y2)[kPairs], float lg, int lane) {
  float mine = -INFINITY;  // lane i: head i of the warp's 32
#pragma unroll
  for (int i = 0; i < kPairs; ++i) {
    float y0, y1;
    unpack2(y2[i], y0, y1);
    const float r0 = ptx::redux_max_f32(y0 + lg), r1 = ptx::redux_max_f32(y1 + lg);
    if (lane == 2 * i) mine = r0;
    if (lane == 2 * i + 1) mine = r1;
  }
  const int b = __float_as_int(mine);
  asm volatile("red.shared.max.s32 [%0], %1;" ::"r"(notes + 4 * lane), "r"(b ^ ((b >> 31) & 0x7fffffff)) : "memory");
}
// m += d and f = 2^-d with d = top - shift, where that is positive; d = 0 and f = 1 for all other heads.  In the first tile of a
// segment d = top - shift whatever its sign, and f is 0: there are no sums yet, and a first top far below zero would make f
// infinite and the empty sums NaN.
__device__ __forceinline__ void refresh_references(uint32_t smem, uint32_t notes, uint32_t cur, bool first, int half, int lane) {
  const uint32_t at = 4u * (32u * uint32_t(half) + uint32_t(lane));
  const int b = int(lds_u32(notes + 4 * lane));
  const float above = __int_as_float(b ^ ((b >> 31) & 0x7fffffff)) - kPShift;
  const float d = first ? above : fmaxf(above, 0.f);
  sts_f32(smem + kOffM + 256 * (cur ^ 1u) + at, lds_f32(smem + kOffM + 256 * cur + at) - d);
  sts_f32(smem + kOffF + at, first ? 0.f : ptx::ex2(-d));
  sts_f32(smem + kOffF + 256 + at, d);
  __syncwarp();
}

// O^T *= f per head column, in TMEM (all four 128-dim blocks of this thread's lane).  With few heads moved, as a new maximum
// usually has it, column by column.
__device__ __noinline__ void rescale_output(uint32_t smem, uint32_t tmem_lane, uint32_t half, int lane) {
  const uint32_t base = tmem_lane + kColO + 32u * half;
  const float mine = lds_f32(smem + kOffF + 4 * (32u * half + uint32_t(lane)));
  uint32_t moved = __ballot_sync(0xffffffffu, mine != 1.f);
  if (__popc(moved) <= 8) {
#pragma unroll 1
    while (moved) {  // two heads at a time (or one, twice)
      const uint32_t h0 = uint32_t(__ffs(moved)) - 1u;
      moved &= moved - 1u;
      const uint32_t h1 = moved ? uint32_t(__ffs(moved)) - 1u : h0;
      moved &= moved - 1u;
      const float f0 = __shfl_sync(0xffffffffu, mine, int(h0)), f1 = __shfl_sync(0xffffffffu, mine, int(h1));
      uint32_t o[kBlocks], u[kBlocks];
#pragma unroll
      for (int j = 0; j < kBlocks; ++j) ptx::tmem_ld1(base + 64u * j + h0, o[j]);
#pragma unroll
      for (int j = 0; j < kBlocks; ++j) ptx::tmem_ld1(base + 64u * j + h1, u[j]);
      ptx::tmem_wait_ld();
#pragma unroll
      for (int j = 0; j < kBlocks; ++j) ptx::tmem_st1(base + 64u * j + h0, __float_as_uint(__uint_as_float(o[j]) * f0));
#pragma unroll
      for (int j = 0; j < kBlocks; ++j) ptx::tmem_st1(base + 64u * j + h1, __float_as_uint(__uint_as_float(u[j]) * f1));
    }
  } else {
#pragma unroll 1
    for (uint32_t jc = 0; jc < kBlocks; ++jc) {  // 16 heads of two blocks at a time
      uint32_t o[2][16];
      const uint32_t c = 16u * (jc & 1), ta = base + 128u * (jc >> 1) + c;
      ptx::tmem_ld16(ta, o[0]);
      ptx::tmem_ld16(ta + 64u, o[1]);
      const uint32_t f = smem + kOffF + 4 * (32u * half + c);
      ptx::tmem_wait_ld();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 v = lds_f32x4(f + 16 * q);
        const float vs[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          o[0][4 * q + e] = __float_as_uint(__uint_as_float(o[0][4 * q + e]) * vs[e]);
          o[1][4 * q + e] = __float_as_uint(__uint_as_float(o[1][4 * q + e]) * vs[e]);
        }
      }
      ptx::tmem_st16(ta, o[0]);
      ptx::tmem_st16(ta + 64u, o[1]);
    }
  }
  ptx::tmem_wait_st();
}

// Normalise O^T and write it to the output tensor (a segment that covers its request).  Runs once per segment, so
// its instructions are fetched cold, and a workload of many short requests runs it between every few tiles: rolled
// loops over (block, 16 heads), a small body (unrolled four times it slowed the variable-length workload by 10 %).
// One instantiation per output type and for a full group of 64 heads (no per-head predicates: half the instructions):
// a call fetches the instructions of its own form only.
template <int kOutDtype, bool kAllHeads>
__device__ __noinline__ void write_final(const DecodeParams& p, uint32_t smem, uint32_t tmem_lane, int row, int half,
                                         int tid, int b, int g) {
  int qpos, head0;
  group_coords(g, p.num_heads, qpos, head0);
  const int heads_here = min(kGroupHeads, p.num_heads - head0);
  const size_t row0 = (size_t(b) * p.q_len + qpos) * p.num_heads + head0;
  constexpr uint32_t esz = kOutDtype == MLA_FP4_OUT_F32 ? 4u : (kOutDtype == MLA_FP4_OUT_BF16 ? 2u : 1u);
#pragma unroll 1
  for (int jb = 0; jb < kBlocks; ++jb) {  // a block of 128 dims: this thread's 32 heads as two TMEM loads in flight together
    uint32_t o[2][16];
    ptx::tmem_ld16(tmem_lane + kColO + 64u * uint32_t(jb) + uint32_t(32 * half), o[0]);
    ptx::tmem_ld16(tmem_lane + kColO + 64u * uint32_t(jb) + uint32_t(32 * half + 16), o[1]);
    const int dim = 128 * jb + row;
    ptx::tmem_wait_ld();
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int h0 = 32 * half + 16 * hh;
      char* dst = static_cast<char*>(p.out) + ((row0 + h0) * kLatent + dim) * esz;
#pragma unroll
      for (int q = 0; q < 4; ++q) {  // output_scale / l of four heads per shared load
        const float4 f = lds_f32x4(smem + kOffLinv + 4 * (h0 + 4 * q));
        const float fs[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = 4 * q + e;
          if (kAllHeads || h0 + i < heads_here) {
            const float v = __uint_as_float(o[hh][i]) * fs[e];
            char* d = dst + size_t(i) * kLatent * esz;
            if (kOutDtype == MLA_FP4_OUT_BF16) *reinterpret_cast<__nv_bfloat16*>(d) = __float2bfloat16_rn(v);
            else if (kOutDtype == MLA_FP4_OUT_F32) *reinterpret_cast<float*>(d) = v;
            else *reinterpret_cast<uint8_t*>(d) = __nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
          }
        }
      }
    }
  }
  if (p.lse && tid < heads_here) p.lse[row0 + tid] = lds_f32(smem + kOffLse + 4 * tid);
}

// The same for BF16, the common output: a block of 128 dims is transposed in the P buffer (idle between two segments) and
// written in rows.  O^T has dims on the lanes, so direct stores are two bytes wide: 128 of them per thread and their
// predicates took 3.7 us for 16 heads.  Here the accumulator is read in fragments, stmatrix transposes 8x8 of them at a time, and a
// thread stores 16 bytes, 16 threads a row.  Chunks of 16 bytes are swizzled by the head so that neither side has conflicts.
// With at most 32 heads the warps of the upper 32 have none: they take the next block of dims (two == 1), two blocks between barriers.
// 2x256 tokens, 16 heads: 8.55 -> 8.07 us.  (A template: one body for both cost the main loop two registers, 87.0 -> 88.3 us for 128
// requests of 128..32768 tokens.)
template <int two>
__device__ __noinline__ void write_final_bf16(const DecodeParams& p, uint32_t smem, uint32_t tmem_lane, int quarter, int half, int tid, int b, int g) {
  int qpos, head0;
  group_coords(g, p.num_heads, qpos, head0);
  const int heads_here = min(kGroupHeads, p.num_heads - head0), lane = tid & 31;
  const size_t row0 = (size_t(b) * p.q_len + qpos) * p.num_heads + head0;
  const uint32_t buf = smem + kOffP;
  // lane 8i + j addresses head 8k + j, dims [8i, 8i + 8) of the warp's 32
  const uint32_t st_row = buf + (32u * half + uint32_t(lane & 7)) * 256u + (((4u * quarter + uint32_t(lane >> 3)) ^ uint32_t(lane & 7)) << 4);
  const int heads_at = two ? 0 : 32 * half;
  const uint32_t fac = smem + kOffLinv + 4u * (uint32_t(heads_at) + 2u * uint32_t(lane & 3));
  const int c = tid & 15, h_ld = tid >> 4;  // reading: 16-byte chunk c of heads h_ld + 16 r
  const uint32_t ld_at = buf + uint32_t(h_ld) * 256u + ((uint32_t(c) ^ uint32_t(h_ld & 7)) << 4);
  __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(p.out) + (row0 + h_ld) * kLatent + 8 * c;
#pragma unroll 1
  for (int jb = 0; jb < kBlocks; jb += 1 + two) {
    uint32_t o[2][16];
    const uint32_t ta = tmem_lane + kColO + 64u * uint32_t(jb + two * half) + uint32_t(heads_at);
    if (heads_at < heads_here) {
      ptx::tmem_ld_16x256b_x4(ta, o[0]);
      ptx::tmem_ld_16x256b_x4(ta + (16u << 16), o[1]);
      ptx::tmem_wait_ld();
#pragma unroll
      for (int k = 0; k < 4; ++k) {  // eight heads
        float f0, f1;
        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(f0), "=f"(f1) : "r"(fac + 32u * k) : "memory");
        uint32_t m[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t* v = &o[i >> 1][4 * k + 2 * (i & 1)];
          const __nv_bfloat162 t = __floats2bfloat162_rn(__uint_as_float(v[0]) * f0, __uint_as_float(v[1]) * f1);
          m[i] = *reinterpret_cast<const uint32_t*>(&t);
        }
        ptx::stmatrix_x4_trans(st_row + uint32_t(k) * (8u * 256u), m[0], m[1], m[2], m[3]);
      }
    }
    ptx::bar_sync(1, kSoftmaxThreads);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int upper = two & (r >> 1), hr = 16 * (r - 2 * upper);
      if (h_ld + hr < heads_here) *reinterpret_cast<uint4*>(dst + size_t(hr) * kLatent + 128 * (jb + upper)) = lds_u32x4(ld_at + uint32_t(r) * (16u * 256u));
    }
    ptx::bar_sync(1, kSoftmaxThreads);  // before the next block overwrites the buffer (and, in the end, the next segment's P')
  }
  if (p.lse && tid < heads_here) p.lse[row0 + tid] = lds_f32(smem + kOffLse + 4 * tid);
}

// Normalise O^T and write it to a split-KV partial slot, as fp16 divided by the slot scale (the factors in shared memory
// include that division).  A block of 128 dims per round, rolled.
__device__ __noinline__ void write_partial(const DecodeParams& p, uint32_t smem, uint32_t tmem_lane, int row, int half, int slot) {
  __half* so = reinterpret_cast<__half*>(slot_o(p.workspace, slot)) + slot_o_index(row, 32 * half);
#pragma unroll 1
  for (int jb = 0; jb < kBlocks; ++jb, so += 128 * 8) {
    uint32_t o[2][16];
    ptx::tmem_ld16(tmem_lane + kColO + 64u * uint32_t(jb) + uint32_t(32 * half), o[0]);
    ptx::tmem_ld16(tmem_lane + kColO + 64u * uint32_t(jb) + uint32_t(32 * half + 16), o[1]);
    ptx::tmem_wait_ld();
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      uint32_t pk[8];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 f = lds_f32x4(smem + kOffLinv + 4 * (32 * half + 16 * hh + 4 * q));
        __half2 a = __floats2half2_rn(__uint_as_float(o[hh][4 * q]) * f.x, __uint_as_float(o[hh][4 * q + 1]) * f.y);
        __half2 b = __floats2half2_rn(__uint_as_float(o[hh][4 * q + 2]) * f.z, __uint_as_float(o[hh][4 * q + 3]) * f.w);
        pk[2 * q] = *reinterpret_cast<uint32_t*>(&a);
        pk[2 * q + 1] = *reinterpret_cast<uint32_t*>(&b);
      }
      // the warp's 32 dims x 8 heads are 512 contiguous bytes of the slot
      *reinterpret_cast<uint4*>(so + size_t(2 * hh) * kLatent * 8) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
      *reinterpret_cast<uint4*>(so + size_t(2 * hh + 1) * kLatent * 8) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
    }
  }
}

template <bool kSoftCap>
__device__ __forceinline__ void softmax_role(const DecodeParams& p, uint32_t smem, uint32_t tmem, int tid, RoleState& st) {
  Misc* misc = misc_of(smem);
  const int nseg = misc->nseg;
  const Segment* sg = segs_of(smem);
  const int warp = tid >> 5, lane = tid & 31;
  const int quarter = warp & 3;           // TMEM lane quarter this warp may access
  const int half = warp >> 2;             // heads [32*half, 32*half + 32)
  const int row = quarter * 32 + lane;    // token of the tile (S) / dim of the block (O) of this thread
  const uint32_t tmem_lane = tmem + ((uint32_t(quarter) * 32u) << 16);
  const float cscale = p.softmax_scale * kLog2e;
  SoftmaxTile t;
  t.cs2 = pack2(cscale, cscale);
  const float cap = kSoftCap ? p.soft_cap : 0.f;
  t.cap2 = pack2(cap, cap);
  t.rcap2 = pack2(kSoftCap ? 1.f / cap : 0.f, kSoftCap ? 1.f / cap : 0.f);
  // this thread's P' row: two 16-byte chunks of hi and two of lo, swizzled
  const uint32_t psw = (uint32_t(row) >> 1) & 3u;
  const uint32_t p_row = smem + kOffP + uint32_t(row) * 64u;
  const uint32_t notes = smem + kOffNotes + 128 * half;
  bool noted = false;  // this warp's notes of the tile before are not cleared
  bool pending = false;  // a partial has been written in this call

#pragma unroll 1
  for (int si = 0; si < nseg; ++si, ++st.seg) {
    const Segment g = sg[si];
    uint64_t l2[kPairs];
#pragma unroll
    for (int h = 0; h < kPairs; ++h) l2[h] = 0ull;
    float sc_max = 0.f;  // largest |token scale| this thread has seen in the segment
#pragma unroll 1
    for (int tt = g.tile_begin; tt < g.tile_end; ++tt, ++st.it, st.advance(2), st.mod3 = st.mod3 == 2 ? 0 : st.mod3 + 1) {
      const uint32_t it = st.it, s = it & 1;
      const bool first = tt == g.tile_begin;
      // per-token scale (it counts on the barrier of the tile's first pair)
      (void)wait(smem, bar_kv_full(st.slot), st.lap & 1);
      t.valid = (tt * kTile + row) < g.seq_len;
      float sc = lds_f32(smem + kOffScale + 4 * ((it & (kScaleStages - 1)) * kTile + row));
      sc = t.valid ? sc : 0.f;
      sc_max = fmaxf(sc_max, fabsf(sc));
      const float lg = t.valid ? __log2f(fmaxf(fabsf(sc), 8.67361738e-19f)) : 0.f;  // floor 2^-60
      t.sc2 = pack2(sc, sc);
      t.t_lat = tmem_lane + kColSLat + 64u * s + uint32_t(kHalfHeads * half);
      t.t_rope = tmem_lane + kColSRope + 64u * s + uint32_t(kHalfHeads * half);

      (void)wait(smem, bar_s_full(s), (it >> 1) & 1);
      ptx::tc_fence_after();

      // The exponents are taken with the reference as it stands, which holds unless some score beat it by more than the lazy
      // threshold (P' would leave the E4M3 range).  Then the references are moved, and the exponents, the sums and, below, O^T
      // follow.
      uint64_t e2[kPairs];
      t.negm = smem + kOffM + 256 * st.m + 4 * kHalfHeads * half;
      const float mx = exponents<kSoftCap>(t, e2);
      ptx::tc_fence_before();  // orders the S reads before the arrival
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(bar_addr(smem, bar_s_empty(s)));
      const bool beaten = first || mx + lg > kPShift + kLazyThreshold;
      const bool note = __any_sync(0xffffffffu, first || mx + lg > kPShift + kNoteMargin);
      const uint32_t here = notes + 256 * st.mod3;
      if (note) note_tops(here, e2, lg, lane);
      const bool moved = ptx::bar_or(1, kSoftmaxThreads, beaten);
      if (noted) sts_f32(notes + 256 * (st.mod3 == 0 ? 2 : st.mod3 - 1) + 4 * lane, __int_as_float(kNoScore));
      noted = note;
      if (moved) {
        refresh_references(smem, here, st.m, first, half, lane);
        st.m ^= 1u;
        const uint32_t f = smem + kOffF + 4 * kHalfHeads * half;
        const uint64_t minus = pack2(-1.f, -1.f);
#pragma unroll
        for (int q = 0; q < kPairs / 2; ++q) {
          uint64_t d[2], g2[2];
          lds_pairs(f + 256 + 16 * q, d[0], d[1]);
          lds_pairs(f + 16 * q, g2[0], g2[1]);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            e2[2 * q + h] = fma2(d[h], minus, e2[2 * q + h]);
            l2[2 * q + h] = mul2(l2[2 * q + h], g2[h]);
          }
        }
      }
#pragma unroll
      for (int q = 0; q < kPairs; ++q) {
        float y0, y1;
        unpack2(e2[q], y0, y1);
        e2[q] = pack2(ptx::ex2(y0), ptx::ex2(y1));
      }
      // Second half: row sums, and P' = e * scale_t split into two E4M3 terms
      uint32_t hi[8], lo[8];
#pragma unroll
      for (int q = 0; q < kPairs / 2; ++q) {
        uint32_t l0, l1;
        const uint32_t h0 = split_e4m3x2(mul2(e2[2 * q], t.sc2), l0), h1 = split_e4m3x2(mul2(e2[2 * q + 1], t.sc2), l1);
        hi[q] = h0 | (h1 << 16);
        lo[q] = l0 | (l1 << 16);
        l2[2 * q] = add2(l2[2 * q], e2[2 * q]);
        l2[2 * q + 1] = add2(l2[2 * q + 1], e2[2 * q + 1]);
      }
      // The one P buffer (and, for a rescale, O^T) is free once the PV of the previous tile has completed; until then
      // this tile's P' stays in registers.
      if (it >= 1) (void)wait(smem, kBarPvDone, (it - 1) & 1);
      if (moved && !first) {  // O^T holds earlier tiles of the segment
        ptx::tc_fence_after();
        rescale_output(smem, tmem_lane, uint32_t(half), lane);
      }
#pragma unroll
      for (int cidx = 0; cidx < 2; ++cidx) {
        const uint32_t at = p_row + (((2 * uint32_t(half) + uint32_t(cidx)) ^ psw) << 4);
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(hi[4 * cidx]), "r"(hi[4 * cidx + 1]),
                     "r"(hi[4 * cidx + 2]), "r"(hi[4 * cidx + 3]) : "memory");
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at + kTile * 64), "r"(lo[4 * cidx]), "r"(lo[4 * cidx + 1]),
                     "r"(lo[4 * cidx + 2]), "r"(lo[4 * cidx + 3]) : "memory");
      }
      ptx::fence_proxy_async_smem();
      ptx::tc_fence_before();  // orders the O^T writes of a rescale before the arrival
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(bar_addr(smem, kBarPFull));
    }

    // ---- segment epilogue
    const float r = warp_transpose_sum32(l2, lane);  // lane L: this warp's tokens, head 32*half + L
    const uint32_t wred = smem + kOffNotes;
    ptx::bar_sync(1, kSoftmaxThreads);  // nobody reads notes any more
    noted = false;
    sts_f32(wred + 4 * (quarter * kGroupHeads + kHalfHeads * half + lane), r);
    const float sc_warp = ptx::redux_max_f32(sc_max);
    if (lane == 0) sts_f32(smem + kOffScMax + 4 * warp, sc_warp);
    ptx::bar_sync(1, kSoftmaxThreads);
    if (tid < kGroupHeads) {
      float L = 0.f;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        L += lds_f32(wred + 4 * (q * kGroupHeads + tid));
        sts_f32(wred + 4 * (q * kGroupHeads + tid), __int_as_float(kNoScore));
      }
      float m = -lds_f32(smem + kOffM + 256 * st.m + 4 * tid);
      sts_f32(smem + kOffM + 256 * st.m + 4 * tid, 0.f);  // for the next segment
      float Ls = L, fo = p.output_scale;
      if (p.sink && g.tile_begin == 0) {  // the sink: a virtual token with a zero value row, counted with the first tile of a request
        int qpos, head0;
        group_coords(g.g, p.num_heads, qpos, head0);
        if (head0 + tid < p.num_heads) {
          const float sk = __ldg(p.sink + head0 + tid) * kLog2e;
          const float mm = fmaxf(m, sk);
          const float fs = ptx::ex2(m - mm);  // the reference may lie far below the sink: fold it into the output factor, not into L
          fo *= fs;
          Ls = L * fs + ptx::ex2(sk - mm);
          m = mm;
        }
      }
      float slot_scale_v = 1.f;
      if (g.slot >= 0) {  // a partial is stored divided by its slot scale
        const float4 a = lds_f32x4(smem + kOffScMax), b = lds_f32x4(smem + kOffScMax + 16);
        const float sc_all = fmaxf(fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w)), fmaxf(fmaxf(b.x, b.y), fmaxf(b.z, b.w)));
        slot_scale_v = slot_scale_for(6.f * sc_all * fabsf(p.output_scale));
        fo *= __frcp_rn(slot_scale_v);  // a power of two: exact
      }
      const float lse = __log2f(Ls) + m;
      sts_f32(smem + kOffLinv + 4 * tid, __fdividef(fo, Ls));
      sts_f32(smem + kOffLse + 4 * tid, lse);
      if (g.slot >= 0) {
        slot_lse(p.workspace, g.slot)[tid] = lse;
        if (tid == 0) slot_scale(p.workspace, g.slot)[0] = slot_scale_v;
        // The LSEs and the scale of a CTA's last partial go out at once (publish): the merge weights are made from them while O is
        // on its way.
        if (p.fused_merge && si == nseg - 1 && !misc->more) asm volatile("bar.arrive 6, %0;" ::"n"(kGroupHeads + 32) : "memory");
      }
    }
    (void)wait(smem, kBarPvDone, (st.it - 1) & 1);  // the PV of the last tile
    ptx::tc_fence_after();
    if (!ptx::bar_or(1, kSoftmaxThreads, misc->abort != 0)) {  // (all or none: the writers meet at barriers)
      if (g.slot >= 0) write_partial(p, smem, tmem_lane, row, half, g.slot);
      else if (p.out_dtype == MLA_FP4_OUT_BF16) {
        if (p.num_heads <= 32) write_final_bf16<1>(p, smem, tmem_lane, quarter, half, tid, g.b, g.g);
        else write_final_bf16<0>(p, smem, tmem_lane, quarter, half, tid, g.b, g.g);
      }
      else if ((p.num_heads & (kGroupHeads - 1)) == 0) {  // every group is full
        if (p.out_dtype == MLA_FP4_OUT_F32) write_final<MLA_FP4_OUT_F32, true>(p, smem, tmem_lane, row, half, tid, g.b, g.g);
        else write_final<MLA_FP4_OUT_E4M3, true>(p, smem, tmem_lane, row, half, tid, g.b, g.g);
      } else {
        if (p.out_dtype == MLA_FP4_OUT_F32) write_final<MLA_FP4_OUT_F32, false>(p, smem, tmem_lane, row, half, tid, g.b, g.g);
        else write_final<MLA_FP4_OUT_E4M3, false>(p, smem, tmem_lane, row, half, tid, g.b, g.g);
      }
    }
    ptx::tc_fence_before();
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive(bar_addr(smem, kBarOFree));
    pending |= g.slot >= 0;
  }
  if (pending && p.fused_merge) {
    if (!misc->more) {  // (publish)
      asm volatile("bar.arrive 9, %0;" ::"n"(kSoftmaxThreads + 32) : "memory");
    } else {  // a round of whole segments but for the first: others follow
      ptx::bar_sync(1, kSoftmaxThreads);
      if (tid == 0) {
        const int slot = slot_of(blockIdx.x, true);
        st_release(slot_lse_flag(p.workspace, slot), misc->gen);
        st_release(slot_flag(p.workspace, slot), misc->gen);
      }
    }
  }
}

// Publishing the partials, by the QK warp in the last round: the merging CTAs wait for these flags.  A release takes a microsecond,
// until every store before it is in L2, and the softmax warps have the merge weights to make meanwhile.  One release for O of
// both partials, after the last segment: nobody can use a partial before this CTA, itself a writer of the later request, is
// done anyway.  The barriers order the writers' stores before lane 0's release, and a release is cumulative.
// With the softmax warps no longer waiting for either: 4x4096 tokens (64 heads) 14.0 -> 13.25 us, 8x32768 34.8 -> 33.85, 128 requests of
// 128..32768 88.2 -> 87.2, 32 requests with 128 heads 40.9 -> 39.9.
// (On the way, the commit for kBarDrain: nobody can have advanced the generation before this CTA counts itself out, which it does
// after the drain.)
template <bool kPair>
__device__ __noinline__ void publish(const DecodeParams& p, uint32_t smem, int lane) {
  const int nseg = misc_of(smem)->nseg;
  const Segment* sg = segs_of(smem);  // (only a round's first and last segment can be partial)
  const int even = slot_of(cta_of<kPair>(misc_of(smem)), true), first = nseg > 0 ? sg[0].slot : -1, last = nseg > 0 ? sg[nseg - 1].slot : -1;
  const bool head = first == even, tail = last == even + 1;
  const int gen = head || tail ? ld_acquire(ws_generation(p.workspace)) + 1 : 0;
  if (!kPair) {
    if (ptx::elect_one()) ptx::umma_commit(bar_addr(smem, kBarDrain));
  } else if (!(blockIdx.x & 1)) {
    if (ptx::elect_one()) ptx::umma_commit_pair(bar_addr(smem, kBarDrain));
  }
  __syncwarp();
  if (!head && !tail) return;
  if (last >= 0) {
    ptx::bar_sync(6, kGroupHeads + 32);
    if (lane == 0) st_release(slot_lse_flag(p.workspace, last), gen);
    __syncwarp();
  }
  ptx::bar_sync(9, kSoftmaxThreads + 32);
  if (lane == 0) {
    if (head && last != even) st_release(slot_lse_flag(p.workspace, even), gen);
    if (head) st_release(slot_flag(p.workspace, even), gen);
    if (tail) st_release(slot_flag(p.workspace, even + 1), gen);
  }
  __syncwarp();
}

// ------------------------------------------------------------------------------------------
// tail: merge of the split-KV partials inside the decode kernel
// ------------------------------------------------------------------------------------------
// Every CTA that wrote a partial of a split request stamps the slot's flag with the generation of this step.  Two forms:
//
// kMergeShared: the CTAs whose partial of a request was their first segment merge it, each a share of the slots' bytes
// (units of 16: eight heads of one dim).  A CTA has published everything it will ever publish before it waits for anybody
// else, so the waits cannot form a cycle; but it may only wait for CTAs that are running.
//
// kMergeLast: nobody waits; the CTA that publishes the last partial of a request (an arrival counter per request) merges
// it alone.  Slower (one CTA reads every partial), and right whether or not the whole grid is resident.
//
// The first CTA to reach its tail decides for the whole grid: kMergeShared when every CTA has started by then, which is the
// case whenever the grid has the GPU to itself for a moment.  A cooperative launch gave the same guarantee and cost 3.3 us
// per step launched outside a graph (it does not overlap the kernel before it): 22.7 -> 19.4 us for 4 x 4096 tokens.
constexpr int kMergeShared = 1, kMergeLast = 2;
constexpr uint32_t kTailBytes = uint32_t(kSlotTailBytes);               // a slot's tail: 64 LSEs, the slot scale, the flag, an arrival counter, the flag of the LSEs
constexpr uint32_t kTailStage = kOffKV;                                 // staging: [slots][this CTA's bytes of a slot], then the tails
constexpr uint32_t kTailRed = kOffScale - kThreads * 32;                // [384][8] f32: sums of a unit that several threads share
constexpr uint32_t kTailStageBytes = kOffP - kTailStage;                // the KV ring, RoPE and Q; not P, where the last segment's output may still be in transit
static_assert(kTailStageBytes >= 2 * (kSlotOBytes + kTailBytes), "two whole slots fit (a request cut once)");
static_assert(kTailStageBytes >= kSlotOBytes + kSlotOBytes / 8 + kWsTailsBytes, "a request cut 148 times fits");

// Requests without tokens: zero rows and LSE -inf (the sink's logit when there is a sink).
__device__ __noinline__ void zero_empty_requests(const DecodeParams& p, int lane) {
  const int total = p.groups * p.batch;
  const uint32_t esz = uint32_t(out_elem_bytes(p.out_dtype));
#pragma unroll 1
  for (int v = blockIdx.x; v < total; v += gridDim.x) {
    const int g = v / p.batch, b = v - g * p.batch;
    if (capped_len(p.seq_lens, b, p.seq_cap) > 0) continue;
    int qpos, head0;
    group_coords(g, p.num_heads, qpos, head0);
    const int heads_here = min(kGroupHeads, p.num_heads - head0);
    const size_t row0 = (size_t(b) * p.q_len + qpos) * p.num_heads + head0;
    uint4* dst = reinterpret_cast<uint4*>(static_cast<char*>(p.out) + row0 * kLatent * esz);
    const uint32_t n16 = uint32_t(heads_here) * kLatent * esz / 16u;
#pragma unroll 4
    for (uint32_t i = lane; i < n16; i += 32) dst[i] = make_uint4(0u, 0u, 0u, 0u);
    if (p.lse)
      for (int h = lane; h < heads_here; h += 32) p.lse[row0 + h] = p.sink ? __ldg(p.sink + head0 + h) * kLog2e : -INFINITY;
  }
}

// The merge plan of one split request, made by one warp: the slots of its writers in CTA order, how many CTAs merge it in
// the shared form (those whose partial was their first segment: every CTA then takes part in at most one merge) and this
// CTA's place among them.  The writers are the CTAs whose range holds a real tile; they are consecutive, as no CTA that shares
// the work is without a tile.
template <bool kPair>
__device__ __noinline__ void plan_merge(uint32_t smem, int which, int lane) {
  Misc* misc = misc_of(smem);
  const MergeReq m = misc->merge[which];
  if (m.vtiles == 0) {
    if (lane == 0) misc->n_slots = 0;
    return;
  }
  const int n = misc->n, cta = cta_of<kPair>(misc);
  const flat_t Tt = misc->Tt;
  const flat_t f0 = m.start + kPhantom;
  const int ends = cta_of_tile(Tt, n, (lane & 1) ? m.start + m.vtiles - 1 : f0);
  const int c0 = __shfl_sync(0xffffffffu, ends, 0), c1 = __shfl_sync(0xffffffffu, ends, 1);
  const int ns = min(c1 - c0 + 1, kMaxCombineSlots);  // (work_ctas leaves no CTA of these without a tile: Tt >= n)
  const bool head_even = cta_lo(Tt, n, c0) >= m.start;  // the first writer's range starts with the request
#pragma unroll 1
  for (int k = lane; k < ns; k += 32) {
    sts_f32(smem + kOffTail + 4u * uint32_t(k), __int_as_float(slot_of(c0 + k, k > 0 || head_even)));
  }
  if (lane == 0) {
    const int skip = head_even ? 0 : 1;
    const int rank = cta - c0 - skip, part = ns - skip;
    misc->m = m;
    misc->n_slots = ns;
    misc->n_part = part;
    misc->rank = rank;
    misc->unit0 = (4096 * rank) / part;
    misc->unit1 = (4096 * (rank + 1)) / part;
  }
  __syncwarp();
}

// How this step merges (see above); one lane per CTA asks.
__device__ __noinline__ int merge_mode(const DecodeParams& p) {
  int32_t* mode = ws_mode(p.workspace);
  int m = ld_relaxed(mode);
  if (m == 0) {
    const int mine = (!p.merge_last && ld_relaxed(ws_started(p.workspace)) == int(gridDim.x)) ? kMergeShared : kMergeLast;
    m = atomicCAS(mode, 0, mine);
    if (m == 0) m = mine;
  }
  return m;
}

// Fetching the partials, by three of the issue warps: slot i (and i + 96) belongs to lane i / 3 of helper warp i % 3, which waits
// for its flag (shared form) and fetches this CTA's share of it with a bulk copy.  In the shared form that
// starts as soon as the last tile's MMAs have drained, while the softmax warps still write and publish this CTA's own
// partial.  A bulk copy costs about fifty clocks to issue whatever its size and the lanes of a warp issue theirs one after the
// other, so the slots are dealt round the warps.  The lanes of a warp poll in step.
__device__ __noinline__ void tail_fetch(const DecodeParams& p, uint32_t smem, int hw, int lane, bool flags) {
  Misc* misc = misc_of(smem);
  void* ws = p.workspace;
  const int ns = misc->n_slots, gen = misc->gen;
  const uint32_t U0 = uint32_t(misc->unit0), share = (uint32_t(misc->unit1) - U0) * 16u;
  const uint32_t rows = smem + kTailStage;
  const uint32_t bar = bar_addr(smem, kBarTail), polls = misc->polls;
#pragma unroll 1
  for (int i = lane * kFetchWarps + hw; __any_sync(0xffffffffu, i < ns); i += 32 * kFetchWarps) {
    const int slot = i < ns ? int(lds_u32(smem + kOffTail + 4u * uint32_t(i))) : 0;
    bool done = i >= ns;
#pragma unroll 1
    for (uint32_t it = 0; it < polls; ++it) {
      // acquire: the slot's bytes, written before the flag, are read after it; they were written by ordinary stores and the copy
      // belongs to the async proxy, hence the fence (of global memory alone: 0.05 us; a full one cost microseconds here).
      if (!done && (!flags || ld_acquire(slot_flag(ws, slot)) == gen)) {
        done = true;
        ptx::fence_proxy_async_global();
        ptx::mbar_expect_tx(bar, share);
        ptx::bulk_load(rows + uint32_t(i) * share, reinterpret_cast<const char*>(slot_o(ws, slot)) + size_t(U0) * 16, share, bar);
      }
      if (__all_sync(0xffffffffu, done) || __any_sync(0xffffffffu, misc->abort)) break;
      __nanosleep(32);
    }
    if (!done && !misc->abort) flag_timeout(smem, 100, uint32_t(slot));  // the budget ran out
    __syncwarp();
    if (misc->abort) break;
  }
  __syncwarp();
  if (lane == 0) ptx::mbar_arrive(bar);  // one of kFetchWarps
}

// eight heads of one dim
template <typename Store>
__device__ __forceinline__ void store_unit(const float (&acc)[8], const float4& i0, const float4& i1, int heads, Store store) {
  const float inv[8] = {i0.x, i0.y, i0.z, i0.w, i1.x, i1.y, i1.z, i1.w};
#pragma unroll
  for (int e = 0; e < 8; ++e)
    if (e < heads) store(e, acc[e] * inv[e]);
}

// eight dims of one head
__device__ __forceinline__ void store_dims(const DecodeParams& p, const float (&acc)[8], float inv, size_t at) {
  if (p.out_dtype == MLA_FP4_OUT_F32) {
    float4* d = reinterpret_cast<float4*>(static_cast<float*>(p.out) + at);
    d[0] = make_float4(acc[0] * inv, acc[1] * inv, acc[2] * inv, acc[3] * inv);
    d[1] = make_float4(acc[4] * inv, acc[5] * inv, acc[6] * inv, acc[7] * inv);
  } else {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (p.out_dtype == MLA_FP4_OUT_BF16) {
        const __nv_bfloat162 t = __floats2bfloat162_rn(acc[2 * i] * inv, acc[2 * i + 1] * inv);
        w[i] = *reinterpret_cast<const uint32_t*>(&t);
      } else {
        w[i] = __nv_cvt_float2_to_fp8x2(make_float2(acc[2 * i] * inv, acc[2 * i + 1] * inv), __NV_SATFINITE, __NV_E4M3);
      }
    }
    if (p.out_dtype == MLA_FP4_OUT_BF16) *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.out) + at) = make_uint4(w[0], w[1], w[2], w[3]);
    else *reinterpret_cast<uint2*>(static_cast<uint8_t*>(p.out) + at) = make_uint2(w[0] | (w[1] << 16), w[2] | (w[3] << 16));
  }
}

// The merge weights w_i = 2^(lse_i - max) * slot scale of the 64 heads, and the inverse of their sum, by the eight softmax
// warps: four lanes per head split the slots, butterflies give all four the results.  They are computed while the shares of the
// slots are on their way: the LSEs come straight from L2, under flags of their own (shared form).
// A round of loads takes 0.65 us: eight slots of a lane go together, and the scales, one to a thread, beside the first of them (five
// slots with their scales in every lane before): 1x16000 tokens 16.35 -> 15.3 us, 1x32768 19.3 -> 18.25, 7 ragged requests 13.2 -> 12.75.
__device__ __noinline__ void merge_weights(const DecodeParams& p, uint32_t smem, int tid, bool flags, bool with_lse) {
  Misc* misc = misc_of(smem);
  const int ns = misc->n_slots;
  const uint32_t tails = smem + kTailStage + uint32_t(ns) * (uint32_t(misc->unit1 - misc->unit0) * 16u);
  const int h = tid >> 2, j = tid & 3;
  const uint32_t col = tails + 4u * uint32_t(h);
  if (flags) {
    const int lane = tid & 31, gen = misc->gen;
    const uint32_t polls = misc->polls;
    bool all = false;
#pragma unroll 1
    for (uint32_t it = 0; it < polls && !all; ++it) {
      bool up = true;
      for (int i = lane; i < ns; i += 32) up &= ld_acquire(slot_lse_flag(p.workspace, int(lds_u32(smem + kOffTail + 4u * uint32_t(i))))) == gen;
      all = __all_sync(0xffffffffu, up);
      if (__any_sync(0xffffffffu, misc->abort)) break;
    }
    if (!all && lane == 0 && !misc->abort) flag_timeout(smem, 101, uint32_t(ns));
    __syncwarp();
  }
  float sc = 0.f;
  if (tid < ns) sc = __ldcg(slot_scale(p.workspace, int(lds_u32(smem + kOffTail + 4u * uint32_t(tid)))));  // (at most 148 slots)
  float mx = -INFINITY;
#pragma unroll 1
  for (int i0 = j; i0 < ns; i0 += 4 * 8) {  // eight slots' loads in flight together
    float l[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) l[k] = __ldcg(slot_lse(p.workspace, int(lds_u32(smem + kOffTail + 4u * uint32_t(min(i0 + 4 * k, ns - 1))))) + h);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int i = i0 + 4 * k;
      mx = fmaxf(mx, l[k]);  // (a repeated last slot changes nothing)
      if (i < ns) sts_f32(col + uint32_t(i) * kTailBytes, l[k]);
    }
  }
  if (tid < ns) sts_f32(tails + uint32_t(tid) * kTailBytes + 4u * kGroupHeads, sc);
  mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
  mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
  ptx::bar_sync(1, kSoftmaxThreads);
  float dsum = 0.f;
#pragma unroll 2
  for (int i = j; i < ns; i += 4) {
    const uint32_t at = uint32_t(i) * kTailBytes;
    const float l = lds_f32(col + at);
    const float e = (l == -INFINITY) ? 0.f : ptx::ex2(l - mx);
    sts_f32(col + at, e * lds_f32(tails + at + 4u * kGroupHeads));
    dsum += e;
  }
  dsum += __shfl_xor_sync(0xffffffffu, dsum, 1);
  dsum += __shfl_xor_sync(0xffffffffu, dsum, 2);
  if (j == 0) {
    sts_f32(smem + kOffLinv + 4u * uint32_t(h), dsum > 0.f ? __frcp_rn(dsum) : 0.f);
    const MergeReq m = misc->m;
    int qpos, head0;
    group_coords(m.g, p.num_heads, qpos, head0);
    if (with_lse && p.lse && head0 + h < p.num_heads)
      p.lse[(size_t(m.b) * p.q_len + qpos) * p.num_heads + head0 + h] = (dsum > 0.f) ? (__log2f(dsum) + mx) : -INFINITY;
  }
}

// out = sum_i w_i * O_i / sum, over the staged shares, in an order that depends on the number of slots and units alone and not on
// the order of arrival: both forms cut the units into the same shares, so they agree to the bit.  All threads of the CTA; the
// weights are there.
template <bool kPair>
__device__ __noinline__ void tail_merge_of(const DecodeParams& p, uint32_t smem, int tid, uint32_t parity) {
  Misc* misc = misc_of(smem);
  const int ns = misc->n_slots;
  const MergeReq m = misc->m;
  int qpos, head0;
  group_coords(m.g, p.num_heads, qpos, head0);
  const int heads_here = min(kGroupHeads, p.num_heads - head0);
  const size_t row0 = (size_t(m.b) * p.q_len + qpos) * p.num_heads + head0;
  const int U0 = misc->unit0, nu = misc->unit1 - U0;
  const uint32_t share = uint32_t(nu) * 16u, rows = smem + kTailStage, tails = rows + uint32_t(ns) * share;
  const bool landed = wait(smem, kBarTail, parity);
  if (!landed && (tid & 31) == 0) drain_wait(smem, kBarTail, parity);  // giving up: copies in flight land first
  if (__syncthreads_or(!landed || misc->abort)) return;  // (uniform: there is a barrier below)
  // A thread per unit, or, when there are fewer units than threads, S threads per unit, each with every S-th slot.
  const int S = min(max(kThreads / nu, 1), ns);
  const int s = S > 1 ? tid / nu : 0;
#pragma unroll 1
  for (int u0 = 0; u0 < nu; u0 += kThreads) {  // (one pass when S > 1)
    const int u = u0 + tid - s * nu;
    bool active = s < S && u < nu;
    // (a unit is eight heads of a dim, or, in the pair kernel, eight dims of a head)
    const int unit = U0 + u, hg = unit >> 9, dim = unit & 511, head = unit >> 6;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (active) {
      uint64_t sum[4] = {0ull, 0ull, 0ull, 0ull};  // pairs of heads
      uint32_t src = rows + uint32_t(s) * share + uint32_t(u) * 16u, w = tails + uint32_t(s) * kTailBytes + (kPair ? 4u * uint32_t(head) : 32u * uint32_t(hg));
#pragma unroll 4
      for (int i = s; i < ns; i += S) {
        const uint4 v = lds_u32x4(src);
        uint64_t wp[4];
        if (kPair) {
          const float wh = lds_f32(w);
          wp[0] = wp[1] = wp[2] = wp[3] = pack2(wh, wh);
        } else {
          lds_pairs(w, wp[0], wp[1]);
          lds_pairs(w + 16u, wp[2], wp[3]);
        }
        src += uint32_t(S) * share;
        w += uint32_t(S) * kTailBytes;
        const uint32_t vs[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&vs[e]));
          sum[e] = fma2(wp[e], pack2(f.x, f.y), sum[e]);
        }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) unpack2(sum[e], acc[2 * e], acc[2 * e + 1]);
    }
    if (S > 1) {
      const uint32_t red = smem + kTailRed + uint32_t(tid) * 4u;  // [8][384]: conflict-free
#pragma unroll
      for (int e = 0; e < 8; ++e) sts_f32(red + uint32_t(e) * (kThreads * 4), acc[e]);
      __syncthreads();
      active = active && s == 0;
      if (active)
#pragma unroll 1
        for (int k = 1; k < S; ++k)
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[e] += lds_f32(red + uint32_t(e) * (kThreads * 4) + uint32_t(k * nu) * 4u);
    }
    if (!active) continue;
    if (kPair) {
      if (head < heads_here) store_dims(p, acc, lds_f32(smem + kOffLinv + 4u * uint32_t(head)), (row0 + head) * kLatent + 8 * (unit & 63));
      continue;
    }
    const float4 i0 = lds_f32x4(smem + kOffLinv + 32u * uint32_t(hg)), i1 = lds_f32x4(smem + kOffLinv + 32u * uint32_t(hg) + 16u);
    const size_t idx = (row0 + 8 * hg) * kLatent + dim;
    const int heads = heads_here - 8 * hg;
    if (p.out_dtype == MLA_FP4_OUT_BF16) {
      __nv_bfloat16* d = static_cast<__nv_bfloat16*>(p.out) + idx;
      store_unit(acc, i0, i1, heads, [&](int e, float v) { d[e * kLatent] = __float2bfloat16_rn(v); });
    } else if (p.out_dtype == MLA_FP4_OUT_F32) {
      float* d = static_cast<float*>(p.out) + idx;
      store_unit(acc, i0, i1, heads, [&](int e, float v) { d[e * kLatent] = v; });
    } else {
      uint8_t* d = static_cast<uint8_t*>(p.out) + idx;
      store_unit(acc, i0, i1, heads, [&](int e, float v) { d[e * kLatent] = __nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3); });
    }
  }
}

// The last-writer form: for each request this CTA wrote a partial of, count it in; the last to arrive merges it, share by share.
// A CTA that has given up counts itself in all the same: the counters are back to zero after every step, whatever became of it.
template <bool kPair>
__device__ __noinline__ void merge_as_last(const DecodeParams& p, uint32_t smem, int tid) {
  constexpr auto& tail_merge = tail_merge_of<kPair>;
  Misc* misc = misc_of(smem);
  uint32_t parity = 0;
#pragma unroll 1
  for (int which = 0; which < 2; ++which) {
    if (misc->merge[which].vtiles == 0) continue;
    if (tid < 32) plan_merge<kPair>(smem, which, tid);
    __syncthreads();
    const int ns = misc->n_slots, part = misc->n_part;  // (the shares of the shared form, so that both sum in the same order)
    if (tid == 0) {
      int32_t* arrivals = slot_arrivals(p.workspace, int(lds_u32(smem + kOffTail)));
      __threadfence();  // this CTA's partial (published after a barrier of its writers) before the count
      misc->last = atomicAdd(arrivals, 1) == ns - 1;
      __threadfence();
      if (misc->last) *arrivals = 0;
    }
    __syncthreads();
    if (!misc->last) continue;
#pragma unroll 1
    for (int r = 0; r < part; ++r, parity ^= 1u) {
      if (__syncthreads_or(misc->abort)) break;
      if (tid == 0) {
        misc->unit0 = (4096 * r) / part;
        misc->unit1 = (4096 * (r + 1)) / part;
      }
      __syncthreads();
      if (tid < 32 * kFetchWarps) tail_fetch(p, smem, tid >> 5, tid & 31, false);
      else if (tid >= 128) merge_weights(p, smem, tid - 128, false, r == 0);
      __syncthreads();
      tail_merge(p, smem, tid, parity);
      ptx::fence_proxy_async_smem();  // the weights written here and the shares read give way to the copies of the next share
      __syncthreads();
    }
  }
}

// ------------------------------------------------------------------------------------------
// kernel
// ------------------------------------------------------------------------------------------
template <bool kSoftCap, Form F>
__global__ void __launch_bounds__(kThreads, 1)
mla_fp4_decode_sm100_kernel(const __grid_constant__ DecodeParams p, const __grid_constant__ CUtensorMap map_q_lat,
                            const __grid_constant__ CUtensorMap map_q_rope, const __grid_constant__ CUtensorMap map_rope,
                            const __grid_constant__ CUtensorMap map_lat) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  Misc* misc = misc_of(smem);
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = int(ptx::uniform_u32(uint32_t(tid >> 5)));

  // What needs nothing an earlier kernel wrote comes first: with a programmatic dependent launch this part runs
  // while the kernel before this one on the stream is still draining.
  if (warp == kWarpQK) {
    ptx::tmem_alloc(smem + kOffMisc + offsetof(Misc, tmem_base), 512);
    ptx::tmem_relinquish();
  } else if (warp == kWarpPV) {
    if (lane < kNumBars) {  // lane i: barrier i
      uint32_t count = 1;
      if (lane == kBarPFull || lane == kBarOFree || lane == bar_s_empty(0) || lane == bar_s_empty(1)) count = kSoftmaxWarps;
      if (lane == kBarDrain) count = 2;  // the two MMA warps
      if (lane == kBarTail) count = kFetchWarps;
      ptx::mbar_init(bar_addr(smem, lane), count);
    }
    ptx::fence_barrier_init();
    if (lane == 0) {
      misc->abort = 0;
      misc->polls = p.wait_polls;
      misc->status = p.status;
      misc->n_slots = 0;
    }
  } else if (warp == kWarpPlan) {
    asm volatile("bar.arrive 7, %0;" ::"n"(kThreads) : "memory");
    if (p.pdl_wait) {  // a first plan, from the lengths as they are in memory; the TMA warp decides whether it stands
      stage_segments<F>(p, smem, lane, true, false);
      ptx::fence_proxy_async_smem();
      __threadfence_block();
      asm volatile("bar.arrive 8, 64;" ::: "memory");
    }
  } else if (warp == kWarpSoftmax0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) sts_f32(smem + kOffNotes + 4 * (lane + 32 * i), __int_as_float(kNoScore));
    sts_f32(smem + kOffM + 4 * lane, 0.f);
    sts_f32(smem + kOffM + 4 * (lane + 32), 0.f);
  } else if (warp == kWarpTMA2 && lane == 0) {
    ptx::prefetch_tensormap(&map_q_lat);
    ptx::prefetch_tensormap(&map_q_rope);
    ptx::prefetch_tensormap(&map_rope);
    ptx::prefetch_tensormap(&map_lat);
  }
  ptx::tc_fence_before();
  if (warp != kWarpPlan) ptx::bar_sync(7, kThreads);
  RoleState st{};
  if (warp != kWarpTMA && warp != kWarpTMA2) {  // (these two: in their role, after a first pass without effect)
    start_work<F>(p, smem, warp, lane);
  }
  ptx::tc_fence_after();
  const uint32_t tmem = ptx::uniform_u32(misc->tmem_base);
  // Rounds: almost always exactly one; more only when a CTA's range spans more than kMaxSeg requests.
  bool first_round = true;
  int finished = -1;
#pragma unroll 1
  for (;;) {
    if (warp >= kWarpSoftmax0) {
      softmax_role<kSoftCap>(p, smem, tmem, tid - 32 * kWarpSoftmax0, st);
      if (p.fused_merge && !misc->more && misc->n_slots > 0) {
        ptx::bar_sync(5, kThreads - 32);
        if (misc->mode == kMergeShared) merge_weights(p, smem, tid - 32 * kWarpSoftmax0, true, misc->rank == 0);
      }
    } else if (warp == kWarpQK) {
      qk_role(p, smem, tmem, &map_q_lat, &map_q_rope, st);
    } else if (warp == kWarpPV) {
      if (first_round && p.fused_merge) {  // (the two-kernel modes leave all this to the combine kernel); the first P is far away
        // The generation of this step: one more than that of the last completed step.  No CTA of this step can have advanced it
        // yet (that takes every CTA of the grid to have finished).
        if (lane == 0) {
          atomicAdd(ws_started(p.workspace), 1);
          misc->gen = ld_acquire(ws_generation(p.workspace)) + 1;
        }
        plan_merge<false>(smem, 0, lane);
        zero_empty_requests(p, lane);
      }
      pv_role(smem, tmem, st);
    } else {
      tma_role<F>(p, smem, warp == kWarpTMA2 ? 1u : 0u, &map_rope, &map_lat, st, first_round);
    }
    const int more = misc->more;
    if (!more && warp < kWarpSoftmax0) {
      // Last round: drain (everything issued has completed before TMEM is released and before shared memory is reused:
      // a commit covers the MMAs of the thread that executes it), then these warps, idle from here on, publish this CTA's
      // partials and fetch those of the request it merges while the softmax warps finish with its own.
      const bool publishes = warp == kWarpQK && p.fused_merge;
      if (((warp == kWarpQK && !publishes) || warp == kWarpPV) && ptx::elect_one()) ptx::umma_commit(bar_addr(smem, kBarDrain));
      __syncwarp();
      if (publishes) {
        publish<false>(p, smem, lane);
      } else {
        if (lane == 0) drain_wait(smem, kBarDrain, 0);
        __syncwarp();
      }
      if (p.fused_merge && !publishes) {
        if (warp == kWarpPV && lane == 0) {
          if (misc->merge[0].vtiles | misc->merge[1].vtiles) misc->mode = merge_mode(p);
        }
        ptx::bar_sync(3, 32 * kFetchWarps);
        if (misc->n_slots > 0) {
          __threadfence_block();
          asm volatile("bar.arrive 5, %0;" ::"n"(kThreads - 32) : "memory");  // the mode is known
          if (misc->mode == kMergeShared) tail_fetch(p, smem, warp - kWarpTMA, lane, true);
        }
        // This CTA has no more use for the header.  (The count comes back while the merge goes on.)
        if (warp == kWarpPV && lane == 0) finished = atomicAdd(ws_finished(p.workspace), 1);
      }
    }
    __syncthreads();  // every role is done with the staged segments
    if (!more) break;
    first_round = false;
    if (warp == kWarpTMA) {
      stage_segments<F>(p, smem, lane, false, false);
      ptx::fence_proxy_async_smem();
    }
    __syncthreads();
  }
  if (warp == kWarpQK) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 512);
  }
  if (p.fused_merge) {
    if (misc->merge[0].vtiles | misc->merge[1].vtiles) {
      if (misc->mode == kMergeLast) merge_as_last<false>(p, smem, tid);
      else if (misc->n_slots > 0) tail_merge_of<false>(p, smem, tid, 0);
    }
    // The last CTA to have counted itself out advances the generation (the next step's flags differ from all of this one's) and
    // resets the counters.
    if (finished == int(gridDim.x) - 1) {
      *ws_finished(p.workspace) = 0;
      *ws_started(p.workspace) = 0;
      *ws_mode(p.workspace) = 0;
      st_release(ws_generation(p.workspace), misc->gen);
    }
  }
}

#include "decode_pair.cuh"  // (in this namespace: it is the other half of this file)

// ------------------------------------------------------------------------------------------ host

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      return reinterpret_cast<EncodeTiledFn>(ptr);
    return static_cast<EncodeTiledFn>(nullptr);
  }();
  return fn;
}

bool encode_map(CUtensorMap* m, const void* base, int rank, const uint64_t* dims, const uint64_t* strides_bytes,
                const uint32_t* box, CUtensorMapSwizzle swz) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return false;
  cuuint64_t gd[5], gs[4];
  cuuint32_t bx[5], es[5];
  for (int i = 0; i < rank; ++i) { gd[i] = dims[i]; bx[i] = box[i]; es[i] = 1; }
  for (int i = 0; i + 1 < rank; ++i) gs[i] = strides_bytes[i];
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, rank, const_cast<void*>(base), gd, gs, bx, es,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// The four tensor maps of a launch depend only on addresses, strides and shapes: two on the query, two on the cache.
// Encoding a map costs about a microsecond of host time, and a serving program calls with the same sets again and again,
// one cache per layer: each thread keeps the last maps in a small direct-mapped table (a bounded 2 x 64 entries; one
// entry, the form before, was overwritten by every layer's call).
struct QKey {
  const void* q;
  int64_t sb, sq, sh;
  int32_t batch, q_len, num_heads, dev;
  bool operator==(const QKey& o) const {
    return q == o.q && sb == o.sb && sq == o.sq && sh == o.sh && batch == o.batch && q_len == o.q_len && num_heads == o.num_heads && dev == o.dev;
  }
};
struct KvKey {
  const void* kv;
  int64_t num_pages;
  int32_t page_size, rows, dev;  // rows: of a box
  bool operator==(const KvKey& o) const { return kv == o.kv && num_pages == o.num_pages && page_size == o.page_size && rows == o.rows && dev == o.dev; }
};
template <typename Key>
struct MapPair {
  CUtensorMap a, b;  // (aligned first)
  Key key;
  bool valid = false;
};
constexpr uint32_t kMapEntries = 64;
uint32_t map_slot(const void* p) {
  return uint32_t((reinterpret_cast<uintptr_t>(p) >> 8) * 0x9E3779B97F4A7C15ull >> 58);
}

// q viewed as [576, H, q_len, B] bytes: a box of 128 latent values (or the 64 RoPE values) of 64 heads
bool encode_q_maps(const DecodeParams& p, CUtensorMap* lat, CUtensorMap* rope) {
  const uint64_t sq = p.q_len > 1 ? uint64_t(p.q_stride_qpos) : uint64_t(p.q_stride_head) * uint64_t(p.num_heads);
  const uint64_t sb = p.batch > 1 ? uint64_t(p.q_stride_batch) : sq * uint64_t(p.q_len);
  const uint64_t dims[4] = {uint64_t(kQDim), uint64_t(p.num_heads), uint64_t(p.q_len), uint64_t(p.batch)};
  const uint64_t strides[3] = {uint64_t(p.q_stride_head), sq, sb};
  const uint32_t box_lat[4] = {128, uint32_t(kGroupHeads), 1, 1};
  const uint32_t box_rope[4] = {64, uint32_t(kGroupHeads), 1, 1};
  return encode_map(lat, p.q, 4, dims, strides, box_lat, CU_TENSOR_MAP_SWIZZLE_128B) &&
         encode_map(rope, p.q, 4, dims, strides, box_rope, CU_TENSOR_MAP_SWIZZLE_64B);
}
// the RoPE bytes of a page, and the cache as 4-bit elements: 640 per row (the 512 latent codes, then the RoPE bytes seen as
// nibbles and never fetched through this map), page_size rows per page; a box is one 128-dim block of `rows` rows of a page
bool encode_kv_maps(const DecodeParams& p, uint32_t rows, CUtensorMap* lat, CUtensorMap* rope) {
  const uint64_t dims[3] = {uint64_t(kRowBytes), uint64_t(p.page_size), uint64_t(p.num_pages)};
  const uint64_t strides[2] = {uint64_t(kRowBytes), uint64_t(kRowBytes) * uint64_t(p.page_size)};
  const uint32_t box[3] = {64, rows, 1};
  if (!encode_map(rope, p.kv_cache, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B)) return false;
  EncodeTiledFn fn = get_encode_fn();
  cuuint64_t gd[3] = {cuuint64_t(2 * kRowBytes), cuuint64_t(p.page_size), cuuint64_t(p.num_pages)};
  cuuint64_t gs[2] = {cuuint64_t(kRowBytes), cuuint64_t(kRowBytes) * cuuint64_t(p.page_size)};
  cuuint32_t bx[3] = {128, cuuint32_t(rows), 1};
  cuuint32_t es[3] = {1, 1, 1};
  return fn(lat, CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B, 3, const_cast<void*>(p.kv_cache), gd, gs, bx, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

cudaError_t launch_decode_sm100(const DecodeParams& p, int num_ctas, cudaStream_t stream, const char** err) {
  *err = nullptr;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  static thread_local MapPair<QKey> q_maps[kMapEntries];
  static thread_local MapPair<KvKey> kv_maps[kMapEntries];
  MapPair<QKey>& qm = q_maps[map_slot(p.q)];
  MapPair<KvKey>& km = kv_maps[map_slot(p.kv_cache)];
  const QKey qkey{p.q, p.q_stride_batch, p.q_stride_qpos, p.q_stride_head, p.batch, p.q_len, p.num_heads, dev};
  const DecodeForm form = p.fused_merge ? decode_form({p.batch, p.groups, p.num_heads, p.page_size, p.longest, num_ctas, p.out_dtype, p.soft_cap > 0.f, p.phase_mask})
                                        : DecodeForm{false, num_ctas, 1};
  const bool pair = form.pair;
  const uint32_t rows = pair && p.page_size > 64 ? 64u : uint32_t(p.page_size);
  const KvKey kvkey{p.kv_cache, p.num_pages, p.page_size, int32_t(rows), dev};
  if (!(qm.valid && qm.key == qkey)) {
    qm.valid = false;
    if (!encode_q_maps(p, &qm.a, &qm.b)) {
      *err = "cuTensorMapEncodeTiled failed for q (check alignment and strides)";
      return cudaErrorInvalidValue;
    }
    qm.key = qkey;
    qm.valid = true;
  }
  if (!(km.valid && km.key == kvkey)) {
    km.valid = false;
    if (!encode_kv_maps(p, rows, &km.a, &km.b)) {
      *err = "cuTensorMapEncodeTiled failed for kv_cache (it must be 32-byte aligned)";
      return cudaErrorInvalidValue;
    }
    km.key = kvkey;
    km.valid = true;
  }
  const CUtensorMap &map_q_lat = qm.a, &map_q_rope = qm.b, &map_rope = km.b, &map_lat = km.a;
  // the attention variant with a score transform is a kernel of its own, as is each form: none carries another's instructions
  using Kernel = void (*)(DecodeParams, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap);
  static constexpr Kernel kernels[3][2] = {
      {mla_fp4_decode_sm100_kernel<false, kFormAlone>, mla_fp4_decode_sm100_kernel<true, kFormAlone>},
      {mla_fp4_decode_sm100_kernel<false, kFormShared>, mla_fp4_decode_sm100_kernel<true, kFormShared>},
      {mla_fp4_decode_pair_kernel<false>, mla_fp4_decode_pair_kernel<true>}};
  {
    // (all of them with the first step: a later one may be under capture, where no kernel should be loaded)
    static std::atomic<bool> attr_done[64];  // zero-initialised; setting the attribute twice is harmless
    if (dev < 0 || dev >= 64 || !attr_done[dev].load(std::memory_order_acquire)) {
      for (const Kernel(&forms)[2] : kernels) {
        for (const Kernel k : forms) {
          e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemAlloc));
          if (e != cudaSuccess) return e;
        }
      }
      if (dev >= 0 && dev < 64) attr_done[dev].store(true, std::memory_order_release);
    }
  }
  const Kernel kernel = kernels[pair ? kFormPair : (form.share > 1 ? kFormShared : kFormAlone)][p.soft_cap > 0.f];
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(form.grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemAlloc;
  cfg.stream = stream;
  // Programmatic dependent launch: the CTAs are placed and run their prologue while the kernel before this one on the
  // stream drains, then wait for that kernel's completion.
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.pdl ? 1 : 0;
  DecodeParams pp = p;
  pp.pdl_wait = p.pdl;
  pp.page_shift = __builtin_ctz(unsigned(p.page_size));
  return cudaLaunchKernelEx(&cfg, kernel, pp, map_q_lat, map_q_rope, map_rope, map_lat);
}

}  // namespace mla
