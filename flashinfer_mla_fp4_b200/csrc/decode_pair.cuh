// Decode kernel for an even number of head groups: a cluster of two CTAs decodes two groups (128 query rows) of the same tiles.
// Part of decode_sm100.cu, with its waits, partition, exchange of partials and shared-memory map.
//
// Here the heads are on the M axis.  The MMAs are those of a CTA pair (cta_group::2, M = 128): CTA r holds the 64 rows of its group, in
// A and in the accumulators, and half of the columns of B:
//
//   S_lat[64 head, 128 tok] = Q_lat(E4M3, 64x512) . K_lat(E2M1)   16 x tcgen05.mma N=128 K=32; CTA r has tokens [64 r, 64 r + 64)
//   S_rope                  = Q_rope . K_rope                      2 x
//   P' hi, lo (E4M3, K-major, in the shared memory of the CTA whose heads they are)
//   O[64 head, 512 dim] += (P'_hi + P'_lo) . V (E2M1, MN-major)   16 x tcgen05.mma N=256 K=32; CTA r has blocks 2 j + r of 128 dims
//
// so every latent byte is read twice from L2, once by the CTA that has its token and once by the one that has its dim, as often
// as by two CTAs with a group each, and the operand reads from shared memory, which bound the other kernel (decode_sm100.cu), are a third
// less: 4 KiB an MMA of QK^T and 5 of PV (P' read once for both halves of the dims) for as many products as take 6 and 8 there.
// Measured back to back, a tile's MMAs take 576 + 1040 = 1616 clk (the rate of the tensor cores; 2111 there); in the kernel a tile takes 1780 (2300
// there).  2x131072 tokens, 128 heads, q_len 2: 105.4 -> 96.5 us, at 1.38 GHz under the 1000 W cap.
//
// An accumulator of 64 rows per CTA lies in all 128 TMEM lanes: lanes 0-63 hold the heads for the first half of the columns, lanes
// 64-127 the same heads for the second.  A softmax thread has one head and 64 tokens of every second tile: its reference and its sum are scalars, and
// four threads share a head.
//
// CTA 0 of the cluster issues all MMAs.  What it waits for it is told by both CTAs at its own barriers (remote arrivals, copies that
// report to it); what both wait for arrives as a commit with multicast.  An arrival at the other CTA that stands for work done (S read, P' stored, O
// rescaled or read out) releases at cluster scope, behind its proxy and tcgen05 fences, and every wait acquires at that scope.  The release is a
// fence of shared memory alone: 2x131072 tokens, 128 heads, q_len 2 95.9 us without it, 95.8 with it, 1x200 8.68 and 8.72; as
// mbarrier.arrive.release.cluster, which waits for stores to global memory too, 142, and passed on by the idle issue warps of CTA 1 102.6.  The roles and the merge are those of the other kernel; the two issue
// warps take no turns (with QK^T held to two tiles ahead of PV a tile took 2670 to 2800 clk).

// shared memory map of the big part; from kOffP on as in the other kernel
constexpr uint32_t kPairQkBytes = kBlocks * 64 * 128 + 64 * 64;  // 36 KiB: 64 tokens, four blocks [64][128 B] and RoPE [64][64 B]
constexpr uint32_t kPairPvBytes = 2 * kBlockBytes;               // 32 KiB: 128 tokens, two blocks [128][128 B]
constexpr uint32_t kPairOffQk = 0, kPairOffPv = 2 * kPairQkBytes;  // two stages each
constexpr uint32_t kPairOffP1 = kPairOffPv + 2 * kPairPvBytes;     // P' of odd tiles; that of even ones is at kOffP
constexpr uint32_t kPairOffTok = kPairOffP1 + 2 * kTile * 64;      // scales and their logarithms as a softmax warp reads them: [8 warps][2][64 tokens] f32
static_assert(kPairOffTok + kSoftmaxWarps * 512 <= kOffQLat && kPairOffP1 % 1024 == 0, "room between the stages and Q");
// 1 KiB of notes (row sums in the epilogue) and the references, where the other kernel has its own: the merge does not stage over them
constexpr uint32_t kPairOffNotes = kOffM, kPairOffRefs = kOffM + 4 * kGroupHeads * 4;
static_assert(kOffLinv - kOffM >= 5 * kGroupHeads * 4, "notes and references");
// barriers: QK^T stages use the first two of the other kernel's pair slots, PV stages the next two
__device__ __forceinline__ constexpr int pbar_qk_full(uint32_t s) { return bar_kv_full(int(s)); }
__device__ __forceinline__ constexpr int pbar_qk_empty(uint32_t s) { return bar_kv_empty(int(s)); }
__device__ __forceinline__ constexpr int pbar_pv_full(uint32_t s) { return bar_kv_full(2 + int(s)); }
__device__ __forceinline__ constexpr int pbar_pv_empty(uint32_t s) { return bar_kv_empty(2 + int(s)); }
// (barriers of the other kernel that have no use here)
__device__ __forceinline__ constexpr int pbar_p_full(uint32_t s) { return s ? kBarRopeFull : kBarPFull; }
constexpr int kGroupWarps = kSoftmaxWarps / 2, kGroupThreads = 32 * kGroupWarps;  // the softmax warps of one parity of tiles

constexpr uint32_t kFmtE2M1B = 5u << 10;
constexpr uint32_t kPairIdescQKRope = ptx::idesc_e4m3(128, 128, false, false);
constexpr uint32_t kPairIdescQK = ptx::idesc_e4m3(128, 128, false, false) | kFmtE2M1B;
constexpr uint32_t kPairIdescPV = ptx::idesc_e4m3(128, 256, false, true) | kFmtE2M1B;

__device__ __forceinline__ uint32_t leader_bar(uint32_t smem, int idx) { return ptx::mapa(bar_addr(smem, idx), 0); }
// Bounded wait as in the other kernel, acquiring at cluster scope.  A CTA that gives up takes its partner along, whichever role's wait it was, and
// the partner is flagged first: once a CTA is, its softmax warps run through the rest of their tiles and still report them, two of which CTA 0
// could take for one of both CTAs'; but whatever CTA 0 does after such a report, it does as a flagged CTA, which writes no rows.  (Softmax warps that
// report nothing after a failed wait instead: 1x200 8.69 -> 8.84 us, by the flag, -> 8.92, by the waits' results.)
__device__ __noinline__ bool pair_wait_slow(uint32_t smem, int idx, uint32_t parity, uint32_t tiles) {
  Misc* m = misc_of(smem);
  const uint32_t bar = bar_addr(smem, idx);
  const uint64_t polls = uint64_t(m->polls) * tiles;
#pragma unroll 1
  for (uint64_t i = 0; i < polls; ++i) {
    if (__all_sync(0xffffffffu, ptx::mbar_try_wait_cluster(bar, parity))) return true;
    if (__any_sync(0xffffffffu, m->abort)) return false;
    if (i > 4096) __nanosleep(128);
  }
  if ((threadIdx.x & 31) == 0) {
    ptx::st_cluster_u32(ptx::mapa(smem + kOffMisc + uint32_t(offsetof(Misc, abort)), ptx::cluster_ctarank() ^ 1u), 1u);
    ptx::fence_cluster();
    flag_timeout(smem, idx, parity);
  }
  __syncwarp();
  return false;
}
// tiles: how many tiles the wait may span (the budget of polls is that of one)
__device__ __forceinline__ bool pair_wait(uint32_t smem, int idx, uint32_t parity, uint32_t tiles = 1) {
  if (__all_sync(0xffffffffu, ptx::mbar_try_wait_cluster(bar_addr(smem, idx), parity))) return true;
  return __all_sync(0xffffffffu, pair_wait_slow(smem, idx, parity, tiles));
}

// ------------------------------------------------------------------------------------------
// role: TMA issue (warp 1: K of QK^T and the scales; warp 3: V of PV and the prefetch into L2)
// ------------------------------------------------------------------------------------------
// Copies go by sub-pages of at most 64 rows (a page of 128 tokens is two), so that the 64 tokens a CTA has for QK^T are whole ones.
// Stage t mod 2 of tile t is free when tile t-2 has been through it.  The scales of a tile (all 128 tokens in both CTAs) have
// a barrier of their own in each CTA and four stages.
__device__ __forceinline__ void pair_tma_role(const DecodeParams& p, uint32_t smem, uint32_t which, const CUtensorMap* map_rope,
                                              const CUtensorMap* map_lat, RoleState& st, bool starting) {
  const Segment* sg = segs_of(smem);
  const int lane = threadIdx.x & 31;
  const uint32_t rank = ptx::uniform_u32(ptx::cluster_ctarank());
  const int ppt = kTile >> p.page_shift;  // pages per tile
  const uint32_t ps = uint32_t(p.page_size);
  const int sub_shift = min(p.page_shift, 6), per_page_shift = p.page_shift - sub_shift;  // rows of a sub-page, sub-pages of a page (log2)
  const uint32_t sub = 1u << sub_shift;
  const int half_subs = 64 >> sub_shift;  // sub-pages of half a tile
  bool ok = true;
  bool dry = starting && p.pdl_wait;  // (as in the other kernel)
  uint32_t nseg = 0;
  if (!dry) {
    if (starting) start_work<kFormPair>(p, smem, which ? kWarpTMA2 : kWarpTMA, lane);
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
      const int subs = np << per_page_shift;
      // this warp's sub-pages: [from, from + count) of the tile
      const int from = which ? 0 : half_subs * int(rank);
      const int count = which ? subs : max(0, min(half_subs, subs - from));
      int pg[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) pg[i] = uniform_page(cur, at + ((from + i) >> per_page_shift));
      const uint32_t e = ptx::elect_one() && !dry;
      const uint32_t s = st.it & 1u;
      // The scales: by warp 1 behind K, but those of the very first tile by warp 3 ahead of V.  (By warp 3 in every tile they came too
      // late, behind PV.)  Stage t mod 4 is free: QK^T of t-2 has been issued, for which the softmax of t-4 had to be over.
      auto scales = [&] {
        const uint32_t sbar = bar_addr(smem, kBarScale + int(st.it & (kScaleStages - 1))), dst_sc = smem + kOffScale + (st.it & (kScaleStages - 1)) * (kTile * 4);
        if (e) ptx::mbar_arrive_expect_tx(sbar, uint32_t(np) * ps * 4u);
#pragma unroll 1
        for (int i = 0; i < np; ++i) {
          const int page = uniform_page(cur, at + i);
          ptx::bulk_load_if(e && page >= 0 ? 1u : 0u, dst_sc + uint32_t(i) * ps * 4u, p.kv_cache_sf + int64_t(page) * ps, ps * 4u, sbar);
        }
      };
      if (which && st.it == 0) scales();
      if (st.it >= 2) ok = pair_wait(smem, which ? pbar_pv_empty(s) : pbar_qk_empty(s), ((st.it >> 1) - 1) & 1);
      if (!ok) break;
      const int full = which ? pbar_pv_full(s) : pbar_qk_full(s);
      // the bytes of both CTAs (a 4-bit copy counts its packed bytes: 64 per row and block)
      if (e && rank == 0) ptx::mbar_arrive_expect_tx(bar_addr(smem, full), uint32_t(subs) * sub * (which ? 256u : 320u));
      const uint32_t bar = leader_bar(smem, full);
      // (CTA 1 may have nothing to copy for QK^T, in a tile of at most 64 tokens; CTA 0 must not run ahead of this warp's waits then)
      if (e && rank && !which) ptx::mbar_arrive_relaxed_cluster(bar);
      const uint32_t dst = smem + (which ? kPairOffPv + s * kPairPvBytes : kPairOffQk + s * kPairQkBytes);
      auto copy = [&](uint32_t issue, int page, int i) {
        const uint32_t rows = uint32_t(i) * sub;                                          // in the destination
        const int row0 = int((uint32_t(from + i) & ((1u << per_page_shift) - 1u)) * sub);  // in the page
        if (which) {
#pragma unroll
          for (uint32_t j = 0; j < 2; ++j) ptx::tma_load_3d_pair_if(issue, dst + j * kBlockBytes + rows * 128u, map_lat, bar, int(256u * j + 128u * rank), row0, page);
        } else {
          ptx::tma_load_3d_pair_if(issue, dst + kBlocks * 8192u + rows * 64u, map_rope, bar, kLatent / 2, row0, page);
#pragma unroll
          for (uint32_t j = 0; j < kBlocks; ++j) ptx::tma_load_3d_pair_if(issue, dst + j * 8192u + rows * 128u, map_lat, bar, int(128u * j), row0, page);
        }
      };
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (i < count) copy(e && pg[i] >= 0 ? 1u : 0u, pg[i], i);
#pragma unroll 1
      for (int i = 4; i < count; ++i) {
        const int page = uniform_page(cur, at + ((from + i) >> per_page_shift));
        copy(e && page >= 0 ? 1u : 0u, page, i);
      }
      if (!which && st.it > 0) scales();
      if (which) {  // the rows of the tile four ahead into L2, half of the pages by each CTA
        const int i = at + 4 * ppt + lane;
        const int in_cur = __shfl_sync(0xffffffffu, cur, i & 31), in_nxt = __shfl_sync(0xffffffffu, nxt, i & 31);
        const int page = i < 32 ? in_cur : (i < 64 ? in_nxt : -1);
        if (lane < ppt && (uint32_t(lane) & 1u) == rank && page >= 0)
          asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(static_cast<const uint8_t*>(p.kv_cache) + size_t(page) * ps * kRowBytes),
                       "r"(ps * kRowBytes) : "memory");
      }
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
      start_work<kFormPair>(p, smem, which ? kWarpTMA2 : kWarpTMA, lane);
      nseg = ptx::uniform_u32(uint32_t(misc_of(smem)->nseg));
    }
  }
  if (!ok && lane == 0) {
    // Copies that were issued but never consumed land before exit (bounded).  CTA 0 has the barriers of both; the phase after the last armed
    // one never completes and runs to its bound, which gives copies of the partner that CTA 0 has not armed time to land.
    if (rank == 0) {
      for (uint32_t k = st.it > 2u ? st.it - 2u : 0u; k <= st.it; ++k) drain_wait(smem, which ? pbar_pv_full(k & 1u) : pbar_qk_full(k & 1u), (k >> 1) & 1);
    }
    if (!which)
      for (uint32_t k = st.it > 4u ? st.it - 4u : 0u; k < st.it; ++k) drain_wait(smem, kBarScale + int(k & 3u), (k >> 2) & 1);
  }
  __syncwarp();
}

// ------------------------------------------------------------------------------------------
// roles: MMA issue (CTA 0) and Q loads (both)
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ void pair_qk_role(const DecodeParams& p, uint32_t smem, uint32_t tmem, const CUtensorMap* map_q_lat,
                                             const CUtensorMap* map_q_rope, RoleState& st) {
  const uint32_t nseg = ptx::uniform_u32(uint32_t(misc_of(smem)->nseg));
  const uint32_t rank = ptx::uniform_u32(ptx::cluster_ctarank());
  const Segment* sg = segs_of(smem);
  const Desc q_rope = make_desc(smem + kOffQRope, 16, 512, 4), q_lat = make_desc(smem + kOffQLat, 16, 1024, 2);
  const Desc k_lat = make_desc(smem + kPairOffQk, 16, 1024, 2), k_rope = make_desc(smem + kPairOffQk + kBlocks * 8192, 16, 512, 4);
  bool ok = true;
  uint32_t spans = 1;  // CTA 1 has no QK^T to issue: its wait for the end of a segment's spans all of its tiles
#pragma unroll 1
  for (uint32_t si = 0; si < nseg && ok; ++si, ++st.seg) {
    const Segment g = sg[si];
    if (st.seg >= 1 && !pair_wait(smem, kBarQEmpty, (st.seg - 1) & 1, spans)) break;
    int qpos, head0;
    group_coords(g.g, p.num_heads, qpos, head0);
    if (ptx::elect_one()) {
      if (rank == 0) ptx::mbar_arrive_expect_tx(bar_addr(smem, kBarQFull), 2 * kGroupHeads * kQDim);
      const uint32_t bar = leader_bar(smem, kBarQFull);
      ptx::tma_load_4d_pair(smem + kOffQRope, map_q_rope, bar, kLatent, head0, qpos, g.b);
#pragma unroll 1
      for (int j = 0; j < kBlocks; ++j)
        ptx::tma_load_4d_pair(smem + kOffQLat + j * kGroupHeads * 128, map_q_lat, bar, 128 * j, head0, qpos, g.b);
    }
    __syncwarp();
    const uint32_t n = ptx::uniform_u32(uint32_t(g.tile_end - g.tile_begin));
    if (rank) {
      spans = n + 1;
      continue;
    }
    ok = pair_wait(smem, kBarQFull, st.seg & 1);
#pragma unroll 1
    for (uint32_t t = 0; t < n && ok; ++t, ++st.it) {
      const uint32_t it = st.it, s = it & 1u, s64 = 64u * s;
      // S of this stage has been read by the softmax of tile it-2; K has landed
      if (it >= 2) ok = pair_wait(smem, bar_s_empty(int(s)), ((it >> 1) - 1) & 1);
      ok = ok && pair_wait(smem, pbar_qk_full(s), (it >> 1) & 1);
      if (!ok) break;
      ptx::tc_fence_after();
      const uint32_t e = ptx::elect_one();
      const uint32_t k = s * (kPairQkBytes >> 4);
#pragma unroll
      for (uint32_t ks = 0; ks < 2; ++ks) ptx::umma_f8_pair(e, tmem + kColSRope + s64, q_rope.at(2 * ks), k_rope.at(k + 2 * ks), kPairIdescQKRope, ks);
#pragma unroll
      for (uint32_t j = 0; j < kBlocks; ++j)
#pragma unroll
        for (uint32_t ks = 0; ks < 4; ++ks)
          ptx::umma_f8_pair(e, tmem + kColSLat + s64, q_lat.at(j * 512 + 2 * ks), k_lat.at(k + j * 512 + 2 * ks), kPairIdescQK, (j | ks) ? 1u : 0u);
      if (e) {
        ptx::umma_commit_pair(bar_addr(smem, bar_s_full(int(s))));
        ptx::umma_commit_pair(bar_addr(smem, pbar_qk_empty(s)));
      }
      __syncwarp();
    }
    if (ptx::elect_one()) ptx::umma_commit_pair(bar_addr(smem, kBarQEmpty));
    __syncwarp();
  }
  if (misc_of(smem)->abort && rank == 0 && (threadIdx.x & 31) == 0) {  // Q loads in flight land (one of the two waits runs to its bound)
    drain_wait(smem, kBarQFull, 0);
    drain_wait(smem, kBarQFull, 1);
  }
  __syncwarp();
}

__device__ __forceinline__ void pair_pv_role(uint32_t smem, uint32_t tmem, RoleState& st) {
  if (ptx::uniform_u32(ptx::cluster_ctarank())) return;
  const uint32_t nseg = ptx::uniform_u32(uint32_t(misc_of(smem)->nseg));
  const Segment* sg = segs_of(smem);
  const Desc v = make_desc(smem + kPairOffPv, kBlockBytes, 1024, 2);  // MN-major, 128B swizzle; 32 tokens per step = 4096 B
  const Desc pd = make_desc(smem, 16, 1024, 2);                       // K-major: 64 rows of 128 tokens, hi then lo
#pragma unroll 1
  for (uint32_t si = 0; si < nseg; ++si, ++st.seg) {
    const uint32_t n = ptx::uniform_u32(uint32_t(sg[si].tile_end - sg[si].tile_begin));
    if (st.seg >= 1 && !pair_wait(smem, kBarOFree, (st.seg - 1) & 1)) return;  // O of the previous segment has been read out
#pragma unroll 1
    for (uint32_t t = 0; t < n; ++t, ++st.it) {
      const uint32_t s = st.it & 1u;
      if (!pair_wait(smem, pbar_pv_full(s), (st.it >> 1) & 1)) return;
      if (!pair_wait(smem, pbar_p_full(s), (st.it >> 1) & 1)) return;
      ptx::tc_fence_after();
      const uint32_t e = ptx::elect_one(), keep = t ? 1u : 0u, a = s * (kPairPvBytes >> 4), pa = (s ? kPairOffP1 : kOffP) >> 4;
#pragma unroll
      for (uint32_t ks = 0; ks < 4; ++ks)
#pragma unroll
        for (uint32_t w = 0; w < 2; ++w) {  // hi, lo: read once for both blocks of 256 dims
          const uint64_t ad = pd.at(pa + 512 * w + 2 * ks);
          ptx::umma_f8_pair_a_fill(e, tmem + kColO, ad, v.at(a + 256 * ks), kPairIdescPV, (ks | w) ? 1u : keep);
          ptx::umma_f8_pair_a_lastuse(e, tmem + kColO + 128u, ad, v.at(a + (kBlockBytes >> 4) + 256 * ks), kPairIdescPV, (ks | w) ? 1u : keep);
        }
      if (e) ptx::umma_commit_pair(bar_addr(smem, pbar_pv_empty(s)));  // (V's stage, this tile's P, and O)
      __syncwarp();
    }
  }
}

// ------------------------------------------------------------------------------------------
// role: softmax / rescale / epilogue (warps 4..11; TMEM lane = head, twice)
// ------------------------------------------------------------------------------------------
// Two groups of four warps, one for the even tiles and one for the odd: a tile's chain of waits (S, the vote, P's buffer, fences) is
// longer than a tile of the tensor pipe, and with all warps on the same tile nothing else runs meanwhile (2400 clk a tile, now
// 1780).  What passes from tile to tile is the heads' references alone: the scores are made without them, and a group takes
// them over when the other one has moved them (or not), by a named barrier each way.  A group's row sums are relative to the
// reference that it last saw.
// Rows of the accumulators, scaled, to memory: head h of the CTA at dst + h * 512 elements.  A warp's 32 lanes are 32 heads, so a direct
// store would touch 32 rows; the rows go through 2 KiB of the P buffer (idle between two segments) that the warp has to itself, 64 bytes of
// each at a time, and leave in runs of that length: whole sectors, and no barrier but the warp's.  16-byte chunks are swizzled by
// the head, so that neither side has bank conflicts.
constexpr int kRowsF16 = 100;  // partials
template <int kDtype>
__device__ __noinline__ void write_rows(uint32_t smem, uint32_t tmem_lane, int tid, char* dst, int heads_here) {
  constexpr uint32_t esz = kDtype == MLA_FP4_OUT_F32 ? 4u : (kDtype == MLA_FP4_OUT_E4M3 ? 1u : 2u);
  constexpr uint32_t kCols = 64u / esz;         // dims of a thread and round: 64 bytes
  constexpr uint32_t kRounds = 64u / kCols;     // per block of 256 dims
  const uint32_t lane = tid & 31, quarter = (tid >> 5) & 3, half = tid >> 7, upper = quarter >> 1, head0 = 32u * (quarter & 1u);
  const float f = lds_f32(smem + kOffLinv + 4 * (head0 + lane));
  const uint32_t buf = smem + kOffP + uint32_t(tid >> 5) * 2048u, st = buf + lane * 64u, st_sw = (lane >> 1) & 3u;
  const uint32_t row = lane >> 2, c = lane & 3u;  // reading: chunk c of heads row + 8 k
  const uint32_t ld_at = buf + row * 64u + ((c ^ ((row >> 1) & 3u)) << 4);
  char* d = dst + size_t(head0 + row) * (kLatent * esz) + upper * (128u * esz) + half * 64u + c * 16u;
#pragma unroll 1
  for (uint32_t r = 0; r < 2 * kRounds; ++r) {
    const uint32_t j = r / kRounds, cc = r % kRounds;
    uint32_t o[kCols / 16][16];
#pragma unroll
    for (uint32_t k = 0; k < kCols / 16; ++k) ptx::tmem_ld16(tmem_lane + kColO + 128u * j + kCols * (2u * cc + half) + 16u * k, o[k]);
    ptx::tmem_wait_ld();
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {  // 16 bytes
      uint32_t w[4];
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i) {
        constexpr uint32_t per = 4u / esz;
        const uint32_t e0 = per * (4u * q + i);
        float x[4];
#pragma unroll
        for (uint32_t u = 0; u < per; ++u) x[u] = __uint_as_float(o[(e0 + u) >> 4][(e0 + u) & 15u]) * f;
        if (kDtype == MLA_FP4_OUT_F32) {
          w[i] = __float_as_uint(x[0]);
        } else if (kDtype == MLA_FP4_OUT_BF16) {
          const __nv_bfloat162 t = __floats2bfloat162_rn(x[0], x[1]);
          w[i] = *reinterpret_cast<const uint32_t*>(&t);
        } else if (kDtype == kRowsF16) {
          const __half2 t = __floats2half2_rn(x[0], x[1]);
          w[i] = *reinterpret_cast<const uint32_t*>(&t);
        } else {
          w[i] = __nv_cvt_float2_to_fp8x2(make_float2(x[0], x[1]), __NV_SATFINITE, __NV_E4M3) |
                 (uint32_t(__nv_cvt_float2_to_fp8x2(make_float2(x[2], x[3]), __NV_SATFINITE, __NV_E4M3)) << 16);
        }
      }
      asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(st + ((q ^ st_sw) << 4)), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
    }
    __syncwarp();
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k)
      if (int(head0 + row + 8u * k) < heads_here) *reinterpret_cast<uint4*>(d + size_t(8 * k) * (kLatent * esz) + j * (256u * esz) + cc * 128u) = lds_u32x4(ld_at + k * 512u);
    __syncwarp();  // before the next round overwrites the buffer
  }
}

// O *= f, the factor of the thread's head.
__device__ __noinline__ void pair_rescale(uint32_t tmem_lane, float f) {
#pragma unroll 1
  for (uint32_t k = 0; k < 8; ++k) {
    uint32_t o[2][16];
    const uint32_t ta = tmem_lane + kColO + 32u * k;
    ptx::tmem_ld16(ta, o[0]);
    ptx::tmem_ld16(ta + 16u, o[1]);
    ptx::tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      o[0][i] = __float_as_uint(__uint_as_float(o[0][i]) * f);
      o[1][i] = __float_as_uint(__uint_as_float(o[1][i]) * f);
    }
    ptx::tmem_st16(ta, o[0]);
    ptx::tmem_st16(ta + 16u, o[1]);
  }
  ptx::tmem_wait_st();
}

template <bool kSoftCap>
__device__ __forceinline__ void pair_softmax_role(const DecodeParams& p, uint32_t smem, uint32_t tmem, int tid, RoleState& st) {
  Misc* misc = misc_of(smem);
  const int nseg = misc->nseg;
  const Segment* sg = segs_of(smem);
  const int warp = tid >> 5, lane = tid & 31;
  const int quarter = warp & 3, grp = warp >> 2;
  const int upper = quarter >> 1;  // which 64 tokens of a tile
  const int head = 32 * (quarter & 1) + lane;
  const uint32_t tmem_lane = tmem + ((uint32_t(quarter) * 32u) << 16);
  const float cscale = p.softmax_scale * kLog2e;
  const uint64_t cs2 = pack2(cscale, cscale);
  const float cap = kSoftCap ? p.soft_cap : 0.f;
  const uint64_t cap2 = pack2(cap, cap), rcap2 = pack2(kSoftCap ? 1.f / cap : 0.f, kSoftCap ? 1.f / cap : 0.f);
  const uint32_t tok = smem + kPairOffTok + 512u * uint32_t(warp);  // this warp's scales; + 256: their logarithms
  // this thread's 64 bytes of P' hi (and of lo, 8 KiB on): row of 128 tokens, four 16-byte chunks, 128-byte swizzle
  const uint32_t p_row = smem + (grp ? kPairOffP1 : kOffP) + uint32_t(head) * 128u, p_sw = uint32_t(head) & 7u;
  const uint32_t note = smem + kPairOffNotes + 4u * uint32_t(128 * grp + head);  // + 256: the other half's
  const uint32_t ref = smem + kPairOffRefs + 4u * uint32_t(head);
  const uint32_t bar_s = leader_bar(smem, bar_s_empty(grp)), bar_p = leader_bar(smem, pbar_p_full(uint32_t(grp))), bar_o = leader_bar(smem, kBarOFree);
  bool pending = false;
  uint32_t r = 0;  // tiles of this round before this one

#pragma unroll 1
  for (int si = 0; si < nseg; ++si, ++st.seg) {
    const Segment g = sg[si];
    float negm = 0.f;  // minus the head's reference as this group last saw it
    bool any = false;  // ... in this segment
    uint64_t l2 = 0ull;
    float sc_max = 0.f;
    const uint32_t it0 = st.it;
#pragma unroll 1
    for (int tt = g.tile_begin + ((int(it0) ^ grp) & 1); tt < g.tile_end; tt += 2) {
      const uint32_t it = it0 + uint32_t(tt - g.tile_begin), half_it = it >> 1;
      const bool first = tt == g.tile_begin;
      (void)pair_wait(smem, kBarScale + int(it & (kScaleStages - 1)), (it / kScaleStages) & 1);
      const int live = g.seq_len - (tt * kTile + 64 * upper);  // tokens of this warp's 64 that exist (any number)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float sc = lds_f32(smem + kOffScale + 4 * ((it & (kScaleStages - 1)) * kTile + 64 * upper + 32 * i + lane));
        sc = lane + 32 * i < live ? sc : 0.f;
        sc_max = fmaxf(sc_max, fabsf(sc));
        sts_f32(tok + 128 * i + 4 * lane, sc);
        sts_f32(tok + 256 + 128 * i + 4 * lane, __log2f(fmaxf(fabsf(sc), 8.67361738e-19f)));  // floor 2^-60
      }
      __syncwarp();
      (void)pair_wait(smem, bar_s_full(grp), half_it & 1);
      ptx::tc_fence_after();
      // The scores, and the largest x c + log2|scale|.
      uint64_t x2[2 * kPairs];
      float mx = -INFINITY;
      {
        const uint32_t t_lat = tmem_lane + kColSLat + 64u * uint32_t(grp), t_rope = tmem_lane + kColSRope + 64u * uint32_t(grp);
        uint32_t a[2][16], b[2][16];
        ptx::tmem_ld16(t_lat, a[0]);
        ptx::tmem_ld16(t_rope, b[0]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          ptx::tmem_wait_ld();
          if (c < 3) {
            ptx::tmem_ld16(t_lat + 16 * (c + 1), a[(c + 1) & 1]);
            ptx::tmem_ld16(t_rope + 16 * (c + 1), b[(c + 1) & 1]);
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {  // four tokens per shared load
            uint64_t sc2[2], lg2[2];
            lds_pairs(tok + 64 * c + 16 * q, sc2[0], sc2[1]);
            lds_pairs(tok + 256 + 64 * c + 16 * q, lg2[0], lg2[1]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int i = 4 * q + 2 * h;
              uint64_t x = fma2(pack2u(a[c & 1][i], a[c & 1][i + 1]), sc2[h], pack2u(b[c & 1][i], b[c & 1][i + 1]));
              if (kSoftCap) {
                float x0, x1;
                unpack2(mul2(x, rcap2), x0, x1);
                x = mul2(pack2(tanh_approx(x0), tanh_approx(x1)), cap2);
              }
              x2[8 * c + 2 * q + h] = x;
              float z0, z1;
              unpack2(fma2(x, cs2, lg2[h]), z0, z1);
              mx = max3(mx, z0, z1);
            }
          }
        }
      }
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive_release_cluster(bar_s);
      if (live < 64) {  // tokens beyond seq_len have no say
        mx = -INFINITY;
#pragma unroll
        for (int q = 0; q < 2 * kPairs; ++q) {
          float z0, z1;
          uint64_t lg2;
          asm volatile("ld.shared.b64 %0, [%1];" : "=l"(lg2) : "r"(tok + 256 + 8 * q) : "memory");
          unpack2(fma2(x2[q], cs2, lg2), z0, z1);
          if (2 * q < live) mx = fmaxf(mx, z0);
          if (2 * q + 1 < live) mx = fmaxf(mx, z1);
        }
      }
      // The references as the tile before left them.  When a score beats its reference by more than the lazy threshold, all heads of the
      // group move to the tops of this tile (those whose tops are above their references; in a segment's first tile all of them).
      if (r + uint32_t(tt - g.tile_begin) > 0) ptx::bar_sync(10 + (grp ^ 1), kSoftmaxThreads);
      const float old = first ? 0.f : lds_f32(ref);
      sts_f32(note + 256 * upper, mx + old);
      const bool beaten = first || mx + old > kPShift + kLazyThreshold;
      const bool moved = ptx::bar_or(grp ? 7 : 4, kGroupThreads, beaten);
      float now = old, f = 1.f;
      if (moved) {
        const float above = fmaxf(lds_f32(note), lds_f32(note + 256)) - kPShift;
        const float d = first ? above : fmaxf(above, 0.f);
        now = old - d;
        f = ptx::ex2(-d);
        if (!upper) sts_f32(ref, now);
      }
      if (!(si == nseg - 1 && tt == g.tile_end - 1)) asm volatile("bar.arrive %0, %1;" ::"r"(10 + grp), "n"(kSoftmaxThreads) : "memory");
      if (any && now != negm) {
        const float fl = ptx::ex2(now - negm);
        l2 = mul2(l2, pack2(fl, fl));
      }
      negm = now;
      any = true;
      const uint64_t nm2 = pack2(now, now);
#pragma unroll
      for (int q = 0; q < 2 * kPairs; ++q) {
        float y0, y1;
        unpack2(fma2(x2[q], cs2, nm2), y0, y1);
        x2[q] = pack2(ptx::ex2(y0), ptx::ex2(y1));
      }
      if (live < 64) {  // weight exactly zero, whatever their rows hold
#pragma unroll
        for (int q = 0; q < 2 * kPairs; ++q) {
          float y0, y1;
          unpack2(x2[q], y0, y1);
          x2[q] = pack2(2 * q < live ? y0 : 0.f, 2 * q + 1 < live ? y1 : 0.f);
        }
      }
      uint32_t hi[16], lo[16];
      uint64_t t2[2] = {0ull, 0ull};  // this tile's sum
#pragma unroll
      for (int q = 0; q < kPairs; ++q) {
        uint64_t sc2[2];
        lds_pairs(tok + 16 * q, sc2[0], sc2[1]);
        uint32_t l0, l1;
        const uint32_t h0 = split_e4m3x2(mul2(x2[2 * q], sc2[0]), l0), h1 = split_e4m3x2(mul2(x2[2 * q + 1], sc2[1]), l1);
        hi[q] = h0 | (h1 << 16);
        lo[q] = l0 | (l1 << 16);
        t2[0] = add2(t2[0], x2[2 * q]);
        t2[1] = add2(t2[1], x2[2 * q + 1]);
      }
      l2 = add2(l2, add2(t2[0], t2[1]));
      if (it >= 2) (void)pair_wait(smem, pbar_pv_empty(uint32_t(grp)), (half_it - 1) & 1);  // this group's P buffer is free
      if (moved && !first && __any_sync(0xffffffffu, f != 1.f)) {  // O holds earlier tiles of the segment, all of them now
        (void)pair_wait(smem, pbar_pv_empty(uint32_t(grp ^ 1)), ((it - 1) >> 1) & 1);
        ptx::tc_fence_after();
        pair_rescale(tmem_lane, f);
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint32_t at = p_row + (((4u * uint32_t(upper) + uint32_t(c)) ^ p_sw) << 4);
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(hi[4 * c]), "r"(hi[4 * c + 1]), "r"(hi[4 * c + 2]), "r"(hi[4 * c + 3]) : "memory");
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at + kTile * 64), "r"(lo[4 * c]), "r"(lo[4 * c + 1]), "r"(lo[4 * c + 2]), "r"(lo[4 * c + 3]) : "memory");
      }
      ptx::fence_proxy_async_smem();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive_release_cluster(bar_p);
    }
    st.it = it0 + uint32_t(g.tile_end - g.tile_begin);
    r += uint32_t(g.tile_end - g.tile_begin);

    // ---- segment epilogue
    ptx::bar_sync(1, kSoftmaxThreads);  // nobody reads notes any more, and the references are final
    const float last = lds_f32(ref);
    {
      float l0, l1;
      unpack2(l2, l0, l1);
      sts_f32(note + 256 * upper, any ? (l0 + l1) * ptx::ex2(last - negm) : 0.f);
      const float sc_warp = ptx::redux_max_f32(sc_max);
      if (lane == 0) sts_f32(smem + kOffScMax + 4 * warp, sc_warp);
    }
    ptx::bar_sync(1, kSoftmaxThreads);
    if (tid < kGroupHeads) {  // (head == tid)
      const uint32_t n0 = smem + kPairOffNotes + 4u * uint32_t(tid);
      const float L = (lds_f32(n0) + lds_f32(n0 + 256)) + (lds_f32(n0 + 512) + lds_f32(n0 + 768));
      float m = -last;
      float Ls = L, fo = p.output_scale;
      if (p.sink && g.tile_begin == 0) {  // (as in the other kernel)
        int qpos, head0;
        group_coords(g.g, p.num_heads, qpos, head0);
        if (head0 + tid < p.num_heads) {
          const float sk = __ldg(p.sink + head0 + tid) * kLog2e;
          const float mm = fmaxf(m, sk);
          const float fs = ptx::ex2(m - mm);
          fo *= fs;
          Ls = L * fs + ptx::ex2(sk - mm);
          m = mm;
        }
      }
      float slot_scale_v = 1.f;
      if (g.slot >= 0) {
        const float4 a = lds_f32x4(smem + kOffScMax), b = lds_f32x4(smem + kOffScMax + 16);
        const float sc_all = fmaxf(fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w)), fmaxf(fmaxf(b.x, b.y), fmaxf(b.z, b.w)));
        slot_scale_v = slot_scale_for(6.f * sc_all * fabsf(p.output_scale));
        fo *= __frcp_rn(slot_scale_v);
      }
      const float lse = __log2f(Ls) + m;
      sts_f32(smem + kOffLinv + 4 * tid, __fdividef(fo, Ls));
      sts_f32(smem + kOffLse + 4 * tid, lse);
      if (g.slot >= 0) {
        slot_lse(p.workspace, g.slot)[tid] = lse;
        if (tid == 0) slot_scale(p.workspace, g.slot)[0] = slot_scale_v;
        if (si == nseg - 1 && !misc->more) asm volatile("bar.arrive 6, %0;" ::"n"(kGroupHeads + 32) : "memory");
      }
    }
    (void)pair_wait(smem, pbar_pv_empty((st.it - 1) & 1), ((st.it - 1) >> 1) & 1);  // the PV of the last tile
    ptx::tc_fence_after();
    if (!ptx::bar_or(1, kSoftmaxThreads, misc->abort != 0)) {
      if (g.slot >= 0) {
        write_rows<kRowsF16>(smem, tmem_lane, tid, reinterpret_cast<char*>(slot_o(p.workspace, g.slot)), kGroupHeads);
      } else {
        int qpos, head0;
        group_coords(g.g, p.num_heads, qpos, head0);
        const int heads_here = min(kGroupHeads, p.num_heads - head0);
        const size_t row0 = (size_t(g.b) * p.q_len + qpos) * p.num_heads + head0;
        char* dst = static_cast<char*>(p.out) + row0 * kLatent * uint32_t(out_elem_bytes(p.out_dtype));
        if (p.out_dtype == MLA_FP4_OUT_BF16) write_rows<MLA_FP4_OUT_BF16>(smem, tmem_lane, tid, dst, heads_here);
        else if (p.out_dtype == MLA_FP4_OUT_F32) write_rows<MLA_FP4_OUT_F32>(smem, tmem_lane, tid, dst, heads_here);
        else write_rows<MLA_FP4_OUT_E4M3>(smem, tmem_lane, tid, dst, heads_here);
        if (p.lse && tid < heads_here) p.lse[row0 + tid] = lds_f32(smem + kOffLse + 4 * tid);
      }
    }
    ptx::tc_fence_before();
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive_release_cluster(bar_o);
    if (si + 1 < nseg) ptx::bar_sync(1, kSoftmaxThreads);  // the rows of all warps have left the P buffer
    pending |= g.slot >= 0;
  }
  if (pending) {
    if (!misc->more) {  // (publish)
      asm volatile("bar.arrive 9, %0;" ::"n"(kSoftmaxThreads + 32) : "memory");
    } else {
      ptx::bar_sync(1, kSoftmaxThreads);
      if (tid == 0) {
        const int slot = slot_of(misc->cta, true);
        st_release(slot_lse_flag(p.workspace, slot), misc->gen);
        st_release(slot_flag(p.workspace, slot), misc->gen);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------
// kernel
// ------------------------------------------------------------------------------------------
template <bool kSoftCap>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
mla_fp4_decode_pair_kernel(const __grid_constant__ DecodeParams p, const __grid_constant__ CUtensorMap map_q_lat,
                           const __grid_constant__ CUtensorMap map_q_rope, const __grid_constant__ CUtensorMap map_rope,
                           const __grid_constant__ CUtensorMap map_lat) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  Misc* misc = misc_of(smem);
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = int(ptx::uniform_u32(uint32_t(tid >> 5)));

  if (warp == kWarpQK) {
    ptx::tmem_alloc_pair(smem + kOffMisc + offsetof(Misc, tmem_base), 512);
    ptx::tmem_relinquish_pair();
  } else if (warp == kWarpPV) {
    if (lane < kNumBars) {  // lane i: barrier i
      uint32_t count = 1;
      if (lane == kBarOFree) count = 2 * kSoftmaxWarps;  // (of both CTAs)
      if (lane == pbar_p_full(0) || lane == pbar_p_full(1) || lane == bar_s_empty(0) || lane == bar_s_empty(1)) count = 2 * kGroupWarps;
      if (lane == kBarDrain || lane == pbar_qk_full(0) || lane == pbar_qk_full(1)) count = 2;  // the two MMA warps of CTA 0; a copy warp of each CTA
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
    __syncwarp();
  } else if (warp == kWarpTMA2 && lane == 0) {
    ptx::prefetch_tensormap(&map_q_lat);
    ptx::prefetch_tensormap(&map_q_rope);
    ptx::prefetch_tensormap(&map_rope);
    ptx::prefetch_tensormap(&map_lat);
  }
  __syncwarp();
  ptx::tc_fence_before();
  ptx::cluster_arrive();  // (from here on the partner may arrive at this CTA's barriers)
  if (warp == kWarpPlan && p.pdl_wait) {
    stage_segments<kFormPair>(p, smem, lane, true, false);
    ptx::fence_proxy_async_smem();
    __threadfence_block();
    asm volatile("bar.arrive 8, 64;" ::: "memory");
  }
  ptx::cluster_wait();
  RoleState st{};
  if (warp != kWarpTMA && warp != kWarpTMA2) start_work<kFormPair>(p, smem, warp, lane);
  ptx::tc_fence_after();
  const uint32_t tmem = ptx::uniform_u32(misc->tmem_base);
  bool first_round = true;
  int finished = -1;
#pragma unroll 1
  for (;;) {
    if (warp >= kWarpSoftmax0) {
      pair_softmax_role<kSoftCap>(p, smem, tmem, tid - 32 * kWarpSoftmax0, st);
      if (!misc->more && misc->n_slots > 0) {
        ptx::bar_sync(5, kThreads - 32);
        if (misc->mode == kMergeShared) merge_weights(p, smem, tid - 32 * kWarpSoftmax0, true, misc->rank == 0);
      }
    } else if (warp == kWarpQK) {
      pair_qk_role(p, smem, tmem, &map_q_lat, &map_q_rope, st);
    } else if (warp == kWarpPV) {
      if (first_round) {
        if (lane == 0) {
          atomicAdd(ws_started(p.workspace), 1);
          misc->gen = ld_acquire(ws_generation(p.workspace)) + 1;
        }
        plan_merge<true>(smem, 0, lane);
        zero_empty_requests(p, lane);
      }
      pair_pv_role(smem, tmem, st);
    } else {
      pair_tma_role(p, smem, warp == kWarpTMA2 ? 1u : 0u, &map_rope, &map_lat, st, first_round);
    }
    const int more = misc->more;
    if (!more && warp < kWarpSoftmax0) {
      // Last round: as in the other kernel; the commits of CTA 0's MMA warps arrive in both CTAs.
      if (warp == kWarpPV && !(blockIdx.x & 1) && ptx::elect_one()) ptx::umma_commit_pair(bar_addr(smem, kBarDrain));
      __syncwarp();
      if (warp == kWarpQK) {
        publish<true>(p, smem, lane);
      } else {
        if (lane == 0) drain_wait<true>(smem, kBarDrain, 0);
        __syncwarp();
        if (warp == kWarpPV && lane == 0) {
          if (misc->merge[0].vtiles | misc->merge[1].vtiles) misc->mode = merge_mode(p);
        }
        ptx::bar_sync(3, 32 * kFetchWarps);
        if (misc->n_slots > 0) {
          __threadfence_block();
          asm volatile("bar.arrive 5, %0;" ::"n"(kThreads - 32) : "memory");
          if (misc->mode == kMergeShared) tail_fetch(p, smem, warp - kWarpTMA, lane, true);
        }
        if (warp == kWarpPV && lane == 0) finished = atomicAdd(ws_finished(p.workspace), 1);
      }
    }
    __syncthreads();
    if (!more) break;
    first_round = false;
    if (warp == kWarpTMA) {
      stage_segments<kFormPair>(p, smem, lane, false, false);
      ptx::fence_proxy_async_smem();
    }
    __syncthreads();
  }
  // Nothing of the partner's is needed any more, and TMEM has been read; its arrivals here may still be under way.
  ptx::tc_fence_before();
  ptx::cluster_arrive();
  if (misc->merge[0].vtiles | misc->merge[1].vtiles) {
    if (misc->mode == kMergeLast) merge_as_last<true>(p, smem, tid);
    else if (misc->n_slots > 0) tail_merge_of<true>(p, smem, tid, 0);
  }
  if (finished == int(gridDim.x) - 1) {
    *ws_finished(p.workspace) = 0;
    *ws_started(p.workspace) = 0;
    *ws_mode(p.workspace) = 0;
    st_release(ws_generation(p.workspace), misc->gen);
  }
  __syncwarp();
  ptx::cluster_wait();
  ptx::tc_fence_after();
  if (warp == kWarpQK) ptx::tmem_dealloc_pair(tmem, 512);
}
