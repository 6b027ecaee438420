// Persistent mixed-precision grouped GEMM for sm_100a on CTA PAIRS (tcgen05 cta_group::2): the default of every launch of
// two CTAs or more.
//
// Same contract and operand roles as gg_swap_kernel.cu (one launch walks a device-side list of problems
// C[M,N] = A[M,K] x B[N,K]^T, each with its own scheme; reference: mxmoe/kernels/compose_kernel.py:150-295,
// cta_gemm.cuh:7-107, :291-421, :423-608): the MMA computes C^T, weights = M side, tokens = N side, 4-bit weights are
// converted straight into tensor memory.  A cluster of two CTAs works on 256 output channels x one token tile: each CTA
// loads (and converts) its own 128 weight rows and HALF of the token tile by its own plain TMA loads (no multicast), the
// leader (cluster rank 0) issues one M = 256 MMA per 32 bytes of K for both, each CTA drains its own 128 channels.
//
// What bounds it.  Single CTAs with tiles of 128 x 176 move 38 KB from L2 into shared memory per 352 tensor cycles
// (8- and 16-bit operands) and read as much back: both the L2 -> SM path (64 B/clk) and shared memory saturate and a
// stage takes 620 cycles.  A pair moves 32 KB per 512 cycles (256 tokens) or 20-28 KB per 384 (192 tokens), so the tensor
// pipe is the limit for 8- and 16-bit operands: 516-529 cycles per stage of 512.  The chip then runs at its power
// limit (1000 W at 1.2-1.3 GHz): fp16 1215 and int8 2413 TFLOP/s held for seconds, cuBLAS on the same operands 1211 and
// 2322.  8 x [4096, 2816, 2048], short runs, us, single CTAs -> pairs: w8a8 172 -> 132, fp16 325 -> 270, w4a4 162 -> 143
// (packed activations 310 -> 243), w4a16 389 -> 334; 8 x [4096, 2048, 1408]: 109 -> 75, 172 -> 140, 124 -> 88 (184 -> 137),
// 213 -> 175.
//
// Tiles.  Without 4-bit weights 256 tokens (both accumulators fill tensor memory), ring of six 32 KiB stages.  With them
// 192 tokens: two accumulators of 192 columns leave room for four A slots of 32 columns (128 channels x 128 bytes of K
// per CTA), ring of seven 28 KiB stages; A slots are a ring of their own, so that a launch can have more loads in flight
// than it has slots.  Launches whose problems all have few rows (a decode batch) take 32 tokens and ten 20 KiB stages: what
// counts there is how many weight bytes are in flight (16 tokens of the mixtral shape 215.7 us on single CTAs, 207.7 here).
//
// One CTA (768 threads; 384 without 4-bit weights), one role per warp:
//   0       producer of the weights;  2  producer of the activations (one thread doing both was the limit of the ring)
//   1       MMA issuer (leader only); with packed activations warps 1 and 3 of the second CTA forward its converters' arrivals
//   4-11    epilogue, two warps per TMEM lane quarter, alternating 32-token chunks; scales and problem fields are loaded
//           one tile ahead (loading them per tile cost w8a8 8 x [4096, 2048, 1408] 20 us of 94)
//   12-23   converters in three groups of four warps that take converted K blocks in turn (two groups: packed w4a4 and
//           w4a16 5-8 % slower; four groups have 72 registers per thread and spill more than the 2-5 words of
//           the long-tile instances at 80, which costs more than they bring)
//
// Barriers.  full[s] (leader): everything the MMAs of stage s read is in place in both CTAs - the loads of both (the
// cta_group::2 form of a load completes on the leader's barrier) and, for converted weights, eight arrivals of converter
// warps, without release semantics: their payload is in tensor memory.  Packed activations are expanded into shared
// memory, which a thread of the leader makes MMAs read: there the leader's converters release to full[s] at CTA scope,
// those of the second CTA to their own xdone[s], and two otherwise idle warps pass that on to full[s] with a release at
// cluster scope, which the issuer acquires.  That release takes some 2 000 cycles, now in the latency of a turn of the ring;
// 8 x [4096, 2816, 2048], 8 x [4096, 2048, 1408], 60 x [24, 2816, 2048], us: no release at cluster scope (not sound)
// 169 / 101 / 49, by the converters in their own chain 271 / 148 / 85, by two forwarders, one release for all stages that
// are ready, 243 / 137 / 67, by one 272 / 151 / 69, by two with a release per stage 242 / 140 / 85.
// empty[s]: the MMAs of the stage have completed, committed to both CTAs; nothing else is needed, since they read what the
// converters wrote from what the stage held.  wfull[n % kWBars]: this CTA's packed weights of converted K block n have
// landed.  Every wait is bounded; a role whose wait runs out reports, raises the CTA's abort flag and leaves its loop, the
// others follow by the flag or by their own limit.
#include "gg_tile.cuh"
#include "launch.cuh"

namespace mxb {

using namespace ptx;
using namespace ggc;

namespace {

constexpr int kDuoRecs     = 256;   // tiles per pair kept in the table of tile records
constexpr int kFirstEpi    = 4;
constexpr int kFirstCvt    = 12;
constexpr int kCvtGroups   = 3;     // groups of four warps (one per TMEM lane quarter)

// kMode 0: no 4-bit operand in the launch.  1: 4-bit weights.  2: packed 4-bit activations as well.
// kShort: token tiles of 32 rows (decode batches), ring of ten 20 KiB stages.
template <int kMode, bool kShort>
struct DuoGeo {
  static constexpr int kTok        = kShort ? kDuoTokShort : (kMode ? kDuoTokCvt : kDuoTok);   // tokens per tile (tcgen05 N)
  static constexpr int kHalf       = kTok / 2;               // token rows one CTA needs
  static constexpr int kXRows      = kHalf < kXBoxSmall ? kXBoxSmall : kHalf;   // token rows one CTA loads
  static constexpr int kStages     = kShort ? 10 : (kMode ? 7 : 6);
  static constexpr int kXSlotBytes = kXRows * kRowBytes;
  static constexpr int kStageBytes = kWSlotBytes + kXSlotBytes;
  static constexpr int kRingBytes  = kStages * kStageBytes;
  // A operands of converted K blocks in tensor memory.  Short tiles leave room for one per stage: a slot is then free
  // whenever its stage is.
  static constexpr int kASlots     = kMode ? (kShort ? kStages : 4) : 1;
  // Barriers of converted K blocks: one per block in turn, not per stage.  A wait by parity is good only for a waiter that saw
  // the barrier's previous phase end, and loads land out of order: a barrier must belong to one converter group for good.
  static constexpr int kWBars      = (kStages + kCvtGroups - 1) / kCvtGroups * kCvtGroups;
  static constexpr int kXBars      = kMode == 2 ? kStages : 1;   // barriers of expanded activations
  static constexpr uint32_t kACol0 = 2 * kTok;
  static constexpr int kThreads    = (kFirstCvt + (kMode ? kCvtGroups * kCvtGroup : 0)) * 32;
  static constexpr int kEpiChunks  = (kTok + 63) / 64;       // 32-token chunks of a tile one epilogue warp takes
  static constexpr int kEpiBufs    = kShort ? kEpiWarps / 2 : kEpiWarps;   // (short tiles: one chunk, the second group stores nothing)
  static_assert(2 * kTok + (kMode ? kASlots * (int)kASlotCols : 0) <= 512, "tensor memory budget");
  static_assert(kXRows % 32 == 0 && kStageBytes % 1024 == 0, "token boxes of 32 rows, swizzle atoms");
};

template <typename G>
struct CtrlD {
  uint64_t full[G::kStages];     // leader: all operands of the stage are in place in both CTAs (loads have landed, weights are converted)
  uint64_t wfull[G::kWBars];     // this CTA's packed weights (and packed activations) of converted K block n have landed: barrier n % kWBars
  uint64_t empty[G::kStages];    // the MMAs of the stage have completed (committed to both CTAs)
  uint64_t tfull[2];             // accumulator b is complete (committed to both CTAs)
  uint64_t tempty[2];            // leader: both CTAs have drained accumulator b
  unsigned long long timeout_ns; // limit of every wait
  long long t0;                  // clock when the first CTA began (PROF_TOTAL)
  uint32_t tmem_base;
  int abort_flag;
  int pad[4];                    // outcome of a group's wait for an accumulator (kExt)
  int pad2[2];
  Sched sched;
  alignas(16) __half sa_stage[kEpiWarps][G::kEpiChunks * 32];   // per epilogue warp: per-token scales of its chunks
  alignas(16) TileRec recs[kDuoRecs];
  uint64_t xdone[G::kXBars];     // second CTA: its converters have expanded the packed activations of the stage
};

template <typename G>
constexpr int smem_bytes_duo() { return 1024 + G::kRingBytes + G::kEpiBufs * kEpiStageS + (int)sizeof(CtrlD<G>); }
static_assert(smem_bytes_duo<DuoGeo<0, false>>() <= 232448 && smem_bytes_duo<DuoGeo<1, false>>() <= 232448 &&
                  smem_bytes_duo<DuoGeo<1, true>>() <= 232448,
              "227 KiB per CTA");

template <typename G>
constexpr uint32_t kCtrlOff = G::kRingBytes + G::kEpiBufs * kEpiStageS;   // CtrlD behind the ring and the transpose buffers
#define MXB_CTRL(field) (kCtrlOff<G> + (uint32_t)offsetof(CtrlD<G>, field))

// Bounded wait.  Everything it needs besides the barrier is in shared memory at a fixed distance from `sb`, so that a
// role carries one register for all its waits.  kAcquire: see mbar_try_wait_cluster.
template <typename G, bool kAcquire = false>
__device__ __forceinline__ bool bar_wait(uint32_t sb, uint32_t bar, uint32_t parity) {
  if (kAcquire ? mbar_try_wait_cluster(bar, parity) : mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  for (uint32_t it = 1;; ++it) {
    if (kAcquire ? mbar_try_wait_cluster(bar, parity) : mbar_try_wait(bar, parity)) return true;
    if ((it & 63u) == 0) {
      if (lds32(sb + MXB_CTRL(abort_flag))) return false;
      if ((long long)(globaltimer_ns() - t0) > (long long)lds64(sb + MXB_CTRL(timeout_ns))) {
        sts32(sb + MXB_CTRL(abort_flag), 1u);
        return false;
      }
    }
  }
}
// The whole warp polls (one instruction for the 32 lanes).
template <typename G, bool kAcquire = false>
__device__ __forceinline__ bool wwait(uint32_t sb, uint32_t bar, uint32_t parity) {
  return __all_sync(0xffffffffu, bar_wait<G, kAcquire>(sb, bar, parity));
}

// tcgen05 N of a tile: the M = 256 form takes multiples of 32
__device__ __forceinline__ int pair_tokens(int ntok) { return (ntok + 31) & ~31; }

// position in the ring of stages, and in the ring of A slots
template <typename G>
struct MmaPos {
  int stage, a;
  uint32_t phase;
  bool ready;      // stage `stage` was seen complete already
};

// kAcquire: converters of both CTAs wrote an operand of the tile to shared memory (packed activations)
template <int kV, bool kAcquire, typename G>
__device__ __forceinline__ bool mma_tile(int nkb, MmaPos<G>& c, uint32_t smem_base, uint32_t d_tmem, uint32_t a0_tmem, uint32_t idesc) {
  const uint64_t desc0   = smem_desc_sw128(smem_base);
  const uint32_t desc_hi = (uint32_t)(desc0 >> 32);
  const uint32_t w0      = (uint32_t)desc0;
  const uint32_t full0 = smem_base + MXB_CTRL(full), empty0 = smem_base + MXB_CTRL(empty);
  for (int kb = 0; kb < nkb; ++kb) {
    const int s = c.stage;
    if (!c.ready && !wwait<G, kAcquire>(smem_base, full0 + 8 * s, c.phase)) return false;
    if (++c.stage == G::kStages) { c.stage = 0; c.phase ^= 1u; }
    // the next stage's barrier is looked at before this stage's MMAs are issued: the round trip of the poll to shared
    // memory then overlaps the issue (test_wait: try_wait could suspend the warp)
    const bool peek = kAcquire ? mbar_test_wait_cluster(full0 + 8 * c.stage, c.phase) : mbar_test_wait(full0 + 8 * c.stage, c.phase);
    tc_fence_after_sync();
    const uint32_t wlo = w0 + s * (G::kStageBytes >> 4);
    if (elect_one_sync())
      mma_stage<kV, true>(d_tmem, wlo, a0_tmem + c.a * kASlotCols, wlo + (kWSlotBytes >> 4), desc_hi, idesc, kb > 0 ? 1u : 0u,
                          empty0 + 8 * s);
    c.ready = __all_sync(0xffffffffu, peek);
    if (kV >= 2) c.a = (c.a + 1) % G::kASlots;
  }
  return true;
}

// A forwarder (packed activations, second CTA): stages with s & 1 == odd, so that each xdone barrier has one waiter, which
// sees all its phases.  One thread.
template <typename G>
__device__ __forceinline__ void forward_arrivals(const CtrlD<G>* ctrl, uint32_t smem_base, int count, int cta, int nctas, int my_tiles,
                                                 int odd, GGStatus* status) {
  const uint32_t full0 = smem_base + MXB_CTRL(full), xdone0 = smem_base + MXB_CTRL(xdone);
  int stage = 0, i = -1, kb = 0, nkb = 0;
  // the next of its stages that holds packed activations, -1 at the end
  auto next_stage = [&]() -> int {
    for (;;) {
      while (kb == nkb) {
        if (++i >= my_tiles) return -1;
        const TileS ti = decode_rec(i < kDuoRecs ? ctrl->recs[i] : make_rec(&ctrl->sched, count, cta + i * nctas, G::kTok, G::kTok, 1));
        kb  = 0;
        nkb = ti.nkb;
        if (ti.scheme != SCH_W4A4) {
          stage = (stage + nkb) % G::kStages;
          kb    = nkb;
        }
      }
      const int s = stage;
      ++kb;
      if (++stage == G::kStages) stage = 0;
      if ((s & 1) == odd) return s;
    }
  };
  uint32_t parities = 0;   // of the next use of every stage's barrier
  int s = next_stage();
  while (s >= 0) {
    if (!bar_wait<G>(smem_base, xdone0 + 8 * s, (parities >> s) & 1u)) {
      report_s(status, 5, cta + i * nctas);
      break;
    }
    // one release for all stages that are ready by now
    uint32_t ready = 0;
    do {
      ready |= 1u << s;
      parities ^= 1u << s;
      s = next_stage();
    } while (s >= 0 && !((ready >> s) & 1u) && mbar_test_wait(xdone0 + 8 * s, (parities >> s) & 1u));
    tc_fence_after_sync();
    tc_fence_before_sync();
    fence_acq_rel_cluster();
    for (; ready; ready &= ready - 1) mbar_arrive_leader_relaxed_n(full0 + 8 * (__ffs(ready) - 1), kCvtGroup);
  }
}

}  // namespace

template <int kMode, bool kShort, bool kExt>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__((DuoGeo<kMode, kShort>::kThreads), 1)
gg_duo_kernel(const GGSwapProblemDev* __restrict__ problems, int count, GGStatus* __restrict__ status) {
  using G = DuoGeo<kMode, kShort>;
  constexpr bool kCvt = kMode != 0;
  // arrivals of the producers of activations at a stage's full[s].  With packed activations the other CTA's producer loads
  // nothing for some tiles; its arrival keeps it from falling a ring behind.
  constexpr int kXArrivals = kMode == 2 ? 2 : 1;
  const int rank  = (int)cluster_ctarank();
  const int cta   = (int)(blockIdx.x >> 1);
  const int nctas = (int)(gridDim.x >> 1);
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen        = smem_raw + (smem_base - smem_u32(smem_raw));
  CtrlD<G>* ctrl           = reinterpret_cast<CtrlD<G>*>(smem_gen + kCtrlOff<G>);
  const uint32_t epi_base  = smem_base + G::kRingBytes;
  Sched* sc                = &ctrl->sched;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (count > kMaxProblems) {
    grid_dependency_wait();
    if (tid == 0 && blockIdx.x == 0) atomicCAS(&status->error, 0, kDevErrTooMany);
    return;
  }
  auto wslot = [&](int s) { return smem_base + s * G::kStageBytes; };
  auto xslot = [&](int s) { return smem_base + s * G::kStageBytes + kWSlotBytes; };

  // ------------------------------------------------------------------ setup
  if (tid == 0) {
    for (int s = 0; s < G::kStages; ++s) {
      mbar_init(smem_u32(&ctrl->full[s]), kCvt ? kXArrivals + 2 * kCvtGroup : 1);
      mbar_init(smem_u32(&ctrl->empty[s]), 1);
    }
    for (int n = 0; n < G::kWBars; ++n) mbar_init(smem_u32(&ctrl->wfull[n]), 1);
    if (kMode == 2)
      for (int s = 0; s < G::kStages; ++s) mbar_init(smem_u32(&ctrl->xdone[s]), kCvtGroup);
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&ctrl->tfull[b]), 1);
      mbar_init(smem_u32(&ctrl->tempty[b]), 2 * kEpiWarps);
    }
    ctrl->abort_flag = 0;
    ctrl->t0         = clock64();
    ctrl->timeout_ns = status->timeout_ms > 0 ? (uint64_t)status->timeout_ms * 1000000ull : kTimeoutNs;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc2(smem_u32(&ctrl->tmem_base), 512);
    tmem_relinquish2();
  }
  grid_dependency_wait();   // row counts and operands come from the kernels before this one
  build_sched(sc, problems, count, G::kTok, 2 * kWT, G::kTok);
  const int total_tiles = sc->total_tiles;
  const int my_tiles    = total_tiles > cta ? (total_tiles - cta + nctas - 1) / nctas : 0;
  for (int i = tid; i < my_tiles && i < kDuoRecs; i += blockDim.x)
    ctrl->recs[i] = make_rec(sc, count, cta + i * nctas, G::kTok, G::kTok, rank);
  acquire_tile_maps<3>(problems, sc, count, cta, nctas, my_tiles);
  auto tile_rec = [&](int i) -> TileRec {
    if (i < kDuoRecs) return ctrl->recs[i];
    return make_rec(sc, count, cta + i * nctas, G::kTok, G::kTok, rank);
  };
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();   // both CTAs' barriers exist before either signals the other's
  tc_fence_after_sync();

  const int skip_stage     = blockIdx.x == 0 ? status->skip_stage - 1 : -1;   // test hook, see GGStatus
  const uint32_t tmem_base = ctrl->tmem_base;
  const uint32_t full0 = smem_base + MXB_CTRL(full), wfull0 = smem_base + MXB_CTRL(wfull), empty0 = smem_base + MXB_CTRL(empty);

  // ------------------------------------------------------------------ roles
  if (warp == 0) {
    // ===== producer of the weights (and of packed activations, which travel with them) =====
    if (elect_one_sync()) {
      int stage = 0, n_stage = 0, wbar = 0;
      uint32_t phase = 0;
      bool ok = true;
      TileRec nrec = tile_rec(0);
      for (int i = 0; ok && i < my_tiles; ++i) {
        const TileS ti = decode_rec(nrec);
        if (i + 1 < my_tiles) nrec = tile_rec(i + 1);
        const GGSwapProblemDev* pr = problems + ti.p;
        uint32_t wbytes;
        int wx_step, wy, wz = 0;
        weight_coords(ti.scheme, ti.n_tile * kWT, wbytes, wx_step, wy);
        if (kExt && pr->silu_inter) { wz = ti.n_tile * 4; wy = 0; }
        const bool convert    = kCvt && is_cvt_scheme(ti.scheme);
        const bool packed_x   = kMode == 2 && ti.scheme == SCH_W4A4;
        const int half        = pair_tokens(ti.ntok) >> 1;
        const int nbox        = packed_x ? (half + kXBoxSmall - 1) / kXBoxSmall : 0;
        const int xr          = ti.x_row + rank * half;
        const uint32_t bytes  = wbytes + (uint32_t)(nbox * kXBoxSmall) * 64u;
        // this tile's K block for which the test hook (GGStatus::skip_stage) announces more weight bytes than will arrive
        const int skip_kb     = (skip_stage >= n_stage && skip_stage < n_stage + ti.nkb) ? skip_stage - n_stage : -1;
        n_stage += ti.nkb;
        for (int kb = 0; kb < ti.nkb; ++kb) {
          if (!bar_wait<G>(smem_base, empty0 + 8 * stage, phase ^ 1u)) {
            report_s(status, 1, cta + i * nctas);
            ok = false;
            break;
          }
          if (convert) {
            const uint32_t wb = wfull0 + 8 * wbar;
            if (++wbar == G::kWBars) wbar = 0;
            mbar_expect_tx(wb, bytes + (kb == skip_kb ? 16u : 0u));
            if (kExt) tma_load_4d(wslot(stage), &pr->tmW, wb, kb * wx_step, wy, 0, wz);
            else      tma_load_2d(wslot(stage), &pr->tmW, wb, kb * wx_step, wy);
            // packed activation rows (64 bytes of K each) go behind the packed weights; the converters expand them
            for (int b = 0; b < nbox; ++b)
              tma_load_2d(wslot(stage) + kWSlotBytes / 2 + b * kXBoxSmall * 64, &pr->tmXs, wb, kb * 64, xr + b * kXBoxSmall);
          } else {
            // announced by the leader's producer of activations
            const uint32_t fb = full0 + 8 * stage;
            if (kExt) tma_load_4d_pair(wslot(stage), &pr->tmW, fb, kb * wx_step, wy, 0, wz);
            else      tma_load_2d_pair(wslot(stage), &pr->tmW, fb, kb * wx_step, wy);
          }
          if (++stage == G::kStages) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 2) {
    // ===== producer of the activations: this CTA's half of the token tile; the leader's announces what the MMAs of
    // the stage wait for =====
    if (elect_one_sync()) {
      int stage = 0, n_stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      TileRec nrec = tile_rec(0);
      for (int i = 0; ok && i < my_tiles; ++i) {
        const TileS ti = decode_rec(nrec);
        if (i + 1 < my_tiles) nrec = tile_rec(i + 1);
        const GGSwapProblemDev* pr = problems + ti.p;
        const int half = pair_tokens(ti.ntok) >> 1;
        const int nbox = (half + kXBoxSmall - 1) / kXBoxSmall;
        const bool big = !kShort && nbox == G::kHalf / kXBoxSmall;
        const int xr   = ti.x_row + rank * half;
        uint32_t wbytes;
        int wx_step, wy;
        weight_coords(ti.scheme, 0, wbytes, wx_step, wy);
        const int xx_step     = (ti.scheme == SCH_FP16 || ti.scheme == SCH_W4A16G128) ? 64 : 128;
        const bool convert    = kCvt && is_cvt_scheme(ti.scheme);
        const bool packed_x   = kMode == 2 && ti.scheme == SCH_W4A4;
        const uint32_t bytes  = packed_x ? 0u : 2u * ((uint32_t)(nbox * kXBoxSmall * kRowBytes) + (convert ? 0u : wbytes));
        const int skip_kb     = (!convert && skip_stage >= n_stage && skip_stage < n_stage + ti.nkb) ? skip_stage - n_stage : -1;
        n_stage += ti.nkb;
        for (int kb = 0; kb < ti.nkb; ++kb) {
          if (!bar_wait<G>(smem_base, empty0 + 8 * stage, phase ^ 1u)) {
            report_s(status, 1, cta + i * nctas);
            ok = false;
            break;
          }
          const uint32_t fb = full0 + 8 * stage;
          if (rank == 0) {
            mbar_expect_tx(fb, bytes + (kb == skip_kb ? 16u : 0u));
            if (kCvt && !convert) mbar_arrive_n(fb, 2 * kCvtGroup);   // nobody converts: the converters' arrivals
          }
          if (kXArrivals == 2 && rank == 1) mbar_arrive_leader_relaxed(fb);
          if (!packed_x) {
            if (big) {
              tma_load_2d_pair(xslot(stage), &pr->tmXh, fb, kb * xx_step, xr);
            } else {
              for (int b = 0; b < nbox; ++b)
                tma_load_2d_pair(xslot(stage) + b * kXBoxSmall * kRowBytes, &pr->tmXs, fb, kb * xx_step, xr + b * kXBoxSmall);
            }
          }
          if (++stage == G::kStages) { stage = 0; phase ^= 1u; }
        }
      }
      if (blockIdx.x == 0) {
        status->prof[PROF_TILES]  = my_tiles;
        status->prof[PROF_STAGES] = n_stage;
      }
    }
  } else if (kMode == 2 && rank == 1 && (warp == 1 || warp == 3)) {
    if constexpr (kMode == 2) {
      if (elect_one_sync()) forward_arrivals<G>(ctrl, smem_base, count, cta, nctas, my_tiles, warp >> 1, status);
    }
  } else if (warp == 1) {
    // ===== MMA issuer: the leader's warp 1 issues for both CTAs =====
    if (rank == 0) {
      MmaPos<G> pos{0, 0, 0u, false};
      int acc = 0;
      TileRec nrec = tile_rec(0);
      for (int i = 0; i < my_tiles; ++i) {
        const TileS ti = decode_rec(nrec);
        if (i + 1 < my_tiles) nrec = tile_rec(i + 1);
        if (i >= 2 && !wwait<G>(smem_base, smem_base + MXB_CTRL(tempty) + 8 * acc, (uint32_t)((i >> 1) - 1) & 1u)) {
          if (lane == 0) report_s(status, 2, cta + i * nctas);
          break;
        }
        tc_fence_after_sync();
        const int npad        = pair_tokens(ti.ntok);
        const uint32_t d_tmem = tmem_base + acc * G::kTok;
        const uint32_t a_tmem = tmem_base + G::kACol0;
        const bool is_int     = is_int_scheme(ti.scheme);
        const bool convert    = kCvt && is_cvt_scheme(ti.scheme);
        const uint32_t idesc  = is_int ? idesc_i8(2 * kWT, npad) : idesc_f16(2 * kWT, npad);
        bool ok;
        if (!convert)
          ok = is_int ? mma_tile<0, kMode == 2, G>(ti.nkb, pos, smem_base, d_tmem, a_tmem, idesc)
                      : mma_tile<1, kMode == 2, G>(ti.nkb, pos, smem_base, d_tmem, a_tmem, idesc);
        else
          ok = is_int ? mma_tile<2, kMode == 2, G>(ti.nkb, pos, smem_base, d_tmem, a_tmem, idesc)
                      : mma_tile<3, kMode == 2, G>(ti.nkb, pos, smem_base, d_tmem, a_tmem, idesc);
        if (!ok) {
          if (lane == 0) report_s(status, 3, cta + i * nctas);
          break;
        }
        if (elect_one_sync()) mma_commit2(smem_base + MXB_CTRL(tfull) + 8 * acc, 3);
        __syncwarp();
        acc ^= 1;
      }
    }
  } else if (warp >= kFirstEpi && warp < kFirstCvt) {
    // ===== epilogue (TMEM lane quarter = warp % 4; lane = output channel, columns = tokens) =====
    // the first four warps take the even 32-token chunks of a tile, the other four the odd ones
    const int q    = warp & 3;
    const int ew   = warp - kFirstEpi;
    const int half = ew >> 2;
    int acc = 0;
    uint32_t acc_phase = 0;
    __half* saw        = ctrl->sa_stage[ew];
    const uint32_t stg = epi_base + ew * kEpiStageS;
    // Everything of a tile that does not depend on its accumulator - fields of the problem, per-token scales of this
    // warp's chunks (lane = token of the chunk), the scale of this thread's channel - is loaded one tile ahead.
    struct Pre {
      TileRec rec;
      int N, ldc, out_mode, silu;
      void* C;
      __half sa[G::kEpiChunks], sb;
    };
    auto channel_of = [&](const TileS& ti, int silu) {
      return silu ? (lane >> 4) * silu + ti.n_tile * (kWT / 2) + q * 16 + (lane & 15) : ti.n_tile * kWT + q * 32 + lane;
    };
    auto prefetch = [&](int i) {
      Pre p;
      p.rec = tile_rec(i);
      const TileS ti = decode_rec(p.rec);
      const GGSwapProblemDev* pr = problems + ti.p;
      p.N = pr->N; p.ldc = pr->ldc; p.out_mode = pr->out_mode; p.C = pr->C;
      p.silu = kExt ? pr->silu_inter : 0;   // > 0: lanes 0-15 of the warp hold gate rows, lanes 16-31 the up rows of the same 16 columns of C
      const bool scaled = is_int_scheme(ti.scheme) && p.out_mode != OUT_ACC;
      const int n_ch    = channel_of(ti, p.silu);
      p.sb = scaled && n_ch < p.N ? __ldg(pr->scale_b + n_ch) : __float2half(0.f);
#pragma unroll
      for (int c = 0; c < G::kEpiChunks; ++c) {
        const int tk = (2 * c + half) * 32 + lane;
        p.sa[c] = scaled && tk < ti.ntok ? pr->scale_a[((int64_t)ti.x_row + tk) * pr->sa_stride] : __float2half(0.f);
      }
      return p;
    };
    Pre next;
    if (my_tiles > 0) next = prefetch(0);
    for (int i = 0; i < my_tiles; ++i) {
      const Pre cur  = next;
      const TileS ti = decode_rec(cur.rec);
      const int ntok      = ti.ntok;
      const int64_t crow0 = ti.c_row;   // row of C of token 0 of the tile
      const int N = cur.N, ldc = cur.ldc, out_mode = cur.out_mode, silu = cur.silu;
      const bool bulk     = kExt && problems[ti.p].bulk_out != 0;
      const int64_t* row_ptrs = kExt ? problems[ti.p].c_row_ptrs : nullptr;
      const bool is_int   = is_int_scheme(ti.scheme);
      const int acc_shift = (ti.scheme == SCH_W4A4 || ti.scheme == SCH_W4A4_XA) ? 8 : 0;
      const int c_col     = ti.n_tile * (kWT / 2) + q * 16 + (lane & 15);
      const int n_ch      = channel_of(ti, silu);
      const __half2 sb2   = __half2half2(cur.sb);
#pragma unroll
      for (int c = 0; c < G::kEpiChunks; ++c) saw[c * 32 + lane] = cur.sa[c];
      __syncwarp();
      bool ok;
      if (kExt) {
        // the four warps of a group meet named barriers below (row-wide stores): one of them waits for all four, so
        // that they agree on the outcome
        if ((ew & 3) == 0) {
          ok = wwait<G>(smem_base, smem_base + MXB_CTRL(tfull) + 8 * acc, acc_phase);
          if (lane == 0) ctrl->pad[half + 2 * (i & 1)] = ok ? 1 : 0;
          __syncwarp();
        }
        nbar_sync(5 + half, 128);
        ok = *reinterpret_cast<volatile int*>(&ctrl->pad[half + 2 * (i & 1)]) != 0;
      } else {
        ok = wwait<G>(smem_base, smem_base + MXB_CTRL(tfull) + 8 * acc, acc_phase);
      }
      if (!ok) {
        if (lane == 0) report_s(status, 4, cta + i * nctas);
        break;
      }
      tc_fence_after_sync();
      if (i + 1 < my_tiles) next = prefetch(i + 1);
      const uint32_t taddr = tmem_base + acc * G::kTok + ((uint32_t)(q * 32) << 16);
      const int nchunk     = (ntok + 31) >> 5;
#pragma unroll 1
      for (int ch = half; ch < nchunk; ch += 2) {
        __syncwarp();   // the lanes left the previous chunk's stores one by one; tcgen05.ld takes the whole warp
        int64_t row_ptr = 0;
        if (row_ptrs && lane < 8 && ch * 32 + q * 8 + lane < ntok) row_ptr = row_ptrs[crow0 + ch * 32 + q * 8 + lane];
        uint32_t v[32];
        tmem_ld_32x32(taddr + ch * 32, v);
        tmem_ld_wait();
        if (out_mode == OUT_ACC) {
          uint32_t* dst = reinterpret_cast<uint32_t*>(cur.C);
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const int tk = ch * 32 + j;
            if (tk < ntok && n_ch < N)
              dst[(crow0 + tk) * ldc + n_ch] = is_int ? (uint32_t)((int)v[j] >> acc_shift) : v[j];
          }
          continue;
        }
        uint32_t h[16];
        if (is_int) {
          // C = fp16_rn( float(acc) * float( fp16_rn(sa * sb) ) )   (mm_tile.cuh:490-493)
          const uint4* sap = reinterpret_cast<const uint4*>(saw + (ch >> 1) * 32);
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            const uint4 sv    = sap[g];
            const __half2* s2 = reinterpret_cast<const __half2*>(&sv);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int j    = g * 4 + e;
              const float2 p = __half22float2(__hmul2(s2[e], sb2));
              const float f0 = (float)((int)v[2 * j] >> acc_shift) * p.x;
              const float f1 = (float)((int)v[2 * j + 1] >> acc_shift) * p.y;
              __half2 r      = __floats2half2_rn(f0, f1);
              h[j]           = *reinterpret_cast<uint32_t*>(&r);
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            __half2 r = __floats2half2_rn(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
            h[j]      = *reinterpret_cast<uint32_t*>(&r);
          }
        }
        if (silu) {
          // h = fp16( fp16(silu(gate)) * up ) on the fp16 results, the arithmetic of the stand-alone silu-mul kernel
          const bool up = lane >= 16;
          uint32_t other[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) other[j] = __shfl_xor_sync(0xffffffffu, up ? h[j] : h[8 + j], 16);
          __half* dst   = reinterpret_cast<__half*>(cur.C) + (crow0 + ch * 32 + (up ? 16 : 0)) * ldc + c_col;
          const int tk0 = ch * 32 + (up ? 16 : 0);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint32_t gw = up ? other[j] : h[j], uw = up ? h[8 + j] : other[j];
            const float2 gf   = __half22float2(*reinterpret_cast<const __half2*>(&gw));
            const float s0    = __fdividef(gf.x, 1.f + __expf(-gf.x));
            const float s1    = __fdividef(gf.y, 1.f + __expf(-gf.y));
            const __half2 r   = __hmul2(__floats2half2_rn(s0, s1), *reinterpret_cast<const __half2*>(&uw));
            if (c_col < silu) {
              if (tk0 + 2 * j < ntok) dst[(2 * j) * ldc] = __low2half(r);
              if (tk0 + 2 * j + 1 < ntok) dst[(2 * j + 1) * ldc] = __high2half(r);
            }
          }
          continue;
        }
        if (bulk) {
          // row-wide stores: the four warps of a group lay the chunk down as 32 token rows of 256 bytes in their joint
          // 8 KiB buffer and hand every row to the copy engine as one piece (outputs that cross NVLink)
          const uint32_t gb = epi_base + half * 4 * kEpiStageS;
          if (lane < 8) bulk_wait_read();
          nbar_sync(1 + 2 * half, 128);
          const uint32_t col = gb + (uint32_t)(q * 32 + lane) * 2;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            sts16(col + (2 * j) * 256, h[j]);
            sts16(col + (2 * j + 1) * 256, h[j] >> 16);
          }
          fence_proxy_async_smem();
          nbar_sync(2 + 2 * half, 128);
          if (lane < 8) {
            const int row = q * 8 + lane, tk = ch * 32 + row;
            const int n0  = ti.n_tile * kWT;
            if (tk < ntok && n0 < N) {
              __half* dst = row_ptrs ? reinterpret_cast<__half*>(row_ptr) + n0
                                     : reinterpret_cast<__half*>(cur.C) + (crow0 + tk) * ldc + n0;
              bulk_store_row(dst, gb + row * 256, (uint32_t)min(kWT, N - n0) * 2u);
            }
            bulk_commit();
          }
          continue;
        }
        // transpose through the warp's 2 KiB buffer: row = token pair (128 bytes = 32 channels x 2 tokens),
        // 16-byte slots XOR-swizzled by the row so that writes and reads are conflict-free
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 16; ++j) sts32(stg + j * 128 + (((lane >> 2) ^ (j & 7)) << 4) + (lane & 3) * 4, h[j]);
        __syncwarp();
        const int p8 = lane & 3;
#pragma unroll
        for (int rd = 0; rd < 2; ++rd) {
          const int tp   = (lane >> 2) + 8 * rd;
          const uint4 a0 = lds128(stg + tp * 128 + (((2 * p8) ^ (tp & 7)) << 4));
          const uint4 a1 = lds128(stg + tp * 128 + (((2 * p8 + 1) ^ (tp & 7)) << 4));
          uint4 lo, hi;
          lo.x = __byte_perm(a0.x, a0.y, 0x5410); hi.x = __byte_perm(a0.x, a0.y, 0x7632);
          lo.y = __byte_perm(a0.z, a0.w, 0x5410); hi.y = __byte_perm(a0.z, a0.w, 0x7632);
          lo.z = __byte_perm(a1.x, a1.y, 0x5410); hi.z = __byte_perm(a1.x, a1.y, 0x7632);
          lo.w = __byte_perm(a1.z, a1.w, 0x5410); hi.w = __byte_perm(a1.z, a1.w, 0x7632);
          const int tk   = ch * 32 + 2 * tp;
          const int ncol = ti.n_tile * kWT + q * 32 + 8 * p8;
          __half* dst    = reinterpret_cast<__half*>(cur.C) + (crow0 + tk) * ldc + ncol;
          if (ncol < N) {
            if (tk < ntok) *reinterpret_cast<uint4*>(dst) = lo;
            if (tk + 1 < ntok) *reinterpret_cast<uint4*>(dst + ldc) = hi;
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_leader_relaxed(smem_base + MXB_CTRL(tempty) + 8 * acc);
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
    if (kExt && lane < 8) bulk_wait_all();
  } else if (kCvt && warp >= kFirstCvt) {
    // ===== converters: three groups of four warps take the converted K blocks in turn =====
    // Thread = weight row (channel) 32*q + lane of the tile = its TMEM lane.
    const int q     = warp & 3;
    const int group = (warp - kFirstCvt) / kCvtGroup;
    const int row   = q * 32 + lane;
    // Where a tile starts: stage, barrier of its first converted K block with the parity of its next use, A slot, the group
    // whose turn it is, stages walked so far.  A group steps from one of its own K blocks to the next: its chain of dependent
    // instructions is what bounds launches with 4-bit weights, so nothing is walked or divided per block.
    int stage0 = 0, wbar0 = 0, slot0 = 0, turn = 0;
    uint32_t wphase0 = 0, it0 = 0;
    constexpr uint32_t kLongAgo = 0u - 64u;
    uint32_t i1 = kLongAgo, i2 = kLongAgo, i3 = kLongAgo, i4 = kLongAgo;   // stage counts of the last four converted K blocks before the tile (none: long ago)
    bool ok = true;
    TileRec nrec = tile_rec(0);
    for (int i = 0; ok && i < my_tiles; ++i) {
      const TileS ti = decode_rec(nrec);
      if (i + 1 < my_tiles) nrec = tile_rec(i + 1);
      if (!is_cvt_scheme(ti.scheme)) {
        stage0 = (stage0 + ti.nkb) % G::kStages;
        it0 += ti.nkb;
        continue;
      }
      const GGSwapProblemDev* pr = problems + ti.p;
      const int N                = pr->N;
      const int gn               = ti.n_tile * kWT + row;
      // w4a16: (scale, zero) of the group's next K block is fetched while the current one is converted
      const bool has_sz   = ti.scheme == SCH_W4A16G128 && gn < N;
      const __half2* szp  = reinterpret_cast<const __half2*>(pr->scale_b) + gn;
      const int gsh       = pr->one_group ? 30 : 1;
      const int kb_first  = group >= turn ? group - turn : group + kCvtGroups - turn;
      __half2 sz_next = __float2half2_rn(0.f);
      if (has_sz && kb_first < ti.nkb) sz_next = __ldg(szp + (int64_t)(kb_first >> gsh) * N);
      int s = (stage0 + kb_first) % G::kStages, wb = wbar0 + kb_first, slot = (slot0 + kb_first) % G::kASlots;
      uint32_t wpar = wphase0;
      if (wb >= G::kWBars) { wb -= G::kWBars; wpar ^= 1u; }
      for (int kb = kb_first; kb < ti.nkb; kb += kCvtGroups) {
        const __half2 sz = sz_next;
        if (has_sz && kb + kCvtGroups < ti.nkb) sz_next = __ldg(szp + (int64_t)((kb + kCvtGroups) >> gsh) * N);
        if (!wwait<G>(smem_base, wfull0 + 8 * wb, wpar)) {
          if (lane == 0) report_s(status, 5, cta + i * nctas);
          ok = false;
          break;
        }
        // The row's 128 bytes of the A slot are formed and stored in two halves of 16 words (fewer registers), the first
        // while the slot may still be in use.
        const uint32_t a_addr = tmem_base + ((uint32_t)(q * 32) << 16) + G::kACol0 + slot * kASlotCols;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t o[16];
          if (ti.scheme != SCH_W4A16G128) {
            const uint32_t src = wslot(s) + row * 64;
            const int sw       = (row >> 1) & 3;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const uint4 w = lds128(src + (((2 * hf + j) ^ sw) << 4));
              o[8 * j + 0] = w.x & 0xF0F0F0F0u; o[8 * j + 4] = (w.x << 4) & 0xF0F0F0F0u;
              o[8 * j + 1] = w.y & 0xF0F0F0F0u; o[8 * j + 5] = (w.y << 4) & 0xF0F0F0F0u;
              o[8 * j + 2] = w.z & 0xF0F0F0F0u; o[8 * j + 6] = (w.z << 4) & 0xF0F0F0F0u;
              o[8 * j + 3] = w.w & 0xF0F0F0F0u; o[8 * j + 7] = (w.w << 4) & 0xF0F0F0F0u;
            }
          } else {
            // channel n = 32*q + 8*f + r lives in packed row 8*q + r; the 16-k block kb16 is the 16-byte chunk
            // 2*kb16 + (f >> 1) (128-byte swizzle: XOR r), nibble 2*(f & 1) + c of word d holds k = 16*kb16 + 8*c + d
            const int f = lane >> 3, r = lane & 7;
            const uint32_t src = wslot(s) + (8 * q + r) * 128;
            const __half2 sc2 = __half2half2(__low2half(sz)), z2 = __half2half2(__high2half(sz));
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              uint4 w = lds128(src + (((4 * hf + 2 * j + (f >> 1)) ^ r) << 4));
              const int sh = 8 * (f & 1);
              w.x >>= sh; w.y >>= sh; w.z >>= sh; w.w >>= sh;
              dequant_two(w.x, sc2, z2, o[8 * j + 0], o[8 * j + 4]);
              dequant_two(w.y, sc2, z2, o[8 * j + 1], o[8 * j + 5]);
              dequant_two(w.z, sc2, z2, o[8 * j + 2], o[8 * j + 6]);
              dequant_two(w.w, sc2, z2, o[8 * j + 3], o[8 * j + 7]);
            }
          }
          if (hf == 0) {
            if (kMode == 2 && ti.scheme == SCH_W4A4) {
              const int half_rows = pair_tokens(ti.ntok) >> 1;
              convert_w4a4<kCvtGroup * 32>(wslot(s) + kWSlotBytes / 2, xslot(s), (half_rows + 31) & ~31, q * 32 + lane);
              fence_proxy_async_smem();
            }
            // The slot's previous content has been read: the MMAs of the fourth converted K block back have completed.  If
            // that was a whole ring ago they have (this stage was refilled after the MMAs a ring back), and its barrier may
            // have moved on.
            if (G::kASlots < G::kStages) {
              const uint32_t it   = it0 + kb;
              const uint32_t last = kb >= 4 ? it - 4 : (kb == 0 ? i4 : (kb == 1 ? i3 : (kb == 2 ? i2 : i1)));
              if (it - last < (uint32_t)G::kStages &&
                  !wwait<G>(smem_base, empty0 + 8 * (last % G::kStages), (last / G::kStages) & 1u)) {
                if (lane == 0) report_s(status, 6, cta + i * nctas);
                ok = false;
                break;
              }
            }
            tc_fence_after_sync();
          }
          tmem_st_32x16(a_addr + 16 * hf, o);
        }
        if (!ok) break;
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          // expanded activations lie in shared memory: release them, in the second CTA to its forwarders
          if (kMode == 2 && ti.scheme == SCH_W4A4) mbar_arrive((rank == 0 ? full0 : smem_base + MXB_CTRL(xdone)) + 8 * s);
          else                                     mbar_arrive_leader_relaxed(full0 + 8 * s);
        }
        s += kCvtGroups;
        if (s >= G::kStages) s -= G::kStages;
        wb += kCvtGroups;
        if (wb >= G::kWBars) { wb -= G::kWBars; wpar ^= 1u; }
        slot += kCvtGroups;
        if (slot >= G::kASlots) slot -= G::kASlots;
      }
      for (int kb = max(ti.nkb - 4, 0); kb < ti.nkb; ++kb) { i4 = i3; i3 = i2; i2 = i1; i1 = it0 + kb; }
      stage0  = (stage0 + ti.nkb) % G::kStages;
      slot0   = (slot0 + ti.nkb) % G::kASlots;
      turn    = (turn + ti.nkb) % kCvtGroups;
      wbar0 += ti.nkb;
      wphase0 ^= (uint32_t)(wbar0 / G::kWBars) & 1u;
      wbar0 %= G::kWBars;
      it0 += ti.nkb;
    }
  }

  // ---------------------------------------------------------------- teardown
  __syncthreads();
  if (blockIdx.x == 0 && tid == 0) status->prof[PROF_TOTAL] = clock64() - ctrl->t0;
  if (*reinterpret_cast<volatile int*>(&ctrl->abort_flag)) {
    // give copies that are still in flight time to land before shared memory is released
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  cluster_sync_all();   // the other CTA may still signal this CTA's barriers or read its shared memory
  if (warp == 1) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc2(tmem_base, 512);
  }
}

namespace {
template <int kMode, bool kShort>
cudaError_t configure_duo() {
  constexpr int kBytes = smem_bytes_duo<DuoGeo<kMode, kShort>>();
  cudaError_t e = cudaFuncSetAttribute(gg_duo_kernel<kMode, kShort, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(gg_duo_kernel<kMode, kShort, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
}
template <int kMode, bool kShort>
cudaError_t launch_duo(const GGSwapProblemDev* problems, int count, GGStatus* status, bool ext, int num_ctas, cudaStream_t stream) {
  using G = DuoGeo<kMode, kShort>;
  return launch_dependent(ext ? gg_duo_kernel<kMode, kShort, true> : gg_duo_kernel<kMode, kShort, false>, num_ctas & ~1, G::kThreads,
                          smem_bytes_duo<G>(), stream, problems, count, status);
}
template <bool kShort>
cudaError_t launch_mode(const GGSwapProblemDev* problems, int count, GGStatus* status, int cvt_mode, bool ext, int num_ctas,
                        cudaStream_t stream) {
  if (cvt_mode == 2) return launch_duo<2, kShort>(problems, count, status, ext, num_ctas, stream);
  if (cvt_mode)      return launch_duo<1, kShort>(problems, count, status, ext, num_ctas, stream);
  return launch_duo<0, kShort>(problems, count, status, ext, num_ctas, stream);
}
}  // namespace

cudaError_t gg_configure_duo() {
  cudaError_t e;
  if ((e = configure_duo<0, false>()) != cudaSuccess) return e;
  if ((e = configure_duo<1, false>()) != cudaSuccess) return e;
  if ((e = configure_duo<2, false>()) != cudaSuccess) return e;
  if ((e = configure_duo<0, true>()) != cudaSuccess) return e;
  if ((e = configure_duo<1, true>()) != cudaSuccess) return e;
  return configure_duo<2, true>();
}

cudaError_t gg_launch_duo(const GGSwapProblemDev* problems, int count, GGStatus* status, int cvt_mode, bool short_tiles, bool ext,
                          int num_ctas, cudaStream_t stream) {
  return short_tiles ? launch_mode<true>(problems, count, status, cvt_mode, ext, num_ctas, stream)
                     : launch_mode<false>(problems, count, status, cvt_mode, ext, num_ctas, stream);
}

}  // namespace mxb
