// Device code shared by the grouped GEMM kernels with swapped operands (weights = M side of the MMA, tokens = N
// side): what a role knows about one tile, named barriers, stores, and the issue sequence of a pipeline stage.
#pragma once
#include "gg_common.cuh"

namespace mxb {
namespace ggc {

constexpr int kWSlotBytes  = kWT * kRowBytes;   // 16 KiB: plain weights, or 8 / 4 KiB of packed ones
constexpr int kEpiStageS   = 2048;              // per epilogue warp: 16 token pairs x 32 channels x 4 bytes
constexpr uint32_t kASlotCols = 32;             // TMEM columns of one converted K block (128 bytes of K per channel)
constexpr int kCvtGroup    = 4;                 // warps per converter group (one per TMEM lane quarter)
constexpr int kEpiWarps    = 8;                 // two per TMEM lane quarter

// What every role needs to know about one tile, precomputed once per CTA: looking a tile up in the
// scheduling tables is a chain of dependent shared-memory loads, each of which takes hundreds of cycles
// while the tensor core streams operands from shared memory.
struct TileRec {
  int pk;       // problem | scheme << 8 | k-blocks << 12
  int x_row;    // buffer row of the tile's first token (A and scale_a)
  int nt;       // channel tile | tokens in the tile (1 .. the kernel's longest) << 16
  int c_row;    // row of C of the tile's first token
};
constexpr int kMaxRecs = 512;   // tiles per CTA kept in the single-CTA kernel's table; later ones are looked up on the fly

struct TileS {
  int p, scheme, nkb, x_row, n_tile, ntok, c_row;
};

__device__ __forceinline__ void report_s(GGStatus* status, int role, int tile) {
  atomicCAS(&status->error, 0, kDevErrTimeout);
  atomicCAS(&status->where, 0, (role << 24) | tile);
}

__device__ __forceinline__ bool is_int_scheme(int s) { return s != SCH_FP16 && s != SCH_W4A16G128; }
__device__ __forceinline__ bool is_cvt_scheme(int s) { return s == SCH_W4A4_XA || s == SCH_W4A16G128 || s == SCH_W4A4; }

// bytes per stage of a weight tile and its coordinates (x step per K block, y) in the weight tensor map
__device__ __forceinline__ void weight_coords(int scheme, int w_row, uint32_t& wbytes, int& wx_step, int& wy) {
  constexpr uint32_t kFull = kWT * kRowBytes;   // 128 channels x 128 bytes of K
  if (scheme == SCH_W8A8)         { wbytes = kFull;     wx_step = 128; wy = w_row; }
  else if (scheme == SCH_FP16)    { wbytes = kFull;     wx_step = 64;  wy = w_row; }
  else if (scheme == SCH_W4A4_XA || scheme == SCH_W4A4) { wbytes = kFull / 2; wx_step = 64;  wy = w_row; }   // 64 packed bytes per row
  else                            { wbytes = kFull / 4; wx_step = 128; wy = w_row / 4; }   // w4a16: 32 packed rows x 128 B
}

// `pair_rank` >= 0: the schedule counts channel tiles of 256 (a CTA pair); this CTA takes the pair_rank-th half
__device__ __forceinline__ TileRec make_rec(const Sched* sc, int count, int t, int tok, int tok_packed, int pair_rank = -1) {
  Tile ti            = find_tile(sc, count, t);
  if (pair_rank >= 0) ti.n_tile = 2 * ti.n_tile + pair_rank;
  const int tile_tok = ti.scheme == SCH_W4A4 ? tok_packed : tok;   // problems with packed activations: shorter tiles
  TileRec r;
  r.pk     = ti.p | (ti.scheme << 8) | (ti.nkb << 12);
  r.x_row  = sc->row0[ti.p] + ti.m_tile * tile_tok;
  r.nt     = ti.n_tile | (min(tile_tok, sc->m_eff[ti.p] - ti.m_tile * tile_tok) << 16);
  r.c_row  = r.x_row + sc->c_shift[ti.p];
  return r;
}
// Acquire the tensor maps this CTA's tiles use (all threads, in parallel; before the barrier that ends the setup).
// Only the first tile of a run of tiles of one problem does it: acquiring every map of a launch of 64 problems in
// every CTA costs the launch 4 us, this 0.5 us.  kBig: index of the map for full token tiles (1 tmX, 3 tmXh).
template <int kBig>
__device__ __forceinline__ void acquire_tile_maps(const GGSwapProblemDev* problems, const Sched* sc, int count, int cta, int nctas,
                                                  int my_tiles) {
  for (int j = threadIdx.x; j < 3 * my_tiles; j += blockDim.x) {
    const int i = j / 3, m = j - 3 * i;
    const int p = find_tile(sc, count, cta + i * nctas).p;
    if (i > 0 && find_tile(sc, count, cta + (i - 1) * nctas).p == p) continue;
    tensormap_acquire(reinterpret_cast<const char*>(problems + p) + (m == 0 ? 0 : (m == 1 ? 2 : kBig)) * sizeof(CUtensorMap));
  }
}
__device__ __forceinline__ TileS decode_rec(const TileRec& r) {
  TileS t;
  t.p = r.pk & 0xff; t.scheme = (r.pk >> 8) & 15; t.nkb = (r.pk >> 12) & 0x3FFFF;
  t.x_row = r.x_row; t.n_tile = r.nt & 0xffff; t.ntok = r.nt >> 16; t.c_row = r.c_row;
  return t;
}

// named barriers (the single-CTA kernel's ids are in its Geo, the CTA-pair kernel uses them in the epilogue only)
__device__ __forceinline__ void nbar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
__device__ __forceinline__ void nbar_arrive(int id, int nthreads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.volatile.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long lds64(uint32_t addr) {
  unsigned long long v;
  asm volatile("ld.volatile.shared.b64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void sts16(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr), "h"((unsigned short)v) : "memory");
}
// one row of the output tile, shared memory -> global memory (this GPU's or a peer's), by the copy engine
__device__ __forceinline__ void bulk_store_row(void* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// One pipeline stage = four MMAs (32 bytes of K each) and the commit that releases the stage, as ONE block of
// straight-line PTX: the issuing warp shares its scheduler with an epilogue warp and converter warps of the same
// TMEM lane quarter, so every instruction it does not need (a predicate set-up per MMA, descriptor arithmetic
// recomputed per stage) delays the issue of the next stage.  `first` == 0: the first MMA overwrites D.
//   kV 0 int8 / weights from shared memory, 1 fp16 / shared memory, 2 int8 / tensor memory, 3 fp16 / tensor memory.
#define MXB_MMA_STAGE_SS(KIND)                                                                              \
  asm volatile(                                                                                             \
      "{\n\t"                                                                                               \
      ".reg .pred p, t;\n\t"                                                                                \
      ".reg .b64 w0, w1, w2, w3, x0, x1, x2, x3;\n\t"                                                       \
      ".reg .b32 a1, a2, a3, b1, b2, b3;\n\t"                                                               \
      "setp.ne.b32 p, %5, 0;\n\t"                                                                           \
      "setp.eq.b32 t, 0, 0;\n\t"                                                                            \
      "add.u32 a1, %1, 2;  add.u32 a2, %1, 4;  add.u32 a3, %1, 6;\n\t"                                      \
      "add.u32 b1, %2, 2;  add.u32 b2, %2, 4;  add.u32 b3, %2, 6;\n\t"                                      \
      "mov.b64 w0, {%1, %3}; mov.b64 w1, {a1, %3}; mov.b64 w2, {a2, %3}; mov.b64 w3, {a3, %3};\n\t"         \
      "mov.b64 x0, {%2, %3}; mov.b64 x1, {b1, %3}; mov.b64 x2, {b2, %3}; mov.b64 x3, {b3, %3};\n\t"         \
      "tcgen05.mma.cta_group::1.kind::" KIND " [%0], w0, x0, %4, p;\n\t"                                    \
      "tcgen05.mma.cta_group::1.kind::" KIND " [%0], w1, x1, %4, t;\n\t"                                    \
      "tcgen05.mma.cta_group::1.kind::" KIND " [%0], w2, x2, %4, t;\n\t"                                    \
      "tcgen05.mma.cta_group::1.kind::" KIND " [%0], w3, x3, %4, t;\n\t"                                    \
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%6];\n\t"                     \
      "}"                                                                                                   \
      :                                                                                                     \
      : "r"(d_tmem), "r"(wlo), "r"(xlo), "r"(desc_hi), "r"(idesc), "r"(first), "r"(empty_bar)               \
      : "memory")
#define MXB_MMA_STAGE_TS(KIND)                                                                              \
  asm volatile(                                                                                             \
      "{\n\t"                                                                                               \
      ".reg .pred p, t;\n\t"                                                                                \
      ".reg .b64 x0, x1, x2, x3;\n\t"                                                                       \
      ".reg .b32 a1, a2, a3, b1, b2, b3;\n\t"                                                               \
      "setp.ne.b32 p, %5, 0;\n\t"                                                                           \
      "setp.eq.b32 t, 0, 0;\n\t"                                                                            \
      "add.u32 a1, %1, 8;  add.u32 a2, %1, 16;  add.u32 a3, %1, 24;\n\t"                                    \
      "add.u32 b1, %2, 2;  add.u32 b2, %2, 4;  add.u32 b3, %2, 6;\n\t"                                      \
      "mov.b64 x0, {%2, %3}; mov.b64 x1, {b1, %3}; mov.b64 x2, {b2, %3}; mov.b64 x3, {b3, %3};\n\t"         \
      "tcgen05.mma.cta_group::1.kind::" KIND " [%0], [%1], x0, %4, p;\n\t"                                  \
      "tcgen05.mma.cta_group::1.kind::" KIND " [%0], [a1], x1, %4, t;\n\t"                                  \
      "tcgen05.mma.cta_group::1.kind::" KIND " [%0], [a2], x2, %4, t;\n\t"                                  \
      "tcgen05.mma.cta_group::1.kind::" KIND " [%0], [a3], x3, %4, t;\n\t"                                  \
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%6];\n\t"                     \
      "}"                                                                                                   \
      :                                                                                                     \
      : "r"(d_tmem), "r"(a_tmem), "r"(xlo), "r"(desc_hi), "r"(idesc), "r"(first), "r"(empty_bar)            \
      : "memory")

// The same for a CTA pair: one M = 256 MMA over both CTAs' weights and token halves, and a commit that arrives at
// the "stage may be refilled" barrier of both CTAs.
#define MXB_MMA_STAGE_SS2(KIND)                                                                             \
  asm volatile(                                                                                             \
      "{\n\t"                                                                                               \
      ".reg .pred p, t;\n\t"                                                                                \
      ".reg .b64 w0, w1, w2, w3, x0, x1, x2, x3;\n\t"                                                       \
      ".reg .b32 a1, a2, a3, b1, b2, b3;\n\t"                                                               \
      "setp.ne.b32 p, %5, 0;\n\t"                                                                           \
      "setp.eq.b32 t, 0, 0;\n\t"                                                                            \
      "add.u32 a1, %1, 2;  add.u32 a2, %1, 4;  add.u32 a3, %1, 6;\n\t"                                      \
      "add.u32 b1, %2, 2;  add.u32 b2, %2, 4;  add.u32 b3, %2, 6;\n\t"                                      \
      "mov.b64 w0, {%1, %3}; mov.b64 w1, {a1, %3}; mov.b64 w2, {a2, %3}; mov.b64 w3, {a3, %3};\n\t"         \
      "mov.b64 x0, {%2, %3}; mov.b64 x1, {b1, %3}; mov.b64 x2, {b2, %3}; mov.b64 x3, {b3, %3};\n\t"         \
      "tcgen05.mma.cta_group::2.kind::" KIND " [%0], w0, x0, %4, p;\n\t"                                    \
      "tcgen05.mma.cta_group::2.kind::" KIND " [%0], w1, x1, %4, t;\n\t"                                    \
      "tcgen05.mma.cta_group::2.kind::" KIND " [%0], w2, x2, %4, t;\n\t"                                    \
      "tcgen05.mma.cta_group::2.kind::" KIND " [%0], w3, x3, %4, t;\n\t"                                    \
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%6], %7;\n\t" \
      "}"                                                                                                   \
      :                                                                                                     \
      : "r"(d_tmem), "r"(wlo), "r"(xlo), "r"(desc_hi), "r"(idesc), "r"(first), "r"(empty_bar),              \
        "h"((unsigned short)3)                                                                              \
      : "memory")
#define MXB_MMA_STAGE_TS2(KIND)                                                                             \
  asm volatile(                                                                                             \
      "{\n\t"                                                                                               \
      ".reg .pred p, t;\n\t"                                                                                \
      ".reg .b64 x0, x1, x2, x3;\n\t"                                                                       \
      ".reg .b32 a1, a2, a3, b1, b2, b3;\n\t"                                                               \
      "setp.ne.b32 p, %5, 0;\n\t"                                                                           \
      "setp.eq.b32 t, 0, 0;\n\t"                                                                            \
      "add.u32 a1, %1, 8;  add.u32 a2, %1, 16;  add.u32 a3, %1, 24;\n\t"                                    \
      "add.u32 b1, %2, 2;  add.u32 b2, %2, 4;  add.u32 b3, %2, 6;\n\t"                                      \
      "mov.b64 x0, {%2, %3}; mov.b64 x1, {b1, %3}; mov.b64 x2, {b2, %3}; mov.b64 x3, {b3, %3};\n\t"         \
      "tcgen05.mma.cta_group::2.kind::" KIND " [%0], [%1], x0, %4, p;\n\t"                                  \
      "tcgen05.mma.cta_group::2.kind::" KIND " [%0], [a1], x1, %4, t;\n\t"                                  \
      "tcgen05.mma.cta_group::2.kind::" KIND " [%0], [a2], x2, %4, t;\n\t"                                  \
      "tcgen05.mma.cta_group::2.kind::" KIND " [%0], [a3], x3, %4, t;\n\t"                                  \
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%6], %7;\n\t" \
      "}"                                                                                                   \
      :                                                                                                     \
      : "r"(d_tmem), "r"(a_tmem), "r"(xlo), "r"(desc_hi), "r"(idesc), "r"(first), "r"(empty_bar),           \
        "h"((unsigned short)3)                                                                              \
      : "memory")

template <int kV, bool kPair>
__device__ __forceinline__ void mma_stage(uint32_t d_tmem, uint32_t wlo, uint32_t a_tmem, uint32_t xlo, uint32_t desc_hi,
                                          uint32_t idesc, uint32_t first, uint32_t empty_bar) {
  if (kPair) {
    if (kV == 0)      { MXB_MMA_STAGE_SS2("i8"); }
    else if (kV == 1) { MXB_MMA_STAGE_SS2("f16"); }
    else if (kV == 2) { MXB_MMA_STAGE_TS2("i8"); }
    else              { MXB_MMA_STAGE_TS2("f16"); }
  } else {
    if (kV == 0)      { MXB_MMA_STAGE_SS("i8"); }
    else if (kV == 1) { MXB_MMA_STAGE_SS("f16"); }
    else if (kV == 2) { MXB_MMA_STAGE_TS("i8"); }
    else              { MXB_MMA_STAGE_TS("f16"); }
  }
}

}  // namespace ggc
}  // namespace mxb
