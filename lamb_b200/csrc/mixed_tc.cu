// Mixed-precision numeric phase on the 5th-generation tensor cores
// (tcgen05.mma kind::i8, accumulators in tensor memory).  No reference
// counterpart: the reference's sector_multiply (src/lamb_multiplication.F90:
// 206-225) is a stub; this computes the same C = A.B as the FP64 path from
// exact int8 digit products (the split-and-sum idea of Ozaki, Ogita, Oishi
// and Rump, Numer. Algorithms 59 (2012), with fixed-point int8 digits).
//
// Digits.  Every element row r of A gets a power-of-two scale 2^ea_r >=
// max_k |A(r,k)|, every element column c of B 2^eb_c >= max_k |B(k,c)|; a
// scaled value x in (-1, 1) is written x = sum_p d_p / (127 * 254^p) + rest
// with integer digits |d_p| <= 127 (t = 127 x; d_p = rint(t);
// t = 254 (t - d_p)), i.e. almost 8 bits a digit: six digits carry 47 bits.
// For S digits,
//   C(r,c) = 2^(ea_r + eb_c) sum_{L=0}^{S-1} sum_{p+q=L} (D_p E_q)(r,c) / (127^2 254^L),
// every D_p E_q is an exact int32 sum (S * 127^2 per inner index keeps
// 22,190 inner indices exact for S = 6), and the recombination runs in FP64.
// Pairs with p + q >= S are dropped (weight below 127^-2 254^-S).
//
// Tiles.  Block rows are too small for tcgen05 (M = 128), so the multiply is
// done on spatial clusters: row atoms (nearby ones, k_tc_pool, or without
// coordinates runs of the row processing order) form clusters of at most 128
// rows, column atoms clusters of at most 64 columns.  A cluster pair
// (I, J) holding at least one C block is one tile; its inner dimension is the
// concatenation of every inner atom k that couples to both clusters (some
// A_ik with i in I and some B_kj with j in J), so only M and N are padded.
// Operands live in "panels" built once per multiply: for row cluster I and
// every inner atom k it touches, b_k panel rows of 128 bytes (the cluster's
// rows, zero where A_ik is absent), one array per digit plane; B likewise
// with 64-byte rows.  A K-row of a tile is thus one 128-byte A panel row and
// one 64-byte B panel row, which the producer warps gather into shared memory
// (cp.async, 16 bytes a thread) in the canonical MN-major layouts of UMMA
// (128B swizzle for A, 64B swizzle for B).  Products that the product filter
// would skip are included (they are bounded by eps each); the C pattern is
// the filtered one, so only C blocks of the pattern are written.
//
// Kernel roles (one CTA of 512 threads per SM, persistent over the tiles):
//   warps 0-5  producers: gather the tile's K rows, 32 per pipeline stage
//              (four warps the A chunks, two warps the B chunks);
//   warp 6     allocates the tensor memory (6 levels x 64 columns in 512); one
//              of its threads, alone (a vote a stage: 5 % slower at 200 waters),
//              issues nine MMAs (M=128, K=32, N=64..256) per
//              stage, one per A digit plane and run of up to four B digit
//              planes;
//   warp 7     expands the tiles' inner lists (runs of panel rows) into the 32
//              (A row, B row) pairs of every stage, up to kRing stages ahead
//              of the producers;
//   warps 8-15 epilogue, two threads a tile row: tensor memory -> FP64 staging
//              tile in shared memory (the six levels of a column recombined
//              exactly in two int64 sums); then every thread writes its row,
//              scaled, into the C blocks of its row atom and keeps the sums
//              of squares per column atom, from which the block norms are
//              summed.  The tile's block list (built before the kernel) and
//              exponents are loaded one tile ahead into registers.
// What bounds it: the MMAs of a stage take ~665 clocks (the tensor pipe and its
// operand reads from shared memory, ~590), the copies of a stage ~350 of the
// producers' time.  With three stages the MMAs waited a third of the time for
// data; the fourth stage's 36 KB come from the inner lists, which no longer lie
// in shared memory, and from the row sums, which overwrite the staged columns
// they came from.  Tiles alone: 200 waters, cutoff 8 (65 stages a tile): 0.73 ->
// 0.68 ms, 2,850 of the probe's 4,340 TOP/s; 1,536 waters, cutoff 7 (11 stages a
// tile, bound by the epilogue's ~14 k clocks): 5.54 -> 4.75 ms (4.57 since; the
// roles' leaving together took 0.5 % of it).  Slower there:
// storing straight from tensor memory (6.2 ms: it stays occupied), whole blocks
// by a warp (5.9), eight columns loaded ahead of their stores (6.3).
// Every wait on an mbarrier is bounded (2 s of %globaltimer); on a timeout
// the kernel records an error code, every role stops, and the host returns
// an error status.  Whoever left a role alone would be missing from the barriers
// of the others, which have no limit: a producer warp's lanes leave at the vote
// after a stage's copies, the epilogue's warps at the vote after staging, and the
// MMA issuer is a single thread.  MMAs and copies in flight are waited for.
#include <cub/cub.cuh>

#include <algorithm>
#include <climits>
#include <numeric>

#include "lamb_probe.h"
#include "multiply.cuh"
#include "ptx.cuh"

namespace lamb {
namespace tc {

constexpr int kS = 6;                 // digits per operand
constexpr int kM = 128, kN = 64, kK = 32;
constexpr int kStages = 4;
constexpr int kRing = 8;              // stages whose rows are listed ahead
constexpr int kPlaneA = kK * kM;      // bytes of one digit plane of one stage (A)
constexpr int kPlaneB = kK * kN;
constexpr int kStageA = kS * kPlaneA;
constexpr int kStageB = kS * kPlaneB;
constexpr int kStageBytes = kStageA + kStageB;  // 36,864: a multiple of 1,024
constexpr int kMaxRowAtoms = 32;      // atoms of one row cluster
constexpr int kMaxColAtoms = 16;      // atoms of one column cluster
constexpr int kMaxBlocks = kMaxRowAtoms * kMaxColAtoms;  // C blocks of one tile
// An integer x with |x| < 2^51 added to the bit pattern of 2^52 + 2^51 gives
// the double 2^52 + 2^51 + x exactly; subtracting that constant leaves x.
constexpr long long kBias = 0x4338000000000000LL;
constexpr double kBiasD = 6755399441055744.0;
// Exponents up to this size scale by multiplying with exact powers of two
// (no intermediate can under- or overflow); larger ones go through ldexp.
constexpr int kExactExp = 500;
constexpr int kProdWarps = 6;                 // warps 0-5: producers
constexpr int kProducers = 32 * kProdWarps;
constexpr int kMmaWarp = kProdWarps;          // warp 6: MMA issuer
constexpr int kListWarp = kMmaWarp + 1;       // warp 7: lists the rows of the stages
constexpr int kEpiWarp0 = kListWarp + 1;      // warps 8-15: epilogue
constexpr int kEpiThreads = 2 * kM;           // two threads a tile row
constexpr int kTileThreads = 32 * kEpiWarp0 + kEpiThreads;
constexpr int kUnits = 32 * (8 + 4);          // 16-byte (row, chunk) copies of a stage and plane
static_assert(kUnits % kProducers == 0, "units split evenly over the producers");
constexpr int kTmemCols = 512;
constexpr int64_t kRowMask = (1 << 25) - 1;  // panel row of an entry (its row count in the top 7 bits)
// Level accumulators stay exact while (K rows) * S * 127^2 < 2^31.
constexpr int64_t kMaxKRows = (int64_t)INT_MAX / (kS * 127 * 127);
// Inner-list entries (runs of panel rows) of one tile.  The kernel has no such
// limit; products with longer lists have always had the mma.sync kernel's
// digits (seven, or the caller's LAMB_GPU_MIXED_SLICES), and six are less exact:
// 1,100 runs of 13, 5 and 5 rows, error against 64 bits 1.07e-13 with six,
// 0.56e-13 with seven.
constexpr int64_t kMaxEntries = 1024;
constexpr double kFirst = 127.0, kBase = 254.0;
// Weight of level L: 1 / (127^2 254^L).
__device__ constexpr double kLevelW[kS] = {1.0 / 16129.0, 1.0 / (16129.0 * 254.0), 1.0 / (16129.0 * 64516.0),
                                          1.0 / (16129.0 * 16387064.0), 1.0 / (16129.0 * 4162314256.0),
                                          1.0 / (16129.0 * 1057227821024.0)};

enum : int { kErrTimeoutFull = 1, kErrTimeoutEmpty = 2, kErrTimeoutTmemFull = 4, kErrTimeoutTmemEmpty = 8,
             kErrTimeoutRows = 16, kErrTimeoutDone = 32 };

// ---- shared-memory layout of the tile kernel --------------------------------------------
struct __align__(16) TileSmem {
  // the tile's scaled FP64 values: element (m, n) at m * kN + (n ^ (m % 16));
  // once a column atom of a row is written out, its first element holds the
  // sum of squares of the row over the atom's columns
  double stg[kM * kN];
  // (A panel row, B panel row) of the inner rows of the next stages; A row
  // kPadRow: zeros, kEndRow: no further stage
  int2 rows[kRing][kK];
  // epilogue tables of the current tile
  long long boff[kMaxBlocks];     // data offset of C block (row atom a, column atom b) at a * 16 + b, or -1
  int32_t blk_id[kMaxBlocks];     // C blocks of the tile in list order: index in C
  int32_t blk_geom[kMaxBlocks];   // and geometry (first tile row | bi << 7 | row atom << 14 | column atom << 19)
  double col_scale[kN];           // 2^exponent of every tile column (when not wide)
  int32_t col_exp[kN];
  int32_t col_atom[kMaxColAtoms]; // first tile column | width << 8 of every column atom
  int32_t n_blk;
  int32_t n_col_atoms;
  unsigned long long bar_full[kStages], bar_empty[kStages];
  unsigned long long bar_tmem_full, bar_tmem_empty, bar_row_full[kRing], bar_row_empty[kRing], bar_done;
  uint32_t tmem_base;
  int abort;
};

constexpr size_t kSmemBytes = (size_t)kStages * kStageBytes + sizeof(TileSmem) + 1024;  // + alignment slack
static_assert(kSmemBytes <= 232448, "tile kernel exceeds the shared memory of one CTA");
constexpr int kPadRow = -1, kEndRow = -2;

struct TcArgs {
  const int2* tiles;
  int64_t n_tiles;
  const int64_t* ent_base;
  const int64_t* ent_cnt;
  const int32_t* krows;
  const uint2* ent;
  const int8_t* pan_a;
  int64_t plane_a;  // bytes between digit planes of the A panels
  const int8_t* pan_b;
  int64_t plane_b;
  const int32_t* cc_first;  // atoms before every column cluster
  // C blocks of every tile: tile t owns blist[lbase[t] .. lbase[t + 1]),
  // each (C block index, geometry, data offset low, high word)
  const int4* blist;
  const int64_t* lbase;
  // per row cluster and tile row m: the row's exponent (0 for padding) and
  // (row atom << 16 | element << 8 | block size) or -1 for padding
  const int32_t* rc_exp;
  const int32_t* rc_row;
  // per column cluster and tile column n the column's exponent; per column
  // atom (first tile column | width << 8)
  const int32_t* cc_exp;
  const int32_t* cc_ab;
  double* c_data;
  double* c_nrm;
  int* err;
};

// ---- PTX helpers -----------------------------------------------------------------------------------
// x * 2^e for any e, out of line: the scatter loop is unrolled 64 times and
// only exponents beyond kExactExp (not met in practice) take this path.
__device__ __noinline__ double scale_wide(double x, int e) { return ldexp(x, e); }
// 2^e for -1022 <= e <= 1023, exactly.
__device__ __forceinline__ double pow2(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }
// Waits until the phase with the given parity has completed; gives up after
// 2 s (or when another role aborted), recording `code`.  The waiting threads
// sleep between checks, leaving the issue slots to the other warps of their SM
// sub-partition.  Called by a whole warp, and then the answer is the same for
// every lane, or (ALONE) with an answer for the calling thread only.
constexpr uint64_t kWaitNs = 2000000000ull;
template <bool ALONE = false>
__device__ __forceinline__ bool bar_wait(unsigned long long* b, uint32_t parity, TileSmem* sm, int* err, int code) {
  auto all = [](bool x) { return ALONE ? x : (bool)__all_sync(0xffffffffu, x); };
  auto any = [](bool x) { return ALONE ? x : (bool)__any_sync(0xffffffffu, x); };
  if (all(bar_try(b, parity))) return true;
  const uint64_t t0 = now_ns();
  for (;;) {
    if (all(bar_try_sleep(b, parity, 200000u))) return true;
    if (any(*(volatile int*)&sm->abort)) return false;
    if (any(now_ns() - t0 > kWaitNs)) {
      if (ALONE || (threadIdx.x & 31) == 0) {
        atomicOr(err, code);
        *(volatile int*)&sm->abort = 1;
      }
      return false;
    }
  }
}
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// Arrive on the mbarrier once every cp.async this thread issued so far has
// landed (counts as one of the barrier's expected arrivals).
__device__ __forceinline__ void cp_arrive(unsigned long long* b) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void named_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
// Named barrier that also returns the OR of every participant's predicate.
__device__ __forceinline__ bool named_sync_or(int id, int n, bool pred) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, %2, %3, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)pred), "r"(id), "r"(n)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor (tcgen05): start address, leading / stride
// byte offsets (16-byte units), version 1, swizzle mode.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo, uint32_t swizzle) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3fff);
  d |= (uint64_t)((lbo >> 4) & 0x3fff) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3fff) << 32;
  d |= (uint64_t)1 << 46;              // descriptor version (Blackwell)
  d |= (uint64_t)(swizzle & 7) << 61;  // 2: 128-byte swizzle, 4: 64-byte swizzle
  return d;
}
// Instruction descriptor: kind::i8, signed A and B, int32 accumulator, both
// operands MN-major, M = 128, the given N (a multiple of 16 up to 256).
constexpr uint32_t idesc_i8(int n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(kM >> 4) << 24);
}

__device__ __forceinline__ void mma_i8(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void mma_commit(unsigned long long* b) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(b))
               : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, int (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Byte offset of (inner row kk, 16-byte chunk c) of one digit plane of a
// stage: A rows are 128 bytes, 128-byte swizzle (chunk ^= row % 8); B rows
// are 64 bytes, 64-byte swizzle (chunk ^= (row / 2) % 4).
__device__ __forceinline__ uint32_t a_swz(int kk, int c) { return (uint32_t)(kk * 128 + ((c ^ (kk & 7)) << 4)); }
__device__ __forceinline__ uint32_t b_swz(int kk, int c) { return (uint32_t)(kk * 64 + ((c ^ ((kk >> 1) & 3)) << 4)); }

// ---- the tile kernel ------------------------------------------------------------------------
__global__ void __launch_bounds__(kTileThreads, 1) k_tc_tiles(TcArgs g) {
  extern __shared__ unsigned char smem_raw[];
  // 1024-byte aligned base by pointer arithmetic on the shared array, so that
  // the compiler keeps the shared state space (shared loads and stores, not
  // generic ones)
  unsigned char* base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  unsigned char* stages = base;
  TileSmem* sm = reinterpret_cast<TileSmem*>(base + (size_t)kStages * kStageBytes);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      bar_init(&sm->bar_full[s], kProducers);
      bar_init(&sm->bar_empty[s], 1);
    }
    bar_init(&sm->bar_tmem_full, 1);
    bar_init(&sm->bar_tmem_empty, kEpiThreads);
    for (int b = 0; b < kRing; ++b) {
      bar_init(&sm->bar_row_full[b], 32);
      bar_init(&sm->bar_row_empty[b], kProdWarps);
    }
    bar_init(&sm->bar_done, 1);
    sm->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm->tmem_base)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm->tmem_base;
  const int64_t n_tiles = g.n_tiles;

  if (warp < kProdWarps) {
    // ================= producers =================
    const int pt = tid;  // 0..kProducers-1
    // A stage is 32 inner rows x (8 A chunks + 4 B chunks) of 16 bytes per
    // digit plane: 384 (row, chunk) units, two per producer thread.  Units
    // 0..255 are A (row u / 8, chunk u % 8), 256..383 are B (row v / 4,
    // chunk v % 4): consecutive lanes copy consecutive chunks of one panel
    // row, so a warp reads whole 128-byte (A) or 64-byte (B) rows.
    // A lane whose wait ran out copies nothing more and leaves with its warp at
    // the vote after the stage's copies, which also shows that every lane has
    // read its rows: a vote at each wait cost 1 % of the mixed multiply.
    for (int64_t gs = 0;; ++gs) {
      const int ring = (int)(gs % kRing), stg = (int)(gs % kStages);
      bool go = bar_wait<true>(&sm->bar_row_full[ring], (uint32_t)((gs / kRing) & 1), sm, g.err, kErrTimeoutRows);
      int2 prow[kUnits / kProducers];
#pragma unroll
      for (int i = 0; i < kUnits / kProducers; ++i) {
        const int u = pt + kProducers * i;
        prow[i] = sm->rows[ring][u < 256 ? (u >> 3) : ((u - 256) >> 2)];
      }
      go = go && prow[0].x != kEndRow &&
           bar_wait<true>(&sm->bar_empty[stg], (uint32_t)(((gs / kStages) & 1) ^ 1), sm, g.err, kErrTimeoutEmpty);
      if (go) {
        const uint32_t sa = smem_u32(stages + (size_t)stg * kStageBytes);
        const uint32_t sb = sa + kStageA;
#pragma unroll
        for (int i = 0; i < kUnits / kProducers; ++i) {
          const int u = pt + kProducers * i;
          const bool is_a = u < 256;  // uniform over the warp
          const int row = is_a ? (u >> 3) : ((u - 256) >> 2);
          const int ch = is_a ? (u & 7) : ((u - 256) & 3);
          const bool valid = prow[i].x >= 0;
          const uint32_t bytes = valid ? 16u : 0u;
          if (is_a) {
            const int8_t* src = g.pan_a + (int64_t)(valid ? prow[i].x : 0) * 128 + 16 * ch;
#pragma unroll
            for (int p = 0; p < kS; ++p) cp16(sa + p * kPlaneA + a_swz(row, ch), src + p * g.plane_a, bytes);
          } else {
            const int8_t* src = g.pan_b + (int64_t)(valid ? prow[i].y : 0) * 64 + 16 * ch;
#pragma unroll
            for (int p = 0; p < kS; ++p) cp16(sb + p * kPlaneB + b_swz(row, ch), src + p * g.plane_b, bytes);
          }
        }
        cp_arrive(&sm->bar_full[stg]);
      }
      if (!__all_sync(0xffffffffu, go)) break;
      if (lane == 0) bar_arrive(&sm->bar_row_empty[ring]);
    }
    // copies that no stage waited for (after an abort) land before the CTA ends
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp >= kEpiWarp0) {
    // ================= epilogue =================
    const int ew = warp & 3;        // tensor-memory lane quarter (warp id mod 4)
    const int et = 32 * ew + lane;  // tile row m
    const int half = (warp - kEpiWarp0) >> 2;  // columns of the tile this thread stages
    const int e2 = kM * half + et;
    // Tables of the next tile, loaded into registers while the current tile
    // is written out: this thread's row exponent and row descriptor, the
    // column exponents (threads < kN), column atoms (threads < 16) and
    // count, block count and up to kMaxBlocks / 256 block-list entries per
    // thread.  The list bounds and clusters of the tile after next are
    // loaded one tile earlier still, so no load waits on another.
    constexpr int kBlkRegs = kMaxBlocks / kEpiThreads;
    int nx_er = 0, nx_ri = -1, nx_ec = 0, nx_cab = 0, nx_nca = 0, nx_nb = 0;
    int4 nx_b[kBlkRegs];
    int64_t lb_lo = 0, lb_hi = 0;  // list bounds of the tile being prefetched
    int2 lb_tile = make_int2(0, 0);  // and its clusters
    auto bounds = [&](int64_t t) {
      lb_lo = t < n_tiles ? g.lbase[t] : 0;
      lb_hi = t < n_tiles ? g.lbase[t + 1] : 0;
      lb_tile = t < n_tiles ? g.tiles[t] : make_int2(0, 0);
    };
    auto prefetch = [&]() {
      const int I = lb_tile.x, J = lb_tile.y;
      nx_er = g.rc_exp[(int64_t)I * kM + et];
      nx_ri = g.rc_row[(int64_t)I * kM + et];
      if (e2 < kN) nx_ec = g.cc_exp[(int64_t)J * kN + e2];
      if (e2 < kMaxColAtoms) nx_cab = g.cc_ab[(int64_t)J * kMaxColAtoms + e2];
      nx_nca = g.cc_first[J + 1] - g.cc_first[J];
      nx_nb = (int)(lb_hi - lb_lo);
#pragma unroll
      for (int j = 0; j < kBlkRegs; ++j) {
        const int k = e2 + kEpiThreads * j;
        nx_b[j] = k < nx_nb ? g.blist[lb_lo + k] : make_int4(0, 0, 0, 0);
      }
    };
    // Writes the prefetched tables to shared memory; returns whether some
    // exponent of the tile lies beyond kExactExp (the same for every thread).
    auto publish = [&]() -> bool {
#pragma unroll
      for (int j = 0; j < kBlkRegs; ++j) sm->boff[e2 + kEpiThreads * j] = -1;
      if (e2 < kN) {
        sm->col_exp[e2] = nx_ec;
        sm->col_scale[e2] = pow2(nx_ec < -kExactExp || nx_ec > kExactExp ? 0 : nx_ec);
      }
      if (e2 < kMaxColAtoms) sm->col_atom[e2] = nx_cab;
      if (e2 == 0) {
        sm->n_blk = nx_nb;
        sm->n_col_atoms = nx_nca;
      }
      named_sync(2, kEpiThreads);  // every slot reset before the blocks are entered
#pragma unroll
      for (int j = 0; j < kBlkRegs; ++j) {
        const int k = e2 + kEpiThreads * j;
        if (k < nx_nb) {
          const int geo = nx_b[j].y;
          sm->blk_id[k] = nx_b[j].x;
          sm->blk_geom[k] = geo;
          sm->boff[((geo >> 14) & 31) * kMaxColAtoms + ((geo >> 19) & 15)] =
              (long long)(((uint64_t)(uint32_t)nx_b[j].w << 32) | (uint32_t)nx_b[j].z);
        }
      }
      const bool w = nx_er < -kExactExp || nx_er > kExactExp || (e2 < kN && (nx_ec < -kExactExp || nx_ec > kExactExp));
      return named_sync_or(2, kEpiThreads, w);
    };
    int64_t local = 0;
    bool wide = false;
    int er = 0, ri = -1;  // this thread's row: exponent and descriptor
    if ((int64_t)blockIdx.x < n_tiles) {
      bounds(blockIdx.x);
      prefetch();
      bounds(blockIdx.x + (int64_t)gridDim.x);
      er = nx_er;
      ri = nx_ri;
      wide = publish();
    }
    for (int64_t t = blockIdx.x; t < n_tiles; t += gridDim.x, ++local) {
      const bool has_next = t + gridDim.x < n_tiles;
      // ---- accumulators: tensor memory -> staging tile, 16 columns a round
      // (a rolled loop: the epilogue's code stays small next to the other
      // roles' in the instruction cache).  Per column the six level sums v_L
      // recombine as (v0 254^2 + v1 254 + v2) w_2 + (v3 254^2 + v4 254 + v5) w_5
      // with w_L = 1 / (127^2 254^L): both brackets are exact in int64
      // (|v_L| < 2^31), below 2^51 in magnitude, and convert exactly to FP64
      // by the 2^52 + 2^51 bias.  The row's power of two is folded into w_2
      // and w_5 (exact: |er| <= kExactExp).  Tensor memory is released as
      // soon as the tile is staged: the next tile's MMAs wait for nothing else. ----
      const bool ok = bar_wait(&sm->bar_tmem_full, (uint32_t)(local & 1), sm, g.err, kErrTimeoutTmemFull);
      double* row = sm->stg + et * kN;
      const int sw = et & 15;
      if (ok) {
        tc_fence_after();
        const double rs = wide ? 1.0 : pow2(er);
        const double w2 = kLevelW[2] * rs, w5 = kLevelW[5] * rs;
        const uint32_t lane_base = tmem + ((uint32_t)(32 * ew) << 16);
#pragma unroll 1
        for (int c0 = (kN / 2) * half; c0 < (kN / 2) * (half + 1); c0 += 16) {
          int v[kS][16];
#pragma unroll
          for (int L = 0; L < kS; ++L) tmem_ld16(lane_base + (uint32_t)(64 * L + c0), v[L]);
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            const long long hi = kBias + (long long)v[0][c] * 64516 + (long long)v[1][c] * 254 + v[2][c];
            const long long lo = kBias + (long long)v[3][c] * 64516 + (long long)v[4][c] * 254 + v[5][c];
            const double hd = __longlong_as_double(hi) - kBiasD, ld = __longlong_as_double(lo) - kBiasD;
            row[(c0 + c) ^ sw] = __fma_rn(hd, w2, ld * w5);
          }
        }
        tc_fence_before();
        bar_arrive(&sm->bar_tmem_empty);  // the MMAs of the next tile may start
      }
      if (has_next) {
        prefetch();
        bounds(t + 2 * (int64_t)gridDim.x);
      }
      // both halves of every row are staged, or all leave
      if (named_sync_or(2, kEpiThreads, !ok)) break;
      // ---- write-out: each thread writes its tile row into the C blocks of
      // its row atom, one column atom after the other (those that start in its
      // half of the columns; a block's column is
      // bi consecutive doubles, so a warp's store covers its rows' runs),
      // scaling by the column's power of two, and keeps the row's sum of
      // squares per column atom for the block norms ----
      if (ri >= 0) {
        const int a = ri >> 16, pe = (ri >> 8) & 0xff, bi = ri & 0xff;
        const int nca = sm->n_col_atoms;
        for (int b = 0; b < nca; ++b) {
          const int cab = sm->col_atom[b];
          const int c0 = cab & 0xff, bj = cab >> 8;
          if ((c0 >= kN / 2) != (half != 0)) continue;
          const long long bo = sm->boff[a * kMaxColAtoms + b];
          double sq = 0.0;
          if (bo >= 0) {
            double* __restrict__ dst = g.c_data + bo + pe;
            if (!wide) {
#pragma unroll 4
              for (int q = 0; q < bj; ++q) {
                const int n = c0 + q;
                const double v = row[n ^ sw] * sm->col_scale[n];
                dst[q * bi] = v;
                sq = __fma_rn(v, v, sq);
              }
            } else {  // rare: exponents beyond kExactExp, scaled out of line
              for (int q = 0; q < bj; ++q) {
                const int n = c0 + q;
                const double v = scale_wide(row[n ^ sw], er + sm->col_exp[n]);
                dst[q * bi] = v;
                sq = __fma_rn(v, v, sq);
              }
            }
          }
          if (bj > 0) row[c0 ^ sw] = sq;
        }
      }
      named_sync(2, kEpiThreads);
      // ---- block norms: rows of the block in ascending order ----
      const int nb = sm->n_blk;
      for (int k = e2; k < nb; k += kEpiThreads) {
        const int geo = sm->blk_geom[k];
        const int r0 = geo & 127, bi = (geo >> 7) & 127, cab = sm->col_atom[(geo >> 19) & 15];
        double sq = 0.0;
        if (cab >> 8)
          for (int r = r0; r < r0 + bi; ++r) sq += sm->stg[r * kN + ((cab & 0xff) ^ (r & 15))];
        g.c_nrm[sm->blk_id[k]] = __dsqrt_rn(sq);
      }
      named_sync(2, kEpiThreads);  // the staging tile and the tables are free again
      if (has_next) {
        er = nx_er;
        ri = nx_ri;
        wide = publish();
      }
    }
  } else if (warp == kListWarp) {
    // ================= rows of the stages =================
    // The tile's list holds runs (first A panel row | rows << 25, first B panel
    // row).  A lane holds one run of the current 32, of the next 32 and, on its
    // way, of the 32 after that, with its first inner row P; the run of a
    // stage's row r is the last one with P <= r, counted in the bit mask of
    // the runs that start inside the stage (32 rows: at most 32 of them).
    int64_t gs = 0, nb_cnt = 0, nb_base = 0;
    int nb_k = 0;
    bool ok = true;
    auto bounds = [&](int64_t t) {
      nb_cnt = t < n_tiles ? g.ent_cnt[t] : 0;
      nb_base = t < n_tiles ? g.ent_base[t] : 0;
      nb_k = t < n_tiles ? g.krows[t] : 0;
    };
    auto slot = [&]() -> int2* {  // the next stage's list, once the producers are past its last use
      const int ring = (int)(gs % kRing);
      ok = bar_wait(&sm->bar_row_empty[ring], (uint32_t)(((gs / kRing) & 1) ^ 1), sm, g.err, kErrTimeoutRows);
      return sm->rows[ring];
    };
    auto filled = [&]() {
      bar_arrive(&sm->bar_row_full[(int)(gs % kRing)]);
      ++gs;
    };
    bounds(blockIdx.x);
    for (int64_t t = blockIdx.x; ok && t < n_tiles; t += gridDim.x) {
      const int n = (int)nb_cnt, K = nb_k;
      const uint2* __restrict__ ent = g.ent + nb_base;
      const int nst = K > 0 ? (K + kK - 1) / kK : 1;
      auto load = [&](int e) { return e < n ? ent[e] : make_uint2(0u, 0u); };
      uint2 x0 = load(lane), x1 = load(32 + lane), x2 = load(64 + lane);
      bounds(t + (int64_t)gridDim.x);
      int carry = 0;
      auto place = [&](const uint2& x) {
        const int cnt = (int)(x.x >> 25);
        const int incl = warp_incl_scan(cnt, lane);
        const int P = cnt ? carry + incl - cnt : INT_MAX / 2;
        carry += __shfl_sync(0xffffffffu, incl, 31);
        return P;
      };
      int p0 = place(x0), p1 = place(x1);
      int base = 0, started = 0;  // first run held; runs that start before the stage
      for (int s = 0; s < nst; ++s) {
        const int r0 = s * kK;
        const unsigned d0 = (unsigned)(p0 - r0), d1 = (unsigned)(p1 - r0);
        const unsigned mask =
            __reduce_or_sync(0xffffffffu, (d0 < (unsigned)kK ? 1u << d0 : 0u) | (d1 < (unsigned)kK ? 1u << d1 : 0u));
        const int e = started + __popc(mask & ((2u << lane) - 1u)) - 1 - base;
        const int from = e & 31;
        const bool first = e < 32;
        const uint32_t a0 = __shfl_sync(0xffffffffu, x0.x, from), a1 = __shfl_sync(0xffffffffu, x1.x, from);
        const uint32_t b0 = __shfl_sync(0xffffffffu, x0.y, from), b1 = __shfl_sync(0xffffffffu, x1.y, from);
        const int q0 = __shfl_sync(0xffffffffu, p0, from), q1 = __shfl_sync(0xffffffffu, p1, from);
        const int in = r0 + lane - (first ? q0 : q1);
        int2* list = slot();
        if (!ok) break;
        list[lane] = r0 + lane < K ? make_int2((int)((first ? a0 : a1) & kRowMask) + in, (int)(first ? b0 : b1) + in)
                                   : make_int2(kPadRow, 0);
        filled();
        started += __popc(mask);
        if (started - 1 - base >= 32) {  // the next stage's first row lies in the second 32
          x0 = x1;
          p0 = p1;
          x1 = x2;
          p1 = place(x1);
          base += 32;
          x2 = load(base + 64 + lane);
        }
      }
    }
    if (ok) {
      int2* list = slot();
      if (ok) {
        list[lane] = make_int2(kEndRow, 0);
        filled();
      }
    }
  } else {
    // ================= MMA issuer =================
    if (lane == 0) {
      int64_t gs = 0, local_mma = 0;
      bool ok = true;
      int next_k = (int64_t)blockIdx.x < n_tiles ? g.krows[blockIdx.x] : 0;  // K rows, loaded one tile ahead
      for (int64_t t = blockIdx.x; ok && t < n_tiles; t += gridDim.x, ++local_mma) {
        const int K = next_k;
        next_k = t + gridDim.x < n_tiles ? g.krows[t + gridDim.x] : 0;
        const int nst = K > 0 ? (K + kK - 1) / kK : 1;
        // tensor memory is free once the epilogue has read the previous tile
        if (!bar_wait<true>(&sm->bar_tmem_empty, (uint32_t)((local_mma & 1) ^ 1), sm, g.err, kErrTimeoutTmemEmpty)) break;
        tc_fence_after();
        for (int s = 0; s < nst; ++s, ++gs) {
          const int stg = (int)(gs % kStages);
          ok = bar_wait<true>(&sm->bar_full[stg], (uint32_t)((gs / kStages) & 1), sm, g.err, kErrTimeoutFull);
          if (!ok) break;
          tc_fence_after();
          fence_async_smem();
          const uint32_t sa = smem_u32(stages + (size_t)stg * kStageBytes);
          const uint32_t sb = sa + kStageA;
          // A plane p times B planes q0 .. q0 + nq - 1 in one MMA of N = 64 nq:
          // the B planes lie kPlaneB apart, which the descriptor's leading
          // byte offset steps through as consecutive 64-column chunks of N,
          // and their products land on consecutive level accumulators
          // 64 (p + q) of tensor memory.  Nine MMAs per stage cover the 21
          // pairs p + q < 6 (N <= 256 per instruction), reading A nine times
          // instead of 21.
#pragma unroll
          for (int p = 0; p < kS; ++p) {
            const uint64_t da = smem_desc(sa + p * kPlaneA, 128, 1024, 2);
#pragma unroll
            for (int q0 = 0; q0 < kS - p; q0 += 4) {
              const int nq = (kS - p - q0) < 4 ? (kS - p - q0) : 4;
              const uint64_t db = smem_desc(sb + q0 * kPlaneB, kPlaneB, 512, 4);
              mma_i8(tmem + (uint32_t)(64 * (p + q0)), da, db, idesc_i8(64 * nq), (s > 0 || p > 0) ? 1u : 0u);
            }
          }
          mma_commit(&sm->bar_empty[stg]);
        }
        if (ok) mma_commit(&sm->bar_tmem_full);
      }
      // every MMA issued by this CTA has completed before tensor memory is
      // released, after an abort too (so this wait does not look at it)
      mma_commit(&sm->bar_done);
      const uint64_t t0 = now_ns();
      while (!bar_try_sleep(&sm->bar_done, 0, 200000u))
        if (now_ns() - t0 > kWaitNs) {
          atomicOr(g.err, kErrTimeoutDone);
          break;
        }
    }
    __syncwarp();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == kMmaWarp)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

}  // namespace tc
}  // namespace lamb

// ============================================================================================
// Preparation: clusters, inner-atom bitmaps, digit panels, tiles and their inner lists.
// ============================================================================================
namespace lamb {
namespace tc {

// Warps a block row in the kernels below that list blocks: with one, 288 dense
// rows leave most of the GPU idle (bitmaps, pair blocks, tile flags and tile
// lists together 98 -> 65 us there; no change at 4,608 rows of 380 blocks).
constexpr int kRowWays = 8;

// Bitmap bit (cluster, inner atom k): A (by_row): cluster of row r, k = column;
// B (!by_row): cluster of column c, k = row r.  The lanes whose bits share a word
// join them, and write only what is missing: dense rows hit the same words over
// and over (288 rows: 34 and 25 -> 11 and 21 us).
__global__ void k_tc_bitmap(int32_t n_rows, const int64_t* __restrict__ row_p, const int32_t* __restrict__ col,
                            const int32_t* __restrict__ clus, int by_row, int32_t W, uint32_t* bm) {
  const int lane = threadIdx.x & 31;
  for (int64_t gw = global_warp(); gw < (int64_t)n_rows * kRowWays; gw += grid_warps()) {
    const int64_t r = gw / kRowWays;
    for (int64_t b = row_p[r] + 32 * (gw % kRowWays) + lane; b < row_p[r + 1]; b += 32 * kRowWays) {
      const int c = col[b];
      const int cl = by_row ? clus[r] : clus[c];
      const int k = by_row ? c : (int)r;
      const int64_t word = (int64_t)cl * W + (k >> 5);
      const unsigned peers = __match_any_sync(__activemask(), (unsigned long long)word);
      const uint32_t bits = __reduce_or_sync(peers, 1u << (k & 31));
      if (lane == __ffs(peers) - 1 && (__ldcg(&bm[word]) & bits) != bits) atomicOr(&bm[word], bits);
    }
  }
}

// Panel rows and pairs (cluster, inner atom) of every cluster before each bitmap word, and their totals.
__global__ void k_tc_word_prefix(int32_t n_cl, int32_t W, const uint32_t* __restrict__ bm,
                                 const int8_t* __restrict__ kbs, int2* __restrict__ before,
                                 int64_t* __restrict__ tot_row, int64_t* __restrict__ tot_pair) {
  const int lane = threadIdx.x & 31;
  for (int64_t c = global_warp(); c < n_cl; c += grid_warps()) {
    int carry = 0, pairs = 0;
    for (int w0 = 0; w0 < W; w0 += 32) {
      const int w = w0 + lane;
      uint32_t bits = w < W ? bm[c * W + w] : 0u;
      const int n = __popc(bits);
      int rows = 0;
      while (bits) {
        const int bit = __ffs(bits) - 1;
        bits &= bits - 1u;
        rows += kbs[32 * w + bit];
      }
      const int incl = warp_incl_scan(rows, lane), incl_n = warp_incl_scan(n, lane);
      if (w < W) before[c * W + w] = make_int2(carry + incl - rows, pairs + incl_n - n);
      carry += __shfl_sync(0xffffffffu, incl, 31);
      pairs += __shfl_sync(0xffffffffu, incl_n, 31);
    }
    if (lane == 0) {
      tot_row[c] = carry;
      tot_pair[c] = pairs;
    }
  }
}

// Exclusive sums of four short arrays, a CTA each: array i has n[i] values, one after the other.
struct Sums {
  int64_t n[4];
};
__global__ void __launch_bounds__(1024) k_tc_sums(Sums a, const int64_t* __restrict__ in, int64_t* __restrict__ out) {
  typedef cub::BlockScan<long long, 1024> BS;
  __shared__ typename BS::TempStorage ts;
  const int64_t n = a.n[blockIdx.x];
  for (int i = 0; i < (int)blockIdx.x; ++i) {
    in += a.n[i];
    out += a.n[i];
  }
  long long carry = 0;
  for (int64_t x0 = 0; x0 < n; x0 += 1024) {
    const int64_t x = x0 + threadIdx.x;
    long long v = x < n ? in[x] : 0, sum = 0;
    BS(ts).ExclusiveSum(v, v, sum);
    __syncthreads();
    if (x < n) out[x] = carry + v;
    carry += sum;
  }
}

// The pairs: (cluster, inner atom, first panel row, rows).
__global__ void k_tc_pairs(int32_t n_cl, int32_t W, const uint32_t* __restrict__ bm, const int8_t* __restrict__ kbs,
                           const int2* __restrict__ before, const int64_t* __restrict__ row_base,
                           const int64_t* __restrict__ pair_base, int4* __restrict__ pair) {
  for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < (int64_t)n_cl * W;
       x += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(x / W), w = (int)(x % W);
    int row = (int)row_base[c] + before[x].x;
    int4* out = pair + pair_base[c] + before[x].y;
    for (uint32_t bits = bm[x]; bits; bits &= bits - 1u) {
      const int k = 32 * w + __ffs(bits) - 1, bk = kbs[k];
      *out++ = make_int4(c, k, row, bk);
      row += bk;
    }
  }
}

// Where the blocks of every pair lie: data offset of the block of the
// cluster's atom x at pair * per + x (-1, set before, where it is absent).
template <bool A_SIDE>
__global__ void k_tc_pair_blocks(int32_t n_rows, int32_t W, const int64_t* __restrict__ row_p,
                                 const int32_t* __restrict__ col, const int64_t* __restrict__ off,
                                 const int32_t* __restrict__ clus, const int32_t* __restrict__ idx,
                                 const uint32_t* __restrict__ bm, const int2* __restrict__ before,
                                 const int64_t* __restrict__ pair_base, long long* __restrict__ tab) {
  constexpr int per = A_SIDE ? kMaxRowAtoms : kMaxColAtoms;
  const int lane = threadIdx.x & 31;
  for (int64_t gw = global_warp(); gw < (int64_t)n_rows * kRowWays; gw += grid_warps()) {
    const int64_t i = gw / kRowWays;
    for (int64_t b = row_p[i] + 32 * (gw % kRowWays) + lane; b < row_p[i + 1]; b += 32 * kRowWays) {
      const int j = col[b], a = A_SIDE ? (int)i : j, k = A_SIDE ? j : (int)i, c = clus[a];
      const int64_t x = (int64_t)c * W + (k >> 5);
      const int64_t pair = pair_base[c] + before[x].y + __popc(bm[x] & ((1u << (k & 31)) - 1u));
      tab[pair * per + idx[a]] = off[b];
    }
  }
}

// x * 2^-e: an exact power-of-two multiply where 2^-e is a normal double
// (the result rounds once either way), ldexp outside that range.
__device__ __forceinline__ double scale_down(double x, int e) {
  return e > -1000 && e < 1000 ? x * __longlong_as_double((long long)(1023 - e) << 52) : ldexp(x, -e);
}

// Digit panels: panel row base[c] + row(c, k) + r holds one byte per element row
// (A, 128) or column (B, 64) of cluster c and digit plane, zero where the block
// is absent.  A warp writes whole panel rows, pair by pair: its lanes hold the
// elements lane + 32 j (A; two rows of lane % 16 + 16 j, B), so that loads run
// along a block's storage, and exchange their four digits with three neighbours
// for words of four consecutive bytes: one full line stored per plane and row,
// and no plane to clear beforehand.  The pairs' blocks are listed first (the
// search for them cost more than the digits).
// Digits.  s = t + 1.5 2^52 rounds t (|t| <= 127) to the integer digit d in its
// low bits; 254 (t - d) is one fused operation from t and another, exact, for
// 254 d: 17 FP64 operations an element.  Bound by instruction issue (about 250 a
// panel row) and the latency of a pair's first loads.  1,536 waters, all of the
// preparation, with panels cleared and written byte by byte, block by block:
// 2.12 -> 1.34 ms (0.39 the A panels, 0.31 B); 200 waters 0.52 -> 0.41 ms.
constexpr double kRound = 6755399441055744.0;  // 1.5 2^52

// The 4 x 4 bytes of four neighbouring lanes transposed: lane i of them gets byte i of each.
__device__ __forceinline__ uint32_t transpose4(uint32_t w, int lane) {
  const uint32_t u = __shfl_xor_sync(0xffffffffu, w, 2);
  const uint32_t a = (lane & 2) ? __byte_perm(u, w, 0x7632) : __byte_perm(w, u, 0x5410);
  const uint32_t v = __shfl_xor_sync(0xffffffffu, a, 1);
  return (lane & 1) ? __byte_perm(v, a, 0x7351) : __byte_perm(a, v, 0x6240);
}

constexpr int kDigitPairs = 4;  // a warp takes: mostly of one cluster

template <bool A_SIDE>
__global__ void __launch_bounds__(128, 5) k_tc_digits(
    int64_t n_pairs, const int4* __restrict__ pairs, const long long* __restrict__ tab,
    const int32_t* __restrict__ geo, const int32_t* __restrict__ exps, const double* __restrict__ data, int64_t plane,
    int8_t* __restrict__ pan) {
  constexpr int width = A_SIDE ? kM : kN, lanes = width / 4, per = A_SIDE ? kMaxRowAtoms : kMaxColAtoms;
  constexpr int rows_at_once = 32 / lanes;
  const int lane = threadIdx.x & 31, l = lane % lanes, sub = lane / lanes;
  int have = -1;       // cluster of the scales
  double scale[4] = {};  // 127 2^-exponent: x times it rounds once, as x 2^-exponent (exact) times 127 does
  bool wide = false;
  for (int64_t p0 = global_warp() * kDigitPairs; p0 < n_pairs; p0 += grid_warps() * kDigitPairs) {
    int4 nxt = pairs[p0];
    long long nxt_o = tab[p0 * per + lane % per];
    for (int64_t q = p0; q < min(n_pairs, p0 + kDigitPairs); ++q) {
      const int c = nxt.x, bk = nxt.w;
      const int64_t prow = nxt.z;
      const long long o = nxt_o;
      if (q + 1 < min(n_pairs, p0 + kDigitPairs)) {
        nxt = pairs[q + 1];
        nxt_o = tab[(q + 1) * per + lane % per];
      }
      const int32_t* __restrict__ g = geo + (int64_t)c * width + l;
      const int32_t* __restrict__ ex = exps + (int64_t)c * width + l;
      if (c != have) {
        have = c;
        wide = false;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int e = ex[lanes * j];
          wide |= !(e > -1000 && e < 1000);
          scale[j] = kFirst * __longlong_as_double((long long)(1023 - e) << 52);
        }
        wide = __any_sync(0xffffffffu, wide);
      }
      const double* src[4];
      bool some[2] = {false, false};  // any block of the warp's elements 2 h and 2 h + 1
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int gj = g[lanes * j];
        const long long oj = __shfl_sync(0xffffffffu, o, gj >= 0 ? gj >> 16 : 0);
        const int e = (gj >> 8) & 0xff;
        src[j] = gj >= 0 && oj >= 0 ? data + oj + (A_SIDE ? e : e * bk + sub) : nullptr;
        some[j / 2] |= src[j] != nullptr;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) some[h] = __any_sync(0xffffffffu, some[h]);
      for (int r0 = 0; r0 < bk; r0 += rows_at_once) {
        const int r = r0 + sub;
        double t[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          t[j] = src[j] && r < bk ? *src[j] : 0.0;
          if (src[j]) src[j] += A_SIDE ? g[lanes * j] & 0xff : rows_at_once;
        }
        uint32_t d[kS] = {};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (!some[h]) continue;
#pragma unroll
          for (int j = 2 * h; j < 2 * h + 2; ++j)
            t[j] = !wide ? t[j] * scale[j] : scale_down(t[j], ex[lanes * j]) * kFirst;
#pragma unroll
          for (int p = 0; p < kS; ++p)
#pragma unroll
            for (int j = 2 * h; j < 2 * h + 2; ++j) {
              const double s = t[j] + kRound;
              const int sel = j == 0 ? 0x3214 : j == 1 ? 0x3240 : j == 2 ? 0x3410 : 0x4210;  // byte j
              d[p] = __byte_perm(d[p], (uint32_t)__double2loint(s), sel);
              if (p + 1 < kS) t[j] = __fma_rn(t[j], kBase, __fma_rn(s, -kBase, kRound * kBase));
            }
        }
        int8_t* dst = pan + (prow + r) * width + lanes * (lane & 3) + (l & ~3);
#pragma unroll
        for (int p = 0; p < kS; ++p) {
          const uint32_t v = transpose4(d[p], lane);
          if (r < bk) *reinterpret_cast<uint32_t*>(dst + p * plane) = v;
        }
      }
    }
  }
}

// Tiles are numbered, and so processed, by groups of kRowGroup row clusters,
// inside a group by column cluster, then row cluster: the tiles in flight
// share A and B panels (1,536 waters: 5.66 -> 5.54 ms; groups of 4 or 16 the same).
constexpr int kRowGroup = 8;
__device__ __forceinline__ int64_t tile_slot(int I, int J, int32_t n_cc) {
  return ((int64_t)(I / kRowGroup) * n_cc + J) * kRowGroup + I % kRowGroup;
}

// Tile flags: (row cluster, column cluster) pairs holding a C block.
__global__ void k_tc_tile_flags(int32_t n_rows, const int64_t* __restrict__ row_p, const int32_t* __restrict__ col,
                                const int32_t* __restrict__ rcl, const int32_t* __restrict__ ccl, int32_t n_cc,
                                int64_t* __restrict__ flag) {
  const int lane = threadIdx.x & 31;
  for (int64_t gw = global_warp(); gw < (int64_t)n_rows * kRowWays; gw += grid_warps()) {
    const int64_t i = gw / kRowWays;
    const int I = rcl[i];
    for (int64_t b = row_p[i] + 32 * (gw % kRowWays) + lane; b < row_p[i + 1]; b += 32 * kRowWays)
      flag[tile_slot(I, ccl[col[b]], n_cc)] = 1;
  }
}

__global__ void k_tc_tile_list(int64_t n_map, int32_t n_cc, const int64_t* __restrict__ flag,
                               const int64_t* __restrict__ pos, int2* __restrict__ tiles) {
  for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n_map; x += (int64_t)gridDim.x * blockDim.x)
    if (flag[x]) {
      const int64_t g = x / kRowGroup;
      tiles[pos[x]] = make_int2((int)(g / n_cc) * kRowGroup + (int)(x % kRowGroup), (int)(g % n_cc));
    }
}

// C blocks of every tile.  Count pass: blocks per tile.  Fill pass: one
// list entry per block at lbase[t] + (arrival order within the tile), each
// (block index, geometry, data offset) with geometry = first tile row |
// bi << 7 | row atom << 14 | column atom << 19.  The order within a tile
// decides nothing but which thread computes which norm.
template <bool FILL>
__global__ void k_tc_tile_blocks(int32_t n_rows, const int64_t* __restrict__ row_p, const int32_t* __restrict__ col,
                                 const int64_t* __restrict__ off, const int8_t* __restrict__ row_bs,
                                 const int32_t* __restrict__ rcl, const int32_t* __restrict__ roff,
                                 const int32_t* __restrict__ ratom, const int32_t* __restrict__ ccl,
                                 const int32_t* __restrict__ catom, int32_t n_cc,
                                 const int64_t* __restrict__ pos, int64_t* __restrict__ cnt,
                                 const int64_t* __restrict__ lbase, int4* __restrict__ blist) {
  const int lane = threadIdx.x & 31;
  for (int64_t gw = global_warp(); gw < (int64_t)n_rows * kRowWays; gw += grid_warps()) {
    const int64_t i = gw / kRowWays;
    const int I = rcl[i];
    const int geo_r = roff[i] | ((int)row_bs[i] << 7) | (ratom[i] << 14);
    for (int64_t b = row_p[i] + 32 * (gw % kRowWays) + lane; b < row_p[i + 1]; b += 32 * kRowWays) {
      const int j = col[b];
      const int64_t t = pos[tile_slot(I, ccl[j], n_cc)];
      const int64_t slot = (int64_t)atomicAdd(reinterpret_cast<unsigned long long*>(&cnt[t]), 1ull);
      if (FILL) {
        const int geo = geo_r | (catom[j] << 19);
        const uint64_t o = (uint64_t)off[b];
        blist[lbase[t] + slot] = make_int4((int)b, geo, (int)(uint32_t)o, (int)(uint32_t)(o >> 32));
      }
    }
  }
}

// Inner atoms of every tile: k with A_ik for some i in I and B_kj for some j
// in J (and b_k > 0), in increasing k.  Consecutive such atoms whose panel
// rows follow on in both panels (no atom of only one cluster between them)
// merge into one entry of up to 127 rows, within one 32-atom bitmap word.
// Count pass: entries and panel rows per tile.  Fill pass: (A panel row |
// rows << 25, B panel row) per entry.  One warp per tile, a lane per word.
template <bool FILL>
__device__ __forceinline__ int tile_word_entries(uint32_t xa, uint32_t xb, int w, const int8_t* __restrict__ kbs,
                                                 int64_t ar, int64_t br, uint2* __restrict__ out, int* nrows,
                                                 int* slot) {
  const uint32_t x = xa & xb;
  int n = 0, open = 0;  // rows of the open entry (0: none)
  int64_t oa = 0, ob = 0;
  for (uint32_t y = xa | xb; y;) {
    const int bit = __ffs(y) - 1;
    y &= y - 1u;
    const uint32_t mb = 1u << bit;
    const int bk = kbs[32 * w + bit];
    if (bk > 0) {
      if (x & mb) {
        *nrows += bk;
        if (open > 0 && open + bk <= 127) {
          open += bk;
        } else {
          if (open > 0) {
            if (FILL) out[atomicAdd(slot, 1)] = make_uint2((uint32_t)oa | ((uint32_t)open << 25), (uint32_t)ob);
            ++n;
          }
          oa = ar;
          ob = br;
          open = bk;
        }
      } else if (open > 0) {  // rows of one panel only: the next entry starts apart
        if (FILL) out[atomicAdd(slot, 1)] = make_uint2((uint32_t)oa | ((uint32_t)open << 25), (uint32_t)ob);
        ++n;
        open = 0;
      }
    }
    if (xa & mb) ar += bk;
    if (xb & mb) br += bk;
  }
  if (open > 0) {
    if (FILL) out[atomicAdd(slot, 1)] = make_uint2((uint32_t)oa | ((uint32_t)open << 25), (uint32_t)ob);
    ++n;
  }
  return n;
}

template <bool FILL>
__global__ void __launch_bounds__(256) k_tc_tile_k(int64_t n_tiles, const int2* __restrict__ tiles, int32_t W,
                                                   const uint32_t* __restrict__ bma, const uint32_t* __restrict__ bmb,
                                                   const int2* __restrict__ wra, const int2* __restrict__ wrb,
                                                   const int64_t* __restrict__ basea, const int64_t* __restrict__ baseb,
                                                   const int8_t* __restrict__ kbs, int64_t* __restrict__ cnt,
                                                   int32_t* __restrict__ rows, const int64_t* __restrict__ ebase,
                                                   uint2* __restrict__ ent) {
  // Fill pass: entries take the next free slot of their tile (a per-warp
  // counter); the K-row order inside a tile does not change the exact int32
  // level sums, and the producers' row prefix follows the stored order.
  __shared__ int slot[8];
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  for (int64_t t = global_warp(); t < n_tiles; t += grid_warps()) {
    const int64_t I = tiles[t].x, J = tiles[t].y;
    int64_t carry = 0;
    int nrows = 0;
    if (FILL && lane == 0) slot[wl] = 0;
    __syncwarp();
    uint2* out = FILL ? ent + ebase[t] : nullptr;
    for (int w0 = 0; w0 < W; w0 += 32) {
      const int w = w0 + lane;
      const uint32_t xa = w < W ? bma[I * W + w] : 0u, xb = w < W ? bmb[J * W + w] : 0u;
      int c = 0;
      if (xa & xb) {
        const int64_t ar = basea[I] + wra[I * W + w].x, br = baseb[J] + wrb[J * W + w].x;
        c = tile_word_entries<FILL>(xa, xb, w, kbs, ar, br, out, &nrows, &slot[wl]);
      }
      if (!FILL) carry += warp_sum_ll(c);
    }
    if (!FILL) {
      nrows = (int)warp_sum_ll(nrows);
      if (lane == 0) {
        cnt[t] = carry;
        rows[t] = nrows;
      }
    }
    __syncwarp();
  }
}

// Longest inner list and largest K of any tile, and the pipeline stages of
// all tiles (ceil(K / 32), at least one), into out[0..2].
__global__ void k_tc_tile_stats(int64_t n_tiles, const int64_t* __restrict__ cnt, const int32_t* __restrict__ rows,
                                unsigned long long* __restrict__ out) {
  long long me = 0, mr = 0, st = 0;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n_tiles; t += (int64_t)gridDim.x * blockDim.x) {
    me = max(me, (long long)cnt[t]);
    mr = max(mr, (long long)rows[t]);
    st += rows[t] > 0 ? (rows[t] + kK - 1) / kK : 1;
  }
  for (int o = 16; o; o >>= 1) {
    me = max(me, __shfl_xor_sync(0xffffffffu, me, o));
    mr = max(mr, __shfl_xor_sync(0xffffffffu, mr, o));
    st += __shfl_xor_sync(0xffffffffu, st, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&out[0], (unsigned long long)me);
    atomicMax(&out[1], (unsigned long long)mr);
    atomicAdd(&out[2], (unsigned long long)st);
  }
}

// Exponent of every tile row / column of every cluster (0 for padding).
__global__ void k_tc_cluster_exp(int64_t n, const int32_t* __restrict__ elem, const int* __restrict__ e,
                                 int32_t* __restrict__ out) {
  for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (int64_t)gridDim.x * blockDim.x)
    out[x] = elem[x] >= 0 ? e[elem[x]] : 0;
}

// ---- clusters ------------------------------------------------------------------------------
// Clusters of nearby atoms.  A tile's inner dimension is the union of what its
// atoms couple to, so its work grows with the extent of its clusters; cutting
// the processing order (a Morton curve) into runs leaves clusters that straddle
// the curve's jumps.  One warp holds the next 256 unplaced atoms of the order
// in registers, starts a cluster at the first of them and adds the nearest to
// the cluster's centre (minimum image) that still fits until none does.  One
// block per range of the order and operand width: a chain of ~0.2 us steps, run
// once per order.  1,536 waters, cutoff 7: 13.3 -> 10.1 T tensor operations,
// tiles 6.68 -> 5.66 ms; 200 waters, cutoff 8: 2.50 -> 1.93 T, 0.95 -> 0.77 ms.
// (A pool of 64 or 512 gives 10.8 or 9.7 T.)
constexpr int kPoolLane = 8;       // atoms a lane holds: a pool of 256
constexpr int kPoolRange = 1024;  // atoms of a range at least: each range ends with one cluster to fill

__global__ void __launch_bounds__(32) k_tc_pool(int32_t n, int32_t ranges, const int32_t* __restrict__ order,
                                                const float* __restrict__ pos, float bx, float by, float bz,
                                                const int8_t* __restrict__ bs, int32_t* __restrict__ out) {
  const int lane = threadIdx.x;
  const bool cols = blockIdx.y != 0;
  const int cap = cols ? kN : kM, max_atoms = cols ? kMaxColAtoms : kMaxRowAtoms;
  int next = (int)((int64_t)n * blockIdx.x / ranges);
  const int end = (int)((int64_t)n * (blockIdx.x + 1) / ranges);
  int32_t* dst = out + (cols ? n : 0) + next;  // the atoms in cluster order, ~atom where a cluster starts
  int id[kPoolLane], sz[kPoolLane];
  unsigned rank[kPoolLane];
  float x[kPoolLane], y[kPoolLane], z[kPoolLane];
#pragma unroll
  for (int j = 0; j < kPoolLane; ++j) {
    id[j] = -1;
    rank[j] = 0xffffffffu;
    sz[j] = 0;
    x[j] = y[j] = z[j] = 0.f;
  }
  for (int placed = 0, total = end - next; placed < total;) {
    // ---- refill the free slots from the order ----
#pragma unroll
    for (int j = 0; j < kPoolLane; ++j) {
      const unsigned free_ = __ballot_sync(0xffffffffu, id[j] < 0);
      const int t = next + __popc(free_ & ((1u << lane) - 1u));
      if (id[j] < 0 && t < end) {
        const int a = order[t];
        id[j] = a;
        rank[j] = (unsigned)t;
        sz[j] = bs[a];
      }
      next = min(end, next + __popc(free_));
    }
    // ---- the first unplaced atom starts the cluster; the others' offsets from it ----
    unsigned first = 0xffffffffu;
#pragma unroll
    for (int j = 0; j < kPoolLane; ++j) first = min(first, rank[j]);
    first = __reduce_min_sync(0xffffffffu, first);
    const int seed = order[first];
    const float sx = pos[3 * seed], sy = pos[3 * seed + 1], sz0 = pos[3 * seed + 2];
    int rows = bs[seed], atoms = 1;
    if (lane == 0) dst[placed] = ~seed;
    ++placed;
#pragma unroll
    for (int j = 0; j < kPoolLane; ++j) {
      if (rank[j] == first) {
        id[j] = -1;
        rank[j] = 0xffffffffu;
      }
      if (id[j] >= 0) {
        const float dx = pos[3 * id[j]] - sx, dy = pos[3 * id[j] + 1] - sy, dz = pos[3 * id[j] + 2] - sz0;
        x[j] = dx - bx * rintf(dx / bx);
        y[j] = dy - by * rintf(dy / by);
        z[j] = dz - bz * rintf(dz / bz);
      }
    }
    float cx = 0.f, cy = 0.f, cz = 0.f;  // sum of the cluster's offsets
    while (rows < cap && atoms < max_atoms) {
      const float inv = 1.f / (float)atoms;
      const float mx = cx * inv, my = cy * inv, mz = cz * inv;
      unsigned best = 0xffffffffu;
#pragma unroll
      for (int j = 0; j < kPoolLane; ++j) {
        const float dx = x[j] - mx, dy = y[j] - my, dz = z[j] - mz;
        const unsigned key = (__float_as_uint(dx * dx + dy * dy + dz * dz) & ~255u) | (unsigned)(lane << 3 | j);
        if (id[j] >= 0 && rows + sz[j] <= cap) best = min(best, key);
      }
      best = __reduce_min_sync(0xffffffffu, best);
      if (best == 0xffffffffu) break;
      const int owner = (best >> 3) & 31;
      int a = 0, b = 0;
      float ax = 0.f, ay = 0.f, az = 0.f;
#pragma unroll
      for (int j = 0; j < kPoolLane; ++j)
        if ((int)(best & 7u) == j) {
          a = id[j];
          b = sz[j];
          ax = x[j];
          ay = y[j];
          az = z[j];
          if (lane == owner) {
            id[j] = -1;
            rank[j] = 0xffffffffu;
          }
        }
      a = __shfl_sync(0xffffffffu, a, owner);
      rows += __shfl_sync(0xffffffffu, b, owner);
      cx += __shfl_sync(0xffffffffu, ax, owner);
      cy += __shfl_sync(0xffffffffu, ay, owner);
      cz += __shfl_sync(0xffffffffu, az, owner);
      if (lane == 0) dst[placed] = a;
      ++placed;
      ++atoms;
    }
  }
}

}  // namespace tc

// Clusters of one axis with the tables the kernels read, in one device buffer.
struct ClusterTab {
  Ctx* ctx = nullptr;
  char* buf = nullptr;
  int32_t n = 0;
  bool cols = false;
  std::vector<int8_t> bs;       // the block sizes it was made for
  int32_t *of = nullptr, *idx = nullptr, *off = nullptr;  // [atoms] cluster, index and first element in it
  int32_t* geo = nullptr;       // [n * kM or kN] atom << 16 | element << 8 | block size of every tile row / column, -1 for padding
  int32_t* cab = nullptr;       // columns: [n * kMaxColAtoms] first tile column | width << 8 of every column atom
  int32_t* elem = nullptr;      // [n * kM or kN] element row / column of the matrix, -1 for padding
  int32_t* first = nullptr;     // [n + 1] atoms before the cluster
  ~ClusterTab() {
    if (buf) cudaFreeAsync(buf, ctx->stream);
  }
};

namespace tc {

// Cuts `order` into clusters: a new one where the next atom would pass max_rows
// rows or max_atoms atoms, and before every complemented atom.
static int32_t make_clusters(Ctx* ctx, const int32_t* order, const std::vector<int8_t>& bs, bool cols,
                             std::shared_ptr<ClusterTab>* out) {
  const int max_rows = cols ? kN : kM, max_atoms = cols ? kMaxColAtoms : kMaxRowAtoms;
  const int64_t n = (int64_t)bs.size();
  auto t = std::make_shared<ClusterTab>();
  t->ctx = ctx;
  t->cols = cols;
  t->bs = bs;
  std::vector<int32_t> h(3 * n), base(n + 1, 0), geo, cab, elem, first;
  int32_t *of = h.data(), *idx = of + n, *off = idx + n;
  for (int64_t a = 0; a < n; ++a) base[a + 1] = base[a] + bs[a];
  int rows = 0, atoms = 0;
  for (int64_t p = 0; p < n; ++p) {
    const bool head = order[p] < 0;
    const int a = head ? ~order[p] : order[p], b = bs[a];
    if (p == 0 || head || rows + b > max_rows || atoms == max_atoms) {
      ++t->n;
      first.push_back((int32_t)p);
      geo.resize((size_t)t->n * max_rows, -1);
      if (cols) cab.resize((size_t)t->n * kMaxColAtoms, 0);
      elem.resize((size_t)t->n * max_rows, -1);
      rows = atoms = 0;
    }
    const int64_t I = t->n - 1;
    of[a] = (int32_t)I;
    idx[a] = atoms;
    off[a] = b > 0 ? rows : 0;  // an atom without elements may follow the last row: 128 has no place in 7 bits
    if (cols) cab[I * kMaxColAtoms + atoms] = rows | (b << 8);
    for (int e = 0; e < b; ++e) {
      geo[I * max_rows + rows + e] = (atoms << 16) | (e << 8) | b;
      elem[I * max_rows + rows + e] = base[a] + e;
    }
    rows += b;
    ++atoms;
  }
  first.push_back((int32_t)n);
  for (const auto* v : {&geo, &cab, &elem, &first}) h.insert(h.end(), v->begin(), v->end());
  LAMB_TRY(dalloc(ctx, &t->buf, (int64_t)(h.size() * sizeof(int32_t))));
  LAMB_CUDA(ctx, cudaMemcpyAsync(t->buf, h.data(), h.size() * sizeof(int32_t), cudaMemcpyHostToDevice, ctx->stream));
  t->of = reinterpret_cast<int32_t*>(t->buf);
  t->idx = t->of + n;
  t->off = t->idx + n;
  t->geo = t->off + n;
  t->cab = t->geo + geo.size();
  t->elem = t->cab + cab.size();
  t->first = t->elem + elem.size();
  *out = std::move(t);
  return LAMB_GPU_OK;
}

// Row clusters of A and, if asked for, column clusters of the same atoms: kept with the matrix.
static int32_t ensure_clusters(Ctx* ctx, DevMatrix* A, bool cols) {
  auto have = [&](const std::shared_ptr<ClusterTab>& t) { return t && t->bs == A->h_row_bs; };
  if (have(A->rclu) && (!cols || have(A->cclu))) return LAMB_GPU_OK;
  const int32_t n = A->n_rows;
  std::vector<int32_t> ord(2 * (size_t)n);
  if ((int64_t)A->h_pos.size() == 3ll * n && A->order) {
    float* d_pos = nullptr;
    int32_t* d_out = nullptr;
    LAMB_TRY(dalloc(ctx, &d_pos, 3ll * n));
    LAMB_TRY(dalloc(ctx, &d_out, 2ll * n));
    LAMB_CUDA(ctx, cudaMemcpyAsync(d_pos, A->h_pos.data(), sizeof(float) * 3 * n, cudaMemcpyHostToDevice, ctx->stream));
    const int ranges = std::max(1, n / kPoolRange);
    k_tc_pool<<<dim3((unsigned)ranges, cols ? 2 : 1), 32, 0, ctx->stream>>>(n, ranges, A->order, d_pos, A->box[0], A->box[1],
                                                                 A->box[2], A->row_bs, d_out);
    LAMB_LAUNCHED(ctx);
    LAMB_CUDA(ctx, cudaMemcpyAsync(ord.data(), d_out, sizeof(int32_t) * (cols ? 2 : 1) * n, cudaMemcpyDeviceToHost, ctx->stream));
    LAMB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    dfree(ctx, d_pos);
    dfree(ctx, d_out);
  } else {
    std::copy(A->h_order.begin(), A->h_order.end(), ord.begin());
    std::copy(A->h_order.begin(), A->h_order.end(), ord.begin() + n);
  }
  LAMB_TRY(make_clusters(ctx, ord.data(), A->h_row_bs, false, &A->rclu));
  return !cols ? LAMB_GPU_OK : make_clusters(ctx, ord.data() + n, A->h_row_bs, true, &A->cclu);
}

// Device buffers of one call, released (stream-ordered) when it returns.
struct Bufs {
  Ctx* ctx;
  std::vector<void*> p;
  ~Bufs() {
    for (void* x : p)
      if (x) cudaFreeAsync(x, ctx->stream);
  }
  template <typename T>
  int32_t alloc(T** d, int64_t n) {
    LAMB_TRY(dalloc(ctx, d, std::max<int64_t>(n, 1)));
    p.push_back(*d);
    return LAMB_GPU_OK;
  }
};

}  // namespace tc

bool mixed_tc_eligible(const DevMatrix* A, const DevMatrix* B) {
  return max_block(A->h_row_bs) <= tc::kM && max_block(B->h_col_bs) <= tc::kN && A->n_rows > 0 && B->n_cols > 0 &&
         A->nnz > 0 && B->nnz > 0;
}

// Numeric phase of a mixed multiply on tcgen05 (C's pattern, layout and data
// buffer already set by a pattern-only symbolic phase).  Sets *ran = false,
// leaving C untouched, when a tile's inner list or its rows exceed the limits;
// the caller then uses the mma.sync path.
int32_t numeric_mixed_tc(Ctx* ctx, DevMatrix* A, DevMatrix* B, DevMatrix* C, const MixedPlanes& mp, double* c_nrm,
                         bool* ran, cudaEvent_t ev_prepared, double* tensor_ops) {
  using namespace tc;
  *ran = false;
  *tensor_ops = 0.0;
  if (C->nnz == 0) { *ran = true; return LAMB_GPU_OK; }
  // ---- clusters (host, from the row processing order) ----
  if ((int)A->h_order.size() != A->n_rows) return fail(ctx, LAMB_LEVEL_FAILURE, LAMB_TYPE_INTERNAL_ERROR, "mixed: row order missing");
  // columns of the rows' atoms share their order and coordinates
  const bool same = B->n_cols == A->n_rows && B->h_col_bs == A->h_row_bs;
  LAMB_TRY(ensure_clusters(ctx, A, same));
  std::shared_ptr<ClusterTab> ccp = A->cclu;
  if (!same) {
    std::vector<int32_t> ident(B->n_cols);
    std::iota(ident.begin(), ident.end(), 0);
    LAMB_TRY(make_clusters(ctx, ident.data(), B->h_col_bs, true, &ccp));
  }
  const ClusterTab &rc = *A->rclu, &cc = *ccp;
  const int32_t nk = A->n_cols, W = (nk + 31) / 32;
  Bufs m{ctx, {}};
  const int32_t *d_rcl = rc.of, *d_ratom = rc.idx, *d_roff = rc.off, *d_ccl = cc.of, *d_catom = cc.idx;
  int32_t *d_rc_exp, *d_cc_exp;
  LAMB_TRY(m.alloc(&d_rc_exp, (int64_t)rc.n * kM)); LAMB_TRY(m.alloc(&d_cc_exp, (int64_t)cc.n * kN));
  k_tc_cluster_exp<<<grid_for((int64_t)rc.n * kM), 256, 0, ctx->stream>>>((int64_t)rc.n * kM, rc.elem, mp.ea, d_rc_exp);
  LAMB_LAUNCHED(ctx);
  k_tc_cluster_exp<<<grid_for((int64_t)cc.n * kN), 256, 0, ctx->stream>>>((int64_t)cc.n * kN, cc.elem, mp.eb, d_cc_exp);
  LAMB_LAUNCHED(ctx);
  // ---- inner-atom bitmaps and panel row offsets ----
  int2 *wra, *wrb;
  LAMB_TRY(m.alloc(&wra, (int64_t)rc.n * W)); LAMB_TRY(m.alloc(&wrb, (int64_t)cc.n * W));
  // panel rows and pairs of every cluster of A, then of B, each with a zero
  // behind, and the bitmaps; what lies before each cluster
  const int64_t n_a = rc.n + 1, n_b = cc.n + 1;
  int64_t *tra, *basea;
  const int64_t zeroed = sizeof(int64_t) * 2 * (n_a + n_b) + sizeof(uint32_t) * ((int64_t)rc.n + cc.n) * W;
  LAMB_TRY(m.alloc(&tra, zeroed / 8 + 1));
  LAMB_TRY(m.alloc(&basea, 2 * (n_a + n_b)));
  int64_t *tpa = tra + n_a, *trb = tpa + n_a, *tpb = trb + n_b;
  int64_t *pba = basea + n_a, *baseb = pba + n_a, *pbb = baseb + n_b;
  uint32_t *bma = reinterpret_cast<uint32_t*>(tpb + n_b), *bmb = bma + (int64_t)rc.n * W;
  LAMB_CUDA(ctx, cudaMemsetAsync(tra, 0, (size_t)zeroed, ctx->stream));
  k_tc_bitmap<<<grid_for(32ll * kRowWays * A->n_rows, 256), 256, 0, ctx->stream>>>(A->n_rows, A->row_p, A->col, d_rcl, 1, W, bma);
  LAMB_LAUNCHED(ctx);
  k_tc_bitmap<<<grid_for(32ll * kRowWays * B->n_rows, 256), 256, 0, ctx->stream>>>(B->n_rows, B->row_p, B->col, d_ccl, 0, W, bmb);
  LAMB_LAUNCHED(ctx);
  k_tc_word_prefix<<<grid_for(32ll * rc.n, 256), 256, 0, ctx->stream>>>(rc.n, W, bma, A->col_bs, wra, tra, tpa);
  LAMB_LAUNCHED(ctx);
  k_tc_word_prefix<<<grid_for(32ll * cc.n, 256), 256, 0, ctx->stream>>>(cc.n, W, bmb, B->row_bs, wrb, trb, tpb);
  LAMB_LAUNCHED(ctx);
  k_tc_sums<<<4, 1024, 0, ctx->stream>>>(Sums{{n_a, n_a, n_b, n_b}}, tra, basea);
  LAMB_LAUNCHED(ctx);
  // ---- tiles: cluster pairs holding a C block ----
  const int64_t n_map = (int64_t)(rc.n + kRowGroup - 1) / kRowGroup * kRowGroup * cc.n;
  int64_t *flag, *pos;
  LAMB_TRY(m.alloc(&flag, n_map + 1)); LAMB_TRY(m.alloc(&pos, n_map + 1));
  LAMB_CUDA(ctx, cudaMemsetAsync(flag, 0, sizeof(int64_t) * (size_t)(n_map + 1), ctx->stream));
  k_tc_tile_flags<<<grid_for(32ll * kRowWays * C->n_rows, 256), 256, 0, ctx->stream>>>(C->n_rows, C->row_p, C->col, d_rcl, d_ccl,
                                                                         cc.n, flag);
  LAMB_LAUNCHED(ctx);
  LAMB_TRY(exclusive_scan_i64(ctx, flag, pos, n_map + 1));
  // panel rows and pairs of A and B and the tile count
  auto* h_sizes = reinterpret_cast<volatile int64_t*>(ctx->pin + kPinTc);
  const int64_t* d_sizes[5] = {basea + rc.n, baseb + cc.n, pba + rc.n, pbb + cc.n, pos + n_map};
  for (int i = 0; i < 5; ++i)
    LAMB_CUDA(ctx, cudaMemcpyAsync((void*)&h_sizes[i], d_sizes[i], sizeof(int64_t), cudaMemcpyDeviceToHost, ctx->stream));
  LAMB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  const int64_t ra = h_sizes[0], rb = h_sizes[1], na = h_sizes[2], nbp = h_sizes[3], n_tiles = h_sizes[4];
  if (ra + 1 > kRowMask || rb + 1 > INT_MAX) return LAMB_GPU_OK;  // panel rows beyond the entry format: not run
  // ---- digit panels ----
  const int64_t plane_a = ((ra + 1) * 128 + 255) & ~255ll, plane_b = ((rb + 1) * 64 + 255) & ~255ll;
  int8_t *pan_a = nullptr, *pan_b = nullptr;
  LAMB_TRY(scratch(ctx, kScrPlaneA, plane_a * kS, &pan_a));
  LAMB_TRY(scratch(ctx, kScrPlaneB, plane_b * kS, &pan_b));
  int4 *pairs_a, *pairs_b;
  long long *tab_a, *tab_b;
  LAMB_TRY(m.alloc(&pairs_a, na)); LAMB_TRY(m.alloc(&pairs_b, nbp));
  const int64_t n_tab = na * kMaxRowAtoms + nbp * kMaxColAtoms;
  LAMB_TRY(m.alloc(&tab_a, n_tab));
  tab_b = tab_a + na * kMaxRowAtoms;
  LAMB_CUDA(ctx, cudaMemsetAsync(tab_a, 0xff, sizeof(long long) * n_tab, ctx->stream));
  k_tc_pairs<<<grid_for((int64_t)rc.n * W, 64), 64, 0, ctx->stream>>>(rc.n, W, bma, A->col_bs, wra, basea, pba, pairs_a);
  LAMB_LAUNCHED(ctx);
  k_tc_pairs<<<grid_for((int64_t)cc.n * W, 64), 64, 0, ctx->stream>>>(cc.n, W, bmb, B->row_bs, wrb, baseb, pbb, pairs_b);
  LAMB_LAUNCHED(ctx);
  k_tc_pair_blocks<true><<<grid_for(32ll * kRowWays * A->n_rows, 256), 256, 0, ctx->stream>>>(
      A->n_rows, W, A->row_p, A->col, A->off, rc.of, rc.idx, bma, wra, pba, tab_a);
  LAMB_LAUNCHED(ctx);
  k_tc_pair_blocks<false><<<grid_for(32ll * kRowWays * B->n_rows, 256), 256, 0, ctx->stream>>>(
      B->n_rows, W, B->row_p, B->col, B->off, cc.of, cc.idx, bmb, wrb, pbb, tab_b);
  LAMB_LAUNCHED(ctx);
  auto warps = [](int64_t n) { return 32 * ((n + kDigitPairs - 1) / kDigitPairs); };
  k_tc_digits<true><<<grid_for(warps(na), 128), 128, 0, ctx->stream>>>(na, pairs_a, tab_a, rc.geo, d_rc_exp, A->data,
                                                                       plane_a, pan_a);
  LAMB_LAUNCHED(ctx);
  k_tc_digits<false><<<grid_for(warps(nbp), 128), 128, 0, ctx->stream>>>(nbp, pairs_b, tab_b, cc.geo, d_cc_exp, B->data,
                                                                         plane_b, pan_b);
  LAMB_LAUNCHED(ctx);
  // ---- tile list, C block lists, inner lists ----
  int2* tiles;
  int32_t* krows;
  int64_t *ecnt, *ebase, *lcnt, *lbase;
  int4* blist;
  LAMB_TRY(m.alloc(&tiles, n_tiles));
  LAMB_TRY(m.alloc(&lcnt, n_tiles + 1));
  LAMB_TRY(m.alloc(&lbase, n_tiles + 1));
  LAMB_TRY(m.alloc(&blist, C->nnz));
  LAMB_TRY(m.alloc(&krows, n_tiles));
  LAMB_TRY(m.alloc(&ecnt, n_tiles + 1));
  LAMB_TRY(m.alloc(&ebase, n_tiles + 1));
  k_tc_tile_list<<<grid_for(n_map, 256), 256, 0, ctx->stream>>>(n_map, cc.n, flag, pos, tiles);
  LAMB_LAUNCHED(ctx);
  LAMB_CUDA(ctx, cudaMemsetAsync(lcnt, 0, sizeof(int64_t) * (size_t)(n_tiles + 1), ctx->stream));
  k_tc_tile_blocks<false><<<grid_for(32ll * kRowWays * C->n_rows, 256), 256, 0, ctx->stream>>>(
      C->n_rows, C->row_p, C->col, C->off, C->row_bs, d_rcl, d_roff, d_ratom, d_ccl, d_catom, cc.n, pos, lcnt, nullptr,
      nullptr);
  LAMB_LAUNCHED(ctx);
  LAMB_TRY(exclusive_scan_i64(ctx, lcnt, lbase, n_tiles + 1));
  LAMB_CUDA(ctx, cudaMemsetAsync(lcnt, 0, sizeof(int64_t) * (size_t)(n_tiles + 1), ctx->stream));
  k_tc_tile_blocks<true><<<grid_for(32ll * kRowWays * C->n_rows, 256), 256, 0, ctx->stream>>>(
      C->n_rows, C->row_p, C->col, C->off, C->row_bs, d_rcl, d_roff, d_ratom, d_ccl, d_catom, cc.n, pos, lcnt, lbase,
      blist);
  LAMB_LAUNCHED(ctx);
  LAMB_CUDA(ctx, cudaMemsetAsync(ecnt + n_tiles, 0, sizeof(int64_t), ctx->stream));
  k_tc_tile_k<false><<<grid_for(32ll * n_tiles, 256), 256, 0, ctx->stream>>>(
      n_tiles, tiles, W, bma, bmb, wra, wrb, basea, baseb, A->col_bs, ecnt, krows, nullptr, nullptr);
  LAMB_LAUNCHED(ctx);
  LAMB_TRY(exclusive_scan_i64(ctx, ecnt, ebase, n_tiles + 1));
  // {longest list, largest K, stages, entries} in one read-back
  unsigned long long* d_stats;
  LAMB_TRY(m.alloc(&d_stats, 4));
  LAMB_CUDA(ctx, cudaMemsetAsync(d_stats, 0, 4 * sizeof(unsigned long long), ctx->stream));
  k_tc_tile_stats<<<grid_for(n_tiles, 256), 256, 0, ctx->stream>>>(n_tiles, ecnt, krows, d_stats);
  LAMB_LAUNCHED(ctx);
  LAMB_CUDA(ctx, cudaMemcpyAsync(d_stats + 3, ebase + n_tiles, sizeof(int64_t), cudaMemcpyDeviceToDevice, ctx->stream));
  auto* h_stats = reinterpret_cast<volatile unsigned long long*>(ctx->pin + kPinTc + 5);
  LAMB_CUDA(ctx, cudaMemcpyAsync((void*)h_stats, d_stats, 4 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, ctx->stream));
  LAMB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  const int64_t max_ent = (int64_t)h_stats[0], max_rows = (int64_t)h_stats[1], n_ent = (int64_t)h_stats[3];
  *tensor_ops = (double)h_stats[2] * (kS * (kS + 1) / 2) * 2.0 * kM * kN * kK;
  if (max_ent > kMaxEntries || max_rows > kMaxKRows) return LAMB_GPU_OK;  // not run
  uint2* ent;
  LAMB_TRY(m.alloc(&ent, n_ent));
  k_tc_tile_k<true><<<grid_for(32ll * n_tiles, 256), 256, 0, ctx->stream>>>(
      n_tiles, tiles, W, bma, bmb, wra, wrb, basea, baseb, A->col_bs, nullptr, nullptr, ebase, ent);
  LAMB_LAUNCHED(ctx);
  if (ev_prepared) LAMB_CUDA(ctx, cudaEventRecord(ev_prepared, ctx->stream));
  // ---- the tile kernel ----
  int* d_err;
  LAMB_TRY(m.alloc(&d_err, 1));
  LAMB_CUDA(ctx, cudaMemsetAsync(d_err, 0, sizeof(int), ctx->stream));
  TcArgs g{};
  g.tiles = tiles; g.n_tiles = n_tiles; g.ent_base = ebase; g.ent_cnt = ecnt; g.krows = krows; g.ent = ent;
  g.pan_a = pan_a; g.plane_a = plane_a; g.pan_b = pan_b; g.plane_b = plane_b;
  g.cc_first = cc.first;
  g.blist = blist; g.lbase = lbase; g.c_data = C->data; g.c_nrm = c_nrm; g.err = d_err;
  g.rc_exp = d_rc_exp; g.rc_row = rc.geo; g.cc_exp = d_cc_exp; g.cc_ab = cc.cab;
  LAMB_CUDA(ctx, cudaFuncSetAttribute(k_tc_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes));
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  const int grid = (int)std::min<int64_t>(n_tiles, sms);
  k_tc_tiles<<<grid, kTileThreads, kSmemBytes, ctx->stream>>>(g);
  LAMB_LAUNCHED(ctx);
  auto* p_err = reinterpret_cast<volatile int*>(ctx->pin + kPinTc + 9);
  LAMB_CUDA(ctx, cudaMemcpyAsync((void*)p_err, d_err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  LAMB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  const int h_err = *p_err;
  if (h_err)
    return fail(ctx, LAMB_LEVEL_FAILURE, LAMB_TYPE_INTERNAL_ERROR,
                "mixed: tensor-core tile kernel stopped (code " + std::to_string(h_err) + ")");
  *ran = true;
  return LAMB_GPU_OK;
}

}  // namespace lamb

// ---- throughput probe of the tile kernel's instruction -------------------------------------
namespace lamb {
namespace tc {

// One CTA per SM: lane 0 of warp 0 issues `iters` rounds of tcgen05.mma
// kind::i8 (M = 128, K = 32, operands from one zeroed shared-memory stage),
// then waits for their completion (bounded).  N = 64 or 256: S(S+1)/2 MMAs
// of that width a round.  N = 0: the tile kernel's stage, the same nine
// MMAs (one per A digit plane and run of up to four B digit planes, N = 64
// to 256) with the same descriptors.
template <int N>
__global__ void __launch_bounds__(128, 1) k_tc_probe(int iters, int* err) {
  extern __shared__ unsigned char smem_raw[];
  // 1024-byte aligned base by pointer arithmetic on the shared array, so that
  // the compiler keeps the shared state space (shared loads and stores, not
  // generic ones)
  unsigned char* base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  __shared__ unsigned long long bar;
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < (N == 0 ? kStageBytes : kStageA + N * kK * kS) / 16; i += blockDim.x)
    reinterpret_cast<int4*>(base)[i] = make_int4(0, 0, 0, 0);
  if (threadIdx.x == 0) {
    bar_init(&bar, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base;
  if (warp == 0) {
    if (lane == 0) {
      constexpr uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                                 ((uint32_t)(N >> 3) << 17) | ((uint32_t)(kM >> 4) << 24);
      const uint32_t sa = smem_u32(base), sb = sa + kStageA;
      // B rows of N bytes: 64-byte swizzle for N = 64, 128-byte for N >= 128 (one atom of 128 per 128 columns)
      const uint32_t bsw = N == 64 ? 4u : 2u, bsbo = N == 64 ? 512u : 1024u, blbo = N == 64 ? 64u : 4096u;
      const int levels = N <= 64 ? kS : 2;  // 512 tensor-memory columns hold 512 / N accumulators
      if (N == 0) {
        for (int it = 0; it < iters; ++it)
#pragma unroll
          for (int p = 0; p < kS; ++p) {
            const uint64_t da = smem_desc(sa + p * kPlaneA, 128, 1024, 2);
#pragma unroll
            for (int q0 = 0; q0 < kS - p; q0 += 4) {
              const int nq = (kS - p - q0) < 4 ? (kS - p - q0) : 4;
              const uint64_t db = smem_desc(sb + q0 * kPlaneB, kPlaneB, 512, 4);
              mma_i8(tmem + (uint32_t)(64 * (p + q0)), da, db, idesc_i8(64 * nq), 1u);
            }
          }
      } else
      for (int it = 0; it < iters; ++it)
        for (int L = 0; L < kS; ++L)
          for (int p = 0; p <= L; ++p) {
            const uint64_t da = smem_desc(sa + p * kPlaneA, 128, 1024, 2);
            const uint64_t db = smem_desc(sb + (L - p) * (N * kK), blbo, bsbo, bsw);
            asm volatile(
                "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, q;\n\t}" ::"r"(tmem + (uint32_t)(N * (L % levels))),
                "l"(da), "l"(db), "r"(idesc), "r"(1u)
                : "memory");
          }
      mma_commit(&bar);
    }
    __syncwarp();
    const uint64_t t0 = now_ns();
    while (!bar_try(&bar, 0)) {
      if (now_ns() - t0 > 4000000000ull) {
        atomicOr(err, 1);
        break;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

template <int N>
static int32_t probe_n(int device, int reps, double* tops) {
  *tops = 0.0;
  if (cudaSetDevice(device) != cudaSuccess) return make_status(LAMB_LEVEL_FAILURE, LAMB_TYPE_EXTERNAL_ERROR);
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  const size_t smem = (N == 0 ? (size_t)kStageBytes : (size_t)kStageA + (size_t)N * kK * kS) + 1024;
  if (cudaFuncSetAttribute(k_tc_probe<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return make_status(LAMB_LEVEL_FAILURE, LAMB_TYPE_EXTERNAL_ERROR);
  int* err = nullptr;
  if (cudaMalloc(&err, sizeof(int)) != cudaSuccess) return make_status(LAMB_LEVEL_MEMORY, LAMB_TYPE_EXTERNAL_ERROR);
  cudaMemset(err, 0, sizeof(int));
  const int iters = 2000;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  k_tc_probe<N><<<sms, 128, smem>>>(10, err);  // warm-up
  float best = 1e30f;
  for (int r = 0; r < std::max(reps, 1); ++r) {
    cudaEventRecord(e0);
    k_tc_probe<N><<<sms, 128, smem>>>(iters, err);
    cudaEventRecord(e1);
    cudaEventSynchronize(e1);
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    best = std::min(best, ms);
  }
  int h_err = 0;
  const cudaError_t ce = cudaMemcpy(&h_err, err, sizeof(int), cudaMemcpyDeviceToHost);
  cudaFree(err);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (ce != cudaSuccess || h_err) return make_status(LAMB_LEVEL_FAILURE, LAMB_TYPE_EXTERNAL_ERROR);
  const double ops = 2.0 * kM * (N == 0 ? kN : N) * kK * (kS * (kS + 1) / 2) * (double)iters * sms;
  *tops = ops / (best * 1e-3) / 1e12;
  return LAMB_GPU_OK;
}

}  // namespace tc
}  // namespace lamb

// int8 tensor-core throughput of tcgen05.mma kind::i8, M = 128, K = 32, for
// N = 64, N = 256 (the widest instruction), or n = 0: the tile kernel's
// stage of nine MMAs of N = 64 to 256.
extern "C" int32_t lamb_probe_int8_tcgen05_tops(int32_t device, int32_t n, int32_t reps, double* tops) {
  if (!tops) return lamb::make_status(LAMB_LEVEL_FAILURE, LAMB_TYPE_WRONG_ARGS);
  if (n == 0) return lamb::tc::probe_n<0>(device, reps, tops);
  if (n == 64) return lamb::tc::probe_n<64>(device, reps, tops);
  if (n == 256) return lamb::tc::probe_n<256>(device, reps, tops);
  return lamb::make_status(LAMB_LEVEL_FAILURE, LAMB_TYPE_WRONG_ARGS);
}
