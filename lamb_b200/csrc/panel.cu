// FP64 block product on group tiles (the numeric body of the reference's
// sector_multiply stub, src/lamb_multiplication.F90:206-225, for whole
// groups of atoms at a time).
//
// A block of a few rows is far below what feeds the FP64 tensor pipe: with one
// warp per C block every MMA needs its own gather of operand fragments, half of
// each 16-row tile is padding, and a 16-byte stack entry is written and read
// per product.  Consecutive atoms that couple to nearly the same atoms (an O and
// its two H) are therefore taken as one group of at most 24 element rows.  Both
// operands are packed once per multiply into panels: for a group and every
// inner group it couples to (a superblock), the inner element rows, each as 24
// consecutive doubles (one per element row of the group, zero where the block
// is absent).  A warp then computes one tile (group x group) of C: it
// intersects the two groups' superblocks, brings in one pair after the other in
// ascending order by two bulk copies and runs mma.m8n8k4 on four rows at a
// time, 3 x 3 MMAs for five shared-memory loads.  Rows of an absent block add
// exact zeros and the tensor pipe adds a row's products one after the other, so
// a C element is the same sum, in the same order, as over its own block
// products: results are the stack kernel's bit for bit.
//
// What bounds it: the FP64 tensor pipe (37.1 TFLOP/s, 16 cycles per m8n8k4).
// At 6,144 waters (cutoff 8) the multiply's 775 GFLOP took 103 ms in the stack
// kernel and 22 ms in its fills; here 48 ms and 2.6 ms for the panels (16.1
// TFLOP/s).  55 to 60 % of the executed MMA work is useful (absent blocks of a
// superblock, 23 of 24 rows), the pipe is about 70 % busy; the rest is a warp's
// own serial work per tile (listing, first copies, writing out), which three
// warps per sub-partition hide only partly.  Tried and slower (768 waters,
// cutoff 7; now 3.2 ms): fragments straight from global memory 7.9 ms, 4 x 4
// tiles behind one copy pipeline 7.4 ms (its warps wait for one another), 2 x 2
// tiles in four such teams 4.3 ms, sixteen warps with rings of 8-row copies
// 4.5 ms (issue-bound).
//
// The product filter is applied exactly: superblock pairs in which every
// product passes run as above; where some products fall below eps, the
// passing ones run in passes whose fragments are masked to the row and column
// atoms they concern.
#include <cub/cub.cuh>

#include <algorithm>
#include <numeric>

#include "multiply.cuh"
#include "panel.cuh"
#include "ptx.cuh"

namespace lamb {

namespace {

constexpr int kTileWarps = 12;   // what two stages of 24 x 24 superblock pairs leave room for
constexpr int kRounds = 4;       // of 32 superblocks listed at a time
constexpr int kSuper = 16;       // macro rows (of two groups) of one super row: its panels stay in L2
constexpr int kPackWarps = 8;
constexpr int kW = kGrpRows;     // doubles of one panel row
constexpr int kRowBytes = 8 * kW;

// ---- arguments ------------------------------------------------------------------------
struct SideArgs {
  const int64_t* row_p;
  const int32_t* col;
  const int64_t* off;
  const double* data;
  const double* norms;
  const int8_t* row_bs;
  const int8_t* col_bs;
  int32_t n_rows, rows_out;
  const int32_t *o_first, *o_map, *o_arow, *o_rows;
  const int32_t *i_first, *i_map, *i_arow, *i_rows;
  int32_t n_out, words, n_sb;
  int32_t* hist;
  uint32_t* bm;
  int32_t* pre;
  int32_t* ptr;
  int32_t* kc;
  int32_t* sbg;
  uint32_t* mask;
  double2* nrange;
  double* nrm;
  double* panel;
};
struct PairArgs {
  SideArgs s[2];
  int32_t kstride, nk_max, na_max[2], n_in;
  int64_t* totals;
};

__device__ __forceinline__ int w8_of(int rows) { return (rows + 7) >> 3; }

// ---- superblock index -------------------------------------------------------------------
__global__ void k_panel_bits(const __grid_constant__ PairArgs p) {
  const SideArgs& s = p.s[blockIdx.y];
  const int lane = threadIdx.x & 31;
  for (int64_t r = global_warp(); r < s.n_rows; r += grid_warps()) {
    const int gr = s.rows_out ? s.o_map[r] : s.i_map[r];
    for (int64_t b = s.row_p[r] + lane; b < s.row_p[r + 1]; b += 32) {
      const int c = s.col[b];
      const int g = s.rows_out ? gr : s.o_map[c], k = s.rows_out ? s.i_map[c] : gr;
      uint32_t* w = &s.bm[(int64_t)g * s.words + (k >> 5)];
      const uint32_t bit = 1u << (k & 31);
      if (!(*w & bit)) atomicOr(w, bit);
    }
  }
}

// Superblocks before every word of a group; the group's count goes to ptr, the
// count of every inner group to hist.
__global__ void k_panel_prefix(const __grid_constant__ PairArgs p) {
  const SideArgs& s = p.s[blockIdx.y];
  const int lane = threadIdx.x & 31;
  for (int64_t g = global_warp(); g < s.n_out; g += grid_warps()) {
    int carry = 0;
    for (int w0 = 0; w0 < s.words; w0 += 32) {
      const int w = w0 + lane;
      uint32_t bits = w < s.words ? s.bm[g * s.words + w] : 0u;
      const int n = __popc(bits);
      for (; bits; bits &= bits - 1u) atomicAdd(&s.hist[32 * w + __ffs(bits) - 1], 1);
      const int incl = warp_incl_scan(n, lane);
      if (w < s.words) s.pre[g * s.words + w] = carry + incl - n;
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) s.ptr[g] = carry;
  }
}

// One CTA per operand: counts -> first superblock of every group.  Totals:
// superblocks of either operand, and superblock pairs of the product.
__global__ void __launch_bounds__(1024) k_panel_scan(const __grid_constant__ PairArgs p) {
  const SideArgs& s = p.s[blockIdx.x];
  typedef cub::BlockScan<int, 1024> BS;
  __shared__ typename BS::TempStorage ts;
  long long carry = 0;  // the host refuses a total beyond 32 bits
  for (int g0 = 0; g0 < s.n_out; g0 += 1024) {
    const int g = g0 + threadIdx.x;
    int e, a;
    BS(ts).ExclusiveSum(g < s.n_out ? s.ptr[g] : 0, e, a);
    __syncthreads();
    if (g < s.n_out) s.ptr[g] = (int)(carry + e);
    carry += a;
  }
  if (threadIdx.x == 0) {
    s.ptr[s.n_out] = (int)carry;
    p.totals[blockIdx.x] = carry;
  }
  if (blockIdx.x == 0) {
    typedef cub::BlockReduce<long long, 1024> BR;
    __shared__ typename BR::TempStorage tr;
    long long n = 0;
    for (int k = threadIdx.x; k < p.n_in; k += 1024) n += (long long)p.s[0].hist[k] * p.s[1].hist[k];
    n = BR(tr).Sum(n);
    if (threadIdx.x == 0) p.totals[2] = n;
  }
}

__global__ void k_panel_list(const __grid_constant__ PairArgs p) {
  const SideArgs& s = p.s[blockIdx.y];
  const int lane = threadIdx.x & 31;
  for (int64_t g = global_warp(); g < s.n_out; g += grid_warps()) {
    const int p0 = s.ptr[g];
    for (int w = lane; w < s.words; w += 32) {
      uint32_t bits = s.bm[g * s.words + w];
      int q = p0 + s.pre[g * s.words + w];
      while (bits) {
        s.kc[q] = 32 * w + __ffs(bits) - 1;
        s.sbg[q] = (int32_t)g;
        bits &= bits - 1u;
        ++q;
      }
    }
  }
}

// ---- panels -----------------------------------------------------------------------------
// One warp per superblock: the blocks of its (out atom, inner atom) pairs by
// one binary search per matrix row, then the inner element rows one after the
// other, 192 bytes each (24 doubles; zero beyond the group's rows, where a
// block is absent, and in the rows that pad the superblock to a multiple of
// four).  Element e of row r sits at position e ^ 4 ((r / 2) % 2): the eight
// bytes a warp's lanes take from four rows then fall into distinct banks.
template <bool FILT>
__global__ void __launch_bounds__(32 * kPackWarps) k_panel_pack(const __grid_constant__ PairArgs p) {
  const SideArgs& s = p.s[blockIdx.y];
  __shared__ long long blk_all[kPackWarps][kGrpAtoms * kGrpAtoms];
  const int lane = threadIdx.x & 31;
  long long* blk = blk_all[threadIdx.x >> 5];
  bool odd = false;  // an infinity or a NaN among the values
  for (int64_t sb = global_warp(); sb < s.n_sb; sb += grid_warps()) {
    const int g = s.sbg[sb], kg = s.kc[sb];
    const int o0 = s.o_first[g], no = s.o_first[g + 1] - o0;
    const int k0 = s.i_first[kg], nk = s.i_first[kg + 1] - k0;
    const int rows_i = s.i_rows[kg];
    // blocks of the pairs, at blk[out atom * 8 + inner atom]
    const int n_search = s.rows_out ? no : nk, n_run = s.rows_out ? nk : no;
    double lo_n = INFINITY, hi_n = 0.0;
    if (lane < n_search) {
      const int r = (s.rows_out ? o0 : k0) + lane, c0 = s.rows_out ? k0 : o0;
      const int64_t end = s.row_p[r + 1];
      int64_t pos = lower_col(s.col, s.row_p[r], end, c0);
      for (int x = 0; x < n_run; ++x) {
        const bool hit = pos < end && s.col[pos] == c0 + x;
        const int o = s.rows_out ? lane : x, k = s.rows_out ? x : lane;
        blk[o * kGrpAtoms + k] = hit ? s.off[pos] : -1;
        if (FILT) {
          const bool real = hit && s.row_bs[r] > 0 && s.col_bs[c0 + x] > 0;
          const double nv = real ? s.norms[pos] : -1.0;
          s.nrm[(sb * p.na_max[blockIdx.y] + o) * p.nk_max + k] = nv;
          if (real) {
            lo_n = fmin(lo_n, nv);
            hi_n = fmax(hi_n, nv);
          }
        }
        pos += hit;
      }
    }
    __syncwarp();
    // this lane as an inner element row, and as an element of the group
    int ki = 0, ke = 0, kb = 0, oi = -1, oe = 0, ob = 0;
    for (int x = 0; x < nk; ++x) {
      const int a = s.i_arow[k0 + x], b = s.rows_out ? s.col_bs[k0 + x] : s.row_bs[k0 + x];
      if (lane >= a && lane < a + b) { ki = x; ke = lane - a; kb = b; }
    }
    for (int x = 0; x < no; ++x) {
      const int a = s.o_arow[o0 + x], b = s.rows_out ? s.row_bs[o0 + x] : s.col_bs[o0 + x];
      if (lane >= a && lane < a + b) { oi = x; oe = lane - a; ob = b; }
    }
    bool any = false;
    if (lane < rows_i)
      for (int x = 0; x < no; ++x) any |= blk[x * kGrpAtoms + ki] >= 0;
    const uint32_t m = __ballot_sync(0xffffffffu, any);
    if (FILT) {
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        lo_n = fmin(lo_n, __shfl_xor_sync(0xffffffffu, lo_n, o));
        hi_n = fmax(hi_n, __shfl_xor_sync(0xffffffffu, hi_n, o));
      }
    }
    if (lane == 0) {
      s.mask[sb] = m;
      if (FILT) s.nrange[sb] = make_double2(lo_n, hi_n);
    }
    // the element stored at this lane's position in rows with the other bit
    const int oi4 = __shfl_xor_sync(0xffffffffu, oi, 4), oe4 = __shfl_xor_sync(0xffffffffu, oe, 4);
    const int ob4 = __shfl_xor_sync(0xffffffffu, ob, 4);
    double* dst = s.panel + (size_t)sb * p.kstride * kW;
#pragma unroll 4
    for (int kk = 0; kk < p.kstride; ++kk) {
      const int xk = __shfl_sync(0xffffffffu, ki, kk), xe = __shfl_sync(0xffffffffu, ke, kk);
      const int xb = __shfl_sync(0xffffffffu, kb, kk);
      const bool sw = (kk >> 1) & 1;
      const int yi = sw ? oi4 : oi, ye = sw ? oe4 : oe, yb = sw ? ob4 : ob;
      double v = 0.0;
      if (yi >= 0 && kk < rows_i) {
        const long long o = blk[yi * kGrpAtoms + xk];
        if (o >= 0) v = __ldg(s.data + o + (s.rows_out ? ye + xe * yb : xe + ye * xb));
      }
      if (lane < kW) dst[kk * kW + lane] = v;
      odd |= !(fabs(v) < INFINITY);
    }
    __syncwarp();
  }
  if (odd) p.totals[3] = 1;
}

// ---- macro tiles ------------------------------------------------------------------------
// Super row S holds the row groups of ranks 32 S .. 32 S + 31 (16 macro rows
// of 2).  For every macro column the 16 x 4 bits say which tiles hold a C block.
struct MaskArgs {
  const int64_t* row_p;
  const int32_t* col;
  const int32_t *r_first, *r_order, *c_map, *c_rank;
  int32_t n_rg, n_mj;
  const int32_t* c_order;
  uint2* masks;     // [n_super * n_mj]
  int32_t* count;   // [n_super + 1] tiles, then their exclusive scan
  int2* items;      // (row group, column group) of every tile
};

__global__ void __launch_bounds__(512) k_panel_masks(const __grid_constant__ MaskArgs p) {
  extern __shared__ uint32_t msk[];  // [n_mj][2]
  const int S = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int x = threadIdx.x; x < 2 * p.n_mj; x += blockDim.x) msk[x] = 0u;
  __syncthreads();
  for (int q = warp; q < 2 * kSuper; q += nw) {
    const int rk = 2 * kSuper * S + q;
    if (rk >= p.n_rg) break;
    const int g = p.r_order[rk];
    const int64_t b1 = p.row_p[p.r_first[g + 1]];
    const int sh = 2 * (q & 15);
    for (int64_t b = p.row_p[p.r_first[g]] + lane; b < b1; b += 32) {
      const int c = p.c_rank[p.c_map[p.col[b]]];
      uint32_t* w = &msk[2 * (c >> 1) + (q >> 4)];
      const uint32_t bit = 1u << (sh + (c & 1));
      if (!(*w & bit)) atomicOr(w, bit);
    }
  }
  __syncthreads();
  int n = 0;
  for (int x = threadIdx.x; x < p.n_mj; x += blockDim.x) {
    const uint2 v = reinterpret_cast<const uint2*>(msk)[x];
    p.masks[(int64_t)S * p.n_mj + x] = v;
    n += __popc(v.x) + __popc(v.y);
  }
  typedef cub::BlockReduce<int, 512> BR;
  __shared__ typename BR::TempStorage ts;
  n = BR(ts).Sum(n);
  if (threadIdx.x == 0) p.count[S] = n;
}

__global__ void __launch_bounds__(1024) k_panel_mask_scan(int32_t n, int32_t* __restrict__ v) {
  typedef cub::BlockScan<int, 1024> BS;
  __shared__ typename BS::TempStorage ts;
  int carry = 0;
  for (int x0 = 0; x0 < n; x0 += 1024) {
    const int x = x0 + threadIdx.x;
    int e, a;
    BS(ts).ExclusiveSum(x < n ? v[x] : 0, e, a);
    __syncthreads();
    if (x < n) v[x] = carry + e;
    carry += a;
  }
  if (threadIdx.x == 0) v[n] = carry;
}

// Tiles of a super row by macro column, then macro row: warps that run side by
// side share the column panels while the super row's panels stay in L2.
__global__ void __launch_bounds__(256) k_panel_items(const __grid_constant__ MaskArgs p) {
  typedef cub::BlockScan<int, 256> BS;
  __shared__ typename BS::TempStorage ts;
  __shared__ int32_t rg[2 * kSuper];
  const int S = blockIdx.x;
  if (threadIdx.x < 2 * kSuper) {
    const int rk = 2 * kSuper * S + threadIdx.x;
    rg[threadIdx.x] = rk < p.n_rg ? p.r_order[rk] : -1;
  }
  int pos = p.count[S];
  for (int x0 = 0; x0 < p.n_mj; x0 += 256) {
    const int x = x0 + threadIdx.x;
    uint2 v = make_uint2(0, 0);
    if (x < p.n_mj) v = p.masks[(int64_t)S * p.n_mj + x];
    int e, a;
    BS(ts).ExclusiveSum(__popc(v.x) + __popc(v.y), e, a);
    __syncthreads();
    int q = pos + e;
    for (int h = 0; h < 2; ++h)
      for (uint32_t w = h ? v.y : v.x; w; w &= w - 1u) {
        const int bit = __ffs(w) - 1;
        p.items[q++] = make_int2(rg[16 * h + (bit >> 1)], p.c_order[2 * x + (bit & 1)]);
      }
    pos += a;
  }
}

// ---- tiles --------------------------------------------------------------------------------
struct TileSide {
  const uint32_t* bm;
  const int32_t *pre, *ptr;
  const uint32_t* mask;
  const double2* nrange;
  const double* nrm;
  const double* panel;
  const int32_t *first, *rows;
  const uint16_t* geo;  // GroupTab::geo
  int32_t max_atoms;
};
struct TileArgs {
  TileSide s[2];
  int32_t words, kstride;
  // C: its pattern as a bitmap over the columns with the row's blocks before every word
  int32_t c_words;
  const uint32_t* c_bm;
  const int32_t* c_pre;
  const int64_t* row_p;
  const int64_t* off;
  double* data;
  double* c_nrm;
  // product filter
  double eps;
  const int32_t *kc_a, *i_first, *i_arow;
  const int8_t* i_bs;
  int32_t nk_max;
  const int2* items;
  const int32_t* seg;  // first item of every super row
  int32_t s0, s1;
  int32_t* head;  // items taken
  uint64_t wait_ns;  // longest wait for a copy
  int* err;
};

struct __align__(128) WarpSm {
  double ring[2][2][kW * kW];
  unsigned long long full[2];
};
constexpr size_t kTileSmem = sizeof(WarpSm) * kTileWarps + 128;
static_assert(kTileSmem <= 232448, "the tile kernel exceeds the shared memory of one CTA");

// Waits for the phase of the given parity, at most limit_ns; then records
// `code` and stops the CTA.  The answer is the whole warp's: lanes that left
// by themselves would be missing from the shuffles of the others (389 waters
// with 23-row O blocks: 8.39 ms with an answer a lane, 7.93 with the votes).  A
// limit of 0 counts every wait as run out, without looking.
__device__ __forceinline__ bool tile_wait(unsigned long long* b, uint32_t parity, uint64_t limit_ns, int* abort,
                                          int* err, int code) {
  if (__all_sync(0xffffffffu, limit_ns != 0 && bar_try(b, parity))) return true;
  const uint64_t t0 = now_ns();
  for (;;) {
    if (__all_sync(0xffffffffu, limit_ns != 0 && bar_try_sleep(b, parity, 20000u))) return true;
    if (__any_sync(0xffffffffu, *(volatile int*)abort)) return false;
    if (__any_sync(0xffffffffu, now_ns() - t0 >= limit_ns)) {
      if ((threadIdx.x & 31) == 0) {
        atomicOr(err, code);
        *(volatile int*)abort = 1;
      }
      return false;
    }
  }
}

__device__ __forceinline__ void dmma884(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// Tile row (0-based) that fragment position x (0..7) of 8-row slab i stands
// for, with T slabs: two slabs share a 16-byte load.  Columns lie in order.
__device__ __forceinline__ int frag_row(int i, int x, int T) {
  return (i == T - 1 && (T & 1)) ? 8 * i + x : 16 * (i >> 1) + 2 * x + (i & 1);
}

// Adds the products of group q of four rows (rows 4 q + lane % 4) of the two
// parts.  pa, ps: this lane's positions in the row part (two slabs share a
// 16-byte load, the third is single), pb: in the column part.  DYN: mt x nt
// slabs instead of 3 x 3.  MASK: only rows [k0, k1), the row atoms rset and the
// column atoms cset take part.
template <bool DYN, bool MASK>
__device__ __forceinline__ void run_group(double (&acc)[3][3][2], int q, const double* pa, const double* ps,
                                          const double* pb, int mt, int nt, int k0 = 0, int k1 = 0, uint32_t rset = 0,
                                          uint32_t cset = 0, uint32_t atoms = 0) {
  const double2 va = *reinterpret_cast<const double2*>(pa + q * (4 * kW));
  const double wa = ps[q * (4 * kW)];
  double a0 = DYN && mt == 1 ? wa : va.x, a1 = va.y, a2 = wa;
  double b0 = pb[q * (4 * kW)], b1 = pb[q * (4 * kW) + 8], b2 = pb[q * (4 * kW) + 16];
  if (MASK) {
    const int k = 4 * q + (threadIdx.x & 3);
    const bool in = k >= k0 && k < k1;
    if (!in || !((rset >> (atoms & 7)) & 1u)) a0 = 0.0;
    if (!in || !((rset >> ((atoms >> 4) & 7)) & 1u)) a1 = 0.0;
    if (!in || !((rset >> ((atoms >> 8) & 7)) & 1u)) a2 = 0.0;
    if (!((cset >> ((atoms >> 16) & 7)) & 1u)) b0 = 0.0;
    if (!((cset >> ((atoms >> 20) & 7)) & 1u)) b1 = 0.0;
    if (!((cset >> ((atoms >> 24) & 7)) & 1u)) b2 = 0.0;
  }
  dmma884(acc[0][0], a0, b0);
  if (!DYN || nt > 1) dmma884(acc[0][1], a0, b1);
  if (!DYN || nt > 2) dmma884(acc[0][2], a0, b2);
  if (!DYN || mt > 1) {
    dmma884(acc[1][0], a1, b0);
    if (!DYN || nt > 1) dmma884(acc[1][1], a1, b1);
    if (!DYN || nt > 2) dmma884(acc[1][2], a1, b2);
  }
  if (!DYN || mt > 2) {
    dmma884(acc[2][0], a2, b0);
    if (!DYN || nt > 1) dmma884(acc[2][1], a2, b1);
    if (!DYN || nt > 2) dmma884(acc[2][2], a2, b2);
  }
}

// All groups of four rows that have a row in m.  A warp issues a dependent
// instruction every four to six cycles, so the loop is unrolled with constant
// offsets: the MMAs (16 cycles each) then cover the loads and the tests.
template <bool DYN>
__device__ __forceinline__ void run_rows(double (&acc)[3][3][2], uint32_t m, const double* pa, const double* ps,
                                         const double* pb, int mt, int nt) {
#pragma unroll
  for (int q = 0; q < kW / 4; ++q)
    if (m & (0xfu << (4 * q))) run_group<DYN, false>(acc, q, pa, ps, pb, mt, nt);
}

// C block of the tile's atom pair x (row atom x / nb, column atom x % nb): its
// index (32 bits: kPanelMaxBlocks), and in *hit whether it is in the pattern.
__device__ __forceinline__ int find_block(const TileArgs& p, int a0, int b0, int nb, int x, uint32_t* hit) {
  const int a = x / nb, c = b0 + x - a * nb;
  const int64_t r = a0 + a, w = r * p.c_words + (c >> 5);
  const uint32_t word = p.c_bm[w], bit = 1u << (c & 31);
  *hit = word & bit;
  return (int)p.row_p[r] + p.c_pre[w] + __popc(word & (bit - 1u));
}

// Warps are independent: each takes one tile (group x group) after another
// from a queue, lists the inner groups both sides couple to, copies their
// superblocks (one bulk copy a side) into two stages of its own shared memory
// and runs the MMAs on one stage while the other fills.  What a warp waits for
// (its tile's list, the first copies, writing the tile out) overlaps the MMAs
// of the other warps of its sub-partition.
template <bool FILT>
__global__ void __launch_bounds__(32 * kTileWarps, 1) k_panel_tiles(const __grid_constant__ TileArgs p) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  WarpSm& ws = reinterpret_cast<WarpSm*>(smem)[warp];
  int* abort = reinterpret_cast<int*>(smem + sizeof(WarpSm) * kTileWarps);
  if (threadIdx.x == 0) *abort = 0;
  if (lane == 0) {
    bar_init(&ws.full[0], 1);
    bar_init(&ws.full[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const int it1 = p.seg[p.s1], it0 = p.seg[p.s0];
  const uint32_t bytes = (uint32_t)p.kstride * kRowBytes;
  const int g = lane >> 2, t = lane & 3;
  const int sw = (t & 2) << 1;  // this lane's rows are 4 q + t
  const int pair = t * kW + ((2 * g) ^ sw), col = t * kW + (g ^ sw);
  uint32_t ph = 0;  // parity of either stage's barrier
  int slot = 0;
  // the item after this one is read while a tile is computed
  int nx = 0;
  if (lane == 0) nx = it0 + atomicAdd(p.head, 1);
  nx = __shfl_sync(0xffffffffu, nx, 0);
  int2 item = nx < it1 ? p.items[nx] : make_int2(-1, 0);
  while (item.x >= 0) {
    const int I = item.x, J = item.y;
    if (lane == 0) nx = it0 + atomicAdd(p.head, 1);
    const int a_ptr = p.s[0].ptr[I], la = p.s[0].ptr[I + 1] - a_ptr, b_ptr = p.s[1].ptr[J];
    const int rows = p.s[0].rows[I], cols = p.s[1].rows[J];
    const int a0 = p.s[0].first[I], na = p.s[0].first[I + 1] - a0;
    const int b0 = p.s[1].first[J], nb = p.s[1].first[J + 1] - b0;
    const int row_geo = lane < kW ? p.s[0].geo[I * kW + lane] : 0;
    const int col_geo = lane < kW ? p.s[1].geo[J * kW + lane] : 0;
    const int mt = w8_of(rows), nt = w8_of(cols);
    const bool full = mt == 3 && nt == 3;
    const int single = t * kW + ((8 * max(mt - 1, 0) + g) ^ sw);
    double acc[3][3][2];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    uint32_t atoms = 0;
    if (FILT) {
      // row / column atom of every fragment element: 4 bits a slab
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int xa = __shfl_sync(0xffffffffu, row_geo, i < mt ? frag_row(i, g, mt) : 0) & 7;
        const int xb = __shfl_sync(0xffffffffu, col_geo, 8 * i + g) & 7;
        atoms |= (xa << (4 * i)) | (xb << (16 + 4 * i));
      }
    }
    // ---- superblock pairs of the two groups, 32 of I's superblocks a round, kRounds rounds at a time ----
    int e0 = -32 * kRounds, rd = kRounds - 1;
    uint32_t hits = 0, m[kRounds];
    int sb[kRounds];
    bool part[FILT ? kRounds : 1];
    uint32_t nm = 0;
    int nsa = 0, nsb = 0;
    bool nsplit = false;
    auto advance = [&]() -> bool {
      while (!hits) {
        if (++rd == kRounds) {
          rd = 0;
          e0 += 32 * kRounds;
          if (e0 >= la) return false;
          int kc[kRounds];
          uint32_t word[kRounds], ma[kRounds];
#pragma unroll
          for (int r = 0; r < kRounds; ++r) {
            const int e = e0 + 32 * r + lane;
            kc[r] = e < la ? p.kc_a[a_ptr + e] : -1;
            ma[r] = e < la ? p.s[0].mask[a_ptr + e] : 0u;
          }
#pragma unroll
          for (int r = 0; r < kRounds; ++r) {
            word[r] = 0;
            sb[r] = 0;
            if (kc[r] >= 0) {
              const int64_t w = (int64_t)J * p.words + (kc[r] >> 5);
              word[r] = p.s[1].bm[w];
              sb[r] = p.s[1].pre[w];
            }
          }
#pragma unroll
          for (int r = 0; r < kRounds; ++r) {
            const uint32_t bit = 1u << (kc[r] & 31);
            m[r] = 0;
            if (word[r] & bit) {
              sb[r] += b_ptr + __popc(word[r] & (bit - 1u));
              m[r] = ma[r] & p.s[1].mask[sb[r]];
            }
          }
          if (FILT) {
#pragma unroll
            for (int r = 0; r < kRounds; ++r)
              if (m[r]) {
                const double2 ra = p.s[0].nrange[a_ptr + e0 + 32 * r + lane], rn = p.s[1].nrange[sb[r]];
                if (ra.y * rn.y < p.eps) m[r] = 0;  // every product falls below eps
                else part[r] = ra.x * rn.x < p.eps;
              }
          }
        }
        uint32_t x = 0;
#pragma unroll
        for (int r = 0; r < kRounds; ++r)
          if (r == rd) x = m[r];
        hits = __ballot_sync(0xffffffffu, x != 0);
      }
      const int src = __ffs(hits) - 1;
      hits &= hits - 1u;
      uint32_t x = 0;
      int y = 0;
      bool z = false;
#pragma unroll
      for (int r = 0; r < kRounds; ++r)
        if (r == rd) {
          x = m[r];
          y = sb[r];
          if (FILT) z = part[r];
        }
      nm = __shfl_sync(0xffffffffu, x, src);
      nsb = __shfl_sync(0xffffffffu, y, src);
      if (FILT) nsplit = __shfl_sync(0xffffffffu, (int)z, src);
      nsa = a_ptr + e0 + 32 * rd + src;
      return true;
    };
    auto issue = [&](int s) {
      __syncwarp();  // every lane is past what the stage held
      if (lane == 0) {
        bar_expect(&ws.full[s], 2 * bytes);
        bulk_copy(smem_u32(ws.ring[s][0]), p.s[0].panel + (size_t)nsa * p.kstride * kW, bytes, &ws.full[s]);
        bulk_copy(smem_u32(ws.ring[s][1]), p.s[1].panel + (size_t)nsb * p.kstride * kW, bytes, &ws.full[s]);
      }
    };
    bool have = mt > 0 && nt > 0 && advance();
    if (have) issue(slot);
    nx = __shfl_sync(0xffffffffu, nx, 0);
    item = nx < it1 ? p.items[nx] : make_int2(-1, 0);
    // C block of atom pair `lane` (row atom major): index, data offset (-1: none)
    int cid = 0;
    uint32_t look = 0;
    long long coff = -1;
    if (lane < na * nb) cid = find_block(p, a0, b0, nb, lane, &look);
    if (look) coff = p.off[cid];
    bool ok = true;
    while (have) {
      const uint32_t cm = nm;
      const int csa = nsa, csb = nsb;
      const bool csplit = nsplit;
      have = advance();
      if (have) issue(slot ^ 1);
      if (!(ok = tile_wait(&ws.full[slot], (ph >> slot) & 1u, p.wait_ns, abort, p.err, 1))) break;
      ph ^= 1u << slot;
      const double* pa = ws.ring[slot][0] + pair;
      const double* ps = ws.ring[slot][0] + single;
      const double* pb = ws.ring[slot][1] + col;
      if (!FILT || !csplit) {
        if (full)
          run_rows<false>(acc, cm, pa, ps, pb, 3, 3);
        else
          run_rows<true>(acc, cm, pa, ps, pb, mt, nt);
      } else if (FILT) {
        // some products of this superblock pair fall below eps: one pass per
        // inner atom and set of passing columns, with the row atoms it serves
        const int kg = p.kc_a[csa], k0 = p.i_first[kg], nk = p.i_first[kg + 1] - k0;
        for (int x = 0; x < nk; ++x) {
          const int kr = p.i_arow[k0 + x], ke = kr + p.i_bs[k0 + x];
          if (ke == kr || !((cm >> kr) & 1u)) continue;
          // passing (row atom, column atom) pairs: 8 bits per row atom
          const int cb = lane & 7;
          const double nbv = cb < nb ? p.s[1].nrm[((int64_t)csb * p.s[1].max_atoms + cb) * p.nk_max + x] : -1.0;
          uint32_t kp[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int ra = (lane >> 3) + 4 * h;
            const double nav = ra < na ? p.s[0].nrm[((int64_t)csa * p.s[0].max_atoms + ra) * p.nk_max + x] : -1.0;
            kp[h] = __ballot_sync(0xffffffffu, nav >= 0.0 && nbv >= 0.0 && !(nav * nbv < p.eps));
          }
          uint32_t todo = 0;
          for (int a = 0; a < kGrpAtoms; ++a)
            if ((kp[a >> 2] >> (8 * (a & 3))) & 0xffu) todo |= 1u << a;
          while (todo) {
            const int a1 = __ffs(todo) - 1;
            const uint32_t cset = (kp[a1 >> 2] >> (8 * (a1 & 3))) & 0xffu;
            uint32_t rset = 0;
            for (int a = a1; a < kGrpAtoms; ++a)
              if (((todo >> a) & 1u) && ((kp[a >> 2] >> (8 * (a & 3))) & 0xffu) == cset) rset |= 1u << a;
            todo &= ~rset;
#pragma unroll 1
            for (int q = kr >> 2; 4 * q < ke; ++q)
              run_group<true, true>(acc, q, pa, ps, pb, mt, nt, kr, ke, rset, cset, atoms);
          }
        }
      }
      slot ^= 1;
    }
    if (!ok) {  // copies still in flight land before the CTA gives up its shared memory
      for (int s = 0; s < 2; ++s) {
        if (s == (slot ^ 1) && !have) continue;  // nothing on its way to the other stage
        const uint64_t t0 = now_ns();
        while (!bar_try_sleep(&ws.full[s], (ph >> s) & 1u, 20000u))
          if (now_ns() - t0 > 2000000000ull) break;
      }
      break;
    }
    // ---- the tile through shared memory, then a lane writes its row of every
    // column (a column of a block is one run of consecutive stores) ----
    if (mt > 0 && nt > 0) {
      __syncwarp();
      double* stg = ws.ring[0][0];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
          if (i < mt && j < nt) {
            const int r = frag_row(i, g, mt);
            stg[(8 * j + 2 * t) * kW + r] = acc[i][j][0];
            stg[(8 * j + 2 * t + 1) * kW + r] = acc[i][j][1];
          }
      const bool in = row_geo & kGeoRow;
      const int ra = row_geo & 7, rr = (row_geo >> 3) & 31, bi = (row_geo >> 8) & 31;
      const int rem = in ? bi - 1 - rr : 0;
      long long coff2 = -1;  // atom pairs beyond the 32nd
      int cid2 = 0;
      if (na * nb > 32) {
        uint32_t word = 0;
        if (lane + 32 < na * nb) cid2 = find_block(p, a0, b0, nb, lane + 32, &word);
        if (word) coff2 = p.off[cid2];
      }
      __syncwarp();
      int c = 0;
      for (int b = 0; c < cols; ++b) {
        const int bj = (__shfl_sync(0xffffffffu, col_geo, c) >> 8) & 31, x = ra * nb + (__shfl_sync(0xffffffffu, col_geo, c) & 7);
        long long o = __shfl_sync(0xffffffffu, coff, x & 31);
        int cn = __shfl_sync(0xffffffffu, cid, x & 31);
        if (na * nb > 32) {
          const long long o2 = __shfl_sync(0xffffffffu, coff2, x & 31);
          const int n2 = __shfl_sync(0xffffffffu, cid2, x & 31);
          if (x >= 32) {
            o = o2;
            cn = n2;
          }
        }
        const bool put = in && o >= 0;
        double* dst = p.data + (put ? o + rr : 0);
        const double* from = stg + c * kW + (lane < kW ? lane : 0);
        double sq = 0.0;
#pragma unroll 4
        for (int q = 0; q < bj; ++q) {
          const double v = from[q * kW];
          if (put) __stcs(dst + q * bi, v);
          sq = __fma_rn(v, v, sq);
        }
        c += bj;
        if (p.c_nrm) {
          // norm: the sum over the block's rows, one lane each
#pragma unroll
          for (int s = 1; s < 32; s <<= 1) {
            const double w = __shfl_down_sync(0xffffffffu, sq, s);
            if (s <= rem) sq += w;
          }
          if (put && rr == 0) p.c_nrm[cn] = __dsqrt_rn(sq);
        }
      }
      // the next tile's copies overwrite what was written and read here
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
  }
}

}  // namespace

// ---- groups of atoms ----------------------------------------------------------------------
namespace {

// Blocks per column, and rows that hold both a column and the next one.
__global__ void k_grp_cols(int32_t n_rows, const int64_t* __restrict__ row_p, const int32_t* __restrict__ col,
                           int32_t* __restrict__ cnt, int32_t* __restrict__ both) {
  const int lane = threadIdx.x & 31;
  for (int64_t r = global_warp(); r < n_rows; r += grid_warps()) {
    const int64_t end = row_p[r + 1];
    for (int64_t b = row_p[r] + lane; b < end; b += 32) {
      const int c = col[b];
      atomicAdd(&cnt[c], 1);
      if (b + 1 < end && col[b + 1] == c + 1) atomicAdd(&both[c], 1);
    }
  }
}

// Blocks per row, and columns held by both a row and the next one.
__global__ void k_grp_rows(int32_t n_rows, const int64_t* __restrict__ row_p, const int32_t* __restrict__ col,
                           int32_t* __restrict__ cnt, int32_t* __restrict__ both) {
  const int lane = threadIdx.x & 31;
  for (int64_t r = global_warp(); r < n_rows; r += grid_warps()) {
    const int64_t b0 = row_p[r], b1 = row_p[r + 1], e1 = r + 1 < n_rows ? row_p[r + 2] : b1;
    int n = 0;
    for (int64_t x = b0; x < b1; x += 32) {
      bool hit = false;
      if (x + lane < b1) {
        const int c = col[x + lane];
        const int64_t y = lower_col(col, b1, e1, c);
        hit = y < e1 && col[y] == c;
      }
      n += __popc(__ballot_sync(0xffffffffu, hit));
    }
    if (lane == 0) {
      cnt[r] = (int32_t)(b1 - b0);
      both[r] = n;
    }
  }
}

// Cuts the atoms 0 .. n - 1 into runs: at most kGrpRows rows and kGrpAtoms
// atoms, neighbours only joined when at least
// half of the longer one's blocks are shared, and among those cuts the one
// whose runs share the most blocks (so that an O and its two H stay together
// whatever precedes them).
std::vector<int32_t> cut_groups(const std::vector<int8_t>& bs, const std::vector<int32_t>& cnt,
                                const std::vector<int32_t>& both) {
  const int n = (int)bs.size();
  std::vector<int64_t> best(n + 1, 0);
  std::vector<int32_t> from(n + 1, 0);
  for (int i = 1; i <= n; ++i) {
    int rows = bs[i - 1];
    int64_t link = 0;
    best[i] = best[i - 1];
    from[i] = i - 1;
    for (int j = i - 2; j >= 0 && i - j <= kGrpAtoms; --j) {
      rows += bs[j];
      if (rows > kGrpRows || 2 * both[j] < std::max(cnt[j], cnt[j + 1])) break;
      link += both[j] + 1;
      if (best[j] + link > best[i]) {
        best[i] = best[j] + link;
        from[i] = j;
      }
    }
  }
  std::vector<int32_t> first;
  for (int i = n; i > 0; i = from[i]) first.push_back(from[i]);
  std::reverse(first.begin(), first.end());
  first.push_back(n);
  return first;
}

// Device tables of the runs `first`; ranks by the smallest processing position
// of a run's atoms (order empty: as they come).
int32_t make_groups(Ctx* ctx, const std::vector<int32_t>& first, const std::vector<int8_t>& bs,
                    const std::vector<int32_t>& order, std::shared_ptr<GroupTab>* out) {
  auto t = std::make_shared<GroupTab>();
  t->ctx = ctx;
  t->n = (int)first.size() - 1;
  t->n_atoms = (int)bs.size();
  const int n = t->n, na = t->n_atoms;
  const size_t words = (size_t)4 * n + 1 + 2 * (size_t)na;
  std::vector<int32_t> h(words + ((size_t)n * kW + 1) / 2, 0);
  uint16_t* hg = reinterpret_cast<uint16_t*>(h.data() + words);
  int32_t *hf = h.data(), *ho = hf + n + 1, *hr = ho + n, *hw = hr + n, *hm = hw + n, *ha = hm + na;
  std::vector<int32_t> pos(na);
  t->ordered = (int)order.size() == na;
  if (t->ordered)
    for (int w = 0; w < na; ++w) pos[order[w]] = w;
  else
    std::iota(pos.begin(), pos.end(), 0);
  std::vector<std::pair<int32_t, int32_t>> key(n);
  for (int g = 0; g < n; ++g) {
    int rows = 0, mp = na;
    for (int a = first[g]; a < first[g + 1]; ++a) {
      hm[a] = g;
      ha[a] = rows;
      for (int x = 0; x < bs[a]; ++x)
        hg[(size_t)g * kW + rows + x] = (uint16_t)(kGeoRow | (a - first[g]) | (x << 3) | (bs[a] << 8));
      rows += bs[a];
      mp = std::min(mp, pos[a]);
    }
    hf[g] = first[g];
    hw[g] = rows;
    key[g] = {mp, g};
    t->max_rows = std::max(t->max_rows, rows);
    t->max_atoms = std::max(t->max_atoms, first[g + 1] - first[g]);
  }
  hf[n] = na;
  std::sort(key.begin(), key.end());
  t->h_minpos.resize(n);
  for (int x = 0; x < n; ++x) {
    ho[x] = key[x].second;
    hr[key[x].second] = x;
    t->h_minpos[x] = key[x].first;
  }
  LAMB_TRY(dalloc(ctx, &t->first, (int64_t)h.size()));
  LAMB_CUDA(ctx, cudaMemcpyAsync(t->first, h.data(), sizeof(int32_t) * h.size(), cudaMemcpyHostToDevice, ctx->stream));
  LAMB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));  // h dies here
  t->order = t->first + n + 1;
  t->rank = t->order + n;
  t->rows = t->rank + n;
  t->map = t->rows + n;
  t->arow = t->map + na;
  t->geo = reinterpret_cast<const uint16_t*>(t->first + words);
  *out = std::move(t);
  return LAMB_GPU_OK;
}

int32_t adjacency(Ctx* ctx, const DevMatrix* m, bool cols, std::vector<int32_t>* cnt, std::vector<int32_t>* both) {
  const int n = cols ? m->n_cols : m->n_rows;
  std::vector<int32_t> h(2 * (size_t)n, 0);
  if (n && m->nnz) {
    int32_t* d = nullptr;
    LAMB_TRY(dalloc(ctx, &d, 2 * (int64_t)n));
    LAMB_CUDA(ctx, cudaMemsetAsync(d, 0, sizeof(int32_t) * 2 * n, ctx->stream));
    if (cols)
      k_grp_cols<<<grid_for(32ll * m->n_rows), kThreads, 0, ctx->stream>>>(m->n_rows, m->row_p, m->col, d, d + n);
    else
      k_grp_rows<<<grid_for(32ll * m->n_rows), kThreads, 0, ctx->stream>>>(m->n_rows, m->row_p, m->col, d, d + n);
    LAMB_LAUNCHED(ctx);
    LAMB_CUDA(ctx, cudaMemcpyAsync(h.data(), d, sizeof(int32_t) * 2 * n, cudaMemcpyDeviceToHost, ctx->stream));
    LAMB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    dfree(ctx, d);
  }
  cnt->assign(h.begin(), h.begin() + n);
  both->assign(h.begin() + n, h.end());
  return LAMB_GPU_OK;
}

}  // namespace

GroupTab::~GroupTab() {
  if (first) cudaFreeAsync(first, ctx->stream);
}

int32_t ensure_groups(Ctx* ctx, DevMatrix* m) {
  if (m->rgrp && !m->rgrp->ordered && !m->h_order.empty()) {  // made before the order was known
    m->rgrp.reset();
    m->cgrp.reset();
  }
  if (m->rgrp && m->cgrp) return LAMB_GPU_OK;
  std::vector<int32_t> cnt, both;
  if (!m->cgrp) {
    LAMB_TRY(adjacency(ctx, m, true, &cnt, &both));
    const bool square = m->n_rows == m->n_cols && m->h_row_bs == m->h_col_bs;
    LAMB_TRY(make_groups(ctx, cut_groups(m->h_col_bs, cnt, both), m->h_col_bs,
                         square ? m->h_order : std::vector<int32_t>(), &m->cgrp));
    if (square && !m->rgrp) m->rgrp = m->cgrp;
  }
  if (!m->rgrp) {
    LAMB_TRY(adjacency(ctx, m, false, &cnt, &both));
    LAMB_TRY(make_groups(ctx, cut_groups(m->h_row_bs, cnt, both), m->h_row_bs, m->h_order, &m->rgrp));
  }
  return LAMB_GPU_OK;
}

// Mean number of 16-row slabs of the stack kernel over the atoms with elements.
static double mean_slabs(const std::vector<int8_t>& bs) {
  int64_t n = 0, s = 0;
  for (int8_t b : bs)
    if (b > 0) {
      ++n;
      s += (b + 15) / 16;
    }
  return n ? (double)s / n : 1.0;
}

double panel_gain(const PanelPair* p, const GroupTab& rows, const GroupTab& inner, const GroupTab& cols,
                  const std::vector<int8_t>& row_bs, const std::vector<int8_t>& col_bs, int64_t products,
                  const int64_t* totals) {
  const double per_pair = p ? (double)products / std::max<int64_t>(totals[2], 1)
                            : (double)rows.n_atoms / rows.n * inner.n_atoms / inner.n * cols.n_atoms / cols.n;
  return per_pair * mean_slabs(row_bs) * mean_slabs(col_bs);
}

bool panel_shapes_ok(const std::vector<int8_t>& rows, const std::vector<int8_t>& inner,
                     const std::vector<int8_t>& cols) {
  return panel_atoms_ok((int64_t)rows.size(), (int64_t)inner.size(), (int64_t)cols.size()) &&
         max_block(rows) <= kGrpRows && max_block(inner) <= kGrpRows && max_block(cols) <= kGrpRows;
}

bool panel_worth(const DevMatrix* A, const DevMatrix* B) {
  return A->n_cols > 0 && panel_blocks_ok(A->nnz, B->nnz, 0) &&
         (double)A->nnz * B->nnz >= (double)(1 << 19) * A->n_cols;
}

int32_t product_groups(Ctx* ctx, DevMatrix* A, DevMatrix* B, std::shared_ptr<GroupTab>* cols) {
  LAMB_TRY(ensure_groups(ctx, A));
  if (A->h_row_bs == A->h_col_bs && B->h_row_bs == A->h_row_bs && B->h_col_bs == A->h_row_bs) {
    *cols = A->rgrp;
    return LAMB_GPU_OK;
  }
  LAMB_TRY(ensure_groups(ctx, B));
  *cols = B->cgrp;
  return LAMB_GPU_OK;
}

void PanelPair::release() {
  for (PanelSide* s : {&a, &b}) {
    if (s->buf) cudaFreeAsync(s->buf, ctx->stream);
    if (s->buf2) cudaFreeAsync(s->buf2, ctx->stream);
    s->buf = s->buf2 = nullptr;
  }
}

namespace {

PairArgs pair_args(const PanelPair& p) {
  PairArgs r{};
  const PanelSide* sd[2] = {&p.a, &p.b};
  for (int k = 0; k < 2; ++k) {
    const PanelSide& s = *sd[k];
    const DevMatrix* m = s.m;
    SideArgs& q = r.s[k];
    q.row_p = m->row_p; q.col = m->col; q.off = m->off; q.data = m->data; q.norms = m->norms;
    q.row_bs = m->row_bs; q.col_bs = m->col_bs; q.n_rows = m->n_rows; q.rows_out = s.rows_out;
    q.o_first = s.out->first; q.o_map = s.out->map; q.o_arow = s.out->arow; q.o_rows = s.out->rows;
    q.i_first = s.in->first; q.i_map = s.in->map; q.i_arow = s.in->arow; q.i_rows = s.in->rows;
    q.n_out = s.out->n; q.words = s.words; q.n_sb = s.n_sb;
    q.hist = s.hist; q.bm = s.bm; q.pre = s.pre; q.ptr = s.ptr; q.kc = s.kc; q.sbg = s.sbg; q.mask = s.mask;
    q.nrange = s.nrange; q.nrm = s.nrm; q.panel = s.panel;
    r.na_max[k] = s.out->max_atoms;
  }
  r.kstride = p.kstride;
  r.nk_max = p.a.in->max_atoms;
  r.n_in = p.a.in->n;
  r.totals = p.totals;
  return r;
}

}  // namespace

int32_t panel_index(Ctx* ctx, PanelPair* p, const DevMatrix* ma, bool a_rows_out, const DevMatrix* mb, bool b_rows_out,
                    std::shared_ptr<GroupTab> out_a, std::shared_ptr<GroupTab> in, std::shared_ptr<GroupTab> out_b,
                    int64_t* totals) {
  p->ctx = ctx;
  p->keep[0] = out_a; p->keep[1] = in; p->keep[2] = out_b;
  p->a.m = ma; p->a.rows_out = a_rows_out; p->a.out = out_a.get();
  p->b.m = mb; p->b.rows_out = b_rows_out; p->b.out = out_b.get();
  p->kstride = std::max((in->max_rows + 3) & ~3, 4);
  p->totals = nullptr;
  for (PanelSide* s : {&p->a, &p->b}) {
    s->in = in.get();
    s->words = (in->n + 31) / 32;
    const int64_t nw = (int64_t)s->out->n * s->words, n1 = s->out->n + 1;
    char* d = nullptr;
    LAMB_TRY(dalloc(ctx, &d, 4 * (in->n + 2 * nw + n1) + 64));
    s->buf = d;
    if (!p->totals) p->totals = reinterpret_cast<int64_t*>(d);
    s->hist = reinterpret_cast<int32_t*>(d + 64);
    s->bm = reinterpret_cast<uint32_t*>(s->hist + in->n);
    s->pre = reinterpret_cast<int32_t*>(s->bm + nw);
    s->ptr = s->pre + nw;
    LAMB_CUDA(ctx, cudaMemsetAsync(d, 0, 64 + sizeof(uint32_t) * (in->n + nw), ctx->stream));
  }
  PairArgs r = pair_args(*p);
  const int rows = std::max(ma->n_rows, mb->n_rows), outs = std::max(p->a.out->n, p->b.out->n);
  k_panel_bits<<<dim3(grid_for(32ll * rows), 2), kThreads, 0, ctx->stream>>>(r);
  LAMB_LAUNCHED(ctx);
  k_panel_prefix<<<dim3(grid_for(32ll * outs), 2), kThreads, 0, ctx->stream>>>(r);
  LAMB_LAUNCHED(ctx);
  k_panel_scan<<<2, 1024, 0, ctx->stream>>>(r);
  LAMB_LAUNCHED(ctx);
  LAMB_CUDA(ctx, cudaMemcpyAsync(totals, p->totals, 3 * sizeof(int64_t), cudaMemcpyDeviceToHost, ctx->stream));
  return LAMB_GPU_OK;
}

int32_t panel_pack(Ctx* ctx, PanelPair* p, const int64_t* totals, bool filt, bool* ok) {
  *ok = false;
  PanelSide* sd[2] = {&p->a, &p->b};
  const int slot[2] = {kScrPlaneA, kScrPlaneB};
  // the panels take at most an eighth of the device's memory (they stay with the context)
  if ((double)(totals[0] + totals[1]) * p->kstride * kRowBytes > (double)ctx->total_mem / 8 ||
      totals[0] > kPanelMaxBlocks || totals[1] > kPanelMaxBlocks)
    return LAMB_GPU_OK;
  for (int k = 0; k < 2; ++k) {
    PanelSide& s = *sd[k];
    s.n_sb = (int32_t)totals[k];
    const int64_t n = std::max(s.n_sb, 1), per = (int64_t)s.out->max_atoms * s.in->max_atoms;
    char* d = nullptr;
    LAMB_TRY(dalloc(ctx, &d, 16 * n + (filt ? n * (16 + 8 * per) : 0)));
    s.buf2 = d;
    s.nrange = reinterpret_cast<double2*>(d);  // 16-byte elements first
    if (filt) d += 16 * n;
    s.nrm = reinterpret_cast<double*>(d);
    if (filt) d += 8 * n * per;
    s.kc = reinterpret_cast<int32_t*>(d);
    s.sbg = s.kc + n;
    s.mask = reinterpret_cast<uint32_t*>(s.sbg + n);
    LAMB_TRY(scratch(ctx, slot[k], n * p->kstride * kW, &s.panel));
  }
  PairArgs r = pair_args(*p);
  const int outs = std::max(p->a.out->n, p->b.out->n), sbs = std::max(p->a.n_sb, p->b.n_sb);
  k_panel_list<<<dim3(grid_for(32ll * outs), 2), kThreads, 0, ctx->stream>>>(r);
  LAMB_LAUNCHED(ctx);
  const dim3 g(grid_for(32ll * std::max(sbs, 1)), 2);
  if (filt)
    k_panel_pack<true><<<g, 32 * kPackWarps, 0, ctx->stream>>>(r);
  else
    k_panel_pack<false><<<g, 32 * kPackWarps, 0, ctx->stream>>>(r);
  LAMB_LAUNCHED(ctx);
  *ok = true;
  return LAMB_GPU_OK;
}

// Bitmap of a block pattern and every row's blocks before each word, one warp per row.
__global__ void k_pattern_bits(int32_t n_rows, int32_t n_words, const int64_t* __restrict__ row_p,
                               const int32_t* __restrict__ col, uint32_t* __restrict__ bm, int32_t* __restrict__ pre) {
  const int lane = threadIdx.x & 31;
  for (int64_t r = global_warp(); r < n_rows; r += grid_warps()) {
    const int64_t b0 = row_p[r], b1 = row_p[r + 1];
    uint32_t* w = bm + r * n_words;
    int32_t* q = pre + r * n_words;
    int64_t b = b0;  // first block of the words to come
    for (int w0 = 0; w0 < n_words; w0 += 32) {
      uint32_t mine = 0;
      const int64_t end = lower_col(col, b, b1, 32 * (w0 + 32));
      for (int64_t x = b; x < end; x += 32) {
        // a block's column names its word among the 32 of this step
        const int c = x + lane < end ? col[x + lane] : -1;
        for (int s = 0; s < 32; ++s) {
          const int cs = __shfl_sync(0xffffffffu, c, s);
          if (cs >= 0 && (cs >> 5) == w0 + lane) mine |= 1u << (cs & 31);
        }
      }
      const int n = __popc(mine), incl = warp_incl_scan(n, lane);
      if (w0 + lane < n_words) {
        w[w0 + lane] = mine;
        q[w0 + lane] = (int32_t)(b - b0) + incl - n;
      }
      b = end;
    }
  }
}

int32_t panel_pattern(Ctx* ctx, const DevMatrix* Z, uint32_t** bm, int32_t** pre) {
  const int32_t words = (Z->n_cols + 31) / 32;
  LAMB_TRY(dalloc(ctx, bm, (int64_t)Z->n_rows * words));
  LAMB_TRY(dalloc(ctx, pre, (int64_t)Z->n_rows * words));
  k_pattern_bits<<<grid_for(32ll * Z->n_rows), kThreads, 0, ctx->stream>>>(Z->n_rows, words, Z->row_p, Z->col, *bm, *pre);
  LAMB_LAUNCHED(ctx);
  return LAMB_GPU_OK;
}

int32_t panel_tiles(Ctx* ctx, const PanelPair& p, const DevMatrix* C, const uint32_t* c_bm, const int32_t* c_pre,
                    double* c_nrm, bool filt, double eps, int chunks, std::vector<int32_t>* done_pos) {
  const GroupTab &R = *p.a.out, &K = *p.a.in, &Q = *p.b.out;
  const int n_mi = (R.n + 1) / 2, n_mj = (Q.n + 1) / 2;
  const int n_sup = (n_mi + kSuper - 1) / kSuper;
  // ---- macro tiles with a C block ----
  MaskArgs q{};
  q.row_p = C->row_p; q.col = C->col;
  q.r_first = R.first; q.r_order = R.order; q.c_map = Q.map; q.c_rank = Q.rank;
  q.n_rg = R.n; q.n_mj = n_mj; q.c_order = Q.order;
  char* d = nullptr;
  const int64_t n_items = std::min<int64_t>((int64_t)R.n * Q.n, std::max<int64_t>(C->nnz, 1));
  LAMB_TRY(dalloc(ctx, &d, 8 * (int64_t)n_sup * n_mj + 8 * n_items + 4 * (n_sup + 1 + kMaxChunks)));
  struct Free {
    Ctx* ctx;
    char* p;
    ~Free() { cudaFreeAsync(p, ctx->stream); }
  } fr{ctx, d};
  q.masks = reinterpret_cast<uint2*>(d);
  q.items = reinterpret_cast<int2*>(q.masks + (int64_t)n_sup * n_mj);
  q.count = reinterpret_cast<int32_t*>(q.items + n_items);
  LAMB_CUDA(ctx, cudaMemsetAsync(q.count + n_sup + 1, 0, sizeof(int32_t) * kMaxChunks, ctx->stream));
  const size_t msk = 8 * (size_t)n_mj;
  LAMB_TRY(allow_smem(ctx, k_panel_masks, msk));
  k_panel_masks<<<n_sup, 512, msk, ctx->stream>>>(q);
  LAMB_LAUNCHED(ctx);
  k_panel_mask_scan<<<1, 1024, 0, ctx->stream>>>(n_sup, q.count);
  LAMB_LAUNCHED(ctx);
  k_panel_items<<<n_sup, 256, 0, ctx->stream>>>(q);
  LAMB_LAUNCHED(ctx);
  // ---- tiles ----
  TileArgs t{};
  const PanelSide* sd[2] = {&p.a, &p.b};
  for (int k = 0; k < 2; ++k) {
    const PanelSide& x = *sd[k];
    t.s[k] = TileSide{x.bm, x.pre, x.ptr, x.mask, x.nrange, x.nrm, x.panel, x.out->first, x.out->rows,
                      x.out->geo, x.out->max_atoms};
  }
  t.words = p.b.words; t.kstride = p.kstride;
  t.c_words = (C->n_cols + 31) / 32; t.c_bm = c_bm; t.c_pre = c_pre;
  t.row_p = C->row_p; t.off = C->off;
  t.data = C->data; t.c_nrm = c_nrm; t.eps = eps;
  t.kc_a = p.a.kc; t.i_first = K.first; t.i_arow = K.arow;
  t.i_bs = p.a.rows_out ? p.a.m->col_bs : p.a.m->row_bs;
  t.nk_max = K.max_atoms;
  t.items = q.items; t.seg = q.count; t.head = q.count + n_sup + 1; t.err = ctx->tile_err;
  t.wait_ns = ctx->wait_ns;
  const size_t smem = kTileSmem;
  auto kern = filt ? k_panel_tiles<true> : k_panel_tiles<false>;
  LAMB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  const int nc = std::max(1, std::min(chunks, n_sup));
  if (done_pos) done_pos->clear();
  for (int c = 0; c < nc; ++c) {
    t.s0 = (int)((int64_t)n_sup * c / nc);
    t.s1 = (int)((int64_t)n_sup * (c + 1) / nc);
    LAMB_CUDA(ctx, cudaEventRecord(ctx->kern_ev[0][c], ctx->stream));
    kern<<<sms, 32 * kTileWarps, smem, ctx->stream>>>(t);
    LAMB_LAUNCHED(ctx);
    ++t.head;
    LAMB_CUDA(ctx, cudaEventRecord(ctx->kern_ev[1][c], ctx->stream));
    LAMB_CUDA(ctx, cudaEventRecord(ctx->chunk_ev[c], ctx->stream));
    // rows before the first row of the next super row's groups are complete
    const int g = t.s1 * 2 * kSuper;
    if (done_pos) done_pos->push_back(g < R.n ? R.h_minpos[g] : R.n_atoms);
  }
  ctx->kern_chunks = nc;
  LAMB_CUDA(ctx, cudaMemcpyAsync(ctx->pin + kPinTileErr, ctx->tile_err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  return LAMB_GPU_OK;
}

}  // namespace lamb
