// Panel products: the FP64 block product on group tiles (panel.cu).
#pragma once
#include "common.cuh"
#include "panel_limits.cuh"

namespace lamb {

constexpr int kGrpRows = 24;  // element rows of a group at most: the MMA tile is 3 x 3 slabs of 8
constexpr int kGrpAtoms = 8;  // atoms of a group at most
constexpr int kGeoRow = 1 << 15;
// Runs of consecutive atoms of one axis (groups) whose block rows couple to
// nearly the same atoms, and where the groups lie in the processing order.
struct GroupTab {
  Ctx* ctx = nullptr;
  int32_t n = 0, n_atoms = 0;
  int32_t max_rows = 0, max_atoms = 0;  // of any group
  bool ordered = false;                 // ranks follow a processing order (otherwise the atoms' own)
  std::vector<int32_t> h_minpos;        // [n] by rank: smallest processing position of the group's atoms
  // one device buffer holding, in this order:
  int32_t* first = nullptr;  // [n + 1]
  int32_t* order = nullptr;  // [n] rank -> group (ranks follow the processing order)
  int32_t* rank = nullptr;   // [n] group -> rank
  int32_t* rows = nullptr;   // [n] element rows
  int32_t* map = nullptr;    // [n_atoms] atom -> group
  int32_t* arow = nullptr;   // [n_atoms] first element row of the atom in its group
  const uint16_t* geo = nullptr;  // [n * kGrpRows] atom | row of its block << 3 | block rows << 8 | kGeoRow; 0 past the end
  ~GroupTab();
};

// Groups of m's rows and columns (kept with the matrix, inherited by results).
int32_t ensure_groups(Ctx* ctx, DevMatrix* m);

// One operand in panel form.  rows_out: the groups tiled over are m's rows
// and the inner dimension its columns; otherwise the other way round.
struct PanelSide {
  const DevMatrix* m = nullptr;
  bool rows_out = true;
  const GroupTab* out = nullptr;
  const GroupTab* in = nullptr;
  int32_t words = 0;          // bitmap words of one group (inner groups / 32)
  int32_t* hist = nullptr;    // [in->n] superblocks of every inner group
  uint32_t* bm = nullptr;     // [out->n * words] inner groups the group couples to
  int32_t* pre = nullptr;     // [out->n * words] superblocks of the group before the word
  int32_t* ptr = nullptr;     // [out->n + 1] superblocks before the group
  int32_t* kc = nullptr;      // [n_sb] inner group of every superblock
  int32_t* sbg = nullptr;     // [n_sb] out group of every superblock
  uint32_t* mask = nullptr;   // [n_sb] inner element rows that hold a block
  double2* nrange = nullptr;  // [n_sb] smallest and largest block norm (product filter only)
  double* nrm = nullptr;      // [n_sb * na * nk] block norms, < 0 where absent (product filter only)
  double* panel = nullptr;    // context scratch
  int32_t n_sb = 0;           // known once the totals have arrived
  void* buf = nullptr;        // device buffer of bm .. ptr
  void* buf2 = nullptr;       // device buffer of kc .. nrm
};

struct PanelPair {
  Ctx* ctx = nullptr;
  PanelSide a, b;
  std::shared_ptr<GroupTab> keep[3];
  int32_t kstride = 0;  // panel rows of a superblock (a multiple of four)
  // device: superblocks of a and b, superblock pairs, and (after the packing)
  // whether a value is infinite or NaN
  int64_t* totals = nullptr;
  void release();  // gives the device buffers back (stream-ordered)
  ~PanelPair() { release(); }
};

// Whether the panel kernel may be considered for A.B (or its adjoint): about
// half a million block products (below that the launches that prepare the
// panels, some 60 us, cost more than the stacks: 48 atoms of 0 to 3 rows, 53,000
// products, 625 us a call with stacks, 690 us with panels; 64 waters, 1.6
// million, even).
bool panel_worth(const DevMatrix* A, const DevMatrix* B);
// Whether its tiles can hold the product of these row, inner and column atoms:
// the roles of each product by itself (those of dA are A's rows, B's columns and
// A's columns, those of dB A's columns, A's rows and B's columns).
bool panel_shapes_ok(const std::vector<int8_t>& rows, const std::vector<int8_t>& inner,
                     const std::vector<int8_t>& cols);
// Groups of A.B's columns (those of its rows and inner atoms are A's): A's when
// B lives on the same atoms (both then describe the same runs), B's own otherwise.
int32_t product_groups(Ctx* ctx, DevMatrix* A, DevMatrix* B, std::shared_ptr<GroupTab>* cols);
// What the panel kernel has to gain on the stack kernel: block products per
// superblock pair times the stack kernel's 16 x 16 slabs per product.  Measured
// (ms, stacks -> panels): 1 (atoms of 13 rows that form no groups) 3.1 -> 6.4,
// 1.8 (23 / 5 rows, no groups) 11.7 -> 14.7, 2.7 (9 rows, groups of two and one)
// 2.2 -> 2.6, 4 (17 rows, no groups) 17.9 -> 8.0, 4.8 (23 / 5 / 5) 12.4 -> 8.4,
// 12 (13 / 5 / 5) 7.2 -> 3.3.  The panels are taken from kPanelGain on.  Without
// p (the superblocks not yet counted): the estimate with every block present.
constexpr double kPanelGain = 3.0;
double panel_gain(const PanelPair* p, const GroupTab& rows, const GroupTab& inner, const GroupTab& cols,
                  const std::vector<int8_t>& row_bs, const std::vector<int8_t>& col_bs, int64_t products,
                  const int64_t* totals);
// Superblock index of both operands; the totals (superblocks of a and of b,
// superblock pairs) are copied to `totals` (pinned, 3 int64) on the stream.
int32_t panel_index(Ctx* ctx, PanelPair* p, const DevMatrix* ma, bool a_rows_out, const DevMatrix* mb, bool b_rows_out,
                    std::shared_ptr<GroupTab> out_a, std::shared_ptr<GroupTab> in, std::shared_ptr<GroupTab> out_b,
                    int64_t* totals);
// Panels of both operands (after the totals have arrived); filt: with block
// norms.  *ok = false, and nothing queued, when they are too large.  What cannot
// be allocated, here or in the other calls, is the callers' to do without: they
// give the memory back and take the stacks.
int32_t panel_pack(Ctx* ctx, PanelPair* p, const int64_t* totals, bool filt, bool* ok);
// Pattern bitmap of Z for panel_tiles (freed by the caller).
int32_t panel_pattern(Ctx* ctx, const DevMatrix* Z, uint32_t** bm, int32_t** pre);
// C := product on C's pattern (row_p, off and data set; c_bm / c_pre: the
// pattern's bitmap over the columns, 32 to a word, and the row's blocks before
// every word).  c_nrm may be null.  `chunks` launches; done_pos gets the rows
// (processing positions) complete after each, the events of chunk p are
// recorded after it.
int32_t panel_tiles(Ctx* ctx, const PanelPair& p, const DevMatrix* C, const uint32_t* c_bm, const int32_t* c_pre,
                    double* c_nrm, bool filt, double eps, int chunks, std::vector<int32_t>* done_pos);

}  // namespace lamb
