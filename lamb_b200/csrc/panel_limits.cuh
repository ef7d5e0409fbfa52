// What the group tiles (panel.cu) can hold.  Host C++ only, so that the rules
// can be checked without a GPU.
#pragma once
#include <cstdint>

namespace lamb {

// The tile kernel counts superblocks, tiles and C blocks in 32 bits.  A
// superblock holds at least one block of its operand and a tile at least one of
// C, so the block counts bound all three.  Beyond: the stacks, whose work items
// carry 64-bit offsets.
constexpr int64_t kPanelMaxBlocks = INT32_MAX;
inline bool panel_blocks_ok(int64_t a_blocks, int64_t b_blocks, int64_t c_blocks) {
  return a_blocks <= kPanelMaxBlocks && b_blocks <= kPanelMaxBlocks && c_blocks <= kPanelMaxBlocks;
}

// Atoms of a product by the role they have in its tiles.  Columns: one super
// row's masks, 8 bytes for two column groups, lie in shared memory (51,200
// groups of one atom take 204,800 of 232,448 bytes).  Rows and inner atoms: the
// superblock bitmaps (groups x inner groups bits) stay below a few GB.
constexpr int64_t kPanelMaxRows = 262144, kPanelMaxInner = 65536, kPanelMaxCols = 51200;
inline bool panel_atoms_ok(int64_t rows, int64_t inner, int64_t cols) {
  return rows > 0 && inner > 0 && cols > 0 && rows <= kPanelMaxRows && inner <= kPanelMaxInner && cols <= kPanelMaxCols;
}

// The stack and the mixed kernels write block norms through a 32-bit index:
// without norms (no result filter, FP64) a C may have more blocks.
inline bool norm_index_ok(int64_t c_blocks, bool norms) { return !norms || c_blocks <= INT32_MAX; }

}  // namespace lamb
