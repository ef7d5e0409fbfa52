// Goods messages: one sector in the wire format of the reference's sector
// exchange (lamb_goods_X_create, src/lamb_goods_X_types.F90:79-268;
// lamb_goods_X_unpack, src/lamb_goods_X_methods.F90:166-218).
//
// The index is an int64 word array: 12 slots of 1-based (offset, size) for
// the index itself, the data, row_p, col_i, extents and flags
// (src/lamb_goods_X_types.F90:79-91), then row_p (int64 words), col_i
// (int16 values, four to a word, little-endian), extents (int64 pairs) and
// flags (zero); every section is at least one word.  The data travel as a
// separate float64 array: the sector's data store, which the extents index
// (1-based).  Followed by intent: row_p carries all n_rows + 1 offsets (the
// reference packs n_rows, :160-162, :196) and col_i is read back as int16.
//
// Pack and unpack accept host or device buffers (unified addressing), so a
// message can go straight from one GPU's memory to another's over NVLink
// (NCCL send/recv of the two arrays) or through the host.
#include <cub/cub.cuh>

#include <cstring>

#include "common.cuh"

namespace lamb {

constexpr int kSlots = 12;
enum GoodsSlot : int {
  kIdxOff = 0, kIdxSize, kDataOff, kDataSize, kRowPOff, kRowPSize, kColIOff, kColISize, kExtOff, kExtSize,
  kFlagsOff, kFlagsSize
};

static int64_t words_of(int64_t bytes) { return std::max<int64_t>(1, (bytes + 7) / 8); }

struct GoodsLayout {
  int64_t hdr[kSlots];
  int64_t w_rows, w_cols, w_ext, w_flags, n_words;
};

static GoodsLayout goods_layout(int64_t n_rows, int64_t n_blks, int64_t data_len) {
  GoodsLayout g{};
  g.w_rows = words_of(8 * (n_rows + 1));
  g.w_cols = words_of(2 * n_blks);
  g.w_ext = words_of(16 * n_blks);
  g.w_flags = words_of(n_blks);
  g.n_words = kSlots + g.w_rows + g.w_cols + g.w_ext + g.w_flags;
  int64_t off = 1 + kSlots;
  g.hdr[kIdxOff] = 1;
  g.hdr[kIdxSize] = g.n_words;
  g.hdr[kDataOff] = 1;
  g.hdr[kDataSize] = data_len;
  g.hdr[kRowPOff] = off; g.hdr[kRowPSize] = n_rows + 1; off += g.w_rows;
  g.hdr[kColIOff] = off; g.hdr[kColISize] = n_blks; off += g.w_cols;
  g.hdr[kExtOff] = off; g.hdr[kExtSize] = n_blks; off += g.w_ext;
  g.hdr[kFlagsOff] = off; g.hdr[kFlagsSize] = n_blks;
  return g;
}

// ---- index message on the device ------------------------------------------------------
// The index of one sector straight into its message: three launches that read
// the sector's rows only.  Built on the host and copied (with the whole matrix's
// sector index built for every sector asked for) the four messages of a
// 6,144-water product, 0.7 GB of index each, took 238 ms.
struct GoodsArgs {
  int64_t hdr[kSlots];
  int64_t* msg;
  int64_t n_words;
  const int64_t* row_p;
  const int32_t* col;
  const int64_t* off;
  const int8_t *row_bs, *col_bs;
  int32_t r0, n_rows, c0, c1;  // rows and columns of the sector
  int64_t base;                // its first element in the data
};

// Blocks per row: lanes 2 i and 2 i + 1 search row i's first block and its end.
__global__ void k_goods_rows(const __grid_constant__ GoodsArgs p) {
  int64_t* rp = p.msg + p.hdr[kRowPOff] - 1;
  const int64_t n = 2ll * p.n_rows, step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < (n + 31) / 32 * 32; x += step) {
    const int64_t l = x >> 1;
    int64_t at = 0;
    if (x < n && p.row_p) at = lower_col(p.col, p.row_p[p.r0 + l], p.row_p[p.r0 + l + 1], x & 1 ? p.c1 : p.c0);
    const int64_t end = __shfl_down_sync(0xffffffffu, at, 1);
    if (x < n && !(x & 1)) rp[l + 1] = end - at;
  }
}

// Row counts -> offsets, the header, and the words that only partly belong to
// blocks (one CTA; a sector has at most 32,767 rows).
__global__ void __launch_bounds__(1024) k_goods_scan(const __grid_constant__ GoodsArgs p) {
  typedef cub::BlockScan<long long, 1024> BS;
  __shared__ typename BS::TempStorage ts;
  int64_t* rp = p.msg + p.hdr[kRowPOff] - 1;
  long long carry = 0;
  for (int l0 = 0; l0 < p.n_rows; l0 += 1024) {
    const int l = l0 + threadIdx.x;
    long long v = l < p.n_rows ? rp[l + 1] : 0, a;
    BS(ts).InclusiveSum(v, v, a);
    __syncthreads();
    if (l < p.n_rows) rp[l + 1] = carry + v;
    carry += a;
  }
  if (threadIdx.x < kSlots) p.msg[threadIdx.x] = p.hdr[threadIdx.x];
  if (threadIdx.x == 0) {
    rp[0] = 0;
    p.msg[p.hdr[kExtOff] - 2] = 0;                              // last word of the columns
    if (p.hdr[kExtSize] == 0) p.msg[p.hdr[kExtOff] - 1] = 0;    // the extents' one word without blocks
    if (p.hdr[kExtSize] == 0) p.msg[p.hdr[kFlagsOff] - 1] = 0;  // and the flags'
  }
}

// Columns (int16, 1-based), extents (1-based within the sector's data) and
// zero flags.
__global__ void k_goods_blocks(const __grid_constant__ GoodsArgs p) {
  const int lane = threadIdx.x & 31;
  const int64_t* rp = p.msg + p.hdr[kRowPOff] - 1;
  int16_t* col16 = reinterpret_cast<int16_t*>(p.msg + p.hdr[kColIOff] - 1);
  int64_t* ext = p.msg + p.hdr[kExtOff] - 1;
  for (int64_t l = global_warp(); l < p.n_rows; l += grid_warps()) {
    const int64_t q0 = rp[l], n = rp[l + 1] - q0;
    if (n == 0) continue;
    const int64_t r = p.r0 + l, lo = lower_col(p.col, p.row_p[r], p.row_p[r + 1], p.c0);
    const int64_t bi = p.row_bs[r];
    for (int64_t x = lane; x < n; x += 32) {
      const int c = p.col[lo + x];
      const int64_t e1 = p.off[lo + x] - p.base + 1;
      col16[q0 + x] = (int16_t)(c - p.c0 + 1);
      ext[2 * (q0 + x)] = e1;
      ext[2 * (q0 + x) + 1] = e1 + bi * p.col_bs[c] - 1;
    }
  }
  for (int64_t w = p.hdr[kFlagsOff] - 1 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < p.n_words;
       w += (int64_t)gridDim.x * blockDim.x)
    p.msg[w] = 0;
}

}  // namespace lamb

using namespace lamb;

extern "C" {

int32_t lamb_gpu_goods_size(lamb_gpu_ctx* c, lamb_gpu_matrix h, int32_t sector, int64_t* index_words,
                            int64_t* data_len) {
  auto* ctx = reinterpret_cast<Ctx*>(c);
  if (!ctx || !index_words || !data_len) return make_status(LAMB_LEVEL_FAILURE, LAMB_TYPE_WRONG_ARGS);
  DevMatrix* m = get_matrix(ctx, h);
  if (!m) return fail(ctx, LAMB_LEVEL_FAILURE, LAMB_TYPE_WRONG_ARGS, "goods: invalid handle");
  const int n_sec = m->n_rsub * m->n_csub;
  if (sector < 0 || sector >= n_sec) return fail(ctx, LAMB_LEVEL_FAILURE, LAMB_TYPE_WRONG_ARGS, "goods: no such sector");
  const GoodsLayout g = goods_layout(m->rsub_cnt[sector / m->n_csub], m->sec_nblk[sector], m->sec_dlen[sector]);
  *index_words = g.n_words;
  *data_len = m->sec_dlen[sector];
  return LAMB_GPU_OK;
}

int32_t lamb_gpu_goods_pack(lamb_gpu_ctx* c, lamb_gpu_matrix h, int32_t sector, int64_t* index, double* data) {
  auto* ctx = reinterpret_cast<Ctx*>(c);
  if (!ctx) return make_status(LAMB_LEVEL_FAILURE, LAMB_TYPE_WRONG_ARGS);
  DevMatrix* m = get_matrix(ctx, h);
  if (!m) return fail(ctx, LAMB_LEVEL_FAILURE, LAMB_TYPE_WRONG_ARGS, "goods: invalid handle");
  const int S = m->n_csub, n_sec = m->n_rsub * S;
  if (sector < 0 || sector >= n_sec) return fail(ctx, LAMB_LEVEL_FAILURE, LAMB_TYPE_WRONG_ARGS, "goods: no such sector");
  cudaSetDevice(ctx->device);
  const int a = sector / S, b = sector % S;
  const int64_t n_rows = m->rsub_cnt[a], n_blks = m->sec_nblk[sector], dlen = m->sec_dlen[sector];
  if (!index || (dlen && !data)) return fail(ctx, LAMB_LEVEL_FAILURE, LAMB_TYPE_WRONG_ARGS, "goods: NULL buffer");
  const GoodsLayout g = goods_layout(n_rows, n_blks, dlen);
  // The index is written where it is wanted when that is this GPU's memory,
  // and into a temporary that is then copied otherwise.
  cudaPointerAttributes at{};
  const bool here = cudaPointerGetAttributes(&at, index) == cudaSuccess && at.type == cudaMemoryTypeDevice &&
                    at.device == ctx->device && reinterpret_cast<uintptr_t>(index) % sizeof(int64_t) == 0;
  if (!here) cudaGetLastError();  // a pointer the driver does not know is plain host memory
  int64_t* msg = index;
  if (!here) LAMB_TRY(dalloc(ctx, &msg, g.n_words));
  GoodsArgs q{};
  memcpy(q.hdr, g.hdr, sizeof(g.hdr));
  q.msg = msg;
  q.n_words = g.n_words;
  q.row_p = m->row_p; q.col = m->col; q.off = m->off; q.row_bs = m->row_bs; q.col_bs = m->col_bs;
  q.r0 = m->rsub_base[a]; q.n_rows = (int32_t)n_rows;
  q.c0 = m->csub_base[b]; q.c1 = m->csub_base[b + 1];
  q.base = m->sec_base[sector];
  auto body = [&]() -> int32_t {
    if (m->nnz == 0) q.row_p = nullptr;  // no index arrays to read
    if (n_rows) {
      k_goods_rows<<<grid_for(2 * n_rows), kThreads, 0, ctx->stream>>>(q);
      LAMB_LAUNCHED(ctx);
    }
    k_goods_scan<<<1, 1024, 0, ctx->stream>>>(q);
    LAMB_LAUNCHED(ctx);
    if (n_blks) {
      k_goods_blocks<<<grid_for(32 * n_rows), kThreads, 0, ctx->stream>>>(q);
      LAMB_LAUNCHED(ctx);
    }
    if (!here)
      LAMB_CUDA(ctx, cudaMemcpyAsync(index, msg, sizeof(int64_t) * g.n_words, cudaMemcpyDefault, ctx->stream));
    if (dlen)
      LAMB_CUDA(ctx, cudaMemcpyAsync(data, m->data + m->sec_base[sector], sizeof(double) * dlen, cudaMemcpyDefault,
                                     ctx->stream));
    return LAMB_GPU_OK;
  };
  const int32_t rc = body();
  if (!here) dfree(ctx, msg);
  LAMB_TRY(rc);
  return finish(ctx);
}

int32_t lamb_gpu_goods_unpack(lamb_gpu_ctx* c, const int64_t* index, int64_t index_words, const double* data,
                              int32_t n_cols, const int8_t* row_blk_sizes, const int8_t* col_blk_sizes,
                              lamb_gpu_matrix* handle) {
  auto* ctx = reinterpret_cast<Ctx*>(c);
  if (!ctx) return make_status(LAMB_LEVEL_FAILURE, LAMB_TYPE_WRONG_ARGS);
  if (!index || !handle || index_words < kSlots || n_cols < 0 || (n_cols && !col_blk_sizes))
    return fail(ctx, LAMB_LEVEL_FAILURE, LAMB_TYPE_WRONG_ARGS, "goods: bad arguments");
  *handle = 0;
  cudaSetDevice(ctx->device);
  std::vector<int64_t> w(index_words);
  LAMB_CUDA(ctx, cudaMemcpyAsync(w.data(), index, sizeof(int64_t) * index_words, cudaMemcpyDefault, ctx->stream));
  LAMB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  const int64_t n_rows = w[kRowPSize] - 1, n_blks = w[kColISize], dlen = w[kDataSize];
  if (w[kIdxOff] != 1 || w[kIdxSize] != index_words || n_rows < 0 || n_blks < 0 || w[kExtSize] != n_blks ||
      dlen < 0 || (dlen && !data) || (n_rows && !row_blk_sizes))
    return fail(ctx, LAMB_LEVEL_FAILURE, LAMB_TYPE_WRONG_ARGS, "goods: index header does not describe a sector");
  const GoodsLayout g = goods_layout(n_rows, n_blks, dlen);
  for (int k = 0; k < kSlots; ++k)
    if (g.hdr[k] != w[k]) return fail(ctx, LAMB_LEVEL_FAILURE, LAMB_TYPE_WRONG_ARGS, "goods: inconsistent index header");
  std::vector<int16_t> col(std::max<int64_t>(n_blks, 1));
  if (n_blks) memcpy(col.data(), w.data() + g.hdr[kColIOff] - 1, sizeof(int16_t) * n_blks);
  lamb_c_sector sec{};
  sec.subset_row = 1;
  sec.subset_col = 1;
  sec.n_rows = (int32_t)n_rows;
  sec.n_cols = n_cols;
  sec.row_blk_sizes = row_blk_sizes;
  sec.col_blk_sizes = col_blk_sizes;
  sec.row_p = w.data() + g.hdr[kRowPOff] - 1;
  sec.col_i = col.data();
  sec.extents = w.data() + g.hdr[kExtOff] - 1;
  sec.data = data;
  sec.n_blks = n_blks;
  sec.data_len = dlen;
  return lamb_gpu_matrix_upload(c, &sec, 1, handle);
}

}  // extern "C"
