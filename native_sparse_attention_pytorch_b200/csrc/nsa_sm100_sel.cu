// Tensor-core (tcgen05 / TMEM / TMA) family for the selected-block branch.
//
// The computation is organised KV-block-stationary.  An integer pre-pass turns
// the per-query selection (idx, mask) into, for every (batch, KV head, KV
// block j), the list of queries that attend block j -- the selected slots and,
// for the own block, its 64 queries.  A list is cut into chunks of 128/G
// queries; with the G query heads of the group that makes a dense 128-row
// tile.  A persistent CTA takes an item (one list, up to kChunksPerItem
// chunks), brings the K and V tiles of block j into shared memory once with
// TMA, and for every chunk gathers the 128 query rows and runs dense tcgen05
// MMAs against the resident tiles:
//
//   forward : S = Q K^T -> per-row softmax of that block -> O_part = P V.
//             Every (row, slot) writes its partial output (sum of p v, bf16)
//             and its (max, sum); a second kernel merges the partials of a row
//             into the output and the log-sum-exp.
//   backward: S = Q K^T and dP = dO V^T -> P = exp(S - lse), dS = P (dP - delta)
//             -> dV += P^T dO and dK += dS^T Q stay in tensor memory across the
//             chunks of the item (flushed once with fp32 reductions), and
//             dQ_chunk = dS K goes out as a partial per (row, slot) that a
//             last kernel sums into dq.
//
// All operand tiles are [rows x 64 columns] bf16 with 128-byte rows and the
// 128-byte swizzle, which serves both as a K-major and as an MN-major operand.
// Every wait on an mbarrier is bounded; a wait that runs out raises a status
// word in the work buffer instead of hanging, and the CTA still frees its
// tensor memory.

#include <cuda_bf16.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "nsa_common.cuh"
#include "nsa_kernels.h"
#include "nsa_sm100_ptx.cuh"

namespace nsa {

using namespace ptx;

constexpr int kBlock = 64;           // keys per selection block served by this family
constexpr int kRows = 128;           // rows of a chunk tile (queries x heads of the group)
constexpr int kChunksPerItem = 16;   // chunks a CTA processes per resident K/V tile
constexpr uint32_t kInvalidEntry = 0xffffffffu;

// Which keys a query attends.  The three NSA branches differ only in this rule; everything after the index pre-pass
// (lists of (query, slot) per key block, dense 128-row chunks) is shared.
//   kModeSel : the blocks named by idx/mask plus the own block as `diag` says         (slot = position in idx; own = nsel)
//   kModeSwa : causal window, keys i-window..i                                         (slot = own block - key block)
//   kModeCmp : compressed keys, rows 0 .. num_mem + i/stride - 1 of a [num_mem + ncb]-row key tensor (slot = key block)
enum { kModeSel = 0, kModeSwa = 1, kModeCmp = 2 };

struct BlockRule {
  const int64_t* idx;
  const uint8_t* mask;
  int N;        // queries
  int nkb;      // key blocks of 64 rows
  int nsel;     // slots in idx (kModeSel)
  int ns;       // slots a query can have: the partial results of a query are indexed 0..ns-1
  int diag, mode, window, stride, num_mem;
};

// Slot s of query i (selection head bh): does it exist, and which key block is it?
template <int MODE>
__device__ __forceinline__ bool slot_block(const BlockRule& R, int bh, int i, int s, int* blk) {
  if (MODE == kModeSel) {
    if (s == R.nsel) {
      *blk = i / 64;
      return R.diag != NSA_DIAG_NONE;
    }
    const int64_t at = ((int64_t)bh * R.N + i) * R.nsel + s;
    const int64_t b = R.idx[at];
    *blk = (int)b;
    return R.mask[at] != 0 && b >= 0 && b < R.nkb;
  }
  if (MODE == kModeSwa) {
    *blk = i / 64 - s;
    return *blk >= 0 && *blk * 64 + 63 >= i - R.window;
  }
  *blk = s;
  return s * 64 < R.num_mem + i / R.stride;
}

struct SelPlan {
  int nqb, nkb, ns, G, QT, nlists;
  int64_t entries_cap, items_cap;
  // byte offsets into the work buffer
  int words;             // 32-bit words of slot bits per query
  int64_t off_status, off_num_items, off_totals, off_list_base, off_list_item, off_cursors, off_bits, off_items, off_entries, off_positions;
  int64_t off_partial, off_stats, off_delta;
  int slices, pairs_per_slice;   // backward: launches over the (batch, KV head) pairs
  int64_t index_bytes;   // the leading part that holds the index (what the backward can take from the forward)
  int64_t total_bytes;
};

struct SelParams {
  const __nv_bfloat16 *q, *dout;
  __nv_bfloat16* out;
  int64_t q_sb, q_sh, q_sn, do_sb, do_sh, do_sn, o_sb, o_sh, o_sn;
  const int64_t* idx;
  const uint8_t* mask;
  const uint32_t* entries;
  const int4* items;
  const int* num_items;    // [0] items, [1] the tag the item kernel left
  const int* list_item;    // per list (and one more): its first item
  const int* positions;    // kModeSel: [B*Hkv*N][ns], the entry of every (query, slot), -1 where the query does not have it
  int bh0, bh1;            // backward: the (batch, KV head) pairs of this launch, whose partial results share the buffer
  const uint32_t* bits;    // [B*Hkv*N][words]: the slots a query has (kModeSel)
  int words;
  __nv_bfloat16* dq_lp;    // optional bf16 dq with its own batch / head / row strides (dq merge)
  int64_t dq_sb, dq_sh, dq_sn;
  __nv_bfloat16* dkv_lp;   // optional: where the dq merge rounds dk and dv (which lie one behind the other) to
  uint32_t index_tag;
  __nv_bfloat16* partial;
  float2* stats;
  float* lse;
  const float* delta;
  float *dq, *dk, *dv, *slot_grads;
  int* status;
  int B, Hq, Hkv, N, Nk, G, nsel, nfb, diag;   // nfb = key blocks (lists per head); N queries, Nk key rows
  int ns;                                       // slots per query in the partial buffers
  float scale, scale_log2;
  BlockRule rule;
  // compressed branch only: the head-averaged logits of every compressed block column, [B, Hkv, N, ncb] fp32
  float* importance;
  int ncb, round_bf16;
  // or, instead of it, those logits averaged over runs of `cpf` columns (one value per selection block of
  // pool_block = cpf * stride queries) and rounded to bf16: [B, Hkv, N, pool_cols], written for the blocks that lie
  // wholly before the query's own block
  __nv_bfloat16* pooled;
  int cpf, pool_cols, pool_block;
};

// The partial results of the forward lie chunk by chunk, as they leave shared memory: row r of chunk c at (128 c + r) * 2 D
// bytes, its 16-byte pieces exchanged by r & 7.  A chunk is then one bulk store, which leaves the load / store units to
// the gathers; the merge finds the row of (query, slot) through `positions` (row = entry * G + head of the group) and
// reads the G heads side by side.
template <int D>
__device__ __forceinline__ const uint4* partial_piece(const __nv_bfloat16* partial, int64_t row, int part) {
  return reinterpret_cast<const uint4*>(partial) + row * (D / 8) + (part ^ (int)(row & 7));
}

// Number of items of the index, or 0 (and status 2) when the index was not built for these sizes: a caller-kept
// index that belongs to another problem, or a buffer nobody filled, must not steer any address.
__device__ __forceinline__ bool foreign_index(const SelParams& P) { return (uint32_t)P.num_items[1] != P.index_tag; }
__device__ __forceinline__ int item_count(const SelParams& P) {
  if (foreign_index(P)) {
    if (threadIdx.x == 0) atomicOr(P.status, 2);
    return 0;
  }
  return P.num_items[0];
}

// ---- index pre-pass --------------------------------------------------------------
//
// Four short integer kernels, at batch 4, 8192 tokens, 4 KV heads, 16 slots 2 + 16 + 11 + 40 us, most of it the latency of the
// look-ups: clear the list totals, count, lay the lists out, fill them.  A block owns 128 queries of one (batch, KV head); it counts in shared memory and touches a list's total and cursor once, so the order of the
// query blocks inside a list is whatever order the blocks arrive in.  Nothing downstream depends on it: every
// (row, slot) partial is computed from its own row alone, and dk / dv are sums of fp32 reductions in any case.
constexpr int kIndexQueries = 128;

__global__ void __launch_bounds__(256) sel_clear_kernel(int* totals, int nlists) {
  const int l = blockIdx.x * 256 + threadIdx.x;
  if (l < nlists) totals[l] = 0;
}

// Takes a place in hist[blk] for every lane with a block.  The queries of a warp mostly select different blocks: each adds for
// itself, and the slots of a batch go side by side.  Own, sliding and compressed blocks are the same for neighbours: lanes that
// hit the same list are added together (for the selected ones this took 100 cycles per slot: 2 x 3333 positions, 4 KV heads, 17
// slots filling 18.7 -> 15 us, counting 8.6 -> 6.9; 4 x 8192, 4 KV heads 42 -> 41 and 18 -> 16).
__device__ __forceinline__ void count_block(int* hist, bool valid, int blk, int lane) {
  const unsigned vm = __ballot_sync(kFullMask, valid);
  if (valid) {
    const unsigned peers = __match_any_sync(vm, blk);
    if (lane == __ffs(peers) - 1) atomicAdd(&hist[blk], __popc(peers));
  }
}

// The key blocks of kSlotBatch slots of a query, -1 where it does not have one, read together.
constexpr int kSlotBatch = 16;
template <int MODE>
__device__ __forceinline__ void load_blocks(const BlockRule& R, int bh, int i, int s0, int (&blk)[kSlotBatch]) {
#pragma unroll
  for (int u = 0; u < kSlotBatch; ++u) {
    int b = -1;
    const bool valid = i < R.N && s0 + u < R.ns && slot_block<MODE>(R, bh, i, s0 + u, &b);
    blk[u] = valid ? b : -1;
  }
}

// totals[list] += entries of this block's queries; bits[(bh*N + i)*words + w]: which of its slots query i has
template <int MODE>
__global__ void __launch_bounds__(kIndexQueries) sel_count_kernel(const BlockRule R, int* totals, uint32_t* bits, int words) {
  extern __shared__ int hist[];
  const int bh = blockIdx.y * gridDim.z + blockIdx.z;  // bh = b*Hkv + h
  const int lane = threadIdx.x & 31;
  for (int j = threadIdx.x; j < R.nkb; j += kIndexQueries) hist[j] = 0;
  __syncthreads();
  const int i = blockIdx.x * kIndexQueries + threadIdx.x;
  for (int w = 0; w < words; ++w) {
    uint32_t mine = 0;
    const int s_end = min(R.ns, w * 32 + 32);
    for (int s = w * 32; s < s_end; s += kSlotBatch) {
      int blk[kSlotBatch];
      load_blocks<MODE>(R, bh, i, s, blk);
#pragma unroll
      for (int u = 0; u < kSlotBatch; ++u) {
        if (s + u >= s_end) break;
        mine |= blk[u] >= 0 ? 1u << ((s + u) & 31) : 0u;
        if (MODE == kModeSel && s + u < R.nsel) {
          if (blk[u] >= 0) atomicAdd(&hist[blk[u]], 1);
        } else {
          count_block(hist, blk[u] >= 0, blk[u], lane);
        }
      }
    }
    if (i < R.N) bits[((int64_t)bh * R.N + i) * words + w] = mine;
  }
  __syncthreads();
  for (int j = threadIdx.x; j < R.nkb; j += kIndexQueries)
    if (hist[j] > 0) atomicAdd(&totals[bh * R.nkb + j], hist[j]);
}

// Exclusive prefix over the block's 1024 threads of two values at once; returns the totals.
__device__ __forceinline__ int2 block_scan2(int2 v, int2* total, int2 (*warp_sums)[32]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int2 inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(kFullMask, inc.x, o), b = __shfl_up_sync(kFullMask, inc.y, o);
    if (lane >= o) { inc.x += a; inc.y += b; }
  }
  if (lane == 31) (*warp_sums)[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int2 s = (*warp_sums)[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(kFullMask, s.x, o), b = __shfl_up_sync(kFullMask, s.y, o);
      if (lane >= o) { s.x += a; s.y += b; }
    }
    (*warp_sums)[lane] = s;
  }
  __syncthreads();
  const int2 before = warp > 0 ? (*warp_sums)[warp - 1] : make_int2(0, 0);
  *total = (*warp_sums)[31];
  __syncthreads();
  return make_int2(before.x + inc.x - v.x, before.y + inc.y - v.y);
}

// List bases (padded to whole chunks), the fill cursors and the item table; one CTA, every thread owns a run of lists.
// A list is cut into items of at most kChunksPerItem chunks, fewer when the whole problem has few chunks: an item is
// what one CTA walks serially, so a problem of a few hundred chunks in items of sixteen leaves most of the chip idle.
// The line is 16 items per SM at dim_head 64 and 8 at 128, where an item's K/V loads and dK/dV flush cost twice as much
// and the forward has two CTAs per SM instead of four; below it these costs outweigh the imbalance of long items.  All
// kernels of the selected branch, forward + backward, in us with 4 / 8 / 16 / 32 items per SM:
//   64:  1 x 3001, 16 / 4 heads 145 147 160 160; 4 x 2048, 8 / 4 307 285 288 311; 2 x 4096, 16 / 2 537 521 505 528;
//        1 x 8192, 32 / 4 1024 1023 994 989; 4 x 8192, 32 / 4 the same within 0.2 % (3763)
//   128: 1 x 3001, 16 / 2 273 268 308 308; 4 x 2048, 8 / 4 558 519 514 589; 2 x 4096, 16 / 2 1061 1024 981 1020;
//        2 x 8192, 16 / 4 1371 1370 1278 1281; 1 x 8192, 32 / 4 2093 2093 2035 2024
// so either line is right for some sizes and costs others: 8 at 128 keeps the short ones from losing 15 %, where 16 would
// give the longer ones 3 to 7 %.
static int items_target(int D) { return 148 * (D == 64 ? 16 : 8); }
__global__ void __launch_bounds__(1024) sel_items_kernel(const int* totals, int* list_base, int* list_item, int* cursors, int4* items,
                                                         int* num_items, int nlists, int QT, int target, uint32_t tag) {
  __shared__ int2 warp_sums[32];
  const int per = (nlists + 1023) / 1024;
  const int l0 = min(nlists, (int)threadIdx.x * per), l1 = min(nlists, l0 + per);
  int chunks = 0;
  for (int l = l0; l < l1; ++l) chunks += (totals[l] + QT - 1) / QT;
  int2 all;
  block_scan2(make_int2(chunks, 0), &all, &warp_sums);
  const int cpi = max(1, min(kChunksPerItem, all.x / target));
  int nit = 0;
  for (int l = l0; l < l1; ++l) nit += ((totals[l] + QT - 1) / QT + cpi - 1) / cpi;
  int2 at = block_scan2(make_int2(chunks, nit), &all, &warp_sums);
  int base = at.x * QT, ibase = at.y;
  for (int l = l0; l < l1; ++l) {
    const int nch = (totals[l] + QT - 1) / QT;
    list_base[l] = base;
    list_item[l] = ibase;
    cursors[l] = base;
    for (int c0 = 0; c0 < nch; c0 += cpi) items[ibase++] = make_int4(l, c0, min(cpi, nch - c0), base + c0 * QT);
    base += nch * QT;
  }
  if (threadIdx.x == 0) {
    list_item[nlists] = all.y;
    num_items[0] = all.y;
    num_items[1] = (int)tag;   // marks the index as built, and for which sizes
  }
}

// writes the entries (query | slot << 24) and, for the forward, where each one is, and pads every list to whole chunks
template <int MODE>
__global__ void __launch_bounds__(kIndexQueries) sel_fill_kernel(const BlockRule R, const int* totals, const int* list_base,
                                                                 int* cursors, uint32_t* entries, int* positions, int QT) {
  extern __shared__ int cursor[];
  const int bh = blockIdx.y * gridDim.z + blockIdx.z;
  const int lane = threadIdx.x & 31;
  for (int j = threadIdx.x; j < R.nkb; j += kIndexQueries) cursor[j] = 0;
  __syncthreads();
  const int i = blockIdx.x * kIndexQueries + threadIdx.x;
  for (int s = 0; s < R.ns; s += kSlotBatch) {
    int blk[kSlotBatch];
    load_blocks<MODE>(R, bh, i, s, blk);
#pragma unroll
    for (int u = 0; u < kSlotBatch; ++u) {
      if (s + u >= R.ns) break;
      if (MODE == kModeSel && s + u < R.nsel) {
        if (blk[u] >= 0) atomicAdd(&cursor[blk[u]], 1);
      } else {
        count_block(cursor, blk[u] >= 0, blk[u], lane);
      }
    }
  }
  __syncthreads();
  for (int j = threadIdx.x; j < R.nkb; j += kIndexQueries) {
    const int mine = cursor[j];
    if (mine > 0) cursor[j] = atomicAdd(&cursors[bh * R.nkb + j], mine);
    if (blockIdx.x == 0) {
      const int l = bh * R.nkb + j, end = list_base[l] + totals[l], stop = (end + QT - 1) / QT * QT;   // bases are multiples of QT
      for (int p = end; p < stop; ++p) entries[p] = kInvalidEntry;
    }
  }
  __syncthreads();
  for (int s = 0; s < R.ns; s += kSlotBatch) {
    int blk[kSlotBatch];
    load_blocks<MODE>(R, bh, i, s, blk);
    int pos[kSlotBatch];
#pragma unroll
    for (int u = 0; u < kSlotBatch; ++u) {
      pos[u] = -1;
      if (s + u >= R.ns) continue;
      const bool valid = blk[u] >= 0;
      if (MODE == kModeSel && s + u < R.nsel) {
        if (valid) pos[u] = atomicAdd(&cursor[blk[u]], 1);
        continue;
      }
      const unsigned vm = __ballot_sync(kFullMask, valid);
      if (valid) {
        const unsigned peers = __match_any_sync(vm, blk[u]);
        const int leader = __ffs(peers) - 1;
        if (lane == leader) pos[u] = atomicAdd(&cursor[blk[u]], __popc(peers));
        pos[u] = __shfl_sync(peers, pos[u], leader) + __popc(peers & ((1u << lane) - 1u));
      }
    }
#pragma unroll
    for (int u = 0; u < kSlotBatch; ++u) {
      if (s + u >= R.ns) break;
      if (pos[u] >= 0) entries[pos[u]] = (uint32_t)i | ((uint32_t)(s + u) << 24);
      if (MODE == kModeSel && i < R.N) positions[((int64_t)bh * R.N + i) * R.ns + s + u] = pos[u];
    }
  }
}

// ---- shared pieces of the two main kernels -----------------------------------------

struct RowInfo {
  int i, slot;
  int lo, lim;   // first and last visible key column of the block (lim = -1: the row is padding)
  bool valid;
};

__device__ __forceinline__ RowInfo decode_row(uint32_t e, int j, const BlockRule& R) {
  RowInfo r;
  r.valid = e != kInvalidEntry;
  r.i = (int)(e & 0xffffffu);
  r.slot = (int)(e >> 24);
  r.lo = 0;
  r.lim = kBlock - 1;
  if (R.mode == kModeSel) {
    if (r.slot == R.nsel && R.diag == NSA_DIAG_CAUSAL) r.lim = r.i - j * kBlock;
  } else if (R.mode == kModeSwa) {
    r.lim = min(kBlock - 1, r.i - j * kBlock);
    r.lo = max(0, r.i - R.window - j * kBlock);
  } else {
    r.lim = min(kBlock - 1, R.num_mem + r.i / R.stride - 1 - j * kBlock);
  }
  if (!r.valid) {
    r.lo = 0;      // (the index of a padding entry would put it past the eight bits the backward keeps it in)
    r.lim = -1;
  }
  return r;
}

// The largest of 32 values
__device__ __forceinline__ float max32(const float (&s)[32]) {
  float m[4] = {fmaxf(s[0], s[1]), fmaxf(s[2], s[3]), fmaxf(s[4], s[5]), fmaxf(s[6], s[7])};
#pragma unroll
  for (int x = 8; x < 32; x += 8)
#pragma unroll
    for (int k = 0; k < 4; ++k) m[k] = max3(m[k], s[x + 2 * k], s[x + 2 * k + 1]);
  return fmaxf(max3(m[0], m[1], m[2]), m[3]);
}
// s = 2^(s * scale2 - off) in place; the sum, in fp32 (four partial sums: values x with equal x % 4)
__device__ __forceinline__ float exp_row32(float (&s)[32], float scale_log2, float off) {
  const uint64_t scale2 = pack2(scale_log2, scale_log2), off2 = pack2(-off, -off);
  uint64_t l0 = 0ull, l1 = 0ull;
#pragma unroll
  for (int x = 0; x < 32; x += 4) {
    unpack2(fma2(pack2(s[x], s[x + 1]), scale2, off2), s[x], s[x + 1]);
    unpack2(fma2(pack2(s[x + 2], s[x + 3]), scale2, off2), s[x + 2], s[x + 3]);
#pragma unroll
    for (int k = 0; k < 4; ++k) s[x + k] = ex2(s[x + k]);
    l0 = add2(l0, pack2(s[x], s[x + 1]));
    l1 = add2(l1, pack2(s[x + 2], s[x + 3]));
  }
  float a, b, c, d;
  unpack2(l0, a, b);
  unpack2(l1, c, d);
  return (a + b) + (c + d);
}

// ---- forward -------------------------------------------------------------------------

// Forward of the selected-block branch.  A CTA of 256 threads walks gather -> S -> softmax -> P V -> store chunk by
// chunk; several CTAs share an SM (4 at dim_head 64) and fill each other's waits.  Two threads share a row (32 of the
// block's 64 columns each; they exchange maximum and sum through shared memory), which halves the serial work per thread.
// What bounds it: the gather of the Q rows, 18 bytes per clock and SM out of the L2 (900 cycles for the 16 KB of a chunk
// at dim_head 64, measured with nothing else running, whatever the number of copying warps; as TMA boxes or gathers 1900
// and more), plus 440 for the bulk store of the partial rows; the chunk takes 1700.  Batch 4, 8192 positions, 32 / 4 heads of
// 64: 1.10 ms with the partial rows stored row by row through the load / store units, 0.96 with bulk stores, 0.90 with waits
// of whole warps (a lane that polls takes a quarter of the issue slots), 0.85 with two values per instruction, three-way
// maxima and gathers of one multiplication per row; 65536 positions, 64 / 8 heads of 128 9.1, 7.8 and now 7.0 ms.
// A thread's rows are RPP apart, with up to RPP heads per KV head all of the same head (at dim_head 128 every row of 16 heads:
// RPP is 16): `head` is that head's row 0 at the thread's piece.  Row strides are 32-bit (see problem_fwd).
template <int D>
struct GatherTile {
  static constexpr int CH = D / 8;               // 16-byte pieces per row
  static constexpr int RPP = 2 * kRows / CH;     // rows covered by one pass of the 256 threads
  __device__ __forceinline__ static void issue(uint32_t tile, const __nv_bfloat16* head, uint32_t stride_n, const uint32_t* entries,
                                               int g_shift, int tid) {
    const int sub = tid % CH, r0 = tid / CH;
    uint32_t ev[kRows / RPP];
#pragma unroll
    for (int it = 0; it < kRows / RPP; ++it) ev[it] = __ldg(entries + ((r0 + it * RPP) >> g_shift));
    const uint32_t dst = tile + (sub / 8) * (kRows * 128) + sw128_offset(r0, sub % 8);   // (RPP is a multiple of 8)
#pragma unroll
    for (int it = 0; it < kRows / RPP; ++it) {
      const bool valid = ev[it] != kInvalidEntry;
      const uint32_t i = valid ? ev[it] & 0xffffffu : 0u;
      cp_async16(dst + it * RPP * 128, head + (uint64_t)i * stride_n, valid ? 16u : 0u);
    }
  }
};

template <int D>
__global__ void __launch_bounds__(2 * kRows, D == 64 ? 4 : 2)
sel_fwd_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const SelParams P) {
  constexpr int NC = D / 64;
  extern __shared__ uint8_t smem_raw[];
  __shared__ int abort_flag;
  __shared__ uint32_t tmem_slot;
  __shared__ __align__(8) uint64_t bars[3];
  __shared__ float xmax[2][kRows], xsum[2][kRows];
  const int nitems = item_count(P);
  if ((int)blockIdx.x >= nitems) return;

  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sQ = base, sK = sQ + NC * 16384, sV = sK + NC * 8192, sStage = sV + NC * 8192;
  const uint32_t bar_kv = smem_u32(&bars[0]), bar_s = smem_u32(&bars[1]), bar_o = smem_u32(&bars[2]);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int half = tid >> 7, row = tid & (kRows - 1);   // this thread: columns 32*half .. 32*half+31 of row `row`
  constexpr uint32_t kCols = D == 64 ? 128 : 256;

  if (tid == 0) {
    abort_flag = 0;
    mbar_init(bar_kv, 1);
    mbar_init(bar_s, 1);
    mbar_init(bar_o, 1);
    fence_mbar_init();
    prefetch_tensormap(&tmK);
    prefetch_tensormap(&tmV);
  }
  __syncthreads();
  if (warp == 0) {
    tmem_alloc(smem_u32(&tmem_slot), kCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tm = tmem_slot;
  const uint32_t tm_lane = tm + ((uint32_t)((warp & 3) * 32) << 16);   // warps w and w + 4 share a lane quarter
  const uint32_t tS = 0, tO = 64;

  const int G = P.G, QT = kRows / G, g_shift = 31 - __clz(G);
  const int q_local = row >> g_shift;
  uint32_t ph_kv = 0, ph_s = 0, ph_o = 0;
  constexpr uint32_t idS = instr_desc_bf16(128, 64, false, false);
  constexpr uint32_t idO = instr_desc_bf16(128, D, false, true);

  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const int4 item = P.items[it];
    const int list = item.x, j = list % P.nfb, bh = list / P.nfb, h = bh % P.Hkv, b = bh / P.Hkv;
    if (tid == 0) {
      mbar_arrive_expect_tx(bar_kv, 2 * NC * 8192);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        tma_load_4d(sK + c * 8192, &tmK, bar_kv, c * 64, j * kBlock, h, b);
        tma_load_4d(sV + c * 8192, &tmV, bar_kv, c * 64, j * kBlock, h, b);
      }
    }
    const __nv_bfloat16* const q_head =
        P.q + b * P.q_sb + (int64_t)(h * G + (tid / GatherTile<D>::CH & (G - 1))) * P.q_sh + tid % GatherTile<D>::CH * 8;
    bool prefetched = false;
    for (int c = 0; c < item.z; ++c) {
      const uint32_t* chunk_entries = P.entries + item.w + c * QT;
      const uint32_t e = chunk_entries[q_local];
      if (!prefetched) GatherTile<D>::issue(sQ, q_head, (uint32_t)P.q_sn, chunk_entries, g_shift, tid);
      cp_async_commit();
      cp_async_wait<0>();
      fence_proxy_async_smem();
      __syncthreads();
      if (warp == 0) {   // the whole warp runs the issue code, one elected lane issues
        if (c == 0) {
          mbar_wait_bounded(bar_kv, ph_kv, &abort_flag);
          __syncwarp();
        }
        tc_fence_after_sync();
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t ch = k / 4, in = (k % 4) * 32;
          mma_bf16_elect(tm + tS, smem_desc_sw128(sQ + ch * 16384 + in, 16), smem_desc_sw128(sK + ch * 8192 + in, 16),
                         idS, k > 0);
        }
        mma_commit_elect(bar_s);
      }
      __syncwarp();
      mbar_wait_warp(bar_s, ph_s, &abort_flag);
      ph_s ^= 1;
      tc_fence_after_sync();
      // S is complete, so the Q tile is free: request the next chunk's rows now; they travel while this chunk's
      // softmax, second MMA and output run
      prefetched = c + 1 < item.z;
      if (prefetched)
        GatherTile<D>::issue(sQ, q_head, (uint32_t)P.q_sn, chunk_entries + QT, g_shift, tid);
      __syncwarp();
      const RowInfo r = decode_row(e, j, P.rule);
      const int lim = r.lim - half * 32;   // last visible column of this thread's half (negative: none)
      float s[32];
      tmem_ld32(tm_lane + tS + half * 32, s);
      tmem_ld_wait();
      const bool all_full = __all_sync(kFullMask, lim >= 31);
      float m = -INFINITY;
      if (all_full) {
        m = max32(s);
      } else {
#pragma unroll
        for (int x = 0; x < 32; ++x) m = x <= lim ? fmaxf(m, s[x]) : m;
      }
      xmax[half][row] = m;
      if (tid == 0) bulk_wait_read();   // the staging tile's last store has left shared memory (written again behind the barriers)
      __syncthreads();
      m = fmaxf(m, xmax[half ^ 1][row]);
      const float m2 = r.valid ? m * P.scale_log2 : 0.f;
      float l_half;          // the fp32 sum: the log-sum-exp stays exact although P is rounded to bf16 for the MMA
      if (all_full) {
        l_half = exp_row32(s, P.scale_log2, m2);
      } else {
        float ll[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int x = 0; x < 32; ++x) {
          s[x] = x <= lim ? ex2(fmaf(s[x], P.scale_log2, -m2)) : 0.f;
          ll[x & 3] += s[x];
        }
        l_half = (ll[0] + ll[1]) + (ll[2] + ll[3]);
      }
      xsum[half][row] = l_half;
      // P goes to the tensor cores through tensor memory, over the first half of this row's S columns (both threads
      // of the row have read their S columns: the exchange of the maxima lies in between)
      tmem_st_bf16_row32(tm_lane + tS + half * 16, s);
      tmem_st_wait();
      tc_fence_before_sync();
      __syncthreads();
      if (warp == 0) {
        tc_fence_after_sync();
#pragma unroll
        for (int k = 0; k < 4; ++k)
          mma_bf16_tmem_a_elect(tm + tO, tm + tS + k * 8, smem_desc_sw128(sV + k * 2048, 8192), idO, k > 0);
        mma_commit_elect(bar_o);
      }
      const float l = xsum[0][row] + xsum[1][row];
      const int64_t chunk = item.w / QT + c;
      __syncwarp();
      mbar_wait_warp(bar_o, ph_o, &abort_flag);
      ph_o ^= 1;
      tc_fence_after_sync();
      __syncwarp();
      // the partial row stays unnormalised (sum of p * v, at most 64 max|v|): the merge divides once per row
#pragma unroll
      for (int c2 = 0; c2 < D / 64; ++c2) {
        float t[32];
        tmem_ld32(tm_lane + tO + half * (D / 2) + c2 * 32, t);
        tmem_ld_wait();
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          uint4 v;
          v.x = pack_bf16(t[x * 8 + 0], t[x * 8 + 1]);
          v.y = pack_bf16(t[x * 8 + 2], t[x * 8 + 3]);
          v.z = pack_bf16(t[x * 8 + 4], t[x * 8 + 5]);
          v.w = pack_bf16(t[x * 8 + 6], t[x * 8 + 7]);
          const int piece = half * (D / 16) + c2 * 4 + x;   // 16-byte piece of the row
          sts_v4(sStage + row * (D * 2) + ((piece ^ (row & 7)) << 4), v);
        }
      }
      if (half == 0) P.stats[chunk * kRows + row] = make_float2(m2, l);
      fence_proxy_async_smem();
      tc_fence_before_sync();
      __syncthreads();
      if (tid == 0) {
        bulk_store(reinterpret_cast<uint8_t*>(P.partial) + chunk * (NC * 16384), sStage, NC * 16384);
        bulk_commit();
      }
    }
    ph_kv ^= 1;
    __syncthreads();   // every thread is done with this item's tiles before the next TMA overwrites them
  }

  if (tid == 0) bulk_wait_all();
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, kCols);
  if (tid == 0 && abort_flag) atomicOr(P.status, 1);
}

// Merges the partial results of head g of the group (batch, KV head) bh at query i: acc[8] of a thread's 16-byte piece
// (unnormalised), the reference maximum and the sum.  The D/8 threads of a row (neighbouring lanes) share the work on the
// slots: each looks up the position and the statistics of every D/8-th one, and hands them on by shuffles.  The kernel is a
// stream over the partial buffer: the rows' loads go six at a time (selected blocks and own block are 17 slots in the
// layers here: three rounds), the first six beside the statistics, as soon as the positions are there.
template <int D>
__device__ __forceinline__ void merge_row(const SelParams& P, int bh, int i, int g, int part, float (&acc)[8], float* M_out, float* L_out) {
  constexpr int TPR = D / 8, PER = 32 / TPR, BATCH = 6;
  const unsigned mask = (TPR == 8 ? 0xffu : 0xffffu) << (threadIdx.x & 31 & ~(TPR - 1));
  const int ns = P.ns;
  const int* positions = P.positions + ((int64_t)bh * P.N + i) * ns;
  float M = -INFINITY, L = 0.f;
#pragma unroll
  for (int x = 0; x < 8; ++x) acc[x] = 0.f;
  for (int s0 = 0; s0 < ns; s0 += 32) {
    int pos[PER];
    float2 st[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k) pos[k] = s0 + k * TPR + part < ns ? positions[s0 + k * TPR + part] : -1;
#pragma unroll
    for (int k = 0; k < PER; ++k) st[k] = pos[k] >= 0 ? P.stats[(int64_t)pos[k] * P.G + g] : make_float2(-INFINITY, 0.f);
    float w[PER];
#pragma unroll
    for (int b0 = 0; b0 < 32; b0 += BATCH) {
      if (s0 + b0 >= ns) break;
      uint4 v[BATCH];
#pragma unroll
      for (int u = 0; u < BATCH; ++u) {
        const int p = b0 + u < 32 ? __shfl_sync(mask, pos[(b0 + u) % 32 / TPR], (b0 + u) % TPR, TPR) : -1;
        v[u] = ldg_stream_if(p >= 0, partial_piece<D>(P.partial, (int64_t)p * P.G + g, part));
      }
      if (b0 == 0) {
        float m = -INFINITY, lsum = 0.f;
#pragma unroll
        for (int k = 0; k < PER; ++k) m = fmaxf(m, st[k].x);
#pragma unroll
        for (int o = TPR / 2; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(mask, m, o));
        if (m == -INFINITY) break;           // none of these slots (the same for all threads of the row)
        const float top = fmaxf(M, m), keep = ex2(M - top);
#pragma unroll
        for (int k = 0; k < PER; ++k) {
          w[k] = ex2(st[k].x - top);
          lsum = fmaf(w[k], st[k].y, lsum);
        }
#pragma unroll
        for (int o = TPR / 2; o > 0; o >>= 1) lsum += __shfl_xor_sync(mask, lsum, o);
        L = fmaf(L, keep, lsum);
        M = top;
#pragma unroll
        for (int x = 0; x < 8; ++x) acc[x] *= keep;
      }
#pragma unroll
      for (int u = 0; u < BATCH; ++u) {
        if (b0 + u >= 32) break;
        const float wu = __shfl_sync(mask, w[(b0 + u) % 32 / TPR], (b0 + u) % TPR, TPR);
        const uint32_t q[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          acc[2 * x] = fmaf(wu, __uint_as_float(q[x] << 16), acc[2 * x]);
          acc[2 * x + 1] = fmaf(wu, __uint_as_float(q[x] & 0xffff0000u), acc[2 * x + 1]);
        }
      }
    }
  }
  *M_out = M;
  *L_out = L;
}

// One group of D/8 threads per row; the heads of a group, whose partial rows are neighbours, next to each other.  Bound by
// the partial buffer's bytes: 17 slots of 1 M rows of 64 take 414-421 us = 0.89 of the copy bandwidth (478 us with branches
// around the loads and nine rows at a time, 520 us with eight behind the statistics), 7 slots of 48 k rows of 128 27 us (42).
// Four blocks per SM (64 registers) with six rows in flight per thread; measured beside them, at 64 and (with the combine,
// 65536 positions, 64 heads) 128 features: three blocks and nine rows 456 us and 4.89 ms, two and seventeen 542 and 5.86, four and nine
// 460 and 4.57, five and six 482 and 4.75, five and four 545 and 4.54, six and four 554 and 5.26; four and six 421 and 4.39.
template <int D>
__global__ void __launch_bounds__(256, 4) sel_merge_kernel(const SelParams P) {
  constexpr int TPR = D / 8;
  const uint32_t t = blockIdx.x * (256 / TPR) + threadIdx.x / TPR;     // 32 bits hold every row id (see `supported`)
  const int part = threadIdx.x % TPR;
  if (t >= (uint32_t)P.B * P.Hq * P.N || foreign_index(P)) return;
  const uint32_t g_shift = 31 - __clz(P.G), query = t >> g_shift;
  const int g = (int)(t & (P.G - 1)), bh = (int)(query / (uint32_t)P.N), i = (int)query - bh * P.N;
  const int b = bh / P.Hkv, hq = (bh - b * P.Hkv) * P.G + g;
  float acc[8], M, L;
  merge_row<D>(P, bh, i, g, part, acc, &M, &L);
  const float inv = L > 0.f ? 1.f / L : 0.f;
  uint4 o;
  o.x = pack_bf16(acc[0] * inv, acc[1] * inv);
  o.y = pack_bf16(acc[2] * inv, acc[3] * inv);
  o.z = pack_bf16(acc[4] * inv, acc[5] * inv);
  o.w = pack_bf16(acc[6] * inv, acc[7] * inv);
  *reinterpret_cast<uint4*>(P.out + b * P.o_sb + (int64_t)hq * P.o_sh + (int64_t)i * P.o_sn + part * 8) = o;
  if (part == 0) P.lse[((int64_t)b * P.Hq + hq) * P.N + i] = L > 0.f ? (M + log2f(L)) * kLn2 : -INFINITY;
}

// The merge of the selected branch that also does the gated combine and the head merge (and, with several
// destinations, the all-gather of the head-sharded layout): the merged selected row is rounded to bf16 as the tensor
// between the two kernels would be, combined with the compressed and the sliding row exactly as combine_gather_kernel
// does (the same three fused multiply-adds in the same order), and stored into every destination.  The selected
// branch's own output tensor is written where the caller wants it.  Thread groups walk the rows position-major
// (b, i, head), so that the heads of one position land next to each other in the destinations' [B, N, features] rows.
template <int D, bool MC>
__global__ void __launch_bounds__(256, 4) sel_merge_combine_kernel(const SelParams P, const CombineParams Cp, const GatherTargets Gt) {
  constexpr int TPR = D / 8;
  const uint32_t t = blockIdx.x * (256 / TPR) + threadIdx.x / TPR;     // 32 bits hold every row id (see `supported`)
  const int part = threadIdx.x % TPR;
  if (t < (uint32_t)P.B * P.Hq * P.N && !foreign_index(P)) {
    const uint32_t token = t / (uint32_t)P.Hq;
    const int hq = (int)(t - token * P.Hq), b = (int)(token / (uint32_t)P.N), i = (int)token - b * P.N, g_shift = 31 - __clz(P.G);
    const int64_t row = ((int64_t)b * P.Hq + hq) * P.N + i;
    float acc[8], M, Lsum;
    merge_row<D>(P, b * P.Hkv + (hq >> g_shift), i, hq & (P.G - 1), part, acc, &M, &Lsum);
    const float inv = Lsum > 0.f ? 1.f / Lsum : 0.f;
    if (part == 0 && P.lse != nullptr) P.lse[row] = Lsum > 0.f ? (M + log2f(Lsum)) * kLn2 : -INFINITY;
    // combine: gates in the order compressed, selected, sliding
    const __nv_bfloat16* g = (const __nv_bfloat16*)Cp.gates + b * Cp.g_sb + hq * Cp.g_sh + (int64_t)i * Cp.g_sn;
    const float g0 = gate_value(g[0], Cp.logits), g1 = gate_value(g[1], Cp.logits), g2 = gate_value(g[2], Cp.logits);
    const uint4 rc = *reinterpret_cast<const uint4*>((const __nv_bfloat16*)Cp.o[0] + b * Cp.o_sb[0] + hq * Cp.o_sh[0] +
                                                     (int64_t)i * Cp.o_sn[0] + part * 8);
    const uint4 rw = *reinterpret_cast<const uint4*>((const __nv_bfloat16*)Cp.o[2] + b * Cp.o_sb[2] + hq * Cp.o_sh[2] +
                                                     (int64_t)i * Cp.o_sn[2] + part * 8);
    const uint32_t qc[4] = {rc.x, rc.y, rc.z, rc.w}, qw[4] = {rw.x, rw.y, rw.z, rw.w};
    uint32_t packed[4], sel[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      // the selected row as its bf16 tensor holds it
      const uint32_t os = sel[x] = pack_bf16(acc[2 * x] * inv, acc[2 * x + 1] * inv);
      float lo = fmaf(g0, __uint_as_float(qc[x] << 16), 0.f);
      float hi = fmaf(g0, __uint_as_float(qc[x] & 0xffff0000u), 0.f);
      lo = fmaf(g1, __uint_as_float(os << 16), lo);
      hi = fmaf(g1, __uint_as_float(os & 0xffff0000u), hi);
      lo = fmaf(g2, __uint_as_float(qw[x] << 16), lo);
      hi = fmaf(g2, __uint_as_float(qw[x] & 0xffff0000u), hi);
      packed[x] = pack_bf16(lo, hi);
    }
    if (P.out != nullptr)
      *reinterpret_cast<uint4*>(P.out + b * P.o_sb + (int64_t)hq * P.o_sh + (int64_t)i * P.o_sn + part * 8) = make_uint4(sel[0], sel[1], sel[2], sel[3]);
    const int64_t at = ((int64_t)b * P.N + i) * Gt.total_features + Gt.feature_offset + (int64_t)hq * D + part * 8;
    if (MC) {
      asm volatile("multimem.st.weak.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"((__nv_bfloat16*)Gt.outs[0] + at),
                   "f"(__uint_as_float(packed[0])), "f"(__uint_as_float(packed[1])), "f"(__uint_as_float(packed[2])),
                   "f"(__uint_as_float(packed[3]))
                   : "memory");
    } else {
      const int rot = (int)(blockIdx.x % (unsigned)Gt.num_outs);
      for (int r = 0; r < Gt.num_outs; ++r) {
        int k = r + rot;
        if (k >= Gt.num_outs) k -= Gt.num_outs;
        *reinterpret_cast<uint4*>((__nv_bfloat16*)Gt.outs[k] + at) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
      }
    }
  }
  if (MC) __threadfence_system();
}

// ---- forward of the dense causal branches, query-tile stationary ---------------------------------------------
//
// The compressed and the sliding-window branch attend a contiguous range of key blocks per query, the same range for
// neighbouring queries.  For them the key-block-stationary form above pays for partial results it does not need: here a
// tile of 128/G consecutive queries (128 rows with the G heads of the group) stays, the key blocks it can see pass by,
// and the output accumulator stays in tensor memory, as in a flash-attention forward.  No index, no partial results.
// One persistent CTA per SM with fixed roles:
//   warps 0-7, 8-15 two streams: each has its own query tile (neighbours of one head), two S buffers and its own O in
//                   tensor memory.  Two threads share a row (32 of a block's 64 columns each; they exchange maxima).
//                   Softmax of block t: read S, importance, maximum, exponentials, P back over S's columns as bf16.
//   warps 16, 17    issue the tcgen05.mma of a stream each: PV(t), then S(t+2) into the buffer that PV(t) has just read;
//                   S of the next tile's first blocks follows the last PV without a gap.
//   warp 18         TMA: K and V blocks through a ring shared by both streams, and the next Q tiles as soon as the last S
//                   of the present ones is complete.
// What bounds it: per 128 x 64 tile the exponentials take 512 cycles (16 per clock) and the tensor cores 512 at dim_head
// 128; the roles reach about three times that (compressed branch with pooled importance 2000 cycles, sliding 1500), most
// of it waits inside the softmax warps.  Sharing K / V matters: tile loads run at 29 bytes per clock and SM, 1100 cycles
// for the 32 KB of a key block at dim_head 128.  One issuing warp per stream, because an issuing warp needs some 100
// cycles per MMA next to the softmax warps: one for both streams took 15 % longer.
// 65536 positions, 64 / 8 heads of 128: compressed 11.5 -> 7.8 ms, sliding (window 512) 2.6 -> 1.6 ms; 2 x 16384, 16 / 4
// heads of 64: 419 -> 289 us and 290 -> 160 us (before: two CTAs per SM that walked the stages one after the other).
//   * The accumulator is rescaled lazily: a row keeps its reference maximum until a block exceeds it by more than 2^8;
//     only then is the O row read from tensor memory, scaled and written back (P stays below 2^8, exact in bf16's
//     range, and the sum is fp32).
//   * MODE compressed with IMP also writes the head-averaged logits of the visible columns (the importance), or with
//     POOL their per-selection-block means: the head means of the last 128 compressed columns of every query wait in
//     a ring in shared memory, and after every key block its two warps average the selection blocks it completed.
namespace dense {
constexpr int kStreams = 2, kSoftmaxWarps = 16, kThreads = (kSoftmaxWarps + kStreams + 1) * 32;
constexpr int kRingCols = 192 + 16;          // POOL: columns per query, three key blocks' worth (rows padded against bank conflicts)
constexpr uint32_t kImpTile = 32 * 64;       // per warp: the scaled logits of its half rows as bf16
template <int D>
struct Shape {
  static constexpr int NC = D / 64;
  static constexpr int kBufs = D == 64 ? 4 : 3;                                 // K and V blocks in flight
  static constexpr uint32_t kTileQ = NC * 16384, kTileKV = NC * 8192;
  static constexpr uint32_t kTiles = kStreams * kTileQ + 2 * kBufs * kTileKV;
};
__host__ __device__ constexpr uint32_t pool_bytes(int G) { return (uint32_t)(32 / G) * kRingCols * 2; }   // per pair of warps
template <int D>
constexpr uint32_t smem_bytes(int imp_heads, bool pool) {
  return Shape<D>::kTiles + (imp_heads > 0 ? kSoftmaxWarps * kImpTile : 0) + (pool ? 8 * pool_bytes(imp_heads) : 0);
}
struct Bars {
  uint64_t q_full[2], q_free[2];
  uint64_t k_full[4], k_free[4], v_full[4], v_free[4];
  // per S buffer: a stream may be two blocks ahead of its PV, and a waiter must know the phase before its own complete
  uint64_t s_full[2][2], p_full[2][2], pv_done[2][2];
  uint64_t drain[2];
};
// Byte offset of 16-byte piece c of row r in a warp's tile of 64-byte rows: no bank conflicts between the rows of eight
// lanes that write, nor between the lanes of neighbouring queries (G rows each) that read.
template <int G>
__device__ __forceinline__ uint32_t imp_offset(int r, int c) {
  return (uint32_t)((r * 64) ^ (((r / G) & 1) << 6)) + ((uint32_t)(c ^ ((r >> 1) & 3)) << 4);
}
// The sums of G pairs of values, each in the order of a butterfly over neighbouring lanes
template <int G>
__device__ __forceinline__ uint64_t tree_sum(const uint64_t* a) {
  if constexpr (G == 1) return a[0];
  else return add2(tree_sum<G / 2>(a), tree_sum<G / 2>(a + G / 2));
}
// A word of two bf16 as two fp32 values
__device__ __forceinline__ uint64_t widen2(uint32_t w) { return pack2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
}  // namespace dense

template <int D, int MODE, int GI, bool POOL = false>   // GI: 0 = no importance output, else the heads per KV head
__global__ void __launch_bounds__(dense::kThreads, 1)
dense_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                 const SelParams P, const int streams) {
  using namespace dense;
  using S = Shape<D>;
  constexpr int NC = S::NC, kBufs = S::kBufs;
  constexpr uint32_t kTileQ = S::kTileQ, kTileKV = S::kTileKV;
  extern __shared__ __align__(1024) uint8_t dense_smem[];
  __shared__ int abort_flag;
  __shared__ uint32_t tmem_slot;
  __shared__ __align__(8) Bars bars;
  __shared__ float xchg[2][kStreams][2][kRows];   // maxima (and, at the end, sums) of the two threads of a row

  const uint32_t sQ0 = smem_u32(dense_smem), sK0 = sQ0 + kStreams * kTileQ, sV0 = sK0 + kBufs * kTileKV;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    abort_flag = 0;
    if (sQ0 & 1023u) abort_flag = 1;   // the tiles would be mis-swizzled: report instead of computing
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&bars.q_full[s]), 1);
      mbar_init(smem_u32(&bars.q_free[s]), 1);
      for (int i = 0; i < 2; ++i) {
        mbar_init(smem_u32(&bars.s_full[s][i]), 1);
        mbar_init(smem_u32(&bars.p_full[s][i]), 2 * kRows);
        mbar_init(smem_u32(&bars.pv_done[s][i]), 1);
      }
    }
    for (int i = 0; i < kBufs; ++i) {
      mbar_init(smem_u32(&bars.k_full[i]), 1);
      mbar_init(smem_u32(&bars.k_free[i]), streams);
      mbar_init(smem_u32(&bars.v_full[i]), 1);
      mbar_init(smem_u32(&bars.v_free[i]), streams);
    }
    mbar_init(smem_u32(&bars.drain[0]), 1);
    mbar_init(smem_u32(&bars.drain[1]), 1);
    fence_mbar_init();
    prefetch_tensormap(&tmQ);
    prefetch_tensormap(&tmK);
    prefetch_tensormap(&tmV);
  }
  __syncthreads();
  if (warp == 0) {
    tmem_alloc(smem_u32(&tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tm = tmem_slot;                 // stream s: S buffers at 256 s and 256 s + 64, O at 256 s + 128
  constexpr uint32_t tO = 128;

  // The n-th pair of tiles: late queries, which see the most blocks, first; heads side by side
  constexpr bool IMP = GI > 0;
  const int G = IMP ? GI : P.G, QT = kRows / G, g_shift = 31 - __clz(G), span = QT * streams;
  const int spans = (P.N + span - 1) / span, heads = P.B * P.Hkv, total = spans * heads;
  struct Tile { int i0, h, b, jb, nb; };
  auto tile_at = [&](int n) {
    Tile t;
    const int back = n / heads, bh = n - back * heads;
    t.b = bh / P.Hkv;
    t.h = bh - t.b * P.Hkv;
    t.i0 = (spans - 1 - back) * span;
    const int i_last = min(t.i0 + span - 1, P.N - 1);
    int je;
    if (MODE == kModeCmp) {
      t.jb = 0;
      je = min(P.nfb, (P.rule.num_mem + i_last / P.rule.stride + kBlock - 1) / kBlock);
    } else {
      t.jb = max(0, t.i0 - P.rule.window) / kBlock;
      je = i_last / kBlock + 1;
    }
    t.nb = je - t.jb;
    return t;
  };

  if (warp < kSoftmaxWarps) {
    // ------------------------------------------------------------------ softmax: two threads per row, 32 columns each
    const int s = warp >> 3, half = (warp >> 2) & 1, row = (warp & 3) * 32 + lane;
    const int q_local = row >> g_shift, g = row - (q_local << g_shift);
    const uint32_t tm_lane = tm + s * 256 + ((uint32_t)((warp & 3) * 32) << 16);   // warps w and w + 4 share a lane quarter
    const int pair = s * 4 + (warp & 3);
    const uint32_t imp_tile = sQ0 + S::kTiles + warp * kImpTile;
    __nv_bfloat16* const ring = reinterpret_cast<__nv_bfloat16*>(dense_smem + S::kTiles + kSoftmaxWarps * kImpTile + pair * pool_bytes(IMP ? GI : 1));
    auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + pair) : "memory"); };
    const int cpf_shift = POOL ? 31 - __clz(P.cpf) : 0, kb_shift = 6 - cpf_shift;   // selection blocks per key block
    const float inv_cpf = POOL ? 1.f / (float)P.cpf : 1.f;
    uint32_t u = 0;
    int slot = 0;                                // POOL: the ring's place for the present key block
    for (int n = s < streams ? (int)blockIdx.x : total; n < total; n += gridDim.x) {
      const Tile tile = tile_at(n);
      const int i = tile.i0 + s * QT + q_local;
      const bool valid = i < P.N;
      // last and first visible key, relative to this thread's half of a block
      const int lim_tile = (MODE == kModeCmp ? P.rule.num_mem + i / P.rule.stride - 1 : i) - half * 32;
      const int lo_tile = i - P.rule.window - half * 32;
      float m_ref = -INFINITY, l = 0.f;          // l: this thread's half of the row sum
      for (int t = 0; t < tile.nb; ++t, ++u) {
        const int j = tile.jb + t;
        const uint32_t tS = tm_lane + (u & 1) * 64;
        mbar_wait_warp(smem_u32(&bars.s_full[s][u & 1]), (u >> 1) & 1, &abort_flag);
        tc_fence_after_sync();
        float x0[32];
        tmem_ld32(tS + half * 32, x0);
        tmem_ld_wait();
        const int lim = valid ? lim_tile - j * kBlock : -1;
        const int lo = MODE == kModeCmp ? 0 : lo_tile - j * kBlock;
        if constexpr (IMP) {
          // the scaled logit of every visible block column, averaged over the G heads of the query (G neighbouring
          // rows), as the tensor of that dtype would hold it upstream: product, scaled logit and mean each rounded to
          // bf16.  The half rows of the warp go through shared memory; every lane then sums 32/G columns of its query
          // over the heads (half the instructions of a reduce-scatter by shuffles).
          constexpr int OWN = 32 / (IMP ? GI : 1);
          constexpr float inv_g = 1.f / (float)(IMP ? GI : 1);
          float mean[OWN];
          const uint64_t logit_scale = pack2(P.scale, P.scale);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const uint32_t r = pack_bf16(x0[c * 8 + 2 * k], x0[c * 8 + 2 * k + 1]);   // (one value at a time would convert at a quarter of the rate)
              float a, b2;
              unpack2(mul2(widen2(r), logit_scale), a, b2);
              w[k] = pack_bf16(a, b2);
            }
            if constexpr (GI == 1) {
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                mean[c * 8 + 2 * k] = __uint_as_float(w[k] << 16);
                mean[c * 8 + 2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
              }
            } else {
              sts_v4(imp_tile + imp_offset<GI>(lane, c), make_uint4(w[0], w[1], w[2], w[3]));
            }
          }
          const int group = lane & ((IMP ? GI : 1) - 1), first_row = lane - group, first = group * OWN;
          if constexpr (GI > 1) {
            __syncwarp();
            constexpr int PIECE = OWN < 8 ? OWN : 8;          // columns per load
#pragma unroll
            for (int p = 0; p < OWN / PIECE; ++p) {
              uint32_t w[GI][PIECE / 2];
#pragma unroll
              for (int k = 0; k < GI; ++k) {
                const int col = first + p * PIECE;
                const uint32_t at = imp_tile + imp_offset<GI>(first_row + k, col >> 3) + (col & 7) * 2;
                if constexpr (PIECE == 8) {
                  const uint4 v = lds_v4(at);
                  w[k][0] = v.x; w[k][1] = v.y; w[k][2] = v.z; w[k][3] = v.w;
                } else if constexpr (PIECE == 4) {
                  const uint2 v = lds_v2(at);
                  w[k][0] = v.x; w[k][1] = v.y;
                } else {
                  w[k][0] = lds_u32(at);
                }
              }
#pragma unroll
              for (int c = 0; c < PIECE / 2; ++c) {
                uint64_t a[GI];
#pragma unroll
                for (int k = 0; k < GI; ++k) a[k] = widen2(w[k][c]);
                unpack2(tree_sum<GI>(a), mean[p * PIECE + 2 * c], mean[p * PIECE + 2 * c + 1]);
              }
            }
          }
          if constexpr (POOL) {
            uint32_t* dst = reinterpret_cast<uint32_t*>(ring + (lane >> g_shift) * kRingCols + slot * kBlock + half * 32 + first);
#pragma unroll
            for (int x = 0; x < OWN / 2; ++x) dst[x] = pack_bf16(mean[2 * x] * inv_g, mean[2 * x + 1] * inv_g);
          } else {
            float* imp_row = P.importance + (((int64_t)tile.b * P.Hkv + tile.h) * P.N + (valid ? i : 0)) * P.ncb;
            const int col0 = j * kBlock + half * 32 + first - P.rule.num_mem;
#pragma unroll
            for (int x = 0; x < OWN; ++x) {
              const int col = col0 + x;
              if (first + x <= lim && col >= 0 && col < P.ncb) imp_row[col] = round_bf16(mean[x] * inv_g);
            }
          }
        }
        // most blocks are fully visible to every row of the warp: the others are masked first
        if (!__all_sync(kFullMask, lim >= 31 && lo <= 0)) {
#pragma unroll
          for (int x = 0; x < 32; ++x)
            if (x < lo || x > lim) x0[x] = -INFINITY;
        }
        float m = max32(x0);
        // the row maximum over both halves; behind the barrier both have also read their S columns and written the ring
        xchg[u & 1][s][half][row] = m;
        pair_sync();
        m = fmaxf(m, xchg[u & 1][s][half ^ 1][row]);
        if constexpr (POOL) {
          // the selection blocks whose last column this key block brought: mean of their cpf columns in the order and
          // with the roundings of the selection kernel's own averaging; only blocks wholly before the query's own block
          // are stored (all others have probability 0 in the selection, whatever their logits)
          const int nm = P.rule.num_mem, before = slot == 0 ? 2 : slot - 1;
          const int b_lo = t == 0 ? 0 : (j * kBlock - nm) >> cpf_shift;
          const int b_hi = min(P.pool_cols, (j * kBlock + kBlock - nm) >> cpf_shift);
          const int q0 = tile.i0 + s * QT + (((warp & 3) * 32) >> g_shift);
          __nv_bfloat16* const pooled_head = P.pooled + ((int64_t)tile.b * P.Hkv + tile.h) * P.N * P.pool_cols;
          for (int e = half * 32 + lane; e < ((32 / GI) << kb_shift); e += 64) {
            const int pq = e >> kb_shift, bb = b_lo + (e & ((1 << kb_shift) - 1));
            const int qi = q0 + pq;
            if (bb < b_hi && qi < P.N && (bb + 1) * P.pool_block <= qi) {
              const __nv_bfloat16* src = ring + pq * kRingCols;
              const int c0 = (bb << cpf_shift) + nm - j * kBlock;   // negative: in the key block before
              float sum = 0.f;
              for (int c = 0; c < (1 << cpf_shift); ++c)
                sum += __bfloat162float(src[c0 + c >= 0 ? slot * kBlock + c0 + c : (before + 1) * kBlock + c0 + c]);
              pooled_head[(int64_t)qi * P.pool_cols + bb] = __float2bfloat16_rn(sum * inv_cpf);   // cpf is a power of two
            }
          }
          slot = slot == 2 ? 0 : slot + 1;   // three places: the next block's may be written while a slow warp still reads
        }
        const float m_blk2 = m * P.scale_log2;   // -inf: nothing visible
        bool need = false;
        float alpha = 1.f;
        if (m_ref == -INFINITY) {
          m_ref = m_blk2;
        } else if (m_blk2 > m_ref + 8.f) {
          alpha = ex2(m_ref - m_blk2);
          m_ref = m_blk2;
          l *= alpha;
          need = true;
        }
        if (t > 0 && __any_sync(kFullMask, need)) {
          // some row of this warp outgrew its reference maximum: scale the accumulator rows (PV(t-1) must be complete);
          // each half scales its half of the output columns
          mbar_wait_warp(smem_u32(&bars.pv_done[s][(u - 1) & 1]), ((u - 1) >> 1) & 1, &abort_flag);
          tc_fence_after_sync();
#pragma unroll 1
          for (int c = half * (D / 2); c < (half + 1) * (D / 2); c += 16) {
            float o[16];
            tmem_ld16(tm_lane + tO + c, o);
            tmem_ld_wait();
#pragma unroll
            for (int x = 0; x < 16; ++x) o[x] *= alpha;
            tmem_st16(tm_lane + tO + c, o);
          }
          tmem_st_wait();
        }
        // a masked logit is -inf and gives 0; a row that has seen nothing yet must not compute -inf - -inf
        l += exp_row32(x0, P.scale_log2, m_ref == -INFINITY ? 0.f : m_ref);
        // P through tensor memory, over the first 32 columns of the row's S; S(t+2), which is issued after PV(t) by the
        // same lane, overwrites them only after PV(t) has read them
        tmem_st_bf16_row32(tS + half * 16, x0);
        tmem_st_wait();
        tc_fence_before_sync();
        mbar_arrive(smem_u32(&bars.p_full[s][u & 1]));
      }
      // output row: O / l
      xchg[u & 1][s][half][row] = l;
      mbar_wait_warp(smem_u32(&bars.pv_done[s][(u - 1) & 1]), ((u - 1) >> 1) & 1, &abort_flag);
      tc_fence_after_sync();
      pair_sync();
      l += xchg[u & 1][s][half ^ 1][row];
      const int64_t row_global = ((int64_t)tile.b * P.Hq + (int64_t)tile.h * G + g) * P.N + (valid ? i : 0);
      const float inv = l > 0.f ? 1.f / l : 0.f;
      // every thread stores its half of the row: four 16-byte pieces (two whole sectors) at a time, once per tile
      __nv_bfloat16* const out_row = P.out + row_global * D + half * (D / 2);
#pragma unroll 1
      for (int c = 0; c < D / 2; c += 32) {
        float o[32];
        tmem_ld32(tm_lane + tO + half * (D / 2) + c, o);
        tmem_ld_wait();
        if (valid) {
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            uint4 v;
            v.x = pack_bf16(o[x * 8 + 0] * inv, o[x * 8 + 1] * inv);
            v.y = pack_bf16(o[x * 8 + 2] * inv, o[x * 8 + 3] * inv);
            v.z = pack_bf16(o[x * 8 + 4] * inv, o[x * 8 + 5] * inv);
            v.w = pack_bf16(o[x * 8 + 6] * inv, o[x * 8 + 7] * inv);
            *reinterpret_cast<uint4*>(out_row + c + x * 8) = v;
          }
        }
        __syncwarp();
      }
      if (half == 0 && valid) P.lse[row_global] = l > 0.f ? (m_ref + log2f(l)) * kLn2 : -INFINITY;
      pair_sync();   // both have read the sums: the next tile's first block may write the same place
    }
  } else if (warp < kSoftmaxWarps + kStreams) {
    // ------------------------------------------------------------------ MMA issuer of a stream: the whole warp runs the
    // loop, one elected lane issues
    const int s = warp - kSoftmaxWarps;
    constexpr uint32_t idS = instr_desc_bf16(128, 64, false, false);
    constexpr uint32_t idO = instr_desc_bf16(128, D, false, true);
    const uint32_t tStream = tm + s * 256;
    const uint64_t dQ = smem_desc_sw128(sQ0 + s * kTileQ, 16);
    // S is issued two key blocks ahead of PV, across tile boundaries: its own position in the work
    int sn = s < streams ? (int)blockIdx.x : total, s_left = sn < total ? tile_at(sn).nb : 0;
    bool s_first = true;
    uint32_t su = 0, s_tiles = 0;
    auto issue_s = [&]() {
      const uint32_t buf = su % kBufs;
      if (s_first) mbar_wait_bounded(smem_u32(&bars.q_full[s]), s_tiles & 1, &abort_flag);
      mbar_wait_bounded(smem_u32(&bars.k_full[buf]), (su / kBufs) & 1, &abort_flag);
      __syncwarp();
      tc_fence_after_sync();
      const uint64_t dK = smem_desc_sw128(sK0 + buf * kTileKV, 16);
#pragma unroll
      for (int k = 0; k < D / 16; ++k)
        mma_bf16_elect(tStream + (su & 1) * 64, desc_advance(dQ, (k / 4) * 16384 + (k % 4) * 32),
                       desc_advance(dK, (k / 4) * 8192 + (k % 4) * 32), idS, k > 0);
      mma_commit_elect(smem_u32(&bars.s_full[s][su & 1]));
      mma_commit_elect(smem_u32(&bars.k_free[buf]));
      ++su;
      s_first = --s_left == 0;
      if (s_first) {
        mma_commit_elect(smem_u32(&bars.q_free[s]));
        sn += gridDim.x;
        ++s_tiles;
        s_left = sn < total ? tile_at(sn).nb : 0;
      }
    };
    if (s_left > 0) issue_s();
    if (s_left > 0) issue_s();
    uint32_t u = 0;
    for (int n = s < streams ? (int)blockIdx.x : total; n < total; n += gridDim.x) {
      const int nb = tile_at(n).nb;
      for (int t = 0; t < nb; ++t, ++u) {
        const uint32_t buf = u % kBufs;
        mbar_wait_bounded(smem_u32(&bars.v_full[buf]), (u / kBufs) & 1, &abort_flag);
        mbar_wait_bounded(smem_u32(&bars.p_full[s][u & 1]), (u >> 1) & 1, &abort_flag);
        __syncwarp();
        tc_fence_after_sync();
        const uint64_t dV = smem_desc_sw128(sV0 + buf * kTileKV, 8192);
        const uint32_t tP = tStream + (u & 1) * 64;
#pragma unroll
        for (int k = 0; k < 4; ++k) mma_bf16_tmem_a_elect(tStream + tO, tP + k * 8, desc_advance(dV, k * 2048), idO, t > 0 || k > 0);
        mma_commit_elect(smem_u32(&bars.pv_done[s][u & 1]));
        mma_commit_elect(smem_u32(&bars.v_free[buf]));
        if (s_left > 0) issue_s();
      }
    }
    // nothing of this CTA may still be running on the tensor cores when tensor memory is freed
    mma_commit_elect(smem_u32(&bars.drain[s]));
    mbar_wait_drain(smem_u32(&bars.drain[s]), 0);
  } else {
    // ------------------------------------------------------------------ TMA
    if (lane == 0) {
      uint32_t u = 0, tiles = 0;
      for (int n = blockIdx.x; n < total; n += gridDim.x, ++tiles) {
        const Tile tile = tile_at(n);
        for (int t = 0; t < tile.nb; ++t, ++u) {
          const uint32_t buf = u % kBufs, round = u / kBufs;
          const int key = (tile.jb + t) * kBlock;
          if (round >= 1) mbar_wait_bounded(smem_u32(&bars.k_free[buf]), (round - 1) & 1, &abort_flag);
          mbar_arrive_expect_tx(smem_u32(&bars.k_full[buf]), kTileKV);
#pragma unroll
          for (int c = 0; c < NC; ++c) tma_load_4d(sK0 + buf * kTileKV + c * 8192, &tmK, smem_u32(&bars.k_full[buf]), c * 64, key, tile.h, tile.b);
          if (t == 0) {
            for (int s = 0; s < streams; ++s) {   // rows past the end of the sequence are zero
              if (tiles >= 1) mbar_wait_bounded(smem_u32(&bars.q_free[s]), (tiles - 1) & 1, &abort_flag);
              mbar_arrive_expect_tx(smem_u32(&bars.q_full[s]), kTileQ);
#pragma unroll
              for (int c = 0; c < NC; ++c)
                tma_load_4d(sQ0 + s * kTileQ + c * 16384, &tmQ, smem_u32(&bars.q_full[s]), c * 64, tile.h * G, tile.i0 + s * QT, tile.b);
            }
          }
          if (round >= 1) mbar_wait_bounded(smem_u32(&bars.v_free[buf]), (round - 1) & 1, &abort_flag);
          mbar_arrive_expect_tx(smem_u32(&bars.v_full[buf]), kTileKV);
#pragma unroll
          for (int c = 0; c < NC; ++c) tma_load_4d(sV0 + buf * kTileKV + c * 8192, &tmV, smem_u32(&bars.v_full[buf]), c * 64, key, tile.h, tile.b);
        }
      }
      // every request must have landed before the block may exit (also when it gave up)
      for (uint32_t back = 1; back <= (uint32_t)kBufs && back <= u; ++back) {
        const uint32_t w = u - back;
        mbar_wait_drain(smem_u32(&bars.k_full[w % kBufs]), (w / kBufs) & 1);
        mbar_wait_drain(smem_u32(&bars.v_full[w % kBufs]), (w / kBufs) & 1);
      }
      for (int s = 0; s < streams && tiles > 0; ++s) mbar_wait_drain(smem_u32(&bars.q_full[s]), (tiles - 1) & 1);
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 512);
  if (tid == 0 && abort_flag) atomicOr(P.status, 1);
}

// ---- backward --------------------------------------------------------------------------

// delta[row] = sum_c out[row][c] * dout[row][c]; D/8 threads per row.  The blocks behind those of the rows clear dk and dv
// (`clear` 16-byte pieces from P.dk on).
template <int D>
__global__ void __launch_bounds__(256) sel_delta_kernel(const SelParams P, float* delta, unsigned row_blocks, int64_t clear) {
  constexpr int TPR = D / 8;
  if (blockIdx.x >= row_blocks) {
    const int64_t step = (int64_t)(gridDim.x - row_blocks) * 256;
    for (int64_t e = (int64_t)(blockIdx.x - row_blocks) * 256 + threadIdx.x; e < clear; e += step)
      reinterpret_cast<float4*>(P.dk)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    return;
  }
  const uint32_t row = blockIdx.x * (256 / TPR) + threadIdx.x / TPR, nrows = (uint32_t)P.B * P.Hq * P.N;   // (see `supported`)
  const int part = threadIdx.x % TPR;
  float acc = 0.f;
  if (row < nrows) {
    const uint32_t head = row / (uint32_t)P.N;
    const int i = (int)(row - head * P.N), b = (int)(head / (uint32_t)P.Hq), hq = (int)head - b * P.Hq;
    const uint4 o = *reinterpret_cast<const uint4*>(P.out + b * P.o_sb + (int64_t)hq * P.o_sh + (int64_t)i * P.o_sn + part * 8);
    const uint4 g = *reinterpret_cast<const uint4*>(P.dout + b * P.do_sb + (int64_t)hq * P.do_sh + (int64_t)i * P.do_sn + part * 8);
    const uint32_t ou[4] = {o.x, o.y, o.z, o.w}, gu[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      acc = fmaf(__uint_as_float(ou[x] << 16), __uint_as_float(gu[x] << 16), acc);
      acc = fmaf(__uint_as_float(ou[x] & 0xffff0000u), __uint_as_float(gu[x] & 0xffff0000u), acc);
    }
  }
#pragma unroll
  for (int o = TPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(kFullMask, acc, o);
  if (row < nrows && part == 0) delta[row] = acc;
}


// ---- backward, warp-specialised ---------------------------------------------------------------
//
// One CTA per SM, 23 warps with fixed roles, so that the gathers, the tensor-core work and the per-row arithmetic of
// different chunks overlap instead of taking turns:
//   warps 0-7, 8-15  two softmax groups; chunk n (counted per CTA) belongs to group n % 2.  Two threads share a row (32
//                    of the block's 64 columns each): they read S and dP from tensor memory, write P and dS (bf16) for
//                    the second set of MMAs and then store the dQ row as a partial result (summed by
//                    sel_dq_merge_kernel): at dim_head 128 at once, at 64, where either group has a dQ of its own in tensor
//                    memory, under the arithmetic of the group's next chunk.  The group of an item's last chunk flushes its dK / dV with fp32 reductions.
//   warp 16, 17      issue the tcgen05.mma: S / dP, which run a chunk ahead, and dV, dQ, dK.  Two of them, because an MMA
//                    is accepted when the one before it starts: the waits and addresses in between leave the tensor
//                    cores idle unless another warp issues meanwhile.
//   warp 18          one thread requests the K / V tiles of each item by TMA.  It is a role of its own because it waits
//                    for the consumer: a gathering thread that did so would hold back the announcements the consumer is
//                    waiting for.
//   warps 19-22      gather the Q and dO rows with 16-byte cp.async into a ring of stages; a stage announces itself
//                    (cp.async.mbarrier.arrive) when the copies have landed, the threads never wait for data.  At dim_head 64
//                    they leave what they know of the rows (dQ destination, visible columns) beside the stage.
// What bounds it: the chain of a group's chunk (wait for S, arithmetic, dV and dQ, dQ read-out) with two groups in flight
// (issue slots 42 % busy, tensor pipe 29 %); the gathers alone (32 KB per chunk at 18 bytes per clock and SM, the rate of scattered 128-byte rows out
// of the L2) would take 1800 cycles per chunk, the MMAs 1100.  Batch 4, 8192 positions, 32 / 4 heads of 64: 1.76 ms with one
// lane polling each barrier, 1.62 with waits of whole warps, 1.54 with dQ under the next chunk and two values per
// instruction, 1.43 with the row data from the loaders (four stages and one K / V buffer 1.48, S released before the
// arithmetic the same, row ids and pointers in registers 1.54).  Batch 1, 3001 positions, 16 / 2 heads of 128: 113 -> 104 us.
// Tensor memory (512 columns): S and dP of either group (64 columns each); dV and dK share D columns, dV in lanes 0-15 and
// dK in lanes 16-31 of every quarter (a 64-row accumulator occupies half of the lanes); dQ: D columns, one buffer per
// group at dim_head 64, one for both at 128.
// Every hand-over is an mbarrier with one waiting role; every wait is bounded.
namespace ws {
constexpr int kSoftmaxWarps = 16, kThreads = 23 * 32;
constexpr int kGroupThreads = 256, kLoaderThreads = 128;
constexpr uint32_t kPBytes = 32768;         // P and dS tiles of a group

template <int D>
struct Shape {
  static constexpr int NC = D / 64;
  static constexpr int kStages = D == 64 ? 3 : 2;
  static constexpr int kKv = D == 64 ? 2 : 1;              // K / V buffers
  static constexpr int kDq = D == 64 ? 2 : 1;              // dQ buffers in tensor memory
  static constexpr uint32_t kTileQ = NC * 16384, kStageBytes = 2 * kTileQ, kTileK = NC * 8192, kKvBytes = 2 * kTileK;
  // Per stage: lse and delta of every row of the chunk; where there is room, also what the loaders know of the rows already:
  // the (row, slot) id its dQ goes to, the visible columns, and for an item's last chunk the keys whose dK / dV are complete
  static constexpr bool kRowMeta = D == 64;
  static constexpr uint32_t kMetaBytes = kRowMeta ? 4 * kRows * 4 + 16 : 2 * kRows * 4;
  static constexpr uint32_t kBytes = kStages * kStageBytes + 2 * kPBytes + kKv * kKvBytes + kStages * kMetaBytes;
  static constexpr uint32_t tGroup = 128, tDP = 64, tAcc = 256, tDQ = tAcc + D;   // tensor-memory columns
};
constexpr uint32_t kLaneDK = 16u << 16;     // dK: lanes 16-31 of every quarter
// dQ partials: bf16 at dim_head 64; fp32 at 128, where dq has always been summed from fp32 terms
template <int D>
constexpr int kDqElem = D == 64 ? 2 : 4;
constexpr uint32_t kDqRow = 64, kDqStage = 32 * kDqRow;   // read-out: bytes of a row that a warp stages at a time, in the P tile

struct Bars {
  uint64_t q_full[3], q_free[3];
  uint64_t s_full[2], p_full[2], dq_done[2], tiles_free[2], dq_free;
  uint64_t kv_full[2], kv_free[2], acc_full[2], acc_free;
  uint64_t drain[2];
};

// The chunks of a CTA in order: chunk c of item `it` (the t-th of the CTA) is its n-th chunk.  The next item is requested
// when the present one is entered.
struct Cursor {
  const int4* items;
  int nitems, it, c, t, n;
  int4 item, ahead;
  __device__ __forceinline__ Cursor(const int4* items_, int nitems_, int first) : items(items_), nitems(nitems_), it(first), c(0), t(0), n(0) {
    item = items[it];                      // a CTA without any item has returned
    ahead = items[min(it + (int)gridDim.x, nitems - 1)];
  }
  __device__ __forceinline__ bool live() const { return it < nitems; }
  __device__ __forceinline__ bool last() const { return c == item.z - 1; }
  __device__ __forceinline__ bool next() {   // true: entered another item
    ++n;
    if (++c < item.z) return false;
    c = 0;
    ++t;
    it += gridDim.x;
    item = ahead;
    ahead = items[min(it + (int)gridDim.x, nitems - 1)];
    return true;
  }
};
}  // namespace ws

template <int D, bool SLOTS>   // SLOTS: the gradients of the slot scales are wanted
__global__ void __launch_bounds__(ws::kThreads, 1)
sel_bwd_ws_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const SelParams P) {
  using namespace ws;
  using S = Shape<D>;
  constexpr int NC = S::NC, kStages = S::kStages;
  extern __shared__ __align__(1024) uint8_t ws_smem[];
  __shared__ int abort_flag;
  __shared__ uint32_t tmem_slot;
  __shared__ __align__(8) Bars bars;
  if (item_count(P) == 0) return;
  const int nitems = P.list_item[P.bh1 * P.nfb], first_item = P.list_item[P.bh0 * P.nfb] + (int)blockIdx.x;   // of the slice
  if (first_item >= nitems) return;

  const uint32_t base = smem_u32(ws_smem);
  // stage s: Q tiles then dO tiles; group g: P tile then dS tile; K / V buffer: K tiles then V tiles
  const uint32_t sQ0 = base, sP0 = sQ0 + kStages * S::kStageBytes, sKV0 = sP0 + 2 * kPBytes, sMeta0 = sKV0 + S::kKv * S::kKvBytes;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    abort_flag = 0;
    if (base & 1023u) abort_flag = 1;   // the tiles would be mis-swizzled: report instead of computing
    for (int i = 0; i < 3; ++i) {
      mbar_init(smem_u32(&bars.q_full[i]), (S::kRowMeta ? 2 : 1) * kLoaderThreads);
      mbar_init(smem_u32(&bars.q_free[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&bars.s_full[i]), 1);
      mbar_init(smem_u32(&bars.p_full[i]), kGroupThreads);
      mbar_init(smem_u32(&bars.dq_done[i]), 1);
      mbar_init(smem_u32(&bars.tiles_free[i]), 1);
      mbar_init(smem_u32(&bars.kv_full[i]), 1);
      mbar_init(smem_u32(&bars.kv_free[i]), 1);
      mbar_init(smem_u32(&bars.acc_full[i]), 1);
    }
    mbar_init(smem_u32(&bars.dq_free), kGroupThreads);
    mbar_init(smem_u32(&bars.acc_free), kGroupThreads);
    mbar_init(smem_u32(&bars.drain[0]), 1);
    mbar_init(smem_u32(&bars.drain[1]), 1);
    fence_mbar_init();
    prefetch_tensormap(&tmK);
    prefetch_tensormap(&tmV);
  }
  __syncthreads();
  if (warp == 0) {
    tmem_alloc(smem_u32(&tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tm = tmem_slot;
  const int G = P.G, QT = kRows / G, g_shift = 31 - __clz(G);

  if (warp < kSoftmaxWarps) {
    // ------------------------------------------------------------------ softmax groups
    const int wg = warp >> 3, half = (warp >> 2) & 1, row = (warp & 3) * 32 + lane;
    const uint32_t tm_quarter = tm + ((uint32_t)((warp & 3) * 32) << 16);   // warps w and w + 4 share a lane quarter
    const uint32_t tS = tm_quarter + wg * S::tGroup;
    const int q_local = row >> g_shift, g = row - (q_local << g_shift);
    const uint32_t sP = sP0 + wg * kPBytes, sDS = sP + 16384;
    const uint32_t sDq = sP + (warp & 3) * 4096 + half * kDqStage;   // in the warp's own rows of the P tile
    // dQ of the chunk just handed over: the thread's half of the columns of its row, to the (row, slot) partial `dst_row`
    // (plain stores run at memory speed, fp32 reductions into dq are limited by the L2 atomic units).  A thread that
    // stored its own piece would make every store instruction touch 32 lines; the warp stages 32 columns at a time in
    // the group's P tile, which the completed dV product no longer reads, and stores eight rows per instruction.
    auto dq_out = [&](const int dst_row) {
      tc_fence_after_sync();
      __syncwarp();
      uint8_t* const pbase = reinterpret_cast<uint8_t*>(P.partial);
      constexpr int kCols = (int)kDqRow / kDqElem<D>, kPieces = D / 2 / kCols;   // columns per piece, pieces per half row
#pragma unroll 1
      for (int piece = 0; piece < kPieces; ++piece) {
        const int col = (half * kPieces + piece) * kCols;
        {
          float tq[kCols];
          if constexpr (kCols == 32) tmem_ld32(tm_quarter + S::tDQ + (S::kDq == 2 ? wg * D : 0) + col, tq);
          else tmem_ld16(tm_quarter + S::tDQ + (S::kDq == 2 ? wg * D : 0) + col, tq);
          tmem_ld_wait();
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            uint4 v;
            if constexpr (kCols == 32) {
              v.x = pack_bf16(tq[x * 8 + 0], tq[x * 8 + 1]); v.y = pack_bf16(tq[x * 8 + 2], tq[x * 8 + 3]);
              v.z = pack_bf16(tq[x * 8 + 4], tq[x * 8 + 5]); v.w = pack_bf16(tq[x * 8 + 6], tq[x * 8 + 7]);
            } else {
              v = make_uint4(__float_as_uint(tq[x * 4]), __float_as_uint(tq[x * 4 + 1]), __float_as_uint(tq[x * 4 + 2]), __float_as_uint(tq[x * 4 + 3]));
            }
            sts_v4(sDq + lane * kDqRow + ((x ^ ((lane >> 1) & 3)) << 4), v);   // conflict-free to write and to read
          }
        }
        if (S::kDq == 1 && piece == kPieces - 1) {
          tc_fence_before_sync();
          mbar_arrive(smem_u32(&bars.dq_free));   // the other group's dQ may overwrite the columns
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int rr = k * 8 + (lane >> 2);
          const int dst = __shfl_sync(kFullMask, dst_row, rr);
          const uint4 v = lds_v4(sDq + rr * kDqRow + (((lane & 3) ^ ((rr >> 1) & 3)) << 4));
          if (dst >= 0) *reinterpret_cast<uint4*>(pbase + ((int64_t)dst * D + col) * kDqElem<D> + (lane & 3) * 16) = v;
        }
        __syncwarp();
      }
      // the two warps that share these rows have read what they staged before either writes P again
      asm volatile("bar.sync %0, 64;" ::"r"(1 + wg * 4 + (warp & 3)) : "memory");
    };
    // The chunks of the group: every second one of the CTA
    int chunks = 0;
    for (int t = first_item + lane * (int)gridDim.x; t < nitems; t += 32 * (int)gridDim.x) chunks += P.items[t].z;
    chunks = (int)__reduce_add_sync(kFullMask, (unsigned)chunks);
    uint32_t use = 0, flushes = 0;
    int stage = wg % kStages;
    // Without room for the rows' data beside the stage the groups look them up themselves: chunk c of `item`; the next item is
    // requested when this one is entered
    int it = first_item, c = wg, j = 0, key_row0 = 0, dst0 = 0;
    int4 item = make_int4(0, 0, 0, 0), ahead = item;
    auto settle = [&](bool entered) {       // onto the item that holds chunk c
      while (it < nitems && c >= item.z) {
        c -= item.z;
        it += gridDim.x;
        item = ahead;
        ahead = P.items[min(it + (int)gridDim.x, nitems - 1)];
        entered = true;
      }
      if (!entered || it >= nitems) return;
      const int bh = item.x / P.nfb;
      j = item.x - bh * P.nfb;
      key_row0 = bh * P.Nk;                 // 32 bits hold every row id (see `supported`)
      dst0 = ((bh - P.bh0) * G + g) * P.N * P.ns;
    };
    auto entry_of = [&]() { return it < nitems ? __ldg(P.entries + item.w + c * QT + q_local) : kInvalidEntry; };
    uint32_t e_next = kInvalidEntry;
    if constexpr (!S::kRowMeta) {
      item = P.items[it];
      ahead = P.items[min(it + (int)gridDim.x, nitems - 1)];
      settle(true);
      e_next = entry_of();
    }
    int dst_prev = -1;
    for (int n = wg; n < chunks; n += 2) {
      const uint32_t sMeta = sMeta0 + stage * S::kMetaBytes + row * 4;
      mbar_wait_warp(smem_u32(&bars.s_full[wg]), use & 1, &abort_flag);
      tc_fence_after_sync();
      const float lse2 = __uint_as_float(lds_u32(sMeta)) * kLog2e;
      const float delta = __uint_as_float(lds_u32(sMeta + kRows * 4));
      int dst, lo, lim, key_row, keys;      // first visible column, last one (-1: padding); key_row < 0: not an item's last chunk
      if constexpr (S::kRowMeta) {
        dst = (int)lds_u32(sMeta + 2 * kRows * 4);
        const int cols = (int)lds_u32(sMeta + 3 * kRows * 4);
        lo = cols & 0xff;
        lim = cols >> 8;
        const uint2 last = lds_v2(sMeta0 + stage * S::kMetaBytes + 4 * kRows * 4);
        key_row = (int)last.x;
        keys = (int)last.y;
      } else {
        const RowInfo r = decode_row(e_next, j, P.rule);
        dst = r.valid ? dst0 + r.i * P.ns + r.slot : -1;
        lo = r.lo;
        lim = r.lim;
        key_row = c == item.z - 1 ? key_row0 + j * kBlock : -1;
        keys = P.Nk - j * kBlock;
      }
      float slot_part = 0.f;
      // rows that see the whole block need no per-column test; only own-block (causal) and padding rows do
      const bool all_full = __all_sync(kFullMask, lim == kBlock - 1 && lo == 0);
      const uint64_t scale2 = pack2(P.scale_log2, P.scale_log2), lse2n = pack2(-lse2, -lse2), delta2n = pack2(-delta, -delta);
#pragma unroll 1
      for (int q = 0; q < 2; ++q) {         // 16 columns at a time: the body stays small enough for the instruction cache
        const int col = half * 32 + q * 16;
        uint32_t pw[8], dsw[8];             // P and dS as bf16
        {
          float sv[16], dv[16];
          tmem_ld16(tS + col, sv);
          tmem_ld16(tS + S::tDP + col, dv);
          tmem_ld_wait();
          const int rem = lim - col, rlo = lo - col;       // columns rlo..rem of this group are visible
#pragma unroll
          for (int x = 0; x < 8; ++x) {
            float p0, p1, d0, d1;
            unpack2(fma2(pack2(sv[2 * x], sv[2 * x + 1]), scale2, lse2n), p0, p1);
            p0 = ex2(p0);
            p1 = ex2(p1);
            if (!all_full) {
              p0 = 2 * x >= rlo && 2 * x <= rem ? p0 : 0.f;
              p1 = 2 * x + 1 >= rlo && 2 * x + 1 <= rem ? p1 : 0.f;
            }
            unpack2(mul2(pack2(p0, p1), add2(pack2(dv[2 * x], dv[2 * x + 1]), delta2n)), d0, d1);
            if constexpr (SLOTS) slot_part = fmaf(d1, sv[2 * x + 1], fmaf(d0, sv[2 * x], slot_part));
            pw[x] = pack_bf16(p0, p1);
            dsw[x] = pack_bf16(d0, d1);
          }
        }
        // dK of the group's previous chunk, the last product to read the tiles, is complete
        if (q == 0 && use > 0) mbar_wait_warp(smem_u32(&bars.tiles_free[wg]), (use - 1) & 1, &abort_flag);
#pragma unroll
        for (int x = 0; x < 2; ++x)
          sts_v4(sDS + sw128_offset(row, col / 8 + x), make_uint4(dsw[4 * x], dsw[4 * x + 1], dsw[4 * x + 2], dsw[4 * x + 3]));
        // with a dQ buffer for either group that chunk's rows leave here: its products have run under the arithmetic above
        if constexpr (S::kDq == 2) {
          if (q == 0 && use > 0) dq_out(dst_prev);
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
          sts_v4(sP + sw128_offset(row, col / 8 + x), make_uint4(pw[4 * x], pw[4 * x + 1], pw[4 * x + 2], pw[4 * x + 3]));
      }
      fence_proxy_async_smem();
      tc_fence_before_sync();
      mbar_arrive(smem_u32(&bars.p_full[wg]));
      dst_prev = dst;
      if constexpr (SLOTS) {   // two threads of a row, in different warps: two additions to a cleared slot
        for (int o = G / 2; o > 0; o >>= 1) slot_part += __shfl_xor_sync(kFullMask, slot_part, o);
        if (dst >= 0 && g == 0) {           // dst = (row of the slice) ns + slot
          const int part_row = dst / P.ns, slot = dst - part_row * P.ns, pair = part_row / P.N;   // (batch, query head) of the slice
          const int64_t query = (int64_t)(P.bh0 + pair / G) * P.N + (part_row - pair * P.N);
          if (slot < P.nsel) atomicAdd(P.slot_grads + query * P.nsel + slot, slot_part * P.scale);
        }
      }
      stage += 2;
      if (stage >= kStages) stage -= kStages;
      if constexpr (!S::kRowMeta) {         // on to the group's next chunk: its entry travels under what is left of this one
        c += 2;
        settle(false);
        e_next = entry_of();
      }
      if constexpr (S::kDq == 1) {          // one dQ buffer for both groups: the other one is waiting for it
        mbar_wait_warp(smem_u32(&bars.dq_done[wg]), use & 1, &abort_flag);
        dq_out(dst_prev);
      }
      ++use;
      if (key_row >= 0) {
        // flush dK/dV of this item: keys 16w..16w+15 live in the lanes of quarter w, either half of the group takes half of
        // the columns.  "Accumulator complete" has one barrier per flushing group, counted by
        // that group: with one barrier for both, a group that reached its wait before the other group's item was complete
        // saw the phase before that one (same parity) as its own and flushed early.
        mbar_wait_warp(smem_u32(&bars.acc_full[wg]), flushes & 1, &abort_flag);
        ++flushes;
        tc_fence_after_sync();
        __syncwarp();
        const float f = lane < 16 ? 1.f : P.scale;
        const int key = (warp & 3) * 16 + (lane & 15);
        float* const dstp = (lane < 16 ? P.dv : P.dk) + ((int64_t)key_row + key) * D + half * (D / 2);
#pragma unroll 1
        for (int cc = 0; cc < D / 2; cc += 32) {
          float tk[32];
          tmem_ld32(tm_quarter + S::tAcc + half * (D / 2) + cc, tk);
          tmem_ld_wait();
          if (key < keys) {
#pragma unroll
            for (int x = 0; x < 8; ++x) red_add_v4(dstp + cc + x * 4, tk[x * 4] * f, tk[x * 4 + 1] * f, tk[x * 4 + 2] * f, tk[x * 4 + 3] * f);
          }
        }
        tc_fence_before_sync();
        mbar_arrive(smem_u32(&bars.acc_free));
      }
    }
    if constexpr (S::kDq == 2) {
      if (use > 0) {
        mbar_wait_warp(smem_u32(&bars.tiles_free[wg]), (use - 1) & 1, &abort_flag);
        dq_out(dst_prev);
      }
    }
  } else if (warp == kSoftmaxWarps) {
    // ------------------------------------------------------------------ issuer of S and dP.  The whole warp runs the
    // loop (so that its state lives in uniform registers), one elected lane issues.  The lbo field of a descriptor serves
    // the tiles read MN-major (the distance to the next 64 columns); the others ignore it.  One descriptor per tile: every
    // MMA then costs one 64-bit add to issue.
    constexpr uint32_t idS = instr_desc_bf16(128, 64, false, false);
    int stage = 0, round = 0;
    for (Cursor cur(P.items, nitems, first_item); cur.live(); cur.next()) {
      const int grp = cur.n & 1, kb = S::kKv == 2 ? cur.t & 1 : 0;
      const uint32_t sQ = sQ0 + stage * S::kStageBytes, sK = sKV0 + kb * S::kKvBytes, tS = tm + grp * S::tGroup;
      const uint64_t dQt = smem_desc_sw128(sQ, 16384), dDOt = smem_desc_sw128(sQ + S::kTileQ, 16384);
      const uint64_t dKt = smem_desc_sw128(sK, 8192), dVt = smem_desc_sw128(sK + S::kTileK, 8192);
      // the group has read the S and dP before these
      if (cur.n >= 2) mbar_wait_bounded(smem_u32(&bars.p_full[grp]), (uint32_t)((cur.n >> 1) - 1) & 1, &abort_flag);
      mbar_wait_bounded(smem_u32(&bars.q_full[stage]), round & 1, &abort_flag);
      if (cur.c == 0) mbar_wait_bounded(smem_u32(&bars.kv_full[kb]), (uint32_t)(S::kKv == 2 ? cur.t >> 1 : cur.t) & 1, &abort_flag);
      __syncwarp();
      tc_fence_after_sync();
#pragma unroll
      for (int k = 0; k < D / 16; ++k) {
        const uint32_t a = (k / 4) * 16384 + (k % 4) * 32, bb = (k / 4) * 8192 + (k % 4) * 32;
        mma_bf16_elect(tS, desc_advance(dQt, a), desc_advance(dKt, bb), idS, k > 0);
        mma_bf16_elect(tS + S::tDP, desc_advance(dDOt, a), desc_advance(dVt, bb), idS, k > 0);
      }
      mma_commit_elect(smem_u32(&bars.s_full[grp]));
      if (++stage == kStages) { stage = 0; ++round; }
    }
    mma_commit_elect(smem_u32(&bars.drain[0]));
    mbar_wait_drain(smem_u32(&bars.drain[0]), 0);
  } else if (warp == kSoftmaxWarps + 1) {
    // ------------------------------------------------------------------ issuer of dV, dQ and dK
    constexpr uint32_t idDQ = instr_desc_bf16(128, D, false, true);
    constexpr uint32_t idKV = instr_desc_bf16(64, D, true, true);
    int stage = 0;
    for (Cursor cur(P.items, nitems, first_item); cur.live(); cur.next()) {
      const int grp = cur.n & 1, kb = S::kKv == 2 ? cur.t & 1 : 0;
      const uint32_t sQ = sQ0 + stage * S::kStageBytes, sP = sP0 + grp * kPBytes;
      const uint64_t dQt = smem_desc_sw128(sQ, 16384), dDOt = smem_desc_sw128(sQ + S::kTileQ, 16384);
      const uint64_t dPt = smem_desc_sw128(sP, 16384), dDSt = smem_desc_sw128(sP + 16384, 16384);
      const uint64_t dKt = smem_desc_sw128(sKV0 + kb * S::kKvBytes, 8192);
      mbar_wait_bounded(smem_u32(&bars.p_full[grp]), (uint32_t)(cur.n >> 1) & 1, &abort_flag);
      // the accumulators are single: the first chunk of an item waits until the previous item has been flushed
      if (cur.c == 0 && cur.t >= 1) mbar_wait_bounded(smem_u32(&bars.acc_free), (uint32_t)(cur.t - 1) & 1, &abort_flag);
      __syncwarp();
      tc_fence_after_sync();
      // dV += P^T dO over the 128 rows of the chunk, then dQ = dS K: the group waits for both (it stages its dQ rows in
      // the P tile).  dQ's columns: the group (or, with one buffer, the other one) has read the dQ before it out.
#pragma unroll
      for (int k = 0; k < 8; ++k)
        mma_bf16_elect(tm + S::tAcc, desc_advance(dPt, k * 2048), desc_advance(dDOt, k * 2048), idKV, cur.c > 0 || k > 0);
      if (S::kDq == 1 && cur.n >= 1) {
        mbar_wait_bounded(smem_u32(&bars.dq_free), (uint32_t)(cur.n - 1) & 1, &abort_flag);
        __syncwarp();
        tc_fence_after_sync();
      }
      const uint32_t tDQ = tm + S::tDQ + (S::kDq == 2 ? grp * D : 0);
#pragma unroll
      for (int k = 0; k < 4; ++k) mma_bf16_elect(tDQ, desc_advance(dDSt, k * 32), desc_advance(dKt, k * 2048), idDQ, k > 0);
      if (S::kDq == 1) mma_commit_elect(smem_u32(&bars.dq_done[grp]));
      // dK += dS^T Q
#pragma unroll
      for (int k = 0; k < 8; ++k)
        mma_bf16_elect(tm + S::tAcc + kLaneDK, desc_advance(dDSt, k * 2048), desc_advance(dQt, k * 2048), idKV, cur.c > 0 || k > 0);
      mma_commit_elect(smem_u32(&bars.tiles_free[grp]));
      mma_commit_elect(smem_u32(&bars.q_free[stage]));
      if (cur.last()) {
        mma_commit_elect(smem_u32(&bars.kv_free[kb]));
        mma_commit_elect(smem_u32(&bars.acc_full[grp]));   // the group of the item's last chunk flushes
      }
      if (++stage == kStages) stage = 0;
    }
    // nothing of this block may still be running on the tensor cores when tensor memory is freed
    mma_commit_elect(smem_u32(&bars.drain[1]));
    mbar_wait_drain(smem_u32(&bars.drain[1]), 0);
  } else if (warp == kSoftmaxWarps + 2) {
    // ------------------------------------------------------------------ K/V tiles
    if (lane == 0) {
      int t = 0;
      for (int it = first_item; it < nitems; it += gridDim.x, ++t) {
        const int4 item = P.items[it];
        const int list = item.x, j = list % P.nfb, bh = list / P.nfb, h = bh % P.Hkv, b = bh / P.Hkv;
        const int kb = S::kKv == 2 ? t & 1 : 0, round = S::kKv == 2 ? t >> 1 : t;
        if (round >= 1) mbar_wait_bounded(smem_u32(&bars.kv_free[kb]), (uint32_t)(round - 1) & 1, &abort_flag);
        const uint32_t sK = sKV0 + kb * S::kKvBytes, sV = sK + S::kTileK;
        const uint32_t bar = smem_u32(&bars.kv_full[kb]);
        mbar_arrive_expect_tx(bar, S::kKvBytes);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          tma_load_4d(sK + c * 8192, &tmK, bar, c * 64, j * kBlock, h, b);
          tma_load_4d(sV + c * 8192, &tmV, bar, c * 64, j * kBlock, h, b);
        }
      }
      // the last requests must have landed before the block may exit
      for (int back = 1; back <= S::kKv && t - back >= 0; ++back) {
        const int tt = t - back;
        mbar_wait_drain(smem_u32(&bars.kv_full[S::kKv == 2 ? tt & 1 : 0]), (uint32_t)(S::kKv == 2 ? tt >> 1 : tt) & 1);
      }
    }
  } else {
    // ------------------------------------------------------------------ loaders
    constexpr int CH = D / 8, RPP = kLoaderThreads / CH, kPasses = kRows / RPP;   // pieces per row, rows per pass
    const int lt = tid - (kSoftmaxWarps + 3) * 32;   // 0..127
    const int sub = lt % CH, r0 = lt / CH;
    // A thread's rows are RPP apart: with up to RPP heads per KV head all of the same head (at dim_head 128 and 16 heads the odd
    // passes are eight heads on).  Row strides are 32-bit (see problem_bwd): one multiplication per row and tensor.
    const int g0 = r0 & (G - 1), g1 = (r0 + RPP) & (G - 1);
    const uint32_t q_sn = (uint32_t)P.q_sn, do_sn = (uint32_t)P.do_sn, off0 = sw128_offset(r0, sub % 8);
    const __nv_bfloat16 *q_head[2] = {nullptr, nullptr}, *do_head[2] = {nullptr, nullptr};
    const float *lse_head = nullptr, *delta_head = nullptr;
    int list_of = -1, j = 0, key_row0 = 0, dst0 = 0;
    for (Cursor cur(P.items, nitems, first_item); cur.live(); cur.next()) {
      if (cur.item.x != list_of) {
        list_of = cur.item.x;
        const int bh = list_of / P.nfb, b = bh / P.Hkv, h = bh - b * P.Hkv;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int64_t hq = (int64_t)h * G + (k == 0 ? g0 : g1);
          q_head[k] = P.q + b * P.q_sb + hq * P.q_sh + sub * 8;
          do_head[k] = P.dout + b * P.do_sb + hq * P.do_sh + sub * 8;
        }
        j = list_of - bh * P.nfb;
        key_row0 = bh * P.Nk + j * kBlock;   // 32 bits hold every row id (see `supported`)
        dst0 = ((bh - P.bh0) * G + (lt & (G - 1))) * P.N * P.ns;
        const int64_t row0 = ((int64_t)b * P.Hq + (int64_t)h * G + (lt & (G - 1))) * P.N;
        lse_head = P.lse + row0;
        delta_head = P.delta + row0;
      }
      const int stage = cur.n % kStages;
      const uint32_t* chunk_entries = P.entries + cur.item.w + cur.c * QT;
      // read the entries first: the copies below are compiler barriers, a load placed between them would be
      // waited for eight times
      uint32_t ev[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) ev[k] = __ldg(chunk_entries + ((r0 + k * RPP) >> g_shift));
      const uint32_t es = __ldg(chunk_entries + (lt >> g_shift));
      if (cur.n >= kStages) mbar_wait_warp(smem_u32(&bars.q_free[stage]), (uint32_t)(cur.n / kStages - 1) & 1, &abort_flag);
      const uint32_t sQ = sQ0 + stage * S::kStageBytes + (sub / 8) * 16384 + off0, sDO = sQ + S::kTileQ;
#pragma unroll
      for (int k0 = 0; k0 < kPasses; k0 += 8) {
        if (k0 > 0)
#pragma unroll
          for (int k = 0; k < 8; ++k) ev[k] = __ldg(chunk_entries + ((r0 + (k0 + k) * RPP) >> g_shift));
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const bool valid = ev[k] != kInvalidEntry;
          const uint32_t i = valid ? ev[k] & 0xffffffu : 0u, bytes = valid ? 16u : 0u;
          const uint32_t off = (k0 + k) * RPP * 128;       // RPP is a multiple of 8: the swizzle of all its rows is that of r0
          cp_async16(sQ + off, q_head[k & 1] + (uint64_t)i * q_sn, bytes);
          cp_async16(sDO + off, do_head[k & 1] + (uint64_t)i * do_sn, bytes);
        }
      }
      {
        // the statistics of row lt
        const bool valid = es != kInvalidEntry;
        const uint32_t i = valid ? es & 0xffffffu : 0u, bytes = valid ? 4u : 0u;
        const uint32_t sMeta = sMeta0 + stage * S::kMetaBytes + lt * 4;
        cp_async4(sMeta, lse_head + i, bytes);
        cp_async4(sMeta + kRows * 4, delta_head + i, bytes);
        if constexpr (S::kRowMeta) {
          const RowInfo r = decode_row(es, j, P.rule);
          sts_u32(sMeta + 2 * kRows * 4, (uint32_t)(valid ? dst0 + r.i * P.ns + r.slot : -1));
          sts_u32(sMeta + 3 * kRows * 4, (uint32_t)(r.lim * 256 + r.lo));
          if (lt == 0) {
            const uint32_t last = sMeta + 4 * kRows * 4;
            sts_u32(last, (uint32_t)(cur.last() ? key_row0 : -1));
            sts_u32(last + 4, (uint32_t)(P.Nk - j * kBlock));
          }
          mbar_arrive(smem_u32(&bars.q_full[stage]));   // these are stores: announced apart from the copies
        }
      }
      // the stage announces itself when this thread's copies have landed; the thread moves on at once
      cp_async_arrive_noinc(smem_u32(&bars.q_full[stage]));
    }
    cp_async_commit();
    cp_async_wait<0>();
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 512);
  if (tid == 0 && abort_flag) atomicOr(P.status, 1);
}


// sums the dQ partials of every (batch, query head, query) into the fp32 dq row: D/8 threads per row.  The blocks behind
// those of the rows round dk and dv, which the kernel before has completed, to bf16 (`round` pieces of 8 from P.dk on).
template <int D, int MODE>
__global__ void __launch_bounds__(256, 6) sel_dq_merge_kernel(const SelParams P, unsigned row_blocks, int64_t round) {
  constexpr int TPR = D / 8;
  if (blockIdx.x >= row_blocks) {
    const int64_t step = (int64_t)(gridDim.x - row_blocks) * 256;
    for (int64_t e = (int64_t)(blockIdx.x - row_blocks) * 256 + threadIdx.x; e < round; e += step) {
      const float4 a = reinterpret_cast<const float4*>(P.dk)[2 * e], c = reinterpret_cast<const float4*>(P.dk)[2 * e + 1];
      reinterpret_cast<uint4*>(P.dkv_lp)[e] = make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(c.x, c.y), pack_bf16(c.z, c.w));
    }
    return;
  }
  const uint32_t slice_row = blockIdx.x * (256 / TPR) + threadIdx.x / TPR;   // 32 bits hold every row id (see `supported`)
  const int part = threadIdx.x % TPR;
  if (slice_row >= (uint32_t)(P.bh1 - P.bh0) * P.G * P.N) return;
  const uint32_t row = (uint32_t)P.bh0 * P.G * P.N + slice_row, head = row / (uint32_t)P.N;
  const int i = (int)(row - head * P.N), b = (int)(head / (uint32_t)P.Hq), hq = (int)head - b * P.Hq;
  const int h = hq >> (31 - __clz(P.G));
  const int64_t part_row = slice_row;
  const int ns = P.ns;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  // Rows in flight: nine of 64 (17 slots in two rounds), but eight in the sliding branch (10 slots: with nine 4 % slower, with ten
  // 12 %), four of 128 in fp32 (with six 9 % slower).  Bound by the partials' bytes: 4 x 8192 positions, 32 heads 437 -> 360 us
  // (0.95 of the copy bandwidth), 3001 positions, 16 heads of 128 45 -> 32 us.  The bound of six blocks an SM is what keeps the loads of a
  // batch together: without one the compiler stops at 32 registers and fetches them in turns (445 us; with four blocks 356 us, but
  // the sliding branch 125 us instead of 118 us and the compressed one 163 us instead of 148 us).
  constexpr int BYTES = ws::kDqElem<D>, BATCH = BYTES == 4 ? 4 : MODE == kModeSwa ? 8 : 9, QUADS = BYTES / 2;
  const uint8_t* prow = reinterpret_cast<const uint8_t*>(P.partial) + (part_row * ns * D + part * 8) * BYTES;
  // some slots at a time: first which of them the query has, then their loads together, then the sums
  const uint32_t* bits = P.bits + ((int64_t)(b * P.Hkv + h) * P.N + i) * P.words;
  for (int s0 = 0; s0 < ns; s0 += BATCH) {
    const int word = s0 >> 5;              // (bits behind the last slot are zero)
    const uint32_t has = MODE == kModeSel ? __funnelshift_r(bits[word], word + 1 < P.words ? bits[word + 1] : 0u, s0 & 31) : 0u;
    bool ok[BATCH];
    uint4 v[BATCH][QUADS];
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      int blk_;
      ok[u] = MODE == kModeSel ? (has >> u & 1u) != 0
                               : s0 + u < ns && slot_block<MODE>(P.rule, b * P.Hkv + h, i, s0 + u, &blk_);
    }
#pragma unroll
    for (int u = 0; u < BATCH; ++u)
#pragma unroll
      for (int w = 0; w < QUADS; ++w)
        v[u][w] = ldg_stream_if(ok[u], prow + (int64_t)(s0 + u) * (D * BYTES) + w * 16);
#pragma unroll
    for (int u = 0; u < BATCH; ++u)
#pragma unroll
      for (int w = 0; w < QUADS; ++w) {
        const uint32_t q[4] = {v[u][w].x, v[u][w].y, v[u][w].z, v[u][w].w};
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          if constexpr (BYTES == 2) {
            acc[2 * x] += __uint_as_float(q[x] << 16);
            acc[2 * x + 1] += __uint_as_float(q[x] & 0xffff0000u);
          } else {
            acc[4 * w + x] += __uint_as_float(q[x]);
          }
        }
      }
  }
  // the partials hold dS K without the logit scale
  if (P.dq_lp != nullptr) {   // the caller asked for dq in the dtype and row layout of q
    uint4 o;
    o.x = pack_bf16(acc[0] * P.scale, acc[1] * P.scale); o.y = pack_bf16(acc[2] * P.scale, acc[3] * P.scale);
    o.z = pack_bf16(acc[4] * P.scale, acc[5] * P.scale); o.w = pack_bf16(acc[6] * P.scale, acc[7] * P.scale);
    *reinterpret_cast<uint4*>(P.dq_lp + b * P.dq_sb + hq * P.dq_sh + i * P.dq_sn + part * 8) = o;
    return;
  }
  float4* dst = reinterpret_cast<float4*>(P.dq + (int64_t)row * D + part * 8);
  dst[0] = make_float4(acc[0] * P.scale, acc[1] * P.scale, acc[2] * P.scale, acc[3] * P.scale);
  dst[1] = make_float4(acc[4] * P.scale, acc[5] * P.scale, acc[6] * P.scale, acc[7] * P.scale);
}

__global__ void fill_kernel(float* dst, float value, int64_t count) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) dst[i] = value;
}

// Importance columns a causal query cannot see (column c of row i is visible iff c < i / stride): `value` from the
// first invisible column on; the attention kernel writes the visible ones.  A warp takes query i and query N-1-i of
// a (batch, head) together, so that every warp writes about one row's worth.
__device__ __forceinline__ void fill_row_from(float* r, int first, int ncb, float value, int lane) {
  const int head = min(ncb, (first + 3) & ~3);          // scalar stores up to the next 16-byte boundary
  if (first + lane < head) r[first + lane] = value;
  const float4 v4 = make_float4(value, value, value, value);
  for (int c = head + 4 * lane; c < ncb; c += 128) *reinterpret_cast<float4*>(r + c) = v4;
}

__global__ void __launch_bounds__(256) fill_invisible_kernel(float* dst, float value, int64_t slices, int N, int ncb, int stride) {
  const int lane = threadIdx.x & 31;
  const int half = (N + 1) / 2;
  const int64_t warps = (int64_t)gridDim.x * 8, pairs = slices * half;
  for (int64_t p = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); p < pairs; p += warps) {
    const int64_t slice = p / half;
    const int i = (int)(p % half), i2 = N - 1 - i;
    fill_row_from(dst + (slice * N + i) * ncb, min(ncb, i / stride), ncb, value, lane);
    if (i2 != i) fill_row_from(dst + (slice * N + i2) * ncb, min(ncb, i2 / stride), ncb, value, lane);
  }
}

// ---- host ----------------------------------------------------------------------------------

static int64_t align_up(int64_t x, int64_t a) { return (x + a - 1) / a * a; }

// One problem of any of the three branches, as the host code sees it.
struct SelProblem {
  nsa_tensor q, k, v, out, dout;
  const int64_t* idx;
  const uint8_t* mask;
  float* lse;
  float *dq, *dk, *dv, *slot_grads;
  nsa_tensor dq_out;       // backward, optional: dq in the dtype and strides the caller chose
  void* dkv_out;           // backward, optional: dk and dv (one behind the other) in bf16; dk and dv are then cleared here
  float* importance;
  __nv_bfloat16* pooled;   // compressed forward, instead of importance: per-selection-block means, see SelParams
  int cpf;
  void* workspace;
  int64_t workspace_bytes;
  const CombineParams* fuse_combine;   // selected forward, optional: the merge also combines and stores (see
  const GatherTargets* fuse_targets;   // sel_merge_combine_kernel); `out` may then be missing
  const void* index;       // an index kept from an earlier call, or NULL to build it
  int64_t index_bytes;
  void* index_out;         // optional: where to build it instead of the head of the work buffer
  int64_t index_out_bytes;
  int* status;             // optional: the word the kernels report through
  const float* delta;      // backward, optional: sum_d out * dout per row from the caller
  int B, Hq, Hkv, N, Nk, D;
  int nsel, diag, mode, window, stride, num_mem, ncb, round_bf16;
  float scale;
};

static int slots_per_query(const SelProblem& a) {
  if (a.mode == kModeSel) return a.nsel + 1;
  if (a.mode == kModeSwa) return a.window / kBlock + 2;   // own block + every older block the window can touch
  return (a.Nk + kBlock - 1) / kBlock;
}

// Shapes served by this family; everything else goes to the generic kernels.
static bool supported(const SelProblem& a) {
  if (a.D != 64 && a.D != 128) return false;
  const int G = a.Hq / a.Hkv;
  if (G != 1 && G != 2 && G != 4 && G != 8 && G != 16) return false;
  if (a.N < 1 || a.N >= (1 << 24) || a.Nk < 1 || a.B < 1) return false;
  if (a.mode == kModeSel && a.diag == NSA_DIAG_NONE) return false;   // a query must see at least one key
  const int64_t ns = slots_per_query(a);
  if (ns > 255) return false;
  const int64_t nqb = (a.N + kBlock - 1) / kBlock, nkb = (a.Nk + kBlock - 1) / kBlock;
  if (nkb > 8192) return false;
  const int64_t lists = (int64_t)a.B * a.Hkv * nkb;
  if (lists * nqb > (1ll << 31) - 1) return false;
  if ((int64_t)a.B * a.Hkv * ((int64_t)a.N * ns + nkb * kRows) > (1ll << 31) - 1) return false;
  if ((int64_t)a.B * a.Hq * (int64_t)a.N * ns > (1ll << 31) - 1) return false;   // (row, slot) ids are 32-bit
  if (a.k.stride_n < a.D || a.v.stride_n < a.D) return false;
  return true;
}

// The forward of the compressed and the sliding-window branch runs query-tile stationary (dense_fwd_kernel).  It
// stores whole rows of a plain contiguous output; other layouts of `out` (and a compressed branch without a memory
// slot, where a query may see no key) are left to the generic kernels.
static bool dense_forward(const SelProblem& a) { return a.mode != kModeSel; }
static bool dense_forward_serves(const SelProblem& a) {
  if (a.mode == kModeCmp && a.num_mem < 1) return false;
  return a.out.stride_n == a.D && a.out.stride_h == (int64_t)a.N * a.D && a.out.stride_b == (int64_t)a.Hq * a.N * a.D;
}

constexpr int64_t kPartialBudget = 8ll << 30;

static SelPlan make_plan(const SelProblem& a, bool backward) {
  SelPlan p;
  p.nqb = (a.N + kBlock - 1) / kBlock;
  p.nkb = (a.Nk + kBlock - 1) / kBlock;
  p.ns = slots_per_query(a);
  p.G = a.Hq / a.Hkv;
  p.QT = kRows / p.G;
  p.nlists = a.B * a.Hkv * p.nkb;
  p.entries_cap = (int64_t)a.B * a.Hkv * (int64_t)a.N * p.ns + (int64_t)p.nlists * p.QT;
  p.items_cap = p.entries_cap / p.QT + p.nlists + 1;   // an item holds at least one chunk
  p.words = (p.ns + 31) / 32;
  int64_t off = 0;
  p.off_status = off; off += 256;
  p.off_num_items = p.off_status + 128;
  if (!backward && dense_forward(a)) {   // only the status word is needed
    p.off_totals = p.off_list_base = p.off_list_item = p.off_cursors = p.off_bits = p.off_items = p.off_entries = p.off_positions = off;
    p.off_partial = p.off_stats = p.off_delta = off;
    p.index_bytes = 0;
    p.total_bytes = off;
    return p;
  }
  p.off_totals = off; off = align_up(off + (int64_t)p.nlists * 4, 256);
  p.off_list_base = off; off = align_up(off + (int64_t)p.nlists * 4, 256);
  p.off_list_item = off; off = align_up(off + (int64_t)(p.nlists + 1) * 4, 256);
  p.off_cursors = off; off = align_up(off + (int64_t)p.nlists * 4, 256);
  p.off_bits = off; off = align_up(off + (int64_t)a.B * a.Hkv * a.N * p.words * 4, 256);
  p.off_items = off; off = align_up(off + p.items_cap * 16, 256);
  p.off_entries = off; off = align_up(off + p.entries_cap * 4, 256);
  p.off_positions = off;
  if (a.mode == kModeSel) off = align_up(off + (int64_t)a.B * a.Hkv * a.N * p.ns * 4, 256);
  p.index_bytes = off;   // status word to positions: the same layout forward and backward
  const int64_t rows = (int64_t)a.B * a.Hq * a.N;
  p.off_partial = p.off_stats = p.off_delta = off;
  p.slices = p.pairs_per_slice = 1;
  if (!backward) {
    p.off_partial = off; off = align_up(off + p.entries_cap * p.G * a.D * 2, 256);
    p.off_stats = off; off = align_up(off + p.entries_cap * p.G * 8, 256);
  } else {
    // very long inputs (64 heads of 128 at 65536 positions: 70 GB for the compressed branch) run in slices of whole
    // (batch, KV head) pairs that share a buffer of at most kPartialBudget, or of one pair
    p.off_delta = off; off = align_up(off + rows * 4, 256);
    const int pairs = a.B * a.Hkv;
    const int64_t per_pair = (int64_t)p.G * a.N * p.ns * a.D * (a.D == 64 ? 2 : 4), most = kPartialBudget / per_pair;
    const int per_slice = (int)(most < 1 ? 1 : most < pairs ? most : pairs);
    p.slices = (pairs + per_slice - 1) / per_slice;
    p.pairs_per_slice = (pairs + p.slices - 1) / p.slices;
    p.slices = (pairs + p.pairs_per_slice - 1) / p.pairs_per_slice;
    p.off_partial = off; off = align_up(off + p.pairs_per_slice * per_pair, 256);
  }
  p.total_bytes = off;
  return p;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// Tensor map over a [B, H, N, d] bf16 view; one box is a [64 rows x 64 columns] tile of one head.
static int make_kv_map(CUtensorMap* map, const nsa_tensor& t, int B, int H, int N, int d) {
  EncodeTiledFn enc = encode_fn();
  if (enc == nullptr) return fail(NSA_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t dims[4] = {(cuuint64_t)d, (cuuint64_t)N, (cuuint64_t)H, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)t.stride_n * 2, (cuuint64_t)(H > 1 ? t.stride_h : t.stride_n * N) * 2,
                           (cuuint64_t)(B > 1 ? t.stride_b : (H > 1 ? t.stride_h * H : t.stride_n * N)) * 2};
  cuuint32_t box[4] = {64, 64, 1, 1}, es[4] = {1, 1, 1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, t.ptr, dims, strides, box, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return NSA_ERR_UNSUPPORTED;   // strides the tiled format cannot express
  return NSA_OK;
}

// Tensor map over the queries of a [B, H, N, d] bf16 view; one box is [128 / G positions x G heads x 64 columns], whose
// rows come in the order (position, head of the group).
static int make_q_map(CUtensorMap* map, const nsa_tensor& t, int B, int H, int N, int d, int G) {
  EncodeTiledFn enc = encode_fn();
  if (enc == nullptr) return fail(NSA_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled is not available from this driver");
  const int64_t sn = N > 1 ? t.stride_n : d, sh = H > 1 ? t.stride_h : sn * N, sb = B > 1 ? t.stride_b : (H > 1 ? sh * H : sn * N);
  cuuint64_t dims[4] = {(cuuint64_t)d, (cuuint64_t)H, (cuuint64_t)N, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)sh * 2, (cuuint64_t)sn * 2, (cuuint64_t)sb * 2};
  cuuint32_t box[4] = {64, (cuuint32_t)G, (cuuint32_t)(kRows / G), 1}, es[4] = {1, 1, 1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, t.ptr, dims, strides, box, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return NSA_ERR_UNSUPPORTED;   // strides the tiled format cannot express
  return NSA_OK;
}

#define CUDA_TRY(expr)                                                        \
  do {                                                                        \
    const cudaError_t e_ = (expr);                                            \
    if (e_ != cudaSuccess) return fail((int)e_, cudaGetErrorString(e_));     \
  } while (0)

static BlockRule make_rule(const SelProblem& a, const SelPlan& p) {
  BlockRule R;
  R.idx = a.idx; R.mask = a.mask;
  R.N = a.N; R.nkb = p.nkb; R.nsel = a.nsel; R.ns = p.ns;
  R.diag = a.diag; R.mode = a.mode; R.window = a.window; R.stride = a.stride > 0 ? a.stride : 1; R.num_mem = a.num_mem;
  return R;
}

// A hash of everything the index depends on besides idx/mask themselves: sizes, head grouping, branch and its rule.
static uint32_t index_tag(const SelProblem& a, const SelPlan& p) {
  const uint32_t f[] = {(uint32_t)a.B, (uint32_t)a.Hkv, (uint32_t)p.G, (uint32_t)a.N, (uint32_t)a.Nk, (uint32_t)p.ns,
                        (uint32_t)a.mode, (uint32_t)a.diag, (uint32_t)a.window, (uint32_t)a.stride, (uint32_t)a.num_mem,
                        (uint32_t)a.nsel, (uint32_t)p.QT, (uint32_t)p.entries_cap};
  uint32_t h = 0x4e534149u;
  for (uint32_t v : f) h = (h ^ v) * 0x01000193u + 0x9E3779B1u;
  return h == 0 ? 1u : h;   // 0 is what a cleared buffer holds
}

static int build_index(const SelProblem& a, const SelPlan& p, uint8_t* ix, cudaStream_t st) {
  int* totals = reinterpret_cast<int*>(ix + p.off_totals);
  int* list_base = reinterpret_cast<int*>(ix + p.off_list_base);
  int* cursors = reinterpret_cast<int*>(ix + p.off_cursors);
  uint32_t* bits = reinterpret_cast<uint32_t*>(ix + p.off_bits);
  int4* items = reinterpret_cast<int4*>(ix + p.off_items);
  int* num_items = reinterpret_cast<int*>(ix + p.off_num_items);
  uint32_t* entries = reinterpret_cast<uint32_t*>(ix + p.off_entries);
  int* list_item = reinterpret_cast<int*>(ix + p.off_list_item);
  int* positions = reinterpret_cast<int*>(ix + p.off_positions);
  const BlockRule R = make_rule(a, p);
  const dim3 grid((a.N + kIndexQueries - 1) / kIndexQueries, a.B, a.Hkv);
  const size_t hist_smem = (size_t)p.nkb * sizeof(int);   // at most 32 KB
  sel_clear_kernel<<<(p.nlists + 255) / 256, 256, 0, st>>>(totals, p.nlists);
  if (a.mode == kModeSel) sel_count_kernel<kModeSel><<<grid, kIndexQueries, hist_smem, st>>>(R, totals, bits, p.words);
  else if (a.mode == kModeSwa) sel_count_kernel<kModeSwa><<<grid, kIndexQueries, hist_smem, st>>>(R, totals, bits, p.words);
  else sel_count_kernel<kModeCmp><<<grid, kIndexQueries, hist_smem, st>>>(R, totals, bits, p.words);
  sel_items_kernel<<<1, 1024, 0, st>>>(totals, list_base, list_item, cursors, items, num_items, p.nlists, p.QT, items_target(a.D), index_tag(a, p));
  if (a.mode == kModeSel) sel_fill_kernel<kModeSel><<<grid, kIndexQueries, hist_smem, st>>>(R, totals, list_base, cursors, entries, positions, p.QT);
  else if (a.mode == kModeSwa) sel_fill_kernel<kModeSwa><<<grid, kIndexQueries, hist_smem, st>>>(R, totals, list_base, cursors, entries, positions, p.QT);
  else sel_fill_kernel<kModeCmp><<<grid, kIndexQueries, hist_smem, st>>>(R, totals, list_base, cursors, entries, positions, p.QT);
  CUDA_TRY(cudaGetLastError());
  count_launches(4);   // clear, count, items, fill
  return NSA_OK;
}

// The word the kernels report through: the caller's accumulator, or the first word of the work buffer, cleared here.
static int prepare_status(const SelProblem& a, const SelPlan& p, uint8_t* ws, cudaStream_t st) {
  if (a.status == nullptr) CUDA_TRY(cudaMemsetAsync(ws + p.off_status, 0, 4, st));
  return NSA_OK;
}

// Where the index is: the caller's (kept from an earlier call, or a buffer of its own to build it into), else the
// leading part of the work buffer.
static int prepare_index(const SelProblem& a, const SelPlan& p, uint8_t* ws, const uint8_t** ix, cudaStream_t st) {
  if (a.index != nullptr) {
    if (a.index_bytes != p.index_bytes) return fail(NSA_ERR_WORKSPACE, "index: not the size the matching *_index_bytes reports");
    *ix = static_cast<const uint8_t*>(a.index);
    return NSA_OK;
  }
  uint8_t* build = ws;
  if (a.index_out != nullptr) {
    if (a.index_out_bytes != p.index_bytes) return fail(NSA_ERR_WORKSPACE, "index_out: not the size the matching *_index_bytes reports");
    build = static_cast<uint8_t*>(a.index_out);
  }
  *ix = build;
  return build_index(a, p, build, st);
}

static void fill_params(SelParams& P, const SelProblem& a, const SelPlan& p, uint8_t* ws, const uint8_t* ix) {
  memset(&P, 0, sizeof(P));
  P.q = (const __nv_bfloat16*)a.q.ptr; P.q_sb = a.q.stride_b; P.q_sh = a.q.stride_h; P.q_sn = a.q.stride_n;
  P.out = (__nv_bfloat16*)a.out.ptr; P.o_sb = a.out.stride_b; P.o_sh = a.out.stride_h; P.o_sn = a.out.stride_n;
  P.idx = a.idx; P.mask = a.mask;
  P.entries = reinterpret_cast<const uint32_t*>(ix + p.off_entries);
  P.items = reinterpret_cast<const int4*>(ix + p.off_items);
  P.num_items = reinterpret_cast<const int*>(ix + p.off_num_items);
  P.index_tag = index_tag(a, p);
  P.bits = reinterpret_cast<const uint32_t*>(ix + p.off_bits);
  P.list_item = reinterpret_cast<const int*>(ix + p.off_list_item);
  P.positions = reinterpret_cast<const int*>(ix + p.off_positions);
  P.bh0 = 0; P.bh1 = a.B * a.Hkv;
  P.words = p.words;
  P.status = a.status != nullptr ? a.status : reinterpret_cast<int*>(ws + p.off_status);
  P.lse = a.lse;
  P.B = a.B; P.Hq = a.Hq; P.Hkv = a.Hkv; P.N = a.N; P.Nk = a.Nk; P.G = p.G; P.nsel = a.nsel; P.nfb = p.nkb;
  P.ns = p.ns;
  P.diag = a.diag; P.scale = a.scale; P.scale_log2 = a.scale * kLog2e;
  P.rule = make_rule(a, p);
  P.importance = a.importance; P.ncb = a.ncb; P.round_bf16 = a.round_bf16;
  P.pooled = a.pooled; P.cpf = a.cpf > 0 ? a.cpf : 1; P.pool_cols = a.ncb / P.cpf; P.pool_block = P.cpf * a.stride;
}

static int num_sms() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

template <int D>
static int run_fwd(const SelProblem& a, const SelPlan& p, uint8_t* ws, cudaStream_t st) {
  CUtensorMap tmK, tmV;
  int rc = make_kv_map(&tmK, a.k, a.B, a.Hkv, a.Nk, D);
  if (rc != NSA_OK) return rc;
  rc = make_kv_map(&tmV, a.v, a.B, a.Hkv, a.Nk, D);
  if (rc != NSA_OK) return rc;
  rc = prepare_status(a, p, ws, st);
  if (rc != NSA_OK) return rc;
  if (dense_forward(a)) {
    SelParams P;
    fill_params(P, a, p, ws, ws);
    const int QT = kRows / p.G;
    const int64_t tiles = (int64_t)a.B * a.Hkv * ((a.N + QT - 1) / QT);
    if (tiles > 0x7fffffffLL) return NSA_ERR_UNSUPPORTED;
    CUtensorMap tmQ;
    rc = make_q_map(&tmQ, a.q, a.B, a.Hq, a.N, D, p.G);
    if (rc != NSA_OK) return rc;
    // two streams per CTA (which share the K / V blocks) once there is a tile for every SM; below that a tile has its own SM
    const int streams = tiles > num_sms() ? dense::kStreams : 1;
    const int64_t work = (int64_t)a.B * a.Hkv * ((a.N + QT * streams - 1) / (QT * streams));
    const unsigned grid = (unsigned)(work < num_sms() ? work : num_sms());
#define NSA_DENSE_LAUNCH(MODE, GI, ...)                                                                                \
    do {                                                                                                              \
      const int smem = (int)dense::smem_bytes<D>(GI, P.pooled != nullptr);                                            \
      CUDA_TRY(cudaFuncSetAttribute(dense_fwd_kernel<D, MODE, GI __VA_OPT__(,) __VA_ARGS__>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)); \
      dense_fwd_kernel<D, MODE, GI __VA_OPT__(,) __VA_ARGS__><<<grid, dense::kThreads, smem, st>>>(tmQ, tmK, tmV, P, streams); \
    } while (0)
    if (a.mode == kModeSwa) NSA_DENSE_LAUNCH(kModeSwa, 0);
    else if (P.pooled != nullptr && p.G == 4) NSA_DENSE_LAUNCH(kModeCmp, 4, true);
    else if (P.pooled != nullptr && p.G == 8) NSA_DENSE_LAUNCH(kModeCmp, 8, true);
    else if (P.pooled != nullptr && p.G == 16) NSA_DENSE_LAUNCH(kModeCmp, 16, true);
    else if (P.pooled != nullptr) return NSA_ERR_UNSUPPORTED;
    else if (P.importance == nullptr) NSA_DENSE_LAUNCH(kModeCmp, 0);
    else if (p.G == 1) NSA_DENSE_LAUNCH(kModeCmp, 1);
    else if (p.G == 2) NSA_DENSE_LAUNCH(kModeCmp, 2);
    else if (p.G == 4) NSA_DENSE_LAUNCH(kModeCmp, 4);
    else if (p.G == 8) NSA_DENSE_LAUNCH(kModeCmp, 8);
    else NSA_DENSE_LAUNCH(kModeCmp, 16);
#undef NSA_DENSE_LAUNCH
    CUDA_TRY(cudaGetLastError());
    count_launches(1);
    return NSA_OK;
  }
  const uint8_t* ix = nullptr;
  rc = prepare_index(a, p, ws, &ix, st);
  if (rc != NSA_OK) return rc;
  SelParams P;
  fill_params(P, a, p, ws, ix);
  P.partial = reinterpret_cast<__nv_bfloat16*>(ws + p.off_partial);
  P.stats = reinterpret_cast<float2*>(ws + p.off_stats);
  constexpr int NC = D / 64;
  const int smem = 1024 + NC * (16384 + 8192 + 8192 + 16384);
  const int per_sm = D == 64 ? 4 : 2;
  CUDA_TRY(cudaFuncSetAttribute(sel_fwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  sel_fwd_kernel<D><<<num_sms() * per_sm, 2 * kRows, smem, st>>>(tmK, tmV, P);
  const int64_t threads = (int64_t)a.B * a.Hq * a.N * (D / 8);
  const unsigned mblocks = (unsigned)((threads + 255) / 256);
  if (a.fuse_combine != nullptr) {
    if (a.fuse_targets->multicast) sel_merge_combine_kernel<D, true><<<mblocks, 256, 0, st>>>(P, *a.fuse_combine, *a.fuse_targets);
    else sel_merge_combine_kernel<D, false><<<mblocks, 256, 0, st>>>(P, *a.fuse_combine, *a.fuse_targets);
  } else {
    sel_merge_kernel<D><<<mblocks, 256, 0, st>>>(P);
  }
  CUDA_TRY(cudaGetLastError());
  count_launches(2);   // forward kernel, merge
  return NSA_OK;
}

template <int D>
static int run_bwd(const SelProblem& a, const SelPlan& p, uint8_t* ws, cudaStream_t st) {
  CUtensorMap tmK, tmV;
  int rc = make_kv_map(&tmK, a.k, a.B, a.Hkv, a.Nk, D);
  if (rc != NSA_OK) return rc;
  rc = make_kv_map(&tmV, a.v, a.B, a.Hkv, a.Nk, D);
  if (rc != NSA_OK) return rc;
  rc = prepare_status(a, p, ws, st);
  if (rc != NSA_OK) return rc;
  const uint8_t* ix = nullptr;
  rc = prepare_index(a, p, ws, &ix, st);
  if (rc != NSA_OK) return rc;
  SelParams P;
  fill_params(P, a, p, ws, ix);
  P.dout = (const __nv_bfloat16*)a.dout.ptr; P.do_sb = a.dout.stride_b; P.do_sh = a.dout.stride_h; P.do_sn = a.dout.stride_n;
  float* delta = reinterpret_cast<float*>(ws + p.off_delta);
  P.delta = a.delta != nullptr ? a.delta : delta;
  P.dq = a.dq; P.dk = a.dk; P.dv = a.dv; P.slot_grads = a.slot_grads;
  if (a.dq_out.ptr != nullptr) {
    P.dq_lp = (__nv_bfloat16*)a.dq_out.ptr; P.dq_sb = a.dq_out.stride_b; P.dq_sh = a.dq_out.stride_h; P.dq_sn = a.dq_out.stride_n;
  }
  const int64_t threads = (int64_t)a.B * a.Hq * a.N * (D / 8);
  const int own_delta = a.delta == nullptr ? 1 : 0;   // the caller may hand the row sums over
  // dk and dv together, as 16-byte pieces: cleared beside the row sums, rounded beside the last merge
  const int64_t kv_pieces = a.dkv_out != nullptr ? (int64_t)a.B * a.Hkv * a.Nk * D / 2 : 0;
  const unsigned kv_blocks = (unsigned)((kv_pieces + 255) / 256 < 148 * 4 ? (kv_pieces + 255) / 256 : 148 * 4), row_blocks = (unsigned)((threads + 255) / 256);
  P.dkv_lp = static_cast<__nv_bfloat16*>(a.dkv_out);
  if (own_delta) sel_delta_kernel<D><<<row_blocks + kv_blocks, 256, 0, st>>>(P, delta, row_blocks, kv_pieces);
  else if (kv_pieces > 0) CUDA_TRY(cudaMemsetAsync(a.dk, 0, (size_t)kv_pieces * 16, st));
  if (a.slot_grads != nullptr) CUDA_TRY(cudaMemsetAsync(a.slot_grads, 0, (size_t)a.B * a.Hkv * a.N * a.nsel * sizeof(float), st));
  CUDA_TRY((allow_shared_memory<sel_bwd_ws_kernel<D, false>>()));
  if (a.slot_grads != nullptr) CUDA_TRY((allow_shared_memory<sel_bwd_ws_kernel<D, true>>()));
  P.partial = reinterpret_cast<__nv_bfloat16*>(ws + p.off_partial);
  for (int s = 0; s < p.slices; ++s) {
    P.bh0 = s * p.pairs_per_slice;
    P.bh1 = P.bh0 + p.pairs_per_slice < a.B * a.Hkv ? P.bh0 + p.pairs_per_slice : a.B * a.Hkv;
    if (a.slot_grads != nullptr) sel_bwd_ws_kernel<D, true><<<num_sms(), ws::kThreads, ws::Shape<D>::kBytes, st>>>(tmK, tmV, P);
    else sel_bwd_ws_kernel<D, false><<<num_sms(), ws::kThreads, ws::Shape<D>::kBytes, st>>>(tmK, tmV, P);
    const unsigned mblocks = (unsigned)(((int64_t)(P.bh1 - P.bh0) * p.G * a.N * (D / 8) + 255) / 256);
    const bool last = s == p.slices - 1;
    const unsigned grid = mblocks + (last ? (kv_blocks + 1) / 2 : 0);
    const int64_t round = last ? kv_pieces / 2 : 0;
    if (a.mode == kModeSel) sel_dq_merge_kernel<D, kModeSel><<<grid, 256, 0, st>>>(P, mblocks, round);
    else if (a.mode == kModeSwa) sel_dq_merge_kernel<D, kModeSwa><<<grid, 256, 0, st>>>(P, mblocks, round);
    else sel_dq_merge_kernel<D, kModeCmp><<<grid, 256, 0, st>>>(P, mblocks, round);
  }
  CUDA_TRY(cudaGetLastError());
  count_launches(2 * p.slices + own_delta);   // (delta,) backward kernel and dQ merge per slice
  return NSA_OK;
}

// ---- the three branches as problems ------------------------------------------------------------

static void problem_base(SelProblem& x) { memset(&x, 0, sizeof(x)); x.stride = 1; }

static bool sel_problem(SelProblem& x, const nsa_sel_fwd_args& a) {
  problem_base(x);
  if (a.dtype != NSA_BF16 || a.block != kBlock || a.sel_heads != a.kv_heads || a.nsel > 254) return false;
  x.q = a.q; x.k = a.k; x.v = a.v; x.out = a.out; x.idx = a.idx; x.mask = a.mask; x.lse = a.lse;
  x.workspace = a.workspace; x.workspace_bytes = a.workspace_bytes;
  x.B = a.batch; x.Hq = a.q_heads; x.Hkv = a.kv_heads; x.N = a.seq; x.Nk = a.seq; x.D = a.dim_head;
  x.nsel = a.nsel; x.diag = a.diag; x.mode = kModeSel; x.scale = a.scale; x.status = a.status;
  return supported(x);
}

static bool swa_problem(SelProblem& x, const nsa_swa_fwd_args& a) {
  problem_base(x);
  if (a.dtype != NSA_BF16 || !a.causal) return false;
  x.q = a.q; x.k = a.k; x.v = a.v; x.out = a.out; x.lse = a.lse;
  x.workspace = a.workspace; x.workspace_bytes = a.workspace_bytes;
  x.B = a.batch; x.Hq = a.q_heads; x.Hkv = a.kv_heads; x.N = a.seq; x.Nk = a.seq; x.D = a.dim_head;
  x.mode = kModeSwa; x.window = a.window; x.scale = a.scale; x.status = a.status;
  return supported(x);
}

static bool cmp_problem(SelProblem& x, const nsa_cmp_fwd_args& a) {
  problem_base(x);
  if (a.dtype != NSA_BF16 || !a.causal || a.sel_heads != a.kv_heads) return false;
  x.q = a.q; x.k = a.ck; x.v = a.cv; x.out = a.out; x.lse = a.lse;
  x.workspace = a.workspace; x.workspace_bytes = a.workspace_bytes;
  x.B = a.batch; x.Hq = a.q_heads; x.Hkv = a.kv_heads; x.N = a.seq; x.Nk = a.num_mem + a.ncb; x.D = a.dim_head;
  x.mode = kModeCmp; x.stride = a.stride; x.num_mem = a.num_mem; x.ncb = a.ncb; x.round_bf16 = 1;
  x.importance = a.importance; x.scale = a.scale; x.status = a.status;
  x.pooled = static_cast<__nv_bfloat16*>(a.pooled); x.cpf = a.pool;
  return supported(x);
}

// The forward can average the importance over the selection blocks itself (`pooled`) when the ring of head means fits
// beside the row maxima in shared memory (128 / G queries x 128 columns of bf16: G >= 4) and every key block of 64
// columns completes a whole number of selection blocks' worth of columns (cpf a power of two).
bool sm100_cmp_fwd_pools(const nsa_cmp_fwd_args& a) {
  SelProblem x;
  if (a.impl == NSA_IMPL_SIMT || !cmp_problem(x, a) || !dense_forward_serves(x)) return false;
  const int G = x.Hq / x.Hkv;
  if (G != 4 && G != 8 && G != 16) return false;
  if (a.pool != 1 && a.pool != 2 && a.pool != 4 && a.pool != 8 && a.pool != 16) return false;
  return a.num_mem <= kBlock && a.ncb / a.pool >= 1;
}

static int check_ws(const SelProblem& x, const SelPlan& p, uint8_t** ws) {
  if (x.workspace == nullptr || x.workspace_bytes < p.total_bytes)
    return fail(NSA_ERR_WORKSPACE, "work buffer missing or smaller than the matching *_workspace_bytes says");
  *ws = static_cast<uint8_t*>(x.workspace);
  if (reinterpret_cast<uintptr_t>(*ws) & 255) return fail(NSA_ERR_ALIGN, "work buffer must be 256-byte aligned");
  return NSA_OK;
}

static int problem_fwd(const SelProblem& x, cudaStream_t st) {
  if (x.N > 1 && x.q.stride_n >> 32) return NSA_ERR_UNSUPPORTED;   // the gathers multiply in 32 bits
  const SelPlan p = make_plan(x, false);
  uint8_t* ws = nullptr;
  const int rc = check_ws(x, p, &ws);
  if (rc != NSA_OK) return rc;
  return x.D == 64 ? run_fwd<64>(x, p, ws, st) : run_fwd<128>(x, p, ws, st);
}

static int problem_bwd(const SelProblem& x, cudaStream_t st) {
  if (x.N > 1 && (x.q.stride_n >> 32 || x.dout.stride_n >> 32)) return NSA_ERR_UNSUPPORTED;   // the gathers multiply in 32 bits
  const SelPlan p = make_plan(x, true);
  uint8_t* ws = nullptr;
  const int rc = check_ws(x, p, &ws);
  if (rc != NSA_OK) return rc;
  return x.D == 64 ? run_bwd<64>(x, p, ws, st) : run_bwd<128>(x, p, ws, st);
}

int64_t sm100_sel_workspace_bytes(const nsa_sel_fwd_args& a, bool backward) {
  SelProblem x;
  if (!sel_problem(x, a)) return NSA_ERR_UNSUPPORTED;
  return make_plan(x, backward).total_bytes;
}
int64_t sm100_sel_index_bytes(const nsa_sel_fwd_args& a) {
  SelProblem x;
  if (!sel_problem(x, a)) return 0;
  return make_plan(x, false).index_bytes;
}
int sm100_sel_fwd(const nsa_sel_fwd_args& a, cudaStream_t st) {
  SelProblem x;
  if (!sel_problem(x, a)) return NSA_ERR_UNSUPPORTED;
  x.index = a.index; x.index_bytes = a.index_bytes;
  x.index_out = a.index_out; x.index_out_bytes = a.index_out_bytes;
  return problem_fwd(x, st);
}
int sm100_sel_fwd_combine(const nsa_sel_fwd_args& a, const CombineParams& c, const GatherTargets& t, cudaStream_t st) {
  SelProblem x;
  if (!sel_problem(x, a)) return NSA_ERR_UNSUPPORTED;
  if (c.batch != x.B || c.q_heads != x.Hq || c.seq != x.N || c.d != x.D) return NSA_ERR_UNSUPPORTED;
  x.index = a.index; x.index_bytes = a.index_bytes;
  x.index_out = a.index_out; x.index_out_bytes = a.index_out_bytes;
  x.fuse_combine = &c; x.fuse_targets = &t;
  return problem_fwd(x, st);
}
int sm100_sel_bwd(const nsa_sel_bwd_args& b, void* dkv_out, cudaStream_t st) {
  SelProblem x;
  if (!sel_problem(x, b.fwd)) return NSA_ERR_UNSUPPORTED;
  x.dkv_out = dkv_out;
  x.dout = b.dout; x.dq = b.dq; x.dk = b.dk; x.dv = b.dv; x.slot_grads = b.slot_grads;
  x.index = b.index; x.index_bytes = b.index_bytes; x.dq_out = b.dq_out; x.delta = b.delta;
  return problem_bwd(x, st);
}

// True when the backward of this problem stores every row of dq (partials + ordered merge) instead of adding into it.
bool sm100_sel_bwd_overwrites_dq(const nsa_sel_fwd_args& a) {
  SelProblem x;
  return sel_problem(x, a);
}
bool sm100_swa_bwd_overwrites_dq(const nsa_swa_fwd_args& a) {
  SelProblem x;
  return swa_problem(x, a);
}
bool sm100_cmp_bwd_overwrites_dq(const nsa_cmp_fwd_args& a) {
  SelProblem x;
  return cmp_problem(x, a);
}

// The index of the sliding and the compressed backward depends on the sizes only: a caller may keep it across calls.
int64_t sm100_swa_index_bytes(const nsa_swa_fwd_args& a) {
  SelProblem x;
  if (!swa_problem(x, a)) return 0;
  return make_plan(x, true).index_bytes;
}
int64_t sm100_cmp_index_bytes(const nsa_cmp_fwd_args& a) {
  SelProblem x;
  if (!cmp_problem(x, a)) return 0;
  x.importance = nullptr;
  return make_plan(x, true).index_bytes;
}

int64_t sm100_swa_workspace_bytes(const nsa_swa_fwd_args& a, bool backward) {
  SelProblem x;
  if (!swa_problem(x, a)) return NSA_ERR_UNSUPPORTED;
  return make_plan(x, backward).total_bytes;
}
int sm100_swa_fwd(const nsa_swa_fwd_args& a, cudaStream_t st) {
  SelProblem x;
  if (!swa_problem(x, a) || !dense_forward_serves(x)) return NSA_ERR_UNSUPPORTED;
  return problem_fwd(x, st);
}
int sm100_swa_bwd(const nsa_swa_bwd_args& b, cudaStream_t st) {
  SelProblem x;
  if (!swa_problem(x, b.fwd)) return NSA_ERR_UNSUPPORTED;
  x.dout = b.dout; x.dq = b.dq; x.dk = b.dk; x.dv = b.dv; x.dq_out = b.dq_out;
  x.index = b.index; x.index_bytes = b.index_bytes; x.delta = b.delta;
  return problem_bwd(x, st);
}

int64_t sm100_cmp_workspace_bytes(const nsa_cmp_fwd_args& a, bool backward) {
  SelProblem x;
  if (!cmp_problem(x, a)) return NSA_ERR_UNSUPPORTED;
  return make_plan(x, backward).total_bytes;
}
int sm100_cmp_fwd(const nsa_cmp_fwd_args& a, cudaStream_t st) {
  SelProblem x;
  if (!cmp_problem(x, a) || !dense_forward_serves(x)) return NSA_ERR_UNSUPPORTED;
  if (x.pooled != nullptr) {
    if (!sm100_cmp_fwd_pools(a)) return NSA_ERR_UNSUPPORTED;
    x.importance = nullptr;
  }
  if (x.importance != nullptr) {
    // columns a query cannot see carry the head mean of the sentinel; the kernel overwrites the visible ones
    float fill = 0.f;
    const int G = x.Hq / x.Hkv;
    for (int g = 0; g < G; ++g) fill += a.sentinel;
    fill = __bfloat162float(__float2bfloat16_rn(fill / (float)G));
    const int64_t count = (int64_t)x.B * x.Hkv * x.N * x.ncb;
    const int64_t rows = (int64_t)x.B * x.Hkv * x.N;
    if (x.ncb % 4 == 0 && (reinterpret_cast<uintptr_t>(x.importance) & 15u) == 0 && rows > 0) {
      const int64_t slices = (int64_t)x.B * x.Hkv;
      const int64_t blocks = (slices * ((x.N + 1) / 2) + 7) / 8;
      fill_invisible_kernel<<<(unsigned)(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, st>>>(x.importance, fill, slices, x.N,
                                                                                              x.ncb, x.stride);
    } else {
      fill_kernel<<<(unsigned)((count + 1023) / 1024 < 148 * 16 ? (count + 1023) / 1024 : 148 * 16), 256, 0, st>>>(x.importance, fill, count);
    }
    count_launches(1);
  }
  return problem_fwd(x, st);
}
int sm100_cmp_bwd(const nsa_cmp_bwd_args& b, cudaStream_t st) {
  SelProblem x;
  if (!cmp_problem(x, b.fwd)) return NSA_ERR_UNSUPPORTED;
  x.importance = nullptr;
  x.pooled = nullptr;
  x.dout = b.dout; x.dq = b.dq; x.dk = b.dck; x.dv = b.dcv; x.dq_out = b.dq_out;
  x.index = b.index; x.index_bytes = b.index_bytes; x.delta = b.delta;
  return problem_bwd(x, st);
}

// ---- forward without a caller-provided work buffer ---------------------------------------------
//
// Some callers cannot hand over device memory for the work buffer: code that runs where the CUDA
// allocator must not be entered (a serving loop holding an allocator lock, a plug-in host whose
// memory pool is closed to extensions, an embedder that forbids cudaMalloc after start-up).  For
// them the forward pass can run on a fixed scratch area that is part of the library image.  Every
// device that loads the library reserves kStaticScratchBytes for it until the process ends.
constexpr int64_t kStaticScratchBytes = 96ll << 20;   // (32 MB of partial rows and, at most, twice that of padding to whole chunks)
static __device__ __align__(256) unsigned char g_sel_scratch[kStaticScratchBytes];

// Filled on first use per device without a lock: every thread that races here stores the same address.
constexpr int kMaxDevices = 64;
static unsigned char* g_scratch_ptr[kMaxDevices] = {nullptr};

// The device address of the scratch array for the current device.  In host code the array's name
// is only a handle; the address a kernel can use comes from cudaGetSymbolAddress, asked once per
// device while that device is current.
static int static_scratch(unsigned char** out) {
  int dev = -1;
  CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return fail(NSA_ERR_UNSUPPORTED, "device ordinal beyond the scratch table");
  if (g_scratch_ptr[dev] == nullptr) {
    void* p = nullptr;
    CUDA_TRY(cudaGetSymbolAddress(&p, g_sel_scratch));
    g_scratch_ptr[dev] = static_cast<unsigned char*>(p);
  }
  *out = g_scratch_ptr[dev];
  return NSA_OK;
}

int sm100_sel_fwd_static(const nsa_sel_fwd_args& a, cudaStream_t st) {
  SelProblem x;
  if (!sel_problem(x, a)) return fail(NSA_ERR_UNSUPPORTED, "nsa_sel_fwd_static: shape outside the tensor-core family (bf16, block 64, dim_head 64/128, shared selection, own block included)");
  x.status = nullptr;   // the area's own first word, see sm100_sel_static_status
  const SelPlan p = make_plan(x, false);
  if (p.total_bytes > kStaticScratchBytes) {
    static thread_local char msg[160];
    snprintf(msg, sizeof(msg), "nsa_sel_fwd_static: this problem needs %lld bytes of scratch, the built-in area holds %lld",
             (long long)p.total_bytes, (long long)kStaticScratchBytes);
    return fail(NSA_ERR_WORKSPACE, msg);
  }
  unsigned char* ws = nullptr;
  const int rc = static_scratch(&ws);
  if (rc != NSA_OK) return rc;
  return x.D == 64 ? run_fwd<64>(x, p, ws, st) : run_fwd<128>(x, p, ws, st);
}

int64_t sm100_static_scratch_bytes() { return kStaticScratchBytes; }

// The status word the kernels of the last nsa_sel_fwd_static call on this device left in the built-in area (its
// first four bytes): copied to `out`, host or device memory, in stream order.  Nothing is allocated.
int sm100_sel_static_status(int* out, cudaStream_t st) {
  if (out == nullptr) return fail(NSA_ERR_NULL, "nsa_sel_static_status: NULL output pointer");
  unsigned char* ws = nullptr;
  const int rc = static_scratch(&ws);
  if (rc != NSA_OK) return rc;
  CUDA_TRY(cudaMemcpyAsync(out, ws, sizeof(int), cudaMemcpyDefault, st));
  return NSA_OK;
}

// ---- self-test of the bounded waits ----------------------------------------------------------------
//
// One block that does what every tensor-core kernel here does around a wait -- allocates tensor memory, waits on an
// mbarrier with a limit, and on giving up raises its abort flag, frees the tensor memory and reports status 1 -- except
// that nobody ever arrives on its barrier and the limit is `limit_cycles` (about a millisecond in the test) instead of
// a second.  It returns by itself; nothing traps, faults or spins without a bound.
__global__ void __launch_bounds__(128) wait_selftest_kernel(int* status, long long limit_cycles) {
  __shared__ int abort_flag;
  __shared__ uint32_t tmem_slot;
  __shared__ __align__(8) uint64_t bar;
  const int tid = threadIdx.x, warp = tid >> 5;
  if (tid == 0) {
    abort_flag = 0;
    mbar_init(smem_u32(&bar), 1);
    fence_mbar_init();
  }
  __syncthreads();
  if (warp == 0) {
    tmem_alloc(smem_u32(&tmem_slot), 32);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tm = tmem_slot;
  mbar_wait_warp(smem_u32(&bar), 0, &abort_flag, limit_cycles);   // nobody arrives: every warp runs into the limit
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 32);
  if (tid == 0 && abort_flag) atomicExch(status, 1);
}

int sm100_wait_selftest(int* status_device, int64_t limit_cycles, cudaStream_t st) {
  if (status_device == nullptr) return fail(NSA_ERR_NULL, "nsa_selftest_bounded_wait: NULL status pointer");
  if (limit_cycles < 1 || limit_cycles > kWaitLimitCycles) return fail(NSA_ERR_SHAPE, "nsa_selftest_bounded_wait: limit out of range");
  CUDA_TRY(cudaMemsetAsync(status_device, 0, sizeof(int), st));
  wait_selftest_kernel<<<1, 128, 0, st>>>(status_device, (long long)limit_cycles);
  CUDA_TRY(cudaGetLastError());
  count_launches(1);
  return NSA_OK;
}

}  // namespace nsa
