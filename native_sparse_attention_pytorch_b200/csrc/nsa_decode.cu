// Decoding: one token per batch element against the caches.
//
// decode_kernel is the attention of a step in a single launch: compressed attention over the blocks compressed so far
// (with its per-block logits), block selection, attention over the selected blocks plus the part of the own block that
// exists, sliding window, and the gated combine into the merged row.
//
// A thread-block cluster of S CTAs serves one (batch element, KV head) and the G query heads of that head together, so
// every key / value row is fetched once for the group.  All arithmetic is fp32.  Bound: latency.  A step reads a few
// thousand key rows per KV head; one CTA walking them serially took 370 us at 32768 cached tokens (8 KV heads), while
// spread over the cluster a warp has one or two tiles of 16 keys per branch.  Inside a branch the warps of the cluster
// take tiles in turn, keep an online softmax each and fold through shared memory; the CTAs' results meet at the end
// through distributed shared memory.  The compressed logits are stored into every CTA of the cluster as they are
// computed, so each of them selects the blocks itself, behind the sliding window, which does not depend on them: one cluster
// barrier instead of two.
//   * Key and value rows are staged by cp.async (whole 128-byte lines) into two buffers per warp, the first tile of a
//     branch before the previous branch is folded; two lanes share a key for the dot products.
//
// In a step of the whole layer it also takes the token's row of the qkv projection as it is: it rotates the queries and
// the new key and appends key and value to the caches and to the window that is being filled for the next compressed
// block.  project_*_kernel run before it (norm of the token, qkv projection, sigmoid gates) and after it (output
// projection).  As separate tensor operations a step was some 25 launches and 500 us of host time.

#include "nsa_common.cuh"
#include "nsa_kernels.h"
#include "nsa_sm100_ptx.cuh"

namespace nsa {

template <typename T>
struct DecodeShape {
  static constexpr int kWarps = sizeof(T) == 4 ? 4 : 8;   // fp32 rows are twice as long: half as many staging areas
};
constexpr int kMaxCluster = 8;    // the portable limit: clusters of 16 find room on part of the chip only and ran in two waves

template <typename T>
__device__ __forceinline__ void store_vec(T* dst, const float* x) {
#pragma unroll
  for (int e = 0; e < Elem<T>::kVec; e += 2) Elem<T>::store2(dst + e, x[e], x[e + 1]);
}

using ptx::cluster_arrive;
using ptx::cluster_rank;
using ptx::cluster_wait;
using ptx::map_rank;
using ptx::st_cluster;
using ptx::st_cluster_v2;

// A tile of up to kTile consecutive keys (kLongTile in the form for very long caches): where its rows are
constexpr int kTile = 16, kLongTile = 4;
template <typename T>
struct KeyTile {
  const T *k, *v;
  int64_t k_sn, v_sn;
  int cnt;
};

// Requests the key and value rows of a tile into a staging buffer (ROWS rows of each, padded by 16 bytes so that
// neighbouring rows fall on different banks); one commit group.  Missing rows are zeroed: they take part in products.
template <typename T, int ROWS>
__device__ __forceinline__ void stage_tile(uint32_t buf, const KeyTile<T>& t, int d, int lane) {
  const int row_bytes = d * (int)sizeof(T), padded = row_bytes + 16;
  const int pieces = row_bytes / 16;
  // lanes per row: the largest power of two that fits a row's pieces, the rest of the row in further steps
  const int lpr = pieces >= 32 ? 32 : pieces >= 16 ? 16 : pieces >= 8 ? 8 : pieces >= 4 ? 4 : pieces >= 2 ? 2 : 1;
  const int sub = lane & (lpr - 1);
#pragma unroll 1
  for (int r = lane / lpr; r < ROWS; r += 32 / lpr) {
    const bool ok = r < t.cnt;
    const T *kr = t.k + (ok ? r * t.k_sn : 0), *vr = t.v + (ok ? r * t.v_sn : 0);
    const uint32_t dst = buf + r * padded;
    for (int c = sub; c < pieces; c += lpr) {
      ptx::cp_async16(dst + c * 16, kr + c * (16 / (int)sizeof(T)), ok ? 16u : 0u);
      ptx::cp_async16(dst + ROWS * padded + c * 16, vr + c * (16 / (int)sizeof(T)), ok ? 16u : 0u);
    }
  }
  ptx::cp_async_commit();
}

// The state of a branch in one warp, on CUDA cores (fp32 inputs, and head sizes the tensor form below does not have).
// Two lanes share a key for the dot products; for the values a lane owns feature pairs.
template <typename T, int GT, int ROWS = kTile>
struct ScalarState {
  static constexpr int kHeads = GT, kRows = ROWS;
  float m[GT], l[GT], acc[GT][2][2];

  __device__ __forceinline__ void start(const T*, int, int) {
#pragma unroll
    for (int g = 0; g < GT; ++g) {
      m[g] = -INFINITY;
      l[g] = 0.f;
      acc[g][0][0] = acc[g][0][1] = acc[g][1][0] = acc[g][1][1] = 0.f;
    }
  }
  // One staged tile; `rows` holds the GT query rows; `imp` (or NULL) gets the mean over the first G heads of every
  // key's scaled logit through push(key, mean)
  template <typename Push>
  __device__ __forceinline__ void tile(const uint8_t* buf, const T* rows, int cnt, int d, float scale, int lane, int G, bool want,
                                       Push push) {
    constexpr int V = Elem<T>::kVec;
    const int padded = d * (int)sizeof(T) + 16;
    const bool present = lane / 2 < cnt;
    float logit[GT];
#pragma unroll
    for (int g = 0; g < GT; ++g) logit[g] = 0.f;
    const T* key = reinterpret_cast<const T*>(buf + min(lane / 2, ROWS - 1) * padded);
#pragma unroll 1
    for (int c = (lane & 1) * V; c < d; c += 2 * V) {
      float kv[V];
      Elem<T>::load_vec(key + c, kv);
#pragma unroll
      for (int g = 0; g < GT; ++g) {
        float q[V];
        Elem<T>::load_vec(rows + g * (d + 8) + c, q);
#pragma unroll
        for (int e = 0; e < V; ++e) logit[g] = fmaf(q[e], kv[e], logit[g]);
      }
    }
#pragma unroll
    for (int g = 0; g < GT; ++g) logit[g] = (logit[g] + __shfl_xor_sync(kFullMask, logit[g], 1)) * scale;
    if (want && present && !(lane & 1)) {
      float sum = 0.f;
#pragma unroll
      for (int g = 0; g < GT; ++g) sum += g < G ? logit[g] : 0.f;
      push(lane / 2, sum / (float)G);
    }
    float p[GT];
#pragma unroll
    for (int g = 0; g < GT; ++g) {
      const float m_new = fmaxf(m[g], warp_max(present ? logit[g] : -INFINITY));
      const float alpha = exp2f((m[g] - m_new) * kLog2e);
      p[g] = present ? exp2f((logit[g] - m_new) * kLog2e) : 0.f;
      l[g] = l[g] * alpha + warp_sum(lane & 1 ? 0.f : p[g]);
      m[g] = m_new;
      acc[g][0][0] *= alpha; acc[g][0][1] *= alpha;
      acc[g][1][0] *= alpha; acc[g][1][1] *= alpha;
    }
    const bool in0 = 2 * lane < d, in1 = 64 + 2 * lane < d;
    const uint8_t* vrow = buf + ROWS * padded + 2 * lane * (int)sizeof(T);
#pragma unroll 2
    for (int k = 0; k < cnt; ++k) {
      const T* row = reinterpret_cast<const T*>(vrow + k * padded);
      const float2 v0 = in0 ? Elem<T>::load2(row) : make_float2(0.f, 0.f);
      const float2 v1 = in1 ? Elem<T>::load2(row + 64) : make_float2(0.f, 0.f);
#pragma unroll
      for (int g = 0; g < GT; ++g) {
        const float pg = __shfl_sync(kFullMask, p[g], 2 * k);
        acc[g][0][0] = fmaf(pg, v0.x, acc[g][0][0]);
        acc[g][0][1] = fmaf(pg, v0.y, acc[g][0][1]);
        acc[g][1][0] = fmaf(pg, v1.x, acc[g][1][0]);
        acc[g][1][1] = fmaf(pg, v1.y, acc[g][1][1]);
      }
    }
  }
  // to shared memory: [g][d + 2]: unnormalised row, maximum (base-2 logarithm), sum
  __device__ __forceinline__ void park(float* dst, int d, int lane) const {
#pragma unroll
    for (int g = 0; g < GT; ++g) {
      float* row = dst + g * (d + 2);
      if (lane == 0) { row[d] = m[g] * kLog2e; row[d + 1] = l[g]; }
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int dim = 64 * c + 2 * lane;
        if (dim < d) { row[dim] = acc[g][c][0]; row[dim + 1] = acc[g][c][1]; }
      }
    }
  }
};

// The same on the warp-level tensor instructions (m16n8k16, bf16 operands, fp32 accumulators): keys are the 16 rows of
// S = K Q^T, the query heads its 8 columns, and O^T = V^T P^T has the features as rows.  A tile is some 60 instructions
// instead of 1500 (8 heads of 128), which also keeps the kernel inside the instruction cache: every part of it runs
// once or twice per launch, and fetching its code was most of the time.  (tcgen05 has nothing to offer here: its
// smallest tile is 64 rows, and the work is a few tiles per warp.)  Queries, keys and values are bf16 already; the fp32
// probabilities go in as three bf16 terms (8 bits each), so no precision is given up against fp32 arithmetic.
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <bool TRANS>
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
  if (TRANS)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t transpose_8x8(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}

template <int D, int GT>
struct TensorState {
  using T = __nv_bfloat16;
  static constexpr int kHeads = GT, kRows = kTile;
  static constexpr int NT = (GT + 7) / 8;        // groups of eight heads
  // lane l holds heads 8 n + 2 (l % 4) + {0, 1}; accumulator rows are the features 16 t + l / 4 (+ 8)
  float m[NT][2], l[NT][2], o[NT][D / 16][4];
  uint32_t qf[NT][D / 16][2];                    // the query rows as B operands

  __device__ __forceinline__ void start(const T* rows, int, int lane) {
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      m[n][0] = m[n][1] = -INFINITY;
      l[n][0] = l[n][1] = 0.f;
      const int g = 8 * n + lane / 4;
#pragma unroll
      for (int t = 0; t < D / 16; ++t) {
        o[n][t][0] = o[n][t][1] = o[n][t][2] = o[n][t][3] = 0.f;
        const T* src = rows + g * (D + 8) + t * 16 + 2 * (lane & 3);
        qf[n][t][0] = g < GT ? *reinterpret_cast<const uint32_t*>(src) : 0u;
        qf[n][t][1] = g < GT ? *reinterpret_cast<const uint32_t*>(src + 8) : 0u;
      }
    }
  }
  template <typename Push>
  __device__ __forceinline__ void tile(const uint8_t* buf, const T*, int cnt, int, float scale, int lane, int G, bool want, Push push) {
    constexpr int padded = D * 2 + 16;
    const uint32_t kb = ptx::smem_u32(buf), vb = kb + kTile * padded;
    float s[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
    for (int t = 0; t < D / 16; ++t) {
      uint32_t a[4];   // rows lane % 16, 16-byte half lane / 16 of the 32-byte step
      ldmatrix4<false>(a, kb + (lane & 15) * padded + t * 32 + (lane >> 4) * 16);
#pragma unroll
      for (int n = 0; n < NT; ++n) mma_16816(s[n], a, qf[n][t][0], qf[n][t][1]);
    }
    const int r0 = lane / 4, r1 = r0 + 8;        // this lane's keys
    if (want) {   // mean over the heads: the lane's own, then the other three lanes of the quad
      float a0 = 0.f, a1 = 0.f;
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          if (8 * n + 2 * (lane & 3) + e < G) { a0 += s[n][e] * scale; a1 += s[n][2 + e] * scale; }
      a0 += __shfl_xor_sync(kFullMask, a0, 1); a1 += __shfl_xor_sync(kFullMask, a1, 1);
      a0 += __shfl_xor_sync(kFullMask, a0, 2); a1 += __shfl_xor_sync(kFullMask, a1, 2);
      if ((lane & 3) == 0) {
        if (r0 < cnt) push(r0, a0 / (float)G);
        if (r1 < cnt) push(r1, a1 / (float)G);
      }
    }
    const float c2 = scale * kLog2e;
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      uint32_t b[3][2];                          // P^T in three bf16 terms: [term][keys 0-7, 8-15]
#pragma unroll
      for (int e = 0; e < 4; ++e) s[n][e] = (e < 2 ? r0 : r1) < cnt ? s[n][e] * c2 : -INFINITY;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float mx = fmaxf(s[n][e], s[n][2 + e]);
        mx = fmaxf(mx, __shfl_xor_sync(kFullMask, mx, 4));
        mx = fmaxf(mx, __shfl_xor_sync(kFullMask, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(kFullMask, mx, 16));
        const float m_new = fmaxf(m[n][e], mx);
        const float alpha = exp2f(m[n][e] - m_new);
        m[n][e] = m_new;
        s[n][e] = exp2f(s[n][e] - m_new);
        s[n][2 + e] = exp2f(s[n][2 + e] - m_new);
        l[n][e] = l[n][e] * alpha + s[n][e] + s[n][2 + e];   // of this lane's keys; summed over the lanes in park()
#pragma unroll
        for (int t = 0; t < D / 16; ++t) { o[n][t][e] *= alpha; o[n][t][2 + e] *= alpha; }
      }
#pragma unroll
      for (int term = 0; term < 3; ++term)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float &x = s[n][2 * half], &y = s[n][2 * half + 1];
          const uint32_t w = ptx::pack_bf16(x, y);
          x -= __uint_as_float(w << 16);
          y -= __uint_as_float(w & 0xffff0000u);
          b[term][half] = transpose_8x8(w);
        }
#pragma unroll
      for (int t = 0; t < D / 16; ++t) {
        uint32_t a[4];   // V^T: features 16 t .. + 15 as rows, the 16 keys as columns
        ldmatrix4<true>(a, vb + ((lane & 7) + (lane >> 4) * 8) * padded + t * 32 + ((lane >> 3) & 1) * 16);
#pragma unroll
        for (int term = 0; term < 3; ++term) mma_16816(o[n][t], a, b[term][0], b[term][1]);
      }
    }
  }
  __device__ __forceinline__ void park(float* dst, int, int lane) const {
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float sum = l[n][e];
        sum += __shfl_xor_sync(kFullMask, sum, 4);
        sum += __shfl_xor_sync(kFullMask, sum, 8);
        sum += __shfl_xor_sync(kFullMask, sum, 16);
        const int g = 8 * n + 2 * (lane & 3) + e;
        if (g < GT) {
          float* row = dst + g * (D + 2);
          if (lane < 4) { row[D] = m[n][e]; row[D + 1] = sum; }
#pragma unroll
          for (int t = 0; t < D / 16; ++t) {
            row[16 * t + lane / 4] = o[n][t][e];
            row[16 * t + 8 + lane / 4] = o[n][t][2 + e];
          }
        }
      }
  }
};

// Logit of block column j: mean over its compressed blocks
__device__ __forceinline__ float block_logit(const DecodeParams& P, const float* imp_s, int j, int cpf) {
  if (P.stride == P.block) return imp_s[j];
  if (cpf == 4) {
    const float4 q = *reinterpret_cast<const float4*>(imp_s + 4 * j);
    return (((q.x + q.y) + q.z) + q.w) * 0.25f;
  }
  float sum = 0.f;
  for (int c = 0; c < cpf; ++c) sum += imp_s[j * cpf + c];
  return sum / (float)cpf;
}

// The `want` largest of `cols` probabilities (ties to the lower column); one warp.  The picks are a set: attention does not
// care in which order the blocks come.  The want-th largest of the 32 lanes' maxima bounds them from below, the columns that
// reach it (20 to 30 of 512) are ranked against each other; where they are more than kCandidates, the want-th largest value is
// found by bisection on the values' bit patterns, which order as the values do because probabilities are not negative.
constexpr int kCandidates = 64;
__device__ __forceinline__ void pick_blocks(const float* prob_s, int cols, int want, float* cand_p, int* cand_col, int* sel_idx, int lane) {
  float top = 0.f;
  for (int j = lane; j < cols; j += 32) top = fmaxf(top, prob_s[j]);
  int r = 0;
#pragma unroll
  for (int o = 0; o < 32; ++o) {
    const float other = __shfl_sync(kFullMask, top, o);
    r += other > top || (other == top && o < lane) ? 1 : 0;
  }
  const float bound = __shfl_sync(kFullMask, top, __ffs(__ballot_sync(kFullMask, r == want - 1)) - 1);
  int n = 0;
  for (int j0 = 0; j0 < cols; j0 += 32) {
    const float p = j0 + lane < cols ? prob_s[j0 + lane] : -1.f;
    const unsigned in = __ballot_sync(kFullMask, p >= bound);
    const int at = n + __popc(in & ((1u << lane) - 1u));
    if (p >= bound && at < kCandidates) {
      cand_p[at] = p;
      cand_col[at] = j0 + lane;
    }
    n += __popc(in);
  }
  __syncwarp();
  if (n <= kCandidates) {                       // in the order of their columns
    for (int c = lane; c < n; c += 32) {
      const float p = cand_p[c];
      int rank = 0;
      for (int o = 0; o < n; ++o) rank += cand_p[o] > p || (cand_p[o] == p && o < c) ? 1 : 0;
      if (rank < want) sel_idx[rank] = cand_col[c];
    }
    return;
  }
  auto key_of = [&](int j) { return j < cols ? __float_as_uint(prob_s[j]) : 0u; };
  auto count_from = [&](unsigned from) {
    unsigned c = 0u;
    for (int j = lane; j < cols; j += 32) c += key_of(j) >= from ? 1u : 0u;
    return (int)__reduce_add_sync(kFullMask, c);
  };
  // the largest `cut` with at least `want` columns at or above it
  unsigned cut = __float_as_uint(bound), hi = __reduce_max_sync(kFullMask, __float_as_uint(top)) + 1u;
#pragma unroll 1
  while (hi - cut > 1u) {
    const unsigned mid = cut + (hi - cut) / 2u;
    if (count_from(mid) >= want) cut = mid;
    else hi = mid;
  }
  // everything above the cut, and of the columns at it the lowest
  int at_cut = want - count_from(cut + 1u), count = 0;
  for (int j0 = 0; j0 < cols; j0 += 32) {
    const unsigned key = key_of(j0 + lane);
    const unsigned eq = __ballot_sync(kFullMask, key == cut);
    const bool take = key > cut || (key == cut && __popc(eq & ((1u << lane) - 1u)) < at_cut);
    at_cut -= min(at_cut, __popc(eq));
    const unsigned picked = __ballot_sync(kFullMask, take);
    if (take) sel_idx[count + __popc(picked & ((1u << lane) - 1u))] = j0 + lane;
    count += __popc(picked);
  }
}

// What a CTA needs in shared memory, in bytes from the start of the dynamic segment (the same in all of a cluster)
struct DecodeLayout {
  int stage, q, area, recv, ml, imp, prob, total;
  int shift;      // a CTA finishes 2^shift features of every head of the group
};
__host__ __device__ inline DecodeLayout decode_layout(int el, int GT, int rows, int d, int W, int S, int ncb, int cols) {
  DecodeLayout L;
  auto up = [](int x) { return (x + 15) / 16 * 16; };
  L.shift = 0;
  while ((S << L.shift) < d) ++L.shift;
  L.stage = 0;                                               // [W][2 buffers][keys, values][tile] rows
  L.q = L.stage + W * 4 * rows * (d * el + 16);              // [un-rotated, rotated][GT] rows of d + 8
  L.area = L.q + up(2 * GT * (d + 8) * el);                  // parked warp states [W][GT][d + 2]
  L.recv = L.area + up(W * GT * (d + 2) * 4);                // [S][3 branches][GT][2^shift]: every CTA's part of this CTA's features
  L.ml = L.recv + up(((S * 3 * GT) << L.shift) * 4);         // [S][3][GT][2]: every CTA's maxima and sums
  L.imp = L.ml + up(S * 3 * GT * 2 * 4);                     // head-mean logit of every compressed block
  L.prob = L.imp + up(ncb * 4);                              // block probabilities
  L.total = L.prob + up(cols * 4);
  return L;
}

// `P.chained`: the kernel before it in the stream is the projection it reads the qkv rows and gates from, whose CTAs let this one
// start once everything before the projection is complete.  What does not come from the projection (caches, angles) is then
// fetched while it runs.
template <typename T, typename State>
__global__ void __launch_bounds__(DecodeShape<T>::kWarps * 32, 1) decode_kernel(const DecodeParams P, int S) {
  constexpr int GT = State::kHeads, ROWS = State::kRows;
  const int kThreads = blockDim.x, W = kThreads / 32;
  extern __shared__ __align__(16) uint8_t decode_smem[];
  __shared__ int sel_idx[32];
  __shared__ int sel_count;
  __shared__ float weight[3][GT][kMaxCluster];
  __shared__ float gate_s[3 * GT], turn_s[2][64], fold_s[2][DecodeShape<T>::kWarps];
  __shared__ int live_s[DecodeShape<T>::kWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = (int)cluster_rank();
  const int unit = blockIdx.x / S;
  const int kvh = unit % P.kv_heads, b = unit / P.kv_heads;
  const int G = P.q_heads / P.kv_heads, d = P.d;
  const int cpf = P.block / P.stride;
  const int cols = P.stride != P.block ? P.ncb / cpf : P.ncb;
  const DecodeLayout L = decode_layout((int)sizeof(T), GT, ROWS, d, W, S, P.ncb, cols);
  const int buf_bytes = 2 * ROWS * (d * (int)sizeof(T) + 16);
  uint8_t* const stage = decode_smem + L.stage + warp * 2 * buf_bytes;
  T* const q_s = reinterpret_cast<T*>(decode_smem + L.q);
  float* const area = reinterpret_cast<float*>(decode_smem + L.area);
  float* const imp_s = reinterpret_cast<float*>(decode_smem + L.imp);

  // The three branches as lists of tiles: 0 compressed (memory slots first), 1 sliding window, 2 selected blocks and the
  // part of the own block that exists
  const T* kb = (const T*)P.keys + b * P.k_sb + (int64_t)kvh * P.k_sh;
  const T* vb = (const T*)P.vals + b * P.v_sb + (int64_t)kvh * P.v_sh;
  const int pos = P.T - 1;
  const int mem_tiles = P.ncb > 0 ? (P.num_mem + ROWS - 1) / ROWS : 0;
  const int win0 = max(0, pos - P.window), own0 = pos / P.block * P.block;
  const int per_block = (P.block + ROWS - 1) / ROWS;
  auto tiles_of = [&](int phase) {
    if (phase == 0) return mem_tiles + (P.ncb + ROWS - 1) / ROWS;
    if (phase == 1) return (pos + 1 - win0 + ROWS - 1) / ROWS;
    return sel_count * per_block + (pos + 1 - own0 + ROWS - 1) / ROWS;
  };
  auto locate = [&](int phase, int t) {
    if (phase == 0) {
      if (t < mem_tiles) {
        const int64_t at = ((int64_t)kvh * P.num_mem + t * ROWS) * d;
        return KeyTile<T>{(const T*)P.mem_k + at, (const T*)P.mem_v + at, d, d, min(ROWS, P.num_mem - t * ROWS)};
      }
      const int t0 = (t - mem_tiles) * ROWS;
      return KeyTile<T>{(const T*)P.ck + b * P.ck_sb + (int64_t)kvh * P.ck_sh + t0 * P.ck_sn,
                        (const T*)P.cv + b * P.cv_sb + (int64_t)kvh * P.cv_sh + t0 * P.cv_sn, P.ck_sn, P.cv_sn,
                        min(ROWS, P.ncb - t0)};
    }
    int t0 = win0 + t * ROWS, end = pos + 1;
    if (phase == 2) {
      const int chosen = sel_count * per_block;
      if (t < chosen) {
        const int s = t / per_block;
        t0 = sel_idx[s] * P.block + (t - s * per_block) * ROWS;
        end = min((sel_idx[s] + 1) * P.block, P.T);
      } else {
        t0 = own0 + (t - chosen) * ROWS;
      }
    }
    return KeyTile<T>{kb + t0 * P.k_sn, vb + t0 * P.v_sn, P.k_sn, P.v_sn, min(ROWS, end - t0)};
  };
  // The warps of the cluster take a branch's tiles in turn
  const int first = warp * S + rank;

  ptx::grid_allow_next();
  if (tid == 0) sel_count = 0;
  if (first < tiles_of(0)) stage_tile<T, ROWS>(ptx::smem_u32(stage), locate(0, first), d, lane);
  if (P.qkv != nullptr)
    for (int e = tid; e < d / 2; e += kThreads) {
      const float ang = (float)pos * P.inv_freq[e];
      turn_s[0][e] = cosf(ang);
      turn_s[1][e] = sinf(ang);
    }
  __syncthreads();
  ptx::grid_wait();
  for (int e = tid; e < 3 * G; e += kThreads)
    gate_s[e] = Elem<T>::to_float(((const T*)P.gates)[((int64_t)b * P.q_heads + kvh * G) * 3 + e]);
  {
    constexpr int V = Elem<T>::kVec;
    const int pieces = d / V;
    if (P.qkv != nullptr) {
      // straight from the qkv projection: rotate the queries, and (one CTA) the new key, append key and value
      const int features = (P.q_heads + 2 * P.kv_heads) * d;
      const T* row = (const T*)P.qkv + (int64_t)b * features;
      for (int e = tid; e < (GT + (rank == 0 ? 2 : 0)) * pieces; e += kThreads) {
        const int g = e / pieces, c = (e - g * pieces) * V;
        const int head = g < GT ? kvh * G + g : P.q_heads + (g - GT) * P.kv_heads + kvh;   // GT: the key, GT + 1: the value
        float x[V], y[V];
#pragma unroll
        for (int i = 0; i < V; ++i) x[i] = 0.f;
        if (g < G || g >= GT) Elem<T>::load_vec(row + head * d + c, x);
#pragma unroll
        for (int i = 0; i < V; i += 2) {
          const float co = turn_s[0][(c + i) / 2], si = turn_s[1][(c + i) / 2];
          y[i] = __fadd_rn(__fmul_rn(x[i], co), __fmul_rn(-x[i + 1], si));
          y[i + 1] = __fadd_rn(__fmul_rn(x[i + 1], co), __fmul_rn(x[i], si));
        }
        if (g < GT) {
          store_vec<T>(q_s + g * (d + 8) + c, x);
          store_vec<T>(q_s + (GT + g) * (d + 8) + c, y);
        } else {
          const int64_t cache = b * P.c_sb + kvh * P.c_sh + (int64_t)P.row * d + c;
          const int64_t run = b * P.r_sb + kvh * P.r_sh + (int64_t)P.run_row * d + c;
          if (g == GT) {
            store_vec<T>((T*)P.new_keys + cache, y);
            store_vec<T>((T*)P.run_k + run, x);
          } else {
            store_vec<T>((T*)P.new_vals + cache, x);
            store_vec<T>((T*)P.run_v + run, x);
          }
        }
      }
    } else {
      for (int e = tid; e < 2 * GT * pieces; e += kThreads) {
        const int row = e / pieces, c = (e - row * pieces) * V, g = row >= GT ? row - GT : row;
        const T* src = (const T*)(row >= GT ? P.qr : P.q) + ((int64_t)b * P.q_heads + kvh * G + g) * d + c;
        *reinterpret_cast<uint4*>(q_s + row * (d + 8) + c) = g < G ? *reinterpret_cast<const uint4*>(src) : make_uint4(0u, 0u, 0u, 0u);
      }
    }
  }
  __syncwarp();
  cluster_arrive();     // nobody writes into another CTA's shared memory before that CTA runs, or reads the new cache
  __syncthreads();      // row before it is written
  cluster_wait();

  State state;
#pragma unroll 1
  for (int phase = 0; phase < 3; ++phase) {
    const T* rows = q_s + (phase == 0 ? 0 : GT * (d + 8));
    state.start(rows, d, lane);
    // two staging buffers: the next tile travels under this one's work
    const int total = tiles_of(phase), step = W * S;
    int which = 0;
#pragma unroll 1
    for (int t = first; t < total; t += step) {
      if (t + step < total) {
        stage_tile<T, ROWS>(ptx::smem_u32(stage) + (which ^ 1) * buf_bytes, locate(phase, t + step), d, lane);
        ptx::cp_async_wait<1>();
      } else {
        ptx::cp_async_wait<0>();
      }
      __syncwarp();
      const int cnt = locate(phase, t).cnt;
      const bool want = phase == 0 && t >= mem_tiles;
      if (cnt > 0)
        state.tile(stage + which * buf_bytes, rows, cnt, d, P.scale, lane, G, want, [&](int key, float mean) {
          const uint32_t dst = ptx::smem_u32(imp_s + (t - mem_tiles) * ROWS + key);
          for (int r = 0; r < S; ++r) st_cluster(map_rank(dst, r), mean);
        });
      __syncwarp();
      which ^= 1;
    }
    if (phase == 0) {
      cluster_arrive();       // this warp's logits are on their way to everybody
      // the first tile of the window travels under the fold
      if (first < tiles_of(1)) stage_tile<T, ROWS>(ptx::smem_u32(stage), locate(1, first), d, lane);
    }
    state.park(area + (size_t)warp * GT * (d + 2), d, lane);
    if (phase == 1) {
      // Selection, by every CTA for itself on the logits of the whole cluster: softmax with the sink over the block columns, all
      // threads; then one warp picks.  (One warp for all of it took 11.7 k of the kernel's 46 k cycles at 512 columns.)
      __syncwarp();
      cluster_wait();
      float* const prob_s = reinterpret_cast<float*>(decode_smem + L.prob);
      float mx = -1000.f;     // the sink logit
      for (int j = tid; j < cols; j += kThreads) {
        const float x = block_logit(P, imp_s, j, cpf);
        prob_s[j] = x;
        mx = fmaxf(mx, x);
      }
      mx = warp_max(mx);
      if (lane == 0) fold_s[0][warp] = mx;
      __syncthreads();
      for (int w = 0; w < W; ++w) mx = fmaxf(mx, fold_s[0][w]);
      float part = 0.f;
      for (int j = tid; j < cols; j += kThreads) {
        const float e = expf(prob_s[j] - mx);
        prob_s[j] = e;
        part += e;
      }
      part = warp_sum(part);
      if (lane == 0) fold_s[1][warp] = part;
      __syncthreads();
      float z = expf(-1000.f - mx);
      for (int w = 0; w < W; ++w) z += fold_s[1][w];
      unsigned live = 0u;     // columns above the threshold below which upstream masks a slot out
      for (int j = tid; j < cols; j += kThreads) {
        const float p = prob_s[j] / z;
        prob_s[j] = p;
        live += p > 1e-10f ? 1u : 0u;
      }
      live = __reduce_add_sync(kFullMask, live);
      if (lane == 0) live_s[warp] = (int)live;
      __syncthreads();
      if (warp == 0) {
        int want = 0;
        for (int w = 0; w < W; ++w) want += live_s[w];
        want = min(want, min(min(P.nsel, cols), 32));
        if (want > 0) pick_blocks(prob_s, cols, want, turn_s[0], reinterpret_cast<int*>(turn_s[1]), sel_idx, lane);
        if (lane == 0) sel_count = want;
      }
    }
    __syncthreads();
    if (phase == 1 && first < tiles_of(2)) stage_tile<T, ROWS>(ptx::smem_u32(stage), locate(2, first), d, lane);
    // Fold the warps' states and send every element to the CTA that finishes it: kThreads / GT threads per head, two
    // neighbouring features each
    {
      const int branch = phase == 0 ? 0 : 3 - phase;          // in the order of the gates: compressed, selected, sliding
      const int per = kThreads / GT, g = tid / per, c0 = tid - g * per;
      const float* src = area + (size_t)g * (d + 2);
      const int next = GT * (d + 2);
      float f[8], M = -INFINITY, sum = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        f[w] = w < W ? src[w * next + d] : -INFINITY;
        M = fmaxf(M, f[w]);
      }
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        f[w] = f[w] == -INFINITY ? 0.f : exp2f(f[w] - M);
        if (w < W) sum = fmaf(f[w], src[w * next + d + 1], sum);
      }
      const uint32_t ml = ptx::smem_u32(decode_smem + L.ml) + (uint32_t)(((rank * 3 + branch) * GT + g) * 2) * 4u;
      for (int r = c0; r < S; r += per) st_cluster_v2(map_rank(ml, r), M, sum);
      const uint32_t recv = ptx::smem_u32(decode_smem + L.recv) + ((uint32_t)((rank * 3 + branch) * GT + g) << (L.shift + 2));
#pragma unroll 2
      for (int c = 2 * c0; c < d; c += 2 * per) {
        float2 o = make_float2(0.f, 0.f);
#pragma unroll
        for (int w = 0; w < 8; ++w)
          if (w < W) {
            const float2 x = *reinterpret_cast<const float2*>(src + w * next + c);
            o.x = fmaf(f[w], x.x, o.x);
            o.y = fmaf(f[w], x.y, o.y);
          }
        const int owner = c >> L.shift;
        const uint32_t dst = recv + (uint32_t)(c - (owner << L.shift)) * 4u;
        if (L.shift > 0) {
          st_cluster_v2(map_rank(dst, owner), o.x, o.y);
        } else {              // a CTA finishes one feature
          st_cluster(map_rank(dst, owner), o.x);
          st_cluster(map_rank(dst, owner + 1), o.y);
        }
      }
    }
    __syncthreads();
  }

  // ---- the CTAs' states meet: weight of every (branch, head, CTA) with the gate in it, then this CTA's slice
  cluster_arrive();
  cluster_wait();
  const float* ml = reinterpret_cast<const float*>(decode_smem + L.ml);
  const float* recv = reinterpret_cast<const float*>(decode_smem + L.recv);
  for (int p0 = 0; p0 < 3 * G; p0 += kThreads / kMaxCluster) {     // eight lanes per (branch, head)
    const int p = p0 + tid / kMaxCluster, r = tid % kMaxCluster;
    const int s = min(p, 3 * G - 1) / G, g = min(p, 3 * G - 1) - s * G;
    const float* src = ml + ((r * 3 + s) * GT + g) * 2;
    const float m = r < S ? src[0] : -INFINITY;
    float M = m;
#pragma unroll
    for (int o = kMaxCluster / 2; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(kFullMask, M, o));
    const float f = m == -INFINITY ? 0.f : exp2f(m - M);
    float sum = r < S ? f * src[1] : 0.f;
#pragma unroll
    for (int o = kMaxCluster / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(kFullMask, sum, o);
    if (p < 3 * G) weight[s][g][r] = sum > 0.f ? f * gate_s[g * 3 + s] / sum : 0.f;
  }
  __syncthreads();
  const int width = 1 << L.shift;
  for (int i = tid; i < G << L.shift; i += kThreads) {
    const int g = i >> L.shift, c = (rank << L.shift) + (i & (width - 1));
    if (c >= d) continue;
    float v = 0.f;
#pragma unroll 4
    for (int r = 0; r < S; ++r)
#pragma unroll
      for (int s = 0; s < 3; ++s) v = fmaf(weight[s][g][r], recv[(((r * 3 + s) * GT + g) << L.shift) + (i & (width - 1))], v);
    ((T*)P.out)[((int64_t)b * P.q_heads + kvh * G + g) * d + c] = Elem<T>::from_float(v);
  }
}

// CTAs per (batch, KV head) and warps per CTA; no warps where the logits of all compressed blocks do not fit
template <typename T, typename State>
static void decode_split(const DecodeParams& P, int* S_out, int* W_out, int* smem) {
  constexpr int ROWS = State::kRows;
  constexpr int kMost = 224 * 1024;            // beside the kernel's static part
  const int cpf = P.block / P.stride;
  const int cols = P.stride != P.block ? P.ncb / cpf : P.ncb;
  // enough warps for one tile of the longest branch each, as long as the grid fits one wave
  const int units = P.batch * P.kv_heads;
  const int keys = max(P.ncb, max(P.window + 1, (min(P.nsel, cols) + 1) * P.block));
  int W = DecodeShape<T>::kWarps, S = 1;
  const int tiles = (min(keys, P.T) + ROWS - 1) / ROWS;
  while (S < kMaxCluster && S * W < tiles && units * S * 2 <= 148) S *= 2;
  auto bytes = [&](int warps) { return (int64_t)decode_layout((int)sizeof(T), State::kHeads, ROWS, P.d, warps, S, P.ncb, cols).total; };
  while (W > 2 && bytes(W) > kMost) W /= 2;    // long caches: the logits take the room of staging areas
  *S_out = S;
  *W_out = P.ncb <= (1 << 24) && bytes(W) <= kMost ? W : 0;
  *smem = (int)bytes(W);
}

// NSA_ERR_UNSUPPORTED (without a message) where the compressed logits do not fit beside this form's staging areas
template <typename T, typename State>
static int launch_decode_state(const DecodeParams& P, cudaStream_t stream) {
  int S, W, smem;
  decode_split<T, State>(P, &S, &W, &smem);
  if (W == 0) return NSA_ERR_UNSUPPORTED;
  auto kern = decode_kernel<T, State>;
  cudaError_t err = allow_shared_memory<decode_kernel<T, State>>();
  if (err != cudaSuccess) return fail((int)err, cudaGetErrorString(err));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(P.batch * P.kv_heads * S));
  cfg.blockDim = dim3(W * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)S;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = P.chained ? 2 : 1;
  err = cudaLaunchKernelEx(&cfg, kern, P, S);
  if (err != cudaSuccess) return fail((int)err, cudaGetErrorString(err));
  count_launches(1);
  return NSA_OK;
}

// bf16 with head sizes of 64 and 128 runs on the tensor instructions, everything else on the CUDA cores.  Every CTA holds
// the logits of all compressed blocks; where they leave no room for staging areas of 16 rows (from 300 000 cached tokens on,
// by type, group and head size), tiles of 4 rows on the CUDA cores take their place: slower per tile, but the step is served
// up to 230 KB of logits.
template <typename T, int GT>
static int launch_decode_gt(const DecodeParams& P, cudaStream_t stream) {
  int rc = NSA_ERR_UNSUPPORTED;
  if constexpr (sizeof(T) == 2) {   // the tensor form works on eight heads in any case
    if (P.d == 64) rc = launch_decode_state<T, TensorState<64, GT < 8 ? 8 : GT>>(P, stream);
    else if (P.d == 128) rc = launch_decode_state<T, TensorState<128, GT < 8 ? 8 : GT>>(P, stream);
    else rc = launch_decode_state<T, ScalarState<T, GT>>(P, stream);
  } else {
    rc = launch_decode_state<T, ScalarState<T, GT>>(P, stream);
  }
  if (rc == NSA_ERR_UNSUPPORTED) rc = launch_decode_state<T, ScalarState<T, GT, kLongTile>>(P, stream);
  return rc == NSA_ERR_UNSUPPORTED ? fail(rc, "decode step: too many compressed blocks for one CTA's shared memory") : rc;
}

template <typename T>
static int launch_decode_t(const DecodeParams& P, cudaStream_t stream) {
  const int G = P.q_heads / P.kv_heads;
  if (G == 1) return launch_decode_gt<T, 1>(P, stream);
  if (G == 2) return launch_decode_gt<T, 2>(P, stream);
  if (G <= 4) return launch_decode_gt<T, 4>(P, stream);
  if (G <= 8) return launch_decode_gt<T, 8>(P, stream);
  if (G <= 16) return launch_decode_gt<T, 16>(P, stream);
  return fail(NSA_ERR_UNSUPPORTED, "decode step: more than 16 query heads per KV head");
}

int launch_decode(const DecodeParams& P, int dtype, cudaStream_t stream) {
  if (P.batch == 0) return NSA_OK;
  return dtype == NSA_F32 ? launch_decode_t<float>(P, stream) : launch_decode_t<__nv_bfloat16>(P, stream);
}

// ---- a cache that cannot grow where it is ------------------------------------------------------------------------
//
// Keys and values in one launch, 16 bytes per access and four of them in flight per thread.  Bound: HBM.  As two tensor
// copies (strided, 2 bytes per access) the 134 MB of 4 x 32768 rows of 2 heads of 128 made a pass of 8 steps 568 us, so 453,
// what it takes without any copy; 16 steps at 300 rows 505 -> 479.
__global__ void __launch_bounds__(256) cache_copy_kernel(const CacheCopy P) {
  const int which = blockIdx.z;
  for (int head = blockIdx.y; head < P.heads; head += gridDim.y) {
    const uint4* src = static_cast<const uint4*>(P.src[which]) + head * P.src_step;
    uint4* dst = static_cast<uint4*>(P.dst[which]) + head * P.dst_step;
    for (int64_t i = (int64_t)blockIdx.x * 1024 + threadIdx.x; i < P.pieces; i += (int64_t)gridDim.x * 1024) {
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i + u * 256 < P.pieces) v[u] = src[i + u * 256];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i + u * 256 < P.pieces) dst[i + u * 256] = v[u];
    }
  }
}

int launch_cache_copy(const CacheCopy& P, cudaStream_t stream) {
  if (P.pieces == 0 || P.heads == 0) return NSA_OK;
  if (!aligned16(P.src[0], P.src[1], P.dst[0], P.dst[1])) return fail(NSA_ERR_ALIGN, "cache copy: rows must start on 16-byte boundaries");
  const int64_t chunks = (P.pieces + 1023) / 1024, most = 148 * 16 / (2 * (int64_t)P.heads) + 1;   // about 16 blocks per SM in all
  const dim3 grid((unsigned)(chunks < most ? chunks : most), (unsigned)(P.heads < 65535 ? P.heads : 65535), 2);
  cache_copy_kernel<<<grid, 256, 0, stream>>>(P);
  count_launches(1);
  const cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? NSA_OK : fail((int)err, cudaGetErrorString(err));
}

// ---- the projections of a step ---------------------------------------------------------------------------------
//
// y = norm(x) W^T for up to 16 token rows x, and behind the rows of W the gates: sigmoid(norm(x) Wg^T + bg); also the two
// layers of the compress networks when a window has filled up, keys and values side by side.
// Bound: the weights, read once.  bf16: a CTA owns 16 rows of W and requests all of them with cp.async before it
// normalises the token rows, then its warps share K (m16n8k16 products, fp32 accumulators) and add their parts in order.
// `chained` 1: the first kernel of a step, which may be scheduled before the kernel in front of it has ended but does nothing
// until then; 2: the last one, behind the attention, which fetches its weights meanwhile (nothing in the step writes them, and
// what came before the step was complete before the attention could start).
// fp32: a warp owns a pair of rows and uses CUDA cores.  Beside a library GEMM, which serves more than 16 rows, the results
// agree as two orders of the same fp32 sum do.

constexpr int kProjWarps = 8;
constexpr int kProjRows = 16;

template <typename T>
__device__ __forceinline__ T gate_of(float logit) {   // the logit rounded as a tensor of that type would hold it
  return Elem<T>::from_float(1.f / (1.f + expf(-Elem<T>::to_float(Elem<T>::from_float(logit)))));
}

// Rows to shared memory, `stride` elements apart, normalised or shifted and rounded as the tensor between two operations
// would be; rows past the last are zero.
template <typename T>
__device__ __forceinline__ void load_rows(const ProjectParams& P, T* x_s, int stride, int rows, int warp, int warps, int lane) {
  constexpr int V = Elem<T>::kVec;
  const int set = blockIdx.y;
  for (int t = warp; t < rows; t += warps) {
    T* dst = x_s + t * stride;
    if (t >= P.rows) {
      for (int c = lane * V; c < P.dim; c += 32 * V) *reinterpret_cast<uint4*>(dst + c) = make_uint4(0u, 0u, 0u, 0u);
      continue;
    }
    const int b = t / P.heads, h = t - b * P.heads;
    const T* src = (const T*)P.x[set] + b * P.x_sb + h * P.x_sh;
    const T* extra = P.norm_w != nullptr ? (const T*)P.norm_w : P.add[set] != nullptr ? (const T*)P.add[set] + (int64_t)h * P.dim : nullptr;
    float rstd = 1.f;
    if (P.norm_w != nullptr) {
      float ss = 0.f;
      for (int c = lane * V; c < P.dim; c += 32 * V) {
        float x[V];
        Elem<T>::load_vec(src + c, x);
#pragma unroll
        for (int e = 0; e < V; ++e) ss += x[e] * x[e];
      }
      rstd = rsqrtf(warp_sum(ss) / (float)P.dim + P.eps);
    }
    for (int c = lane * V; c < P.dim; c += 32 * V) {
      if (extra == nullptr) {
        *reinterpret_cast<uint4*>(dst + c) = *reinterpret_cast<const uint4*>(src + c);
        continue;
      }
      float x[V], w[V];
      Elem<T>::load_vec(src + c, x);
      Elem<T>::load_vec(extra + c, w);
#pragma unroll
      for (int e = 0; e < V; ++e) x[e] = P.norm_w != nullptr ? x[e] * rstd * w[e] : x[e] + w[e];
      store_vec<T>(dst + c, x);
    }
  }
}

// One finished value: row t, feature f of the set's projection, or of the gates
template <typename T>
__device__ __forceinline__ void emit(const ProjectParams& P, bool gates, int t, int f, float v) {
  const int set = blockIdx.y;
  if (gates) {
    ((T*)P.gates)[(int64_t)t * P.gates_n + f] = gate_of<T>(v + Elem<T>::to_float(((const T*)P.gate_b)[f]));
    return;
  }
  if (P.bias[set] != nullptr) v += Elem<T>::to_float(((const T*)P.bias[set])[f]);
  if (P.relu) v = fmaxf(v, 0.f);
  const int b = t / P.heads, h = t - b * P.heads;
  ((T*)P.y[set])[b * P.y_sb + h * P.y_sh + f] = Elem<T>::from_float(v);
}

template <int NT>   // groups of eight tokens
__global__ void __launch_bounds__(kProjWarps * 32) project_bf16_kernel(const ProjectParams P) {
  using T = __nv_bfloat16;
  if (P.chained != 2) ptx::grid_wait();
  ptx::grid_allow_next();
  extern __shared__ __align__(16) uint8_t proj_smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int stride = P.dim + 8;                    // elements; 16 bytes of padding keep ldmatrix free of conflicts
  T* const w_s = reinterpret_cast<T*>(proj_smem);
  T* const x_s = w_s + kProjRows * stride;
  const int feature_blocks = (P.features + kProjRows - 1) / kProjRows;
  const bool gates = (int)blockIdx.x >= feature_blocks;
  if (gates && blockIdx.y != 0) return;
  const int f0 = ((int)blockIdx.x - (gates ? feature_blocks : 0)) * kProjRows, end = gates ? P.gates_n : P.features;
  const T* w = (const T*)(gates ? P.gate_w : P.w[blockIdx.y]);
  const int pieces = P.dim / 8;
  for (int c0 = 0; c0 < pieces; c0 += 64) {        // by columns, so that the first of them arrive first
    const int n = min(64, pieces - c0);
    for (int e = tid; e < kProjRows * 64; e += kProjWarps * 32) {
      const int r = e / 64, c = e % 64;
      if (c < n)
        ptx::cp_async16(ptx::smem_u32(w_s + r * stride + (c0 + c) * 8), w + (int64_t)min(f0 + r, end - 1) * P.dim + (c0 + c) * 8, 16u);
    }
  }
  ptx::cp_async_commit();
  if (P.chained == 2) ptx::grid_wait();
  load_rows<T>(P, x_s, stride, 8 * NT, warp, kProjWarps, lane);
  ptx::cp_async_wait<0>();
  __syncthreads();
  float acc[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
  const uint32_t a_at = ptx::smem_u32(w_s + (lane & 15) * stride + (lane >> 4) * 8);
  const T* const b_at = x_s + (lane / 4) * stride + 2 * (lane & 3);
  const int k_end = P.dim / 16 * (warp + 1) / kProjWarps * 16;
#pragma unroll 4
  for (int k = P.dim / 16 * warp / kProjWarps * 16; k < k_end; k += 16) {
    uint32_t a[4];
    ldmatrix4<false>(a, a_at + k * 2);
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const T* src = b_at + 8 * n * stride + k;
      mma_16816(acc[n], a, *reinterpret_cast<const uint32_t*>(src), *reinterpret_cast<const uint32_t*>(src + 8));
    }
  }
  // the warps' parts of the sum, in their order
  __syncthreads();                                 // (over the weights)
  float* const part = reinterpret_cast<float*>(proj_smem);
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) part[(warp * NT * 4 + n * 4 + e) * 32 + lane] = acc[n][e];
  __syncthreads();
  if (tid >= NT * 128) return;
  const int n = tid / 128, e = tid / 32 % 4;
  float v = 0.f;
#pragma unroll
  for (int w = 0; w < kProjWarps; ++w) v += part[w * NT * 128 + tid];
  const int f = f0 + lane / 4 + (e / 2) * 8, t = 8 * n + 2 * (lane & 3) + (e & 1);
  if (f < end && t < P.rows) emit<T>(P, gates, t, f, v);
}

// fp32: the weights come from the L2 or from memory, so a lane requests four 16-byte pieces of either row at a time, the
// first of them before the token rows are ready.
template <int BT>
__global__ void __launch_bounds__(kProjWarps * 32) project_f32_kernel(const ProjectParams P) {
  constexpr int kAhead = BT <= 4 ? 4 : 2, kStep = kAhead * 128;
  extern __shared__ __align__(16) uint8_t proj_smem[];
  float* const x_s = reinterpret_cast<float*>(proj_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int feature_pairs = (P.features + 1) / 2, pairs = feature_pairs + (blockIdx.y == 0 ? (P.gates_n + 1) / 2 : 0);
  float4 a[kAhead], b[kAhead];
  const float *w0 = nullptr, *w1 = nullptr;
  auto aim = [&](int p) {
    const bool gates = p >= feature_pairs;
    const int f = 2 * (gates ? p - feature_pairs : p);
    w0 = (const float*)(gates ? P.gate_w : P.w[blockIdx.y]) + (int64_t)f * P.dim;
    w1 = f + 1 < (gates ? P.gates_n : P.features) ? w0 + P.dim : w0;
  };
  auto fetch = [&](int c0) {
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int c = c0 + (u * 32 + lane) * 4;
      a[u] = c < P.dim ? *reinterpret_cast<const float4*>(w0 + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      b[u] = c < P.dim ? *reinterpret_cast<const float4*>(w1 + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  const int first = blockIdx.x * kProjWarps + warp;
  if (P.chained != 2) ptx::grid_wait();
  ptx::grid_allow_next();
  if (first < pairs) {
    aim(first);
    fetch(0);
  }
  if (P.chained == 2) ptx::grid_wait();
  load_rows<float>(P, x_s, P.dim, BT, warp, kProjWarps, lane);
  __syncthreads();
  for (int p = first; p < pairs; p += gridDim.x * kProjWarps) {
    if (p != first) {
      aim(p);
      fetch(0);
    }
    float acc[2][BT];
#pragma unroll
    for (int t = 0; t < BT; ++t) acc[0][t] = acc[1][t] = 0.f;
    for (int c0 = 0; c0 < P.dim; c0 += kStep) {
      float4 ca[kAhead], cb[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) { ca[u] = a[u]; cb[u] = b[u]; }
      if (c0 + kStep < P.dim) fetch(c0 + kStep);
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int c = c0 + (u * 32 + lane) * 4;
        if (c >= P.dim) break;
#pragma unroll
        for (int t = 0; t < BT; ++t) {
          const float4 x = *reinterpret_cast<const float4*>(x_s + t * P.dim + c);
          acc[0][t] = fmaf(ca[u].w, x.w, fmaf(ca[u].z, x.z, fmaf(ca[u].y, x.y, fmaf(ca[u].x, x.x, acc[0][t]))));
          acc[1][t] = fmaf(cb[u].w, x.w, fmaf(cb[u].z, x.z, fmaf(cb[u].y, x.y, fmaf(cb[u].x, x.x, acc[1][t]))));
        }
      }
    }
    const bool gates = p >= feature_pairs;
    const int f = 2 * (gates ? p - feature_pairs : p), n = gates ? P.gates_n : P.features;
#pragma unroll
    for (int t = 0; t < BT; ++t) {
      const float y0 = warp_sum(acc[0][t]), y1 = warp_sum(acc[1][t]);
      if (lane != t || t >= P.rows) continue;
      emit<float>(P, gates, t, f, y0);
      if (f + 1 < n) emit<float>(P, gates, t, f + 1, y1);
    }
  }
}

// Shared memory of the kernel that would run, or 0 where none serves: more than 16 tokens (a GEMM then reuses every
// weight row often enough), or rows that do not fit.
static int project_smem(int batch, int dim, int dtype) {
  if (batch > 16 || dim % 16) return 0;
  const int tokens = batch <= 8 ? 8 : 16;
  const int64_t parts = kProjWarps * kProjRows * tokens * 4;      // bf16: the warps' sums, over the weights
  const int64_t rows = (int64_t)(kProjRows + tokens) * (dim + 8) * 2;
  const int64_t need = dtype == NSA_F32 ? (int64_t)(batch <= 1 ? 1 : batch <= 4 ? 4 : 16) * dim * 4 : rows > parts ? rows : parts;
  return need <= 220 * 1024 ? (int)need : 0;
}

bool project_serves(int batch, int dim, int dtype) { return project_smem(batch, dim, dtype) > 0; }

template <auto Kernel>
static int launch_project_with(const ProjectParams& P, int blocks, int smem, cudaStream_t stream) {
  cudaError_t err = allow_shared_memory<Kernel>();
  if (err == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks, (unsigned)P.sets);
    cfg.blockDim = dim3(kProjWarps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = P.chained ? 1 : 0;
    err = cudaLaunchKernelEx(&cfg, Kernel, P);
    count_launches(1);
  }
  return err == cudaSuccess ? NSA_OK : fail((int)err, cudaGetErrorString(err));
}

int launch_project(const ProjectParams& P, int dtype, cudaStream_t stream) {
  const int smem = project_smem(P.rows, P.dim, dtype);
  if (P.rows == 0) return NSA_OK;
  if (smem == 0) return fail(NSA_ERR_UNSUPPORTED, "projection of token rows: too many or too long");
  const int V = dtype == NSA_F32 ? 4 : 8;   // (only the first `sets` of the pairs are given; the others are NULL)
  if (!aligned16(P.x[0], P.x[1], P.w[0], P.w[1], P.add[0], P.add[1], P.norm_w, P.gate_w) || P.x_sb % V || P.x_sh % V)
    return fail(NSA_ERR_ALIGN, "projection of token rows: rows and weights must start on 16-byte boundaries");
  if (dtype == NSA_F32) {
    const int pairs = (P.features + 1) / 2 + (P.gates_n + 1) / 2, blocks = min((pairs + kProjWarps - 1) / kProjWarps, 148 * 4);
    if (P.rows <= 1) return launch_project_with<project_f32_kernel<1>>(P, blocks, smem, stream);
    if (P.rows <= 4) return launch_project_with<project_f32_kernel<4>>(P, blocks, smem, stream);
    return launch_project_with<project_f32_kernel<16>>(P, blocks, smem, stream);
  }
  const int blocks = (P.features + kProjRows - 1) / kProjRows + (P.gates_n + kProjRows - 1) / kProjRows;
  if (P.rows <= 8) return launch_project_with<project_bf16_kernel<1>>(P, blocks, smem, stream);
  return launch_project_with<project_bf16_kernel<2>>(P, blocks, smem, stream);
}

}  // namespace nsa
