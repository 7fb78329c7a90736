// Generic CUDA-core kernels for the three NSA attention branches.
//
// One warp serves one (batch, head group, query) task and all query heads of
// the group, so every fetched key/value row is shared by the group (GQA).
// In the compressed and the sliding branch, where neighbours see nearly the
// same keys, the queries of a block also share staged tiles of 32 keys, unless
// they see few (see shares_tiles).
// The keys of a task are runs of consecutive positions:
//   selected branch  : one run per visible slot + the own-block run
//   compressed branch: the memory slots and the visible compressed blocks
//   sliding branch   : the window around the query
// Inside a run, lanes map to keys for the two dot products (q.k and do.v) and
// to feature pairs for the accumulations (p.v, ds.k, ds.q, p.do); values move
// between the two mappings with warp shuffles.  All arithmetic is fp32, which
// is what lets this family meet a 1e-4 relative bound on fp32 inputs; it also
// serves every shape the tensor-core family does not cover.

#include "nsa_common.cuh"
#include "nsa_kernels.h"
#include "nsa_sm100_ptx.cuh"

namespace nsa {

constexpr int kWarpsPerBlock = 4;

// Stages the G query rows (or upstream-gradient rows) of a task as fp32.
template <typename T, int GT>
__device__ __forceinline__ void stage_rows(float* dst, const T* src, int64_t head_stride, int G, int d, int lane) {
  for (int e = lane * 2; e < GT * d; e += 64) {
    const int g = e / d, c = e - g * d;
    float2 val = make_float2(0.f, 0.f);
    if (g < G) val = Elem<T>::load2(src + g * head_stride + c);
    dst[e] = val.x;
    dst[e + 1] = val.y;
  }
}

// s[g] += sum_c rows[g][c] * key[c] for this lane's key row.
template <typename T, int GT>
__device__ __forceinline__ void dot_rows(float (&s)[GT], const float* rows, const T* key, int d) {
  constexpr int V = Elem<T>::kVec;
  for (int c = 0; c < d; c += V) {
    float kv[V];
    Elem<T>::load_vec(key + c, kv);
#pragma unroll
    for (int g = 0; g < GT; ++g) {
      const float* r = rows + g * d + c;
#pragma unroll
      for (int e = 0; e < V; e += 4) {
        const float4 qv = *reinterpret_cast<const float4*>(r + e);
        s[g] = fmaf(qv.x, kv[e], s[g]);
        s[g] = fmaf(qv.y, kv[e + 1], s[g]);
        s[g] = fmaf(qv.z, kv[e + 2], s[g]);
        s[g] = fmaf(qv.w, kv[e + 3], s[g]);
      }
    }
  }
}

// The keys of query i in the compressed and the sliding branch: rows first .. first + total - 1 (compressed: the memory slots, then the visible blocks)
template <int BR>
struct KeyRange {
  int first, total;
  __device__ __forceinline__ KeyRange(const AttnParams& P, int i) {
    if (BR == BR_CMP) {
      first = 0;
      total = P.num_mem + (P.causal ? min(P.ncb, i / P.stride) : P.ncb);
    } else {
      first = max(0, i - P.window);
      total = (P.causal ? i + 1 : min(P.seq, i + P.window + 1)) - first;
    }
  }
};

// The runs of one task.  get(r) yields [start, end) in key-row units.  Selected branch: slot s is run s, the own block is run nsel;
// `uniform`: the query sees no key at all (all logits equal, no gradient to q and k).  The other two: one run.
struct Run {
  int start, end;
  int slot;  // slot index, or -1
};

template <int BR>
struct TaskRuns {
  int count;
  bool uniform;
  int total_keys; // number of keys when uniform
  __device__ __forceinline__ void init(const AttnParams& P, int b, int grp, int i) {
    if (BR != BR_SEL) {
      count = 1;
      uniform = false;
      total_keys = 0;
      return;
    }
    count = P.nsel + (P.diag != NSA_DIAG_NONE ? 1 : 0);
    bool any = P.diag != NSA_DIAG_NONE;
    const int nfb = (P.seq + P.block - 1) / P.block;
    const int64_t base = (((int64_t)b * P.groups + grp) * P.seq + i) * P.nsel;
    int in_range = 0;
    for (int s = 0; s < P.nsel; ++s) {
      const int64_t blk = P.idx[base + s];
      const bool ok = blk >= 0 && blk < nfb;
      in_range += ok ? 1 : 0;
      any = any || (ok && P.mask[base + s] != 0);
    }
    uniform = !any;
    total_keys = in_range * P.block;
  }
  __device__ __forceinline__ Run get(const AttnParams& P, int b, int grp, int i, int r) const {
    Run run;
    run.slot = -1;
    if (BR != BR_SEL) {
      const KeyRange<BR> keys(P, i);
      run.start = keys.first;
      run.end = keys.first + keys.total;
    } else if (r < P.nsel) {
      const int nfb = (P.seq + P.block - 1) / P.block;
      const int64_t base = (((int64_t)b * P.groups + grp) * P.seq + i) * P.nsel;
      const int64_t blk = P.idx[base + r];
      const bool ok = blk >= 0 && blk < nfb && (uniform || P.mask[base + r] != 0);
      run.start = ok ? (int)blk * P.block : 0;
      run.end = ok ? run.start + P.block : 0;
      run.slot = r;
    } else {
      const int own = i / P.block * P.block;
      run.start = own;
      run.end = P.diag == NSA_DIAG_CAUSAL ? i + 1 : own + P.block;
    }
    return run;
  }
};

template <typename T, int GT, int BR>
__global__ void __launch_bounds__(kWarpsPerBlock * 32) attend_query_fwd_kernel(const AttnParams P) {
  extern __shared__ __align__(16) float smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t task = (int64_t)blockIdx.x * kWarpsPerBlock + warp;
  const int64_t ntasks = (int64_t)P.batch * P.groups * P.seq;
  if (task >= ntasks) return;
  const int i = (int)(task % P.seq);
  const int grp = (int)((task / P.seq) % P.groups);
  const int b = (int)(task / ((int64_t)P.seq * P.groups));
  const int G = P.q_heads / P.groups;
  const int kvh = grp / (P.groups / P.kv_heads);
  const int d = P.d;
  float* q_s = smem + warp * GT * d;

  const T* qp = (const T*)P.q + b * P.q_sb + (int64_t)(grp * G) * P.q_sh + (int64_t)i * P.q_sn;
  stage_rows<T, GT>(q_s, qp, P.q_sh, G, d, lane);
  __syncwarp();
  const T* kb = (const T*)P.k + b * P.k_sb + (int64_t)kvh * P.k_sh;
  const T* vb = (const T*)P.v + b * P.v_sb + (int64_t)kvh * P.v_sh;

  float m[GT], l[GT], acc[GT][2][2];
#pragma unroll
  for (int g = 0; g < GT; ++g) {
    m[g] = -INFINITY;
    l[g] = 0.f;
    acc[g][0][0] = acc[g][0][1] = acc[g][1][0] = acc[g][1][1] = 0.f;
  }

  TaskRuns<BR> runs;
  runs.init(P, b, grp, i);
  for (int r = 0; r < runs.count; ++r) {
    const Run run = runs.get(P, b, grp, i, r);
    for (int t0 = run.start; t0 < run.end; t0 += 32) {
      const int pos = t0 + lane;
      const bool present = pos < run.end;
      const bool real = present && pos < P.key_rows;  // rows past the end are zero keys
      float s[GT];
#pragma unroll
      for (int g = 0; g < GT; ++g) s[g] = 0.f;
      if (real && !runs.uniform) dot_rows<T, GT>(s, q_s, kb + (int64_t)pos * P.k_sn, d);
#pragma unroll
      for (int g = 0; g < GT; ++g) s[g] *= P.scale;
      float p[GT];
#pragma unroll
      for (int g = 0; g < GT; ++g) {
        const float tile_max = warp_max(present ? s[g] : -INFINITY);
        const float m_new = fmaxf(m[g], tile_max);
        const float alpha = exp2f((m[g] - m_new) * kLog2e);
        p[g] = present ? exp2f((s[g] - m_new) * kLog2e) : 0.f;
        l[g] = l[g] * alpha + warp_sum(p[g]);
        m[g] = m_new;
        acc[g][0][0] *= alpha; acc[g][0][1] *= alpha;
        acc[g][1][0] *= alpha; acc[g][1][1] *= alpha;
      }
      const int cnt = min(32, min(run.end, P.key_rows) - t0);
      for (int kk = 0; kk < cnt; ++kk) {
        const T* vrow = vb + (int64_t)(t0 + kk) * P.v_sn;
        float2 vv[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int dim = 64 * c + 2 * lane;
          vv[c] = dim < d ? Elem<T>::load2(vrow + dim) : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int g = 0; g < GT; ++g) {
          const float pg = __shfl_sync(kFullMask, p[g], kk);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            acc[g][c][0] = fmaf(pg, vv[c].x, acc[g][c][0]);
            acc[g][c][1] = fmaf(pg, vv[c].y, acc[g][c][1]);
          }
        }
      }
    }
  }

  T* op = (T*)P.out + b * P.o_sb + (int64_t)(grp * G) * P.o_sh + (int64_t)i * P.o_sn;
#pragma unroll
  for (int g = 0; g < GT; ++g) {
    if (g >= G) break;
    const float inv = l[g] > 0.f ? 1.f / l[g] : 0.f;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int dim = 64 * c + 2 * lane;
      if (dim < d) Elem<T>::store2(op + g * P.o_sh + dim, acc[g][c][0] * inv, acc[g][c][1] * inv);
    }
    if (lane == 0)
      P.lse[((int64_t)b * P.q_heads + grp * G + g) * P.seq + i] = l[g] > 0.f ? m[g] + logf(l[g]) : -INFINITY;
  }
}

template <typename T, int GT, int BR>
__global__ void __launch_bounds__(kWarpsPerBlock * 32) attend_query_bwd_kernel(const AttnParams P) {
  extern __shared__ __align__(16) float smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t task = (int64_t)blockIdx.x * kWarpsPerBlock + warp;
  const int64_t ntasks = (int64_t)P.batch * P.groups * P.seq;
  if (task >= ntasks) return;
  const int i = (int)(task % P.seq);
  const int grp = (int)((task / P.seq) % P.groups);
  const int b = (int)(task / ((int64_t)P.seq * P.groups));
  const int G = P.q_heads / P.groups;
  const int kvh = grp / (P.groups / P.kv_heads);
  const int d = P.d;
  float* q_s = smem + warp * 2 * GT * d;
  float* do_s = q_s + GT * d;

  const T* qp = (const T*)P.q + b * P.q_sb + (int64_t)(grp * G) * P.q_sh + (int64_t)i * P.q_sn;
  const T* dop = (const T*)P.dout + b * P.do_sb + (int64_t)(grp * G) * P.do_sh + (int64_t)i * P.do_sn;
  const T* op = (const T*)P.out + b * P.o_sb + (int64_t)(grp * G) * P.o_sh + (int64_t)i * P.o_sn;
  stage_rows<T, GT>(q_s, qp, P.q_sh, G, d, lane);
  stage_rows<T, GT>(do_s, dop, P.do_sh, G, d, lane);
  __syncwarp();
  const T* kb = (const T*)P.k + b * P.k_sb + (int64_t)kvh * P.k_sh;
  const T* vb = (const T*)P.v + b * P.v_sb + (int64_t)kvh * P.v_sh;
  float* dkb = P.dk + ((int64_t)b * P.kv_heads + kvh) * P.key_rows * d;
  float* dvb = P.dv + ((int64_t)b * P.kv_heads + kvh) * P.key_rows * d;

  float lse[GT], delta[GT], dq[GT][2][2];
#pragma unroll
  for (int g = 0; g < GT; ++g) {
    float part = 0.f;
    if (g < G) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int dim = 64 * c + 2 * lane;
        if (dim < d) {
          const float2 o = Elem<T>::load2(op + g * P.o_sh + dim);
          part += o.x * do_s[g * d + dim] + o.y * do_s[g * d + dim + 1];
        }
      }
    }
    delta[g] = warp_sum(part);
    lse[g] = g < G ? P.lse[((int64_t)b * P.q_heads + grp * G + g) * P.seq + i] : 0.f;
    dq[g][0][0] = dq[g][0][1] = dq[g][1][0] = dq[g][1][1] = 0.f;
  }

  TaskRuns<BR> runs;
  runs.init(P, b, grp, i);
  const float p_uniform = runs.total_keys > 0 ? 1.f / (float)runs.total_keys : 0.f;
  for (int r = 0; r < runs.count; ++r) {
    const Run run = runs.get(P, b, grp, i, r);
    float slot_part = 0.f;
    for (int t0 = run.start; t0 < run.end; t0 += 32) {
      const int pos = t0 + lane;
      const bool present = pos < run.end;
      const bool real = present && pos < P.key_rows;
      float s[GT], dp[GT], p[GT], ds[GT];
#pragma unroll
      for (int g = 0; g < GT; ++g) s[g] = dp[g] = 0.f;
      if (real) {
        if (!runs.uniform) dot_rows<T, GT>(s, q_s, kb + (int64_t)pos * P.k_sn, d);
        dot_rows<T, GT>(dp, do_s, vb + (int64_t)pos * P.v_sn, d);
      }
#pragma unroll
      for (int g = 0; g < GT; ++g) {
        s[g] *= P.scale;
        if (runs.uniform) {
          p[g] = present ? p_uniform : 0.f;
          ds[g] = 0.f;
        } else {
          p[g] = (present && g < G) ? exp2f((s[g] - lse[g]) * kLog2e) : 0.f;
          ds[g] = p[g] * (dp[g] - delta[g]);
          slot_part += ds[g] * s[g];
          ds[g] *= P.scale;
        }
      }
      const int cnt = min(32, min(run.end, P.key_rows) - t0);
      for (int kk = 0; kk < cnt; ++kk) {
        const int64_t row = t0 + kk;
        const T* krow = kb + row * P.k_sn;
        float2 kv[2], gk[2], gv[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int dim = 64 * c + 2 * lane;
          kv[c] = dim < d ? Elem<T>::load2(krow + dim) : make_float2(0.f, 0.f);
          gk[c] = gv[c] = make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int g = 0; g < GT; ++g) {
          const float dsg = __shfl_sync(kFullMask, ds[g], kk);
          const float pg = __shfl_sync(kFullMask, p[g], kk);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int dim = 64 * c + 2 * lane;
            if (dim < d) {
              dq[g][c][0] = fmaf(dsg, kv[c].x, dq[g][c][0]);
              dq[g][c][1] = fmaf(dsg, kv[c].y, dq[g][c][1]);
              const float2 qv = *reinterpret_cast<const float2*>(q_s + g * d + dim);
              const float2 dv = *reinterpret_cast<const float2*>(do_s + g * d + dim);
              gk[c].x = fmaf(dsg, qv.x, gk[c].x);
              gk[c].y = fmaf(dsg, qv.y, gk[c].y);
              gv[c].x = fmaf(pg, dv.x, gv[c].x);
              gv[c].y = fmaf(pg, dv.y, gv[c].y);
            }
          }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int dim = 64 * c + 2 * lane;
          if (dim < d) {
            if (!runs.uniform) atomicAdd(reinterpret_cast<float2*>(dkb + row * d + dim), gk[c]);
            atomicAdd(reinterpret_cast<float2*>(dvb + row * d + dim), gv[c]);
          }
        }
      }
    }
    if (BR == BR_SEL && P.slot_grads != nullptr && run.slot >= 0) {
      const float total = warp_sum(slot_part);
      if (lane == 0)
        P.slot_grads[(((int64_t)b * P.groups + grp) * P.seq + i) * P.nsel + run.slot] = total;
    }
  }

  float* dqp = P.dq + (((int64_t)b * P.q_heads + grp * G) * P.seq + i) * d;
#pragma unroll
  for (int g = 0; g < GT; ++g) {
    if (g >= G) break;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int dim = 64 * c + 2 * lane;
      if (dim < d)
        *reinterpret_cast<float2*>(dqp + (int64_t)g * P.seq * d + dim) = make_float2(dq[g][c][0], dq[g][c][1]);
    }
  }
}

// ---- compressed and sliding branch ------------------------------------------------
//
// Neighbouring queries attend nearly the same keys: a block takes several queries of one (batch, head group), a warp each, and
// walks the union of their keys in tiles of 32 that it stages once, whole rows per access.  In the backward the warps leave P
// and dS of a tile in shared memory; then every warp sums dk and dv of its share of the tile's keys over all rows and adds
// them once: one reduction per key and block instead of one per key and query.
// Bound: issue slots and shared memory are busy half of the time each (51 to 55 and 41 to 45 % in the forward, 45 to 48 and 53 to 55 % in the
// backward), a third of the warps is resident and waits for the one or the other.  4 x 512 positions, 8 / 4 heads of 64 in fp32,
// forward and backward in us, against a warp per query that fetches its keys alone: sliding window of 32
// 37 + 85 -> 31 + 52, 64 compressed blocks 50 + 96 -> 33 + 49; 4 x 1024, 8 heads, 512 compressed blocks 826 + 1691 -> 423 + 610.
// Rows of a tile lie 16 bytes further apart than they are long: neighbours fall on other banks.
template <typename T>
__host__ __device__ __forceinline__ int tile_pitch(int d) { return d * (int)sizeof(T) + 16; }
// Requests rows t0 .. of k and v up to `end` (the rest of the 32 is zeroed), a share per warp of the block; one commit group.
template <typename T>
__device__ __forceinline__ void stage_tile(const AttnParams& P, const T* kb, const T* vb, int t0, int end, uint8_t* k_s, uint8_t* v_s, int warp,
                                           int warps, int lane) {
  const int pieces = P.d * (int)sizeof(T) / 16, pitch = tile_pitch<T>(P.d), rows = 32 / warps;
  for (int e = lane; e < 2 * rows * pieces; e += 32) {
    const int which = e / (rows * pieces), x = e - which * rows * pieces, r = warp * rows + x / pieces, c = x % pieces, row = t0 + r;
    const bool ok = row < end;
    const T* src = which == 0 ? kb + (ok ? (int64_t)row * P.k_sn : 0) : vb + (ok ? (int64_t)row * P.v_sn : 0);
    ptx::cp_async16(ptx::smem_u32(which == 0 ? k_s : v_s) + r * pitch + c * 16, src + c * (16 / (int)sizeof(T)), ok ? 16u : 0u);
  }
  ptx::cp_async_commit();
}

template <typename T, int GT>
struct DenseFwd {
  static constexpr int QB = 8;
  static int64_t smem(int d) { return QB * GT * d * 4 + 2 * 32 * tile_pitch<T>(d); }
};
template <typename T, int GT, int BR>
__global__ void __launch_bounds__(DenseFwd<T, GT>::QB * 32) attend_dense_fwd_kernel(const AttnParams P) {
  constexpr int QB = DenseFwd<T, GT>::QB;
  extern __shared__ __align__(16) uint8_t simt_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tiles = (P.seq + QB - 1) / QB;
  const int i0 = (int)(blockIdx.x % tiles) * QB, unit = blockIdx.x / tiles;
  const int grp = unit % P.groups, b = unit / P.groups, i = i0 + warp;
  const int G = P.q_heads / P.groups, kvh = grp / (P.groups / P.kv_heads);
  const int d = P.d, pitch = tile_pitch<T>(d);
  const bool valid = i < P.seq;
  const int iv = min(i, P.seq - 1);            // (a warp past the end works on the last query and keeps nothing)
  float* const q_s = reinterpret_cast<float*>(simt_smem) + warp * GT * d;
  uint8_t *const k_s = simt_smem + QB * GT * d * 4, *const v_s = k_s + 32 * pitch;
  const T* kb = (const T*)P.k + b * P.k_sb + (int64_t)kvh * P.k_sh;
  const T* vb = (const T*)P.v + b * P.v_sb + (int64_t)kvh * P.v_sh;
  const KeyRange<BR> keys(P, iv), front(P, i0), back(P, min(i0 + QB, P.seq) - 1);
  const int lo = keys.first, hi = keys.first + keys.total, end = back.first + back.total;
  stage_tile<T>(P, kb, vb, front.first, end, k_s, v_s, warp, QB, lane);
  stage_rows<T, GT>(q_s, (const T*)P.q + b * P.q_sb + (int64_t)(grp * G) * P.q_sh + (int64_t)iv * P.q_sn, P.q_sh, G, d, lane);

  float m[GT], l[GT], acc[GT][2][2];
#pragma unroll
  for (int g = 0; g < GT; ++g) {
    m[g] = -INFINITY;
    l[g] = 0.f;
    acc[g][0][0] = acc[g][0][1] = acc[g][1][0] = acc[g][1][1] = 0.f;
  }
  for (int t0 = front.first; t0 < end; t0 += 32) {
    if (t0 > front.first) {
      __syncthreads();                         // the tile before has been read
      stage_tile<T>(P, kb, vb, t0, end, k_s, v_s, warp, QB, lane);
    }
    ptx::cp_async_wait<0>();
    __syncthreads();
    if (hi <= t0 || lo >= t0 + 32) continue;   // (the same for the whole warp)
    const int row = t0 + lane;
    const bool present = row >= lo && row < hi;
    float s[GT];
#pragma unroll
    for (int g = 0; g < GT; ++g) s[g] = 0.f;
    if (present) dot_rows<T, GT>(s, q_s, reinterpret_cast<const T*>(k_s + lane * pitch), d);
    if (BR == BR_CMP && P.importance != nullptr && valid && present && row >= P.num_mem) {
      // the logit as upstream's tensor of that dtype would hold it
      const int w = row - P.num_mem;
      float logit[GT];
#pragma unroll
      for (int g = 0; g < GT; ++g)
        logit[g] = P.round_bf16 ? round_bf16(round_bf16(s[g]) * P.scale) : s[g] * P.scale;
      if (P.imp_heads == P.kv_heads) {
        float sum = 0.f;
#pragma unroll
        for (int g = 0; g < GT; ++g) sum += (g < G) ? logit[g] : 0.f;
        float mean = sum / (float)G;
        if (P.round_bf16) mean = round_bf16(mean);
        P.importance[(((int64_t)b * P.imp_heads + kvh) * P.seq + i) * P.ncb + w] = mean;
      } else {
#pragma unroll
        for (int g = 0; g < GT; ++g)
          if (g < G) P.importance[(((int64_t)b * P.imp_heads + kvh * G + g) * P.seq + i) * P.ncb + w] = logit[g];
      }
    }
    float p[GT];
#pragma unroll
    for (int g = 0; g < GT; ++g) {
      s[g] *= P.scale;
      const float m_new = fmaxf(m[g], warp_max(present ? s[g] : -INFINITY));
      const float alpha = exp2f((m[g] - m_new) * kLog2e);
      p[g] = present ? exp2f((s[g] - m_new) * kLog2e) : 0.f;
      l[g] = l[g] * alpha + warp_sum(p[g]);
      m[g] = m_new;
      acc[g][0][0] *= alpha; acc[g][0][1] *= alpha;
      acc[g][1][0] *= alpha; acc[g][1][1] *= alpha;
    }
    const int k0 = max(0, lo - t0), k1 = min(32, hi - t0);
#pragma unroll 4
    for (int kk = k0; kk < k1; ++kk) {
      const T* vrow = reinterpret_cast<const T*>(v_s + kk * pitch);
      float2 vv[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int dim = 64 * c + 2 * lane;
        vv[c] = dim < d ? Elem<T>::load2(vrow + dim) : make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int g = 0; g < GT; ++g) {
        const float pg = __shfl_sync(kFullMask, p[g], kk);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          acc[g][c][0] = fmaf(pg, vv[c].x, acc[g][c][0]);
          acc[g][c][1] = fmaf(pg, vv[c].y, acc[g][c][1]);
        }
      }
    }
  }
  if (!valid) return;

  if (BR == BR_CMP && P.importance != nullptr) {
    // columns the query cannot see carry the sentinel (its head mean, when shared)
    const int vis = P.causal ? min(P.ncb, i / P.stride) : P.ncb;
    float fill = P.sentinel;
    if (P.imp_heads == P.kv_heads) {
      float sum = 0.f;
      for (int g = 0; g < G; ++g) sum += P.sentinel;
      fill = sum / (float)G;
      if (P.round_bf16) fill = round_bf16(fill);
    }
    const int heads_here = P.imp_heads == P.kv_heads ? 1 : G;
    for (int hh = 0; hh < heads_here; ++hh) {
      const int ih = P.imp_heads == P.kv_heads ? kvh : kvh * G + hh;
      float* row = P.importance + (((int64_t)b * P.imp_heads + ih) * P.seq + i) * P.ncb;
      for (int w = vis + lane; w < P.ncb; w += 32) row[w] = fill;
    }
  }
  T* op = (T*)P.out + b * P.o_sb + (int64_t)(grp * G) * P.o_sh + (int64_t)i * P.o_sn;
#pragma unroll
  for (int g = 0; g < GT; ++g) {
    if (g >= G) break;
    const float inv = l[g] > 0.f ? 1.f / l[g] : 0.f;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int dim = 64 * c + 2 * lane;
      if (dim < d) Elem<T>::store2(op + g * P.o_sh + dim, acc[g][c][0] * inv, acc[g][c][1] * inv);
    }
    if (lane == 0)
      P.lse[((int64_t)b * P.q_heads + grp * G + g) * P.seq + i] = l[g] > 0.f ? m[g] + logf(l[g]) : -INFINITY;
  }
}

// The row sums of out * dout of the G heads of a query, and their log-sum-exp
template <typename T, int GT>
__device__ __forceinline__ void row_statistics(const AttnParams& P, const float* do_s, int b, int grp, int G, int i, int lane, float (&lse)[GT],
                                               float (&delta)[GT]) {
  const T* op = (const T*)P.out + b * P.o_sb + (int64_t)(grp * G) * P.o_sh + (int64_t)i * P.o_sn;
#pragma unroll
  for (int g = 0; g < GT; ++g) {
    float part = 0.f;
    if (g < G) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int dim = 64 * c + 2 * lane;
        if (dim < P.d) {
          const float2 o = Elem<T>::load2(op + g * P.o_sh + dim);
          part += o.x * do_s[g * P.d + dim] + o.y * do_s[g * P.d + dim + 1];
        }
      }
    }
    delta[g] = warp_sum(part);
    lse[g] = g < G ? P.lse[((int64_t)b * P.q_heads + grp * G + g) * P.seq + i] : 0.f;
  }
}
template <int GT>
__device__ __forceinline__ void store_dq(const AttnParams& P, const float (&dq)[GT][2][2], int b, int grp, int G, int i, int lane) {
  float* dqp = P.dq + (((int64_t)b * P.q_heads + grp * G) * P.seq + i) * P.d;
#pragma unroll
  for (int g = 0; g < GT; ++g) {
    if (g >= G) break;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int dim = 64 * c + 2 * lane;
      if (dim < P.d)
        *reinterpret_cast<float2*>(dqp + (int64_t)g * P.seq * P.d + dim) = make_float2(dq[g][c][0], dq[g][c][1]);
    }
  }
}

template <typename T, int GT>
struct DenseBwd {
  static constexpr int QB = GT <= 4 ? 8 : 32 / GT;          // 8, 8, 8, 4, 2 queries: at most 32 rows
  static constexpr int ROWS = QB * GT, KPW = 32 / QB;       // keys per warp
  static int64_t smem(int d) { return 2 * ROWS * d * 4 + 2 * ROWS * 32 * 4 + 2 * 32 * tile_pitch<T>(d); }
};
template <typename T, int GT, int BR>
__global__ void __launch_bounds__(DenseBwd<T, GT>::QB * 32) attend_dense_bwd_kernel(const AttnParams P) {
  using S = DenseBwd<T, GT>;
  constexpr int QB = S::QB, ROWS = S::ROWS, KPW = S::KPW;
  extern __shared__ __align__(16) uint8_t simt_smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tiles = (P.seq + QB - 1) / QB;
  const int i0 = (int)(blockIdx.x % tiles) * QB, unit = blockIdx.x / tiles;
  const int grp = unit % P.groups, b = unit / P.groups, i = i0 + warp;
  const int G = P.q_heads / P.groups, kvh = grp / (P.groups / P.kv_heads);
  const int d = P.d, pitch = tile_pitch<T>(d);
  const bool valid = i < P.seq;
  float* const q_s = reinterpret_cast<float*>(simt_smem);   // [QB * GT][d] each; row = query * GT + head
  float* const do_s = q_s + ROWS * d;
  float* const p_s = do_s + ROWS * d;                       // [rows][32] each
  float* const ds_s = p_s + ROWS * 32;
  uint8_t *const k_s = reinterpret_cast<uint8_t*>(ds_s + ROWS * 32), *const v_s = k_s + 32 * pitch;
  float *const q_w = q_s + warp * GT * d, *const do_w = do_s + warp * GT * d;

  const int iv = min(i, P.seq - 1);                         // (a warp past the end works on the last query and keeps nothing)
  const T* kb = (const T*)P.k + b * P.k_sb + (int64_t)kvh * P.k_sh;
  const T* vb = (const T*)P.v + b * P.v_sb + (int64_t)kvh * P.v_sh;
  const KeyRange<BR> keys(P, iv), front(P, i0), back(P, min(i0 + QB, P.seq) - 1);
  const int lo = keys.first, hi = keys.first + keys.total, end = back.first + back.total;
  stage_tile<T>(P, kb, vb, front.first, end, k_s, v_s, warp, QB, lane);
  stage_rows<T, GT>(q_w, (const T*)P.q + b * P.q_sb + (int64_t)(grp * G) * P.q_sh + (int64_t)iv * P.q_sn, P.q_sh, G, d, lane);
  stage_rows<T, GT>(do_w, (const T*)P.dout + b * P.do_sb + (int64_t)(grp * G) * P.do_sh + (int64_t)iv * P.do_sn, P.do_sh, G, d, lane);
  __syncwarp();
  float* dkb = P.dk + ((int64_t)b * P.kv_heads + kvh) * P.key_rows * d;
  float* dvb = P.dv + ((int64_t)b * P.kv_heads + kvh) * P.key_rows * d;
  float lse[GT], delta[GT], dq[GT][2][2];
  row_statistics<T, GT>(P, do_w, b, grp, G, iv, lane, lse, delta);
#pragma unroll
  for (int g = 0; g < GT; ++g) dq[g][0][0] = dq[g][0][1] = dq[g][1][0] = dq[g][1][1] = 0.f;

  // a row with infinities or NaN must not reach the keys it does not see through a product with zero
  bool finite = true;
  for (int e = lane; e < GT * d; e += 32) finite = finite && isfinite(q_w[e]) && isfinite(do_w[e]);
  const bool odd = __syncthreads_or(!finite) != 0;
  for (int t0 = front.first; t0 < end; t0 += 32) {
    if (t0 > front.first) {
      __syncthreads();                          // the tile before, and its P and dS, have been read
      stage_tile<T>(P, kb, vb, t0, end, k_s, v_s, warp, QB, lane);
    }
    ptx::cp_async_wait<0>();
    __syncthreads();
    const int row = t0 + lane;
    const bool sees = valid && row >= lo && row < hi;
    float s[GT], dp[GT], ds[GT];
#pragma unroll
    for (int g = 0; g < GT; ++g) s[g] = dp[g] = 0.f;
    if (__any_sync(kFullMask, sees)) {
      dot_rows<T, GT>(s, q_w, reinterpret_cast<const T*>(k_s + lane * pitch), d);
      dot_rows<T, GT>(dp, do_w, reinterpret_cast<const T*>(v_s + lane * pitch), d);
    }
#pragma unroll
    for (int g = 0; g < GT; ++g) {
      const float p = sees && g < G ? exp2f((s[g] * P.scale - lse[g]) * kLog2e) : 0.f;
      ds[g] = p * (dp[g] - delta[g]) * P.scale;
      if (!sees) ds[g] = 0.f;
      p_s[(warp * GT + g) * 32 + lane] = p;
      ds_s[(warp * GT + g) * 32 + lane] = ds[g];
    }
    __syncthreads();
    if (valid) {
      const int k0 = max(0, lo - t0), k1 = min(32, hi - t0);
#pragma unroll 2
      for (int kk = k0; kk < k1; ++kk) {
        const T* krow = reinterpret_cast<const T*>(k_s + kk * pitch);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int dim = 64 * c + 2 * lane;
          if (64 * c >= d) continue;
          const float2 kv = dim < d ? Elem<T>::load2(krow + dim) : make_float2(0.f, 0.f);
#pragma unroll
          for (int g = 0; g < GT; ++g) {
            const float dsg = ds_s[(warp * GT + g) * 32 + kk];
            dq[g][c][0] = fmaf(dsg, kv.x, dq[g][c][0]);
            dq[g][c][1] = fmaf(dsg, kv.y, dq[g][c][1]);
          }
        }
      }
    }
    // dk and dv of this warp's keys, summed over the rows of the block
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int dim = 64 * c + 2 * lane;
      if (64 * c >= d) continue;
      constexpr int PART = KPW < 4 ? KPW : 4;   // keys at a time
#pragma unroll 1
      for (int kk = warp * KPW; kk < (warp + 1) * KPW; kk += PART) {
        if (t0 + kk >= end) break;
        float2 gk[PART], gv[PART];
#pragma unroll
        for (int x = 0; x < PART; ++x) gk[x] = gv[x] = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int r = 0; r < ROWS; ++r) {
          const float2 qv = dim < d ? *reinterpret_cast<const float2*>(q_s + r * d + dim) : make_float2(0.f, 0.f);
          const float2 dv = dim < d ? *reinterpret_cast<const float2*>(do_s + r * d + dim) : make_float2(0.f, 0.f);
#pragma unroll
          for (int x = 0; x < PART; ++x) {
            const float dsr = ds_s[r * 32 + kk + x], pr = p_s[r * 32 + kk + x];
            if (odd && dsr == 0.f && pr == 0.f) continue;
            gk[x].x = fmaf(dsr, qv.x, gk[x].x);
            gk[x].y = fmaf(dsr, qv.y, gk[x].y);
            gv[x].x = fmaf(pr, dv.x, gv[x].x);
            gv[x].y = fmaf(pr, dv.y, gv[x].y);
          }
        }
#pragma unroll
        for (int x = 0; x < PART; ++x)
          if (t0 + kk + x < end && dim < d) {
            atomicAdd(reinterpret_cast<float2*>(dkb + (int64_t)(t0 + kk + x) * d + dim), gk[x]);
            atomicAdd(reinterpret_cast<float2*>(dvb + (int64_t)(t0 + kk + x) * d + dim), gv[x]);
          }
      }
    }
  }
  if (valid) store_dq<GT>(P, dq, b, grp, G, i, lane);
}

// ---- host side --------------------------------------------------------------

template <auto Kernel>
static int launch_with(const AttnParams& P, int64_t blocks, int threads, int64_t smem, cudaStream_t stream) {
  if (blocks == 0) return NSA_OK;
  if (blocks > 0x7fffffffLL) return fail(NSA_ERR_SHAPE, "too many (batch, head, query) tasks for one launch");
  cudaError_t err = smem > 48 * 1024 ? allow_shared_memory<Kernel>() : cudaSuccess;
  if (err == cudaSuccess) {
    Kernel<<<(unsigned)blocks, threads, (size_t)smem, stream>>>(P);
    count_launches(1);
    err = cudaGetLastError();
  }
  return err == cudaSuccess ? NSA_OK : fail((int)err, cudaGetErrorString(err));
}

// Whether the queries of a block share tiles, or a warp fetches the keys of its query alone (the selected branch always): by the
// most keys that a query sees, because a query of few shares little and a tile costs its staging whatever is seen of it, by the
// heads that share a fetched row anyway, and in the backward by dim_head (fewer queries in a block of 32 rows, and larger ones).
// Measured, the time alone over that with tiles (fp32 and bf16, 1 x 256 to 2 x 4096 positions).  Forward: up to four heads per KV head
// 0.8 to 0.96 with 3 to 9 keys, 1.0 to 1.2 with 11, 1.4 to 2 with 65; eight heads 0.8 to 1.0 up to 15 keys, 0.95 to 1.14 with 21;
// sixteen 0.96 to 1.1 from 11 on, but 0.85 to 1.0 where the blocks do not fill the GPU.  Backward: 0.75 to 0.9 with 3 keys, 0.9 to 1.0
// with 9 (sixteen heads 0.9 to 1.35), 1.0 to 1.3 with 11, 1.6 to 2 with 65; heads of 128, eight of them 0.85 to 1.0 up to 15 keys, 1.04
// to 1.2 with 21; sixteen 0.7 to 0.9 with 9 to 21, 1.0 to 1.2 with 25, with few blocks 0.95 to 1.2 with 11.  Compressed backward: 0.7 to 1.0
// with two keys, 1.0 to 1.3 with three; sixteen heads of 128 in many blocks 0.8 to 1.0 with five to nine; forward 1.0 to 2, but for
// 10 us against 13 with a single block and eight heads or more.
template <int BR>
static bool shares_tiles(const AttnParams& P, int heads, bool backward) {
  if (BR == BR_SEL) return false;
  const bool wide = P.d > 64, fills = (int64_t)P.batch * P.groups * P.seq >= 8 * 148;   // (blocks of eight queries, SMs)
  if (BR == BR_CMP) return !backward || P.num_mem + P.ncb >= (wide && heads > 8 && fills ? 12 : 3);
  const int64_t keys = (int64_t)P.window * (P.causal ? 1 : 2) + 1;
  if (!backward) return heads > 8 ? fills && keys >= 11 : keys >= (heads > 4 ? 20 : 11);
  if (wide && heads > 4) return keys >= (heads <= 8 ? 20 : fills ? 24 : 11);
  return keys >= (heads > 8 ? 9 : 11);
}

template <typename T, int GT, int BR>
static int launch_one(const AttnParams& P, bool backward, cudaStream_t stream) {
  if (!shares_tiles<BR>(P, GT, backward)) {
    const int64_t ntasks = (int64_t)P.batch * P.groups * P.seq, blocks = (ntasks + kWarpsPerBlock - 1) / kWarpsPerBlock;
    const int64_t smem = (int64_t)kWarpsPerBlock * GT * P.d * sizeof(float) * (backward ? 2 : 1);
    if (backward) return launch_with<attend_query_bwd_kernel<T, GT, BR>>(P, blocks, kWarpsPerBlock * 32, smem, stream);
    if constexpr (BR != BR_CMP) return launch_with<attend_query_fwd_kernel<T, GT, BR>>(P, blocks, kWarpsPerBlock * 32, smem, stream);
  }
  if constexpr (BR != BR_SEL) {
    const int queries = backward ? DenseBwd<T, GT>::QB : DenseFwd<T, GT>::QB;
    const int64_t blocks = (int64_t)P.batch * P.groups * ((P.seq + queries - 1) / queries);
    return backward ? launch_with<attend_dense_bwd_kernel<T, GT, BR>>(P, blocks, queries * 32, DenseBwd<T, GT>::smem(P.d), stream)
                    : launch_with<attend_dense_fwd_kernel<T, GT, BR>>(P, blocks, queries * 32, DenseFwd<T, GT>::smem(P.d), stream);
  }
  return NSA_OK;   // (not reached)
}

template <typename T, int BR>
static int launch_gt(const AttnParams& P, bool backward, cudaStream_t stream) {
  const int G = P.q_heads / P.groups;
  if (G <= 1) return launch_one<T, 1, BR>(P, backward, stream);
  if (G <= 2) return launch_one<T, 2, BR>(P, backward, stream);
  if (G <= 4) return launch_one<T, 4, BR>(P, backward, stream);
  if (G <= 8) return launch_one<T, 8, BR>(P, backward, stream);
  if (G <= 16) return launch_one<T, 16, BR>(P, backward, stream);
  return fail(NSA_ERR_UNSUPPORTED, "more than 16 query heads per group");
}

int simt_attend(const AttnParams& P, int branch, int dtype, bool backward, cudaStream_t stream) {
  if (dtype == NSA_F32) {
    if (branch == BR_SEL) return launch_gt<float, BR_SEL>(P, backward, stream);
    if (branch == BR_CMP) return launch_gt<float, BR_CMP>(P, backward, stream);
    return launch_gt<float, BR_SWA>(P, backward, stream);
  }
  if (branch == BR_SEL) return launch_gt<__nv_bfloat16, BR_SEL>(P, backward, stream);
  if (branch == BR_CMP) return launch_gt<__nv_bfloat16, BR_CMP>(P, backward, stream);
  return launch_gt<__nv_bfloat16, BR_SWA>(P, backward, stream);
}

}  // namespace nsa
