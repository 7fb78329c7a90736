// Small and fp32 matrix products of a layer step, several of them per launch, on tcgen05.
//
// A training step has some twenty products between its attention kernels.  As library calls each costs 12 to 17 us of host
// time (heuristics, the call, one or two launches), which is what bounds a step of a thousand tokens whatever the GPU needs;
// here the products of the backward that do not depend on one another share a launch, four in all, with the ReLU mask and the
// column sums of the bias gradient in the same pass.  Whole steps: 2 x 31 fp32, dim 512 612 -> 481 us; 4 x 512 fp32, dim 512
// 1509 -> 1286; 1 x 1024 bf16, dim 256 648 -> 590.
// fp32 products run as bf16 ones: every operand is split into three bf16 terms (together its 24 bits) and the six products
// of terms that reach fp32's last bits are summed.  The library's fp32 kernels use the CUDA cores, an eighth of what the
// tensor cores reach with six products.
//
// A CTA computes a tile of 128 x BN.  Eight (fp32: sixteen) warps bring the operands in K steps of 64 into a ring of stages: bf16 by
// cp.async, fp32 through registers (the next step's loads stand before the split of the present one).  Another warp issues
// the products.  What bounds it: operands out of the L2, 24 (fp32 48 to 64) KB per step and tile.
// Accuracy in fp32: tensor cores do not round their sums to nearest, so long sums lose bits in one direction.  The leading
// products of a slice of K therefore have an accumulator of their own, the five small ones another, and the epilogue adds
// them in fp32.
#include <string.h>

#include <type_traits>

#include "nsa_common.cuh"
#include "nsa_kernels.h"
#include "nsa_sm100_ptx.cuh"

namespace nsa {

using namespace ptx;

namespace gemm {
constexpr int kBM = 128, kBK = 64, kMaxSplit = 8;

template <typename T, int BN>
struct Shape {
  static constexpr int kLoaders = sizeof(T) == 4 ? 512 : 256, kThreads = kLoaders + 32;
  static constexpr int kOwn = kBM * BN / kLoaders;                                // columns of the tile a thread of the epilogue has
  static constexpr int kTerms = sizeof(T) == 4 ? 3 : 1;
  static constexpr int kStages = sizeof(T) == 4 ? 2 : 4;
  static constexpr uint32_t kPlaneA = kBM * 128, kPlaneB = BN * 128;              // one bf16 term of an operand tile
  static constexpr uint32_t kStage = kTerms * (kPlaneA + kPlaneB);
  static constexpr uint32_t kBytes = kStages * kStage + 1024;
  static constexpr int kSlices = sizeof(T) == 4 ? 512 / BN - 1 : 1;               // accumulators for the leading products
  static constexpr uint32_t kCols = sizeof(T) == 4 ? 512 : BN;
};

// Eight consecutive elements of an operand, in memory order; `count` of them exist
template <typename T>
struct Piece;
template <>
struct Piece<float> {
  float x[8];
  __device__ __forceinline__ void load(const float* p, int count, int vec) {
    if (vec == 16 && count >= 8) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
      x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
      x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = i < count ? __ldg(p + i) : 0.f;
    }
  }
};

// x = h + m + l, each term rounded to bf16; the remainders are exact.  False where h is not finite (the terms would give
// NaN for an infinite product, or for a value that rounds to infinity).
__device__ __forceinline__ bool split3(const float (&x)[8], uint32_t (&h)[4], uint32_t (&m)[4], uint32_t (&l)[4]) {
  bool finite = true;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float a = x[2 * i], b = x[2 * i + 1];
    finite = finite && fabsf(a) < 3.38e38f && fabsf(b) < 3.38e38f;
    h[i] = pack_bf16(a, b);
    a -= __uint_as_float(h[i] << 16);
    b -= __uint_as_float(h[i] & 0xffff0000u);
    m[i] = pack_bf16(a, b);
    a -= __uint_as_float(m[i] << 16);
    b -= __uint_as_float(m[i] & 0xffff0000u);
    l[i] = pack_bf16(a, b);
  }
  return finite;
}

// Where the pieces of an operand tile lie: ROWS values of the M / N index, 64 of K.  K-major: memory rows are the M / N
// index, pieces run along K; else memory rows are K and pieces run along M / N (64 of them per swizzled block).
struct Operand {
  const void* p;
  int64_t ld;
  int rows, k;        // extents that exist, from the tile's first row / column on
  bool mn;            // M / N index contiguous in memory
  int vec;            // bytes that one access may move: 16, 4 or an element
};
template <int ROWS>
__device__ __forceinline__ void locate(const Operand& o, int e, int k0, int64_t& at, int& count, uint32_t& off) {
  if (o.mn) {
    const int kr = e / (ROWS / 8), c = e % (ROWS / 8);
    at = (int64_t)(k0 + kr) * o.ld + c * 8;
    count = k0 + kr < o.k ? o.rows - c * 8 : 0;
    off = (c / 8) * 8192 + sw128_offset(kr, c % 8);
  } else {
    const int r = e / 8, c = e % 8;
    at = (int64_t)r * o.ld + k0 + c * 8;
    count = r < o.rows ? o.k - k0 - c * 8 : 0;
    off = sw128_offset(r, c);
  }
}

template <int ROWS, int LOADERS>
__device__ __forceinline__ void fetch(const Operand& o, int k0, int tid, Piece<float> (&v)[ROWS * 8 / LOADERS]) {
#pragma unroll
  for (int i = 0; i < ROWS * 8 / LOADERS; ++i) {
    int64_t at;
    int count;
    uint32_t off;
    locate<ROWS>(o, tid + i * LOADERS, k0, at, count, off);
    v[i].load(static_cast<const float*>(o.p) + at, count, o.vec);
  }
}
template <int ROWS, int LOADERS>
__device__ __forceinline__ bool put(const Operand& o, uint32_t tile, int tid, const Piece<float> (&v)[ROWS * 8 / LOADERS]) {
  bool finite = true;
#pragma unroll
  for (int i = 0; i < ROWS * 8 / LOADERS; ++i) {
    int64_t at;
    int count;
    uint32_t off, h[4], m[4], l[4];
    locate<ROWS>(o, tid + i * LOADERS, 0, at, count, off);
    finite = split3(v[i].x, h, m, l) && finite;
    sts_v4(tile + off, make_uint4(h[0], h[1], h[2], h[3]));
    sts_v4(tile + ROWS * 128 + off, make_uint4(m[0], m[1], m[2], m[3]));
    sts_v4(tile + 2 * ROWS * 128 + off, make_uint4(l[0], l[1], l[2], l[3]));
  }
  return finite;
}
template <int ROWS, int LOADERS>
__device__ __forceinline__ void copy(const Operand& o, uint32_t tile, int k0, int tid) {
#pragma unroll
  for (int i = 0; i < ROWS * 8 / LOADERS; ++i) {
    int64_t at;
    int count;
    uint32_t off;
    locate<ROWS>(o, tid + i * LOADERS, k0, at, count, off);
    const uint16_t* src = static_cast<const uint16_t*>(o.p) + at;
    if (count <= 0) {
      sts_v4(tile + off, make_uint4(0u, 0u, 0u, 0u));
    } else if (o.vec == 16 && count >= 8) {
      cp_async16(tile + off, src, 16u);
    } else if (o.vec >= 4 && count % 2 == 0) {
#pragma unroll
      for (int x = 0; x < 4; ++x) cp_async4(tile + off + x * 4, 2 * x < count ? src + 2 * x : src, 2 * x < count ? 4u : 0u);
    } else {
      uint32_t w[4];
#pragma unroll
      for (int x = 0; x < 4; ++x)
        w[x] = (2 * x < count ? (uint32_t)__ldg(src + 2 * x) : 0u) | (2 * x + 1 < count ? (uint32_t)__ldg(src + 2 * x + 1) << 16 : 0u);
      sts_v4(tile + off, make_uint4(w[0], w[1], w[2], w[3]));
    }
  }
}

struct Bars {
  uint64_t full[4], empty[4], done;
};

// The accumulator that takes the leading products of a step
template <typename T, int BN>
__device__ __forceinline__ int slice_of(int step, int steps) {
  constexpr int N = Shape<T, BN>::kSlices;
  return N == 1 ? 0 : step * N / steps;
}
__device__ __forceinline__ void tmem_ld_cols(uint32_t at, float (&v)[32]) { tmem_ld32(at, v); }
__device__ __forceinline__ void tmem_ld_cols(uint32_t at, float (&v)[16]) { tmem_ld16(at, v); }
}  // namespace gemm

template <typename T, int BN>
__global__ void __launch_bounds__((gemm::Shape<T, BN>::kThreads), sizeof(T) == 4 ? 1 : 2) gemm_kernel(const __grid_constant__ GemmGroup group) {
  using namespace gemm;
  using S = Shape<T, BN>;
  constexpr bool F32 = sizeof(T) == 4;
  constexpr int kStages = S::kStages, kLoaders = S::kLoaders, kOwn = S::kOwn;
  extern __shared__ uint8_t gemm_smem[];
  __shared__ __align__(8) Bars bars;
  __shared__ int abort_flag, odd_input;
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t base = (smem_u32(gemm_smem) + 1023u) & ~1023u;

  // A cluster belongs to one task: to one tile of it, whose K steps its CTAs share, or to as many tiles as it has CTAs
  int which = 0;
  while (which + 1 < group.tasks && (int)blockIdx.x >= group.task[which + 1].first_cta) ++which;
  const GemmTask& task = group.task[which];
  const int split = task.split, rank = split > 1 ? (int)cluster_rank() : 0;
  const int tile = ((int)blockIdx.x - task.first_cta) / split, tiles_n = (task.n + BN - 1) / BN;
  const int m0 = tile / tiles_n * kBM, n0 = tile % tiles_n * BN;
  if (m0 >= task.m) return;                 // padding behind the last tile of a task that is not split
  const bool a_mn = task.op == kGemmTN, b_mn = task.op != kGemmNT;
  const int steps0 = (task.k[0] + kBK - 1) / kBK, all_steps = steps0 + (task.k[1] + kBK - 1) / kBK;
  const int first = (int)((int64_t)all_steps * rank / split), steps = (int)((int64_t)all_steps * (rank + 1) / split) - first;

  if (tid == 0) {
    abort_flag = 0;
    odd_input = 0;
    for (int i = 0; i < kStages; ++i) {
      mbar_init(smem_u32(&bars.full[i]), kLoaders);
      mbar_init(smem_u32(&bars.empty[i]), 1);
    }
    mbar_init(smem_u32(&bars.done), 1);
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(&tmem_slot), S::kCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tm = tmem_slot;

  if (tid < kLoaders) {
    // ------------------------------------------------------------------ operands
    auto operand = [&](bool second, int seg) {
      const int64_t el = sizeof(T);
      const bool mn = second ? b_mn : a_mn;
      const int64_t ld = second ? task.ldb[seg] : task.lda[seg], from = second ? n0 : m0;
      const char* p = static_cast<const char*>(second ? task.b[seg] : task.a[seg]) + (mn ? from : from * ld) * el;
      const uintptr_t odd = reinterpret_cast<uintptr_t>(p) | (uintptr_t)(ld * el);
      return Operand{p, ld, (int)((second ? task.n : task.m) - from), task.k[seg], mn, odd % 16 == 0 ? 16 : odd % 4 == 0 ? 4 : 2};
    };
    int seg = first < steps0 ? 0 : 1, k0 = (seg == 0 ? first : first - steps0) * kBK;    // of the step that is requested next
    Operand A = operand(false, seg), B = operand(true, seg);
    auto advance = [&]() {
      k0 += kBK;
      if (k0 >= task.k[seg] && seg == 0 && task.k[1] > 0) {
        seg = 1;
        k0 = 0;
        A = operand(false, 1);
        B = operand(true, 1);
      }
    };
    auto wait_free = [&](int step) {
      if (step >= kStages) mbar_wait_warp(smem_u32(&bars.empty[step % kStages]), (uint32_t)(step / kStages - 1) & 1, &abort_flag);
    };
    if constexpr (F32) {
      bool finite = true;
      Piece<float> a[2][kBM * 8 / kLoaders], b[2][BN * 8 / kLoaders];
      const Operand shape_a = A, shape_b = B;   // the places in shared memory depend on the layout only
      if (steps > 0) {
        fetch<kBM, kLoaders>(A, k0, tid, a[0]);
        fetch<BN, kLoaders>(B, k0, tid, b[0]);
      }
      for (int step0 = 0; step0 < steps; step0 += 2) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int step = step0 + u;
          if (step < steps) {
            if (step + 1 < steps) {
              advance();
              fetch<kBM, kLoaders>(A, k0, tid, a[u ^ 1]);
              fetch<BN, kLoaders>(B, k0, tid, b[u ^ 1]);
            }
            wait_free(step);
            const uint32_t at = base + (step % kStages) * S::kStage;
            finite = put<kBM, kLoaders>(shape_a, at, tid, a[u]) && finite;
            finite = put<BN, kLoaders>(shape_b, at + 3 * S::kPlaneA, tid, b[u]) && finite;
            fence_proxy_async_smem();
            mbar_arrive(smem_u32(&bars.full[step % kStages]));
          }
        }
      }
      if (!finite) odd_input = 1;
    } else {
      constexpr int kAhead = kStages - 1;
      for (int step = 0; step < steps + kAhead; ++step) {
        if (step < steps) {
          wait_free(step);
          const uint32_t at = base + (step % kStages) * S::kStage;
          copy<kBM, kLoaders>(A, at, k0, tid);
          copy<BN, kLoaders>(B, at + S::kPlaneA, k0, tid);
          advance();
        }
        cp_async_commit();
        if (step >= kAhead) {
          cp_async_wait<kAhead>();
          fence_proxy_async_smem();
          mbar_arrive(smem_u32(&bars.full[(step - kAhead) % kStages]));
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ products
    const uint32_t idesc = instr_desc_bf16(kBM, BN, a_mn, b_mn);
    const uint32_t step_a = a_mn ? 2048 : 32, step_b = b_mn ? 2048 : 32;
    int slice = -1;
    for (int step = 0; step < steps; ++step) {
      const int stage = step % kStages;
      mbar_wait_bounded(smem_u32(&bars.full[stage]), (uint32_t)(step / kStages) & 1, &abort_flag);
      __syncwarp();
      tc_fence_after_sync();
      const uint32_t at = base + stage * S::kStage;
      const uint64_t dA = smem_desc_sw128(at, 8192), dB = smem_desc_sw128(at + S::kTerms * S::kPlaneA, 8192);
      const int now = slice_of<T, BN>(step, steps);
      const bool fresh = now != slice;
      slice = now;
#pragma unroll
      for (int k = 0; k < kBK / 16; ++k) {
        const uint64_t ak = desc_advance(dA, k * step_a), bk = desc_advance(dB, k * step_b);
        mma_bf16_elect(tm + slice * BN, ak, bk, idesc, !fresh || k > 0);
        if constexpr (F32) {
          const uint32_t tR = tm + S::kSlices * BN;
          const uint64_t a1 = desc_advance(ak, S::kPlaneA), a2 = desc_advance(ak, 2 * S::kPlaneA);
          const uint64_t b1 = desc_advance(bk, S::kPlaneB), b2 = desc_advance(bk, 2 * S::kPlaneB);
          mma_bf16_elect(tR, ak, b2, idesc, step > 0 || k > 0);
          mma_bf16_elect(tR, a2, bk, idesc, true);
          mma_bf16_elect(tR, a1, b1, idesc, true);
          mma_bf16_elect(tR, ak, b1, idesc, true);
          mma_bf16_elect(tR, a1, bk, idesc, true);
        }
      }
      mma_commit_elect(smem_u32(&bars.empty[stage]));
    }
    mma_commit_elect(smem_u32(&bars.done));
    mbar_wait_drain(smem_u32(&bars.done), 0);
  }
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();                          // every product is complete, the flags are set
  tc_fence_after_sync();

  // ------------------------------------------------------------------ epilogue
  // what comes behind the sum, and the store, for V neighbouring columns of a row
  auto finish = [&](int row, int col, auto& v) {
    constexpr int V = sizeof(v) / sizeof(float);
    const bool whole = V * sizeof(T) % 8 == 0 && task.c_vec && col + V <= task.n;
    const int64_t at = (int64_t)row * task.n + col;
    if (task.act != nullptr) {
      const T* act = static_cast<const T*>(task.act) + at;
#pragma unroll
      for (int x = 0; x < V; ++x)
        if (col + x < task.n && !(Elem<T>::to_float(act[x]) > 0.f)) v[x] = 0.f;
    }
    T* out = static_cast<T*>(task.c) + at;
    T w[V];
#pragma unroll
    for (int x = 0; x < V; ++x) {
      w[x] = Elem<T>::from_float(v[x]);
      v[x] = Elem<T>::to_float(w[x]);
    }
    if (whole) {
      using Store = typename std::conditional<sizeof(T) * V % 16 == 0, uint4, uint2>::type;
#pragma unroll
      for (int x = 0; x < (int)(sizeof(w) / sizeof(Store)); ++x) {
        Store raw;
        memcpy(&raw, reinterpret_cast<const char*>(w) + x * sizeof(Store), sizeof(Store));
        reinterpret_cast<Store*>(out)[x] = raw;
      }
    } else {
#pragma unroll
      for (int x = 0; x < V; ++x)
        if (col + x < task.n) out[x] = w[x];
    }
  };

  // The sum of this CTA's steps: a thread has a row and kOwn columns
  const int own_row = (warp & 3) * 32 + lane, own_col = (warp >> 2) * kOwn;
  float v[kOwn];
  if (tid < kLoaders) {
    const uint32_t tm_lane = tm + ((uint32_t)((warp & 3) * 32) << 16) + own_col;
#pragma unroll
    for (int x = 0; x < kOwn; ++x) v[x] = 0.f;
    if (steps > 0) {
      tmem_ld_cols(tm_lane + (F32 ? S::kSlices * BN : 0), v);
      tmem_ld_wait();
      if constexpr (F32) {
        int seen = -1;
#pragma unroll 1
        for (int step = 0; step < steps; ++step) {
          const int slice = slice_of<T, BN>(step, steps);
          if (slice == seen) continue;
          seen = slice;
          float t[kOwn];
          tmem_ld_cols(tm_lane + slice * BN, t);
          tmem_ld_wait();
#pragma unroll
          for (int x = 0; x < kOwn; ++x) v[x] += t[x];
        }
      }
    }
    const int row = m0 + own_row, col = n0 + own_col;
    if (F32 && odd_input != 0 && row < task.m) {
      // an operand of the tile is infinite, NaN or next to overflow: in fp32 steps, as IEEE has it
#pragma unroll 1
      for (int x = 0; x < kOwn; ++x) {
        float s = 0.f;
        if (col + x < task.n)
          for (int g = 0; g < 2; ++g) {
            const float* a = static_cast<const float*>(task.a[g]) + (a_mn ? row : (int64_t)row * task.lda[g]);
            const float* b = static_cast<const float*>(task.b[g]) + (b_mn ? col + x : (int64_t)(col + x) * task.ldb[g]);
            const int64_t sa = a_mn ? task.lda[g] : 1, sb = b_mn ? task.ldb[g] : 1;
            // this CTA's steps of the part
            const int from = min(max(first - (g == 0 ? 0 : steps0), 0) * kBK, task.k[g]);
            const int to = min(max(first + steps - (g == 0 ? 0 : steps0), 0) * kBK, task.k[g]);
            for (int k = from; k < to; ++k) s = fmaf(a[k * sa], b[k * sb], s);
          }
#pragma unroll
        for (int y = 0; y < kOwn; ++y)
          if (y == x) v[y] = s;
      }
    }
    if (split == 1) {
      if (row < task.m) finish(row, col, v);
      if (task.sums != nullptr) {
        // column sums of what was stored: every step folds lanes, and halves the columns a lane holds while it can
#pragma unroll
        for (int x = 0; x < kOwn; ++x) v[x] = row < task.m && col + x < task.n ? v[x] : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          if (o >= kOwn) {
#pragma unroll
            for (int x = 0; x < kOwn; ++x) v[x] += __shfl_xor_sync(kFullMask, v[x], o);
          } else {
            const bool up = lane & o;
#pragma unroll
            for (int x = 0; x < o; ++x) {
              const float mine = up ? v[x + o] : v[x], other = up ? v[x] : v[x + o];
              v[x] = mine + __shfl_xor_sync(kFullMask, other, o);
            }
          }
        }
        if (lane < kOwn && col + lane < task.n) atomicAdd(task.sums + col + lane, v[0]);
      }
    }
  }
  if (split > 1) {
    // The CTAs of the tile meet: CTA r finishes columns r BN / split ...; every one sends it its sums, [source][column][row]
    // in the staging area, and they are added in the order of the CTAs.
    __syncwarp();
    cluster_arrive();                       // nobody's products read the staging area any more
    cluster_wait();
    const int share = BN / split;
    if (tid < kLoaders) {
#pragma unroll
      for (int x = 0; x < kOwn; ++x) {
        const int owner = (own_col + x) / share, c = own_col + x - owner * share;
        st_cluster(map_rank(base, owner) + (uint32_t)(((rank * share + c) * kBM + own_row) * 4), v[x]);
      }
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    for (int e = tid; e < kBM * share / 4; e += S::kThreads) {
      const int r = e % kBM, c = e / kBM * 4;
      float s[4] = {0.f, 0.f, 0.f, 0.f};
      for (int from = 0; from < split; ++from)
#pragma unroll
        for (int x = 0; x < 4; ++x) s[x] += __uint_as_float(lds_u32(base + (uint32_t)(((from * share + c + x) * kBM + r) * 4)));
      if (m0 + r < task.m) finish(m0 + r, n0 + rank * share + c, s);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, S::kCols);
  if (tid == 0 && abort_flag && group.status != nullptr) atomicOr(group.status, 1);
}

static int64_t steps_of(const GemmTask& t) { return ((int64_t)t.k[0] + gemm::kBK - 1) / gemm::kBK + ((int64_t)t.k[1] + gemm::kBK - 1) / gemm::kBK; }
static int64_t tiles_of(const GemmTask& t, int cols) { return (int64_t)((t.m + gemm::kBM - 1) / gemm::kBM) * ((t.n + cols - 1) / cols); }
// K steps that fp32 accumulators can take.  Up to ten steps (640 products) per accumulator of the leading products the result
// is nearer to the exact one than fp32 steps are (relative 2-norm, normal operands: K 2048 6.5e-7 against the library's 8.1e-7
// with three accumulators, 2.7e-7 with seven; K 512 1.7e-7 against 4.1e-7); twice as many and it is not (K 4096 1.4e-6 against
// 1.1e-6).  Longer sums are split over the CTAs of a cluster.
static int most_steps(int cols) { return cols == 64 ? 70 : 32; }

// How a group is cut: columns of a tile, CTAs per cluster, and the K steps from which on a task's tiles are shared by a cluster
struct GemmCut {
  int cols, split, from;
  int of(const GemmTask& t) const { return t.sums == nullptr && steps_of(t) >= from ? split : 1; }
};
static GemmCut gemm_cut(const GemmGroup& G, int dtype) {
  int64_t wide = 0, longest = 0;
  for (int t = 0; t < G.tasks; ++t) {
    wide += tiles_of(G.task[t], 128);
    if (steps_of(G.task[t]) > longest) longest = steps_of(G.task[t]);
  }
  // 128 columns halve what the rows cost, as long as such tiles still fill the chip: 2 x [1024 x 1024 x 1024] 45 us, with 64
  // columns 55; but 2048 x 512 x 1024 and its weight gradients, 100 wide tiles, 55 with 64 columns, 82 with 128
  GemmCut cut = {dtype == NSA_F32 && wide >= 128 && longest <= (int64_t)most_steps(128) * gemm::kMaxSplit ? 128 : 64, 1, 1 << 30};
  if (G.cols != 0) cut.cols = dtype == NSA_F32 ? G.cols : 64;
  if (dtype == NSA_F32) {   // what the accumulators need
    cut.from = most_steps(cut.cols) + 1;
    while (cut.split < gemm::kMaxSplit && longest > (int64_t)most_steps(cut.cols) * cut.split) cut.split *= 2;
  }
  // and while the chip has room for it and every CTA keeps two steps (62 x 1536 x 512 24 -> 19 us, 62 rows of the backward's
  // last products 48 -> 28)
  for (int s = cut.split * 2; s <= gemm::kMaxSplit && longest >= 2 * s; s *= 2) {
    const GemmCut more = {cut.cols, s, 2 * s};
    int64_t ctas = 0;
    for (int t = 0; t < G.tasks; ++t) ctas += tiles_of(G.task[t], cut.cols) * more.of(G.task[t]);
    if (ctas > 148) break;
    cut = more;
  }
  if (G.split != 0) cut = {cut.cols, G.split, 2 * G.split};
  return cut;
}

template <typename T, int BN>
static int launch_gemm_as(GemmGroup& G, const GemmCut& cut, cudaStream_t stream) {
  const int split = cut.split;
  int64_t ctas = 0;
  for (int t = 0; t < G.tasks; ++t) {
    GemmTask& k = G.task[t];
    k.split = cut.of(k);
    k.first_cta = (int)ctas;
    ctas += (tiles_of(k, BN) * k.split + split - 1) / split * split;
    if (ctas > 0x7fffffff) return fail(NSA_ERR_SHAPE, "layer: a matrix product with too many tiles for one launch");
  }
  if (ctas == 0) return NSA_OK;
  cudaError_t err = allow_shared_memory<gemm_kernel<T, BN>>();
  if (err == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(gemm::Shape<T, BN>::kThreads);
    cfg.dynamicSmemBytes = gemm::Shape<T, BN>::kBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)split;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    err = cudaLaunchKernelEx(&cfg, gemm_kernel<T, BN>, G);
    count_launches(1);
  }
  return err == cudaSuccess ? NSA_OK : fail((int)err, cudaGetErrorString(err));
}

bool gemm_serves(const GemmGroup& G, int dtype) {
  for (int t = 0; t < G.tasks; ++t)
    if (dtype == NSA_F32 && steps_of(G.task[t]) > (int64_t)most_steps(64) * (G.task[t].sums == nullptr ? gemm::kMaxSplit : 1)) return false;
  return true;
}

int launch_gemm(GemmGroup& G, int dtype, cudaStream_t stream) {
  if (!gemm_serves(G, dtype)) return fail(NSA_ERR_UNSUPPORTED, "layer: a sum too long for the accumulators of a matrix product");
  for (int t = 0; t < G.tasks; ++t) G.task[t].c_vec = aligned16(G.task[t].c) && (int64_t)G.task[t].n * (dtype == NSA_F32 ? 4 : 2) % 16 == 0;
  const GemmCut cut = gemm_cut(G, dtype);
  if (dtype != NSA_F32) return launch_gemm_as<__nv_bfloat16, 64>(G, cut, stream);
  return cut.cols == 128 ? launch_gemm_as<float, 128>(G, cut, stream) : launch_gemm_as<float, 64>(G, cut, stream);
}

}  // namespace nsa
