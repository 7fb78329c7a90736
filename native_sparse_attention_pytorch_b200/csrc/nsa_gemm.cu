// Small and fp32 matrix products of a layer step, several of them per launch, on tcgen05.
//
// A training step has some twenty products between its attention kernels.  As library calls each costs 12 to 17 us of host
// time (heuristics, the call, one or two launches), which is what bounds a step of a thousand tokens whatever the GPU needs;
// here the products of the backward that do not depend on one another share a launch, four in all, with the ReLU mask and the
// column sums of the bias gradient in the same pass.  On the GPU, against the library's launches one after the other: the last
// three products of a backward of 2048 rows, dim 512, fp32 50 us against 126; of 62 rows 18 against 42; of 1024 rows, dim 256, bf16
// 16 against 21.
// fp32 products run as bf16 ones: every operand is split into three bf16 terms (together its 24 bits) and the six products
// of terms that reach fp32's last bits are summed.  The library's fp32 kernels use the CUDA cores, an eighth of what the
// tensor cores reach with six products.
//
// A CTA computes a tile of 128 x BN.  Eight (fp32: sixteen) warps bring the operands in K steps of 64 into a ring of stages: bf16 by
// cp.async, fp32 through registers (an operand's loads for the next step stand behind the split of the present one; 16-byte
// pieces, whole memory rows per warp: with 32 bytes per thread every load takes twice the wavefronts).  Another warp issues
// the products.  What bounds it in fp32: the chain of a step (loads, split, products, sums) with two stages in flight; no unit
// is busy more than half of the time (3744 x 2048 x 2048 twice: shared memory 51 %, issue slots 44 %, tensor pipe 33 %, L2 17 %).
// In bf16, with few steps per SM, the launch and the latency of its few loads (issue slots 18 %, L2 7 %).
// Accuracy in fp32: tensor cores cut their sums instead of rounding them, so a sum of one sign loses about 2^-25 of itself with
// every product added to it.  An accumulator therefore takes the leading products of one K step (four), the loading threads add
// step after step in fp32 while the next ones run, and the small products of all steps have an accumulator of their own.
// Relative 2-norm of the error against 64 bits, operands in [0, 1), 2048 x 2048: K 512 8.6e-8 (library 3.1e-7), K 2048 1.1e-7
// (6.0e-7), K 15000 9.1e-8 (1.7e-6); 1024 x 512 with K 15000, which the library splits, 9.1e-8 (9.9e-8).  With a third of K per
// accumulator, added at the end, it was 2.2e-7, 1.2e-6 and 1.0e-6, and tiles of 128 columns took 15 % less time.
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
  // Tensor memory: bf16 one accumulator; fp32 three for the leading products of a step, in turn, and one for the small products
  static constexpr uint32_t tSmall = 3 * BN, kCols = (sizeof(T) == 4 ? 4 : 1) * BN;
};

// x = h + m + l, each term rounded to bf16; the remainders are exact.  Infinities and NaN are in h as they are, and m and l are
// NaN: the leading products are then what fp32 gives, the small ones are left out (see the epilogue).  A finite x that rounds to
// an infinite h (above 3.39e38) has an infinite m, which stays in `odd`.
__device__ __forceinline__ void split3(const float4& x, uint2& h, uint2& m, uint2& l, __nv_bfloat162& odd) {
  auto pair = [&](float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    hi = pack_bf16(a, b);
    a -= __uint_as_float(hi << 16);
    b -= __uint_as_float(hi & 0xffff0000u);
    mid = pack_bf16(a, b);
    a -= __uint_as_float(mid << 16);
    b -= __uint_as_float(mid & 0xffff0000u);
    lo = pack_bf16(a, b);
    odd = __hmax2(odd, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&mid)));      // (keeps the number beside a NaN)
  };
  pair(x.x, x.y, h.x, m.x, l.x);
  pair(x.z, x.w, h.y, m.y, l.y);
}

// An operand from a tile's first row / column on.  K-major: memory rows are the M / N index; else memory rows are K.
struct Operand {
  const void* p;
  int64_t ld;
  int rows, k;        // extents that exist
  bool mn;            // M / N index contiguous in memory
  int vec;            // bytes that one access may move: 16, 4 or an element
};
// The 16-byte pieces of an operand tile (ROWS x 64 of K) that a thread brings: memory rows `pass` apart, so that one address
// and one place in shared memory serve all of them.
template <typename T, int ROWS, int LOADERS>
struct Places {
  static constexpr int V = 16 / (int)sizeof(T), N = ROWS * kBK / (V * LOADERS);
  const T* p;
  int64_t step, hop;  // elements to the next K step and to the next piece
  int row, left, pass, rows;   // K-major: memory row, K values from the piece on; else K row, values of the M / N index from the piece on
  uint32_t off;
  bool mn;
  int vec;
  __device__ __forceinline__ Places(const Operand& o, int k0, int tid) : mn(o.mn), vec(o.vec) {
    const int per = (mn ? ROWS : kBK) / V, r = tid / per, c = tid % per * V;
    pass = LOADERS / per;
    hop = pass * o.ld;
    if (mn) {
      p = static_cast<const T*>(o.p) + (int64_t)(k0 + r) * o.ld + c;
      step = kBK * o.ld;
      row = k0 + r; rows = o.k; left = o.rows - c;
    } else {
      p = static_cast<const T*>(o.p) + (int64_t)r * o.ld + k0 + c;
      step = kBK;
      row = r; rows = o.rows; left = o.k - k0 - c;
    }
    off = (uint32_t)(c / 64) * 8192 + sw128_offset(r, c % 64 * 2 / sizeof(uint4)) + (c * 2) % 16;
  }
  __device__ __forceinline__ void next() {
    p += step;
    if (mn) row += kBK;
    else left -= kBK;
  }
  __device__ __forceinline__ int count(int i) const { return row + i * pass < rows ? left : 0; }   // (may be negative, or above V)
  __device__ __forceinline__ uint32_t place(int i) const { return off + i * pass * 128; }
};

template <int ROWS, int LOADERS, int N>
__device__ __forceinline__ void fetch(const Places<float, ROWS, LOADERS>& at, float4 (&v)[N]) {
  static_assert(N == Places<float, ROWS, LOADERS>::N, "");
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const float* p = at.p + i * at.hop;
    const int count = at.count(i);
    if (at.vec == 16 && count >= 4) {
      v[i] = __ldg(reinterpret_cast<const float4*>(p));
    } else {
      v[i].x = count > 0 ? __ldg(p) : 0.f;
      v[i].y = count > 1 ? __ldg(p + 1) : 0.f;
      v[i].z = count > 2 ? __ldg(p + 2) : 0.f;
      v[i].w = count > 3 ? __ldg(p + 3) : 0.f;
    }
  }
}
__device__ __forceinline__ void sts_v2(uint32_t addr, uint2 v) {
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(v.x), "r"(v.y) : "memory");
}
template <int ROWS, int LOADERS, int N>
__device__ __forceinline__ void put(const Places<float, ROWS, LOADERS>& at, uint32_t tile, const float4 (&v)[N], __nv_bfloat162& odd) {
#pragma unroll
  for (int i = 0; i < N; ++i) {
    uint2 h, m, l;
    split3(v[i], h, m, l, odd);
    const uint32_t dst = tile + at.place(i);
    sts_v2(dst, h);
    sts_v2(dst + ROWS * 128, m);
    sts_v2(dst + 2 * ROWS * 128, l);
  }
}
template <int ROWS, int LOADERS>
__device__ __forceinline__ void copy(const Places<__nv_bfloat16, ROWS, LOADERS>& at, uint32_t tile) {
#pragma unroll
  for (int i = 0; i < Places<__nv_bfloat16, ROWS, LOADERS>::N; ++i) {
    const uint16_t* src = reinterpret_cast<const uint16_t*>(at.p + i * at.hop);
    const int count = at.count(i);
    const uint32_t dst = tile + at.place(i);
    if (count <= 0) {
      sts_v4(dst, make_uint4(0u, 0u, 0u, 0u));
    } else if (at.vec == 16 && count >= 8) {
      cp_async16(dst, src, 16u);
    } else if (at.vec >= 4 && count % 2 == 0) {
#pragma unroll
      for (int x = 0; x < 4; ++x) cp_async4(dst + x * 4, 2 * x < count ? src + 2 * x : src, 2 * x < count ? 4u : 0u);
    } else {
      uint32_t w[4];
#pragma unroll
      for (int x = 0; x < 4; ++x)
        w[x] = (2 * x < count ? (uint32_t)__ldg(src + 2 * x) : 0u) | (2 * x + 1 < count ? (uint32_t)__ldg(src + 2 * x + 1) << 16 : 0u);
      sts_v4(dst, make_uint4(w[0], w[1], w[2], w[3]));
    }
  }
}

struct Bars {
  uint64_t full[4], empty[4], done;
};

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

  // The sum of this CTA's steps: a loading thread has a row and kOwn columns of the tile.  fp32: the leading products of a step
  const int own_row = (warp & 3) * 32 + lane, own_col = (warp >> 2) * kOwn;
  const uint32_t tm_own = tm + ((uint32_t)((warp & 3) * 32) << 16) + own_col;
  float v[kOwn];
#pragma unroll
  for (int x = 0; x < kOwn; ++x) v[x] = 0.f;
  auto fold = [&](int step) {
#pragma unroll
    for (int c = 0; c < kOwn; c += 8) {
      float t[8];
      tmem_ld8(tm_own + step % 3 * BN + c, t);
      tmem_ld_wait();
#pragma unroll
      for (int x = 0; x < 8; ++x) v[c + x] += t[x];
    }
  };

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
    Places<T, kBM, kLoaders> A(operand(false, seg), k0, tid);
    Places<T, BN, kLoaders> B(operand(true, seg), k0, tid);
    auto advance = [&]() {
      k0 += kBK;
      if (k0 >= task.k[seg] && seg == 0 && task.k[1] > 0) {
        seg = 1;
        k0 = 0;
        A = Places<T, kBM, kLoaders>(operand(false, 1), 0, tid);
        B = Places<T, BN, kLoaders>(operand(true, 1), 0, tid);
      } else {
        A.next();
        B.next();
      }
    };
    auto wait_free = [&](int step) {
      if (step >= kStages) mbar_wait_warp(smem_u32(&bars.empty[step % kStages]), (uint32_t)(step / kStages - 1) & 1, &abort_flag);
    };
    if constexpr (F32) {
      __nv_bfloat162 odd = __floats2bfloat162_rn(0.f, 0.f);
      float4 a[decltype(A)::N], b[decltype(B)::N];
      if (steps > 0) {
        fetch(A, a);
        fetch(B, b);
      }
      for (int step = 0; step < steps; ++step) {
        wait_free(step);
        const uint32_t at = base + (step % kStages) * S::kStage;   // (the places depend on the layout only, not on the part)
        put(A, at, a, odd);
        if (step + 1 < steps) {
          advance();
          fetch(A, a);
        }
        put(B, at + 3 * S::kPlaneA, b, odd);
        if (step + 1 < steps) fetch(B, b);
        fence_proxy_async_smem();
        mbar_arrive(smem_u32(&bars.full[step % kStages]));
        if (step >= 2) {        // (wait_free)
          tc_fence_after_sync();
          fold(step - 2);
          tc_fence_before_sync();
        }
      }
      if (__hisinf(odd.x) || __hisinf(odd.y)) odd_input = 1;
    } else {
      constexpr int kAhead = kStages - 1;
      for (int step = 0; step < steps + kAhead; ++step) {
        if (step < steps) {
          wait_free(step);
          const uint32_t at = base + (step % kStages) * S::kStage;
          copy(A, at);
          copy(B, at + S::kPlaneA);
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
    for (int step = 0; step < steps; ++step) {
      const int stage = step % kStages;
      mbar_wait_bounded(smem_u32(&bars.full[stage]), (uint32_t)(step / kStages) & 1, &abort_flag);
      __syncwarp();
      tc_fence_after_sync();
      const uint32_t at = base + stage * S::kStage;
      const uint64_t dA = smem_desc_sw128(at, 8192), dB = smem_desc_sw128(at + S::kTerms * S::kPlaneA, 8192);
      const uint32_t tL = tm + (F32 ? step % 3 * BN : 0), tR = tm + S::tSmall;
#pragma unroll
      for (int k = 0; k < kBK / 16; ++k) {
        const uint64_t ak = desc_advance(dA, k * step_a), bk = desc_advance(dB, k * step_b);
        mma_bf16_elect(tL, ak, bk, idesc, (!F32 && step > 0) || k > 0);
        if constexpr (F32) {
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

  if (tid < kLoaders) {
    if (F32)
      for (int step = max(steps - 2, 0); step < steps; ++step) fold(step);
    if (steps > 0) {
      float t[kOwn];
      tmem_ld_cols(tm_own + (F32 ? S::tSmall : 0), t);
      tmem_ld_wait();
#pragma unroll
      for (int x = 0; x < kOwn; ++x)
        if (isfinite(v[x])) v[x] += t[x];    // else an operand is not finite and its small terms are NaN; the leading ones are
                                             // fp32's, but for infinity times a number below 2^-134, which is zero in bf16: NaN
    }
    const int row = m0 + own_row, col = n0 + own_col;
    if (F32 && odd_input != 0 && row < task.m) {
      // a finite operand of the tile has no bf16 term next to it: in fp32 steps, as IEEE has it.  Many times as long as the
      // products above, so not for infinities and NaN, which a step with an overflow is full of.
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
// K steps that a CTA adds up in fp32.  Longer sums are split over the CTAs of a cluster: the roundings of a sum of n steps come to
// some 2^-25 sqrt(n / 3) of it, which stays below what the last bit of the leading products loses.
static int most_steps(int cols) { return cols == 64 ? 70 : 32; }

// How a group of products is cut: columns of a tile, CTAs per cluster, and the K steps from which on a task's tiles are shared by a cluster
struct GemmCut {
  int cols, split, from;
  int of(const GemmTask& t) const { return t.sums == nullptr && steps_of(t) >= from ? split : 1; }
};
// The cut with the shortest estimate (against the best of all cuts, measured for 24 groups of 62 to 15000 rows in fp32: 3 % longer on
// average, 12 % at most): the K steps of the longest CTA, or the steps per SM, whichever is more; a step with 128 columns costs
// 1.95 of one with 64, and a CTA that shares a tile spends some three steps (bf16: two, and two more per launch) on every other one.
static GemmCut gemm_cut(const GemmGroup& G, int dtype) {
  const bool f32 = dtype == NSA_F32;
  GemmCut best = {64, 1, 1 << 30};
  double least = -1.;
  for (int cols = 64; cols <= (f32 ? 128 : 64); cols *= 2) {
    if (G.cols != 0 && f32 && cols != G.cols) continue;
    for (int split = 1; split <= gemm::kMaxSplit; split *= 2) {
      if (G.split != 0 && split != G.split) continue;
      // from which length on tasks are shared: all that leave a CTA two steps, or the long ones only
      for (int from = 2 * split; from <= 1024; from *= 2) {
        const GemmCut cut = {cols, split, from};
        int64_t total = 0, longest = 0;
        bool fits = true;
        for (int t = 0; t < G.tasks; ++t) {
          const int64_t per = (steps_of(G.task[t]) + cut.of(G.task[t]) - 1) / cut.of(G.task[t]);
          longest = per > longest && tiles_of(G.task[t], cols) > 0 ? per : longest;
          total += tiles_of(G.task[t], cols) * (steps_of(G.task[t]) + (cut.of(G.task[t]) > 1 ? (f32 ? 3 : 2) * split : 0));
          fits = fits && (!f32 || per <= most_steps(cols));
        }
        const double per_sm = (double)total / 148., estimate = (per_sm > longest ? per_sm : longest + .5 * per_sm) * (cols == 64 ? 1. : 1.95) + (split > 1 && !f32 ? 2. : 0.);
        if (G.split == 0 && !fits) continue;
        if (least < 0. || estimate < least) {
          least = estimate;
          best = cut;
        }
        if (split == 1) break;
      }
    }
  }
  return best;
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
