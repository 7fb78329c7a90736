// The tensor work between the GEMMs and the attention kernels of a layer step: everything that moves whole activations
// between the layouts of the projections and those of the branches, one pass each.  Bound: HBM at training sizes, launch
// count at small ones.  As separate tensor operations these were some 60 of the 140 launches of a training step.
// Measured for the whole step with csrc/host/layer.cpp (forward + backward): dim 512, 8 heads of 64, 2 x 31 fp32 2.77 ->
// 0.47 ms; dim 256, 4 / 2 heads, 1 x 1024 bf16 3.20 -> 0.60 ms; dim 1024, 16 / 4 heads, 2 x 16384 bf16 6.49 -> 4.90 ms.

#include "nsa_common.cuh"
#include "nsa_kernels.h"

namespace nsa {

template <typename T>
struct Vec {
  static constexpr int V = 16 / (int)sizeof(T);
  float x[V];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < V; ++i) x[i] = 0.f;
  }
  __device__ __forceinline__ void load(const T* p) { Elem<T>::load_vec(p, x); }
  __device__ __forceinline__ void add(const T* p) {
    float y[V];
    Elem<T>::load_vec(p, y);
#pragma unroll
    for (int i = 0; i < V; ++i) x[i] += y[i];
  }
  __device__ __forceinline__ void add_f32(const float* p) {
#pragma unroll
    for (int i = 0; i < V; i += 4) {
      const float4 y = *reinterpret_cast<const float4*>(p + i);
      x[i] += y.x; x[i + 1] += y.y; x[i + 2] += y.z; x[i + 3] += y.w;
    }
  }
  __device__ __forceinline__ void store(T* p) const {
    uint4 raw;
    T* v = reinterpret_cast<T*>(&raw);
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = Elem<T>::from_float(x[i]);
    *reinterpret_cast<uint4*>(p) = raw;
  }
  // rotation of the feature pairs by the angles (or, with `back`, against them); no contraction, as the rotary kernel
  __device__ __forceinline__ void rotate(const float* co, const float* si, bool back) {
#pragma unroll
    for (int i = 0; i < V; i += 2) {
      const float a = x[i], b = x[i + 1], c = co[i / 2], s = back ? -si[i / 2] : si[i / 2];
      x[i] = __fadd_rn(__fmul_rn(a, c), __fmul_rn(-b, s));
      x[i + 1] = __fadd_rn(__fmul_rn(b, c), __fmul_rn(a, s));
    }
  }
};

// The cos / sin of the tile's positions, in shared memory: [kTileN][d / 2] each.  Computed once per tile and used by
// every head, so no table has to be kept in memory.
constexpr int kTileN = 8;
__device__ __forceinline__ void fill_angles(const LayerShape& L, const float* inv_freq, int n0, float* co, float* si) {
  const int half = L.d / 2;
  for (int e = threadIdx.x; e < kTileN * half; e += blockDim.x) {
    const float ang = (float)(n0 + e / half) * inv_freq[e % half];
    co[e] = cosf(ang);
    si[e] = sinf(ang);
  }
}

// ---- behind the qkv projection: rotated queries and keys (contiguous heads), the windows of the compress networks,
// and, for a caller that keeps a cache, the values in the cache's layout
template <typename T>
__global__ void __launch_bounds__(256) layer_prep_kernel(const LayerShape L, const LayerPrep P, int rot_blocks) {
  constexpr int V = Vec<T>::V;
  extern __shared__ float angles[];
  const int vpr = L.d / V, F = (L.heads + 2 * L.kv_heads) * L.d;
  const T* qkv = (const T*)P.qkv;
  if ((int)blockIdx.x < rot_blocks) {
    const int tiles = (L.seq + kTileN - 1) / kTileN;
    const int b = blockIdx.x / tiles, n0 = (blockIdx.x - b * tiles) * kTileN;
    float *co = angles, *si = angles + kTileN * (L.d / 2);
    fill_angles(L, P.inv_freq, n0, co, si);
    __syncthreads();
    const int rows = min(kTileN, L.seq - n0), heads = L.heads + (P.v_out != nullptr ? 2 : 1) * L.kv_heads;
    for (int e = threadIdx.x; e < heads * rows * vpr; e += 256) {
      const int c = (e % vpr) * V, t = e / vpr, r = t % rows, h = t / rows;
      const int64_t n = n0 + r;
      Vec<T> x;
      x.load(qkv + (b * (int64_t)L.seq + n) * F + h * L.d + c);
      if (h < L.heads + L.kv_heads) x.rotate(co + r * (L.d / 2) + c / 2, si + r * (L.d / 2) + c / 2, false);
      T* dst;
      if (h < L.heads) dst = (T*)P.qr + (((int64_t)b * L.heads + h) * L.seq + n) * L.d;
      else if (h < L.heads + L.kv_heads) dst = (T*)P.kr + b * P.c_sb + (h - L.heads) * P.c_sh + n * L.d;
      else dst = (T*)P.v_out + b * P.c_sb + (h - L.heads - L.kv_heads) * P.c_sh + n * L.d;
      x.store(dst + c);
    }
    return;
  }
  const int64_t per = (int64_t)L.batch * L.kv_heads * L.ncb * L.cbs * vpr;      // pieces of one of the two window tensors
  for (int64_t e = (int64_t)(blockIdx.x - rot_blocks) * 256 + threadIdx.x; e < 2 * per; e += (int64_t)(gridDim.x - rot_blocks) * 256) {
    const bool val = e >= per;
    const int64_t i = val ? e - per : e;
    const Coord4 at = split4(i, vpr, L.cbs, L.ncb);
    const int c = at.i0 * V, j = at.i1, w = at.i2, h = at.i3 % L.kv_heads;
    const int64_t b = at.i3 / L.kv_heads;
    const int tok = (w + 1) * L.stride - L.cbs + j;
    Vec<T> x;
    if (tok >= 0) x.load(qkv + (b * L.seq + tok) * F + (L.heads + (val ? L.kv_heads : 0) + h) * L.d + c);
    else x.zero();
    x.add((const T*)(val ? P.pos_v : P.pos_k) + ((int64_t)h * L.cbs + j) * L.d + c);
    x.store((T*)(val ? P.vw : P.kw) + i * V);
  }
}

int launch_layer_prep(const LayerShape& L, const LayerPrep& P, int dtype, cudaStream_t stream) {
  const int V = dtype == NSA_F32 ? 4 : 8;
  if (!aligned16(P.qkv, P.pos_k, P.pos_v, P.qr, P.kr, P.v_out, P.kw, P.vw) || P.c_sb % V || P.c_sh % V || L.d % V)
    return fail(NSA_ERR_ALIGN, "layer: qkv rows, positions and outputs must start on 16-byte boundaries");
  const int64_t rot = (int64_t)L.batch * ((L.seq + kTileN - 1) / kTileN);
  const int64_t win = (2 * (int64_t)L.batch * L.kv_heads * L.ncb * L.cbs * (L.d / V) + 255) / 256;
  if (rot > 0x3fffffff) return fail(NSA_ERR_SHAPE, "layer: too many positions for one launch");
  const int64_t grid = rot + (win < 148 * 16 ? win : 148 * 16);
  if (grid == 0) return NSA_OK;
  const size_t smem = (size_t)kTileN * L.d * sizeof(float);
  if (dtype == NSA_F32) layer_prep_kernel<float><<<(unsigned)grid, 256, smem, stream>>>(L, P, (int)rot);
  else layer_prep_kernel<__nv_bfloat16><<<(unsigned)grid, 256, smem, stream>>>(L, P, (int)rot);
  count_launches(1);
  const cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? NSA_OK : fail((int)err, cudaGetErrorString(err));
}

// ---- the memory slots in front of the compressed rows: [2][B, Hkv, num_mem + ncb, d]
template <typename T>
__global__ void __launch_bounds__(256) join_mem_kernel(const LayerShape L, const T* mem, const T* ck, const T* cv, T* out) {
  constexpr int V = Vec<T>::V;
  const int rows = L.num_mem + L.ncb, vpr = L.d / V;
  const int64_t per = (int64_t)L.batch * L.kv_heads * rows * vpr;
  for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < 2 * per; e += (int64_t)gridDim.x * 256) {
    const bool val = e >= per;
    const Coord4 at = split4(val ? e - per : e, vpr, rows, L.kv_heads);
    const int c = at.i0 * V, r = at.i1, h = at.i2;
    const int64_t b = at.i3;
    const T* src = r < L.num_mem ? mem + (((int64_t)(val ? 1 : 0) * L.kv_heads + h) * L.num_mem + r) * L.d + c
                                 : (val ? cv : ck) + ((b * L.kv_heads + h) * L.ncb + r - L.num_mem) * L.d + c;
    *reinterpret_cast<uint4*>(out + e * V) = *reinterpret_cast<const uint4*>(src);
  }
}

int launch_join_mem(const LayerShape& L, const void* mem, const void* ck, const void* cv, void* out, int dtype, cudaStream_t stream) {
  const int V = dtype == NSA_F32 ? 4 : 8;
  if (!aligned16(mem, ck, cv, out) || L.d % V) return fail(NSA_ERR_ALIGN, "layer: memory slots and compressed rows must start on 16-byte boundaries");
  const int64_t blocks = (2 * (int64_t)L.batch * L.kv_heads * (L.num_mem + L.ncb) * (L.d / V) + 255) / 256;
  if (blocks == 0) return NSA_OK;
  const unsigned grid = (unsigned)(blocks < 148 * 8 ? blocks : 148 * 8);
  if (dtype == NSA_F32) join_mem_kernel<float><<<grid, 256, 0, stream>>>(L, (const float*)mem, (const float*)ck, (const float*)cv, (float*)out);
  else
    join_mem_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>(L, (const __nv_bfloat16*)mem, (const __nv_bfloat16*)ck, (const __nv_bfloat16*)cv, (__nv_bfloat16*)out);
  count_launches(1);
  const cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? NSA_OK : fail((int)err, cudaGetErrorString(err));
}

// ---- backward of the joint: fp32 gradients [2][B, Hkv, num_mem + ncb, d] -> rows of the compress networks' outputs in
// the layer's type, their column sums (the bias of the second layer) and the slots' gradient summed over the batch
// Every block takes some rows of one of the two halves; column c of all its rows is summed by the threads that own it.
template <typename T>
__global__ void __launch_bounds__(256) split_mem_kernel(const LayerShape L, const float* grad, T* dc, float* dmem, float* dbias) {
  const int rows = L.num_mem + L.ncb, val = blockIdx.y;
  const int64_t total = (int64_t)L.batch * L.kv_heads * rows;
  const float* src = grad + val * total * L.d;
  const int64_t out_rows = (int64_t)L.batch * L.kv_heads * L.ncb;
  const int c = threadIdx.x % L.d, lane_rows = 256 / L.d;
  float sum = 0.f;
  if ((int)threadIdx.x < lane_rows * L.d) {
    for (int64_t r = (int64_t)blockIdx.x * lane_rows + threadIdx.x / L.d; r < total; r += (int64_t)gridDim.x * lane_rows) {
      const int w = (int)(r % rows);
      const int64_t bh = r / rows;
      const float v = src[r * L.d + c];
      if (w < L.num_mem) {
        atomicAdd(dmem + (((int64_t)val * L.kv_heads + bh % L.kv_heads) * L.num_mem + w) * L.d + c, v);
      } else {
        const T t = Elem<T>::from_float(v);
        dc[(val * out_rows + bh * L.ncb + w - L.num_mem) * L.d + c] = t;
        sum += Elem<T>::to_float(t);
      }
    }
    if (sum != 0.f) atomicAdd(dbias + val * L.d + c, sum);
  }
}

int launch_split_mem(const LayerShape& L, const float* grad, void* dc, float* dmem, float* dbias, int dtype, cudaStream_t stream) {
  const int64_t total = (int64_t)L.batch * L.kv_heads * (L.num_mem + L.ncb);
  if (total == 0) return NSA_OK;
  const int64_t want = (total * L.d + 1023) / 1024;
  const dim3 grid((unsigned)(want < 148 * 2 ? want : 148 * 2), 2);
  if (dtype == NSA_F32) split_mem_kernel<float><<<grid, 256, 0, stream>>>(L, grad, (float*)dc, dmem, dbias);
  else split_mem_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>(L, grad, (__nv_bfloat16*)dc, dmem, dbias);
  count_launches(1);
  const cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? NSA_OK : fail((int)err, cudaGetErrorString(err));
}

// ---- column sums (the bias of the first compress layer) behind the ReLU whose output is `act`: x = act > 0 ? x : 0 in
// place.  A block owns 32 sixteen-byte columns and a slice of the rows; sets side by side in blockIdx.z.  The slices meet in
// float atomics, as those of split_mem_kernel and pos_grad do: the last bits of these sums differ from run to run,
// like those of dk and dv behind them (fp32 reductions of the attention kernels).
template <typename T>
__global__ void __launch_bounds__(256) relu_sums_kernel(const ColumnSums P) {
  constexpr int V = Vec<T>::V;
  __shared__ float fold[8][32 * V];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, set = blockIdx.z;
  const int col = (blockIdx.x * 32 + lane) * V;
  T* x = (T*)P.x[set];
  const T* act = (const T*)P.act[set];
  Vec<T> sum;
  sum.zero();
  if (col < P.cols) {
    const int64_t step = (int64_t)gridDim.y * 8;
    int64_t r = (int64_t)blockIdx.y * 8 + warp;
    for (; r < P.rows; r += step) {
      Vec<T> v, a;
      v.load(x + r * P.cols + col);
      a.load(act + r * P.cols + col);
#pragma unroll
      for (int i = 0; i < V; ++i) {
        v.x[i] = a.x[i] > 0.f ? v.x[i] : 0.f;
        sum.x[i] += v.x[i];
      }
      v.store(x + r * P.cols + col);
    }
  }
#pragma unroll
  for (int i = 0; i < V; ++i) fold[warp][lane * V + i] = sum.x[i];
  __syncthreads();
  for (int i = threadIdx.x; i < 32 * V; i += 256) {
    const int c = blockIdx.x * 32 * V + i;
    if (c < P.cols) {
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) s += fold[w][i];
      atomicAdd(P.out[set] + c, s);
    }
  }
}

int launch_relu_sums(const ColumnSums& P, int dtype, cudaStream_t stream) {
  if (P.rows == 0 || P.cols == 0) return NSA_OK;
  const int V = dtype == NSA_F32 ? 4 : 8;
  if (P.cols % V) return fail(NSA_ERR_ALIGN, "column sums behind a ReLU need rows of whole 16-byte pieces");
  const int gx = (P.cols / V + 31) / 32;
  int64_t gy = 148 * 4 / ((int64_t)gx * P.sets) + 1;              // about four blocks per SM: every block ends in atomics
  const int64_t most = (P.rows + 15) / 16;
  gy = gy < most ? gy : most;
  const dim3 grid((unsigned)gx, (unsigned)(gy < 65535 ? gy : 65535), (unsigned)P.sets);
  if (dtype == NSA_F32) relu_sums_kernel<float><<<grid, 256, 0, stream>>>(P);
  else relu_sums_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>(P);
  count_launches(1);
  const cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? NSA_OK : fail((int)err, cudaGetErrorString(err));
}

// ---- column sums of the gates' gradient (their bias), in a fixed order: nothing before them depends on the order of
// atomics, so their bits repeat from run to run, and must not be lost here.  A block sums a slice of the rows of up to 256
// columns, VEC at a time per thread (one where a row is not whole 16-byte pieces), and leaves its part in `partial`; the
// block that arrives last adds the slices up in their order.  Up to 64 slices: the last block reads them all.
// `arrived`: one counter per 256 columns, zero.
constexpr int kGateSlices = 64;
template <typename T, int VEC>
__device__ __forceinline__ void gate_sums(const GateSums& P, int group, int slice, int slices) {
  __shared__ float fold[256 * VEC];
  __shared__ bool last;
  const T* x = (const T*)P.x;
  float *out = P.out, *partial = P.partial;
  const int64_t rows = P.rows;
  const int cols = P.cols;
  const int c0 = group * 256, width = min(256, cols - c0), units = width / VEC;
  const int tid = threadIdx.x, u = tid % units, r0 = tid / units, step = 256 / units;
  float sum[VEC];
#pragma unroll
  for (int i = 0; i < VEC; ++i) sum[i] = 0.f;
  if (r0 < step) {
    const int64_t per = (rows + slices - 1) / slices, end = min(rows, (slice + 1) * per);
#pragma unroll 4
    for (int64_t r = slice * per + r0; r < end; r += step) {
      const T* at = x + r * cols + c0 + u * VEC;
      if constexpr (VEC == 1) {
        sum[0] += Elem<T>::to_float(*at);
      } else {
        float v[VEC];
        Elem<T>::load_vec(at, v);
#pragma unroll
        for (int i = 0; i < VEC; ++i) sum[i] += v[i];
      }
    }
#pragma unroll
    for (int i = 0; i < VEC; ++i) fold[r0 * width + u * VEC + i] = sum[i];
  }
  __syncthreads();
  if (tid < width) {
    float s = 0.f;
    for (int k = 0; k < step; ++k) s += fold[k * width + tid];
    partial[(int64_t)slice * cols + c0 + tid] = s;
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(P.arrived + group, 1u) == slices - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int groups = 256 / width, c = tid % width, g = tid / width;
  float s = 0.f;
  if (g < groups) {
#pragma unroll 8
    for (int y = g; y < (int)slices; y += groups) s += __ldcg(partial + (int64_t)y * cols + c0 + c);
    fold[g * width + c] = s;
  }
  __syncthreads();
  if (tid < width) {
    s = 0.f;
    for (int k = 0; k < groups; ++k) s += fold[k * width + tid];
    out[c0 + tid] = s;
  }
}

int64_t gate_sums_partial(int cols) { return (int64_t)kGateSlices * cols; }
int gate_sums_counters(int cols) { return (cols + 255) / 256; }

// ---- gradient of the qkv projection's output, [B, N, (Hq + 2 Hkv) d]: per query head the gradient of the un-rotated
// query (compressed branch) plus the two rotated ones turned back; per key head the rotated key's gradient turned back
// plus what arrives through the windows that hold the token; per value head the same without the rotation.  Sums in
// fp32, one rounding.
template <typename T>
__device__ __forceinline__ void qkv_grad(const LayerShape& L, const QkvGrad& P, int block) {
  constexpr int V = Vec<T>::V;
  extern __shared__ float angles[];
  const int vpr = L.d / V, F = (L.heads + 2 * L.kv_heads) * L.d;
  const int tiles = (L.seq + kTileN - 1) / kTileN;
  const int b = block / tiles, n0 = (block - b * tiles) * kTileN;
  float *co = angles, *si = angles + kTileN * (L.d / 2);
  fill_angles(L, P.inv_freq, n0, co, si);
  __syncthreads();
  const int rows = min(kTileN, L.seq - n0), heads = L.heads + 2 * L.kv_heads;
  for (int e = threadIdx.x; e < heads * rows * vpr; e += 256) {
    const int h = (e / vpr) % heads, c = (e % vpr) * V, r = e / (vpr * heads);
    const int n = n0 + r;
    Vec<T> x;
    x.zero();
    const float *cr = co + r * (L.d / 2) + c / 2, *sr = si + r * (L.d / 2) + c / 2;
    if (h < L.heads) {
      const int64_t at = (((int64_t)b * L.heads + h) * L.seq + n) * L.d + c;
#pragma unroll
      for (int s = 1; s < 3; ++s) {
        if (P.dq_f32[s] != nullptr) x.add_f32(P.dq_f32[s] + at);
        else x.add((const T*)P.dq[s] + at);
      }
      x.rotate(cr, sr, true);
      if (P.dq_f32[0] != nullptr) x.add_f32(P.dq_f32[0] + at);
      else x.add((const T*)P.dq[0] + at);
    } else {
      const bool val = h >= L.heads + L.kv_heads;
      const int hk = h - L.heads - (val ? L.kv_heads : 0);
      const int64_t bh = (int64_t)b * L.kv_heads + hk;
      x.add_f32((val ? P.dv : P.dk) + (bh * L.seq + n) * L.d + c);
      if (!val) x.rotate(cr, sr, true);
      const T* dw = (const T*)(val ? P.dvw : P.dkw);
      if (dw != nullptr) {
        const int w_hi = min(L.ncb, (n + L.cbs) / L.stride);       // windows n / stride .. w_hi - 1 hold the token
        for (int w = n / L.stride; w < w_hi; ++w) x.add(dw + ((bh * L.ncb + w) * L.cbs + n - (w + 1) * L.stride + L.cbs) * L.d + c);
      }
    }
    x.store((T*)P.out + ((int64_t)b * L.seq + n) * F + h * L.d + c);
  }
}

// ---- gradients of the intra-block positions: sums over batch and windows of the window gradients, keys and values side
// by side (blockIdx.z); a thread owns a 16-byte piece of the window and a slice of the (batch, window) pairs
template <typename T>
__device__ __forceinline__ void pos_grad(const LayerShape& L, const T* dkw, const T* dvw, float* dpos, int group, int slot_groups, int slice, int slices,
                                         int val) {
  constexpr int V = Vec<T>::V;
  const int slots = L.cbs * L.d / V;
  const int h = group / slot_groups, slot = (group % slot_groups) * 256 + threadIdx.x;
  if (slot >= slots) return;
  const int64_t pairs = (int64_t)L.batch * L.ncb, window = (int64_t)slots * V;
  const int64_t per = (pairs + slices - 1) / slices, k0 = slice * per, k1 = k0 + per < pairs ? k0 + per : pairs;
  const T* base = (val ? dvw : dkw) + (int64_t)slot * V;
  Vec<T> sum;
  sum.zero();
#pragma unroll 4
  for (int64_t k = k0; k < k1; ++k) sum.add(base + (((k / L.ncb) * L.kv_heads + h) * L.ncb + k % L.ncb) * window);
  float* dst = dpos + ((int64_t)val * L.kv_heads + h) * window + (int64_t)slot * V;
#pragma unroll
  for (int i = 0; i < V; ++i) atomicAdd(dst + i, sum.x[i]);
}

// The three passes behind the window gradients, which do not depend on one another, in one launch: first the blocks of
// qkv_grad, then those of the positions, then those of the gates.
struct TailGrid {
  int qkv, pos_groups, slot_groups, pos_slices, gate_groups, gate_slices;
};
template <typename T, int VEC>
__global__ void __launch_bounds__(256, 5) layer_tail_kernel(const LayerShape L, const QkvGrad P, const GateSums S, float* dpos, const TailGrid g) {
  int block = blockIdx.x;
  if (block < g.qkv) {
    qkv_grad<T>(L, P, block);
    return;
  }
  block -= g.qkv;
  if (block < 2 * g.pos_groups * g.pos_slices) {
    const int group = block % g.pos_groups, rest = block / g.pos_groups;
    pos_grad<T>(L, (const T*)P.dkw, (const T*)P.dvw, dpos, group, g.slot_groups, rest % g.pos_slices, g.pos_slices, rest / g.pos_slices);
    return;
  }
  block -= 2 * g.pos_groups * g.pos_slices;
  gate_sums<T, VEC>(S, block % g.gate_groups, block / g.gate_groups, g.gate_slices);
}

int launch_layer_tail(const LayerShape& L, const QkvGrad& P, const GateSums& S, float* dpos, int dtype, cudaStream_t stream) {
  const int V = dtype == NSA_F32 ? 4 : 8;
  const int64_t qkv = (int64_t)L.batch * ((L.seq + kTileN - 1) / kTileN), pairs = (int64_t)L.batch * L.ncb;
  TailGrid g = {};
  g.slot_groups = (L.cbs * L.d / V + 255) / 256;
  g.pos_groups = L.kv_heads * g.slot_groups;
  int64_t slices = (148 * 2 + 2 * (int64_t)g.pos_groups - 1) / (2 * (int64_t)g.pos_groups);   // about two blocks per SM: every slice ends in atomics
  slices = slices < (pairs + 7) / 8 ? slices : (pairs + 7) / 8;
  g.pos_slices = pairs > 0 ? (int)slices : 0;
  const int64_t parts = (S.rows * S.cols + 2047) / 2048;
  g.gate_groups = gate_sums_counters(S.cols);
  g.gate_slices = S.rows > 0 && S.cols > 0 ? (int)(parts < kGateSlices ? parts : kGateSlices) : 0;
  const int64_t grid = qkv + 2 * (int64_t)g.pos_groups * g.pos_slices + (int64_t)g.gate_groups * g.gate_slices;
  if (grid == 0) return NSA_OK;
  if (grid > 0x7fffffff) return fail(NSA_ERR_SHAPE, "layer: too many positions for one launch");
  g.qkv = (int)qkv;
  const size_t smem = (size_t)kTileN * L.d * sizeof(float);
  const bool vec = S.cols % V == 0 && aligned16(S.x);
  if (dtype == NSA_F32) {
    if (vec) layer_tail_kernel<float, 4><<<(unsigned)grid, 256, smem, stream>>>(L, P, S, dpos, g);
    else layer_tail_kernel<float, 1><<<(unsigned)grid, 256, smem, stream>>>(L, P, S, dpos, g);
  } else {
    if (vec) layer_tail_kernel<__nv_bfloat16, 8><<<(unsigned)grid, 256, smem, stream>>>(L, P, S, dpos, g);
    else layer_tail_kernel<__nv_bfloat16, 1><<<(unsigned)grid, 256, smem, stream>>>(L, P, S, dpos, g);
  }
  count_launches(1);
  const cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? NSA_OK : fail((int)err, cudaGetErrorString(err));
}

// ---- the small fp32 gradients (norm, biases, slots, positions) in the layer's type
__global__ void __launch_bounds__(256) round_kernel(const float* src, __nv_bfloat16* dst, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) dst[i] = __float2bfloat16_rn(src[i]);
}

int launch_round(const float* src, void* dst, int64_t n, cudaStream_t stream) {
  if (n == 0) return NSA_OK;
  const int64_t blocks = (n + 255) / 256;
  round_kernel<<<(unsigned)(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, stream>>>(src, (__nv_bfloat16*)dst, n);
  count_launches(1);
  const cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? NSA_OK : fail((int)err, cudaGetErrorString(err));
}

}  // namespace nsa
