// Gradient through the differentiable top-k: d(value of a pick) back through the softmax with the sink, the mean over a
// block's compressed columns and the mean over the heads to the logits, and from there to queries and compressed keys.
//
// Two launches, 37 us for 4 x 512 positions of 8 / 4 heads with 64 compressed columns; as tensor operations with two library products
// 38 launches, 100 us on the GPU and 300 us on the host.
// Bound there: latency of the loads in the products (256 blocks, issue slots 16 % busy); with more rows the CUDA cores (4 d ncb
// operations per row in fp32).
#include "nsa_common.cuh"
#include "nsa_kernels.h"

namespace nsa {

// ---- gradient of the logits: dlog [rows, ncb], one warp per row (batch, selection head, query).
// ds_j = p_j (dp_j - sum p dp) where dp is zero but at the picks: first every column without its dp, then the picks on top.
__global__ void __launch_bounds__(256) topk_logits_kernel(const TopkGrad P) {
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= (int64_t)P.batch * P.sel_heads * P.seq) return;
  const int i = (int)(row % P.seq), cpf = P.cpf, cols = P.ncb / cpf, own = cpf > 1 ? i / P.block : -1;
  const float* imp = P.importance + row * P.ncb;
  float* out = P.dlog + row * P.ncb;
  const int64_t* idx = P.idx + row * P.k;
  const float* dvals = P.dvals + row * P.k;
  auto logit = [&](int j) {
    if (j == own) return -FLT_MAX;
    if (cpf == 1) return imp[j];
    float s = 0.f;
    for (int c = 0; c < cpf; ++c) s += imp[j * cpf + c];
    return s / (float)cpf;
  };
  float mx = -1000.f;                       // the sink
  for (int j = lane; j < cols; j += 32) mx = fmaxf(mx, logit(j));
  mx = warp_max(mx);
  float z = 0.f;
  for (int j = lane; j < cols; j += 32) z += expf(logit(j) - mx);
  z = warp_sum(z) + expf(-1000.f - mx);
  float dot = 0.f;
  for (int t = lane; t < P.k; t += 32) {
    const int64_t j = idx[t];
    if (j >= 0 && j < cols) dot = fmaf(expf(logit((int)j) - mx) / z, dvals[t], dot);
  }
  dot = warp_sum(dot);
  // column c of the compressed blocks: visible before i / stride, and part of a whole selection block
  const float unit = P.scale / (float)cpf;
  const int visible = P.causal ? min(P.ncb, i / P.stride) : P.ncb;
  for (int c = lane; c < P.ncb; c += 32) {
    const int j = c / cpf;
    out[c] = c < visible && j < cols && j != own ? -(expf(logit(j) - mx) / z) * dot * unit : 0.f;
  }
  __syncwarp();
  for (int t = lane; t < P.k; t += 32) {
    const int64_t j = idx[t];
    if (j < 0 || j >= cols || j == own) continue;
    const float add = expf(logit((int)j) - mx) / z * dvals[t] * unit;
    for (int c = 0; c < cpf; ++c)
      if (j * cpf + c < visible) atomicAdd(out + j * cpf + c, add);   // (a block that is picked twice counts twice)
  }
}

// ---- dq += dlog ck for every head that shares the selection, dck += dlog^T (sum of these heads' q): 64 x 64 tiles, 4 x 4
// per thread, 16 steps of the sum at a time in shared memory.
template <typename T>
__global__ void __launch_bounds__(256) topk_products_kernel(const TopkGrad P, int dq_tiles, int dck_slices) {
  constexpr int TILE = 64, KB = 16;
  __shared__ __align__(16) float a_s[KB][TILE + 4], b_s[KB][TILE + 4];   // (read as float4)
  const int tid = threadIdx.x, ty = tid / 16, tx = tid % 16, d0 = blockIdx.y * TILE;
  const int sel_per_kv = P.sel_heads / P.kv_heads, per_sel = P.heads / P.sel_heads, F = (P.heads + 2 * P.kv_heads) * P.d;
  const int kv = P.num_mem + P.ncb, row_tiles = (P.seq + TILE - 1) / TILE, col_tiles = (P.ncb + TILE - 1) / TILE;
  const bool to_q = (int)blockIdx.x < dq_tiles;
  int m0, k0, k1, bs;            // bs: (batch, selection head) for dq, (batch, KV head) for dck
  if (to_q) {
    bs = blockIdx.x / row_tiles;
    m0 = (blockIdx.x - bs * row_tiles) * TILE;
    k0 = 0;
    k1 = P.causal ? min(P.ncb, (min(m0 + TILE, P.seq) - 1) / P.stride) : P.ncb;
  } else {
    int at = blockIdx.x - dq_tiles;
    const int slice = at % dck_slices;
    at /= dck_slices;
    bs = at / col_tiles;
    m0 = (at - bs * col_tiles) * TILE;
    // the rows (selection head of the KV head, query) of this slice
    const int rows = sel_per_kv * P.seq, per = (rows + dck_slices - 1) / dck_slices;
    k0 = slice * per;
    k1 = min(rows, k0 + per);
  }
  const int b = to_q ? bs / P.sel_heads : bs / P.kv_heads, h = to_q ? bs % P.sel_heads : bs % P.kv_heads;
  const int kvh = to_q ? h / sel_per_kv : h;
  const T* ck = (const T*)P.ck + (((int64_t)b * P.kv_heads + kvh) * kv + P.num_mem) * P.d;
  const float* dlog = P.dlog + ((int64_t)b * P.sel_heads + (to_q ? h : h * sel_per_kv)) * P.seq * P.ncb;
  float acc[4][4];
#pragma unroll
  for (int x = 0; x < 4; ++x) acc[x][0] = acc[x][1] = acc[x][2] = acc[x][3] = 0.f;
  for (int k = k0; k < k1; k += KB) {
    __syncthreads();
    for (int e = tid; e < KB * TILE; e += 256) {
      if (to_q) {   // a_s[k][m] = dlog[m0 + m][k], read along the columns; b_s[k][n] = ck[k][d0 + n]
        const int c = e % KB, m = e / KB;
        a_s[c][m] = k + c < k1 && m0 + m < P.seq ? dlog[(int64_t)(m0 + m) * P.ncb + k + c] : 0.f;
        const int n = e % TILE, r = e / TILE;
        b_s[r][n] = k + r < k1 && d0 + n < P.d ? Elem<T>::to_float(ck[(int64_t)(k + r) * P.d + d0 + n]) : 0.f;
      } else {      // a_s[k][m] = dlog[k][m0 + m]; b_s[k][n] = sum over the heads of q[k][d0 + n]
        const int m = e % TILE, r = e / TILE, at = k + r;
        a_s[r][m] = at < k1 && m0 + m < P.ncb ? dlog[(int64_t)at * P.ncb + m0 + m] : 0.f;
        float q = 0.f;
        if (at < k1 && d0 + m < P.d) {
          const int s = at / P.seq, i = at - s * P.seq;
          const T* src = (const T*)P.qkv + ((int64_t)b * P.seq + i) * F + (int64_t)(h * sel_per_kv + s) * per_sel * P.d + d0 + m;
          for (int g = 0; g < per_sel; ++g) q += Elem<T>::to_float(src[g * P.d]);
        }
        b_s[r][m] = q;
      }
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < KB; ++c) {
      const float4 a = *reinterpret_cast<const float4*>(&a_s[c][ty * 4]), v = *reinterpret_cast<const float4*>(&b_s[c][tx * 4]);
      const float am[4] = {a.x, a.y, a.z, a.w}, bn[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) acc[x][y] = fmaf(am[x], bn[y], acc[x][y]);
    }
  }
#pragma unroll
  for (int x = 0; x < 4; ++x) {
    const int m = m0 + ty * 4 + x;
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const int n = d0 + tx * 4 + y;
      if (n >= P.d) continue;
      if (to_q) {
        if (m < P.seq)
          for (int g = 0; g < per_sel; ++g) P.dq[(((int64_t)b * P.heads + (int64_t)h * per_sel + g) * P.seq + m) * P.d + n] += acc[x][y];
      } else if (m < P.ncb) {
        atomicAdd(P.dck + (((int64_t)b * P.kv_heads + h) * kv + P.num_mem + m) * P.d + n, acc[x][y]);
      }
    }
  }
}

int launch_topk_grad(const TopkGrad& P, int dtype, cudaStream_t stream) {
  const int64_t rows = (int64_t)P.batch * P.sel_heads * P.seq;
  if (rows == 0 || P.ncb == 0 || P.k == 0) return NSA_OK;
  const int64_t warps = (rows + 7) / 8, dq_tiles = (int64_t)P.batch * P.sel_heads * ((P.seq + 63) / 64);
  // about four blocks per SM for the sums over the rows, of no fewer than 64 rows each
  const int64_t cols = (int64_t)P.batch * P.kv_heads * ((P.ncb + 63) / 64), sums = (int64_t)(P.sel_heads / P.kv_heads) * P.seq;
  int64_t slices = 148 * 4 / cols + 1;
  slices = slices < (sums + 63) / 64 ? slices : (sums + 63) / 64;
  if (warps > 0x7fffffff || dq_tiles + cols * slices > 0x7fffffff) return fail(NSA_ERR_SHAPE, "layer: too many rows for the gradient of the top-k");
  topk_logits_kernel<<<(unsigned)warps, 256, 0, stream>>>(P);
  const dim3 grid((unsigned)(dq_tiles + cols * slices), (unsigned)((P.d + 63) / 64));
  if (dtype == NSA_F32) topk_products_kernel<float><<<grid, 256, 0, stream>>>(P, (int)dq_tiles, (int)slices);
  else topk_products_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>(P, (int)dq_tiles, (int)slices);
  count_launches(2);
  const cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? NSA_OK : fail((int)err, cudaGetErrorString(err));
}

}  // namespace nsa
