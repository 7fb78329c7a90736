// One decoding step: of the operator (the attention part) and of the whole layer.

#include <algorithm>
#include <cmath>
#include <tuple>

#include "nsa_kernels.h"
#include "rooms.h"

namespace nsa_host {

static nsa_decode_args decode_args(const void* q, const void* qr, const Tensor& keys, const Tensor& vals, const Tensor& ck,
                                   const Tensor& cv, const void* mem_k, const void* mem_v, int64_t num_mem, const void* gates,
                                   void* out, int64_t heads, int64_t stride, int64_t block, int64_t nsel, int64_t window) {
  nsa_decode_args a = {};
  a.q = q; a.qr = qr; a.gates = gates; a.out = out; a.mem_k = mem_k; a.mem_v = mem_v;
  a.keys = t4(keys); a.vals = t4(vals);
  a.ncb = ck.size(2);
  if (a.ncb > 0) { a.ck = t4(ck); a.cv = t4(cv); }
  a.batch = keys.size(0); a.q_heads = heads; a.dim_head = keys.size(3); a.kv_heads = keys.size(1); a.cache_len = keys.size(2);
  a.num_mem = num_mem; a.stride = stride; a.block = block; a.nsel = nsel; a.window = window;
  a.dtype = dtype_code(keys); a.scale = 1.f / std::sqrt((float)keys.size(3));
  return a;
}

// The kernels take batch, heads and row length from one tensor and address the others with them
static void require_shape(bool ok, const char* what) {
  if (!ok) throw Error(std::string("decode step: ") + what);
}
static bool is_cache(const Tensor& k, const Tensor& v, int64_t batch, int64_t heads, int64_t d) {
  return k.dim() == 4 && k.size(0) == batch && k.size(1) == heads && k.size(3) == d && v.sizes() == k.sizes();
}
static void check_compressed(const Tensor& ck, const Tensor& cv, int64_t batch, int64_t heads, int64_t d) {
  require_shape(is_cache(ck, cv, batch, heads, d), "compressed keys and values must both be [batch, kv_heads, blocks, dim_head] of the cache they belong to");
}

// Attention part of a step on tensors the caller holds
static Tensor decode_step(Tensor q, Tensor qr, Tensor keys, Tensor vals, Tensor ck, Tensor cv, Tensor mem_k, Tensor mem_v,
                          Tensor gates, int64_t stride, int64_t block, int64_t nsel, int64_t window) {
  for (const Tensor* t : {&q, &qr, &keys, &vals, &ck, &cv, &mem_k, &mem_v, &gates}) require_cuda(*t);
  require_shape(q.dim() == 3 && qr.sizes() == q.sizes(), "q and qr must both be [batch, q_heads, dim_head]");
  require_shape(keys.dim() == 4 && is_cache(keys, vals, q.size(0), keys.size(1), q.size(2)),
                "keys and values must both be [batch, kv_heads, rows, dim_head] with the batch and dim_head of q");
  check_compressed(ck, cv, q.size(0), keys.size(1), q.size(2));
  require_shape(mem_k.dim() == 3 && mem_k.size(0) == keys.size(1) && mem_k.size(2) == q.size(2) && mem_v.sizes() == mem_k.sizes(),
                "memory keys and values must both be [kv_heads, slots, dim_head]");
  require_shape(gates.numel() == q.size(0) * q.size(1) * 3, "gates must be [batch, q_heads, 3]");
  const c10::cuda::CUDAGuard guard(q.device());
  const auto dt = q.scalar_type();
  q = q.contiguous();
  qr = qr.to(dt).contiguous();
  gates = gates.to(dt).contiguous();
  mem_k = mem_k.to(dt).contiguous();
  mem_v = mem_v.to(dt).contiguous();
  keys = rowwise(keys.to(dt));
  vals = rowwise(vals.to(dt));
  if (ck.size(2) > 0) {
    ck = rowwise(ck.to(dt));
    cv = rowwise(cv.to(dt));
  }
  Tensor out = at::empty({q.size(0), q.size(1) * q.size(2)}, q.options());
  const nsa_decode_args a = decode_args(q.data_ptr(), qr.data_ptr(), keys, vals, ck, cv, mem_k.data_ptr(), mem_v.data_ptr(),
                                        mem_k.size(1), gates.data_ptr(), out.data_ptr(), q.size(1), stride, block, nsel, window);
  check(nsa_decode_step(&a, stream_of(q)));
  return out;
}

// Rows of room behind a cache that has to move: an eighth of it, so that the copies of a long generation add up to a
// small multiple of the final cache, within bounds that keep short caches and the largest ones sensible.
static int64_t room_for(int64_t rows) { return std::min<int64_t>(std::max<int64_t>(rows / 8, 64), 2048); }

// Token rows x [B, 1, dim] against the caches.  -> out, keys, vals, the window being filled (keys, values)
static std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor> layer_decode(
    Tensor x, OptTensor norm_w, double eps, Tensor qkv_w, Tensor gate_w, Tensor gate_b, Tensor out_w, Tensor inv_freq,
    Tensor mem_kv, Tensor past_k, Tensor past_v, Tensor ck, Tensor cv, Tensor run_k, Tensor run_v, int64_t heads,
    int64_t stride, int64_t block, int64_t cbs, int64_t nsel, int64_t window) {
  require_shape(x.dim() == 3 && x.size(1) == 1, "the input must be [batch, 1, dim]");
  require_shape(mem_kv.dim() == 4 && mem_kv.size(0) == 2, "memory slots must be [2, kv_heads, slots, dim_head]");
  const int64_t B = x.size(0), dim = x.size(2), hkv = mem_kv.size(1), d = mem_kv.size(3), rows = 3 * heads;
  require_shape(qkv_w.dim() == 2 && qkv_w.size(0) == (heads + 2 * hkv) * d && qkv_w.size(1) == dim && gate_w.dim() == 2 &&
                    gate_w.size(0) == rows && gate_w.size(1) == dim && gate_b.numel() == rows && out_w.dim() == 2 &&
                    out_w.size(0) == dim && out_w.size(1) == heads * d && (!norm_w.has_value() || norm_w->numel() == dim) &&
                    inv_freq.numel() == d / 2,
                "the weights are not those of a layer with these heads");
  require_shape(is_cache(past_k, past_v, B, hkv, d), "cached keys and values must both be [batch, kv_heads, rows, dim_head] with the batch of the input");
  check_compressed(ck, cv, B, hkv, d);
  require_shape(is_cache(run_k, run_v, B, hkv, d), "the window being filled must be [batch, kv_heads, rows, dim_head], keys and values alike");
  const c10::cuda::CUDAGuard guard(x.device());
  void* st = stream_of(x);
  const int dt = dtype_code(x);
  x = rowwise(x);
  ck = rowwise(ck);
  cv = rowwise(cv);
  GrownPair cache = Rooms::instance().extend(past_k, past_v, room_for(past_k.size(2)));
  GrownPair run = Rooms::instance().extend(run_k, run_v, 4 * cbs);
  // the qkv rows, the merged rows and the gates in one buffer of 16-byte aligned parts
  auto up = [](int64_t n) { return (n + 7) / 8 * 8; };
  const int64_t features = qkv_w.size(0), el = x.element_size();
  const int64_t at_merged = up(B * features), at_gates = at_merged + up(B * heads * d);
  Tensor work = at::empty({at_gates + B * rows}, x.options());
  uint8_t* const w = static_cast<uint8_t*>(work.data_ptr());
  void *qkv = w, *merged = w + at_merged * el, *gates = w + at_gates * el;
  Tensor qkv_rows, gate_rows;
  const bool projected = nsa::project_serves(B, dim, dt);
  if (projected) {
    nsa::ProjectParams p = {};
    p.x[0] = x.data_ptr(); p.x_sb = x.stride(0);
    p.norm_w = norm_w.has_value() ? norm_w->data_ptr() : nullptr; p.eps = (float)eps;
    p.w[0] = qkv_w.data_ptr(); p.gate_w = gate_w.data_ptr(); p.gate_b = gate_b.data_ptr();
    p.y[0] = qkv; p.y_sb = features; p.gates = gates; p.rows = B; p.heads = p.sets = 1; p.dim = dim; p.features = features;
    p.gates_n = rows; p.chained = 1;
    check(nsa::launch_project(p, dt, (cudaStream_t)st));
  } else {
    const Tensor xn = norm_w.has_value() ? at::rms_norm(x, {dim}, norm_w, eps) : x;
    qkv_rows = at::linear(xn, qkv_w);
    gate_rows = at::sigmoid(at::linear(xn, gate_w, gate_b));
    qkv = qkv_rows.data_ptr();
    gates = gate_rows.data_ptr();
  }
  const uint8_t* mem = static_cast<const uint8_t*>(mem_kv.data_ptr());
  const nsa_decode_args a = decode_args(nullptr, nullptr, cache.k, cache.v, ck, cv, mem, mem + mem_kv.numel() / 2 * el,
                                        mem_kv.size(2), gates, merged, heads, stride, block, nsel, window);
  nsa::DecodeParams p;
  check(nsa::fill_decode(p, a));
  p.qkv = qkv; p.inv_freq = ptr<float>(inv_freq);
  p.new_keys = cache.k_buf; p.new_vals = cache.v_buf; p.c_sb = cache.k.stride(0); p.c_sh = cache.k.stride(1); p.row = cache.row;
  p.run_k = run.k_buf; p.run_v = run.v_buf; p.r_sb = run.k.stride(0); p.r_sh = run.k.stride(1); p.run_row = run.row;
  p.chained = projected;
  check(nsa::launch_decode(p, dt, (cudaStream_t)st));
  Tensor out;
  if (nsa::project_serves(B, heads * d, dt)) {
    out = at::empty({B, 1, dim}, x.options());
    nsa::ProjectParams o = {};
    o.x[0] = merged; o.x_sb = heads * d; o.w[0] = out_w.data_ptr(); o.y[0] = out.data_ptr(); o.y_sb = dim;
    o.rows = B; o.heads = o.sets = 1; o.dim = heads * d; o.features = dim; o.chained = 2;
    check(nsa::launch_project(o, dt, (cudaStream_t)st));
  } else {
    out = at::linear(at::as_strided(work, {B, heads * d}, {heads * d, 1}, at_merged), out_w).unsqueeze(1);
  }
  return {out, cache.k, cache.v, run.k, run.v};
}

// The same for a layer that has not looked at its tensors yet: nothing where the step has to run module by module (another
// input than one token, parameters or caches of another type or device, off the 16-byte boundary).  `weights` as in
// layer_takes; cfg: heads, stride, block, cbs, nsel, window.  Asked one by one from Python, these questions were a fifth of a
// step's host time.
static std::optional<std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor>> layer_step(
    const Tensor& x, const std::vector<OptTensor>& w, double eps, const Tensor& inv_freq, const Tensor& past_k, const Tensor& past_v,
    const Tensor& ck, const Tensor& cv, const Tensor& run_k, const Tensor& run_v, const std::vector<int64_t>& cfg) {
  const int64_t heads = cfg.at(0), stride = cfg.at(1), block = cfg.at(2), cbs = cfg.at(3), nsel = cfg.at(4), window = cfg.at(5);
  if (x.dim() != 3 || x.size(1) != 1 || !w.at(5).has_value() || w[5]->dim() != 4) return std::nullopt;
  const Tensor& mem = *w[5];
  if (!layer_takes(x, w, heads, mem.size(1), mem.size(3), cbs, mem.size(2))) return std::nullopt;
  for (const Tensor* t : {&past_k, &past_v, &ck, &cv, &run_k, &run_v})
    if (t->scalar_type() != x.scalar_type() || t->device() != x.device()) return std::nullopt;
  return layer_decode(x, w[0], eps, *w[1], *w[2], *w[3], *w[4], inv_freq, mem, past_k, past_v, ck, cv, run_k, run_v, heads, stride, block, cbs,
                      nsel, window);
}

// The windows being filled (keys, values: [B, H, cbs, d]) have filled up: the two layers of either compress network, each
// one launch for both, and the compressed row appended to ck / cv.  -> ck, cv, or nothing where these kernels do not serve.
static std::optional<std::tuple<Tensor, Tensor>> compress_filled(Tensor run_k, Tensor run_v, OptTensor pos_k, OptTensor pos_v,
                                                                 Tensor k1, Tensor kb1, Tensor k2, Tensor kb2, Tensor v1,
                                                                 Tensor vb1, Tensor v2, Tensor vb2, Tensor ck, Tensor cv) {
  const int64_t B = run_k.size(0), H = run_k.size(1), d = run_k.size(3), width = run_k.size(2) * d, hidden = k1.size(0);
  for (const OptTensor& p : {pos_k, pos_v})
    if (!fits(p, run_k, {H, run_k.size(2), d})) return std::nullopt;
  for (const auto& net : {std::make_tuple(k1, kb1, k2, kb2), std::make_tuple(v1, vb1, v2, vb2)})
    if (!fits(std::get<0>(net), run_k, {hidden, width}) || !fits(std::get<1>(net), run_k, {hidden}) || !fits(std::get<2>(net), run_k, {d, hidden}) ||
        !fits(std::get<3>(net), run_k, {d}))
      return std::nullopt;
  check_compressed(ck, cv, B, H, d);
  const int dt = dtype_code(run_k);
  if (!nsa::project_serves(B * H, width, dt) || !nsa::project_serves(B * H, hidden, dt) || run_k.stride(2) != d ||
      run_k.strides() != run_v.strides() || run_k.stride(3) != 1 || run_v.stride(3) != 1)
    return std::nullopt;
  const c10::cuda::CUDAGuard guard(run_k.device());
  cudaStream_t st = (cudaStream_t)stream_of(run_k);
  GrownPair grown = Rooms::instance().extend(ck, cv, room_for(ck.size(2)));
  Tensor h = at::empty({2, B * H, hidden}, run_k.options());
  nsa::ProjectParams p = {};
  p.x[0] = run_k.data_ptr(); p.x[1] = run_v.data_ptr(); p.x_sb = run_k.stride(0); p.x_sh = run_k.stride(1);
  p.add[0] = pos_k->data_ptr(); p.add[1] = pos_v->data_ptr();
  p.w[0] = k1.data_ptr(); p.w[1] = v1.data_ptr(); p.bias[0] = kb1.data_ptr(); p.bias[1] = vb1.data_ptr();
  p.y[0] = h.data_ptr(); p.y[1] = static_cast<uint8_t*>(h.data_ptr()) + B * H * hidden * h.element_size();
  p.y_sb = H * hidden; p.y_sh = hidden;
  p.rows = B * H; p.heads = H; p.sets = 2; p.dim = width; p.features = hidden; p.relu = 1;
  check(nsa::launch_project(p, dt, st));
  nsa::ProjectParams o = {};
  o.x[0] = p.y[0]; o.x[1] = p.y[1]; o.x_sb = p.y_sb; o.x_sh = p.y_sh;
  o.w[0] = k2.data_ptr(); o.w[1] = v2.data_ptr(); o.bias[0] = kb2.data_ptr(); o.bias[1] = vb2.data_ptr();
  const int64_t at = grown.row * d * run_k.element_size();
  o.y[0] = static_cast<uint8_t*>(grown.k_buf) + at; o.y[1] = static_cast<uint8_t*>(grown.v_buf) + at;
  o.y_sb = grown.k.stride(0); o.y_sh = grown.k.stride(1);
  o.rows = B * H; o.heads = H; o.sets = 2; o.dim = hidden; o.features = d;
  check(nsa::launch_project(o, dt, st));
  return std::make_tuple(grown.k, grown.v);
}

void bind_decode(pybind11::module_& m) {
  namespace py = pybind11;
  m.def("decode_step", &decode_step, py::call_guard<py::gil_scoped_release>());
  m.def("compress_filled", &compress_filled, py::call_guard<py::gil_scoped_release>());
  m.def("layer_step", &layer_step, py::call_guard<py::gil_scoped_release>());
  m.def("layer_decode", &layer_decode, py::call_guard<py::gil_scoped_release>());
}

}  // namespace nsa_host
