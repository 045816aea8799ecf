// The generation engine's launch chains in native code: the prompt prefill and the decode step of
// sizes that the fused step does not take.  In Python a layer of either costs 70-100 us of host time
// (library GEMMs and single kernels through two bindings), several times its kernels at small sizes.
// Included by native.cpp.
#pragma once

struct EngineModel {
  std::vector<Tensor> attn_norm, c_attn, c_proj, mlp_norm, gate_up, down;   // projections transposed: [in, out]
  Tensor wte, out_norm, lm_head, freqs;
  int64_t C, I, heads, head_dim, slots;
  double eps;
  int parity, window, retained_slot, window_slot;
  int dtype;                      // SPSATTN_DTYPE_BF16 or SPSATTN_DTYPE_FP32
  bool f32() const { return dtype == SPSATTN_DTYPE_FP32; }
  int layers() const { return (int)attn_norm.size(); }
};
constexpr const char* kEngineName = "sps_b200.EngineModel";

std::vector<Tensor> tensor_list(PyObject* o, bool transposed) {
  const Items items(o);
  std::vector<Tensor> out;
  for (Py_ssize_t i = 0; i < items.n; ++i) {
    const Tensor& t = tensor_arg(items[i], "weight");
    out.push_back(transposed ? t.t() : t);
  }
  return out;
}

// engine_model(attn_norm, c_attn, c_proj, mlp_norm, gate_up, down, wte, out_norm, lm_head, freqs, heads,
//              head_dim, slots, eps, parity, window, retained_slot, window_slot) -> capsule
PyObject* engine_model_impl(PyObject* const* a, Py_ssize_t n) {
  if (n != 18) fail(PyExc_TypeError, "engine_model takes 18 arguments");
  auto m = std::make_unique<EngineModel>();
  m->attn_norm = tensor_list(a[0], false);
  m->c_attn = tensor_list(a[1], true);
  m->c_proj = tensor_list(a[2], true);
  m->mlp_norm = tensor_list(a[3], false);
  m->gate_up = tensor_list(a[4], true);
  m->down = tensor_list(a[5], true);
  m->wte = tensor_arg(a[6], "wte");
  m->out_norm = tensor_arg(a[7], "out_norm");
  m->lm_head = tensor_arg(a[8], "lm_head").t();
  m->freqs = tensor_arg(a[9], "freqs");
  m->heads = int_arg(a[10]);
  m->head_dim = int_arg(a[11]);
  m->slots = int_arg(a[12]);
  m->eps = float_arg(a[13]);
  m->parity = (int)int_arg(a[14]);
  m->window = (int)int_arg(a[15]);
  m->retained_slot = (int)int_arg(a[16]);
  m->window_slot = (int)int_arg(a[17]);
  m->C = m->wte.size(1);
  m->I = m->down[0].size(0);
  m->dtype = m->wte.scalar_type() == at::kFloat ? SPSATTN_DTYPE_FP32 : SPSATTN_DTYPE_BF16;
  return PyCapsule_New(m.release(), kEngineName, [](PyObject* c) {
    delete reinterpret_cast<EngineModel*>(PyCapsule_GetPointer(c, kEngineName));
  });
}

EngineModel& engine_arg(PyObject* o) {
  void* p = PyCapsule_GetPointer(o, kEngineName);
  if (!p) throw python_error();
  return *reinterpret_cast<EngineModel*>(p);
}

void norm_into(const EngineModel& m, const Tensor& x, const Tensor* delta, const Tensor& weight, const Tensor& y, void* stream) {
  check_rc(spsattn_add_rmsnorm(x.data_ptr(), delta ? delta->data_ptr() : nullptr, weight.data_ptr(), y.data_ptr(), m.dtype,
                               x.size(0), (int)m.C, (float)m.eps, stream),
           "spsattn_add_rmsnorm");
}

// The block behind the attention of one layer, up to the norm that the next one starts with.
void block_tail(const EngineModel& m, int layer, const Tensor& y, const Tensor& x, Tensor& xn, Tensor& delta, Tensor& gate_up,
                Tensor& hidden, void* stream) {
  at::mm_out(delta, y, m.c_proj[layer]);
  norm_into(m, x, &delta, m.mlp_norm[layer], xn, stream);
  at::mm_out(gate_up, xn, m.gate_up[layer]);
  check_rc(spsattn_swiglu(gate_up.data_ptr(), hidden.data_ptr(), m.dtype, hidden.size(0), (int)m.I, stream), "spsattn_swiglu");
  at::mm_out(delta, hidden, m.down[layer]);
  norm_into(m, x, &delta, layer + 1 < m.layers() ? m.attn_norm[layer + 1] : m.out_norm, xn, stream);
}

// engine_scan(model, ids [B, T], eos, pad, predict, empty_after_eos) -> (ids2, pos2, run_start, doc_mask,
//             real_len, ends_on_eos, flags)
PyObject* engine_scan_impl(PyObject* const* a, Py_ssize_t n) {
  if (n != 6) fail(PyExc_TypeError, "engine_scan takes 6 arguments");
  const EngineModel& m = engine_arg(a[0]);
  const Tensor& ids = tensor_arg(a[1], "ids");
  require(ids.is_cuda() && ids.dim() == 2 && ids.scalar_type() == at::kLong && ids.is_contiguous(), "ids must be contiguous int64 [B, T]");
  const int64_t b = ids.size(0), t = ids.size(1), rows = t * m.slots;
  const long long eos = int_arg(a[2]), pad = int_arg(a[3]), predict = int_arg(a[4]);
  const bool empty_after_eos = bool_arg(a[5]);
  Tensor ids2, pos2, runs, mask, real, ends, flags;
  unlocked([&] {
    const c10::cuda::CUDAGuard guard(ids.device());
    auto make = [&](at::IntArrayRef shape, at::ScalarType type) {
      return at::detail::empty_cuda(shape, type, ids.device(), c10::nullopt);
    };
    ids2 = make({b, rows}, at::kLong), pos2 = make({b, rows}, at::kLong), runs = make({b, rows}, at::kInt);
    mask = make({b, t}, at::kByte), real = make({b}, at::kLong), ends = make({b}, at::kByte), flags = make({4}, at::kLong);
    check_rc(spsattn_prompt_scan(ids.data_ptr<int64_t>(), (int)b, (int)t, (int)m.slots, eos, pad, predict, empty_after_eos,
                                 ids2.data_ptr<int64_t>(), pos2.data_ptr<int64_t>(), runs.data_ptr<int>(),
                                 mask.data_ptr<uint8_t>(), real.data_ptr<int64_t>(), ends.data_ptr<uint8_t>(),
                                 flags.data_ptr<int64_t>(), status_ptr(ids), stream_of(ids)),
             "spsattn_prompt_scan");
  });
  PyRef r0(THPVariable_Wrap(ids2)), r1(THPVariable_Wrap(pos2)), r2(THPVariable_Wrap(runs)), r3(THPVariable_Wrap(mask)),
      r4(THPVariable_Wrap(real)), r5(THPVariable_Wrap(ends)), r6(THPVariable_Wrap(flags));
  return PyTuple_Pack(7, r0.p, r1.p, r2.p, r3.p, r4.p, r5.p, r6.p);
}

// Final-norm hidden states [B, N, C] of doubled ids; the caches of all layers (none: empty) filled on the way.
Tensor prefill_chain(const EngineModel& m, const Tensor& ids2, const Tensor& pos2, const Tensor& docs, const std::vector<Tensor>& caches,
                     const Tensor& mask) {
  const int64_t b = ids2.size(0), rows = ids2.size(1), all = b * rows, C = m.C, H = m.heads, D = m.head_dim;
  const bool runs = docs.scalar_type() == at::kInt;
  const c10::cuda::CUDAGuard guard(ids2.device());
  void* stream = stream_of(ids2);
  int* status = status_ptr(ids2);
  Tensor x = m.wte.index_select(0, ids2.reshape(-1));                       // [rows, C] residual stream
  const Tensor fc = m.freqs.index_select(0, pos2.reshape(-1));              // [rows, D/2, 2]
  auto make = [&](at::IntArrayRef shape, at::ScalarType type) {
    return at::detail::empty_cuda(shape, type, x.device(), c10::nullopt);
  };
  const at::ScalarType pt = x.scalar_type();
  Tensor xn = make({all, C}, pt), delta = make({all, C}, pt), qkv = make({all, 3 * C}, pt), gate_up = make({all, 2 * m.I}, pt),
         hidden = make({all, m.I}, pt), ops = make({3, all, C}, at::kBFloat16), y = make({all, C}, at::kBFloat16);
  uint16_t* op[3];
  spsattn_rope_group groups[3] = {};
  for (int g = 0; g < 3; ++g) {
    op[g] = reinterpret_cast<uint16_t*>(ops.data_ptr()) + g * all * C;
    groups[g].out = op[g];
    groups[g].stride_b = rows * C;
    groups[g].stride_n = C;
    groups[g].stride_h = D;
    groups[g].rotate = g < 2;
  }
  const int64_t strides[3] = {rows * C, D, C};                              // token-major: batch, head, row
  const int window = std::min<int64_t>(m.window, rows);
  const float scale = (float)(1.0 / std::sqrt((double)D));
  Tensor ws;
  const size_t ws_bytes = runs ? 0 : spsattn_prefill_workspace_bytes((int)b, (int)H, (int)rows, (int)D);
  if (ws_bytes) ws = empty_bytes(ws_bytes, x);
  norm_into(m, x, nullptr, m.attn_norm[0], xn, stream);
  for (int l = 0; l < m.layers(); ++l) {
    at::mm_out(qkv, xn, m.c_attn[l]);
    check_rc(spsattn_qkv_rope_cast(qkv.data_ptr(), m.f32() ? 2 : 0, rows * 3 * C, 3 * C, D, fc.data_ptr<float>(), rows * (D / 2),
                                   groups, 3, SPSATTN_DTYPE_BF16, (int)b, (int)rows, (int)H, (int)D, stream),
             "spsattn_qkv_rope_cast");
    if (!caches.empty()) {
      const Tensor br_k = caches[4][l], br_v = caches[5][l], br_len = caches[6][l];
      void* ring[2] = {nullptr, nullptr};
      int64_t* count[2] = {nullptr, nullptr};
      if (m.window > 0)
        for (int i = 0; i < 2; ++i) {
          ring[i] = caches[i][l].data_ptr();
          count[i] = caches[2 + i][l].data_ptr<int64_t>();
        }
      // the entry point addresses row 2 * token + slot of a doubled sequence; with one row per token
      // (Standard) half the row stride and slot 0 address row `token`
      check_rc(spsattn_fill_decode_caches(op[1], op[2], rows * C, m.slots == 2 ? C : C / 2, D, mask.data_ptr<uint8_t>(),
                                          br_k.data_ptr(), br_v.data_ptr(), br_len.data_ptr<int64_t>(), ring[0], ring[1], count[0],
                                          count[1], (int)b, (int)(rows / m.slots), (int)H, (int)D, (int)br_k.size(2),
                                          (int)caches[0].size(3), m.window, m.retained_slot, m.window_slot, stream),
               "spsattn_fill_decode_caches");
    }
    const int rc =
        runs ? spsattn_prefill_fwd_runs(op[0], op[1], op[2], y.data_ptr(), nullptr, strides, strides, strides, strides,
                                        docs.data_ptr<int>(), (int)b, (int)H, (int)rows, (int)D, SPSATTN_DTYPE_BF16, scale, m.parity,
                                        window, SPSATTN_NO_WINDOW, 0, status, stream)
             : spsattn_prefill_fwd_strided(op[0], op[1], op[2], y.data_ptr(), nullptr, strides, strides, strides, strides,
                                           docs.data_ptr(), 1, rows, 1, (int)b, (int)H, (int)rows, (int)D, SPSATTN_DTYPE_BF16, scale,
                                           m.parity, window, SPSATTN_NO_WINDOW, 0, ws.data_ptr(), ws_bytes, status, stream);
    check_rc(rc, "spsattn_prefill_fwd");
    block_tail(m, l, m.f32() ? y.to(pt) : y, x, xn, delta, gate_up, hidden, stream);
  }
  return xn.view({b, rows, C});
}

// engine_prefill(model, ids2 [B, N], pos2 [B, N], docs [B, N] int64 | run_start [B, N] int32,
//                caches (nw_k, nw_v, nw_len, nw_pos, br_k, br_v, br_len) or None, doc_mask or None)
//   -> final-norm hidden states [B, N, C]; the caches of all layers filled on the way
PyObject* engine_prefill_impl(PyObject* const* a, Py_ssize_t n) {
  if (n != 6) fail(PyExc_TypeError, "engine_prefill takes 6 arguments");
  const EngineModel& m = engine_arg(a[0]);
  const Tensor &ids2 = tensor_arg(a[1], "ids2"), &pos2 = tensor_arg(a[2], "pos2"), &docs = tensor_arg(a[3], "documents");
  require(docs.dim() == 2 && docs.sizes() == ids2.sizes() && docs.is_contiguous(), "documents must be contiguous [B, N]");
  std::vector<Tensor> caches;
  Tensor mask;
  if (a[4] != Py_None) {
    caches = tensor_list(a[4], false);
    require(caches.size() == 7, "seven cache tensors are needed");
    mask = tensor_arg(a[5], "doc_mask");
  }
  return THPVariable_Wrap(unlocked([&] { return prefill_chain(m, ids2, pos2, docs, caches, mask); }));
}

// engine_step(model, decoder address, source address, rope groups address, buffers (x, xn, delta, qkv, y,
//             gate_up, hidden, fc), logits, blocks): one decode step, its layers by spsattn_decoder_blocks or
//             by library GEMMs and single kernels
PyObject* engine_step_impl(PyObject* const* a, Py_ssize_t n) {
  if (n != 7) fail(PyExc_TypeError, "engine_step takes 7 arguments");
  const EngineModel& m = engine_arg(a[0]);
  const auto* d = reinterpret_cast<const spsattn_decoder*>(PyLong_AsVoidPtr(a[1]));
  const auto* source = reinterpret_cast<const spsattn_token_source*>(PyLong_AsVoidPtr(a[2]));
  const auto* groups = reinterpret_cast<const spsattn_rope_group*>(PyLong_AsVoidPtr(a[3]));
  if (PyErr_Occurred()) throw python_error();
  std::vector<Tensor> buf = tensor_list(a[4], false);
  require(d && source && groups && buf.size() == 8, "engine_step needs its argument blocks and eight buffers");
  Tensor &x = buf[0], &xn = buf[1], &delta = buf[2], &qkv = buf[3], &y = buf[4], &gate_up = buf[5], &hidden = buf[6], &fc = buf[7];
  Tensor logits = tensor_arg(a[5], "logits");
  const bool blocks = bool_arg(a[6]);
  unlocked([&] {
    const c10::cuda::CUDAGuard guard(x.device());
    void* stream = stream_of(x);
    int* status = status_ptr(x);
    const int ns = d->slots, b = d->batch;
    const int64_t C = m.C, D = m.head_dim;
    check_rc(spsattn_decoder_start(d, source, status, stream), "spsattn_decoder_start");
    if (blocks) {
      check_rc(spsattn_decoder_blocks(d, xn.data_ptr(), status, stream), "spsattn_decoder_blocks");
      at::mm_out(logits, xn.view({b, ns, C}).select(1, d->pred_slot), m.lm_head);
      return;
    }
    spsattn_extra extras[2] = {};
    for (int s = 0; s < ns; ++s) {
      extras[s].k = reinterpret_cast<const uint16_t*>(d->k2) + (size_t)s * b * C;
      extras[s].v = reinterpret_cast<const uint16_t*>(d->v2) + (size_t)s * b * C;
      extras[s].query_mask = s == 0 ? (1u << ns) - 1 : 2u;
    }
    norm_into(m, x, nullptr, m.attn_norm[0], xn, stream);
    for (int l = 0; l < m.layers(); ++l) {
      const spsattn_decoder_layer& w = d->layers[l];
      at::mm_out(qkv, xn, m.c_attn[l]);
      check_rc(spsattn_qkv_rope_cast(qkv.data_ptr(), m.f32() ? 2 : 0, 3 * ns * C, 0, D, fc.data_ptr<float>(), D / 2, groups, 3 * ns,
                                     SPSATTN_DTYPE_BF16, b, 1, (int)m.heads, (int)D, stream),
               "spsattn_qkv_rope_cast");
      check_rc(spsattn_decode_step(d->q, ns, d->y, SPSATTN_DTYPE_BF16, w.segments, d->n_segments, extras, ns, &w.append, b,
                                   (int)m.heads, (int)D, SPSATTN_DTYPE_BF16, (float)(1.0 / std::sqrt((double)D)), d->workspace,
                                   d->workspace_bytes, status, stream),
               "spsattn_decode_step");
      block_tail(m, l, m.f32() ? y.to(x.scalar_type()) : y, x, xn, delta, gate_up, hidden, stream);
    }
    at::mm_out(logits, xn.view({b, ns, C}).select(1, d->pred_slot), m.lm_head);
  });
  Py_RETURN_NONE;
}
