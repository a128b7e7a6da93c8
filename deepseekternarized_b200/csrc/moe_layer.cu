// A whole routed-expert layer (boilerplate/engine/model.py:407-422, engine/standard.py:154-176) from one host call: routing
// sort, gather, the two expert GEMMs with SwiGLU between them, the optional shared expert, combine. The same kernels, in
// the same order on one stream, as the layer's steps called one by one; what goes is the host's work between them (some
// twenty small allocations, checks and calls per layer) and, on the decode path, the passes that only moved rows: the
// gather is part of the quantisation, SwiGLU writes the second GEMV's quantised rows, the sort gives the inverse order.
// One token, six of 384 experts, two stacked terms: 198 us per call as single steps (75 us of kernels).
#include <cstring>

#include "dst_common.cuh"

namespace dst {
namespace {

struct Carve {
  uint8_t* base;
  size_t used = 0;
  explicit Carve(void* b) : base(static_cast<uint8_t*>(b)) {}
  template <typename T>
  T* take(size_t count) {
    T* r = reinterpret_cast<T*>(base + used);
    used += (count * sizeof(T) + 255) & ~(size_t)255;
    return r;
  }
};

enum Path { PATH_NONE, PATH_DECODE, PATH_DECODE_TQ1, PATH_PREFILL };

// One of the two GEMMs of a set of experts: its weights and the kernel that AUTO would take for n rows.
struct Gemm {
  GemmArgs a;
  Path path;
};
Gemm make_gemm(const dst_expert_weights& w, bool second, int64_t n, const int64_t* offsets) {
  Gemm g;
  std::memset(&g.a, 0, sizeof(g.a));
  GemmArgs& a = g.a;
  const void* const* dec = second ? w.w2_decode : w.w13_decode;
  const void* const* packed = second ? w.w2 : w.w13;
  const void* const* scale = second ? w.s2 : w.s13;
  a.terms.n = w.n_terms;
  a.scale_dtype = DST_SCALE_F16;
  a.E = w.experts;
  a.T = n;
  a.N = second ? w.hidden : 2 * w.inter;
  a.K = second ? w.inter : w.hidden;
  a.group = 128;
  a.G = a.K / 128;
  a.fmt = w.fmt;
  a.offsets = w.experts == 1 ? nullptr : offsets;
  a.max_rows = w.experts == 1 ? n : -1;
  a.weight_layout = DST_LAYOUT_TILED;
  a.out_dtype = DST_OUT_BF16;
  // the 2-bit decode copy takes the place of TQ1 weights by the rule of TQ2 tiles
  if (w.fmt == DST_FMT_TQ1 && dec[0] != nullptr && cdiv64(n, a.E) <= decode_row_limit(DST_FMT_TQ2, a.E, a.N)) {
    a.fmt = DST_FMT_TQ2;
    packed = dec;
  }
  a.Kp = cdiv64(a.K, a.fmt == DST_FMT_TQ2 ? 4 : 5);
  for (int i = 0; i < w.n_terms; ++i) {
    a.terms.packed[i] = static_cast<const uint8_t*>(packed[i]);
    a.terms.scale[i] = scale[i];
  }
  a.act_dtype = DST_ACT_BF16;
  if (auto_takes_decode(a)) {
    // the second GEMV's rows come quantised from decode_swiglu_quant: a row length it does not take is not covered here
    if (second && a.fmt == DST_FMT_TQ2 && !decode_swiglu_quant_supports(a.K)) {
      g.path = PATH_NONE;
      return g;
    }
    g.path = a.fmt == DST_FMT_TQ2 ? PATH_DECODE : PATH_DECODE_TQ1;
  } else {
    static const float one = 1.f;  // any non-null pointer: only asked whether the shape is covered
    a.act_dtype = DST_ACT_F16_NORM;
    a.row_scale = &one;
    g.path = prefill_supports(a) ? PATH_PREFILL : PATH_NONE;
    a.row_scale = nullptr;
  }
  return g;
}

struct Rows {  // a set of rows in the form one of the GEMM paths reads
  void* data;        // bf16 or fp16 rows
  float* factor;     // of fp16-normalised rows
  void* workspace;   // quantised rows
  size_t workspace_bytes;
};
Rows take_rows(Carve& c, Path path, int64_t n, int64_t K) {
  Rows r = {nullptr, nullptr, nullptr, 0};
  if (path == PATH_DECODE) {
    r.workspace_bytes = decode_workspace_bytes(n, K);
    r.workspace = c.take<uint8_t>(r.workspace_bytes);
  } else {
    r.data = c.take<uint16_t>((size_t)n * K);
    r.factor = c.take<float>(path == PATH_PREFILL ? n : 0);
  }
  return r;
}

struct Buffers {  // of one set of experts
  Rows xs, h;
  __half* gu;
  void* down;
};
// `down` lies over `xs`: the second GEMM writes it after the first one has read those (one stream). What is taken behind the
// returned mark is free again once the second GEMM is done. A layer's single steps hold xs, gu, h and down at once; the call
// needs no more memory than they do.
Buffers take_buffers(Carve& c, const dst_expert_weights& w, const Gemm& g1, const Gemm& g2, int64_t n, size_t* mark) {
  Buffers b;
  const size_t start = c.used;
  b.down = c.take<uint16_t>((size_t)n * w.hidden);
  const size_t down_end = c.used;
  c.used = start;
  b.xs = take_rows(c, g1.path, n, w.hidden);
  if (c.used < down_end) c.used = down_end;
  *mark = c.used;
  b.gu = c.take<__half>((size_t)n * 2 * w.inter);
  b.h = take_rows(c, g2.path, n, w.inter);
  return b;
}

#define DST_TRY(expr)             \
  do {                            \
    const int rc__ = (expr);      \
    if (rc__ != DST_OK) return rc__; \
  } while (0)

int run_gemm(Gemm& g, const Rows& r, void* out, cudaStream_t st) {
  g.a.out = out;
  if (g.path == PATH_PREFILL) {
    g.a.x = r.data;
    g.a.row_scale = r.factor;
    return launch_prefill(g.a, st);
  }
  g.a.x = r.data;
  g.a.workspace = r.workspace;
  g.a.workspace_bytes = r.workspace_bytes;
  return launch_decode(g.a, st);
}

// Rows x[order / top_k] (order null: x) through one set of experts -> b.down
int run_experts(const dst_expert_weights& w, Gemm& g1, Gemm& g2, const Buffers& b, const void* x, const int64_t* order, int top_k, int64_t n,
                const float* weights, float limit, bool standard, cudaStream_t st) {
  Rows xs = b.xs;
  if (g1.path == PATH_PREFILL) {
    DST_TRY(dst_gather_rows_norm(x, order, n, w.hidden, top_k, xs.data, xs.factor, st));
  } else if (g1.path == PATH_DECODE) {
    xs.data = const_cast<void*>(x);  // gathered by the quantisation
    g1.a.gather_order = order;
    g1.a.gather_top_k = top_k;
  } else if (order) {
    DST_TRY(dst_gather_rows(x, order, n, w.hidden, top_k, xs.data, st));
  } else {
    xs.data = const_cast<void*>(x);
  }
  DST_TRY(run_gemm(g1, xs, b.gu, st));
  if (g2.path == PATH_PREFILL) {
    if (standard) DST_TRY(dst_swiglu_std_norm(b.gu, n, w.inter, b.h.data, b.h.factor, st));
    else DST_TRY(dst_swiglu_norm(b.gu, weights, order, n, w.inter, limit, b.h.data, b.h.factor, st));
  } else if (g2.path == PATH_DECODE) {
    DST_TRY(decode_swiglu_quant(b.gu, weights, order, n, w.inter, limit, standard, b.h.workspace, st));
    g2.a.quantised = 1;
  } else if (standard) {
    DST_TRY(dst_swiglu_std(b.gu, n, w.inter, b.h.data, st));
  } else {
    DST_TRY(dst_swiglu(b.gu, weights, order, n, w.inter, limit, b.h.data, st));
  }
  return run_gemm(g2, b.h, b.down, st);
}

bool weights_ok(const dst_expert_weights* w) {
  if (w->n_terms < 1 || w->n_terms > DST_MAX_TERMS || (w->fmt != DST_FMT_TQ1 && w->fmt != DST_FMT_TQ2) || w->experts < 1 || w->hidden < 1 ||
      w->inter < 1)
    return false;
  for (int i = 0; i < w->n_terms; ++i) {
    if (!w->w13[i] || !w->s13[i] || !w->w2[i] || !w->s2[i]) return false;
    if (!w->w13_decode[i] != !w->w13_decode[0] || !w->w2_decode[i] != !w->w2_decode[0]) return false;  // all terms or none
  }
  return true;
}

int layer(const void* x, const float* weights, const int32_t* ids, int64_t T, int top_k, int standard, float limit, const dst_expert_weights* w,
          const dst_expert_weights* shared, void* y, void* workspace, size_t* bytes, cudaStream_t st) {
  if (!w || !weights_ok(w) || (shared && (!weights_ok(shared) || shared->experts != 1 || shared->hidden != w->hidden)) || T < 0 || top_k <= 0)
    return DST_ERR_BAD_ARG;
  if (top_k > 8 || w->hidden % 128 != 0 || w->inter % 128 != 0 || (shared && (shared->inter % 128 != 0 || standard)) || w->experts > 4096)
    return DST_ERR_UNSUPPORTED;
  if (T > 0x3fffffff / top_k) return DST_ERR_BAD_SHAPE;
  const int64_t n = T * top_k;
  Carve c(workspace);
  int64_t* order = c.take<int64_t>(n);
  int64_t* offsets = c.take<int64_t>(w->experts + 1);
  int64_t* inv = c.take<int64_t>(n);
  uint8_t* sort_ws = c.take<uint8_t>(dst_sort_workspace_bytes(n, w->experts));
  Gemm g1 = make_gemm(*w, false, n, offsets), g2 = make_gemm(*w, true, n, offsets);
  if (g1.path == PATH_NONE || g2.path == PATH_NONE) return DST_ERR_UNSUPPORTED;
  size_t mark = 0;
  const Buffers b = take_buffers(c, *w, g1, g2, n, &mark);
  Gemm s1, s2;
  Buffers sb;
  if (shared) {
    s1 = make_gemm(*shared, false, T, nullptr);
    s2 = make_gemm(*shared, true, T, nullptr);
    if (s1.path == PATH_NONE || s2.path == PATH_NONE) return DST_ERR_UNSUPPORTED;
    const size_t end = c.used;
    c.used = mark;  // the shared expert runs after the routed ones, in the memory of their gate, up and SwiGLU rows
    sb = take_buffers(c, *shared, s1, s2, T, &mark);
    if (c.used < end) c.used = end;
  }
  if (bytes) {  // only asked for the size
    *bytes = c.used;
    return DST_OK;
  }
  if (T == 0) return DST_OK;
  if (!x || !weights || !ids || !y || !workspace) return DST_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(x) & 15) != 0 || (reinterpret_cast<uintptr_t>(workspace) & 255) != 0) return DST_ERR_ALIGNMENT;
  DST_TRY(sort_rows(ids, 1, n, w->experts, order, offsets, nullptr, sort_ws, inv, st));
  DST_TRY(run_experts(*w, g1, g2, b, x, order, top_k, n, standard ? nullptr : weights, limit, standard != 0, st));
  if (shared) DST_TRY(run_experts(*shared, s1, s2, sb, x, nullptr, 1, T, nullptr, limit, false, st));
  return combine_rows(b.down, inv, ids, standard ? weights : nullptr, T, top_k, w->hidden, shared ? sb.down : nullptr, y, st);
}

}  // namespace
}  // namespace dst

extern "C" size_t dst_moe_layer_workspace_bytes(int64_t T, int top_k, int standard, const dst_expert_weights* w, const dst_expert_weights* shared) {
  size_t bytes = 0;
  return dst::layer(nullptr, nullptr, nullptr, T, top_k, standard, 0.f, w, shared, nullptr, nullptr, &bytes, nullptr) == DST_OK ? bytes : 0;
}

extern "C" int dst_moe_layer(const void* x_bf16, const float* weights, const int32_t* ids, int64_t T, int top_k, int standard, float limit,
                             const dst_expert_weights* w, const dst_expert_weights* shared, void* y_bf16, void* workspace, size_t workspace_bytes,
                             dst_stream_t stream) {
  size_t need = 0;
  const int rc = dst::layer(nullptr, nullptr, nullptr, T, top_k, standard, limit, w, shared, nullptr, nullptr, &need, nullptr);
  if (rc != DST_OK) return rc;
  if (T > 0 && (workspace == nullptr || workspace_bytes < need)) return DST_ERR_BAD_ARG;
  return dst::layer(x_bf16, weights, ids, T, top_k, standard, limit, w, shared, y_bf16, workspace, nullptr, static_cast<cudaStream_t>(stream));
}
