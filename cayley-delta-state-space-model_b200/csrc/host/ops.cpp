// Operator calls: checks, outputs, one C-ABI call each.
#include "host.h"

#include <map>
#include <mutex>
#include <tuple>

namespace cdssm_host {

PyObject* g_error_type = nullptr;

void check(int rc, const char* what) {
    if (rc == CDSSM_OK) return;
    std::string msg = std::string(what) + ": ";
    switch (rc) {
        case CDSSM_ERR_BAD_ARG: msg += "bad argument (null pointer, non-positive size, odd state_dim, misaligned buffer)"; break;
        case CDSSM_ERR_UNSUPPORTED: msg += "unsupported size (state_dim > 32, head_dim > 128, chunk > 256, ...)"; break;
        case CDSSM_ERR_WORKSPACE: msg += "workspace missing, misaligned or too small"; break;
        case CDSSM_ERR_CUDA: msg += "CUDA runtime error (cudaError " + std::to_string(cdssm_b200_last_cuda_error()) + ")"; break;
        case CDSSM_ERR_TIMEOUT: msg += "device-side wait timed out"; break;
        default: msg += "error " + std::to_string(rc);
    }
    throw Error(msg);
}

namespace {
struct Buffer {
    std::mutex launching;   // held while a call's kernels are put on the stream: two threads may share one
    Tensor memory;
};
std::mutex g_ws_mutex;
// never destroyed: the tensors must not outlive the CUDA context at process exit
Buffer& buffer_of(const std::pair<int, void*>& key) {
    static auto* m = new std::map<std::pair<int, void*>, Buffer>();
    std::lock_guard<std::mutex> lock(g_ws_mutex);
    return (*m)[key];
}
}  // namespace

Workspace workspace(const Tensor& on, size_t bytes) {
    Buffer& b = buffer_of({on.device().index(), stream_of(on)});
    std::unique_lock<std::mutex> hold(b.launching);
    if (!b.memory.defined() || (size_t)b.memory.numel() < bytes + 256)
        b.memory = at::empty({(int64_t)bytes + 512}, on.options().dtype(at::kByte));
    const uintptr_t p = reinterpret_cast<uintptr_t>(b.memory.data_ptr());
    const size_t off = (size_t)(-p & 255);
    return {reinterpret_cast<void*>(p + off), (size_t)b.memory.numel() - off, std::move(hold)};
}

void* workspace_if_any(int device) {
    Buffer& b = buffer_of({device, c10::cuda::getCurrentCUDAStream(device).stream()});
    std::lock_guard<std::mutex> hold(b.launching);
    if (!b.memory.defined()) return nullptr;
    const uintptr_t p = reinterpret_cast<uintptr_t>(b.memory.data_ptr());
    return reinterpret_cast<void*>(p + (size_t)(-p & 255));
}

ScanOut scan_fused(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& gate_, const Tensor& lds_,
                   const Tensor& rope_, const Dyn& dyn, int64_t heads, int64_t N, int64_t C, const Tensor& h0_,
                   double shortcut, int64_t pos0, bool want_tail, int64_t flags, const Tensor& out, int64_t segs) {
    need_cuda(q_, "q");
    const int dt = dtype_code(q_);
    const Tensor q = q_.is_contiguous() ? q_ : q_.contiguous();
    const Tensor k = dense(k_, q.scalar_type(), "k"), v = dense(v_, q.scalar_type(), "v");
    const Tensor g = dense(gate_, q.scalar_type(), "gate_raw");
    if (q.dim() != 4) throw Error("scan_fused: inconsistent shapes");
    const int64_t B = q.size(0), L = q.size(1), H = q.size(2), D = q.size(3);
    if (H != heads || k.sizes() != q.sizes() || v.sizes() != at::IntArrayRef({B, L, H, N}) ||
        g.sizes() != at::IntArrayRef({B, L, (N + 5) * H}))
        throw Error("scan_fused: inconsistent shapes");
    const Tensor lds = f32_vector(lds_, "log_dt_scale"), rope = f32_vector(rope_, "rope_freqs");
    Tensor h0;
    if (h0_.defined()) {
        h0 = dense(h0_, at::kFloat, "h0");
        if (h0.sizes() != at::IntArrayRef({B, H, N, D})) throw Error("h0 must be (B,H,N,D)");
    }
    ScanOut o;
    if (out.defined()) {
        if (out.sizes() != at::IntArrayRef({B, L, H, N}) || out.scalar_type() != q.scalar_type() || !out.is_contiguous())
            throw Error("out must be a contiguous (B,L,H,N) tensor of the input dtype");
        o.y = out;
    }
    const c10::cuda::CUDAGuard guard(q.device());
    if (!o.y.defined()) o.y = empty_like_dims({B, L, H, N}, q);
    o.final_state = empty_f32({B, H, N, D}, q);
    if (want_tail) o.tail = empty_f32({B, H, N, D}, q);
    if (B * L == 0) {   // nothing to scan: the carry passes through
        if (h0.defined()) o.final_state.copy_(h0);
        else o.final_state.zero_();
        if (want_tail) o.tail.copy_(o.final_state);
        return o;
    }
    // (a call that reuses a summary's results asks for what the summary asked for: the buffer must not move)
    const int for_flags = flags & CDSSM_SCAN_REUSE_LOCAL ? 0 : (int)flags;
    const Workspace ws = workspace(q, cdssm_b200_scan_fused_workspace_bytes_for((int)B, (int)L, (int)H, (int)D, (int)N, (int)C, dt, for_flags));
    void* st = stream_of(q);
    if (segs == 1) {
        check(cdssm_b200_scan_fused_fwd(cptr(q), cptr(k), cptr(v), cptr(g), fptr(lds), fptr(rope), fptr(h0), mptr(o.y),
                                        fmut(o.final_state), fmut(o.tail), ws.ptr, ws.bytes, dyn.c[0], dyn.c[1], dyn.c[2],
                                        dyn.c[3], dyn.c[4], (float)shortcut, (int)B, (int)L, (int)H, (int)D, (int)N,
                                        (int)C, (int)pos0, dt, (int)flags, st),
              "scan_fused_fwd");
    } else {
        if (want_tail) throw Error("tail_state is not available for segmented batches");
        check(cdssm_b200_scan_fused_segmented_fwd(cptr(q), cptr(k), cptr(v), cptr(g), fptr(lds), fptr(rope), fptr(h0),
                                                  mptr(o.y), fmut(o.final_state), ws.ptr, ws.bytes, dyn.c[0], dyn.c[1],
                                                  dyn.c[2], dyn.c[3], dyn.c[4], (float)shortcut, (int)B, (int)L, (int)H,
                                                  (int)D, (int)N, (int)C, (int)pos0, (int)segs, dt, (int)flags, st),
              "scan_fused_segmented_fwd");
    }
    return o;
}

// Rows dense inside; only the batch stride may be larger (a column slice of a projection).  Anything else: a dense copy.
static Tensor rows(const Tensor& t, at::ScalarType dt, int64_t n_rows, int64_t inner, const char* name) {
    if (t.is_cuda() && t.scalar_type() == dt && t.dim() > 0 && t.size(0) == n_rows) {
        bool ok = true;
        int64_t run = 1;
        for (int64_t i = t.dim() - 1; i > 0; i--) {
            ok = ok && t.stride(i) == run;
            run *= t.size(i);
        }
        ok = ok && run == inner && t.stride(0) >= inner && (t.stride(0) * t.element_size()) % 16 == 0 &&
             (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15) == 0;
        if (ok) return t;
    }
    return dense(t, dt, name);
}

// One long sequence per batch row, cut into S chunk-aligned segments: summaries of all segments, their carries in series, the
// scan of all segments as a batch on the local results the summaries have left in the workspace.
std::array<Tensor, 2> scan_fused_long(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& gate_, const Tensor& lds_,
                                      const Tensor& rope_, const Dyn& dyn, int64_t heads, int64_t N, int64_t C, const Tensor& h0_,
                                      double shortcut, int64_t pos0, int64_t flags, int64_t S) {
    need_cuda(q_, "q");
    const int dt = dtype_code(q_);
    const Tensor q = q_.is_contiguous() ? q_ : q_.contiguous();
    const Tensor k = dense(k_, q.scalar_type(), "k"), v = dense(v_, q.scalar_type(), "v");
    const Tensor g = dense(gate_, q.scalar_type(), "gate_raw");
    need_dims(q, 4, "q");
    const int64_t B = q.size(0), L = q.size(1), H = q.size(2), D = q.size(3), R = B * S, Ls = L / S;
    if (H != heads || k.sizes() != q.sizes() || v.sizes() != at::IntArrayRef({B, L, H, N}) ||
        g.sizes() != at::IntArrayRef({B, L, (N + 5) * H}))
        throw Error("scan_fused_long: inconsistent shapes");
    const Tensor lds = f32_vector(lds_, "log_dt_scale"), rope = f32_vector(rope_, "rope_freqs");
    Tensor h0;
    if (h0_.defined()) {
        h0 = dense(h0_, at::kFloat, "h0");
        if (h0.numel() != B * H * N * D) throw Error("h0 must be (B,H,N,D)");
    }
    const c10::cuda::CUDAGuard guard(q.device());
    const Tensor y = empty_like_dims({B, L, H, N}, q), final_state = empty_f32({B, H, N, D}, q);
    // carries out of and into the segments, the segments' last carries (not handed out), their decays and the whole one
    const int64_t st_n = (R * H * N * D + 63) & ~63, dc_n = R * H * N;
    const Tensor scratch = empty_f32({3 * st_n + dc_n + B * H * N}, q);
    float* carry = fmut(scratch);
    float *carry_in = carry + st_n, *last = carry_in + st_n, *decay = last + st_n, *total = decay + dc_n;
    const Workspace ws = workspace(q, cdssm_b200_scan_fused_workspace_bytes_for((int)R, (int)Ls, (int)H, (int)D, (int)N, (int)C, dt, (int)flags));
    void* st = stream_of(q);
    check(cdssm_b200_scan_summary_fwd(cptr(k), cptr(v), cptr(g), fptr(lds), fptr(rope), nullptr, carry, decay, ws.ptr, ws.bytes,
                                      dyn.c[0], dyn.c[1], dyn.c[2], dyn.c[3], dyn.c[4], (int)R, (int)Ls, (int)H, (int)D, (int)N,
                                      (int)C, (int)pos0, (int)S, dt, (int)flags & CDSSM_SCAN_FP32_DECAY, st),
          "scan_summary_fwd");
    check(cdssm_b200_compose_carries(decay, carry, fptr(h0), carry_in, fmut(final_state), total, (int)B, (int)S, (int)H, (int)D,
                                     (int)N, S, 1, st),
          "compose_carries");
    check(cdssm_b200_scan_fused_segmented_fwd(cptr(q), cptr(k), cptr(v), cptr(g), fptr(lds), fptr(rope), carry_in, mptr(y), last,
                                              ws.ptr, ws.bytes, dyn.c[0], dyn.c[1], dyn.c[2], dyn.c[3], dyn.c[4], (float)shortcut,
                                              (int)R, (int)Ls, (int)H, (int)D, (int)N, (int)C, (int)pos0, (int)S, dt,
                                              (int)flags | CDSSM_SCAN_REUSE_LOCAL, st),
          "scan_fused_segmented_fwd");
    return {y, final_state};
}

Tensor decode_step(const Tensor& state, const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& gate_,
                   const Tensor& lds_, const Tensor& rope_, const Dyn& dyn, int64_t heads, int64_t N, int64_t pos,
                   const Tensor& pos_dev, double shortcut, const Tensor& out, const Tensor& v_first_, const Tensor& mix_) {
    need_cuda(q_, "q");
    if (q_.dim() != 3) throw Error("decode_step: inconsistent shapes");
    const int64_t B = q_.size(0), H = q_.size(1), D = q_.size(2);
    const auto dt = q_.scalar_type();
    const int code = dtype_code(q_);
    const Tensor q = rows(q_, dt, B, H * D, "q"), k = rows(k_, dt, B, H * D, "k"), v = rows(v_, dt, B, H * N, "v");
    const Tensor g = rows(gate_, dt, B, (N + 5) * H, "gate_raw");
    if (!state.is_cuda() || state.scalar_type() != at::kFloat || !state.is_contiguous())
        throw Error("state must be a contiguous float32 CUDA tensor (B,H,N,D)");
    if (H != heads || state.sizes() != at::IntArrayRef({B, H, N, D}) || k.sizes() != at::IntArrayRef({B, H, D}) ||
        v.sizes() != at::IntArrayRef({B, H, N}) || g.sizes() != at::IntArrayRef({B, (N + 5) * H}))
        throw Error("decode_step: inconsistent shapes");
    if (v_first_.defined() != mix_.defined()) throw Error("decode_step: v_first and mix go together");
    Tensor v_first, mix;
    if (v_first_.defined()) {
        v_first = dense(v_first_, dt, "v_first");
        mix = dense(mix_.reshape({-1}), dt, "mix");
        if (v_first.sizes() != at::IntArrayRef({B, H, N}) || mix.numel() != H)
            throw Error("decode_step: v_first must be (B,H,N) and mix (H)");
    }
    const Tensor lds = f32_vector(lds_, "log_dt_scale"), rope = f32_vector(rope_, "rope_freqs");
    if (pos_dev.defined() && (pos_dev.scalar_type() != at::kInt || !pos_dev.is_cuda()))
        throw Error("a tensor position must be an int32 CUDA tensor");   // device memory: graph-replayable
    const c10::cuda::CUDAGuard guard(q.device());
    const Tensor y = out.defined() ? out : empty_like_dims({B, H, N}, q);
    check(cdssm_b200_decode_step_strided(fmut(state), cptr(q), q.stride(0), cptr(k), k.stride(0), cptr(v), v.stride(0),
                                         cptr(v_first), cptr(mix), cptr(g), g.stride(0), fptr(lds), fptr(rope), mptr(y),
                                         dyn.c[0], dyn.c[1], dyn.c[2], dyn.c[3], dyn.c[4], (float)shortcut, (int)B, (int)H,
                                         (int)D, (int)N, (int)pos, static_cast<const int*>(cptr(pos_dev)), code, stream_of(q)),
          "decode_step");
    return y;
}

Tensor rms_norm(const Tensor& x_, const Tensor& w_, double eps) {
    need_cuda(x_, "x");
    const Tensor x = x_.is_contiguous() ? x_ : x_.contiguous(), w = dense(w_, x.scalar_type(), "weight");
    const int64_t d = x.size(-1);
    if (d == 0) throw Error("rms_norm: the last dimension is empty");
    const c10::cuda::CUDAGuard guard(x.device());
    const Tensor out = at::empty_like(x);
    check(cdssm_b200_rmsnorm_fwd(cptr(x), cptr(w), mptr(out), x.numel() / d, (int)d, (float)eps, dtype_code(x), stream_of(x)),
          "rmsnorm_fwd");
    return out;
}

Tensor groupnorm_gate(const Tensor& y_, const Tensor& gw_, const Tensor& gb_, const Tensor& z_, const Tensor& skip_,
                      const Tensor& x_conv, int64_t groups, double eps, bool per_token) {
    need_cuda(y_, "y");
    const Tensor y = y_.is_contiguous() ? y_ : y_.contiguous();
    const auto dt = y.scalar_type();
    const Tensor xc = dense(x_conv, dt, "x_conv");
    need_dims(y, 3, "y");
    const int64_t B = y.size(0), L = y.size(1), di = y.size(2);
    Tensor z = z_;
    if (!z.is_cuda() || z.scalar_type() != dt || z.sizes() != y.sizes() || z.stride(-1) != 1 ||
        (L > 1 && z.stride(0) != L * z.stride(1)))
        z = z.contiguous();
    int64_t zs = L > 1 ? z.stride(1) : (B > 1 ? z.stride(0) : di);
    if ((zs * z.element_size()) % 16 || (reinterpret_cast<uintptr_t>(z.const_data_ptr()) & 15)) {   // 16-byte pieces
        z = z.contiguous();
        zs = di;
    }
    const Tensor gw = dense(gw_, dt, "groupnorm parameter"), gb = dense(gb_, dt, "groupnorm parameter"),
                 sk = dense(skip_, dt, "groupnorm parameter");
    const c10::cuda::CUDAGuard guard(y.device());
    const Tensor out = at::empty_like(y);
    void* st = stream_of(y);
    const int code = dtype_code(y);
    Tensor stats;
    if (!per_token) {
        stats = empty_f32({(int64_t)cdssm_b200_groupnorm_stats_floats((int)B, (int)L, (int)groups)}, y);   // results, then scratch
        check(cdssm_b200_groupnorm_stats(cptr(y), fmut(stats), (int)B, (int)L, (int)di, (int)groups, (float)eps, code, st),
              "groupnorm_stats");
    }
    check(cdssm_b200_groupnorm_gate_fwd(cptr(y), fptr(stats), cptr(gw), cptr(gb), cptr(z), zs, cptr(sk), cptr(xc), mptr(out),
                                        (int)B, (int)L, (int)di, (int)groups, (float)eps, code, st),
          "groupnorm_gate_fwd");
    return out;
}

Tensor conv1d_silu(const Tensor& x_, const Tensor& w_, const Tensor& b_) {
    need_cuda(x_, "x");
    const Tensor x = x_.is_contiguous() ? x_ : x_.contiguous();
    need_dims(x, 3, "x");
    const Tensor w = dense(w_.detach().to(x.scalar_type()), x.scalar_type(), "weight");
    const Tensor b = dense(b_.detach().to(x.scalar_type()), x.scalar_type(), "bias");
    const c10::cuda::CUDAGuard guard(x.device());
    const Tensor out = at::empty_like(x);
    check(cdssm_b200_conv1d_silu_fwd(cptr(x), cptr(w), cptr(b), mptr(out), (int)x.size(0), (int)x.size(1), (int)x.size(2),
                                     dtype_code(x), stream_of(x)),
          "conv1d_silu_fwd");
    return out;
}

Tensor conv1d_silu_step(const Tensor& x_, const Tensor& hist, const Tensor& w_, const Tensor& b_) {
    const Tensor x = !x_.is_cuda() || x_.stride(-1) != 1 ? x_.contiguous() : x_;
    need_cuda(x, "x");
    need_dims(x, 2, "x");
    const int64_t B = x.size(0), Dm = x.size(1);
    if (hist.scalar_type() != x.scalar_type() || !hist.is_contiguous() || hist.sizes() != at::IntArrayRef({B, 3, Dm}))
        throw Error("conv1d_silu_step: hist must be a contiguous (B,3,Dm) tensor of the input dtype");
    const Tensor w = dense(w_, x.scalar_type(), "weight"), b = dense(b_, x.scalar_type(), "bias");
    const c10::cuda::CUDAGuard guard(x.device());
    const Tensor out = empty_like_dims({B, Dm}, x);
    check(cdssm_b200_conv1d_silu_step(cptr(x), B > 1 ? x.stride(0) : Dm, mptr(hist), cptr(w), cptr(b), mptr(out), (int)B,
                                      (int)Dm, dtype_code(x), stream_of(x)),
          "conv1d_silu_step");
    return out;
}

// ------------------------------------------------------------------------------------------ Python entry points
namespace {

PyObject* py_decode_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        Args in{a, n};
        const Tensor state = in.tensor("state"), q = in.tensor("q"), k = in.tensor("k"), v = in.tensor("v"),
                     g = in.tensor("gate_raw"), lds = in.tensor("log_dt_scale"), rope = in.tensor("rope_freqs");
        const Dyn dyn = in.dyn();
        const int64_t H = in.integer(), N = in.integer();
        Tensor pos_dev;
        int64_t pos = 0;
        if (in.at < n && THPVariable_Check(a[in.at])) pos_dev = in.tensor("pos");
        else pos = in.integer();
        const double shortcut = in.number();
        const Tensor out = in.tensor_or_none("out"), v_first = in.tensor_or_none("v_first"), mix = in.tensor_or_none("mix");
        return wrap(without_gil([&] {
            return decode_step(state, q, k, v, g, lds, rope, dyn, H, N, pos, pos_dev, shortcut, out, v_first, mix);
        }));
    });
}

PyObject* py_scan_fused(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        Args in{a, n};
        const Tensor q = in.tensor("q"), k = in.tensor("k"), v = in.tensor("v"), g = in.tensor("gate_raw"),
                     lds = in.tensor("log_dt_scale"), rope = in.tensor("rope_freqs");
        const Dyn dyn = in.dyn();
        const int64_t H = in.integer(), N = in.integer(), C = in.integer();
        const Tensor h0 = in.tensor_or_none("h0");
        const double shortcut = in.number();
        const int64_t pos0 = in.integer();
        const bool tail = in.flag();
        const int64_t flags = in.integer();
        const Tensor out = in.tensor_or_none("out");
        const int64_t segs = in.integer();
        ScanOut o = without_gil([&] {
            return scan_fused(q, k, v, g, lds, rope, dyn, H, N, C, h0, shortcut, pos0, tail, flags, out, segs);
        });
        PyObject* t = PyTuple_New(tail ? 3 : 2);
        if (!t) return nullptr;
        PyTuple_SET_ITEM(t, 0, wrap(o.y));
        PyTuple_SET_ITEM(t, 1, wrap(o.final_state));
        if (tail) PyTuple_SET_ITEM(t, 2, wrap(o.tail));
        return t;
    });
}

// scan_fused_long(q, k, v, gate_raw, log_dt_scale, rope_freqs, five dynamics scalars, n_heads, state_dim, chunk_size, h0 or None,
//                 shortcut_scale, pos0, flags, segments) -> (y, final_state)
PyObject* py_scan_fused_long(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        Args in{a, n};
        const Tensor q = in.tensor("q"), k = in.tensor("k"), v = in.tensor("v"), g = in.tensor("gate_raw");
        const Tensor lds = in.tensor("log_dt_scale"), rope = in.tensor("rope_freqs");
        const Dyn dyn = in.dyn();
        const int64_t H = in.integer(), N = in.integer(), C = in.integer();
        const Tensor h0 = in.tensor_or_none("h0");
        const double shortcut = in.number();
        const int64_t pos0 = in.integer(), flags = in.integer(), S = in.integer();
        const auto o = without_gil([&] { return scan_fused_long(q, k, v, g, lds, rope, dyn, H, N, C, h0, shortcut, pos0, flags, S); });
        PyObject* t = PyTuple_New(2);
        if (!t) return nullptr;
        PyTuple_SET_ITEM(t, 0, wrap(o[0]));
        PyTuple_SET_ITEM(t, 1, wrap(o[1]));
        return t;
    });
}

PyObject* py_rms_norm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        Args in{a, n};
        const Tensor x = in.tensor("x"), w = in.tensor("weight");
        const double eps = in.number();
        return wrap(without_gil([&] { return rms_norm(x, w, eps); }));
    });
}

PyObject* py_groupnorm_gate(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        Args in{a, n};
        const Tensor y = in.tensor("y"), gw = in.tensor("gn_weight"), gb = in.tensor("gn_bias"), z = in.tensor("z"),
                     sk = in.tensor("skip"), xc = in.tensor("x_conv");
        const int64_t groups = in.integer();
        const double eps = in.number();
        const bool per_token = in.flag();
        return wrap(without_gil([&] { return groupnorm_gate(y, gw, gb, z, sk, xc, groups, eps, per_token); }));
    });
}

PyObject* py_conv1d_silu_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        Args in{a, n};
        const Tensor x = in.tensor("x"), hist = in.tensor("hist"), w = in.tensor("weight"), b = in.tensor("bias");
        return wrap(without_gil([&] { return conv1d_silu_step(x, hist, w, b); }));
    });
}

// workspace(tensor on the device, bytes) -> (address, usable bytes)
PyObject* py_workspace(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        Args in{a, n};
        const Tensor on = in.tensor("tensor");
        const size_t bytes = (size_t)in.integer();
        const Workspace w = without_gil([&] { return workspace(on, bytes); });
        return Py_BuildValue("(Kn)", (unsigned long long)reinterpret_cast<uintptr_t>(w.ptr), (Py_ssize_t)w.bytes);
    });
}

// workspace_address(device index) -> address of the current stream's buffer, 0 if there is none
PyObject* py_workspace_address(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        Args in{a, n};
        const int device = (int)in.integer();
        return PyLong_FromUnsignedLongLong(reinterpret_cast<uintptr_t>(without_gil([&] { return workspace_if_any(device); })));
    });
}

PyObject* py_set_error_type(PyObject*, PyObject* t) {
    Py_INCREF(t);
    Py_XSETREF(g_error_type, t);
    Py_RETURN_NONE;
}

#define FAST(fn) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(fn)), METH_FASTCALL, nullptr
PyMethodDef g_methods[] = {
    {"decode_step", FAST(py_decode_step)},
    {"scan_fused", FAST(py_scan_fused)},
    {"scan_fused_long", FAST(py_scan_fused_long)},
    {"rms_norm", FAST(py_rms_norm)},
    {"groupnorm_gate", FAST(py_groupnorm_gate)},
    {"conv1d_silu_step", FAST(py_conv1d_silu_step)},
    {"workspace", FAST(py_workspace)},
    {"workspace_address", FAST(py_workspace_address)},
    {"set_error_type", py_set_error_type, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_cdssm_host", "Native host path of the CD-SSM operators.", -1, g_methods,
                        nullptr, nullptr, nullptr, nullptr};

}  // namespace
}  // namespace cdssm_host

PyMODINIT_FUNC PyInit__cdssm_host() {
    PyObject* m = PyModule_Create(&cdssm_host::g_module);
    if (m && (PyModule_AddFunctions(m, cdssm_host::model_methods()) < 0 || PyModule_AddFunctions(m, cdssm_host::train_methods()) < 0)) {
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}
