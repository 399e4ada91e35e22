// The six operators of cdssm/ops.py, forward and backward, one native call each: issued through ctypes with their checks and
// allocations in Python a call took some 40 us of host time, and a block's forward and backward makes twelve.
#include "host.h"

namespace cdssm_host {
namespace {

// Contiguous CUDA tensor (of type dt if given), with the operator's message otherwise.
Tensor prep(const Tensor& t, const char* name) {
    need_cuda(t, name);
    return t.is_contiguous() ? t : t.contiguous();
}
Tensor grad_or_zeros(const Tensor& t, at::IntArrayRef sizes, const Tensor& like) {
    if (!t.defined()) return at::zeros(sizes, like.options());
    return prep(t.scalar_type() == like.scalar_type() ? t : t.to(like.scalar_type()), "upstream gradient");
}
Tensor cast(const Tensor& t, at::ScalarType dt) { return t.scalar_type() == dt ? t : t.to(dt); }

template <size_t n>
PyObject* tuple_of(std::array<Tensor, n> ts) {
    PyObject* t = PyTuple_New(n);
    if (!t) return nullptr;
    for (size_t i = 0; i < n; i++) PyTuple_SET_ITEM(t, i, wrap(std::move(ts[i])));
    return t;
}

// conv_fwd(x, weight, bias) -> (out, x, w, b): dense inputs as the backward wants them
PyObject* py_conv_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        Args in{a, n};
        const Tensor x = prep(in.tensor("x"), "x"), weight = in.tensor("weight"), bias = in.tensor("bias");
        if (weight.size(-1) != 4) throw Error("Only kernel_size=4 is supported");   // conv1d_silu.cu:241
        need_dims(x, 3, "x");
        const int64_t B = x.size(0), L = x.size(1), Dm = x.size(2);
        const Tensor w = prep(cast(weight.detach(), x.scalar_type()), "weight").reshape({Dm, 4});
        const Tensor b = prep(cast(bias.detach(), x.scalar_type()), "bias");
        return tuple_of<4>(without_gil([&]() -> std::array<Tensor, 4> {
            const c10::cuda::CUDAGuard guard(x.device());
            const Tensor out = at::empty_like(x);
            check(cdssm_b200_conv1d_silu_fwd(cptr(x), cptr(w), cptr(b), mptr(out), (int)B, (int)L, (int)Dm, dtype_code(x), stream_of(x)),
                  "conv1d_silu_fwd");
            return {out, x, w, b};
        }));
    });
}

// conv_bwd(grad_out, x, w, b) -> (grad_x, grad_w (Dm,4) float32, grad_b float32)
PyObject* py_conv_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        Args in{a, n};
        const Tensor g_ = in.tensor("grad_out"), x = in.tensor("x"), w = in.tensor("w"), b = in.tensor("b");
        const Tensor go = prep(cast(g_, x.scalar_type()), "grad_out");
        return tuple_of<3>(without_gil([&]() -> std::array<Tensor, 3> {
            const c10::cuda::CUDAGuard guard(x.device());
            const int64_t Dm = x.size(2);
            const Tensor gx = at::empty_like(x), gw = empty_f32({Dm, 4}, x), gb = empty_f32({Dm}, x);
            check(cdssm_b200_conv1d_silu_bwd(cptr(go), cptr(x), cptr(w), cptr(b), mptr(gx), fmut(gw), fmut(gb), (int)x.size(0),
                                             (int)x.size(1), (int)Dm, dtype_code(x), stream_of(x)),
                  "conv1d_silu_bwd");
            return {gx, gw, gb};
        }));
    });
}

// dynamics_fwd(gate_raw, log_dt_scale, rope_freqs, c0..c4, H, N) -> (A, vp, beta, sel_C, gate, lds, rope)
PyObject* py_dynamics_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        Args in{a, n};
        const Tensor g = prep(in.tensor("gate_raw"), "gate_raw"), lds_ = in.tensor("log_dt_scale"), rope_ = in.tensor("rope_freqs");
        const Dyn d = in.dyn();
        need_dims(g, 3, "gate_raw");
        const int64_t H = in.integer(), N = in.integer(), B = g.size(0), L = g.size(1);
        if (g.size(2) != (N + 5) * H)
            throw Error("gate_raw last dim " + std::to_string(g.size(2)) + " != (state_dim+5)*n_heads = " + std::to_string((N + 5) * H));
        const Tensor lds = f32_vector(lds_, "log_dt_scale"), rope = f32_vector(rope_, "rope_freqs");
        return tuple_of<7>(without_gil([&]() -> std::array<Tensor, 7> {
            const c10::cuda::CUDAGuard guard(g.device());
            const Tensor A = empty_like_dims({B, L, H, N}, g), vp = empty_like_dims({B, L, H, N / 2}, g);
            const Tensor beta = empty_like_dims({B, L, H}, g), sel = empty_like_dims({B, L, H}, g);
            check(cdssm_b200_dynamics_fwd(cptr(g), fptr(lds), fptr(rope), mptr(A), mptr(vp), mptr(beta), mptr(sel), d.c[0], d.c[1], d.c[2],
                                          d.c[3], d.c[4], (int)B, (int)L, (int)H, (int)N, 0, dtype_code(g), stream_of(g)),
                  "dynamics_fwd");
            return {A, vp, beta, sel, g, lds, rope};
        }));
    });
}

// dynamics_bwd(gA, gvp, gbeta, gsel (each or None), gate, lds, rope, c0..c4, H, N) -> (grad_gate, grad_lds float32)
PyObject* py_dynamics_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        Args in{a, n};
        const Tensor gA_ = in.tensor_or_none("grad_A_bar"), gvp_ = in.tensor_or_none("grad_vp_scale"), gb_ = in.tensor_or_none("grad_beta"),
                     gc_ = in.tensor_or_none("grad_sel_C"), g = in.tensor("gate"), lds = in.tensor("lds"), rope = in.tensor("rope");
        const Dyn d = in.dyn();
        const int64_t H = in.integer(), N = in.integer(), B = g.size(0), L = g.size(1);
        return tuple_of<2>(without_gil([&]() -> std::array<Tensor, 2> {
            const c10::cuda::CUDAGuard guard(g.device());
            const Tensor gA = grad_or_zeros(gA_, {B, L, H, N}, g), gvp = grad_or_zeros(gvp_, {B, L, H, N / 2}, g);
            const Tensor gb = grad_or_zeros(gb_, {B, L, H}, g), gc = grad_or_zeros(gc_, {B, L, H}, g);
            const Tensor gg = at::empty_like(g), gl = empty_f32({H}, g);
            check(cdssm_b200_dynamics_bwd(cptr(gA), cptr(gvp), cptr(gb), cptr(gc), cptr(g), fptr(lds), fptr(rope), mptr(gg), fmut(gl), d.c[0],
                                          d.c[1], d.c[2], d.c[3], d.c[4], (int)B, (int)L, (int)H, (int)N, 0, dtype_code(g), stream_of(g)),
                  "dynamics_bwd");
            return {gg, gl};
        }));
    });
}

// normalize_fwd(K, Q) -> (Ko, Qo, K, Q)
PyObject* py_normalize_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        Args in{a, n};
        const Tensor K = prep(in.tensor("K"), "K"), Q = dense(in.tensor("Q"), K.scalar_type(), "Q");
        if (K.sizes() != Q.sizes()) throw Error("K and Q must have the same shape");
        const int64_t D = K.size(-1);
        if (D == 0) throw Error("K and Q: the last dimension is empty");
        return tuple_of<4>(without_gil([&]() -> std::array<Tensor, 4> {
            const c10::cuda::CUDAGuard guard(K.device());
            const Tensor Ko = at::empty_like(K), Qo = at::empty_like(Q);
            check(cdssm_b200_normalize_kq_fwd(cptr(K), cptr(Q), mptr(Ko), mptr(Qo), K.numel() / D, (int)D, dtype_code(K), stream_of(K)),
                  "normalize_kq_fwd");
            return {Ko, Qo, K, Q};
        }));
    });
}

// normalize_bwd(gKo, gQo (each or None), K, Q) -> (gK, gQ)
PyObject* py_normalize_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        Args in{a, n};
        const Tensor gk_ = in.tensor_or_none("grad_K_out"), gq_ = in.tensor_or_none("grad_Q_out"), K = in.tensor("K"), Q = in.tensor("Q");
        const int64_t D = K.size(-1);
        return tuple_of<2>(without_gil([&]() -> std::array<Tensor, 2> {
            const c10::cuda::CUDAGuard guard(K.device());
            const Tensor gKo = grad_or_zeros(gk_, K.sizes(), K), gQo = grad_or_zeros(gq_, K.sizes(), K);
            const Tensor gK = at::empty_like(K), gQ = at::empty_like(Q);
            check(cdssm_b200_normalize_kq_bwd(cptr(gKo), cptr(gQo), cptr(K), cptr(Q), mptr(gK), mptr(gQ), K.numel() / D, (int)D,
                                              dtype_code(K), stream_of(K)),
                  "normalize_kq_bwd");
            return {gK, gQ};
        }));
    });
}

// intra_fwd(A, K, V, beta, N) -> (local_h, cum_A, A, K, V, beta)
PyObject* py_intra_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        Args in{a, n};
        const Tensor A_ = in.tensor("A_flat"), K = prep(in.tensor("K_flat"), "K_flat"), V_ = in.tensor("V_flat"), b_ = in.tensor("beta_flat");
        const auto dt = K.scalar_type();
        const Tensor A = dense(A_, dt, "A_flat"), V = dense(V_, dt, "V_flat"), be = dense(b_, dt, "beta_flat");
        need_dims(K, 4, "K_flat");
        const int64_t N = in.integer(), M = K.size(0), C = K.size(1), H = K.size(2), D = K.size(3);
        return tuple_of<6>(without_gil([&]() -> std::array<Tensor, 6> {
            const c10::cuda::CUDAGuard guard(K.device());
            const Tensor h = empty_like_dims({M, C, H, N, D}, K), cum = empty_like_dims({M, C, H, N}, K);
            check(cdssm_b200_intra_chunk_scan_fwd(cptr(A), cptr(K), cptr(V), cptr(be), mptr(h), mptr(cum), (int)M, (int)C, (int)H, (int)D,
                                                  (int)N, dtype_code(K), stream_of(K)),
                  "intra_chunk_scan_fwd");
            return {h, cum, A, K, V, be};
        }));
    });
}

// intra_bwd(grad_local_h, grad_cum_A (each or None), A, K, V, beta, local_h, cum_A, N) -> (gA, gK, gV, gB)
PyObject* py_intra_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        Args in{a, n};
        const Tensor gh_ = in.tensor_or_none("grad_local_h"), gc_ = in.tensor_or_none("grad_cum_A"), A = in.tensor("A"), K = in.tensor("K"),
                     V = in.tensor("V"), be = in.tensor("beta"), h = in.tensor("local_h"), cum = in.tensor("cum_A");
        const int64_t N = in.integer(), M = K.size(0), C = K.size(1), H = K.size(2), D = K.size(3);
        return tuple_of<4>(without_gil([&]() -> std::array<Tensor, 4> {
            const c10::cuda::CUDAGuard guard(K.device());
            const Tensor gh = grad_or_zeros(gh_, h.sizes(), K), gc = grad_or_zeros(gc_, cum.sizes(), K);
            const Tensor gA = at::empty_like(A), gV = at::empty_like(V), gK = empty_f32({M, C, H, D}, K), gB = empty_f32({M, C, H}, K);
            check(cdssm_b200_intra_chunk_scan_bwd(cptr(gh), cptr(gc), cptr(A), cptr(K), cptr(V), cptr(be), cptr(h), cptr(cum), mptr(gA),
                                                  fmut(gK), mptr(gV), fmut(gB), (int)M, (int)C, (int)H, (int)D, (int)N, dtype_code(K),
                                                  stream_of(K)),
                  "intra_chunk_scan_bwd");
            return {gA, cast(gK, K.scalar_type()), gV, cast(gB, K.scalar_type())};
        }));
    });
}

// inter_fwd(total_A, final_local_h, N) -> (chunk_states, total_A)
PyObject* py_inter_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        Args in{a, n};
        const Tensor A_ = in.tensor("total_A"), f = prep(in.tensor("final_local_h"), "final_local_h"), A = dense(A_, f.scalar_type(), "total_A");
        need_dims(f, 5, "final_local_h");
        const int64_t N = in.integer();
        return tuple_of<2>(without_gil([&]() -> std::array<Tensor, 2> {
            const c10::cuda::CUDAGuard guard(f.device());
            const Tensor out = at::empty_like(f);
            check(cdssm_b200_inter_chunk_scan_fwd(cptr(A), cptr(f), mptr(out), (int)f.size(0), (int)f.size(1), (int)f.size(2), (int)f.size(4),
                                                  (int)N, dtype_code(f), stream_of(f)),
                  "inter_chunk_scan_fwd");
            return {out, A};
        }));
    });
}

// inter_bwd(grad_chunk_states, total_A, chunk_states, N) -> (gA, gH)
PyObject* py_inter_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        Args in{a, n};
        const Tensor g_ = in.tensor("grad_chunk_states"), A = in.tensor("total_A"), s = in.tensor("chunk_states");
        const int64_t N = in.integer();
        const Tensor g = prep(cast(g_, s.scalar_type()), "grad_chunk_states");
        return tuple_of<2>(without_gil([&]() -> std::array<Tensor, 2> {
            const c10::cuda::CUDAGuard guard(s.device());
            const Tensor gA = at::empty_like(A), gH = at::empty_like(s);
            check(cdssm_b200_inter_chunk_scan_bwd(cptr(g), cptr(A), cptr(s), mptr(gA), mptr(gH), (int)s.size(0), (int)s.size(1), (int)s.size(2),
                                                  (int)s.size(4), (int)N, dtype_code(s), stream_of(s)),
                  "inter_chunk_scan_bwd");
            return {gA, gH};
        }));
    });
}

// correction_fwd(A, K, beta, chunk_states, N) -> (corrections, A, K, beta)
PyObject* py_correction_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        Args in{a, n};
        const Tensor A_ = in.tensor("A_chunk"), K = prep(in.tensor("K_chunk"), "K_chunk"), b_ = in.tensor("beta_chunk"), s_ = in.tensor("chunk_states");
        const auto dt = K.scalar_type();
        const Tensor A = dense(A_, dt, "A_chunk"), be = dense(b_, dt, "beta_chunk"), s = dense(s_, dt, "chunk_states");
        need_dims(K, 5, "K_chunk");
        const int64_t N = in.integer(), B = K.size(0), NC = K.size(1), C = K.size(2), H = K.size(3), D = K.size(4);
        return tuple_of<4>(without_gil([&]() -> std::array<Tensor, 4> {
            const c10::cuda::CUDAGuard guard(K.device());
            const Tensor out = empty_like_dims({B, NC, C, H, N, D}, K);
            check(cdssm_b200_exact_correction_fwd(cptr(A), cptr(K), cptr(be), cptr(s), mptr(out), (int)B, (int)NC, (int)C, (int)H, (int)D, (int)N,
                                                  dtype_code(K), stream_of(K)),
                  "exact_correction_fwd");
            return {out, A, K, be};
        }));
    });
}

// correction_bwd(grad_corrections, A, K, beta, corrections, N, reference_order) -> (gA, gK, gB, gS)
PyObject* py_correction_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&] {
        Args in{a, n};
        const Tensor g_ = in.tensor("grad_corrections"), A = in.tensor("A"), K = in.tensor("K"), be = in.tensor("beta"), c = in.tensor("corrections");
        const int64_t N = in.integer(), order = in.integer(), B = K.size(0), NC = K.size(1), C = K.size(2), H = K.size(3), D = K.size(4);
        const Tensor g = prep(cast(g_, K.scalar_type()), "grad_corrections");
        return tuple_of<4>(without_gil([&]() -> std::array<Tensor, 4> {
            const c10::cuda::CUDAGuard guard(K.device());
            const Tensor gA = at::empty_like(A), gK = empty_f32({B, NC, C, H, D}, K), gB = empty_f32({B, NC, C, H}, K);
            const Tensor gS = empty_like_dims({B, NC, H, N, D}, K);
            check(cdssm_b200_exact_correction_bwd(cptr(g), cptr(A), cptr(K), cptr(be), cptr(c), mptr(gA), fmut(gK), fmut(gB), mptr(gS), (int)B,
                                                  (int)NC, (int)C, (int)H, (int)D, (int)N, (int)order, dtype_code(K), stream_of(K)),
                  "exact_correction_bwd");
            return {gA, cast(gK, K.scalar_type()), cast(gB, K.scalar_type()), gS};
        }));
    });
}

#define FAST(fn) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(fn)), METH_FASTCALL, nullptr
PyMethodDef g_train_methods[] = {
    {"conv_fwd", FAST(py_conv_fwd)},           {"conv_bwd", FAST(py_conv_bwd)},
    {"dynamics_fwd", FAST(py_dynamics_fwd)},   {"dynamics_bwd", FAST(py_dynamics_bwd)},
    {"normalize_fwd", FAST(py_normalize_fwd)}, {"normalize_bwd", FAST(py_normalize_bwd)},
    {"intra_fwd", FAST(py_intra_fwd)},         {"intra_bwd", FAST(py_intra_bwd)},
    {"inter_fwd", FAST(py_inter_fwd)},         {"inter_bwd", FAST(py_inter_bwd)},
    {"correction_fwd", FAST(py_correction_fwd)}, {"correction_bwd", FAST(py_correction_bwd)},
    {nullptr, nullptr, 0, nullptr},
};

}  // namespace

PyMethodDef* train_methods() { return g_train_methods; }

}  // namespace cdssm_host
