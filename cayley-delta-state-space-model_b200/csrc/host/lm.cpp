// The language model's forward, prefill and one-token decode: one native call per pass.  Issued op by op from Python, a
// 12-layer decode step took 2.7 ms of host time around 0.39 ms of kernels and a 500-token prompt 4 ms around 1.8 ms.
// Layer structure as cdssm/models/block.py:140-229 (see model.py).
#include "host.h"

#include <c10/core/GradMode.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>

namespace cdssm_host {
namespace {

struct Weights {   // of a block, as the caller keeps them
    Tensor norm_w, w_in, b_in, conv_w, conv_b, w_gate, b_gate, lds, rope, w_q, w_readout, w_out, gn_w, gn_b, D, v_gate, w_qg,
        b_qg;
    static constexpr int kCount = 18;
    std::array<Tensor*, kCount> all() {
        return {&norm_w, &w_in, &b_in, &conv_w, &conv_b, &w_gate, &b_gate, &lds, &rope, &w_q, &w_readout, &w_out, &gn_w, &gn_b,
                &D, &v_gate, &w_qg, &b_qg};
    }
};
struct Block : Weights {
    double shortcut = 0.0;
    // views of the input projection's row blocks
    Tensor w_z, b_z, w_x, b_x, w_k, b_k, w_v, b_v;
    // w_qg, b_qg are w_q over w_gate and zeros over b_gate in the same memory: one product serves Q and the gates.  (After an
    // assignment to one of them they are not, and each has its own.)
    bool merged = false;
};
// The weights as they lie in memory now; a pass keeps the one that it began with.
struct Layout {
    std::vector<Block> blocks;
    std::vector<const void*> at;   // where and how large each tensor was
    std::vector<int64_t> numel;
    bool dense_bf16 = false;       // every weight bf16, dense, 16-byte aligned and of its size: what the kernels read by pointer
    bool merged = false;           // of all blocks
};

struct Plan {
    int64_t d_model, d_inner, heads, N, chunk, groups;
    double eps_norm;
    Dyn dyn;
    Tensor embedding, final_norm_w;
    std::vector<std::pair<Weights, double>> weights;
    std::shared_ptr<const Layout> layout;
};

constexpr double kFinalEps = 1.0 / 16384;   // 2^-14
constexpr double kGroupEps = 1e-5;
constexpr int64_t kHeadDim = 64;
constexpr int64_t kGraphBatch = 32;
// Prompts beyond this take the CUDA-core scan.  The two scans are equally precise: against float64, 12 layers, width 768, the
// worst layer's cached state is off by 0.0725 / 0.0724 of itself at 523 tokens (CUDA cores / tensor cores, N 16), 0.134 / 0.134
// at 900, 0.381 / 0.381 at 2000.  But the state is a product of one bf16-rounded transition a token, so single bf16 roundings that
// fall the other way drive two such caches apart: 0.014 at 523 tokens, 0.015 at 700, 0.018 at 900, 0.022 at 1200, 0.024 at 2000.
// Up to this length that is inside the 2e-2 within which passes of a model are compared; longer prompts keep the scan that
// their caches have always been filled with.
constexpr int64_t kTensorPrompt = 576;
constexpr int64_t kScanForceSimt = CDSSM_SCAN_FORCE_SIMT;

const char* kCapsule = "cdssm_lm_plan";
Plan& plan_of(PyObject* o) {
    auto* p = static_cast<Plan*>(PyCapsule_GetPointer(o, kCapsule));
    if (!p) throw std::invalid_argument("plan");
    return *p;
}

bool aligned_dense(const Tensor& t, at::ScalarType dt) {
    return t.is_cuda() && t.scalar_type() == dt && t.is_contiguous() && (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15) == 0;
}

// The present layout: laid out anew when a tensor has other memory (`.data` was assigned) than when it was last.  With the GIL.
std::shared_ptr<const Layout> layout_of(Plan& p) {
    auto each = [&](auto&& use) {
        for (Tensor* t : {&p.embedding, &p.final_norm_w}) use(*t);
        for (auto& w : p.weights)
            for (Tensor* t : w.first.all()) use(*t);
    };
    if (p.layout) {
        size_t i = 0;
        bool same = true;
        each([&](const Tensor& t) {
            same = same && t.const_data_ptr() == p.layout->at[i] && t.numel() == p.layout->numel[i];
            i++;
        });
        if (same) return p.layout;
    }
    auto l = std::make_shared<Layout>();
    each([&](const Tensor& t) {
        l->at.push_back(t.const_data_ptr());
        l->numel.push_back(t.numel());
    });
    const int64_t d = p.d_model, di = p.d_inner, H = p.heads, HN = H * p.N, G = (p.N + 5) * H, W = 3 * di + HN;
    l->dense_bf16 = H * kHeadDim == di && aligned_dense(p.embedding, at::kBFloat16) && p.embedding.dim() == 2 &&
                    p.embedding.size(1) == d && aligned_dense(p.final_norm_w, at::kBFloat16) && p.final_norm_w.numel() == d;
    l->merged = true;
    for (auto& pw : p.weights) {
        Block b;
        static_cast<Weights&>(b) = pw.first;
        b.shortcut = pw.second;
        auto rows = [](const Tensor& w, int64_t r0, int64_t r1) { return w.slice(0, r0, r1); };
        b.w_z = rows(b.w_in, 0, di); b.b_z = rows(b.b_in, 0, di);
        b.w_x = rows(b.w_in, di, 2 * di); b.b_x = rows(b.b_in, di, 2 * di);
        b.w_k = rows(b.w_in, 2 * di, 3 * di); b.b_k = rows(b.b_in, 2 * di, 3 * di);
        b.w_v = rows(b.w_in, 3 * di, b.w_in.size(0)); b.b_v = rows(b.b_in, 3 * di, b.b_in.size(0));
        auto vector = [](const Tensor& t, at::ScalarType dt, int64_t n) { return aligned_dense(t, dt) && t.numel() == n; };
        auto matrix = [](const Tensor& t, int64_t m, int64_t k) {
            return aligned_dense(t, at::kBFloat16) && t.dim() == 2 && t.size(0) == m && t.size(1) == k;
        };
        const auto bf = at::kBFloat16;
        l->dense_bf16 = l->dense_bf16 && vector(b.norm_w, bf, d) && matrix(b.w_in, W, d) && vector(b.b_in, bf, W) &&
                        vector(b.conv_w, bf, 4 * di) && vector(b.conv_b, bf, di) && matrix(b.w_q, di, di) && matrix(b.w_gate, G, di) &&
                        vector(b.b_gate, bf, G) && vector(b.lds, at::kFloat, H) && vector(b.rope, at::kFloat, H) &&
                        matrix(b.w_readout, di, HN) && matrix(b.w_out, d, di) && vector(b.gn_w, bf, di) &&
                        vector(b.gn_b, bf, di) && vector(b.D, bf, di);
        auto after = [](const Tensor& t, int64_t n) { return static_cast<const char*>(t.const_data_ptr()) + n * t.element_size(); };
        b.merged = b.w_qg.dim() == 2 && b.w_qg.size(0) == di + G && b.w_qg.size(1) == di && b.b_qg.numel() == di + G &&
                   b.w_qg.is_contiguous() && b.b_qg.is_contiguous() && b.w_q.is_contiguous() && b.w_gate.is_contiguous() &&
                   b.b_gate.is_contiguous() && b.w_q.const_data_ptr() == b.w_qg.const_data_ptr() &&
                   b.w_gate.const_data_ptr() == after(b.w_qg, di * di) && b.b_gate.const_data_ptr() == after(b.b_qg, di) &&
                   b.w_q.scalar_type() == b.w_qg.scalar_type() && b.w_gate.scalar_type() == b.w_qg.scalar_type() &&
                   b.b_gate.scalar_type() == b.b_qg.scalar_type() && b.w_q.numel() == di * di && b.w_gate.numel() == G * di &&
                   b.b_gate.numel() == G;
        l->merged = l->merged && b.merged;
        l->blocks.push_back(std::move(b));
    }
    return p.layout = l;
}

// sigmoid(v_residual_gate) of every layer in the activation type, formed anew in each pass (one small kernel): nothing of an
// earlier pass, stream or graph is read.  Layer 0 has no value residual.
struct Mix {
    std::vector<Tensor> of;   // (H) per layer, layer 0's undefined
    Mix(const Plan& p, const Layout& l, const Tensor& on) : of(l.blocks.size()) {
        const size_t n = of.size();
        if (n < 2) return;
        bool plain = true;
        std::vector<const float*> gates;
        for (size_t i = 1; i < n; i++) {
            const Tensor& g = l.blocks[i].v_gate;
            plain = plain && g.is_cuda() && g.scalar_type() == at::kFloat && g.is_contiguous() && g.numel() == p.heads;
            gates.push_back(plain ? fptr(g) : nullptr);
        }
        if (plain) {
            const Tensor all = at::empty({(int64_t)n - 1, p.heads}, on.options());
            check(cdssm_b200_residual_mix(gates.data(), (int)n - 1, (int)p.heads, mptr(all), dtype_code(on), stream_of(on)),
                  "residual_mix");
            for (size_t i = 1; i < n; i++) of[i] = all.select(0, (int64_t)i - 1);
        } else {
            for (size_t i = 1; i < n; i++)
                of[i] = at::sigmoid(l.blocks[i].v_gate.reshape({-1})).to(on.scalar_type()).expand({p.heads}).contiguous();
        }
    }
    const Tensor& at(size_t i) const { return of[i]; }
};

// GroupNorm(y) * silu(z) + D * x_conv
Tensor norm_gate(const Plan& p, const Block& b, const Tensor& y, const Tensor& z, const Tensor& x_conv, bool per_token) {
    const int64_t B = y.size(0), L = y.size(1), di = p.d_inner;
    if ((di / p.groups) % 8 == 0 && di <= 8192)
        return groupnorm_gate(y, b.gn_w, b.gn_b, z, b.D, x_conv, p.groups, kGroupEps, per_token);
    const auto dt = z.scalar_type();
    Tensor n;
    if (per_token)
        n = at::group_norm(y.to(at::kFloat).reshape({B * L, di, 1}), p.groups, b.gn_w.to(at::kFloat), b.gn_b.to(at::kFloat),
                           kGroupEps).to(dt).reshape({B, L, di});
    else
        n = at::group_norm(y.to(at::kFloat).transpose(1, 2), p.groups, b.gn_w.to(at::kFloat), b.gn_b.to(at::kFloat), kGroupEps)
                .to(dt).transpose(1, 2);
    return n * at::silu(z) + b.D * x_conv;
}

// One block over a sequence; x (B,L,d) is this call's own tensor and takes the residual sum in place.  With a cache the
// state after the last token and the last three conv inputs are handed out.
struct Cache {
    Tensor state, conv;
};
void block_sequence(const Plan& p, const Block& b, const Tensor& mix, const Tensor& x, Tensor& v_first, Cache* cache, bool per_token,
                    int64_t flags, const Tensor& ws) {
    const int64_t B = x.size(0), L = x.size(1), H = p.heads, N = p.N, di = p.d_inner;
    const Tensor xn = rms_norm(x, b.norm_w, p.eps_norm);
    // One product per consumer (row blocks of the in_proj weight): each output is dense, so neither the conv nor the
    // scan has to copy a column slice of a wide projection first.
    const Tensor z = linear(xn, b.w_z, b.b_z, ws), x_gate = linear(xn, b.w_x, b.b_x, ws);
    const Tensor K = linear(xn, b.w_k, b.b_k, ws).view({B, L, H, kHeadDim});
    Tensor V = linear(xn, b.w_v, b.b_v, ws).view({B, L, H, N});
    if (!v_first.defined()) v_first = V;
    else V = at::lerp(v_first, V, mix.view({1, 1, H, 1}));   // value residual (block.py:167-171)
    const Tensor x_conv = conv1d_silu(x_gate, b.conv_w, b.conv_b);
    if (cache) {   // last three inputs of the causal 4-tap conv
        if (L >= 3) {
            cache->conv = x_gate.slice(1, L - 3, L).contiguous();
        } else {
            cache->conv = at::zeros({B, 3, di}, x.options());
            cache->conv.slice(1, 3 - L, 3).copy_(x_gate);
        }
    }
    const Tensor gates = linear(x_conv, b.w_gate, b.b_gate, ws);
    const Tensor Q = linear(x_conv, b.w_q, Tensor(), ws).view({B, L, H, kHeadDim});
    ScanOut s = scan_fused(Q, K, V, gates, b.lds, b.rope, p.dyn, H, N, p.chunk, Tensor(), b.shortcut, 0, cache != nullptr,
                           cache ? (L > kTensorPrompt ? kScanForceSimt : 0) : flags, Tensor(), 1);
    if (cache) cache->state = s.tail;
    const Tensor y = linear(s.y.view({B, L, H * N}), b.w_readout, Tensor(), ws);
    // The reference normalises over (channels of the group) x (ALL positions of the sequence) (block.py:216-222), which
    // makes its forward non-causal.  A cached decode cannot reproduce that, so with a cache - and in forward() when
    // per_token_group_norm is set - the statistics are taken per token instead.
    const Tensor o = norm_gate(p, b, y, z, x_conv, per_token || cache);
    gemm(x.view({B * L, p.d_model}), o.view({B * L, di}), b.w_out, Tensor(), true, ws);   // the residual add rides in the epilogue
}

// The same for bf16 models: every activation of a pass lives in one arena, the kernels are called with pointers and row
// strides, and a layer's products are two wide ones (z | conv input | K | V and Q | gates) whose column slices the conv, the
// scan and the gate read in place; the scan applies the value residual.  Tensor by tensor, a layer took 97 us of host time
// (15 launches, as many allocations and views, nine products) whatever its size.
struct Arena {
    char* base;
    size_t at = 0;
    void* take(size_t bytes) {
        void* p = base ? base + at : nullptr;
        at += (bytes + 255) & ~(size_t)255;
        return p;
    }
};
struct SequenceBuffers {
    void *xn, *proj0, *proj, *x_conv, *qg, *y, *y2, *gated, *gemm_ws;
    float* stats;
    size_t bytes;
};
SequenceBuffers sequence_buffers(const Plan& p, int64_t B, int64_t L, char* base) {
    Arena a{base};
    const size_t T = (size_t)(B * L), es = 2, di = p.d_inner, HN = p.heads * p.N, G = (p.N + 5) * p.heads;
    const size_t pw = (3 * di + HN + 7) & ~(size_t)7, qw = (di + G + 7) & ~(size_t)7;
    SequenceBuffers s;
    s.xn = a.take(T * p.d_model * es);
    s.proj0 = a.take(T * pw * es + 1024);   // layer 0's, kept: its V is every later layer's v_first
    s.proj = a.take(T * pw * es + 1024);
    s.x_conv = a.take(T * di * es);
    s.qg = a.take(T * qw * es + 1024);
    s.y = a.take(T * HN * es);
    s.y2 = a.take(T * di * es);
    s.gated = a.take(T * di * es);
    s.stats = static_cast<float*>(a.take(sizeof(float) * cdssm_b200_groupnorm_stats_floats((int)B, (int)L, (int)p.groups)));
    s.gemm_ws = a.take(kGemmWorkspace);
    s.bytes = a.at;
    return s;
}

void run_sequence(const Plan& p, const Layout& lay, const Mix& mixes, const Tensor& x, std::vector<Cache>* caches, bool per_token,
                  int64_t flags, const SequenceBuffers& s) {
    const int B = (int)x.size(0), L = (int)x.size(1), d = (int)p.d_model, di = (int)p.d_inner, H = (int)p.heads, N = (int)p.N;
    const int64_t T = (int64_t)B * L;
    const int HN = H * N, G = (N + 5) * H, dev = (int)x.device().index();
    void* st = stream_of(x);
    const int scan_flags = (int)(caches ? (L > kTensorPrompt ? kScanForceSimt : 0) : flags);
    const Workspace ws = workspace(x, cdssm_b200_scan_fused_workspace_bytes_for(B, L, H, kHeadDim, N, (int)p.chunk, CDSSM_BF16, scan_flags));
    auto product = [&](void* out, int64_t ldo, const void* in, int64_t K, const Tensor& w, const void* bias, bool accumulate) {
        gemm_raw(dev, out, ldo, in, K, cptr(w), bias, T, w.size(0), K, accumulate, s.gemm_ws, st);
    };
    struct Slice { char* p; int64_t stride; };
    Slice v0{};
    const int64_t pw = (3 * di + HN + 7) & ~7, qw = (di + G + 7) & ~7;
    for (size_t i = 0; i < lay.blocks.size(); i++) {
        const Block& b = lay.blocks[i];
        char* proj = static_cast<char*>(i == 0 ? s.proj0 : s.proj);
        char* qg = static_cast<char*>(s.qg);
        check(cdssm_b200_rmsnorm_fwd(mptr(x), cptr(b.norm_w), s.xn, T, d, (float)p.eps_norm, CDSSM_BF16, st), "rmsnorm_fwd");
        const Slice z{proj, pw}, xg{proj + 2 * di, pw}, k{proj + 4 * di, pw}, v{proj + 6 * di, pw}, q{qg, qw}, g{qg + 2 * di, qw};
        product(proj, pw, s.xn, d, b.w_in, cptr(b.b_in), false);
        if (i == 0) v0 = v;
        Cache* cache = caches ? &(*caches)[i] : nullptr;
        if (cache) {
            cache->conv = at::empty({B, 3, di}, x.options());
            cache->state = empty_f32({B, H, N, kHeadDim}, x);
        }
        check(cdssm_b200_conv1d_silu_strided_fwd(xg.p, xg.stride, cptr(b.conv_w), cptr(b.conv_b), s.x_conv,
                                                 cache ? mptr(cache->conv) : nullptr, B, L, di, CDSSM_BF16, st),
              "conv1d_silu_fwd");
        if (b.merged) {
            product(qg, qw, s.x_conv, di, b.w_qg, cptr(b.b_qg), false);
        } else {
            product(q.p, qw, s.x_conv, di, b.w_q, nullptr, false);
            product(g.p, qw, s.x_conv, di, b.w_gate, cptr(b.b_gate), false);
        }
        const void* mix = i == 0 ? nullptr : cptr(mixes.at(i));
        check(cdssm_b200_scan_fused_strided_fwd(q.p, q.stride, k.p, k.stride, v.p, v.stride, i == 0 ? nullptr : v0.p, v0.stride, mix,
                                                g.p, g.stride, fptr(b.lds), fptr(b.rope), nullptr, s.y, nullptr,
                                                cache ? fmut(cache->state) : nullptr, ws.ptr, ws.bytes, p.dyn.c[0], p.dyn.c[1],
                                                p.dyn.c[2], p.dyn.c[3], p.dyn.c[4], (float)b.shortcut, B, L, H, kHeadDim, N,
                                                (int)p.chunk, 0, CDSSM_BF16,
                                                scan_flags, st),
              "scan_fused_fwd");
        product(s.y2, di, s.y, HN, b.w_readout, nullptr, false);
        const bool token_stats = per_token || caches;   // see block_sequence()
        if (!token_stats)
            check(cdssm_b200_groupnorm_stats(s.y2, s.stats, B, L, di, (int)p.groups, (float)kGroupEps, CDSSM_BF16, st), "groupnorm_stats");
        check(cdssm_b200_groupnorm_gate_fwd(s.y2, token_stats ? nullptr : s.stats, cptr(b.gn_w), cptr(b.gn_b), z.p, z.stride, cptr(b.D),
                                            s.x_conv, s.gated, B, L, di, (int)p.groups, (float)kGroupEps, CDSSM_BF16, st),
              "groupnorm_gate_fwd");
        product(mptr(x), d, s.gated, di, b.w_out, nullptr, true);   // the residual add rides in the epilogue
    }
}

// All layers over a sequence; x (B,L,d) is this call's own tensor and takes the residual sums in place.
void run_blocks(const Plan& p, const Layout& lay, const Tensor& x, std::vector<Cache>* caches, bool per_token, int64_t flags,
                const Tensor& ws) {
    const Mix mixes(p, lay, x);
    if (lay.dense_bf16 && x.numel() > 0 && p.d_model % 8 == 0 && (p.heads * p.N) % 8 == 0 && (p.d_inner / p.groups) % 8 == 0 &&
        p.d_inner <= 8192) {
        const size_t bytes = sequence_buffers(p, x.size(0), x.size(1), nullptr).bytes;
        const Tensor arena = at::empty({(int64_t)bytes + 256}, x.options().dtype(at::kByte));
        char* base = static_cast<char*>(arena.data_ptr());
        run_sequence(p, lay, mixes, x, caches, per_token, flags, sequence_buffers(p, x.size(0), x.size(1), base + (-(uintptr_t)base & 255)));
        return;
    }
    Tensor v_first;
    for (size_t i = 0; i < lay.blocks.size(); i++)
        block_sequence(p, lay.blocks[i], mixes.at(i), x, v_first, caches ? &(*caches)[i] : nullptr, per_token, flags, ws);
}

// One block of a one-token step; x (B,1,d) takes the residual sum in place.
void block_step(const Plan& p, const Block& b, const Tensor& residual_mix, const Tensor& x, Tensor& v_first, const Tensor& state, const Tensor& conv, int64_t pos,
                const Tensor& pos_dev, const Tensor& ws) {
    const int64_t B = x.size(0), H = p.heads, N = p.N, di = p.d_inner;
    const Tensor xn = rms_norm(x.view({B, p.d_model}), b.norm_w, p.eps_norm);
    const Tensor proj = linear(xn, b.w_in, b.b_in, ws);
    const Tensor z = proj.slice(1, 0, di).view({B, 1, di}), x_gate = proj.slice(1, di, 2 * di);
    const Tensor K = proj.slice(1, 2 * di, 3 * di).unflatten(1, {H, kHeadDim}), V = proj.slice(1, 3 * di).unflatten(1, {H, N});
    Tensor mix;
    if (!v_first.defined()) v_first = V.contiguous();   // one small copy per step; the kernels read it densely
    else mix = residual_mix;                            // the decode kernel applies the value residual itself
    const Tensor x_conv = conv1d_silu_step(x_gate, conv, b.conv_w, b.conv_b);
    Tensor Q, gates;
    if (b.merged) {   // one product for Q and the gates; the kernel reads slices
        const Tensor qg = linear(x_conv, b.w_qg, b.b_qg, ws);
        Q = qg.slice(1, 0, di);
        gates = qg.slice(1, di);
    } else {
        Q = linear(x_conv, b.w_q, Tensor(), ws);
        gates = linear(x_conv, b.w_gate, b.b_gate, ws);
    }
    Q = Q.unflatten(1, {H, kHeadDim});
    Tensor y = decode_step(state, Q, K, V, gates, b.lds, b.rope, p.dyn, H, N, pos, pos_dev, b.shortcut, Tensor(),
                           mix.defined() ? v_first : Tensor(), mix);
    y = linear(y.view({B, 1, H * N}), b.w_readout, Tensor(), ws);
    const Tensor o = norm_gate(p, b, y, z, x_conv.view({B, 1, di}), true);
    gemm(x.view({B, p.d_model}), o.view({B, di}), b.w_out, Tensor(), true, ws);
}

// The whole step by the small-batch kernels (csrc/lm_decode.cu); false where they do not apply.
bool decode_small_batch(const Plan& p, const Layout& lay, const Mix& mixes, const Tensor& x, const std::vector<Cache>& caches,
                        const Tensor& logits, int64_t pos, const Tensor& pos_dev) {
    const int64_t B = x.size(0), V = p.embedding.size(0);
    // replayed from a graph, the library's products are not held up by their launches: see lm_decode_takes()
    if (B > kGraphBatch && c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return false;
    const size_t bytes = cdssm_b200_lm_decode_workspace_bytes((int)B, (int)p.d_model, (int)p.N, (int)p.groups, (int)V, CDSSM_BF16);
    if (bytes == 0) return false;
    std::vector<cdssm_lm_layer> layers(caches.size());
    for (size_t i = 0; i < layers.size(); i++) {
        const Cache& c = caches[i];
        if (!aligned_dense(c.state, at::kFloat) || !aligned_dense(c.conv, at::kBFloat16) ||
            c.state.sizes() != at::IntArrayRef({B, p.heads, p.N, kHeadDim}) || c.conv.sizes() != at::IntArrayRef({B, 3, p.d_inner}))
            return false;
        const Block& b = lay.blocks[i];
        layers[i] = {cptr(b.norm_w), cptr(b.w_in), cptr(b.b_in), cptr(b.conv_w), cptr(b.conv_b), cptr(b.w_qg), cptr(b.b_qg),
                     fptr(b.lds), fptr(b.rope), cptr(mixes.at(i)), cptr(b.w_readout), cptr(b.gn_w),
                     cptr(b.gn_b), cptr(b.D), cptr(b.w_out), (float)b.shortcut, mptr(c.state), mptr(c.conv)};
    }
    const Tensor ws = at::empty({(int64_t)bytes}, x.options().dtype(at::kByte));
    check(cdssm_b200_lm_decode(layers.data(), (int)layers.size(), mptr(x), cptr(p.final_norm_w), cptr(p.embedding), mptr(logits),
                               mptr(ws), bytes, (float)p.eps_norm, (float)kGroupEps, (float)kFinalEps, p.dyn.c[0], p.dyn.c[1],
                               p.dyn.c[2], p.dyn.c[3], p.dyn.c[4], (int)B, (int)p.d_model, (int)p.N, (int)p.groups, (int)V,
                               (int)pos, static_cast<const int*>(cptr(pos_dev)), CDSSM_BF16, stream_of(x)),
          "lm_decode");
    return true;
}

Tensor embed(const Plan& p, const Tensor& ids) { return at::index(p.embedding, {std::optional<Tensor>(ids)}); }
Tensor head(const Plan& p, const Tensor& x, const Tensor& ws) {
    return linear(rms_norm(x, p.final_norm_w, kFinalEps), p.embedding, Tensor(), ws);
}

struct NoGrad {
    c10::AutoGradMode no_grad{false};
    at::AutoDispatchBelowADInplaceOrView below;
};

// lm_plan(d_model, d_inner, heads, N, chunk, groups, eps_norm, c0..c4, embedding, final_norm_w, blocks) -> plan;
// blocks: a list of tuples (eighteen tensors in Block's order, shortcut_scale)
PyObject* py_plan(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        Args in{a, n};
        auto p = std::make_unique<Plan>();
        p->d_model = in.integer(); p->d_inner = in.integer(); p->heads = in.integer(); p->N = in.integer();
        p->chunk = in.integer(); p->groups = in.integer();
        p->eps_norm = in.number();
        p->dyn = in.dyn();
        p->embedding = in.tensor("embedding"); p->final_norm_w = in.tensor("final_norm_w");
        PyObject* list = in.next();
        for (Py_ssize_t i = 0; i < PyList_Size(list); i++) {
            PyObject* t = PyList_GET_ITEM(list, i);
            Args f{PySequence_Fast_ITEMS(t), PyTuple_Size(t)};
            Weights w;
            for (Tensor* x : w.all()) *x = f.tensor("weight");
            p->weights.emplace_back(std::move(w), f.number());
        }
        return PyCapsule_New(p.release(), kCapsule, [](PyObject* o) {
            delete static_cast<Plan*>(PyCapsule_GetPointer(o, kCapsule));
        });
    });
}

// (B, L) token ids, or an error as the layers' shapes would have given.
void need_batch(const Tensor& ids) {
    if (ids.dim() != 2) throw Error("input_ids must be (batch, length)");
}

// lm_forward(plan, ids, per_token_group_norm, scan_flags) -> logits (B,L,vocab)
PyObject* py_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        Args in{a, n};
        Plan& p = plan_of(in.next());
        const Tensor ids = in.tensor("input_ids");
        const bool per_token = in.flag();
        const int64_t flags = in.integer();
        need_batch(ids);
        const NoGrad ng;
        const auto lay = layout_of(p);
        return wrap(without_gil([&] {
            const c10::cuda::CUDAGuard guard(p.embedding.device());
            const Tensor x = embed(p, ids), ws = gemm_workspace(x);
            run_blocks(p, *lay, x, nullptr, per_token, flags, ws);
            return head(p, x, ws);
        }));
    });
}

// lm_prefill(plan, ids, last_only) -> (logits, [state, conv, state, conv, ...])
PyObject* py_prefill(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        Args in{a, n};
        Plan& p = plan_of(in.next());
        const Tensor ids = in.tensor("input_ids");
        const bool last_only = in.flag();
        need_batch(ids);
        const NoGrad ng;
        const auto lay = layout_of(p);
        std::vector<Cache> caches(lay->blocks.size());
        Tensor logits = without_gil([&] {
            const c10::cuda::CUDAGuard guard(p.embedding.device());
            Tensor x = embed(p, ids);
            const Tensor ws = gemm_workspace(x);
            run_blocks(p, *lay, x, &caches, true, 0, ws);
            if (last_only) x = x.slice(1, x.size(1) - 1, x.size(1));
            return head(p, x, ws);
        });
        PyObject* list = PyList_New(2 * (Py_ssize_t)caches.size());
        if (!list) return nullptr;
        for (size_t i = 0; i < caches.size(); i++) {
            PyList_SET_ITEM(list, 2 * i, wrap(caches[i].state));
            PyList_SET_ITEM(list, 2 * i + 1, wrap(caches[i].conv));
        }
        return Py_BuildValue("(NN)", wrap(std::move(logits)), list);
    });
}

// lm_decode(plan, token_ids, [state, conv, ...], position: int or int32 CUDA tensor) -> logits (B,vocab)
PyObject* py_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        Args in{a, n};
        Plan& p = plan_of(in.next());
        const Tensor ids = in.tensor("token_ids");
        PyObject* list = in.next();
        if (!PyList_Check(list)) throw Error("decode: the cache is no list");
        // (as many layers as the cache has)
        const size_t layers = std::min(p.weights.size(), (size_t)PyList_GET_SIZE(list) / 2);
        Args c{PySequence_Fast_ITEMS(list), PyList_GET_SIZE(list)};
        std::vector<Cache> caches(layers);
        for (Cache& l : caches) { l.state = c.tensor("state"); l.conv = c.tensor("conv"); }
        Tensor pos_dev;
        int64_t pos = 0;
        if (in.at < n && THPVariable_Check(a[in.at])) pos_dev = in.tensor("pos");
        else pos = in.integer();
        if (ids.dim() != 1) throw Error("token_ids must be (batch)");
        if (pos_dev.defined() && (pos_dev.scalar_type() != at::kInt || !pos_dev.is_cuda()))
            throw Error("a tensor position must be an int32 CUDA tensor");
        const NoGrad ng;
        const auto lay = layout_of(p);
        return wrap(without_gil([&] {
            const c10::cuda::CUDAGuard guard(p.embedding.device());
            const int64_t B = ids.size(0);
            Tensor x = embed(p, ids).view({B, p.d_model}), v_first;
            const Mix mixes(p, *lay, x);
            if (lay->dense_bf16 && lay->merged && layers > 0) {
                const Tensor logits = at::empty({B, p.embedding.size(0)}, x.options());
                if (decode_small_batch(p, *lay, mixes, x, caches, logits, pos, pos_dev)) return logits;
            }
            x = x.view({B, 1, p.d_model});
            const Tensor ws = gemm_workspace(x);
            for (size_t i = 0; i < layers; i++)
                block_step(p, lay->blocks[i], mixes.at(i), x, v_first, caches[i].state, caches[i].conv, pos, pos_dev, ws);
            return head(p, x.view({B, p.d_model}), ws);
        }));
    });
}

#define FAST(fn) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(fn)), METH_FASTCALL, nullptr
PyMethodDef g_model_methods[] = {
    {"lm_plan", FAST(py_plan)},
    {"lm_forward", FAST(py_forward)},
    {"lm_prefill", FAST(py_prefill)},
    {"lm_decode", FAST(py_decode)},
    {nullptr, nullptr, 0, nullptr},
};

}  // namespace

PyMethodDef* model_methods() { return g_model_methods; }

}  // namespace cdssm_host
