// The projections' library products through cublasLt with the choice of algorithm and the descriptors kept per shape.
// at::linear asks the library's heuristics again on every call: 16 us of host time each, nine times a layer, against the 10 to
// 40 us that the product of a prompt takes on the GPU.
#include "host.h"

#include <cublasLt.h>

#include <list>
#include <mutex>
#include <unordered_map>

namespace cdssm_host {
namespace {

void lt_check(cublasStatus_t s, const char* what) {
    if (s != CUBLAS_STATUS_SUCCESS) throw Error(std::string(what) + ": cublasLt status " + std::to_string((int)s));
}

struct Key {
    int device;
    int64_t m, n, k, ldb, ldd;
    int bias, accumulate;
    int align_w, align_x, align_out, align_bias;   // bytes
    int reduction;                                 // the program's setting for partial sums of a split product
    bool operator==(const Key& o) const {
        return device == o.device && m == o.m && n == o.n && k == o.k && ldb == o.ldb && ldd == o.ldd && bias == o.bias &&
               accumulate == o.accumulate && align_w == o.align_w && align_x == o.align_x && align_out == o.align_out &&
               align_bias == o.align_bias && reduction == o.reduction;
    }
};
struct KeyHash {
    size_t operator()(const Key& k) const {
        size_t h = 1469598103934665603ull;
        for (int64_t v : {(int64_t)k.device, k.m, k.n, k.k, k.ldb, k.ldd, (int64_t)(k.bias * 8 + k.accumulate * 4 + k.reduction),
                          (int64_t)k.align_w << 36 | (int64_t)k.align_x << 24 | (int64_t)k.align_out << 12 | k.align_bias})
            h = (h ^ (size_t)v) * 1099511628211ull;
        return h;
    }
};
struct Plan {
    cublasLtMatmulDesc_t op = nullptr;
    cublasLtMatrixLayout_t a = nullptr, b = nullptr, d = nullptr;
    cublasLtMatmulAlgo_t algo;
    ~Plan() {
        if (op) cublasLtMatmulDescDestroy(op);
        for (auto l : {a, b, d})
            if (l) cublasLtMatrixLayoutDestroy(l);
    }
};

// Per host thread, so that the bias pointer can be set in the descriptor without a lock; the oldest plans go beyond kPlans.
constexpr size_t kPlans = 512;
struct Plans {
    std::unordered_map<Key, std::unique_ptr<Plan>, KeyHash> map;
    std::list<Key> order;
};
thread_local Plans t_plans;

cublasLtHandle_t handle(int device) {   // never destroyed: must not outlive the CUDA context at process exit
    static std::mutex mutex;
    static cublasLtHandle_t handles[64] = {};
    std::lock_guard<std::mutex> lock(mutex);
    cublasLtHandle_t& h = handles[device & 63];
    if (!h) lt_check(cublasLtCreate(&h), "cublasLtCreate");
    return h;
}

Plan& plan_for(const Key& key) {
    auto it = t_plans.map.find(key);
    if (it != t_plans.map.end()) return *it->second;
    auto p = std::make_unique<Plan>();
    lt_check(cublasLtMatmulDescCreate(&p->op, CUBLAS_COMPUTE_32F, CUDA_R_32F), "cublasLtMatmulDescCreate");
    const cublasOperation_t trans = CUBLAS_OP_T;
    lt_check(cublasLtMatmulDescSetAttribute(p->op, CUBLASLT_MATMUL_DESC_TRANSA, &trans, sizeof(trans)), "transpose");
    if (key.bias) {
        const cublasLtEpilogue_t ep = CUBLASLT_EPILOGUE_BIAS;
        lt_check(cublasLtMatmulDescSetAttribute(p->op, CUBLASLT_MATMUL_DESC_EPILOGUE, &ep, sizeof(ep)), "epilogue");
    }
    lt_check(cublasLtMatrixLayoutCreate(&p->a, CUDA_R_16BF, key.k, key.m, key.k), "layout");
    lt_check(cublasLtMatrixLayoutCreate(&p->b, CUDA_R_16BF, key.k, key.n, key.ldb), "layout");
    lt_check(cublasLtMatrixLayoutCreate(&p->d, CUDA_R_16BF, key.m, key.n, key.ldd), "layout");
    cublasLtMatmulPreference_t pref;
    lt_check(cublasLtMatmulPreferenceCreate(&pref), "preference");
    const size_t ws = kGemmWorkspace;
    cublasLtMatmulPreferenceSetAttribute(pref, CUBLASLT_MATMUL_PREF_MAX_WORKSPACE_BYTES, &ws, sizeof(ws));
    auto prefer = [&](cublasLtMatmulPreferenceAttributes_t attr, uint32_t v) {
        lt_check(cublasLtMatmulPreferenceSetAttribute(pref, attr, &v, sizeof(v)), "preference");
    };
    // (the library takes operands for 256-byte aligned unless it is told)
    prefer(CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_A_BYTES, key.align_w);
    prefer(CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_B_BYTES, key.align_x);
    prefer(CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_C_BYTES, key.align_out);
    prefer(CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_D_BYTES, key.align_out);
    // torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction, as the framework's own products take it
    using Reduction = at::CuBLASReductionOption;
    if (key.reduction == (int)Reduction::DisallowReducedPrecisionAllowSplitK)
        prefer(CUBLASLT_MATMUL_PREF_REDUCTION_SCHEME_MASK, CUBLASLT_REDUCTION_SCHEME_COMPUTE_TYPE);
    if (key.reduction == (int)Reduction::DisallowReducedPrecisionDisallowSplitK)
        prefer(CUBLASLT_MATMUL_PREF_REDUCTION_SCHEME_MASK, CUBLASLT_REDUCTION_SCHEME_NONE);
    cublasLtMatmulHeuristicResult_t res;
    int found = 0;
    const cublasStatus_t s = cublasLtMatmulAlgoGetHeuristic(handle(key.device), p->op, p->a, p->b, p->d, p->d, pref, 1, &res, &found);
    cublasLtMatmulPreferenceDestroy(pref);
    lt_check(s, "cublasLtMatmulAlgoGetHeuristic");
    if (!found) throw Error("cublasLt: no algorithm");
    p->algo = res.algo;
    if (t_plans.map.size() >= kPlans) {
        t_plans.map.erase(t_plans.order.front());
        t_plans.order.pop_front();
    }
    t_plans.order.push_back(key);
    return *(t_plans.map[key] = std::move(p));
}

int alignment(const void* p) {   // of an address, 256 bytes at most
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    return a ? (int)std::min<uintptr_t>(a & -a, 256) : 256;
}

bool aligned16(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15) == 0; }

}  // namespace

Tensor gemm_workspace(const Tensor& on) { return at::empty({(int64_t)kGemmWorkspace}, on.options().dtype(at::kByte)); }

// bf16: out (rows, M; ldo apart) = x (rows, K; ldx apart) w (M, K)^T [+ bias] [+ out]
void gemm_raw(int device, void* out, int64_t ldo, const void* x, int64_t ldx, const void* w, const void* bias, int64_t rows, int64_t M,
              int64_t K, bool accumulate, void* workspace, void* stream) {
    const Key key{device, M, rows, K, ldx, ldo, bias != nullptr, accumulate, alignment(w), alignment(x), alignment(out),
                  bias ? alignment(bias) : 256, (int)at::globalContext().allowBF16ReductionCuBLAS()};
    Plan& p = plan_for(key);
    if (bias) lt_check(cublasLtMatmulDescSetAttribute(p.op, CUBLASLT_MATMUL_DESC_BIAS_POINTER, &bias, sizeof(bias)), "bias");
    const float one = 1.f, beta = accumulate ? 1.f : 0.f;
    lt_check(cublasLtMatmul(handle(device), p.op, &one, w, p.a, x, p.b, &beta, out, p.d, out, p.d, &p.algo, workspace,
                            kGemmWorkspace, static_cast<cudaStream_t>(stream)),
             "cublasLtMatmul");
}

// out (rows, M; rows out.stride(0) apart) = x (rows, K; rows x.stride(0) apart) w^T [+ bias] [+ out]; w (M, K) dense.
void gemm(const Tensor& out, const Tensor& x, const Tensor& w, const Tensor& bias, bool accumulate, const Tensor& workspace) {
    const int64_t rows = x.size(0), K = x.size(1), M = w.size(0);
    if (rows == 0) return;
    const bool fits = w.dim() == 2 && w.size(1) == K && out.size(0) == rows && out.size(1) == M &&
                      (!bias.defined() || (bias.dim() == 1 && bias.size(0) == M && bias.scalar_type() == w.scalar_type()));
    const bool plain = fits && x.scalar_type() == at::kBFloat16 && w.scalar_type() == at::kBFloat16 && x.stride(1) == 1 &&
                       w.is_contiguous() && out.stride(1) == 1 && (x.stride(0) | out.stride(0) | K) % 8 == 0 && aligned16(x) && aligned16(w) &&
                       aligned16(out) && (!bias.defined() || aligned16(bias));
    if (!plain) {   // float32 models, widths that are no multiple of eight
        if (accumulate) at::addmm_out(const_cast<Tensor&>(out), out, x, w.t());   // one rounding, as in the epilogue (no bias with it)
        else out.copy_(at::linear(x, w, bias));
        return;
    }
    gemm_raw((int)x.device().index(), out.data_ptr(), out.stride(0), x.const_data_ptr(), x.stride(0), w.const_data_ptr(),
             bias.defined() ? bias.const_data_ptr() : nullptr, rows, M, K, accumulate, workspace.data_ptr(), stream_of(x));
}

// x (.., K) w^T [+ bias] as a new tensor (.., M)
Tensor linear(const Tensor& x, const Tensor& w, const Tensor& bias, const Tensor& workspace) {
    if (x.scalar_type() != at::kBFloat16 || !x.is_contiguous()) return at::linear(x, w, bias);
    auto sizes = x.sizes().vec();
    sizes.back() = w.size(0);
    Tensor out = at::empty(sizes, x.options());
    gemm(out.view({-1, w.size(0)}), x.view({-1, x.size(-1)}), w, bias, false, workspace);
    return out;
}

}  // namespace cdssm_host
