// What the CUDA-core scans (scan_simt.cu, scan_short.cu) are launched with, and the dynamics of a token.
#pragma once
#include "cdssm_common.cuh"

namespace cdssm {

struct ScanArgs {
    const void *q, *k, *v, *gate_raw;
    const float *log_dt_scale, *rope_freqs, *h0;
    void* y;
    float *final_state, *tail_state;
    float* total_decay;   // (B,H,N) or NULL: product over the chunks of the (rounded) chunk decays
    int segs;             // batch rows are `segs` consecutive segments of longer sequences
    int run_local;        // 0: the workspace already holds this input's local pass
    int run_output;       // 0: stop after the carry pass (another kernel writes y)
    int publish;          // 0: summary only, the carry pass leaves the local results in place
    int fp32_decay;       // 1: the transition a_t keeps float32 precision (the reference stores it as bf16)
    float4* rec_av;    // (B,NC,H,NP,C): transition and scaled v of a token, or NULL: the walk computes them itself
    float2* rec_bs;    // (B,NC,H,C): beta and sel_C
    float* ws_gamma;   // (B,NC,H,NP,2)
    float* ws_state;   // (B,NC,H,NP,2,D): z_{C-1} after the local pass, s_c after the carry pass
    DynConsts dc;
    float shortcut_scale;
    int B, L, H, D, N, C, NC, pos0;
    // elements between the (batch, token) rows of q, k, v, gate_raw and v_first (column slices of wider projections)
    long long q_rs, k_rs, v_rs, g_rs, vf_rs;
    const void *v_first, *mix;   // or NULL: v <- lerp(v_first, v, mix[head])
    long long units;   // B*NC*H*NP
};

// Dynamics of one (token, head): what its pairs share, then pair j (dynamics_fused.cu:64-139 and the vp scale of
// block.py:194-195).
template <typename T>
struct TokenDynamics {
    const T *gr, *vrow, *vfirst;
    DynShared ds;
    float freq, pos, mix;
    int H, NH, fp32_decay;
    __device__ __forceinline__ TokenDynamics(const ScanArgs& a, int b, int l, int hd) {
        H = a.H; NH = a.N >> 1; fp32_decay = a.fp32_decay;
        const long long bl = (long long)b * a.L + l;
        gr = static_cast<const T*>(a.gate_raw) + bl * a.g_rs + hd;
        vrow = static_cast<const T*>(a.v) + bl * a.v_rs + (long long)hd * a.N;
        vfirst = a.v_first ? static_cast<const T*>(a.v_first) + bl * a.vf_rs + (long long)hd * a.N : nullptr;
        mix = a.v_first ? IO<T>::ld(static_cast<const T*>(a.mix) + hd) : 0.f;
        const T* s5 = gr + a.N * H;
        freq = a.rope_freqs[hd];
        pos = (float)(l + a.pos0 + (b % a.segs) * a.L);
        ds = dyn_shared<IO<T>::kBf16>(IO<T>::ld(gr), IO<T>::ld(gr + NH * H), IO<T>::ld(s5), IO<T>::ld(s5 + H),
                                      IO<T>::ld(s5 + 2 * H), IO<T>::ld(s5 + 3 * H), IO<T>::ld(s5 + 4 * H),
                                      a.log_dt_scale[hd], freq, pos, a.dc);
    }
    __device__ __forceinline__ float2 beta_sel() const { return make_float2(IO<T>::rnd(ds.beta), IO<T>::rnd(ds.sel_c)); }
    __device__ __forceinline__ float4 pair(int j) const {
        float ar, ai, vp;
        dyn_pair<IO<T>::kBf16>(IO<T>::ld(gr + j * H), IO<T>::ld(gr + (NH + j) * H), freq, pos, ds, ar, ai, vp);
        if (!fp32_decay) {
            ar = IO<T>::rnd(ar);
            ai = IO<T>::rnd(ai);
        }
        vp = IO<T>::rnd(vp);
        float v0 = IO<T>::ld(vrow + 2 * j), v1 = IO<T>::ld(vrow + 2 * j + 1);
        if (vfirst) {
            v0 = value_residual<T>(IO<T>::ld(vfirst + 2 * j), v0, mix);
            v1 = value_residual<T>(IO<T>::ld(vfirst + 2 * j + 1), v1, mix);
        }
        return make_float4(ar, ai, IO<T>::rnd(v0 * vp), IO<T>::rnd(v1 * vp));
    }
};

// The walks' sums and products whose grouping is said, not left to the compiler: either walk may run, by size, and has the bits of the other.
// x y - z w, x y + z w, the second product rounded
__device__ __forceinline__ float msub(float x, float y, float z, float w) { return __fmaf_rn(x, y, -__fmul_rn(z, w)); }
__device__ __forceinline__ float madd(float x, float y, float z, float w) { return __fmaf_rn(x, y, __fmul_rn(z, w)); }
// s <- gamma s + l
__device__ __forceinline__ float next_re(float2 g, float sr, float si, float l) { return __fadd_rn(msub(g.x, sr, g.y, si), l); }
__device__ __forceinline__ float next_im(float2 g, float sr, float si, float l) { return __fadd_rn(madd(g.x, si, g.y, sr), l); }
// read-out before the norms: (r.q + a_re (z.q)_re -+ a_im (z.q)_im) + K (k.q)
__device__ __forceinline__ float read_re(float rq, float are, float aim, float zqr, float zqi, float K, float kq) {
    return __fmaf_rn(K, kq, __fmaf_rn(-aim, zqi, __fmaf_rn(are, zqr, rq)));
}
__device__ __forceinline__ float read_im(float rq, float are, float aim, float zqr, float zqi, float K, float kq) {
    return __fmaf_rn(K, kq, __fmaf_rn(aim, zqr, __fmaf_rn(are, zqi, rq)));
}

// scan_short.cu: the walk's local and output pass for few units, bit for bit.  from_chunks: no carry pass has run, the output pass adds up
// the chunks before its own (and writes the final state).
bool scan_short_takes(const ScanArgs& a, int dtype, int sms);
int scan_short_pass(bool output, const ScanArgs& a, int dtype, int from_chunks, cudaStream_t st);

}  // namespace cdssm
