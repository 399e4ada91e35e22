// Device-side math shared by every kernel of the CD-SSM scan path.
//
// The formulas restate the reference's (cdssm/csrc/include/common.cuh:82-91 for the
// activations, cdssm/csrc/include/cayley_math.cuh:51-99 for the Cayley map,
// cdssm/csrc/kernels/dynamics_fused.cu:64-139 for the gate pipeline).  The reference is built
// with --use_fast_math, so its expf/logf/powf and '/' come from the special-function unit; the
// bfloat16 instantiations here take theirs from it too (kFast), and their outputs agree with
// the reference's bit for bit almost everywhere.  The float32 instantiations use the accurate
// library functions instead, to stay within 1e-4 of an fp32 restatement over long sequences.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace cdssm {

constexpr int kMaxStateDim = 32;   // N: even, N/2 complex pairs per head (common.cuh:34)
constexpr int kMaxHeadDim = 128;   // D (common.cuh:35)
constexpr float kEps = 1e-6f;      // common.cuh:142

// ---- storage types: bf16 (the reference's only I/O type) and fp32 ------------------------
template <typename T> struct IO;
template <> struct IO<__nv_bfloat16> {
    static constexpr bool kBf16 = true;
    static __device__ __forceinline__ float ld(const __nv_bfloat16* p) { return __bfloat162float(*p); }
    static __device__ __forceinline__ void st(__nv_bfloat16* p, float x) { *p = __float2bfloat16_rn(x); }
    // value as the reference would see it after a bf16 store
    static __device__ __forceinline__ float rnd(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
};
template <> struct IO<float> {
    static constexpr bool kBf16 = false;
    static __device__ __forceinline__ float ld(const float* p) { return *p; }
    static __device__ __forceinline__ void st(float* p, float x) { *p = x; }
    static __device__ __forceinline__ float rnd(float x) { return x; }
};

// kFast, from the special-function unit by the identities e^x = 2^(x log2 e), ln x = ln 2 log2 x, x^y = 2^(y log2 x) and a / b = a (1 / b).  The
// instructions are good to 2^-22 (PTX ISA); .ftz takes subnormal numbers for zero.  That is harmless where an exponential is added to one, a
// logarithm is of 1 + e^x or of at least 1e-8, a divisor is 1 + e^x, a sum of positive terms or the caller's adt_smoothness.  Powers stand alone: no
// flush there (sfu_exp2_sub).  Against float64 over the range of the gates: test_scan_bits_gpu.py.
__device__ __forceinline__ float sfu_exp2(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ float sfu_exp2_sub(float x) { float r; asm("ex2.approx.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ float sfu_log2(float x) { float r; asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ float sfu_rcp(float x) { float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }

// (of terms beside one)
template <bool kFast> __device__ __forceinline__ float exp_(float x) { return kFast ? sfu_exp2(__fmul_rn(x, 1.44269504f)) : expf(x); }
template <bool kFast> __device__ __forceinline__ float exp_alone(float x) { return kFast ? sfu_exp2_sub(__fmul_rn(x, 1.44269504f)) : expf(x); }
template <bool kFast> __device__ __forceinline__ float log_(float x) { return kFast ? __fmul_rn(sfu_log2(x), 0.693147181f) : logf(x); }
template <bool kFast> __device__ __forceinline__ float pow_(float x, float y) { return kFast ? sfu_exp2_sub(__fmul_rn(y, sfu_log2(x))) : powf(x, y); }
template <bool kFast> __device__ __forceinline__ float div_(float a, float b) { return kFast ? __fmul_rn(a, sfu_rcp(b)) : a / b; }

template <bool kFast> __device__ __forceinline__ float sigmoidf_(float x) {
    return div_<kFast>(1.0f, 1.0f + exp_<kFast>(-x));
}
template <bool kFast> __device__ __forceinline__ float softplusf_(float x) {
    return x > 20.0f ? x : log_<kFast>(1.0f + exp_<kFast>(x));
}
template <bool kFast> __device__ __forceinline__ float siluf_(float x) {
    return div_<kFast>(x, 1.0f + exp_<kFast>(-x));
}

struct DynConsts {
    float gating_c, omega_thresh, adt_delta, adt_smoothness, adt_eps;
};

// Which products and sums go together is said, not left to the compiler: kernels that form the dynamics on their own (records, walks,
// one-token steps, the operator) and versions of one for other sizes have the same bits, but for the angle (omega_at()).
// Per-(token, head) quantities shared by all complex pairs of the head.
struct DynShared {
    float dt, cr, beta, sel_c;   // cr = gating_c * sigmoid(r_gate)
};

// omega + pos freq, rounded once (the records of N = 2) or product and sum each (everywhere else).  Where gate and product all but cancel the
// second way costs up to half an ulp of the product, a transition of position 1000 6e-6; over a model's gates it is 0 to 5 % of the
// transition's error (rms against float64 at positions 0, 1000 and 200 000 of 2^18: 4.27, 3.46, 2.19e-7 once, 4.27, 3.64, 2.20e-7 twice).
template <bool kOnce>
__device__ __forceinline__ float omega_at(float omega_raw, float pos, float freq) {
    return kOnce ? __fmaf_rn(pos, freq, omega_raw) : __fadd_rn(omega_raw, __fmul_rn(pos, freq));
}

// dynamics_fused.cu:64-96,133-139.  alpha0_raw/omega0_raw are pair 0's gates; pos is the
// absolute position of the token.
template <bool kFast, bool kOnce = false>
__device__ __forceinline__ DynShared dyn_shared(float alpha0_raw, float omega0_raw, float sel_B,
                                                float sel_C, float sel_dt, float beta_raw,
                                                float r_raw, float log_dt_scale, float freq,
                                                float pos, const DynConsts& c) {
    DynShared o;
    float r_gate = sigmoidf_<kFast>(r_raw);
    float alpha0 = softplusf_<kFast>(alpha0_raw);
    float w0 = fabsf(omega_at<kOnce>(omega0_raw, pos, freq));
    float dt_scale = softplusf_<kFast>(log_dt_scale);
    float dt_raw = div_<kFast>(dt_scale, alpha0 + w0 + c.adt_eps);
    float dt_max = div_<kFast>(2.0f - c.adt_delta, alpha0 + c.adt_eps);
    float blend = sigmoidf_<kFast>(div_<kFast>(c.omega_thresh - w0, c.adt_smoothness));
    float dt_cap = fminf(dt_raw, dt_max);
    o.dt = __fadd_rn(__fmaf_rn(blend, dt_cap, __fmul_rn(1.0f - blend, dt_raw)), softplusf_<kFast>(sel_dt));
    o.cr = __fmul_rn(c.gating_c, r_gate);
    o.beta = sigmoidf_<kFast>(beta_raw) * sigmoidf_<kFast>(sel_B);
    o.sel_c = sigmoidf_<kFast>(sel_C);
    return o;
}

// One complex pair: Cayley map of lambda = -alpha + i*omega with tau = dt/2, stored as the
// conjugate, scaled by |mu|^(c*r - 1); vp = sqrt(1 - |mu|^(2*c*r)).
// dynamics_fused.cu:98-131, cayley_math.cuh:51-99.
template <bool kFast, bool kOnce = false>
__device__ __forceinline__ void dyn_pair(float alpha_raw, float omega_raw, float freq, float pos,
                                         const DynShared& s, float& a_re, float& a_im, float& vp) {
    float alpha = fmaxf(softplusf_<kFast>(alpha_raw), 0.0f);
    float omega = omega_at<kOnce>(omega_raw, pos, freq);
    const float tau = s.dt * 0.5f, tw = __fmul_rn(tau, omega), tw2 = __fmul_rn(tw, tw);
    const float nr = __fmaf_rn(-tau, alpha, 1.0f), dr = __fmaf_rn(tau, alpha, 1.0f);
    const float ni = tw, di = -tw;
    const float denom = __fadd_rn(__fmaf_rn(dr, dr, tw2), kEps);
    float inv_d = __frcp_rn(denom);
    const float mu_re = __fmul_rn(__fmaf_rn(nr, dr, __fmul_rn(ni, di)), inv_d);
    const float mu_im = __fmul_rn(__fmaf_rn(ni, dr, -__fmul_rn(nr, di)), inv_d);
    const float numer = __fmaf_rn(nr, nr, tw2);
    const float den2 = __fmaf_rn(dr, dr, tw2);
    float eig = fmaxf(div_<kFast>(numer, den2 + kEps), 1e-8f);
    float scale = pow_<kFast>(eig, __fadd_rn(s.cr, -1.0f) * 0.5f);
    a_re = mu_re * scale;
    a_im = -mu_im * scale;
    float eff = kFast ? sfu_exp2(__fmul_rn(s.cr, sfu_log2(eig))) : powf(eig, s.cr);   // (nothing beside one where it is flushed)
    vp = fminf(sqrtf(fmaxf(1.0f - eff, kEps)), 1.0f);
}

// Value residual across layers (block.py:167-171): lerp(first, v, w) rounded like the eager operation's output.
template <typename T>
__device__ __forceinline__ float value_residual(float first, float v, float w) {
    const float d = v - first;
    return IO<T>::rnd(fabsf(w) < 0.5f ? first + w * d : v - d * (1.f - w));
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// 16-byte vector of eight bfloat16 values <-> eight floats.
__device__ __forceinline__ void unpack8(const uint4& r, float* f) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&p);
}

// Rounds two values to the storage type with one conversion instruction.
template <typename T> __device__ __forceinline__ void rnd2(float& a, float& b) {
    if (IO<T>::kBf16) {
        const uint32_t w = pack2(a, b);
        a = __uint_as_float(w << 16);
        b = __uint_as_float(w & 0xffff0000u);
    }
}

// Pairs, for the kernels that are bound by issue slots beside memory: two values an instruction, in float32 or, where the values are
// bf16 already and the result is rounded to it, in bf16 (one rounding, as of the float32 result).
__device__ __forceinline__ float2 unpack2(uint32_t w) { return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
__device__ __forceinline__ __nv_bfloat162 as_bf16x2(uint32_t w) { return *reinterpret_cast<__nv_bfloat162*>(&w); }
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
    __nv_bfloat162 p = __hmul2_rn(as_bf16x2(a), as_bf16x2(b));
    return *reinterpret_cast<uint32_t*>(&p);
}
__device__ __forceinline__ uint32_t add_bf16x2(uint32_t a, uint32_t b) {
    __nv_bfloat162 p = __hadd2_rn(as_bf16x2(a), as_bf16x2(b));
    return *reinterpret_cast<uint32_t*>(&p);
}
// x / (1 + 2^(-x log2 e)).  What the exponential flushes to zero is nothing beside one; the reciprocal flushes below x = -87.3, where the
// result (-1e-36 and nearer to zero) becomes zero.
__device__ __forceinline__ float2 silu2(float2 x) {
    const float2 t = __fmul2_rn(x, make_float2(-1.44269504f, -1.44269504f));
    float2 e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.x) : "f"(t.x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.y) : "f"(t.y));
    const float2 d = __fadd2_rn(e, make_float2(1.f, 1.f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(d.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(d.y));
    return __fmul2_rn(x, r);
}
// Two channels of GroupNorm, gate and skip: rnd(rnd(rnd(GN(f)) rnd(silu(z))) + rnd(skip x)), bf16 pairs
__device__ __forceinline__ uint32_t gate_pair(float2 f, float mean, float rstd, float2 gw, float2 gb, uint32_t z, uint32_t skip, uint32_t x) {
    const float2 n = __ffma2_rn(__fmul2_rn(__fadd2_rn(f, make_float2(-mean, -mean)), make_float2(rstd, rstd)), gw, gb), s = silu2(unpack2(z));
    return add_bf16x2(mul_bf16x2(pack2(n.x, n.y), pack2(s.x, s.y)), mul_bf16x2(skip, x));
}

// Two consecutive elements as one access where `vec` says they are aligned.
template <typename T> __device__ __forceinline__ float2 ld_pair(const T* p, bool vec) {
    if (!vec) return make_float2(IO<T>::ld(p), IO<T>::ld(p + 1));
    if (IO<T>::kBf16) {
        const uint32_t w = *reinterpret_cast<const uint32_t*>(p);
        return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
    }
    return *reinterpret_cast<const float2*>(p);
}
template <typename T> __device__ __forceinline__ void st_pair(T* p, bool vec, float a, float b) {
    if (!vec) {
        IO<T>::st(p, a);
        IO<T>::st(p + 1, b);
    } else if (IO<T>::kBf16) {
        *reinterpret_cast<uint32_t*>(p) = pack2(a, b);
    } else {
        *reinterpret_cast<float2*>(p) = make_float2(a, b);
    }
}

template <typename T> struct Vec8;   // eight consecutive elements
template <> struct Vec8<__nv_bfloat16> {
    static __device__ __forceinline__ void ld(const __nv_bfloat16* p, float* f) {
        unpack8(*reinterpret_cast<const uint4*>(p), f);
    }
    static __device__ __forceinline__ void st(__nv_bfloat16* p, const float* f) {
        uint4 r;
        r.x = pack2(f[0], f[1]); r.y = pack2(f[2], f[3]); r.z = pack2(f[4], f[5]); r.w = pack2(f[6], f[7]);
        *reinterpret_cast<uint4*>(p) = r;
    }
};
template <> struct Vec8<float> {
    static __device__ __forceinline__ void ld(const float* p, float* f) {
        const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
        f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    }
    static __device__ __forceinline__ void st(float* p, const float* f) {
        *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
        *reinterpret_cast<float4*>(p + 4) = make_float4(f[4], f[5], f[6], f[7]);
    }
};

template <typename T> struct Vec4;   // four
template <> struct Vec4<__nv_bfloat16> {
    uint2 v;
    __device__ __forceinline__ void ld(const __nv_bfloat16* p) { v = *reinterpret_cast<const uint2*>(p); }
    __device__ __forceinline__ void get(float* f) const {
        f[0] = __uint_as_float(v.x << 16); f[1] = __uint_as_float(v.x & 0xffff0000u);
        f[2] = __uint_as_float(v.y << 16); f[3] = __uint_as_float(v.y & 0xffff0000u);
    }
    static __device__ __forceinline__ void st(__nv_bfloat16* p, const float* f) {
        *reinterpret_cast<uint2*>(p) = make_uint2(pack2(f[0], f[1]), pack2(f[2], f[3]));
    }
};
template <> struct Vec4<float> {
    float4 v;
    __device__ __forceinline__ void ld(const float* p) { v = *reinterpret_cast<const float4*>(p); }
    __device__ __forceinline__ void get(float* f) const { f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w; }
    static __device__ __forceinline__ void st(float* p, const float* f) {
        *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
    }
};

template <typename T> struct Raw8;   // eight, kept in storage form until used
template <> struct Raw8<__nv_bfloat16> {
    uint4 v;
    __device__ __forceinline__ void ld(const __nv_bfloat16* p) { v = *reinterpret_cast<const uint4*>(p); }
    __device__ __forceinline__ void get(float* f) const { unpack8(v, f); }
};
template <> struct Raw8<float> {
    float4 a, b;
    __device__ __forceinline__ void ld(const float* p) {
        a = *reinterpret_cast<const float4*>(p);
        b = *reinterpret_cast<const float4*>(p + 4);
    }
    __device__ __forceinline__ void get(float* f) const {
        f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    }
};

}  // namespace cdssm
