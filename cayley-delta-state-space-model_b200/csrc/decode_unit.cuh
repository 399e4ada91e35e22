// One decode step of one (sequence, head, complex pair) by eight lanes: dynamics, normalised q and k, one delta-rule step
// on the float32 state in place, read-out.  Shared by the stand-alone step kernel (scan_simt.cu) and the whole-model step
// (lm_decode.cu).
#pragma once
#include "cdssm_common.cuh"
#include "row_slice.cuh"

namespace cdssm {

constexpr int kLanesPerUnit = 8;

// x * rsqrt(sum x^2 + 1e-6) over the unit's row, rounded like the reference's K_norm/Q_norm
// store (normalize_kq.cu:72-79).
template <typename T, int kCols>
__device__ __forceinline__ void normalise(float* f) {
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < kCols; i++) ss += f[i] * f[i];
    const float inv = rsqrtf(group_sum(ss) + kEps);
#pragma unroll
    for (int i = 0; i < kCols; i++) f[i] = IO<T>::rnd(f[i] * inv);
}

// One-token decode step: one pass over the state (read + write), everything else is a few hundred bytes per head.
struct DecodeUnitArgs {
    float* state;                  // (B,H,N,D)
    const void *q, *k, *v, *gate;  // rows with their own strides (column slices of a wider projection), in elements
    long long q_stride, k_stride, v_stride, gate_stride;
    const void *v_first, *mix;     // or NULL: v <- lerp(v_first, v, mix[head]) (value residual)
    long long v_first_stride;
    const float *log_dt_scale, *rope_freqs;
    void* y;                       // (B,H,N)
    DynConsts dc;
    float shortcut_scale;
    int H, D, N, pos;
    long long units;               // B*H*N/2
};

// Unit u of this thread's group of eight lanes; the whole warp calls together (units past the end take part in the
// shuffles and write nothing).  ready() comes before the first read of q and the gates: state, k and v are on their way by then.
// A step of a few units is a chain of trips to memory and of the dynamics' special functions: places in 32 bits (four divisions in 64
// took longer than a trip to the L2 cache).
template <typename T, int kCols, typename Ready>
__device__ __forceinline__ void decode_unit(const DecodeUnitArgs& a, long long u, Ready ready) {
    const int g = threadIdx.x % kLanesPerUnit;
    const bool active = u < a.units;
    if (!active) u = a.units - 1;
    const int NH = a.N >> 1, D = a.D, H = a.H;
    int j, hd;
    long long b;
    if (a.units <= 0xffffffffll) {
        const unsigned n = (unsigned)u / (unsigned)NH, m = n / (unsigned)H;
        j = (int)((unsigned)u - n * (unsigned)NH);
        hd = (int)(n - m * (unsigned)H);
        b = m;
    } else {
        j = (int)(u % NH);
        hd = (int)((u / NH) % H);
        b = u / ((long long)NH * H);
    }
    const bool vec = (D == kCols * kLanesPerUnit);
    const long long bh = b * H + hd;

    RowSlice<T, kCols> kraw, qraw;
    kraw.load(static_cast<const T*>(a.k) + b * a.k_stride + (long long)hd * D, g, D, vec);
    float* st = a.state + (bh * a.N + 2 * j) * D;
    float zr[kCols], zi[kCols];
    if (vec) {
#pragma unroll
        for (int i = 0; i < kCols / 4; i++) {
            const float4 x = *reinterpret_cast<const float4*>(st + g * kCols + 4 * i);
            const float4 w = *reinterpret_cast<const float4*>(st + D + g * kCols + 4 * i);
            zr[4 * i] = x.x; zr[4 * i + 1] = x.y; zr[4 * i + 2] = x.z; zr[4 * i + 3] = x.w;
            zi[4 * i] = w.x; zi[4 * i + 1] = w.y; zi[4 * i + 2] = w.z; zi[4 * i + 3] = w.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < kCols; i++) {
            const int d = g * kCols + i;
            zr[i] = d < D ? st[d] : 0.f;
            zi[i] = d < D ? st[D + d] : 0.f;
        }
    }
    const T* vrow = static_cast<const T*>(a.v) + b * a.v_stride + (long long)hd * a.N + 2 * j;
    float v0 = IO<T>::ld(vrow), v1 = IO<T>::ld(vrow + 1), f0 = 0.f, f1 = 0.f, mix = 0.f;
    if (a.v_first) {
        const T* f = static_cast<const T*>(a.v_first) + b * a.v_first_stride + (long long)hd * a.N + 2 * j;
        mix = IO<T>::ld(static_cast<const T*>(a.mix) + hd);
        f0 = IO<T>::ld(f);
        f1 = IO<T>::ld(f + 1);
    }
    const float lds = a.log_dt_scale[hd], freq = a.rope_freqs[hd], pos = (float)a.pos;
    ready();
    qraw.load(static_cast<const T*>(a.q) + b * a.q_stride + (long long)hd * D, g, D, vec);
    // dynamics (every lane of the unit computes the same scalars; dynamics_fused.cu:64-139)
    const T* gr = static_cast<const T*>(a.gate) + b * a.gate_stride;
    const T* s5 = gr + a.N * H;
    DynShared ds = dyn_shared<IO<T>::kBf16>(IO<T>::ld(gr + hd), IO<T>::ld(gr + NH * H + hd), IO<T>::ld(s5 + hd),
                              IO<T>::ld(s5 + H + hd), IO<T>::ld(s5 + 2 * H + hd),
                              IO<T>::ld(s5 + 3 * H + hd), IO<T>::ld(s5 + 4 * H + hd),
                              lds, freq, pos, a.dc);
    float a_re, a_im, vp;
    dyn_pair<IO<T>::kBf16>(IO<T>::ld(gr + j * H + hd), IO<T>::ld(gr + (NH + j) * H + hd), freq, pos, ds, a_re, a_im, vp);
    a_re = IO<T>::rnd(a_re);
    a_im = IO<T>::rnd(a_im);
    vp = IO<T>::rnd(vp);
    const float be = IO<T>::rnd(ds.beta), sc = IO<T>::rnd(ds.sel_c);
    if (a.v_first) {
        v0 = value_residual<T>(f0, v0, mix);
        v1 = value_residual<T>(f1, v1, mix);
    }
    const float vr = IO<T>::rnd(v0 * vp), vi = IO<T>::rnd(v1 * vp);

    float kk[kCols], qq[kCols];
    kraw.get(kk);
    qraw.get(qq);
    normalise<T, kCols>(kk);
    normalise<T, kCols>(qq);
    float ur = 0.f, ui = 0.f;
#pragma unroll
    for (int i = 0; i < kCols; i++) { ur += zr[i] * kk[i]; ui += zi[i] * kk[i]; }
    ur = be * group_sum(ur);
    ui = be * group_sum(ui);
    const float ivr = be * vr, ivi = be * vi;
    float yr = 0.f, yi = 0.f;
#pragma unroll
    for (int i = 0; i < kCols; i++) {
        const float er = zr[i] - ur * kk[i], ei = zi[i] - ui * kk[i];
        zr[i] = a_re * er - a_im * ei + ivr * kk[i];
        zi[i] = a_re * ei + a_im * er + ivi * kk[i];
        yr += zr[i] * qq[i];
        yi += zi[i] * qq[i];
    }
    yr = group_sum(yr);
    yi = group_sum(yi);
    if (a.shortcut_scale != 0.f) {
        float qk = 0.f;
#pragma unroll
        for (int i = 0; i < kCols; i++) qk += qq[i] * kk[i];
        qk = group_sum(qk);
        const float f = a.shortcut_scale * qk * qk;
        yr += f * vr;
        yi += f * vi;
    }
    if (!active) return;
    if (vec) {
#pragma unroll
        for (int i = 0; i < kCols / 4; i++) {
            *reinterpret_cast<float4*>(st + g * kCols + 4 * i) =
                make_float4(zr[4 * i], zr[4 * i + 1], zr[4 * i + 2], zr[4 * i + 3]);
            *reinterpret_cast<float4*>(st + D + g * kCols + 4 * i) =
                make_float4(zi[4 * i], zi[4 * i + 1], zi[4 * i + 2], zi[4 * i + 3]);
        }
    } else {
#pragma unroll
        for (int i = 0; i < kCols; i++) {
            const int d = g * kCols + i;
            if (d < D) { st[d] = zr[i]; st[D + d] = zi[i]; }
        }
    }
    if (g == 0) {
        T* o = static_cast<T*>(a.y) + bh * a.N + 2 * j;
        IO<T>::st(o, IO<T>::rnd(yr) * sc);
        IO<T>::st(o + 1, IO<T>::rnd(yi) * sc);
    }
}

}  // namespace cdssm
