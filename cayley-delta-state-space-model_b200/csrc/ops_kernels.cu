// The six operator-level forward kernels behind the reference's cdssm/ops.py classes.
//
// These keep the reference's operator boundaries (and therefore its HBM traffic: the
// (B,L,H,N,D) tensors are materialised) so that cdssm/models/ssd.py and block.py can run on
// them unchanged.  The measured path is the fused one (scan_wa.cu, scan_simt.cu); these exist for the
// strict drop-in and as building blocks of the parity tests.
//
// Thread mappings differ from the reference's (one block of D threads per (chunk, head) with
// two block barriers per step):
//   * the complex pairs of a head never interact (each pair owns two state rows; the erase
//     uses a per-row dot product), so the sequential kernels run a few LANES per
//     (chunk, head, pair): the per-step reduction is a few shuffles, no barrier at all;
//   * the dynamics kernel maps consecutive threads to consecutive heads so that every gate
//     segment is read coalesced.
#include "cdssm_common.cuh"
#include "row_slice.cuh"

namespace cdssm {

// ---------------------------------------------------------------- dynamics
template <typename T>
__global__ void __launch_bounds__(256)
dynamics_fwd_kernel(const T* __restrict__ gate_raw, const float* __restrict__ log_dt_scale,
                    const float* __restrict__ rope_freqs, T* __restrict__ A_bar,
                    T* __restrict__ vp_scale, T* __restrict__ beta, T* __restrict__ sel_C,
                    DynConsts c, long long total, int H, int N, int L, int pos0) {
    long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const int h = (int)(idx % H);
    const long long bl = idx / H;
    const int l = (int)(bl % L);
    const int NH = N >> 1;
    const T* g = gate_raw + bl * (long long)((N + 5) * H);
    const T* sc = g + N * H;
    const float freq = rope_freqs[h];
    const float pos = (float)(l + pos0);
    DynShared s = dyn_shared<IO<T>::kBf16>(IO<T>::ld(g + h), IO<T>::ld(g + NH * H + h), IO<T>::ld(sc + h),
                             IO<T>::ld(sc + H + h), IO<T>::ld(sc + 2 * H + h),
                             IO<T>::ld(sc + 3 * H + h), IO<T>::ld(sc + 4 * H + h),
                             log_dt_scale[h], freq, pos, c);
    for (int j = 0; j < NH; j++) {
        float a_re, a_im, vp;
        dyn_pair<IO<T>::kBf16>(IO<T>::ld(g + j * H + h), IO<T>::ld(g + (NH + j) * H + h), freq, pos, s, a_re,
                 a_im, vp);
        IO<T>::st(A_bar + idx * N + 2 * j, a_re);
        IO<T>::st(A_bar + idx * N + 2 * j + 1, a_im);
        IO<T>::st(vp_scale + idx * NH + j, vp);
    }
    IO<T>::st(beta + idx, s.beta);
    IO<T>::st(sel_C + idx, s.sel_c);
}

// ---------------------------------------------------------------- normalise
// Eight lanes per row pair (K row and Q row of a token-head) of 64 columns, 16 of 128, one 16-byte access per row and lane;
// other sizes, and unaligned rows, take a warp each.  Bounded by memory.  Measured on B200, bf16, 98 304 rows of 64: 8.3 us (a warp per row: 23).
template <typename T, int kLanes>
__global__ void __launch_bounds__(256)
normalize_kq_fwd_rows_kernel(const T* __restrict__ K, const T* __restrict__ Q, T* __restrict__ Ko, T* __restrict__ Qo, long long rows) {
    constexpr int kCols = 8, kD = kCols * kLanes;
    const int g = threadIdx.x % kLanes;
    long long row = (long long)blockIdx.x * (256 / kLanes) + threadIdx.x / kLanes;
    const bool on = row < rows;
    if (!on) row = rows - 1;
    RowSlice<T, kCols> rk, rq;
    rk.load(K + row * kD, g, kD, true);
    rq.load(Q + row * kD, g, kD, true);
    auto side = [&](const RowSlice<T, kCols>& x, T* out) {
        float f[kCols], ss = 0.f;
        x.get(f);
#pragma unroll
        for (int i = 0; i < kCols; i++) ss += f[i] * f[i];
        const float n = rsqrtf(group_sum<kLanes>(ss) + kEps);
#pragma unroll
        for (int i = 0; i < kCols; i++) f[i] *= n;
        if (on) RowSlice<T, kCols>::store(out + row * kD, g, kD, true, f);
    };
    side(rk, Ko);
    side(rq, Qo);
}

template <typename T>
__global__ void __launch_bounds__(256)
normalize_kq_fwd_kernel(const T* __restrict__ K, const T* __restrict__ Q, T* __restrict__ Ko,
                        T* __restrict__ Qo, long long rows, int D) {
    const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int lane = threadIdx.x & 31;
    const T* k = K + row * D;
    const T* q = Q + row * D;
    float sk = 0.f, sq = 0.f;
    for (int d = lane; d < D; d += 32) {
        float a = IO<T>::ld(k + d), b = IO<T>::ld(q + d);
        sk += a * a;
        sq += b * b;
    }
    sk = warp_sum(sk);
    sq = warp_sum(sq);
    const float ik = rsqrtf(sk + kEps), iq = rsqrtf(sq + kEps);
    for (int d = lane; d < D; d += 32) {
        IO<T>::st(Ko + row * D + d, IO<T>::ld(k + d) * ik);
        IO<T>::st(Qo + row * D + d, IO<T>::ld(q + d) * iq);
    }
}

// ---------------------------------------------------------------- intra-chunk scan and correction
// kLanes lanes (8 for D <= 64, 16 above) own one (chunk, head, pair), eight contiguous columns of its two state rows each; the
// next token's inputs are on their way while a step is taken.  Bounded by the states written.  Measured on B200, bf16, 64 chunks
// of 64, 24 heads, N 16, D 64 (201 MB written): intra 162 -> 67 us, correction 149 -> 68 us.
template <typename T, int kLanes, bool kInject>
__global__ void __launch_bounds__(128)
chunk_walk_kernel(const T* __restrict__ A, const T* __restrict__ K, const T* __restrict__ V,
                  const T* __restrict__ beta, const T* __restrict__ init,  // correction: carry in
                  T* __restrict__ states,   // local_h or corrections (units,C,H,N,D)
                  T* __restrict__ cum_A,    // intra only
                  long long units, int C, int H, int D, int N, bool vec) {
    constexpr int kCols = 8, kP = kCols / 2;
    const int NH = N >> 1, g = threadIdx.x % kLanes;
    long long w = (long long)blockIdx.x * (128 / kLanes) + threadIdx.x / kLanes;
    const bool active = w < units * H * NH;
    if (!active) w = units * H * NH - 1;                 // keep the lane in the shuffles
    const int j = (int)(w % NH);
    const int hd = (int)((w / NH) % H);
    const long long c = w / ((long long)NH * H);
    const long long row0 = c * C * H + hd;
    const T* Ap = A + row0 * N + 2 * j;
    const T* Kp = K + row0 * D;
    const T* Vp = kInject ? V + row0 * N + 2 * j : nullptr;
    const T* Bp = beta + row0;
    T* out = states + (row0 * N + 2 * j) * (long long)D;
    T* cum = kInject ? cum_A + row0 * N + 2 * j : nullptr;
    float2 zr[kP], zi[kP];
#pragma unroll
    for (int i = 0; i < kP; i++) zr[i] = zi[i] = make_float2(0.f, 0.f);
    if (!kInject) {
        RowSlice<T, kCols> s;
        const T* p = init + ((c * H + hd) * N + 2 * j) * (long long)D;
        s.load(p, g, D, vec);
        s.get(reinterpret_cast<float*>(zr));
        s.load(p + D, g, D, vec);
        s.get(reinterpret_cast<float*>(zi));
    }
    auto store = [&]() {
        if (!active) return;
        RowSlice<T, kCols>::store(out, g, D, vec, reinterpret_cast<const float*>(zr));
        RowSlice<T, kCols>::store(out + D, g, D, vec, reinterpret_cast<const float*>(zi));
    };
    float cr = 1.f, ci = 0.f;
    RowSlice<T, kCols> kraw;
    float a_re, a_im, b, vr = 0.f, vi = 0.f;
    auto fetch = [&]() {
        kraw.load(Kp, g, D, vec);
        a_re = IO<T>::ld(Ap); a_im = IO<T>::ld(Ap + 1);
        b = IO<T>::ld(Bp);
        if (kInject) { vr = IO<T>::ld(Vp); vi = IO<T>::ld(Vp + 1); }
    };
    fetch();
    for (int t = 0; t < C; t++) {
        float2 k[kP];
        kraw.get(reinterpret_cast<float*>(k));
        const float ar = a_re, ai = a_im, be = b, v0 = vr, v1 = vi;
        if (t + 1 < C) {
            Ap += (long long)H * N; Kp += (long long)H * D; Bp += H;
            if (kInject) Vp += (long long)H * N;
            fetch();
        }
        if (!kInject) store();   // correction stores the state BEFORE the step (exact_correction.cu:90-94)
        float2 ur2 = make_float2(0.f, 0.f), ui2 = ur2;
#pragma unroll
        for (int i = 0; i < kP; i++) {
            ur2 = __ffma2_rn(zr[i], k[i], ur2);
            ui2 = __ffma2_rn(zi[i], k[i], ui2);
        }
        const float ur = -be * group_sum<kLanes>(ur2.x + ur2.y), ui = -be * group_sum<kLanes>(ui2.x + ui2.y);
        // z' = a (z + u k) + beta v k
        const float kr = ar * ur - ai * ui + be * v0, ki = ar * ui + ai * ur + be * v1;
        const float2 ar2 = make_float2(ar, ar), ai2 = make_float2(ai, ai), ni2 = make_float2(-ai, -ai);
        const float2 kr2 = make_float2(kr, kr), ki2 = make_float2(ki, ki);
#pragma unroll
        for (int i = 0; i < kP; i++) {
            const float2 x = zr[i], y = zi[i];
            zr[i] = __ffma2_rn(kr2, k[i], __ffma2_rn(ar2, x, __fmul2_rn(ni2, y)));
            zi[i] = __ffma2_rn(ki2, k[i], __ffma2_rn(ar2, y, __fmul2_rn(ai2, x)));
        }
        if (kInject) {           // local scan stores the state AFTER the step (intra_chunk_scan.cu:169-173)
            store();
            const float nr = ar * cr - ai * ci, ni = ar * ci + ai * cr;
            cr = nr;
            ci = ni;
            if (g == 0 && active) {
                IO<T>::st(cum, cr);
                IO<T>::st(cum + 1, ci);
            }
            cum += (long long)H * N;
        }
        out += (long long)H * N * D;
    }
}

// ---------------------------------------------------------------- inter-chunk carry
// One thread per (b, h, pair, d); serial over the chunks (inter_chunk_scan.cu:52-84).
template <typename T>
__global__ void __launch_bounds__(128)
inter_chunk_fwd_kernel(const T* __restrict__ total_A, const T* __restrict__ flh,
                       T* __restrict__ chunk_states, int B, int NC, int H, int D, int N) {
    const int NH = N >> 1;
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)B * H * NH * D) return;
    const int d = (int)(idx % D);
    const int j = (int)((idx / D) % NH);
    const int hd = (int)((idx / ((long long)D * NH)) % H);
    const int b = (int)(idx / ((long long)D * NH * H));
    float sr = 0.f, si = 0.f;
    for (int k = 0; k < NC; k++) {
        const long long u = ((long long)b * NC + k) * H + hd;
        const long long o = (u * N + 2 * j) * (long long)D + d;
        IO<T>::st(chunk_states + o, sr);
        IO<T>::st(chunk_states + o + D, si);
        const float re = IO<T>::ld(total_A + u * N + 2 * j), im = IO<T>::ld(total_A + u * N + 2 * j + 1);
        const float fr = IO<T>::ld(flh + o), fi = IO<T>::ld(flh + o + D);
        const float nr = re * sr - im * si + fr;
        const float ni = re * si + im * sr + fi;
        sr = nr;
        si = ni;
    }
}

// ---------------------------------------------------------------- conv1d + SiLU
// kSeg consecutive positions per thread with the 3-deep history in registers (the reference re-reads the three neighbours from
// global for every output).  hist, if given, receives the last three inputs of every sequence (zeros where it has fewer).
template <typename T, int kSeg>
__global__ void __launch_bounds__(128)
conv1d_silu_fwd_kernel(const T* __restrict__ x, long long x_rs, const T* __restrict__ w, const T* __restrict__ bias,
                       T* __restrict__ out, T* __restrict__ hist, int L, int Dm) {
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= Dm) return;
    const int l0 = blockIdx.y * kSeg;
    const T* xb = x + (long long)blockIdx.z * L * x_rs + d;
    const long long base = (long long)blockIdx.z * L * Dm + d;
    const float w0 = IO<T>::ld(w + d * 4), w1 = IO<T>::ld(w + d * 4 + 1), w2 = IO<T>::ld(w + d * 4 + 2),
                w3 = IO<T>::ld(w + d * 4 + 3), bv = IO<T>::ld(bias + d);
    float x0 = l0 >= 3 ? IO<T>::ld(xb + (long long)(l0 - 3) * x_rs) : 0.f;
    float x1 = l0 >= 2 ? IO<T>::ld(xb + (long long)(l0 - 2) * x_rs) : 0.f;
    float x2 = l0 >= 1 ? IO<T>::ld(xb + (long long)(l0 - 1) * x_rs) : 0.f;
    const int lend = min(l0 + kSeg, L);
    for (int l = l0; l < lend; l++) {
        const float x3 = IO<T>::ld(xb + (long long)l * x_rs);
        const float yv = w0 * x0 + w1 * x1 + w2 * x2 + w3 * x3 + bv;
        IO<T>::st(out + base + (long long)l * Dm, siluf_<IO<T>::kBf16>(yv));
        x0 = x1;
        x1 = x2;
        x2 = x3;
    }
    if (hist != nullptr && lend == L) {
        T* h = hist + (long long)blockIdx.z * 3 * Dm + d;
        IO<T>::st(h, x0);
        IO<T>::st(h + Dm, x1);
        IO<T>::st(h + 2 * Dm, x2);
    }
}

// Four channels per thread, the loads of the next eight positions in flight while eight are worked on (without that the loads
// sank to their uses and every position waited for memory).  Bounded by memory latency, then bandwidth (one read, one write).
// kSeg: 32 positions where that still gives the GPU enough threads, else 8.  Measured on B200, bf16, B 8, L 2048, 1536
// channels: 30 -> 27 us against a channel per thread, 24.7 -> 21.7 (rows of a wider projection) with two channels an instruction; a
// copy takes 18.5 us.
template <typename T, int kSeg>
__global__ void __launch_bounds__(128)
conv1d_silu_vec_kernel(const T* x, long long x_rs, const T* w, const T* bias,
                       T* __restrict__ out, T* __restrict__ hist, int L, int Dm) {
    constexpr int kStep = 8;
    const int d = (blockIdx.x * 128 + threadIdx.x) * 4;
    if (d >= Dm) return;
    const int l0 = blockIdx.y * kSeg;
    const T* xb = x + (long long)blockIdx.z * L * x_rs + d;
    T* ob = out + (long long)blockIdx.z * L * Dm + d;
    float x0[4], x1[4], x2[4], bi[4], wt[4][4];
    auto row = [&](int l, float* f) {
        Vec4<T> v;
        v.ld(xb + (long long)max(l, 0) * x_rs);
        v.get(f);
#pragma unroll
        for (int e = 0; e < 4; e++) f[e] = l >= 0 ? f[e] : 0.f;
    };
    grid_dependency_wait();   // launched while the predecessor drains (glue_kernels.cu)
    {
        Vec4<T> v;
        v.ld(bias + d);
        v.get(bi);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            v.ld(w + (d + i) * 4);
            v.get(wt[i]);
        }
    }
    row(l0 - 3, x0);
    row(l0 - 2, x1);
    row(l0 - 1, x2);
    const int lend = min(l0 + kSeg, L);
    Vec4<T> r[kStep];
#pragma unroll
    for (int s = 0; s < kStep; s++) r[s].ld(xb + (long long)min(l0 + s, L - 1) * x_rs);
#pragma unroll 1
    for (int l1 = l0; l1 < lend; l1 += kStep) {
        Vec4<T> n[kStep];
        if (kSeg > kStep) {   // the next positions travel while these are worked on
#pragma unroll
            for (int s = 0; s < kStep; s++) n[s].ld(xb + (long long)min(l1 + kStep + s, L - 1) * x_rs);
        }
#pragma unroll
        for (int s = 0; s < kStep; s++) {
            float x3[4], y[4];
            r[s].get(x3);
#pragma unroll
            for (int e = 0; e < 4; e += 2) {   // (two channels an instruction)
                auto two = [&](const float* f) { return make_float2(f[e], f[e + 1]); };
                auto tap = [&](int i) { return make_float2(wt[e][i], wt[e + 1][i]); };
                float2 v = __fmul2_rn(tap(0), two(x0));
                v = __ffma2_rn(tap(1), two(x1), v);
                v = __ffma2_rn(tap(2), two(x2), v);
                v = __fadd2_rn(__ffma2_rn(tap(3), two(x3), v), two(bi));
                if constexpr (IO<T>::kBf16) {
                    v = silu2(v);
                } else {
                    v.x = siluf_<false>(v.x);
                    v.y = siluf_<false>(v.y);
                }
                y[e] = v.x;
                y[e + 1] = v.y;
            }
#pragma unroll
            for (int e = 0; e < 4; e++) {
                x0[e] = x1[e];
                x1[e] = x2[e];
                x2[e] = x3[e];
            }
            if (l1 + s < lend) Vec4<T>::st(ob + (long long)(l1 + s) * Dm, y);
            if (kSeg > kStep) r[s] = n[s];
        }
    }
    if (hist != nullptr && lend == L) {
        T* h = hist + (long long)blockIdx.z * 3 * Dm + d;
#pragma unroll
        for (int i = 0; i < 3; i++) {
            float f[4];
            row(L - 3 + i, f);
            Vec4<T>::st(h + (long long)i * Dm, f);
        }
    }
}

// ---------------------------------------------------------------- carries into consecutive segments
// One thread per (b, h, pair, d): carry_in[g] = s; s <- decay[g] (*) s + carry_out[g], g = 0..S-1.
// Segment g of batch element b is found at index b*batch_stride + g*seg_stride (in segments), so the
// same kernel serves segments stored as consecutive batch rows and summaries gathered rank by rank.
__global__ void __launch_bounds__(128)
compose_carries_kernel(const float* __restrict__ decay, const float* __restrict__ carry_out,
                       const float* __restrict__ h0, float* __restrict__ carry_in,
                       float* __restrict__ final_state, float* __restrict__ total_decay, int B, int S, int H,
                       int D, int N, long long batch_stride, long long seg_stride) {
    const int NH = N >> 1;
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)B * H * NH * D) return;
    const int d = (int)(idx % D);
    const int j = (int)((idx / D) % NH);
    const int hd = (int)((idx / ((long long)D * NH)) % H);
    const int b = (int)(idx / ((long long)D * NH * H));
    const long long so = (((long long)b * H + hd) * N + 2 * j) * D + d;
    float sr = 0.f, si = 0.f, pr = 1.f, pi = 0.f;
    if (h0) { sr = h0[so]; si = h0[so + D]; }
    for (int g = 0; g < S; g++) {
        const long long seg = (long long)b * batch_stride + (long long)g * seg_stride;
        const long long o = ((seg * H + hd) * N + 2 * j) * D + d;
        if (carry_in) { carry_in[o] = sr; carry_in[o + D] = si; }
        const float re = decay[(seg * H + hd) * N + 2 * j], im = decay[(seg * H + hd) * N + 2 * j + 1];
        const float nr = re * sr - im * si + carry_out[o];
        const float ni = re * si + im * sr + carry_out[o + D];
        sr = nr;
        si = ni;
        const float qr = re * pr - im * pi, qi = re * pi + im * pr;
        pr = qr;
        pi = qi;
    }
    if (final_state) { final_state[so] = sr; final_state[so + D] = si; }
    if (total_decay && d == 0) {
        total_decay[((long long)b * H + hd) * N + 2 * j] = pr;
        total_decay[((long long)b * H + hd) * N + 2 * j + 1] = pi;
    }
}

}  // namespace cdssm

using namespace cdssm;

#define DISPATCH_DTYPE(dtype, ...)                                 \
    if ((dtype) == CDSSM_BF16) { using T = __nv_bfloat16; __VA_ARGS__; } \
    else if ((dtype) == CDSSM_F32) { using T = float; __VA_ARGS__; }     \
    else return CDSSM_ERR_BAD_ARG;

extern "C" int cdssm_b200_dynamics_fwd(const void* gate_raw, const float* log_dt_scale,
                                       const float* rope_freqs, void* A_bar, void* vp_scale,
                                       void* beta, void* sel_C, float gating_c, float omega_thresh,
                                       float adt_delta, float adt_smoothness, float adt_eps, int B,
                                       int L, int H, int N, int pos0, int dtype, void* stream) {
    if (!gate_raw || !log_dt_scale || !rope_freqs || !A_bar || !vp_scale || !beta || !sel_C)
        return CDSSM_ERR_BAD_ARG;
    if (B < 0 || L < 0 || H <= 0 || N <= 0 || (N & 1)) return CDSSM_ERR_BAD_ARG;
    if (N > kMaxStateDim) return CDSSM_ERR_UNSUPPORTED;
    const long long total = (long long)B * L * H;
    if (total == 0) return CDSSM_OK;
    DynConsts c{gating_c, omega_thresh, adt_delta, adt_smoothness, adt_eps};
    const unsigned blocks = (unsigned)((total + 255) / 256);
    DISPATCH_DTYPE(dtype, (dynamics_fwd_kernel<T><<<blocks, 256, 0, (cudaStream_t)stream>>>(
                              (const T*)gate_raw, log_dt_scale, rope_freqs, (T*)A_bar,
                              (T*)vp_scale, (T*)beta, (T*)sel_C, c, total, H, N, L, pos0)));
    return check_launch();
}

extern "C" int cdssm_b200_normalize_kq_fwd(const void* K, const void* Q, void* K_out, void* Q_out,
                                           int64_t rows, int D, int dtype, void* stream) {
    if (!K || !Q || !K_out || !Q_out || rows < 0 || D <= 0) return CDSSM_ERR_BAD_ARG;
    if (rows == 0) return CDSSM_OK;
    if (((((uintptr_t)K | (uintptr_t)Q | (uintptr_t)K_out | (uintptr_t)Q_out) & 15) == 0) && (D == 64 || D == 128)) {
        DISPATCH_DTYPE(dtype, {
            auto launch = [&](auto kernel, int lanes) {
                const int per = 256 / lanes;
                kernel<<<(unsigned)((rows + per - 1) / per), 256, 0, (cudaStream_t)stream>>>((const T*)K, (const T*)Q, (T*)K_out,
                                                                                             (T*)Q_out, rows);
            };
            if (D == 64) launch(normalize_kq_fwd_rows_kernel<T, 8>, 8);
            else launch(normalize_kq_fwd_rows_kernel<T, 16>, 16);
        });
        return check_launch();
    }
    const unsigned blocks = (unsigned)((rows + 7) / 8);
    DISPATCH_DTYPE(dtype, (normalize_kq_fwd_kernel<T><<<blocks, 256, 0, (cudaStream_t)stream>>>(
                              (const T*)K, (const T*)Q, (T*)K_out, (T*)Q_out, rows, D)));
    return check_launch();
}

static int check_scan_dims(int C, int H, int D, int N) {
    if (C <= 0 || H <= 0 || D <= 0 || N <= 0 || (N & 1)) return CDSSM_ERR_BAD_ARG;
    if (N > kMaxStateDim || D > kMaxHeadDim) return CDSSM_ERR_UNSUPPORTED;
    return CDSSM_OK;
}

extern "C" int cdssm_b200_intra_chunk_scan_fwd(const void* A, const void* K, const void* V,
                                               const void* beta, void* local_h, void* cum_A,
                                               int BNC, int C, int H, int D, int N, int dtype,
                                               void* stream) {
    if (!A || !K || !V || !beta || !local_h || !cum_A || BNC < 0) return CDSSM_ERR_BAD_ARG;
    if (int rc = check_scan_dims(C, H, D, N)) return rc;
    const long long warps = (long long)BNC * H * (N / 2);
    if (warps == 0) return CDSSM_OK;
    const bool aligned = (((uintptr_t)K | (uintptr_t)local_h) & 15) == 0;   // 16-byte pieces of rows
    DISPATCH_DTYPE(dtype, {
        auto launch = [&](auto kernel, int lanes) {
            const int per = 128 / lanes;
            kernel<<<(unsigned)((warps + per - 1) / per), 128, 0, (cudaStream_t)stream>>>(
                (const T*)A, (const T*)K, (const T*)V, (const T*)beta, nullptr, (T*)local_h, (T*)cum_A, BNC, C, H, D, N, D == 8 * lanes && aligned);
        };
        if (D <= 64) launch(chunk_walk_kernel<T, 8, true>, 8);
        else launch(chunk_walk_kernel<T, 16, true>, 16);
    });
    return check_launch();
}

extern "C" int cdssm_b200_exact_correction_fwd(const void* A, const void* K, const void* beta,
                                               const void* chunk_states, void* corrections, int B,
                                               int NC, int C, int H, int D, int N, int dtype,
                                               void* stream) {
    if (!A || !K || !beta || !chunk_states || !corrections || B < 0 || NC < 0)
        return CDSSM_ERR_BAD_ARG;
    if (int rc = check_scan_dims(C, H, D, N)) return rc;
    const long long units = (long long)B * NC;
    const long long warps = units * H * (N / 2);
    if (warps == 0) return CDSSM_OK;
    const bool aligned = (((uintptr_t)K | (uintptr_t)chunk_states | (uintptr_t)corrections) & 15) == 0;
    DISPATCH_DTYPE(dtype, {
        auto launch = [&](auto kernel, int lanes) {
            const int per = 128 / lanes;
            kernel<<<(unsigned)((warps + per - 1) / per), 128, 0, (cudaStream_t)stream>>>(
                (const T*)A, (const T*)K, nullptr, (const T*)beta, (const T*)chunk_states, (T*)corrections, nullptr, units, C, H, D, N, D == 8 * lanes && aligned);
        };
        if (D <= 64) launch(chunk_walk_kernel<T, 8, false>, 8);
        else launch(chunk_walk_kernel<T, 16, false>, 16);
    });
    return check_launch();
}

extern "C" int cdssm_b200_inter_chunk_scan_fwd(const void* total_A, const void* final_local_h,
                                               void* chunk_states, int B, int NC, int H, int D,
                                               int N, int dtype, void* stream) {
    if (!total_A || !final_local_h || !chunk_states || B < 0 || NC < 0) return CDSSM_ERR_BAD_ARG;
    if (int rc = check_scan_dims(1, H, D, N)) return rc;
    const long long threads = (long long)B * H * (N / 2) * D;
    if (threads == 0 || NC == 0) return CDSSM_OK;
    const unsigned blocks = (unsigned)((threads + 127) / 128);
    DISPATCH_DTYPE(dtype, (inter_chunk_fwd_kernel<T><<<blocks, 128, 0, (cudaStream_t)stream>>>(
                              (const T*)total_A, (const T*)final_local_h, (T*)chunk_states, B, NC,
                              H, D, N)));
    return check_launch();
}

extern "C" int cdssm_b200_conv1d_silu_strided_fwd(const void* x, int64_t x_row_stride, const void* weight, const void* bias,
                                                  void* out, void* hist, int B, int L, int Dm, int dtype, void* stream) {
    if (!x || !weight || !bias || !out || B < 0 || L < 0 || Dm <= 0) return CDSSM_ERR_BAD_ARG;
    if (x_row_stride == 0) x_row_stride = Dm;
    if (x_row_stride < Dm) return CDSSM_ERR_BAD_ARG;
    if (B == 0 || L == 0) return CDSSM_OK;
    if (B > 65535) return CDSSM_ERR_UNSUPPORTED;
    cudaStream_t st = (cudaStream_t)stream;
    const size_t es = dtype == CDSSM_F32 ? 4 : 2;
    const uintptr_t all = (uintptr_t)x | (uintptr_t)weight | (uintptr_t)bias | (uintptr_t)out | (uintptr_t)hist |
                          (uintptr_t)(x_row_stride * es);
    if (Dm % 4 == 0 && (all & (4 * es - 1)) == 0) {
        const int cols = (Dm / 4 + 127) / 128;
        const bool many = (long long)cols * ((L + 31) / 32) * B >= 148 * 8;
        const int segs = many ? (L + 31) / 32 : (L + 7) / 8;
        if (segs > 65535) return CDSSM_ERR_UNSUPPORTED;
        const dim3 grid(cols, segs, B);
        DISPATCH_DTYPE(dtype, {
            auto launch = [&](auto kernel) {
                return launch_overlapped(kernel, grid, dim3(128), 0, st, (const T*)x, x_row_stride, (const T*)weight, (const T*)bias,
                                         (T*)out, (T*)hist, L, Dm);
            };
            return many ? launch(conv1d_silu_vec_kernel<T, 32>) : launch(conv1d_silu_vec_kernel<T, 8>);
        });
    }
    constexpr int kSeg = 32;
    dim3 grid((Dm + 127) / 128, (L + kSeg - 1) / kSeg, B);
    if (grid.y > 65535) return CDSSM_ERR_UNSUPPORTED;
    DISPATCH_DTYPE(dtype, (conv1d_silu_fwd_kernel<T, kSeg><<<grid, 128, 0, st>>>(
                              (const T*)x, x_row_stride, (const T*)weight, (const T*)bias, (T*)out, (T*)hist, L, Dm)));
    return check_launch();
}

extern "C" int cdssm_b200_conv1d_silu_fwd(const void* x, const void* weight, const void* bias,
                                          void* out, int B, int L, int Dm, int dtype,
                                          void* stream) {
    return cdssm_b200_conv1d_silu_strided_fwd(x, Dm, weight, bias, out, nullptr, B, L, Dm, dtype, stream);
}

extern "C" int cdssm_b200_compose_carries(const float* decay, const float* carry_out, const float* h0,
                                          float* carry_in, float* final_state, float* total_decay, int B,
                                          int S, int H, int D, int N, int64_t batch_stride,
                                          int64_t seg_stride, void* stream) {
    if (!decay || !carry_out || B < 0 || S < 0) return CDSSM_ERR_BAD_ARG;
    if (int rc = check_scan_dims(1, H, D, N)) return rc;
    const long long threads = (long long)B * H * (N / 2) * D;
    if (threads == 0) return CDSSM_OK;
    compose_carries_kernel<<<(unsigned)((threads + 127) / 128), 128, 0, (cudaStream_t)stream>>>(
        decay, carry_out, h0, carry_in, final_state, total_decay, B, S, H, D, N, batch_stride, seg_stride);
    return check_launch();
}
