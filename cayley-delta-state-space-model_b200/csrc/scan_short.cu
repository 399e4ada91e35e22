// The walk by steps (scan_simt.cu) for few units: a call whose (chunk, head, pair) units leave the SMs a warp or two each is as long as
// the chain of a chunk's steps, and a step as long as the instructions of its warp, so all that the chain need not wait for goes to
// another warp or comes before it.  The same operations on the same operands in the same order, bit for bit: either kernel may run, by size.
//   - Rows come 32 tokens at a time through shared memory, and with them the norms, k.q and the scalars of a step, a lane per token:
//     beside the pass before this one.
//   - In the output pass a unit has sixteen lanes of two warps, eight for z and eight for the correction r, the same instructions on
//     another state.  The first warp has the chain, the sums z.k and r.k and the update; it leaves K, the coefficient that a step adds
//     along its key, and the second warp walks behind it with K at hand for the products with q, which stay in parts, a lane's own,
//     until they are summed up for 32 tokens at a time, a lane per token.
#include "row_slice.cuh"
#include "scan_args.cuh"
#include "sm100_ptx.cuh"
#include <type_traits>

namespace cdssm {
namespace shortwalk {

constexpr int kStage = 32;   // tokens

// shared memory of a thread block (two warps), bytes
template <typename T, int kCols, bool kOutput>
struct Geo {
    static constexpr int kGroup = kOutput ? 16 : 8, kUnits = 32 / kGroup, kM = kOutput ? 2 : 1;
    static constexpr int kRow = 8 * kCols * (int)sizeof(T) + 16;       // rows whose 16-byte pieces eight lanes read at once lie on distinct banks
    static constexpr int kRows = kUnits * kM * 2 * kStage * kRow;      // [unit][k, q][two stages]
    static constexpr int kScal = kUnits * 2 * kStage * 48;             // [unit][two stages]: {a, beta n^2, beta n}, {v, k.q, 1 / |q|}, {n, sel_C, -, -}
    static constexpr int kPart = kOutput ? kStage * 33 * 8 : 0;        // [token][lane]: parts of q.z, q.r
    static constexpr int kCoef = kOutput ? 2 * kStage * 4 * 8 : 0;     // [two stages][token][unit][z, r]: K
    static constexpr int kBytes = kRows + kScal + kPart + kCoef;
};

// the order of a butterfly over eight lanes
__device__ __forceinline__ float tree(const float (&p)[8]) { return ((p[0] + p[1]) + (p[2] + p[3])) + ((p[4] + p[5]) + (p[6] + p[7])); }

template <typename T, int kCols, bool kOutput>
__global__ void __launch_bounds__(64, 1) scan_short_kernel(const __grid_constant__ ScanArgs a, const int from_chunks) {
    using G = Geo<T, kCols, kOutput>;
    constexpr int kGroup = G::kGroup, kUnits = G::kUnits, kM = G::kM, kRow = G::kRow, kP = kCols / 2, D = 8 * kCols;
    constexpr int kPieces = kCols * (int)sizeof(T) / 16;
    extern __shared__ __align__(16) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane & 7, ul = lane / kGroup;
    const bool second = kOutput && (lane & 8);           // the correction's lanes
    float* scal0 = reinterpret_cast<float*>(smem + G::kRows);
    float2* xq = reinterpret_cast<float2*>(smem + G::kRows + G::kScal);
    float2* coef = reinterpret_cast<float2*>(smem + G::kRows + G::kScal + G::kPart);
    const int NH = a.N >> 1, C = a.C, H = a.H, NC = a.NC;
    struct Place { int j, hd, c, b; };
    auto place = [&](int i) {                            // of unit i of this block (behind the end: the last one again, not written)
        const unsigned u = min(blockIdx.x * kUnits + i, (unsigned)a.units - 1);
        const unsigned h = u / NH, n = h / H, b = n / NC;
        return Place{(int)(u - h * NH), (int)(h - n * H), (int)(n - b * NC), (int)b};
    };
    const Place own = place(ul);
    const int j = own.j, hd = own.hd, c = own.c, b = own.b;
    const bool active = blockIdx.x * kUnits + ul < (unsigned)a.units;
    const int Lc = min(C, a.L - c * C);                  // valid tokens of this chunk
    const int Lw = __reduce_max_sync(0xffffffffu, Lc);   // (the units of a warp may sit in different chunks)
    const size_t sidx = (((size_t)b * NC + c) * H + hd) * NH + j;

    // rows of stage s; a token behind the end: zeros (ssd.py:60-67)
    auto fetch = [&](int s) {
        if (s * kStage < Lw) {
#pragma unroll
            for (int m = 0; m < kM; m++) {
                const long long rs = m ? a.q_rs : a.k_rs;
                const T* from = static_cast<const T*>(m ? a.q : a.k) + ((long long)b * a.L + (long long)c * C) * rs + (long long)hd * D;
                unsigned char* to = smem + ((ul * kM + m) * 2 + (s & 1)) * (kStage * kRow);
#pragma unroll 4
                for (int t = 2 * ((lane % kGroup) >> 3) + warp; t < kStage; t += kGroup / 4) {   // (eight lanes a row)
                    const int tok = s * kStage + t;
#pragma unroll
                    for (int p = 0; p < kPieces; p++)
                        sm100::cp_async16(to + t * kRow + (p * 8 + g) * 16, from + min(tok, Lc - 1) * rs + (p * 8 + g) * (16 / (int)sizeof(T)), tok < Lc);
                }
            }
        }
        sm100::cp_async_commit();
    };
    auto slice = [&](const unsigned char* row, float (&x)[kCols], int i) {   // columns i kCols ...
#pragma unroll
        for (int p = 0; p < kPieces; p++) {
            const uint4 w = *reinterpret_cast<const uint4*>(row + (i * kPieces + p) * 16);
            if constexpr (IO<T>::kBf16) {
                unpack8(w, x + 8 * p);
            } else {
                x[4 * p] = __uint_as_float(w.x); x[4 * p + 1] = __uint_as_float(w.y);
                x[4 * p + 2] = __uint_as_float(w.z); x[4 * p + 3] = __uint_as_float(w.w);
            }
        }
    };
    // what stage s's steps take from the rows alone, a lane per token: |k|^-1, k.q, |q|^-1 (each warp half of the units)
    auto norms = [&](int s) {
        if (s * kStage >= Lw) return;
#pragma unroll 1
        for (int i = warp; i < kUnits; i += 2) {
            const unsigned char* base = smem + (i * kM * 2 + (s & 1)) * (kStage * kRow) + lane * kRow;
            float kk[8], kq[8], qq[8];
#pragma unroll
            for (int n = 0; n < 8; n++) {
                float2 x[kP], y[kP], s0 = make_float2(0.f, 0.f), s1 = s0, s2 = s0;
                slice(base, reinterpret_cast<float(&)[kCols]>(x), n);
                if (kOutput) slice(base + 2 * kStage * kRow, reinterpret_cast<float(&)[kCols]>(y), n);
#pragma unroll
                for (int e = 0; e < kP; e++) {
                    s0 = __ffma2_rn(x[e], x[e], s0);
                    if (kOutput) {
                        s1 = __ffma2_rn(x[e], y[e], s1);
                        s2 = __ffma2_rn(y[e], y[e], s2);
                    }
                }
                kk[n] = s0.x + s0.y;
                if (kOutput) { kq[n] = s1.x + s1.y; qq[n] = s2.x + s2.y; }
            }
            float* to = scal0 + ((i * 2 + (s & 1)) * kStage + lane) * 12;
            to[8] = rsqrtf(tree(kk) + kEps);
            if (kOutput) *reinterpret_cast<float2*>(to + 6) = make_float2(tree(kq), rsqrtf(tree(qq) + kEps));
        }
    };
    // the dynamics of kN stages from s on, a lane per token
    constexpr int kMine = kUnits / 2;
    Place mine[kMine];
#pragma unroll
    for (int i = 0; i < kMine; i++) mine[i] = place(warp + 2 * i);
    auto scalars = [&](int s, auto count) {
        constexpr int kN = decltype(count)::value;
        float4 av[kN][kMine];
        float2 bs[kN][kMine];
#pragma unroll
        for (int n = 0; n < kN; n++)
#pragma unroll
            for (int i = 0; i < kMine; i++) {
                const Place& m = mine[i];
                const int tok = (s + n) * kStage + lane;
                av[n][i] = make_float4(0.f, 0.f, 0.f, 0.f);
                bs[n][i] = make_float2(0.f, 0.f);
                if (tok < min(C, a.L - m.c * C)) {
                    const size_t unit = ((size_t)m.b * NC + m.c) * H + m.hd;
                    if (a.rec_av != nullptr) {
                        av[n][i] = __ldcg(a.rec_av + (unit * NH + m.j) * C + tok);
                        bs[n][i] = __ldcg(a.rec_bs + unit * C + tok);
                    } else {
                        const TokenDynamics<T> d(a, m.b, m.c * C + tok, m.hd);
                        av[n][i] = d.pair(m.j);
                        bs[n][i] = d.beta_sel();
                    }
                }
            }
#pragma unroll
        for (int n = 0; n < kN; n++)
#pragma unroll
            for (int i = 0; i < kMine; i++) {
                float* to = scal0 + (((warp + 2 * i) * 2 + ((s + n) & 1)) * kStage + lane) * 12;
                const float ik = to[8], bik = bs[n][i].x * ik;
                *reinterpret_cast<float4*>(to) = make_float4(av[n][i].x, av[n][i].y, bik * ik, bik);
                *reinterpret_cast<float2*>(to + 4) = make_float2(av[n][i].z, av[n][i].w);
                to[9] = bs[n][i].y;
            }
        __syncthreads();
    };

    // The local pass waits for the records, whose kernel starts when everything before it is done (rows and gates are there); the output
    // pass is launched when the one before it has waited for what lies before that, and waits for the states only.
    if (!kOutput && a.rec_av == nullptr) grid_dependency_wait();
    fetch(0);
    fetch(1);
    sm100::cp_async_wait_group<0>();
    __syncthreads();
    norms(0);
    norms(1);
    if (!kOutput) {
        if (a.rec_av != nullptr) grid_dependency_wait();
        grid_launch_dependents();
    }
    scalars(0, std::integral_constant<int, 2>());
    if (kOutput) grid_dependency_wait();

    const float2 zero2 = make_float2(0.f, 0.f);
    float2 xr[kP], xi[kP];                               // z or r, a lane's columns in pairs (both warps of an output pass have them)
#pragma unroll
    for (int i = 0; i < kP; i++) { xr[i] = xi[i] = zero2; }
    if (kOutput) {
        auto state = [&](const float* s) {
#pragma unroll
            for (int i = 0; i < kP; i++) {
                const int d = g * kCols + 2 * i;
                xr[i] = make_float2(__ldcg(s + d), __ldcg(s + d + 1));
                xi[i] = make_float2(__ldcg(s + D + d), __ldcg(s + D + d + 1));
            }
        };
        if (second && !from_chunks) state(a.ws_state + sidx * 2 * D);
        if (second && from_chunks) {                     // s <- gamma s + z over the chunks before
            const size_t head = (((size_t)b * H + hd) * NH + j) * 2 * D;
            if (a.h0) state(a.h0 + head);
            float2 s0r[kP], s0i[kP];
            auto into_chunk = [&]() {
#pragma unroll
                for (int i = 0; i < kP; i++) { s0r[i] = xr[i]; s0i[i] = xi[i]; }
            };
            const bool last = c + 1 == NC && a.final_state != nullptr && warp == 1;   // (the last chunk's own step too)
            const int chunks = c + (last ? 1 : 0);
            constexpr int kBatch = 32 / kCols;
#pragma unroll 1
            for (int n0 = 0; n0 < chunks; n0 += kBatch) {
                float2 lr[kBatch][kP], li[kBatch][kP], gm[kBatch];
#pragma unroll
                for (int k = 0; k < kBatch; k++) {
                    const size_t w = (((size_t)b * NC + min(n0 + k, chunks - 1)) * H + hd) * NH + j;
                    gm[k] = __ldcg(reinterpret_cast<const float2*>(a.ws_gamma) + w);
                    const float2* s = reinterpret_cast<const float2*>(a.ws_state + w * 2 * D + g * kCols);
#pragma unroll
                    for (int i = 0; i < kP; i++) { lr[k][i] = __ldcg(s + i); li[k][i] = __ldcg(s + D / 2 + i); }
                }
#pragma unroll
                for (int k = 0; k < kBatch; k++) {
                    if (n0 + k >= chunks) break;
                    if (n0 + k == c) into_chunk();
#pragma unroll
                    for (int i = 0; i < kP; i++) {
                        const float r0 = next_re(gm[k], xr[i].x, xi[i].x, lr[k][i].x), r1 = next_re(gm[k], xr[i].y, xi[i].y, lr[k][i].y);
                        xi[i] = make_float2(next_im(gm[k], xr[i].x, xi[i].x, li[k][i].x), next_im(gm[k], xr[i].y, xi[i].y, li[k][i].y));
                        xr[i] = make_float2(r0, r1);
                    }
                }
            }
            if (!last) into_chunk();
            else if (active) {
#pragma unroll
                for (int i = 0; i < kP; i++) {
                    float* to = a.final_state + head + g * kCols + 2 * i;
                    to[0] = xr[i].x; to[1] = xr[i].y; to[D] = xi[i].x; to[D + 1] = xi[i].y;
                }
            }
#pragma unroll
            for (int i = 0; i < kP; i++) {               // (chunk_states store)
                xr[i] = make_float2(IO<T>::rnd(s0r[i].x), IO<T>::rnd(s0r[i].y));
                xi[i] = make_float2(IO<T>::rnd(s0i[i].x), IO<T>::rnd(s0i[i].y));
            }
        }
        __syncwarp();
        grid_launch_dependents();
    }
    float cr = 1.f, ci = 0.f;
    // K from the first warp to the second, eight steps at a time: a barrier for every eight steps of two stages.  (At the third stage
    // and later ones both warps have met in between.)
    auto step_barrier = [](int s, int t) { return 1 + (s & 1) * (kStage / 8) + t / 8; };

#pragma unroll 1
    for (int s = 0; s * kStage < Lw; s++) {
        if (s > 0 && Lw > 2 * kStage) {
            __syncthreads();                             // (both are done with stage s - 1, whose place stage s + 1 takes)
            fetch(s + 1);
            if (s > 1) {
                sm100::cp_async_wait_group<1>();
                __syncthreads();
                norms(s);
                scalars(s, std::integral_constant<int, 1>());
            }
        }
        const unsigned char* kr = smem + (ul * kM * 2 + (s & 1)) * (kStage * kRow);
        const unsigned char* qr = kr + 2 * kStage * kRow;
        const float* sc = scal0 + (ul * 2 + (s & 1)) * (kStage * 12);
        float2* cf = coef + (s & 1) * (kStage * 4) + ul * 2 + (second ? 1 : 0);   // 4 t + ...
        const int steps = min(kStage, Lw - s * kStage);
        auto rotated = [&](float4 s1, float2 (&tr)[kP], float2 (&ti)[kP]) {   // a x
            const float2 are2 = make_float2(s1.x, s1.x), aim2 = make_float2(s1.y, s1.y), nim2 = make_float2(-s1.y, -s1.y);
#pragma unroll
            for (int i = 0; i < kP; i++) {
                tr[i] = __ffma2_rn(are2, xr[i], __fmul2_rn(nim2, xi[i]));
                ti[i] = __ffma2_rn(are2, xi[i], __fmul2_rn(aim2, xr[i]));
            }
        };
        auto add = [&](float Kr, float Ki, const float2 (&kk)[kP], const float2 (&tr)[kP], const float2 (&ti)[kP]) {
            const float2 kr2 = make_float2(Kr, Kr), ki2 = make_float2(Ki, Ki);
#pragma unroll
            for (int i = 0; i < kP; i++) {
                xr[i] = __ffma2_rn(kr2, kk[i], tr[i]);
                xi[i] = __ffma2_rn(ki2, kk[i], ti[i]);
            }
        };
        if (warp == 0) {
            // Every dot product of the step is taken against the state BEFORE the update.
            float2 kk[kP];
            slice(kr, reinterpret_cast<float(&)[kCols]>(kk), g);
            float4 s1 = *reinterpret_cast<const float4*>(sc);
            float2 v = *reinterpret_cast<const float2*>(sc + 4);
#pragma unroll 2
            for (int t = 0; t < steps; t++) {
                float2 kn[kP];                           // what the next step needs
                const int tn = min(t + 1, kStage - 1);
                slice(kr + tn * kRow, reinterpret_cast<float(&)[kCols]>(kn), g);
                const float4 n1 = *reinterpret_cast<const float4*>(sc + 12 * tn);
                const float2 nv = *reinterpret_cast<const float2*>(sc + 12 * tn + 4);
                float2 sr2 = zero2, si2 = zero2;
#pragma unroll
                for (int i = 0; i < kP; i++) {
                    sr2 = __ffma2_rn(xr[i], kk[i], sr2);
                    si2 = __ffma2_rn(xi[i], kk[i], si2);
                }
                float sr = sr2.x + sr2.y, si = si2.x + si2.y;
                float2 tr[kP], ti[kP];
                rotated(s1, tr, ti);
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) {
                    const float x = __shfl_xor_sync(0xffffffffu, sr, o), y = __shfl_xor_sync(0xffffffffu, si, o);
                    sr += x;
                    si += y;
                }
                // z' = a (z - beta (z.k^) k^) + beta v k^ = a z + K k;  r' = a (r - beta (r.k^) k^)
                const float cre = __fmul_rn(s1.z, sr), cim = __fmul_rn(s1.z, si);
                const float Kr = __fmaf_rn(s1.w, second ? 0.f : v.x, -msub(s1.x, cre, s1.y, cim));
                const float Ki = __fmaf_rn(s1.w, second ? 0.f : v.y, -madd(s1.x, cim, s1.y, cre));
                add(Kr, Ki, kk, tr, ti);
                if (kOutput) {
                    if (g == 0) cf[4 * t] = make_float2(Kr, Ki);
                    if ((t & 7) == 7 || t == steps - 1) {
                        __syncwarp();
                        asm volatile("bar.arrive %0, 64;" ::"r"(step_barrier(s, t)) : "memory");
                    }
                } else {
                    const float ncr = msub(s1.x, cr, s1.y, ci), nci = madd(s1.x, ci, s1.y, cr);
                    cr = ncr;
                    ci = nci;
                }
#pragma unroll
                for (int i = 0; i < kP; i++) kk[i] = kn[i];
                s1 = n1;
                v = nv;
            }
        } else if (kOutput) {
            const int tail_t = a.tail_state != nullptr && active ? a.L - 1 - c * C - s * kStage : -1;
#pragma unroll 1
            for (int t0 = 0; t0 < steps; t0 += 8) {
                asm volatile("bar.sync %0, 64;" ::"r"(step_barrier(s, t0)) : "memory");
#pragma unroll 2
                for (int t = t0; t < min(t0 + 8, steps); t++) {
                    float2 kk[kP], qq[kP], tr[kP], ti[kP], qr2 = zero2, qi2 = zero2;
                    slice(kr + t * kRow, reinterpret_cast<float(&)[kCols]>(kk), g);
                    slice(qr + t * kRow, reinterpret_cast<float(&)[kCols]>(qq), g);
                    const float4 s1 = *reinterpret_cast<const float4*>(sc + 12 * t);
                    const float2 K = cf[4 * t];
#pragma unroll
                    for (int i = 0; i < kP; i++) {
                        qr2 = __ffma2_rn(xr[i], qq[i], qr2);
                        qi2 = __ffma2_rn(xi[i], qq[i], qi2);
                    }
                    xq[t * 33 + lane] = make_float2(qr2.x + qr2.y, qi2.x + qi2.y);
                    rotated(s1, tr, ti);
                    add(K.x, K.y, kk, tr, ti);
                    if (a.tail_state != nullptr && __any_sync(0xffffffffu, t == tail_t)) {   // z + r
                        float* ts = a.tail_state + (((size_t)b * H + hd) * a.N + 2 * j) * D + g * kCols;
                        const bool here = t == tail_t && !second;
#pragma unroll
                        for (int i = 0; i < kP; i++) {
                            auto sum = [](float x) { return x + __shfl_xor_sync(0xffffffffu, x, 8); };
                            const float2 re = make_float2(sum(xr[i].x), sum(xr[i].y)), im = make_float2(sum(xi[i].x), sum(xi[i].y));
                            if (here) { ts[2 * i] = re.x; ts[2 * i + 1] = re.y; ts[D + 2 * i] = im.x; ts[D + 2 * i + 1] = im.y; }
                        }
                    }
                }
            }
            __syncwarp();
            // read-outs of the stage: sixteen lanes a unit, a lane per token; the post-step product follows from
            // z' = a z + K k  =>  z'.q = a (z.q) + K (k.q)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int tt = 16 * h + (lane & 15), tok = s * kStage + tt;
                if (tok < Lc && active) {
                    const float2* x = xq + tt * 33 + (lane & 16);
                    float zr[8], zi[8], rr[8], ri[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        zr[i] = x[i].x; zi[i] = x[i].y;
                        rr[i] = x[8 + i].x; ri[i] = x[8 + i].y;
                    }
                    const float zqr = tree(zr), zqi = tree(zi), rqr = tree(rr), rqi = tree(ri);
                    const float2 K = coef[(s & 1) * (kStage * 4) + 4 * tt + 2 * ul];
                    const float* t1 = sc + 12 * tt;
                    const float kq = t1[6], iq = t1[7];
                    // correction is read BEFORE its step (exact_correction.cu:90-94), the local state after
                    float yr = __fmul_rn(iq, read_re(rqr, t1[0], t1[1], zqr, zqi, K.x, kq));
                    float yi = __fmul_rn(iq, read_im(rqi, t1[0], t1[1], zqr, zqi, K.y, kq));
                    if (a.shortcut_scale != 0.f) {   // block.py:202-208: sum_d shortcut[s,d] q[d] = (q^.k^)^2 v[s]
                        const float qk = __fmul_rn(__fmul_rn(iq, t1[8]), kq), f = __fmul_rn(__fmul_rn(a.shortcut_scale, qk), qk);
                        yr = __fmaf_rn(f, t1[4], yr);
                        yi = __fmaf_rn(f, t1[5], yi);
                    }
                    T* o = static_cast<T*>(a.y) + (((long long)b * a.L + c * C + tok) * H + hd) * a.N + 2 * j;
                    IO<T>::st(o, IO<T>::rnd(IO<T>::rnd(yr) * t1[9]));
                    IO<T>::st(o + 1, IO<T>::rnd(IO<T>::rnd(yi) * t1[9]));
                }
            }
            __syncwarp();
        }
    }
    if (!kOutput && warp == 0 && active) {
        const bool whole = Lc == C;                      // zero padding wipes the local state and the decay product
        // the carry pass consumes these as the reference's bf16 cum_A[:, -1] / local_h[:, -1]
        float* s = a.ws_state + sidx * 2 * D + g * kCols;
#pragma unroll
        for (int i = 0; i < kP; i++) {
            *reinterpret_cast<float2*>(s + 2 * i) = whole ? make_float2(IO<T>::rnd(xr[i].x), IO<T>::rnd(xr[i].y)) : zero2;
            *reinterpret_cast<float2*>(s + D + 2 * i) = whole ? make_float2(IO<T>::rnd(xi[i].x), IO<T>::rnd(xi[i].y)) : zero2;
        }
        if (g == 0) *reinterpret_cast<float2*>(a.ws_gamma + sidx * 2) = whole ? make_float2(IO<T>::rnd(cr), IO<T>::rnd(ci)) : zero2;
    }
}

template <typename T, int kCols, bool kOutput> struct KernelTag {};

template <typename T, int kCols, bool kOutput>
static int launch(const ScanArgs& a, int from_chunks, cudaStream_t st) {
    using G = Geo<T, kCols, kOutput>;
    static_assert(G::kBytes <= 227 * 1024, "shared memory");
    if (int rc = allow_smem<KernelTag<T, kCols, kOutput>>((const void*)scan_short_kernel<T, kCols, kOutput>, G::kBytes)) return rc;
    return launch_overlapped(scan_short_kernel<T, kCols, kOutput>, dim3((unsigned)((a.units + G::kUnits - 1) / G::kUnits)), dim3(64), G::kBytes, st, a,
                             from_chunks);
}
template <typename T>
static int launch_shape(bool output, const ScanArgs& a, int from_chunks, cudaStream_t st) {
    if (a.D == 64) return output ? launch<T, 8, true>(a, from_chunks, st) : launch<T, 8, false>(a, from_chunks, st);
    return output ? launch<T, 16, true>(a, from_chunks, st) : launch<T, 16, false>(a, from_chunks, st);
}

}  // namespace shortwalk

// As many units as have their rows in shared memory at once, in the output pass: float32 of head_dim 64 four an SM, bf16 eight; half of
// that for 128.  us of a call on B200, walk / this: float32, D 64, 64 units 45.1 / 28.9, 384 47.4 / 34.3, 768 49.4 / 49.4, 1536 50 / 74; D 128,
// 64 129 / 82, 384 139 / 130, 768 133 / 205; bf16, D 64, 240 46.8 / 31.0, 768 49.2 / 39.2, 1536 49.7 / 54.8; D 128, 192 105 / 70, 768
// 108 / 111.
bool scan_short_takes(const ScanArgs& a, int dtype, int sms) {
    using namespace shortwalk;
    const int es = dtype == CDSSM_F32 ? 4 : 2;
    const size_t block = a.D == 64 ? (es == 4 ? Geo<float, 8, true>::kBytes : Geo<__nv_bfloat16, 8, true>::kBytes)
                                   : (es == 4 ? Geo<float, 16, true>::kBytes : Geo<__nv_bfloat16, 16, true>::kBytes);
    const long long an_sm = 2 * (long long)((size_t)227 * 1024 / (block + 1024));
    return (a.D == 64 || a.D == 128) && ((a.k_rs | a.q_rs) * es) % 16 == 0 && a.units <= an_sm * sms;
}

int scan_short_pass(bool output, const ScanArgs& a, int dtype, int from_chunks, cudaStream_t st) {
    return dtype == CDSSM_F32 ? shortwalk::launch_shape<float>(output, a, from_chunks, st) : shortwalk::launch_shape<__nv_bfloat16>(output, a, from_chunks, st);
}

}  // namespace cdssm
