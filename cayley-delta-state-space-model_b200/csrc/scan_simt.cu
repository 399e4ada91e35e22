// Fused CD-SSM scan on CUDA cores (the general path: any even N <= 32, D <= 128, C <= 256,
// bf16 or fp32 storage).  scan_short.cu has the same walk for few units of head_dim 64 and 128.
//
// Reference chunk semantics (cdssm/models/ssd.py:56-111 over intra_chunk_scan.cu:100-195,
// inter_chunk_scan.cu:52-84, exact_correction.cu:89-150), per head and complex pair:
//   z_t : local state, zero at the start of every chunk, delta-rule step per token;
//   s_c : carry into chunk c,  s_{c+1} = gamma_c * s_c + z_{C-1}   (decay product only);
//   r_t : correction, r_0 = s_c, erase+rotate per token, taken BEFORE step t;
//   y_t = sel_C * ((z_t + r_t) . q_t + shortcut).
// Nothing of size (B,L,H,N,D) is stored.  Three launches:
//   local pass  : per (chunk, head, pair) walk z only -> gamma_c and z_{C-1}  (workspace)
//   carry pass  : per (batch, head, pair, d) serial over chunks -> s_c in place of z_{C-1}
//   output pass : per (chunk, head, pair) walk z and r together, read out y
// The local pass re-reads k, v and the gates (about half of the algorithmic bytes).  scan_wa.cu and
// scan_tile.cu hold the tensor-core kernels for the shapes they take; the carry pass here serves both.
//
// Thread mapping: eight lanes own one (chunk, head, pair) unit, each lane D/8 contiguous
// columns of the two state rows, so a k/q row is fetched with 16-byte loads and a dot product
// costs three shuffles.  The sixteen units of a block are consecutive (head, pair) of one chunk
// wherever H*N/2 allows, which makes the strided gate and v reads of a block contiguous.
// The dynamics of a chunk are computed once per unit into shared memory before the walk.
#include "cdssm_common.cuh"
#include "decode_unit.cuh"
#include "scan_args.cuh"
#include "sm100_ptx.cuh"
#include <atomic>

namespace cdssm {

constexpr int kUnitsPerBlock = 16;
constexpr int kSimtThreads = kLanesPerUnit * kUnitsPerBlock;   // 128
constexpr int kMaxChunk = 256;

// Shared-memory staging of one chunk's per-token scalars for the 16 units of a block.
struct ChunkScalars {
    float *a_re, *a_im, *beta, *v_re, *v_im, *sel_c;   // each [kUnitsPerBlock][C]
    __device__ ChunkScalars(float* base, int C, int units_per_block = kUnitsPerBlock) {
        const int n = units_per_block * C;
        a_re = base; a_im = base + n; beta = base + 2 * n; v_re = base + 3 * n;
        v_im = base + 4 * n; sel_c = base + 5 * n;
    }
};

// The dynamics of every (token, head) before the walks: a warp takes four tokens of eight heads.  Computed by the walks
// themselves, eight tokens in a row per lane, they were 10 us (float32: 15) of each of the two walks whatever the size.
template <typename T>
__global__ void __launch_bounds__(256) simt_records_kernel(const ScanArgs a, const bool early) {
    const int lt = threadIdx.x >> 3 & 3, lh = threadIdx.x & 7, warp = threadIdx.x >> 5;
    if (early) grid_launch_dependents();
    const long long tok = (long long)blockIdx.x * 32 + warp * 4 + lt;
    const int hd = blockIdx.y * 8 + lh;
    if (tok >= (long long)a.B * a.L || hd >= a.H) return;
    const int b = (int)(tok / a.L), l = (int)(tok % a.L), c = l / a.C, t = l % a.C, NH = a.N >> 1;
    const TokenDynamics<T> d(a, b, l, hd);
    const size_t unit = ((size_t)b * a.NC + c) * a.H + hd;
    a.rec_bs[unit * a.C + t] = d.beta_sel();
    for (int j = blockIdx.z; j < NH; j += gridDim.z) a.rec_av[(unit * NH + j) * a.C + t] = d.pair(j);
    // (at the end where these blocks fill the SMs: dependents that start meanwhile are packed onto the few with room, and a walk of
    // 24 blocks of head_dim 128 took 104 us instead of 21)
    if (!early) grid_launch_dependents();
}

// Scalars of the unit's chunk into shared memory: lane g handles tokens g, g+8, ...  Padded positions (l >= L) get
// a = k = v = beta = 0 like the reference's zero padding (ssd.py:60-67).
template <typename T, int kLanes>
__device__ __forceinline__ void stage_dynamics(const ScanArgs& a, ChunkScalars& sm, int ul, int g,
                                               int b, int c, int hd, int j) {
    const int Lc = min(a.C, a.L - c * a.C), o0 = ul * a.C;
    const size_t unit = ((size_t)b * a.NC + c) * a.H + hd;
    auto put = [&](int t, float4 av, float2 bs) {
        sm.a_re[o0 + t] = av.x; sm.a_im[o0 + t] = av.y; sm.beta[o0 + t] = bs.x;
        sm.v_re[o0 + t] = av.z; sm.v_im[o0 + t] = av.w; sm.sel_c[o0 + t] = bs.y;
    };
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    if (a.rec_av != nullptr) {
        const float4* av = a.rec_av + (unit * (a.N >> 1) + j) * a.C;
        const float2* bs = a.rec_bs + unit * a.C;
#pragma unroll 8
        for (int t = g; t < Lc; t += kLanes) put(t, __ldcg(av + t), __ldcg(bs + t));
    } else {
        for (int t = g; t < Lc; t += kLanes) {
            const TokenDynamics<T> d(a, b, c * a.C + t, hd);
            put(t, d.pair(j), d.beta_sel());
        }
    }
    for (int t = Lc + (g - Lc % kLanes + kLanes) % kLanes; t < a.C; t += kLanes) put(t, zero, make_float2(0.f, 0.f));
}

// kOutput = false: local pass (z only).  kOutput = true: output pass (z, r, read-out).
// kRing: rows that travel ahead of the step that uses them, as asynchronous copies to shared memory (a lane reads only what it has
// copied itself: no barrier).  0: the next row only, in registers.  A step of a short walk takes less time than a row does to come.
template <typename T, int kCols, int kLanes, bool kOutput, int kRing>
// (No register cap: at most 6 resident blocks of 80 registers cost the output walk its overlap of a step's eleven sums, float32
// 61 -> 34 us at 64 units and 173 -> 90 us at head_dim 128, bf16 with a full GPU 380 -> 368 us.)
__global__ void __launch_bounds__(kSimtThreads, 1)
scan_walk_kernel(const ScanArgs a) {
    constexpr int kUnits = kSimtThreads / kLanes;       // units per block
    extern __shared__ float smem[];
    ChunkScalars sm(smem, a.C, kUnits);
    const int ul = threadIdx.x / kLanes;                 // unit within the block
    const int g = threadIdx.x % kLanes;                  // lane within the unit
    long long u = (long long)blockIdx.x * kUnits + ul;
    const bool active = u < a.units;
    if (!active) u = a.units - 1;                        // keep the lane in the shuffles
    const int NH = a.N >> 1, D = a.D, C = a.C, H = a.H;
    const int j = (int)(u % NH);
    const int hd = (int)((u / NH) % H);
    const int c = (int)((u / ((long long)NH * H)) % a.NC);
    const int b = (int)(u / ((long long)NH * H * a.NC));
    const bool vec = (D == kCols * kLanes);              // rows are 16-byte aligned slices

    // The local walk waits for the records; the output walk is launched when the carry pass, which has waited for the local
    // one, begins: the records are there, and it waits for the carries only.
    if (!kOutput) grid_dependency_wait();
    stage_dynamics<T, kLanes>(a, sm, ul, g, b, c, hd, j);
    if (kOutput) grid_dependency_wait();
    __syncwarp();

    const int Lc = min(C, a.L - c * C);                  // valid tokens of this chunk
    const T* kbase = static_cast<const T*>(a.k) + ((long long)b * a.L + (long long)c * C) * a.k_rs + (long long)hd * D;
    const T* qbase = static_cast<const T*>(a.q) + ((long long)b * a.L + (long long)c * C) * a.q_rs + (long long)hd * D;

    // State columns are held as pairs: every element-wise operation of the step is a packed
    // fp32x2 instruction (Blackwell FFMA2 / FMUL2), which halves the issue slots of a kernel that
    // is bound by instruction issue.
    constexpr int kP = kCols / 2;
    float2 zr[kP], zi[kP], rr[kP], ri[kP];
#pragma unroll
    for (int i = 0; i < kP; i++) { zr[i] = zi[i] = rr[i] = ri[i] = make_float2(0.f, 0.f); }
    const long long sidx = ((((long long)b * a.NC + c) * H + hd) * NH + j);
    if (kOutput) {
        const float* s = a.ws_state + sidx * 2 * D;
#pragma unroll
        for (int i = 0; i < kP; i++) {
            const int d = g * kCols + 2 * i;
            if (d < D) { rr[i].x = s[d]; ri[i].x = s[D + d]; }
            if (d + 1 < D) { rr[i].y = s[d + 1]; ri[i].y = s[D + d + 1]; }
        }
    }
    float cr = 1.f, ci = 0.f;

    RowSlice<T, kCols> kraw, qraw;
    constexpr int kPieces = kCols * (int)sizeof(T) / 16, kRows = kOutput ? 2 : 1;   // 16-byte pieces of a lane's slice; rows a token
    uint4* ring = reinterpret_cast<uint4*>(smem + 6 * kUnits * C) + threadIdx.x;
    auto piece = [&](int t, int row, int p) { return ring + (((t % (kRing > 0 ? kRing : 1)) * kRows + row) * kPieces + p) * kSimtThreads; };
    auto fetch = [&](int t) {
        const int row = min(t, Lc - 1);
#pragma unroll
        for (int p = 0; p < kPieces; p++) {
            sm100::cp_async16(piece(t, 0, p), kbase + (long long)row * a.k_rs + g * kCols + p * (16 / (int)sizeof(T)), t < Lc);
            if (kOutput) sm100::cp_async16(piece(t, 1, p), qbase + (long long)row * a.q_rs + g * kCols + p * (16 / (int)sizeof(T)), t < Lc);
        }
        sm100::cp_async_commit();
    };
    auto take = [&](int t) {   // row t, requested kRing - 1 requests ago
        sm100::cp_async_wait_group<kRing - 2 < 0 ? 0 : kRing - 2>();
#pragma unroll
        for (int p = 0; p < kPieces; p++) {
            *(reinterpret_cast<uint4*>(&kraw) + p) = *piece(t, 0, p);
            if (kOutput) *(reinterpret_cast<uint4*>(&qraw) + p) = *piece(t, 1, p);
        }
    };
    if constexpr (kRing > 0) {
#pragma unroll 1
        for (int t = 0; t < kRing - 1; t++) fetch(t);
        take(0);
    } else {
        kraw.load(kbase, g, D, vec);
        if (kOutput) qraw.load(qbase, g, D, vec);
    }
    const int so = ul * C;
    // The four units of a warp may sit in different chunks (a full one and the ragged last one):
    // every lane walks the warp's longest chunk so that the shuffles stay warp-wide; beyond its
    // own Lc a unit sees the zero padding of the reference (a = k = v = beta = 0, ssd.py:60-67).
    const int Lw = __reduce_max_sync(0xffffffffu, Lc);
    for (int t = 0; t < Lw; t++) {
        float2 kk[kP], qq[kP];
        kraw.get(reinterpret_cast<float*>(kk));
        if (kOutput) qraw.get(reinterpret_cast<float*>(qq));
        if constexpr (kRing > 0) {
            fetch(t + kRing - 1);
            take(t + 1);
        } else if (t + 1 < Lc) {
            kraw.load(kbase + (long long)(t + 1) * a.k_rs, g, D, vec);
            if (kOutput) qraw.load(qbase + (long long)(t + 1) * a.q_rs, g, D, vec);
        } else {
            kraw.zero();
            if (kOutput) qraw.zero();
        }
        const float a_re = sm.a_re[so + t], a_im = sm.a_im[so + t], be = sm.beta[so + t];
        const float vr = sm.v_re[so + t], vi = sm.v_im[so + t];
        // The rows stay raw; the normalisation (normalize_kq.cu:46-79) enters through the scalars
        // ik = |k|^-1, iq = |q|^-1:  k^ = ik k, q^ = iq q.  Every dot product of the step is taken
        // against the state BEFORE the update, so all reductions are issued together; the
        // post-step read-out follows from  z' = a z + Kz k  =>  z'.q = a (z.q) + Kz (k.q).
        // (The reference rounds k^ and q^ to bf16 before use; here they keep fp32 precision.)
        const float2 zero2 = make_float2(0.f, 0.f);
        float2 skk2 = zero2, zkr2 = zero2, zki2 = zero2;
#pragma unroll
        for (int i = 0; i < kP; i++) {
            skk2 = __ffma2_rn(kk[i], kk[i], skk2);
            zkr2 = __ffma2_rn(zr[i], kk[i], zkr2);
            zki2 = __ffma2_rn(zi[i], kk[i], zki2);
        }
        float skk = skk2.x + skk2.y, zkr = zkr2.x + zkr2.y, zki = zki2.x + zki2.y;
        float sqq = 0.f, kq = 0.f, zqr = 0.f, zqi = 0.f, rkr = 0.f, rki = 0.f, rqr = 0.f, rqi = 0.f;
        if (kOutput) {
            float2 sqq2 = zero2, kq2 = zero2, zqr2 = zero2, zqi2 = zero2, rkr2 = zero2, rki2 = zero2,
                   rqr2 = zero2, rqi2 = zero2;
#pragma unroll
            for (int i = 0; i < kP; i++) {
                sqq2 = __ffma2_rn(qq[i], qq[i], sqq2);
                kq2 = __ffma2_rn(kk[i], qq[i], kq2);
                zqr2 = __ffma2_rn(zr[i], qq[i], zqr2);
                zqi2 = __ffma2_rn(zi[i], qq[i], zqi2);
                rkr2 = __ffma2_rn(rr[i], kk[i], rkr2);
                rki2 = __ffma2_rn(ri[i], kk[i], rki2);
                rqr2 = __ffma2_rn(rr[i], qq[i], rqr2);
                rqi2 = __ffma2_rn(ri[i], qq[i], rqi2);
            }
            sqq = sqq2.x + sqq2.y; kq = kq2.x + kq2.y; zqr = zqr2.x + zqr2.y; zqi = zqi2.x + zqi2.y;
            rkr = rkr2.x + rkr2.y; rki = rki2.x + rki2.y; rqr = rqr2.x + rqr2.y; rqi = rqi2.x + rqi2.y;
        }
        skk = group_sum<kLanes>(skk); zkr = group_sum<kLanes>(zkr); zki = group_sum<kLanes>(zki);
        if (kOutput) {
            sqq = group_sum<kLanes>(sqq); kq = group_sum<kLanes>(kq); zqr = group_sum<kLanes>(zqr); zqi = group_sum<kLanes>(zqi);
            rkr = group_sum<kLanes>(rkr); rki = group_sum<kLanes>(rki); rqr = group_sum<kLanes>(rqr); rqi = group_sum<kLanes>(rqi);
        }
        const float ik = rsqrtf(skk + kEps);
        const float bik = be * ik, bik2 = bik * ik;
        // z' = a (z - beta (z.k^) k^) + beta v k^ = a z + Kz k
        const float czr = __fmul_rn(bik2, zkr), czi = __fmul_rn(bik2, zki);
        const float Kzr = __fmaf_rn(bik, vr, -msub(a_re, czr, a_im, czi));
        const float Kzi = __fmaf_rn(bik, vi, -madd(a_re, czi, a_im, czr));
        const float2 are2 = make_float2(a_re, a_re), aim2 = make_float2(a_im, a_im), nim2 = make_float2(-a_im, -a_im);
        {
            const float2 kzr2 = make_float2(Kzr, Kzr), kzi2 = make_float2(Kzi, Kzi);
#pragma unroll
            for (int i = 0; i < kP; i++) {
                const float2 x = zr[i], y = zi[i];
                zr[i] = __ffma2_rn(kzr2, kk[i], __ffma2_rn(are2, x, __fmul2_rn(nim2, y)));
                zi[i] = __ffma2_rn(kzi2, kk[i], __ffma2_rn(are2, y, __fmul2_rn(aim2, x)));
            }
        }
        const float ncr = msub(a_re, cr, a_im, ci), nci = madd(a_re, ci, a_im, cr);
        cr = ncr;
        ci = nci;
        if (kOutput) {
            const float iq = rsqrtf(sqq + kEps);
            // correction is read BEFORE its step (exact_correction.cu:90-94), the local state after
            float yr = __fmul_rn(iq, read_re(rqr, a_re, a_im, zqr, zqi, Kzr, kq));
            float yi = __fmul_rn(iq, read_im(rqi, a_re, a_im, zqr, zqi, Kzi, kq));
            // r' = a (r - beta (r.k^) k^) = a r + Kr k
            const float crr = __fmul_rn(bik2, rkr), cri = __fmul_rn(bik2, rki);
            const float Krr = -msub(a_re, crr, a_im, cri), Kri = -madd(a_re, cri, a_im, crr);
            const float2 krr2 = make_float2(Krr, Krr), kri2 = make_float2(Kri, Kri);
#pragma unroll
            for (int i = 0; i < kP; i++) {
                const float2 x = rr[i], y = ri[i];
                rr[i] = __ffma2_rn(krr2, kk[i], __ffma2_rn(are2, x, __fmul2_rn(nim2, y)));
                ri[i] = __ffma2_rn(kri2, kk[i], __ffma2_rn(are2, y, __fmul2_rn(aim2, x)));
            }
            if (a.shortcut_scale != 0.f) {   // block.py:202-208: sum_d shortcut[s,d] q[d] = (q^.k^)^2 v[s]
                const float qk = __fmul_rn(__fmul_rn(iq, ik), kq), f = __fmul_rn(__fmul_rn(a.shortcut_scale, qk), qk);
                yr = __fmaf_rn(f, vr, yr);
                yi = __fmaf_rn(f, vi, yi);
            }
            if (g == 0) {   // v slots of this step are consumed: reuse them to stage y
                const float sc = sm.sel_c[so + t];
                sm.v_re[so + t] = IO<T>::rnd(IO<T>::rnd(yr) * sc);
                sm.v_im[so + t] = IO<T>::rnd(IO<T>::rnd(yi) * sc);
            }
            if (a.tail_state != nullptr && c * C + t == a.L - 1 && active) {
                float* ts = a.tail_state + (((long long)b * H + hd) * a.N + 2 * j) * D;
#pragma unroll
                for (int i = 0; i < kP; i++) {
                    const int d = g * kCols + 2 * i;
                    if (d < D) { ts[d] = zr[i].x + rr[i].x; ts[D + d] = zi[i].x + ri[i].x; }
                    if (d + 1 < D) { ts[d + 1] = zr[i].y + rr[i].y; ts[D + d + 1] = zi[i].y + ri[i].y; }
                }
            }
        }
    }
    if (!kOutput) {
        if (Lc < C) {   // zero padding wipes the local state and the decay product
#pragma unroll
            for (int i = 0; i < kP; i++) { zr[i] = zi[i] = make_float2(0.f, 0.f); }
            cr = 0.f;
            ci = 0.f;
        }
        if (active) {
            // the carry pass consumes these as the reference's bf16 cum_A[:, -1] / local_h[:, -1]
            float* s = a.ws_state + sidx * 2 * D;
#pragma unroll
            for (int i = 0; i < kP; i++) {
                const int d = g * kCols + 2 * i;
                if (d < D) { s[d] = IO<T>::rnd(zr[i].x); s[D + d] = IO<T>::rnd(zi[i].x); }
                if (d + 1 < D) { s[d + 1] = IO<T>::rnd(zr[i].y); s[D + d + 1] = IO<T>::rnd(zi[i].y); }
            }
            if (g == 0) {
                a.ws_gamma[sidx * 2] = IO<T>::rnd(cr);
                a.ws_gamma[sidx * 2 + 1] = IO<T>::rnd(ci);
            }
        }
    } else {
        __syncwarp();
        if (active) {
            T* y = static_cast<T*>(a.y);
            for (int t = g; t < Lc; t += kLanes) {
                T* o = y + (((long long)b * a.L + c * C + t) * H + hd) * a.N + 2 * j;
                IO<T>::st(o, sm.v_re[so + t]);
                IO<T>::st(o + 1, sm.v_im[so + t]);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// "Exact" semantics: the plain sequential recurrence over the whole sequence (what the reference's
// chunked scan equals inside its first chunk, and what the one-token decode step continues),
//   z_t = a_t (z_{t-1} - beta_t (z_{t-1}.k^_t) k^_t) + beta_t v_t k^_t,  y_t = sel_C (z_t.q^_t + shortcut),
// with z_{-1} = h0.  One 8-lane unit walks one (batch, head, pair) sequence from start to end; the
// dynamics are staged in shared memory kMaxChunk tokens at a time.  Parallel over B*H*N/2 only.
template <typename T, int kCols>
__global__ void __launch_bounds__(kSimtThreads)
scan_recurrent_kernel(const ScanArgs a) {
    constexpr int kLanes = kLanesPerUnit, kP = kCols / 2;
    extern __shared__ float smem[];
    const int CS = a.C;                                   // staging length (tokens per stage)
    ChunkScalars sm(smem, CS);
    const int ul = threadIdx.x / kLanes, g = threadIdx.x % kLanes;
    long long u = (long long)blockIdx.x * kUnitsPerBlock + ul;
    const bool active = u < a.units;
    if (!active) u = a.units - 1;
    const int NH = a.N >> 1, D = a.D, H = a.H;
    const int j = (int)(u % NH);
    const int hd = (int)((u / NH) % H);
    const int b = (int)(u / ((long long)NH * H));
    const bool vec = (D == kCols * kLanes);
    float2 zr[kP], zi[kP];
    {
        const float* h = a.h0 ? a.h0 + (((long long)b * H + hd) * a.N + 2 * j) * D : nullptr;
#pragma unroll
        for (int i = 0; i < kP; i++) {
            const int d = g * kCols + 2 * i;
            zr[i] = make_float2(h && d < D ? h[d] : 0.f, h && d + 1 < D ? h[d + 1] : 0.f);
            zi[i] = make_float2(h && d < D ? h[D + d] : 0.f, h && d + 1 < D ? h[D + d + 1] : 0.f);
        }
    }
    const int so = ul * CS;
    for (int c = 0; c < a.NC; c++) {
        __syncwarp();
        stage_dynamics<T, kLanes>(a, sm, ul, g, b, c, hd, j);
        __syncwarp();
        const int Lc = min(CS, a.L - c * CS);
        const T* kbase = static_cast<const T*>(a.k) + ((long long)b * a.L + (long long)c * CS) * a.k_rs + (long long)hd * D;
        const T* qbase = static_cast<const T*>(a.q) + ((long long)b * a.L + (long long)c * CS) * a.q_rs + (long long)hd * D;
        RowSlice<T, kCols> kraw, qraw;
        kraw.load(kbase, g, D, vec);
        qraw.load(qbase, g, D, vec);
        for (int t = 0; t < Lc; t++) {
            float2 kk[kP], qq[kP];
            kraw.get(reinterpret_cast<float*>(kk));
            qraw.get(reinterpret_cast<float*>(qq));
            if (t + 1 < Lc) {
                kraw.load(kbase + (long long)(t + 1) * a.k_rs, g, D, vec);
                qraw.load(qbase + (long long)(t + 1) * a.q_rs, g, D, vec);
            }
            const float a_re = sm.a_re[so + t], a_im = sm.a_im[so + t], be = sm.beta[so + t];
            const float vr = sm.v_re[so + t], vi = sm.v_im[so + t];
            const float2 zero2 = make_float2(0.f, 0.f);
            float2 skk2 = zero2, sqq2 = zero2, kq2 = zero2, zkr2 = zero2, zki2 = zero2, zqr2 = zero2, zqi2 = zero2;
#pragma unroll
            for (int i = 0; i < kP; i++) {
                skk2 = __ffma2_rn(kk[i], kk[i], skk2);
                sqq2 = __ffma2_rn(qq[i], qq[i], sqq2);
                kq2 = __ffma2_rn(kk[i], qq[i], kq2);
                zkr2 = __ffma2_rn(zr[i], kk[i], zkr2);
                zki2 = __ffma2_rn(zi[i], kk[i], zki2);
                zqr2 = __ffma2_rn(zr[i], qq[i], zqr2);
                zqi2 = __ffma2_rn(zi[i], qq[i], zqi2);
            }
            const float skk = group_sum(skk2.x + skk2.y), sqq = group_sum(sqq2.x + sqq2.y);
            const float kq = group_sum(kq2.x + kq2.y);
            const float zkr = group_sum(zkr2.x + zkr2.y), zki = group_sum(zki2.x + zki2.y);
            const float zqr = group_sum(zqr2.x + zqr2.y), zqi = group_sum(zqi2.x + zqi2.y);
            const float ik = rsqrtf(skk + kEps), iq = rsqrtf(sqq + kEps);
            const float bik = be * ik, bik2 = bik * ik;
            const float czr = bik2 * zkr, czi = bik2 * zki;
            const float Kzr = bik * vr - (a_re * czr - a_im * czi);
            const float Kzi = bik * vi - (a_re * czi + a_im * czr);
            const float2 are2 = make_float2(a_re, a_re), aim2 = make_float2(a_im, a_im), nim2 = make_float2(-a_im, -a_im);
            const float2 kzr2 = make_float2(Kzr, Kzr), kzi2 = make_float2(Kzi, Kzi);
#pragma unroll
            for (int i = 0; i < kP; i++) {
                const float2 x = zr[i], y = zi[i];
                zr[i] = __ffma2_rn(kzr2, kk[i], __ffma2_rn(are2, x, __fmul2_rn(nim2, y)));
                zi[i] = __ffma2_rn(kzi2, kk[i], __ffma2_rn(are2, y, __fmul2_rn(aim2, x)));
            }
            float yr = iq * (a_re * zqr - a_im * zqi + Kzr * kq);
            float yi = iq * (a_re * zqi + a_im * zqr + Kzi * kq);
            if (a.shortcut_scale != 0.f) {
                const float qk = iq * ik * kq;
                yr += a.shortcut_scale * qk * qk * vr;
                yi += a.shortcut_scale * qk * qk * vi;
            }
            if (g == 0) {
                const float sc = sm.sel_c[so + t];
                sm.v_re[so + t] = IO<T>::rnd(IO<T>::rnd(yr) * sc);
                sm.v_im[so + t] = IO<T>::rnd(IO<T>::rnd(yi) * sc);
            }
        }
        __syncwarp();
        if (active) {
            T* y = static_cast<T*>(a.y);
            for (int t = g; t < Lc; t += kLanes) {
                T* o = y + (((long long)b * a.L + c * CS + t) * H + hd) * a.N + 2 * j;
                IO<T>::st(o, sm.v_re[so + t]);
                IO<T>::st(o + 1, sm.v_im[so + t]);
            }
        }
    }
    if (active && a.final_state) {
        float* fs = a.final_state + (((long long)b * H + hd) * a.N + 2 * j) * D;
#pragma unroll
        for (int i = 0; i < kP; i++) {
            const int d = g * kCols + 2 * i;
            if (d < D) { fs[d] = zr[i].x; fs[D + d] = zi[i].x; }
            if (d + 1 < D) { fs[d + 1] = zr[i].y; fs[D + d + 1] = zi[i].y; }
        }
    }
}

template <typename T, int kCols>
static int launch_recurrent(ScanArgs a, cudaStream_t st) {
    a.C = a.L < 128 ? a.L : 128;                          // staging length only: no chunk semantics here
    a.NC = (a.L + a.C - 1) / a.C;
    a.segs = 1;
    a.units = (long long)a.B * a.H * (a.N / 2);
    const size_t smem = (size_t)6 * kUnitsPerBlock * a.C * sizeof(float);
    const unsigned blocks = (unsigned)((a.units + kUnitsPerBlock - 1) / kUnitsPerBlock);
    scan_recurrent_kernel<T, kCols><<<blocks, kSimtThreads, smem, st>>>(a);
    return check_launch();
}

// Carry pass: s_0 = h0 (or 0); for every chunk: publish s_c, then s <- gamma_c * s + z_{C-1}.
// One thread per (b, h, pair, d).  Chunks are taken eight at a time so that the loads of a
// batch are in flight together (the recurrence itself is two FMAs per chunk).
template <typename T>
__global__ void __launch_bounds__(128)
scan_carry_kernel(const ScanArgs a) {
    grid_dependency_wait();
    const int NH = a.N >> 1, D = a.D, H = a.H, NC = a.NC;
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)a.B * H * NH * D) return;
    const int d = (int)(idx % D);
    const int j = (int)((idx / D) % NH);
    const int hd = (int)((idx / ((long long)D * NH)) % H);
    const int b = (int)(idx / ((long long)D * NH * H));
    const long long so = (((long long)b * H + hd) * a.N + 2 * j) * D + d;
    float sr = 0.f, si = 0.f, dr = 1.f, di = 0.f;
    if (a.h0) { sr = a.h0[so]; si = a.h0[so + D]; }
    const long long cstride = (long long)H * NH;            // units per chunk index
    const long long u0 = ((long long)b * NC * H + hd) * NH + j;
    constexpr int kBatch = 8;
    for (int c0 = 0; c0 < NC; c0 += kBatch) {
        float gr[kBatch], gi[kBatch], lr[kBatch], li[kBatch];
#pragma unroll
        for (int i = 0; i < kBatch; i++) {
            if (c0 + i < NC) {
                const long long u = u0 + (long long)(c0 + i) * cstride;
                gr[i] = a.ws_gamma[u * 2];
                gi[i] = a.ws_gamma[u * 2 + 1];
                lr[i] = a.ws_state[u * 2 * D + d];
                li[i] = a.ws_state[u * 2 * D + D + d];
            }
        }
#pragma unroll
        for (int i = 0; i < kBatch; i++) {
            if (c0 + i < NC) {
                const long long u = u0 + (long long)(c0 + i) * cstride;
                if (a.publish) {
                    a.ws_state[u * 2 * D + d] = IO<T>::rnd(sr);       // chunk_states store
                    a.ws_state[u * 2 * D + D + d] = IO<T>::rnd(si);
                }
                const float2 gm = make_float2(gr[i], gi[i]);
                const float nr = next_re(gm, sr, si, lr[i]);
                si = next_im(gm, sr, si, li[i]);
                sr = nr;
                const float pr = msub(gm.x, dr, gm.y, di), pi = madd(gm.x, di, gm.y, dr);
                dr = pr;
                di = pi;
            }
        }
    }
    grid_launch_dependents();
    if (a.final_state) { a.final_state[so] = sr; a.final_state[so + D] = si; }
    if (a.total_decay && d == 0) {
        float* td = a.total_decay + ((long long)b * H + hd) * a.N + 2 * j;
        td[0] = dr;
        td[1] = di;
    }
}

// Whether the walks' rows travel ahead through shared memory: while there is a block per SM at most; more blocks hide each other's
// waits and want the shared memory.  us of a call on B200, next row in registers / ring of eight: float32, D 64, 64 units 49.3 / 45.8,
// 768 52.4 / 49.7, 1536 57.0 / 50.0, 6144 98 / 129; D 128, 1024 units 154 / 135, 4096 236 / 291; bf16, D 64, 240 units 52.5 / 46.9,
// 3072 69.3 / 65.8, 6144 92.3 / 93.6.
static bool walk_with_ring(const ScanArgs& a, int cols, int es, unsigned blocks, int sms) {
    return blocks <= (unsigned)sms && a.D == cols * kLanesPerUnit && a.C <= a.D && ((a.k_rs | a.q_rs) * es) % 16 == 0;
}

template <typename T, int kCols, bool kOutput, int kRing> struct WalkTag {};

template <typename T, int kCols, bool kOutput, int kRing>
static int launch_walk(const ScanArgs& a, unsigned blocks, cudaStream_t st) {
    constexpr int kRows = kOutput ? 2 : 1;
    constexpr size_t ring = (size_t)kRing * kRows * kCols * sizeof(T) * kSimtThreads;
    const size_t scalars = (size_t)6 * kUnitsPerBlock * sizeof(float);
    const size_t smem = scalars * a.C + ring;
    if (smem > 48 * 1024) {   // opt in to more than 48 KB of dynamic shared memory
        const size_t most = kRing ? scalars * kCols * kLanesPerUnit + ring : scalars * kMaxChunk;   // (with a ring: C <= D)
        if (int rc = allow_smem<WalkTag<T, kCols, kOutput, kRing>>((const void*)scan_walk_kernel<T, kCols, kLanesPerUnit, kOutput, kRing>, most)) return rc;
    }
    return launch_overlapped(scan_walk_kernel<T, kCols, kLanesPerUnit, kOutput, kRing>, dim3(blocks), dim3(kSimtThreads), smem, st, a);
}

// Whether a state that the call leaves lies where h0 does (a caller who carries one buffer on).  The carry pass reads and writes an element in one
// thread; where the output pass adds the carry up itself, every chunk's block reads h0 and the last chunk's writes.
static bool writes_into_h0(const ScanArgs& a) {
    const uintptr_t bytes = (uintptr_t)a.B * a.H * a.N * a.D * sizeof(float), h0 = (uintptr_t)a.h0;
    auto meets = [&](const float* out) { return out != nullptr && (uintptr_t)out < h0 + bytes && h0 < (uintptr_t)out + bytes; };
    return h0 != 0 && (meets(a.final_state) || meets(a.tail_state));
}

template <typename T, int kCols>
static int launch_simt(const ScanArgs& a, cudaStream_t st) {
    constexpr int kUnits = kUnitsPerBlock, kRing = 8;
    const unsigned blocks = (unsigned)((a.units + kUnits - 1) / kUnits);
    const bool output = a.y != nullptr && a.run_output;   // else: summary only, or y comes from another kernel
    int sms = 0;
    if (int rc = sm_count(sms)) return rc;
    constexpr int dtype = IO<T>::kBf16 ? CDSSM_BF16 : CDSSM_F32;
    const bool short_walk = scan_short_takes(a, dtype, sms);
    const bool ring = walk_with_ring(a, kCols, (int)sizeof(T), blocks, sms);
    if (a.rec_av != nullptr && (a.run_local || output)) {
        // pairs over the grid as far as one wave goes (what the pairs of a token share is computed again for each)
        const long long wave = ((long long)a.B * a.L + 31) / 32 * ((a.H + 7) / 8);
        const int pairs = wave >= 1024 ? 1 : (int)min((long long)(a.N / 2), 1024 / wave);
        const bool early = short_walk && wave * pairs <= sms;   // (the walk has rows to fetch and norms to form meanwhile)
        simt_records_kernel<T><<<dim3((unsigned)(((long long)a.B * a.L + 31) / 32), (a.H + 7) / 8, pairs), 256, 0, st>>>(a, early);
        if (int rc = check_launch()) return rc;
    }
    if (a.run_local) {
        if (int rc = short_walk ? scan_short_pass(false, a, dtype, 0, st)
                     : ring     ? launch_walk<T, kCols, false, kRing>(a, blocks, st)
                                : launch_walk<T, kCols, false, 0>(a, blocks, st))
            return rc;
    }
    // (the short walk adds a few chunks up itself, instead of a launch and two more trips to memory)
    const bool from_chunks = short_walk && output && a.run_local && a.publish && !a.total_decay && a.NC <= 12 && !writes_into_h0(a);
    if (!from_chunks) {
        const long long th = (long long)a.B * a.H * (a.N / 2) * a.D;
        if (int rc = launch_overlapped(scan_carry_kernel<T>, dim3((unsigned)((th + 127) / 128)), dim3(128), 0, st, a)) return rc;
    }
    if (!output) return CDSSM_OK;
    if (short_walk) return scan_short_pass(true, a, dtype, from_chunks, st);
    return ring ? launch_walk<T, kCols, true, kRing>(a, blocks, st) : launch_walk<T, kCols, true, 0>(a, blocks, st);
}

// Column split: D <= 64 -> 8 lanes x 8 columns, D <= 128 -> 8 lanes x 16 columns (16 lanes x 8 columns was slower: 10.8 ms
// against 8.9 ms at B 16, H 32, L 65536).
int scan_fused_simt(const ScanArgs& a, int dtype, cudaStream_t st) {
    const int cols = (a.D + kLanesPerUnit - 1) / kLanesPerUnit;
    if (dtype == CDSSM_BF16) return cols <= 8 ? launch_simt<__nv_bfloat16, 8>(a, st) : launch_simt<__nv_bfloat16, 16>(a, st);
    return cols <= 8 ? launch_simt<float, 8>(a, st) : launch_simt<float, 16>(a, st);
}

}  // namespace cdssm

namespace cdssm {
// ---------------------------------------------------------------------------------------------
// One-token decode step.  Eight lanes per (batch, head, pair): dynamics for position `pos`,
// normalise q/k, one delta-rule step on the fp32 state in place, read-out.  One pass over the
// state (read + write), everything else is a few hundred bytes per head.
struct DecodeArgs {
    float* state;
    float *corr, *carry, *gamma;   // reference-compatible step only: correction, carry (B,H,N,D), chunk decay (B,H,N)
    int C;                         // chunk length of the reference-compatible step
    const void *q, *k, *v, *gate_raw;
    long long k_stride, v_stride;  // elements between the batch rows of k and v (column slices of a wider projection)
    long long q_stride, g_stride;  // the same for q and gate_raw (plain step only)
    const void *v_first, *mix;     // plain step only, or NULL: v <- lerp(v_first, v, mix[head]) (value residual)
    const float *log_dt_scale, *rope_freqs;
    void* y;
    DynConsts dc;
    float shortcut_scale;
    int B, H, D, N, pos;
    const int* pos_dev;   // if not NULL the position is read from device memory (graph replay)
    long long units;   // B*H*NP
};

template <typename T, int kCols>
__global__ void __launch_bounds__(kSimtThreads)
decode_step_kernel(const DecodeArgs a) {
    grid_dependency_wait();
    grid_launch_dependents();
    DecodeUnitArgs u;
    u.state = a.state;
    u.q = a.q; u.k = a.k; u.v = a.v; u.gate = a.gate_raw;
    u.q_stride = a.q_stride; u.k_stride = a.k_stride; u.v_stride = a.v_stride; u.gate_stride = a.g_stride;
    u.v_first = a.v_first; u.mix = a.mix; u.v_first_stride = (long long)a.H * a.N;
    u.log_dt_scale = a.log_dt_scale; u.rope_freqs = a.rope_freqs;
    u.y = a.y;
    u.dc = a.dc;
    u.shortcut_scale = a.shortcut_scale;
    u.H = a.H; u.D = a.D; u.N = a.N;
    u.pos = a.pos_dev ? *a.pos_dev : a.pos;
    u.units = a.units;
    decode_unit<T, kCols>(u, (long long)blockIdx.x * kUnitsPerBlock + threadIdx.x / kLanesPerUnit, [] {});
}

// The decode step that reproduces the reference's CHUNKED scan token by token (its outputs beyond the first
// chunk are not those of the plain recurrence): per (batch, head) the local state z (zero at every chunk start),
// the correction r (starts from the rounded carry, erase + rotate only, read before its step), the carry s
// and the cumulative decay of the current chunk.  Position pos counts from the sequence start; chunks are
// C tokens.  Same thread mapping as decode_step_kernel.
template <typename T, int kCols>
__global__ void __launch_bounds__(kSimtThreads)
decode_step_ref_kernel(const DecodeArgs a) {
    const int g = threadIdx.x % kLanesPerUnit;
    long long u = (long long)blockIdx.x * kUnitsPerBlock + threadIdx.x / kLanesPerUnit;
    const bool active = u < a.units;
    if (!active) u = a.units - 1;
    const int NH = a.N >> 1, D = a.D, H = a.H;
    const int j = (int)(u % NH);
    const int hd = (int)((u / NH) % H);
    const long long b = u / ((long long)NH * H);
    const bool vec = (D == kCols * kLanesPerUnit);
    const long long bh = b * H + hd;

    RowSlice<T, kCols> kraw, qraw;
    kraw.load(static_cast<const T*>(a.k) + bh * D, g, D, vec);
    qraw.load(static_cast<const T*>(a.q) + bh * D, g, D, vec);
    const long long so = (bh * a.N + 2 * j) * D;
    float* st = a.state + so;
    float* ct = a.corr + so;
    float zr[kCols], zi[kCols], rr[kCols], ri[kCols];
    if (vec) {
#pragma unroll
        for (int i = 0; i < kCols / 4; i++) {
            const float4 x = *reinterpret_cast<const float4*>(st + g * kCols + 4 * i);
            const float4 w = *reinterpret_cast<const float4*>(st + D + g * kCols + 4 * i);
            zr[4 * i] = x.x; zr[4 * i + 1] = x.y; zr[4 * i + 2] = x.z; zr[4 * i + 3] = x.w;
            zi[4 * i] = w.x; zi[4 * i + 1] = w.y; zi[4 * i + 2] = w.z; zi[4 * i + 3] = w.w;
            const float4 p = *reinterpret_cast<const float4*>(ct + g * kCols + 4 * i);
            const float4 r = *reinterpret_cast<const float4*>(ct + D + g * kCols + 4 * i);
            rr[4 * i] = p.x; rr[4 * i + 1] = p.y; rr[4 * i + 2] = p.z; rr[4 * i + 3] = p.w;
            ri[4 * i] = r.x; ri[4 * i + 1] = r.y; ri[4 * i + 2] = r.z; ri[4 * i + 3] = r.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < kCols; i++) {
            const int d = g * kCols + i;
            zr[i] = d < D ? st[d] : 0.f;
            zi[i] = d < D ? st[D + d] : 0.f;
            rr[i] = d < D ? ct[d] : 0.f;
            ri[i] = d < D ? ct[D + d] : 0.f;
        }
    }
    // dynamics (every lane of the unit computes the same scalars; dynamics_fused.cu:64-139)
    const T* gr = static_cast<const T*>(a.gate_raw) + b * (long long)((a.N + 5) * H);
    const T* s5 = gr + a.N * H;
    const float freq = a.rope_freqs[hd], pos = (float)(a.pos_dev ? *a.pos_dev : a.pos);
    DynShared ds = dyn_shared<IO<T>::kBf16>(IO<T>::ld(gr + hd), IO<T>::ld(gr + NH * H + hd), IO<T>::ld(s5 + hd),
                              IO<T>::ld(s5 + H + hd), IO<T>::ld(s5 + 2 * H + hd),
                              IO<T>::ld(s5 + 3 * H + hd), IO<T>::ld(s5 + 4 * H + hd),
                              a.log_dt_scale[hd], freq, pos, a.dc);
    float a_re, a_im, vp;
    dyn_pair<IO<T>::kBf16>(IO<T>::ld(gr + j * H + hd), IO<T>::ld(gr + (NH + j) * H + hd), freq, pos, ds, a_re, a_im, vp);
    a_re = IO<T>::rnd(a_re);
    a_im = IO<T>::rnd(a_im);
    vp = IO<T>::rnd(vp);
    const float be = IO<T>::rnd(ds.beta), sc = IO<T>::rnd(ds.sel_c);
    const T* vrow = static_cast<const T*>(a.v) + bh * a.N + 2 * j;
    const float vr = IO<T>::rnd(IO<T>::ld(vrow) * vp), vi = IO<T>::rnd(IO<T>::ld(vrow + 1) * vp);

    float kk[kCols], qq[kCols];
    kraw.get(kk);
    qraw.get(qq);
    normalise<T, kCols>(kk);
    normalise<T, kCols>(qq);
    float ur = 0.f, ui = 0.f, wr = 0.f, wi = 0.f;
#pragma unroll
    for (int i = 0; i < kCols; i++) {
        ur += zr[i] * kk[i]; ui += zi[i] * kk[i];
        wr += rr[i] * kk[i]; wi += ri[i] * kk[i];
    }
    ur = be * group_sum(ur);
    ui = be * group_sum(ui);
    wr = be * group_sum(wr);
    wi = be * group_sum(wi);
    const float ivr = be * vr, ivi = be * vi;
    float yr = 0.f, yi = 0.f;
#pragma unroll
    for (int i = 0; i < kCols; i++) {
        const float er = zr[i] - ur * kk[i], ei = zi[i] - ui * kk[i];
        zr[i] = a_re * er - a_im * ei + ivr * kk[i];
        zi[i] = a_re * ei + a_im * er + ivi * kk[i];
        // the correction is read BEFORE its step (exact_correction.cu:90-94), then erased and rotated
        yr += (zr[i] + rr[i]) * qq[i];
        yi += (zi[i] + ri[i]) * qq[i];
        const float cr = rr[i] - wr * kk[i], ci = ri[i] - wi * kk[i];
        rr[i] = a_re * cr - a_im * ci;
        ri[i] = a_re * ci + a_im * cr;
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
    // cumulative decay of the chunk; at the chunk's last token the carry takes the (rounded) chunk results, the
    // local state restarts from zero and the correction from the (rounded) carry (inter_chunk_scan.cu:52-84)
    float* gm = a.gamma + bh * a.N + 2 * j;
    const float g0 = gm[0], g1 = gm[1];
    float gr_ = a_re * g0 - a_im * g1, gi_ = a_re * g1 + a_im * g0;
    const int posi = a.pos_dev ? *a.pos_dev : a.pos;
    if (posi % a.C == a.C - 1) {
        float* cy = a.carry + so;
        const float dr = IO<T>::rnd(gr_), di = IO<T>::rnd(gi_);
#pragma unroll
        for (int i = 0; i < kCols; i++) {
            const int d = g * kCols + i;
            if (d < D) {
                const float sr = cy[d], si = cy[D + d];
                const float nr = dr * sr - di * si + IO<T>::rnd(zr[i]), ni = dr * si + di * sr + IO<T>::rnd(zi[i]);
                cy[d] = nr;
                cy[D + d] = ni;
                rr[i] = IO<T>::rnd(nr);
                ri[i] = IO<T>::rnd(ni);
            }
            zr[i] = 0.f;
            zi[i] = 0.f;
        }
        gr_ = 1.f;
        gi_ = 0.f;
    }
    if (g == 0) { gm[0] = gr_; gm[1] = gi_; }
    if (vec) {
#pragma unroll
        for (int i = 0; i < kCols / 4; i++) {
            *reinterpret_cast<float4*>(st + g * kCols + 4 * i) =
                make_float4(zr[4 * i], zr[4 * i + 1], zr[4 * i + 2], zr[4 * i + 3]);
            *reinterpret_cast<float4*>(st + D + g * kCols + 4 * i) =
                make_float4(zi[4 * i], zi[4 * i + 1], zi[4 * i + 2], zi[4 * i + 3]);
            *reinterpret_cast<float4*>(ct + g * kCols + 4 * i) =
                make_float4(rr[4 * i], rr[4 * i + 1], rr[4 * i + 2], rr[4 * i + 3]);
            *reinterpret_cast<float4*>(ct + D + g * kCols + 4 * i) =
                make_float4(ri[4 * i], ri[4 * i + 1], ri[4 * i + 2], ri[4 * i + 3]);
        }
    } else {
#pragma unroll
        for (int i = 0; i < kCols; i++) {
            const int d = g * kCols + i;
            if (d < D) { st[d] = zr[i]; st[D + d] = zi[i]; ct[d] = rr[i]; ct[D + d] = ri[i]; }
        }
    }
    if (g == 0) {
        T* o = static_cast<T*>(a.y) + bh * a.N + 2 * j;
        IO<T>::st(o, IO<T>::rnd(yr) * sc);
        IO<T>::st(o + 1, IO<T>::rnd(yi) * sc);
    }
}

template <typename T, int kCols>
static int launch_decode(const DecodeArgs& a, cudaStream_t st) {
    const unsigned blocks = (unsigned)((a.units + kUnitsPerBlock - 1) / kUnitsPerBlock);
    if (a.corr) decode_step_ref_kernel<T, kCols><<<blocks, kSimtThreads, 0, st>>>(a);
    // launched to overlap its predecessor's drain: back-to-back steps of 3-6 us otherwise pay a launch gap each
    else return launch_overlapped(decode_step_kernel<T, kCols>, dim3(blocks), dim3(kSimtThreads), 0, st, a);
    return check_launch();
}

}  // namespace cdssm

using namespace cdssm;

namespace cdssm {
unsigned long long wait_limit_ns();   // c_abi.cu
// scan_records.cu
size_t scan_record_bytes(int B, int L, int H, int N, int C);
int scan_records(bool wa, const void* v, long long v_rs, const void* v_first, long long vf_rs, const void* mix,
                 const void* gate_raw, long long g_rs, const float* log_dt_scale, const float* rope_freqs, void* rec,
                 int* clear, size_t clear_words, int* clear2, size_t clear2_words, const DynConsts& dc, int B, int L, int H, int N,
                 int C, int pos0, int segs, int fp32_decay, cudaStream_t st);
// scan_wa.cu
bool scan_wa_supported(int D, int N, int C, int dtype);
int scan_wa_pass(bool output, const void* q, long long q_rs, const void* k, long long k_rs, const void* rec, float* ws_gamma, float* ws_state, void* y,
                 float* tail_state, int* status, float shortcut_scale, int B, int L, int H, int D, unsigned long long wait_ns, int withhold,
                 int from_chunks, const float* h0, float* final_state, int parts, cudaStream_t st);
// scan_tile.cu
bool scan_tile_supported(int D, int N, int C, int dtype);
size_t scan_tile_words(int B, int L, int H, int D, int N);
size_t scan_tile_extra_bytes(int B, int L, int H, int D, int N);
int scan_tile_pass(int mode, int from_chunks, const void* q, long long q_rs, const void* k, long long k_rs, void* rec, const float* h0, void* y,
                   float* final_state, float* tail_state, float* ws_gamma, float* ws_state, void* extra, int* status, int* ticket,
                   float shortcut_scale, int B, int L, int H, int D, int N, unsigned long long wait_ns, int withhold, cudaStream_t st);
}

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// What every path needs: status word, chunk decays, chunk states.
static size_t base_workspace_bytes(int B, int L, int H, int D, int N, int C) {
    const size_t NC = ((size_t)L + C - 1) / C;
    const size_t units = (size_t)B * NC * H * (N / 2);
    return 256 + align256(units * 2 * sizeof(float)) + align256(units * 2 * D * sizeof(float));
}
// Per-token records of the CUDA-core walks (which can do without); never less than those of the tensor-core kernels.
static size_t simt_record_bytes(int B, int L, int H, int N, int C) {
    return (size_t)B * (((size_t)L + C - 1) / C) * H * C * ((size_t)(N / 2) * sizeof(float4) + sizeof(float2));
}

// What a call cannot do without: the tensor-core scans' records beside the base.
static size_t least_workspace_bytes(int B, int L, int H, int D, int N, int C) {
    size_t bytes = base_workspace_bytes(B, L, H, D, N, C);
    if (scan_wa_supported(D, N, C, CDSSM_BF16) || scan_tile_supported(D, N, C, CDSSM_BF16)) bytes += align256(scan_record_bytes(B, L, H, N, C));
    return bytes;
}

// Tiles of the whole-chunk scan beside each other: a head (head_dim 128) or two (64) of a sequence.
static long long scan_tiles(int B, int H, int D) { return (long long)B * (D == 128 ? H : (H + 1) / 2); }

// Whether the whole-chunk scan (scan_tile.cu) hands the carry on inside one kernel, or runs as local pass, carry pass and output
// pass: the same arithmetic in the same order, so this choice may go by size.  One kernel forms G once and reads k once, but its
// blocks add up the chunks between theirs and the last finished one, as many as there are blocks on a sequence.  That is too much for
// head_dim 64 (592 blocks at a time for N <= 4, else 296) when few tiles beside each other fill the GPU with long sequences.  us of a
// call on B200, one kernel / passes, by tiles beside each other:
//   N 4:  1 tile, 64 chunks 21.3 / 22.8, 96 26.3 / 25.2, 512 112 / 75; 12 tiles 64 43.5 / 45.2, 96 59.3 / 58.5, 256 159 / 142; 48 tiles 64
//         123 / 125, 128 245 / 236; 96 tiles 128 449 / 446; 192 tiles 64 361 / 439
//   N 8:  1 tile, 96 chunks 29.8 / 29.5, 256 65 / 51; 2 tiles 96 34.8 / 35.9, 128 42 / 39, 512 121 / 124; 6 tiles 256 104 / 137
//   N 16: 1 tile, 25 chunks 25.4 / 26.9, 45 32.1 / 29.9, 256 109 / 62; 4 tiles 25 27.8 / 28.4, 64 47.5 / 42.0, 512 255 / 256; 6 tiles 64 57 / 62,
//         512 384 / 376; 12 tiles 256 337 / 338; 48 tiles 64 286 / 318
static bool hands_carry_on(int B, int H, int NC, int D, int N) {
    if (D == 128) return true;
    const long long tiles = scan_tiles(B, H, D);
    if (N <= 4) return NC <= 90 || tiles >= 96;
    return N <= 8 ? NC <= 110 || tiles >= 2 : NC <= 30 || tiles >= 5;
}

extern "C" size_t cdssm_b200_scan_fused_workspace_bytes(int B, int L, int H, int D, int N, int C) {
    if (B <= 0 || L <= 0 || H <= 0 || D <= 0 || N <= 0 || (N & 1) || C <= 0) return 0;
    size_t bytes = least_workspace_bytes(B, L, H, D, N, C);
    if (scan_tile_supported(D, N, C, CDSSM_BF16) && hands_carry_on(B, H, (L + C - 1) / C, D, N)) bytes += scan_tile_extra_bytes(B, L, H, D, N);
    return bytes;
}
// With room for the CUDA-core walks' records where those kernels run: a tenth faster (8 bytes more per token-head and 8 per pair
// than the tensor-core kernels want, 805 against 537 MB for N = 2 at 16 x 65 536 tokens of 32 heads).
extern "C" size_t cdssm_b200_scan_fused_workspace_bytes_for(int B, int L, int H, int D, int N, int C, int dtype, int flags) {
    const size_t least = cdssm_b200_scan_fused_workspace_bytes(B, L, H, D, N, C);
    if (least == 0 || (flags & CDSSM_SCAN_EXACT)) return least;
    const bool tensor = !(flags & CDSSM_SCAN_FORCE_SIMT) && (scan_wa_supported(D, N, C, dtype) || scan_tile_supported(D, N, C, dtype));
    return tensor ? least : std::max(least_workspace_bytes(B, L, H, D, N, C),
                                     base_workspace_bytes(B, L, H, D, N, C) + align256(simt_record_bytes(B, L, H, N, C)));
}

extern "C" int cdssm_b200_scan_fused_status(const void* workspace, int* status_host, void* stream) {
    if (!workspace || !status_host) return CDSSM_ERR_BAD_ARG;
    if (int rc = check_cuda(cudaMemcpyAsync(status_host, workspace, sizeof(int), cudaMemcpyDeviceToHost,
                                            (cudaStream_t)stream)))
        return rc;
    if (int rc = check_cuda(cudaStreamSynchronize((cudaStream_t)stream))) return rc;
    return *status_host == 0 ? CDSSM_OK : CDSSM_ERR_TIMEOUT;
}

// Whether scan_wa.cu's output pass adds the carry up itself from the local results of the chunks before it (else a carry pass runs
// in between): while it has a chunk of four heads per block, two blocks per SM.  us on B200, carry pass / without: D 64, 936 chunks
// 24.4 / 21.5, 3072 42 / 44; D 128, 528 32.3 / 30.5, 1536 61 / 63.
static bool carry_in_output(int B, int NC, int H) { return (long long)B * NC * ((H + 3) / 4) <= 296 && NC <= 40; }

// Whether the output pass of the whole-chunk scan, where it is not one kernel, adds the carry up itself: a read of NC x N rows by every
// block, in parallel, against a launch and two more trips to memory.  us of a call on B200, carry pass / without, by tiles beside each
// other, D 64: N 4, 2 tiles, 9 chunks 16.8 / 14.3, 25 18.4 / 17.0, 32 19.3 / 20.7; 12 tiles 9 18.5 / 17.9, 25 26.0 / 26.4; N 8, 2 tiles,
// 16 chunks 20.5 / 19.3, 25 22.2 / 22.1; 12 tiles 9 21.7 / 21.0, 16 27.0 / 28.7; N 16, 1 tile, 2 chunks 23.5 / 19.5, 9 24.8 / 23.9, 16
// 25.2 / 27.3; 12 tiles 9 27.5 / 29.1.  D 128, N 8, 4 tiles, 9 chunks 28.8 / 26.2, 25 32.2 / 35.4.
static bool few_chunks(int B, int H, int NC, int D, int N) {
    return NC * N <= 130 && NC <= (scan_tiles(B, H, D) <= 6 ? 20 : 10);
}

struct ScanRows {   // elements between (batch, token) rows, 0: dense; and the value residual
    long long q = 0, k = 0, v = 0, gate = 0, v_first = 0;
    const void *first = nullptr, *mix = nullptr;
};

static int scan_fused_impl(const void* q, const void* k, const void* v, const void* gate_raw,
                           const float* log_dt_scale, const float* rope_freqs, const float* h0, void* y,
                           float* final_state, float* tail_state, float* total_decay, bool summary_only,
                           void* workspace, size_t workspace_bytes, float gating_c, float omega_thresh,
                           float adt_delta, float adt_smoothness, float adt_eps, float shortcut_scale,
                           int B, int L, int H, int D, int N, int C, int pos0, int segs, int dtype,
                           int flags, void* stream, bool small_workspace = false, const ScanRows& rows = ScanRows()) {
    if (summary_only) { q = k; y = nullptr; tail_state = nullptr; }
    if (!q || !k || !v || !gate_raw || !log_dt_scale || !rope_freqs || (!y && !summary_only))
        return CDSSM_ERR_BAD_ARG;
    if (segs < 1 || (B > 0 && B % segs)) return CDSSM_ERR_BAD_ARG;
    if (B < 0 || L < 0 || H <= 0 || D <= 0 || N <= 0 || (N & 1) || C <= 0) return CDSSM_ERR_BAD_ARG;
    if (dtype != CDSSM_BF16 && dtype != CDSSM_F32) return CDSSM_ERR_BAD_ARG;
    const long long es = dtype == CDSSM_F32 ? 4 : 2, hd = (long long)H * D, hn = (long long)H * N, hg = (long long)(N + 5) * H;
    const long long q_rs = rows.q ? rows.q : hd, k_rs = rows.k ? rows.k : hd, v_rs = rows.v ? rows.v : hn,
                    g_rs = rows.gate ? rows.gate : hg, vf_rs = rows.v_first ? rows.v_first : hn;
    if (q_rs < hd || k_rs < hd || v_rs < hn || g_rs < hg || vf_rs < hn || (rows.first != nullptr) != (rows.mix != nullptr))
        return CDSSM_ERR_BAD_ARG;
    if (((uintptr_t)q | (uintptr_t)k) & 15) return CDSSM_ERR_BAD_ARG;   // 16-byte row loads
    if ((D == 64 || D == 128) && (((q_rs | k_rs) * es) & 15)) return CDSSM_ERR_BAD_ARG;
    if (N > kMaxStateDim || D > kMaxHeadDim || C > kMaxChunk) return CDSSM_ERR_UNSUPPORTED;
    if (B == 0 || L == 0) return CDSSM_OK;
    // small_workspace: as many of the records as fit (the walks can do without)
    const size_t base = base_workspace_bytes(B, L, H, D, N, C);
    const size_t need = small_workspace ? base : least_workspace_bytes(B, L, H, D, N, C);
    if (!workspace || workspace_bytes < need || ((uintptr_t)workspace & 255)) return CDSSM_ERR_WORKSPACE;
    // first 256 bytes of the workspace: status word of the tensor-core kernel's bounded waits, ticket counter
    int* status = static_cast<int*>(workspace);
    workspace = static_cast<char*>(workspace) + 256;
    if ((flags & CDSSM_SCAN_EXACT) && (summary_only || segs != 1)) return CDSSM_ERR_UNSUPPORTED;
    ScanArgs a;
    a.q = q; a.k = k; a.v = v; a.gate_raw = gate_raw;
    a.log_dt_scale = log_dt_scale; a.rope_freqs = rope_freqs; a.h0 = h0;
    a.y = y; a.final_state = final_state; a.tail_state = tail_state;
    a.total_decay = total_decay; a.segs = segs;
    a.run_local = (flags & CDSSM_SCAN_REUSE_LOCAL) ? 0 : 1;
    a.run_output = 1;
    a.publish = summary_only ? 0 : 1;
    a.fp32_decay = (flags & CDSSM_SCAN_FP32_DECAY) ? 1 : 0;
    a.dc = DynConsts{gating_c, omega_thresh, adt_delta, adt_smoothness, adt_eps};
    a.shortcut_scale = shortcut_scale;
    a.B = B; a.L = L; a.H = H; a.D = D; a.N = N; a.C = C; a.pos0 = pos0;
    a.q_rs = q_rs; a.k_rs = k_rs; a.v_rs = v_rs; a.g_rs = g_rs; a.vf_rs = vf_rs;
    a.v_first = rows.first; a.mix = rows.mix;
    a.NC = (L + C - 1) / C;
    a.units = (long long)B * a.NC * H * (N / 2);
    a.ws_gamma = static_cast<float*>(workspace);
    a.ws_state = reinterpret_cast<float*>(static_cast<char*>(workspace) +
                                          align256((size_t)a.units * 2 * sizeof(float)));
    cudaStream_t st = (cudaStream_t)stream;
    // Tensor-core kernels for bf16, chunk = head_dim in {64, 128}: N = 2 (scan_wa.cu), any other N <= 16 (scan_tile.cu).  The
    // kernel goes by the head's shape and by what is asked for, never by batch or length: a shard of a batch, and chunk-aligned
    // pieces of a sequence that hand the carry on, give the bits of the whole.  They read v
    // and write y as 4-byte pairs: buffers that are only 2-byte aligned, which the contract allows, stay on the CUDA-core
    // kernels.  (Bits 256 / 512 keep the CUDA-core local / output pass: used by the tests to check each tensor-core pass alone.)
    const bool tensor_ok = (((uintptr_t)v | (uintptr_t)y | (uintptr_t)rows.first | (uintptr_t)(2 * v_rs) |
                              (uintptr_t)(rows.first ? 2 * vf_rs : 0)) & 3) == 0 && ((q_rs | k_rs) & 7) == 0 && workspace_bytes - base >= scan_record_bytes(B, L, H, N, C) &&
                           !(flags & (CDSSM_SCAN_EXACT | CDSSM_SCAN_FORCE_SIMT));
    const bool wa_ok = tensor_ok && scan_wa_supported(D, N, C, dtype), tile_ok = tensor_ok && scan_tile_supported(D, N, C, dtype);
    if ((flags & CDSSM_SCAN_TENSOR_CORE_WA) && !(flags & CDSSM_SCAN_FORCE_SIMT) && (!wa_ok || H % 4)) return CDSSM_ERR_UNSUPPORTED;
    // (the precision that the CUDA-core walk gave these calls before they came here)
    const int wa_parts = (H % 4 == 0 && tail_state == nullptr) || (flags & CDSSM_SCAN_TENSOR_CORE_WA) ? 2 : 3;
    const bool tc_local = !(flags & CDSSM_SCAN_KEEP_SIMT_LOCAL), tc_output = !(flags & CDSSM_SCAN_KEEP_SIMT_OUTPUT);
    // The whole-chunk scan hands the carry on inside one kernel where the scratch has room for the words that do it; else local,
    // carry and output pass: the same arithmetic in the same order, so this choice may go by size.
    const size_t records = align256(scan_record_bytes(B, L, H, N, C));
    const bool one_kernel = tile_ok && tc_local && tc_output && a.run_local && !summary_only && hands_carry_on(B, H, a.NC, D, N) &&
                            workspace_bytes - base >= records + scan_tile_extra_bytes(B, L, H, D, N);
    // Status word; for the one-kernel scan everything from there through the chunks' words, and the carries: cleared by the records
    // kernel where that runs first.
    const bool tensor = wa_ok || tile_ok;
    const bool fill_records = tensor && (a.run_local || (flags & CDSSM_SCAN_TENSOR_CORE_WA));
    void* rec = reinterpret_cast<char*>(a.ws_state) + align256((size_t)a.units * 2 * D * sizeof(float));
    void* extra = static_cast<char*>(rec) + records;
    if (!fill_records)
        if (int rc = check_cuda(cudaMemsetAsync(status, 0, sizeof(int), st))) return rc;
    a.rec_av = nullptr;
    a.rec_bs = nullptr;
    if (!tensor && workspace_bytes - base >= simt_record_bytes(B, L, H, N, C)) {
        a.rec_av = static_cast<float4*>(rec);
        a.rec_bs = reinterpret_cast<float2*>(a.rec_av + (size_t)a.units * C);
    }
    if (flags & CDSSM_SCAN_EXACT) {
        a.rec_av = nullptr;   // (its stages are not the chunks of the records)
        // the recurrent state after the last token is both the "carry" and the tail state
        const int cols = (D + kLanesPerUnit - 1) / kLanesPerUnit;
        float* extra = tail_state;
        if (!a.final_state) { a.final_state = tail_state; extra = nullptr; }
        int rc;
        if (dtype == CDSSM_BF16) rc = cols <= 8 ? launch_recurrent<__nv_bfloat16, 8>(a, st) : launch_recurrent<__nv_bfloat16, 16>(a, st);
        else rc = cols <= 8 ? launch_recurrent<float, 8>(a, st) : launch_recurrent<float, 16>(a, st);
        if (rc == CDSSM_OK && extra && a.final_state)
            rc = check_cuda(cudaMemcpyAsync(extra, a.final_state, sizeof(float) * (size_t)B * H * N * D,
                                            cudaMemcpyDeviceToDevice, st));
        return rc;
    }
    if (!tensor) return scan_fused_simt(a, dtype, st);
    const int withhold = (flags & CDSSM_SCAN_TEST_WITHHOLD) ? 1 : 0;
    const unsigned long long limit = wait_limit_ns();
    const int from_chunks = (wa_ok ? carry_in_output(B, a.NC, H) : few_chunks(B, H, a.NC, D, N)) && tc_local && tc_output && a.run_local && !summary_only &&
                            !writes_into_h0(a);
    auto pass = [&](int mode) {   // 0: local, 1: output, 2: both in one kernel
        if (wa_ok)
            return scan_wa_pass(mode == 1, q, q_rs, k, k_rs, rec, a.ws_gamma, a.ws_state, y, tail_state, status, shortcut_scale, B, L, H, D,
                                limit, withhold, from_chunks, h0, final_state, wa_parts, st);
        return scan_tile_pass(mode, from_chunks, q, q_rs, k, k_rs, rec, h0, y, final_state, tail_state, a.ws_gamma, a.ws_state, one_kernel ? extra : nullptr,
                              status, status + 1, shortcut_scale, B, L, H, D, N, limit, withhold, st);
    };
    // (a summary of the same inputs has left the records in the workspace, in the order of the kernels that sizes alone choose)
    if (fill_records)
        if (int rc = scan_records(wa_ok, v, v_rs, rows.first, vf_rs, rows.mix, gate_raw, g_rs, log_dt_scale, rope_freqs, rec, status,
                                  one_kernel ? 64 + scan_tile_words(B, L, H, D, N) : 1, static_cast<int*>(extra),
                                  one_kernel ? scan_tile_extra_bytes(B, L, H, D, N) / sizeof(int) : 0, a.dc, B, L, H, N, C, pos0, segs,
                                  a.fp32_decay, st))
            return rc;
    if (one_kernel) return pass(2);
    if (a.run_local && tc_local) {
        if (int rc = pass(0)) return rc;
        a.run_local = 0;
    }
    if (from_chunks) return pass(1);
    a.run_output = tc_output ? 0 : 1;
    if (int rc = scan_fused_simt(a, dtype, st)) return rc;   // carry pass (+ whatever was kept)
    return !tc_output || summary_only ? CDSSM_OK : pass(1);
}

static int decode_step_impl(float* state, const void* q, const void* k, const void* v,
                            const void* gate_raw, const float* log_dt_scale, const float* rope_freqs,
                            void* y, float gating_c, float omega_thresh, float adt_delta,
                            float adt_smoothness, float adt_eps, float shortcut_scale, int B, int H, int D,
                            int N, int pos, const int* pos_dev, int dtype, void* stream, float* corr = nullptr,
                            float* carry = nullptr, float* gamma = nullptr, int C = 0, long long k_stride = 0,
                            long long v_stride = 0, const void* v_first = nullptr, const void* mix = nullptr,
                            long long q_stride = 0, long long g_stride = 0) {
    if (!state || !q || !k || !v || !gate_raw || !log_dt_scale || !rope_freqs || !y)
        return CDSSM_ERR_BAD_ARG;
    if (corr && (!carry || !gamma || C <= 0 || (((uintptr_t)corr | (uintptr_t)carry) & 15))) return CDSSM_ERR_BAD_ARG;
    if (B < 0 || H <= 0 || D <= 0 || N <= 0 || (N & 1)) return CDSSM_ERR_BAD_ARG;
    if (dtype != CDSSM_BF16 && dtype != CDSSM_F32) return CDSSM_ERR_BAD_ARG;
    if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)state) & 15) return CDSSM_ERR_BAD_ARG;
    if (N > kMaxStateDim || D > kMaxHeadDim) return CDSSM_ERR_UNSUPPORTED;
    if (B == 0) return CDSSM_OK;
    DecodeArgs a;
    a.state = state; a.q = q; a.k = k; a.v = v; a.gate_raw = gate_raw;
    a.corr = corr; a.carry = carry; a.gamma = gamma; a.C = C;
    a.k_stride = k_stride ? k_stride : (long long)H * D;
    a.v_stride = v_stride ? v_stride : (long long)H * N;
    a.v_first = v_first; a.mix = mix;
    a.q_stride = q_stride ? q_stride : (long long)H * D;
    a.g_stride = g_stride ? g_stride : (long long)(N + 5) * H;
    {
        const long long es = dtype == CDSSM_F32 ? 4 : 2;
        const bool vec_rows = D == 64 || D == 128;                             // 16-byte row loads of k and q
        if (vec_rows && (((a.k_stride | a.q_stride) * es) & 15)) return CDSSM_ERR_BAD_ARG;
        if (a.q_stride < (long long)H * D || a.g_stride < (long long)(N + 5) * H) return CDSSM_ERR_BAD_ARG;
        if (a.k_stride < (long long)H * D || a.v_stride < (long long)H * N) return CDSSM_ERR_BAD_ARG;
        if ((v_first != nullptr) != (mix != nullptr)) return CDSSM_ERR_BAD_ARG;
        if (corr && (v_first || k_stride || v_stride || q_stride || g_stride)) return CDSSM_ERR_UNSUPPORTED;
    }
    a.log_dt_scale = log_dt_scale; a.rope_freqs = rope_freqs; a.y = y;
    a.dc = DynConsts{gating_c, omega_thresh, adt_delta, adt_smoothness, adt_eps};
    a.shortcut_scale = shortcut_scale;
    a.B = B; a.H = H; a.D = D; a.N = N; a.pos = pos; a.pos_dev = pos_dev;
    a.units = (long long)B * H * (N / 2);
    const int cols = (D + kLanesPerUnit - 1) / kLanesPerUnit;
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == CDSSM_BF16)
        return cols <= 8 ? launch_decode<__nv_bfloat16, 8>(a, st) : launch_decode<__nv_bfloat16, 16>(a, st);
    return cols <= 8 ? launch_decode<float, 8>(a, st) : launch_decode<float, 16>(a, st);
}

extern "C" int cdssm_b200_scan_fused_fwd(const void* q, const void* k, const void* v,
                                         const void* gate_raw, const float* log_dt_scale,
                                         const float* rope_freqs, const float* h0, void* y,
                                         float* final_state, float* tail_state, void* workspace,
                                         size_t workspace_bytes, float gating_c,
                                         float omega_thresh, float adt_delta, float adt_smoothness,
                                         float adt_eps, float shortcut_scale, int B, int L, int H,
                                         int D, int N, int C, int pos0, int dtype, int flags,
                                         void* stream) {
    return scan_fused_impl(q, k, v, gate_raw, log_dt_scale, rope_freqs, h0, y, final_state, tail_state,
                           nullptr, false, workspace, workspace_bytes, gating_c, omega_thresh, adt_delta,
                           adt_smoothness, adt_eps, shortcut_scale, B, L, H, D, N, C, pos0, 1, dtype, flags,
                           stream);
}

extern "C" int cdssm_b200_scan_fused_strided_fwd(const void* q, int64_t q_row_stride, const void* k, int64_t k_row_stride,
                                                 const void* v, int64_t v_row_stride, const void* v_first,
                                                 int64_t v_first_row_stride, const void* mix, const void* gate_raw,
                                                 int64_t gate_row_stride, const float* log_dt_scale, const float* rope_freqs,
                                                 const float* h0, void* y, float* final_state, float* tail_state,
                                                 void* workspace, size_t workspace_bytes, float gating_c, float omega_thresh,
                                                 float adt_delta, float adt_smoothness, float adt_eps, float shortcut_scale,
                                                 int B, int L, int H, int D, int N, int C, int pos0, int dtype, int flags,
                                                 void* stream) {
    ScanRows r;
    r.q = q_row_stride; r.k = k_row_stride; r.v = v_row_stride; r.gate = gate_row_stride;
    r.first = v_first; r.v_first = v_first_row_stride; r.mix = mix;
    return scan_fused_impl(q, k, v, gate_raw, log_dt_scale, rope_freqs, h0, y, final_state, tail_state, nullptr, false,
                           workspace, workspace_bytes, gating_c, omega_thresh, adt_delta, adt_smoothness, adt_eps,
                           shortcut_scale, B, L, H, D, N, C, pos0, 1, dtype, flags, stream, false, r);
}

extern "C" int cdssm_b200_scan_fused_segmented_fwd(const void* q, const void* k, const void* v,
                                                   const void* gate_raw, const float* log_dt_scale,
                                                   const float* rope_freqs, const float* h0, void* y,
                                                   float* final_state, void* workspace,
                                                   size_t workspace_bytes, float gating_c,
                                                   float omega_thresh, float adt_delta,
                                                   float adt_smoothness, float adt_eps,
                                                   float shortcut_scale, int B, int L, int H, int D, int N,
                                                   int C, int pos0, int segs, int dtype, int flags,
                                                   void* stream) {
    return scan_fused_impl(q, k, v, gate_raw, log_dt_scale, rope_freqs, h0, y, final_state, nullptr,
                           nullptr, false, workspace, workspace_bytes, gating_c, omega_thresh, adt_delta,
                           adt_smoothness, adt_eps, shortcut_scale, B, L, H, D, N, C, pos0, segs, dtype,
                           flags, stream);
}

extern "C" int cdssm_b200_scan_summary_fwd(const void* k, const void* v, const void* gate_raw,
                                           const float* log_dt_scale, const float* rope_freqs,
                                           const float* h0, float* carry_out, float* total_decay,
                                           void* workspace, size_t workspace_bytes, float gating_c,
                                           float omega_thresh, float adt_delta, float adt_smoothness,
                                           float adt_eps, int B, int L, int H, int D, int N, int C, int pos0,
                                           int segs, int dtype, int flags, void* stream) {
    if (!carry_out || !total_decay) return CDSSM_ERR_BAD_ARG;
    if (flags & ~CDSSM_SCAN_FP32_DECAY) return CDSSM_ERR_BAD_ARG;   // the only option that applies to a summary
    return scan_fused_impl(nullptr, k, v, gate_raw, log_dt_scale, rope_freqs, h0, nullptr, carry_out,
                           nullptr, total_decay, true, workspace, workspace_bytes, gating_c, omega_thresh,
                           adt_delta, adt_smoothness, adt_eps, 0.f, B, L, H, D, N, C, pos0, segs, dtype,
                           flags, stream);
}

// ---------------------------------------------------------------------------------------------
// Allocation-free variant of the fused scan.
//
// Some hosts of this library cannot hand it a workspace: an inference server whose memory pool
// already owns every byte of the device, a plugin that runs inside somebody else's framework and
// is not allowed to call the CUDA allocator (cudaMalloc synchronises the whole device and would
// stall the other streams of that process), or an embedding whose allocator is simply not reachable
// from where the scan is called.  For them the scratch of the three-launch scan lives in a
// file-scope device array that the module carries itself: kNoAllocScratchBytes on every GPU that
// loads the library, for as long as the process lives.
//
// In host code the array's name is only a handle for the symbol, not a device pointer; the device
// address is looked up once per device with cudaGetSymbolAddress (with that device current) and it
// is this address that the kernels receive.
constexpr size_t kNoAllocScratchBytes = 16u << 20;   // 16 MiB
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];
constexpr int kNoAllocMaxDevices = 64;
static std::atomic<void*> g_noalloc_scratch_of_device[kNoAllocMaxDevices];   // device address of the array, per device

extern "C" size_t cdssm_b200_scan_fused_noalloc_max_bytes(void) { return kNoAllocScratchBytes; }

extern "C" int cdssm_b200_scan_fused_fwd_noalloc(const void* q, const void* k, const void* v,
                                                 const void* gate_raw, const float* log_dt_scale,
                                                 const float* rope_freqs, const float* h0, void* y,
                                                 float* final_state, float* tail_state, float gating_c,
                                                 float omega_thresh, float adt_delta,
                                                 float adt_smoothness, float adt_eps,
                                                 float shortcut_scale, int B, int L, int H, int D, int N,
                                                 int C, int pos0, int dtype, int flags, void* stream) {
    if (B <= 0 || L <= 0) {   // nothing to do, but still validate like the allocating entry point
        return cdssm_b200_scan_fused_fwd(q, k, v, gate_raw, log_dt_scale, rope_freqs, h0, y, final_state,
                                         tail_state, nullptr, 0, gating_c, omega_thresh, adt_delta,
                                         adt_smoothness, adt_eps, shortcut_scale, B, L, H, D, N, C, pos0,
                                         dtype, flags, stream);
    }
    if (cdssm_b200_scan_fused_workspace_bytes(B, L, H, D, N, C) == 0) return CDSSM_ERR_BAD_ARG;
    // beyond the built-in scratch?  (the records of the tensor-core kernel of N = 2 are part of it, others only as they fit)
    size_t need = base_workspace_bytes(B, L, H, D, N, C);
    if (scan_wa_supported(D, N, C, CDSSM_BF16) && H % 4 == 0) need += align256(scan_record_bytes(B, L, H, N, C));
    if (need > kNoAllocScratchBytes) return CDSSM_ERR_WORKSPACE;
    int dev = 0;
    if (int rc = check_cuda(cudaGetDevice(&dev))) return rc;
    if (dev < 0 || dev >= kNoAllocMaxDevices) return CDSSM_ERR_UNSUPPORTED;
    void* scratch = g_noalloc_scratch_of_device[dev].load(std::memory_order_acquire);
    if (scratch == nullptr) {
        // one-time set-up for this device (do it before any stream capture begins); two host threads that
        // race here both look up the same address
        if (int rc = check_cuda(cudaGetSymbolAddress(&scratch, g_noalloc_scratch))) return rc;
        g_noalloc_scratch_of_device[dev].store(scratch, std::memory_order_release);
    }
    // Nothing in the scratch has to start at zero except the status word, which the scan itself
    // clears on the stream; gamma/state slots are all written by the local pass before they are read.
    return scan_fused_impl(q, k, v, gate_raw, log_dt_scale, rope_freqs, h0, y, final_state, tail_state, nullptr, false,
                           scratch, kNoAllocScratchBytes, gating_c, omega_thresh, adt_delta, adt_smoothness, adt_eps,
                           shortcut_scale, B, L, H, D, N, C, pos0, 1, dtype, flags, stream, true);
}

extern "C" int cdssm_b200_scan_fused_noalloc_status(int* status_host, void* stream) {
    if (!status_host) return CDSSM_ERR_BAD_ARG;
    int dev = 0;
    if (int rc = check_cuda(cudaGetDevice(&dev))) return rc;
    if (dev < 0 || dev >= kNoAllocMaxDevices) return CDSSM_ERR_UNSUPPORTED;
    void* p = g_noalloc_scratch_of_device[dev].load(std::memory_order_acquire);
    if (!p) return CDSSM_ERR_BAD_ARG;   // no allocation-free call has run on this device yet
    return cdssm_b200_scan_fused_status(p, status_host, stream);
}

extern "C" int cdssm_b200_decode_step(float* state, const void* q, const void* k, const void* v,
                                      const void* gate_raw, const float* log_dt_scale,
                                      const float* rope_freqs, void* y, float gating_c,
                                      float omega_thresh, float adt_delta, float adt_smoothness,
                                      float adt_eps, float shortcut_scale, int B, int H, int D,
                                      int N, int pos, int dtype, void* stream) {
    return decode_step_impl(state, q, k, v, gate_raw, log_dt_scale, rope_freqs, y, gating_c, omega_thresh,
                            adt_delta, adt_smoothness, adt_eps, shortcut_scale, B, H, D, N, pos, nullptr,
                            dtype, stream);
}

extern "C" int cdssm_b200_decode_step_at(float* state, const void* q, const void* k, const void* v,
                                         const void* gate_raw, const float* log_dt_scale,
                                         const float* rope_freqs, void* y, float gating_c,
                                         float omega_thresh, float adt_delta, float adt_smoothness,
                                         float adt_eps, float shortcut_scale, int B, int H, int D, int N,
                                         const int* pos_dev, int dtype, void* stream) {
    if (!pos_dev) return CDSSM_ERR_BAD_ARG;
    return decode_step_impl(state, q, k, v, gate_raw, log_dt_scale, rope_freqs, y, gating_c, omega_thresh,
                            adt_delta, adt_smoothness, adt_eps, shortcut_scale, B, H, D, N, 0, pos_dev,
                            dtype, stream);
}

extern "C" int cdssm_b200_decode_step_strided(float* state, const void* q, int64_t q_row_stride, const void* k,
                                              int64_t k_row_stride, const void* v, int64_t v_row_stride,
                                              const void* v_first, const void* mix, const void* gate_raw,
                                              int64_t gate_row_stride, const float* log_dt_scale,
                                              const float* rope_freqs, void* y, float gating_c, float omega_thresh,
                                              float adt_delta, float adt_smoothness, float adt_eps,
                                              float shortcut_scale, int B, int H, int D, int N, int pos,
                                              const int* pos_dev, int dtype, void* stream) {
    if (k_row_stride <= 0 || v_row_stride <= 0 || q_row_stride <= 0 || gate_row_stride <= 0) return CDSSM_ERR_BAD_ARG;
    return decode_step_impl(state, q, k, v, gate_raw, log_dt_scale, rope_freqs, y, gating_c, omega_thresh,
                            adt_delta, adt_smoothness, adt_eps, shortcut_scale, B, H, D, N, pos, pos_dev, dtype,
                            stream, nullptr, nullptr, nullptr, 0, k_row_stride, v_row_stride, v_first, mix, q_row_stride,
                            gate_row_stride);
}

extern "C" int cdssm_b200_decode_step_reference(float* local_state, float* correction, float* carry, float* chunk_decay,
                                                const void* q, const void* k, const void* v, const void* gate_raw,
                                                const float* log_dt_scale, const float* rope_freqs, void* y,
                                                float gating_c, float omega_thresh, float adt_delta,
                                                float adt_smoothness, float adt_eps, float shortcut_scale, int B,
                                                int H, int D, int N, int C, int pos, const int* pos_dev, int dtype,
                                                void* stream) {
    if (!correction || !carry || !chunk_decay || C <= 0 || pos < 0) return CDSSM_ERR_BAD_ARG;
    return decode_step_impl(local_state, q, k, v, gate_raw, log_dt_scale, rope_freqs, y, gating_c, omega_thresh,
                            adt_delta, adt_smoothness, adt_eps, shortcut_scale, B, H, D, N, pos, pos_dev, dtype,
                            stream, correction, carry, chunk_decay, C);
}
