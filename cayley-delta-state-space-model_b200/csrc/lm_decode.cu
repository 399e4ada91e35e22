// One decode step of the language model for a small batch, five kernels per layer.
//
// At a few sequences per step every product of a layer streams its weights once and does next to nothing with them
// (12 layers of the 768-wide model: 188 MB, 29 us at the measured copy rate), so the step is bounded by its chain of
// dependent phases and by what each of them does before its first load comes back:
//       1 in-projection   RMSNorm of x on the way in; the one-token convolution + SiLU and its history on the way out
//       2 Q and gates     one product
//       3 recurrent step  eight lanes per (sequence, head, pair), decode_unit.cuh
//       4 read-out        a block owns one normalisation group: GroupNorm, silu(z) gate and D * x_conv on the way out
//       5 out-projection  residual sum in place
//     and the head: final RMSNorm, logits.
// A kernel is launched while its predecessor drains (programmatic dependent launch) and requests its weight rows, as mma
// fragments into registers, and the constants of its epilogue BEFORE it waits for the predecessor's results (the step's
// first kernel after: its predecessor is not ours); at most 128
// registers a thread, so that the blocks of two consecutive kernels are resident together.  The activations of all
// sequences go through shared memory as the other operand of mma.sync m16n8k16: the weight rows are the 16-row operand,
// sequences the 8-column one (a tcgen05 tile starts at 128 rows, of which a step of a few sequences could use a
// sixteenth).  Every rounding is where the separate kernels and the library products round.
//
// Measured on B200, 12 layers, d 768, N 2, vocabulary 32000: see lm_decode_takes() for the figures and the line to the
// library products.  One cooperative kernel over all layers, with the same phases and a barrier in global memory between
// them, was slower (B = 16: 396 against 281 us): a meeting of all blocks costs a store drain, an atomic and a poll in a
// row, about 2.4 us, against 1.5 us from one kernel's last store to the next one's first load.
#include "cdssm_common.cuh"
#include "decode_unit.cuh"
#include "sm100_ptx.cuh"
#include <algorithm>

namespace cdssm {
namespace lmstep {

using bf16 = __nv_bfloat16;

constexpr int kThreads = 256, kWarps = 8;
constexpr int kAhead = 6;        // 32-column blocks of weights a warp holds in registers (16 B per row, lane and block)
constexpr size_t kSmemMost = 227 * 1024;

enum Mode { kInProj, kQGates, kReadout, kOutProj, kHead };

struct Args {
    bf16 *x, *proj, *x_conv, *qg, *y, *gated, *logits;
    const bf16 *v_first, *final_norm_w, *head_w;   // v_first: layer 0's V (rows proj_stride apart), or nullptr in layer 0
    float eps_norm, eps_group, eps_final;
    DynConsts dc;
    int B, d, di, H, N, vocab, pos;
    int first;                  // the step's first kernel: the one before it is the caller's and may write the weights
    const int* pos_dev;
    long long proj_stride, qg_stride;
    const void* ahead[2];       // weights of the kernels behind the next one, requested into the L2 cache
    unsigned ahead_bytes[2];
};

// The blocks of a kernel share the request for later weights: at 2.5 us a kernel, the trip to HBM is as long as the kernel,
// and a request a kernel earlier than the register loads hides it.
__device__ __forceinline__ void request_ahead(const Args& a) {
    if (threadIdx.x != 0) return;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const unsigned share = ((a.ahead_bytes[i] + gridDim.x - 1) / gridDim.x + 127) & ~127u, at = share * blockIdx.x;
        if (at < a.ahead_bytes[i])
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(static_cast<const char*>(a.ahead[i]) + at),
                         "r"(min(share, a.ahead_bytes[i] - at)) : "memory");
    }
}

__host__ __device__ inline int x_pitch(int K) {   // bytes: rows 64 bytes off each other's banks
    const int b = ((K + 31) / 32) * 64;
    return (b & 64) ? b : b + 64;
}

// One product of a phase.
struct Product {
    const bf16* w;            // (M, K) row-major
    const bf16* x;            // (B, x_stride)
    long long x_stride;
    int M, K;
    int apart;                // the partial sums have shared memory of their own, beside the activations
};

// Weight rows of work item `item` to registers: rows g and g + 8 of the warp's fragment, columns 8 t .. 8 t + 7 of the
// 32-column blocks kp, kp + KW, ...
template <int MT>
__device__ __forceinline__ void fetch_block(const Product& p, int tile, int i, uint4 (&r)[2]) {
    constexpr int KW = kWarps / MT;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int col = (warp / MT + i * KW) * 32 + 8 * (lane & 3), row = tile * 16 * MT + (warp % MT) * 16 + (lane >> 2);
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    const bool on = col < p.K && warp < MT * KW;
    r[0] = on && row < p.M ? __ldg(reinterpret_cast<const uint4*>(p.w + (size_t)row * p.K + col)) : zero;
    r[1] = on && row + 8 < p.M ? __ldg(reinterpret_cast<const uint4*>(p.w + (size_t)(row + 8) * p.K + col)) : zero;
}
template <int MT>
__device__ __forceinline__ void fetch_first(const Product& p, int tile, uint4 (&wr)[kAhead][2]) {
#pragma unroll
    for (int i = 0; i < kAhead; i++) fetch_block<MT>(p, tile, i, wr[i]);
}

// One product: every work item (row tile, batch tile) of the block.  Only the head has more items than blocks.
template <int NT, int MT, Mode kMode>
__global__ void __launch_bounds__(kThreads, NT == 8 ? 1 : 2)
lm_product_kernel(const Args a, const cdssm_lm_layer w, const Product p, bf16* const out, const long long out_stride) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int KW = kWarps / MT, kRows = 16 * MT, kRP = kRows + 4;
    constexpr bool kNorm = kMode == kInProj || kMode == kHead;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int mt = warp % MT, kp = warp / MT;
    const int pitch = x_pitch(p.K), kblocks = (p.K + 31) / 32;
    const int mine = warp < MT * KW ? (kblocks - kp + KW - 1) / KW : 0;
    const int tiles = (p.M + kRows - 1) / kRows, btiles = (a.B + NT * 8 - 1) / (NT * 8), items = tiles * btiles;
    float* red = reinterpret_cast<float*>(smem + (kMode == kHead || p.apart ? (size_t)NT * 8 * pitch : 0));
    uint4 wr[kAhead][2];
    if (kMode == kInProj && a.first) grid_dependency_wait();
    if ((int)blockIdx.x < items) fetch_first<MT>(p, (int)blockIdx.x % tiles, wr);
    constexpr int kNormAhead = 3;   // 256-column pieces of the norm's weights that are there before the activations are; wider rows load the rest
                                    // afterwards (more of them would be registers of every width's kernel)
    uint4 nwr[kNormAhead];
    const bf16* nw = kMode == kHead ? a.final_norm_w : (const bf16*)w.norm_w;
    if (kNorm) {
#pragma unroll
        for (int i = 0; i < kNormAhead; i++)
            if (lane * 8 + 256 * i < p.K) nwr[i] = __ldg(reinterpret_cast<const uint4*>(nw + lane * 8 + 256 * i));
    }
    request_ahead(a);
    bool waited = false;
    int staged = -1;      // batch tile whose activations are in shared memory
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
        const int tile = item % tiles, b0 = (item / tiles) * NT * 8, nb = min(NT * 8, a.B - b0);
        if (item != (int)blockIdx.x) {
            __syncthreads();                        // the previous item's sums have been read
        }
        // ---- operands of the epilogue: constants first, then what predecessors wrote.  Outputs of a thread: sequence
        // tid / kRows + e * (256 / kRows), always the same row (read-out: sequence warp + 8 e, rows lane + 32 i)
        constexpr int kPer = (kRows + 31) / 32, kOut = kMode == kReadout ? NT : (NT * 8 * kRows + 255) / 256;
        constexpr int kBStep = 256 / kRows;
        const int r_own = tid % kRows, b_own = tid / kRows, m_own = tile * kRows + r_own;
        float bias = 0.f, cw[5], hist[kOut][3], res[kOut], zz[kOut][kPer], xc[kOut][kPer], gnw[kPer], gnb[kPer], skip[kPer];
        const bool conv = kMode == kInProj && m_own >= a.di && m_own < 2 * a.di;
        const int ch = m_own - a.di;
        if (kMode == kReadout) {
#pragma unroll
            for (int i = 0; i < kPer; i++) {
                const int r = lane + 32 * i, m = tile * kRows + r;
                const bool on = r < kRows;
                gnw[i] = on ? IO<bf16>::ld((const bf16*)w.gn_w + m) : 0.f;
                gnb[i] = on ? IO<bf16>::ld((const bf16*)w.gn_b + m) : 0.f;
                skip[i] = on ? IO<bf16>::ld((const bf16*)w.skip + m) : 0.f;
            }
        } else if (m_own < p.M) {
            if (kMode == kInProj) bias = IO<bf16>::ld((const bf16*)w.b_in + m_own);
            if (kMode == kQGates) bias = IO<bf16>::ld((const bf16*)w.b_qg + m_own);
            if (conv) {
#pragma unroll
                for (int j = 0; j < 4; j++) cw[j] = IO<bf16>::ld((const bf16*)w.conv_w + ch * 4 + j);
                cw[4] = IO<bf16>::ld((const bf16*)w.conv_b + ch);
            }
        }
        if (!waited) {
            grid_dependency_wait();
            grid_launch_dependents();
            waited = true;
        }
        // ---- activations to shared memory (zero rows and columns where the batch or K ends): asynchronous 16-byte
        // copies, all in flight at once; the norm is applied in place by the warp that copied the row
        if (kMode != kHead || staged != b0) {
            for (int b = warp; b < NT * 8; b += kWarps)
                for (int c = lane * 8; c < kblocks * 32; c += 256) {
                    const bool on = b < nb && c < p.K;
                    sm100::cp_async16(smem + (size_t)b * pitch + 2 * c, p.x + (on ? (size_t)(b0 + b) * p.x_stride + c : 0), on);
                }
            sm100::cp_async_commit();
        }
        if (kMode == kReadout) {
#pragma unroll
            for (int i = 0; i < kPer; i++) {
                const int r = lane + 32 * i, m = tile * kRows + r;
#pragma unroll
                for (int e = 0; e < kOut; e++) {
                    const int b = warp + e * kWarps;
                    const bool use = r < kRows && b < nb;
                    zz[e][i] = use ? IO<bf16>::ld(a.proj + (size_t)(b0 + b) * a.proj_stride + m) : 0.f;
                    xc[e][i] = use ? IO<bf16>::ld(a.x_conv + (size_t)(b0 + b) * a.di + m) : 0.f;
                }
            }
        } else if (m_own < p.M) {
#pragma unroll
            for (int e = 0; e < kOut; e++) {
                const int b = b_own + e * kBStep;
                if (b < nb) {
                    const size_t row = (size_t)(b0 + b);
                    if (kMode == kOutProj) res[e] = IO<bf16>::ld(out + row * out_stride + m_own);
                    if (conv) {
#pragma unroll
                        for (int j = 0; j < 3; j++) hist[e][j] = IO<bf16>::ld((const bf16*)w.conv + row * 3 * a.di + j * a.di + ch);
                    }
                }
            }
        }
        if (kMode != kHead || staged != b0) {
            sm100::cp_async_wait_all();
            __syncwarp();
            if (kNorm) {
                const float eps = kMode == kHead ? a.eps_final : a.eps_norm;
                for (int b = warp; b < nb; b += kWarps) {
                    bf16* xs = reinterpret_cast<bf16*>(smem + (size_t)b * pitch);
                    float ss = 0.f;
                    for (int c = lane * 8; c < p.K; c += 256) {
                        float f[8];
                        Vec8<bf16>::ld(xs + c, f);
#pragma unroll
                        for (int e = 0; e < 8; e++) ss += f[e] * f[e];
                    }
                    const float rms = rsqrtf(warp_sum(ss) / (float)p.K + eps);
                    auto scale = [&](int c, const uint4& weights) {
                        float f[8], n[8];
                        Vec8<bf16>::ld(xs + c, f);
                        unpack8(weights, n);
#pragma unroll
                        for (int e = 0; e < 8; e++) f[e] = IO<bf16>::rnd(f[e] * rms) * n[e];
                        Vec8<bf16>::st(xs + c, f);
                    };
#pragma unroll
                    for (int i = 0; i < kNormAhead; i++)
                        if (lane * 8 + 256 * i < p.K) scale(lane * 8 + 256 * i, nwr[i]);
                    for (int c = lane * 8 + 256 * kNormAhead; c < p.K; c += 256) scale(c, __ldg(reinterpret_cast<const uint4*>(nw + c)));
                }
            }
            staged = b0;
            __syncthreads();
        }
        // ---- the product
        float acc[NT][4];
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[j][e] = 0.f;
        for (int i0 = 0; i0 < mine; i0 += kAhead) {
#pragma unroll
            for (int s = 0; s < kAhead; s++) {
                if (i0 + s < mine) {
                    const uint4 lo = wr[s][0], hi = wr[s][1];
                    const uint32_t a0[4] = {lo.x, hi.x, lo.y, hi.y}, a1[4] = {lo.z, hi.z, lo.w, hi.w};
                    const unsigned char* xs = smem + (size_t)g * pitch + ((kp + (i0 + s) * KW) * 32 + 8 * t) * 2;
                    if (i0 + s + kAhead < mine) fetch_block<MT>(p, tile, i0 + s + kAhead, wr[s]);   // the slot is free
#pragma unroll
                    for (int j = 0; j < NT; j++) {
                        const uint4 b = *reinterpret_cast<const uint4*>(xs + (size_t)j * 8 * pitch);
                        sm100::mma_bf16_m16n8k16(acc[j], a0, b.x, b.y);
                        sm100::mma_bf16_m16n8k16(acc[j], a1, b.z, b.w);
                    }
                }
            }
        }
        if (kMode == kHead && item + (int)gridDim.x < items)   // the next item's weights travel during the epilogue
            fetch_first<MT>(p, (item + gridDim.x) % tiles, wr);
        if (kMode != kHead && !p.apart) __syncthreads();   // the sums take the place of the activations
        if (warp < MT * KW) {
            float* mr = red + (size_t)kp * NT * 8 * kRP;
#pragma unroll
            for (int j = 0; j < NT; j++) {
                mr[(8 * j + 2 * t) * kRP + mt * 16 + g] = acc[j][0];
                mr[(8 * j + 2 * t + 1) * kRP + mt * 16 + g] = acc[j][1];
                mr[(8 * j + 2 * t) * kRP + mt * 16 + g + 8] = acc[j][2];
                mr[(8 * j + 2 * t + 1) * kRP + mt * 16 + g + 8] = acc[j][3];
            }
        }
        __syncthreads();
        auto total = [&](int b, int r) {
            float s = 0.f;
#pragma unroll
            for (int q = 0; q < KW; q++) s += red[((size_t)q * NT * 8 + b) * kRP + r];
            return s;
        };
        if (kMode == kReadout) {   // one warp per sequence: the item's rows are one group
#pragma unroll
            for (int e = 0; e < kOut; e++) {
                const int b = warp + e * kWarps;
                if (b >= nb) break;
                float f[kPer], s = 0.f, q = 0.f;
#pragma unroll
                for (int i = 0; i < kPer; i++) {
                    const int r = lane + 32 * i;
                    f[i] = r < kRows ? IO<bf16>::rnd(total(b, r)) : 0.f;
                    s += f[i];
                    q += f[i] * f[i];
                }
                s = warp_sum(s);
                q = warp_sum(q);
                const float mean = s / (float)kRows;
                const float rstd = rsqrtf(fmaxf(q / (float)kRows - mean * mean, 0.f) + a.eps_group);
#pragma unroll
                for (int i = 0; i < kPer; i++) {
                    const int r = lane + 32 * i;
                    if (r < kRows) {
                        const float n = IO<bf16>::rnd((f[i] - mean) * rstd * gnw[i] + gnb[i]);
                        const float z = IO<bf16>::rnd(siluf_<true>(zz[e][i]));
                        IO<bf16>::st(out + (size_t)(b0 + b) * out_stride + tile * kRows + r,
                                     IO<bf16>::rnd(n * z) + IO<bf16>::rnd(skip[i] * xc[e][i]));
                    }
                }
            }
        } else if (m_own < p.M && (kRows == 16 || kRows == 32)) {
#pragma unroll
            for (int e = 0; e < kOut; e++) {
                const int b = b_own + e * kBStep;
                if (b >= nb) break;
                const size_t row = (size_t)(b0 + b);
                float v = total(b, r_own) + bias;
                if (kMode == kOutProj) v += res[e];
                if (conv) {
                    const float x3 = IO<bf16>::rnd(v);
                    const float y = cw[0] * hist[e][0] + cw[1] * hist[e][1] + cw[2] * hist[e][2] + cw[3] * x3 + cw[4];
                    IO<bf16>::st(a.x_conv + row * a.di + ch, siluf_<true>(y));
                    bf16* h = (bf16*)w.conv + row * 3 * a.di + ch;
                    IO<bf16>::st(h, hist[e][1]);
                    IO<bf16>::st(h + a.di, hist[e][2]);
                    IO<bf16>::st(h + 2 * a.di, x3);
                } else {
                    IO<bf16>::st(out + row * out_stride + m_own, v);
                }
            }
        }
    }
}

// The recurrent step of a layer: eight lanes per (sequence, head, pair).
__global__ void __launch_bounds__(128) lm_step_kernel(const Args a, const cdssm_lm_layer w) {
    request_ahead(a);
    // (the state is the step's before, k and v are two kernels back: the one before this has waited for both)
    DecodeUnitArgs u;
    u.state = (float*)w.state;
    u.q = a.qg; u.q_stride = a.qg_stride;
    u.k = a.proj + 2 * a.di; u.k_stride = a.proj_stride;
    u.v = a.proj + 3 * a.di; u.v_stride = a.proj_stride;
    u.v_first = a.v_first; u.v_first_stride = a.proj_stride;
    u.mix = w.mix;
    u.gate = a.qg + a.di; u.gate_stride = a.qg_stride;
    u.log_dt_scale = w.log_dt_scale; u.rope_freqs = w.rope_freqs;
    u.y = a.y;
    u.dc = a.dc;
    u.shortcut_scale = w.shortcut_scale;
    u.H = a.H; u.D = 64; u.N = a.N;
    u.pos = a.pos_dev ? *a.pos_dev : a.pos;
    u.units = (long long)a.B * a.H * (a.N / 2);
    decode_unit<bf16, 8>(u, (long long)blockIdx.x * 16 + threadIdx.x / 8, [] {
        grid_dependency_wait();
        grid_launch_dependents();
    });
}

template <int NT, int MT, bool kHeadMode>
static size_t smem_bytes(int K, bool apart = false) {
    const size_t xs = (size_t)NT * 8 * x_pitch(K), red = sizeof(float) * NT * 8 * (kWarps / MT) * (16 * MT + 4);
    return kHeadMode || apart ? xs + red : (xs > red ? xs : red);
}

template <int NT, int MT, Mode kMode> struct KernelTag {};

template <int NT, int MT, Mode kMode>
static int launch(const Args& a, const cdssm_lm_layer& w, const Product& product, bf16* out, long long out_stride, int max_blocks,
                  cudaStream_t st) {
    Product p = product;
    p.apart = smem_bytes<NT, MT, false>(p.K, true) <= kSmemMost / 2 - 1024;   // (a block of the next kernel has room beside it)
    const size_t smem = smem_bytes<NT, MT, kMode == kHead>(p.K, p.apart);
    if (smem > 48 * 1024)
        if (int rc = allow_smem<KernelTag<NT, MT, kMode>>((const void*)lm_product_kernel<NT, MT, kMode>, kSmemMost)) return rc;
    const int items = ((p.M + 16 * MT - 1) / (16 * MT)) * ((a.B + NT * 8 - 1) / (NT * 8));
    const int grid = kMode == kHead && items > max_blocks ? max_blocks : items;
    return launch_overlapped(lm_product_kernel<NT, MT, kMode>, dim3(grid), dim3(kThreads), smem, st, a, w, p, out, out_stride);
}

// The whole batch in one tile where it fits (up to 64 sequences), else the largest tile that does: further tiles of the
// batch read the same weights from the L2 cache.
template <int MT, Mode kMode>
static int launch_batch(const Args& a, const cdssm_lm_layer& w, const Product& p, bf16* out, long long out_stride,
                        int max_blocks, cudaStream_t st) {
    constexpr bool kH = kMode == kHead;
    if (a.B > 32 && smem_bytes<8, MT, kH>(p.K) <= kSmemMost) return launch<8, MT, kMode>(a, w, p, out, out_stride, max_blocks, st);
    if (a.B > 16 && smem_bytes<4, MT, kH>(p.K) <= kSmemMost) return launch<4, MT, kMode>(a, w, p, out, out_stride, max_blocks, st);
    if (a.B > 8 && smem_bytes<2, MT, kH>(p.K) <= kSmemMost) return launch<2, MT, kMode>(a, w, p, out, out_stride, max_blocks, st);
    return launch<1, MT, kMode>(a, w, p, out, out_stride, max_blocks, st);
}

// us per step on B200, these kernels / the library's products with this library's glue kernels, issued natively (in brackets replayed from a
// CUDA graph), all of one build; 12 layers, N 2, vocabulary 32000 (d 512: 8 layers, N 16; d 256: 4 layers):
//     d 256    B 16:  70 / 219  (63 / 86)     B 32:  94 / 223  (86 / 94)     B 128: 162 / 226 (154 / 101)
//     d 512    B 16: 151 / 490 (140 / 233)    B 32: 212 / 459 (199 / 240)    B 128: 469 / 411 (445 / 274)
//     d 768    B 1:  207 / 596 (203 / 396)    B 16: 239 / 587 (226 / 374)    B 32:  349 / 602 (329 / 335)    B 64: 502 / 595 (480 / 335)
//     d 1024   B 16: 300 / 604 (279 / 416)    B 32: 444 / 612 (426 / 415)    B 64:  748 / 605 (728 / 411)
// Issued call by call the library path is bounded by the host that issues its 112 launches (300 to 920 us on a slower host than this one), and
// these kernels win until the activations every block reads (B x d) weigh more: d 512, B 128 and d 1024, B 64 are ahead with the slower host only.
// Inside a captured graph the line is at 32 sequences (the caller's check).
static bool lm_decode_takes(int B, int d, int di, int H, int N, int groups) {
    // 16-byte pieces of every row; a read-out item is one normalisation group of one to four 16-row fragments
    if (d % 32 || (H * N) % 8 || di % groups) return false;
    const int cg = di / groups;
    if (cg != 16 && cg != 32 && cg != 48 && cg != 64) return false;
    if (smem_bytes<1, 1, false>(di) > kSmemMost || smem_bytes<1, 2, true>(d) > kSmemMost) return false;
    return B <= 128 && (long long)B * d <= 65536;
}

}  // namespace lmstep
}  // namespace cdssm

using namespace cdssm;

static size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }

struct DecodeBuffers {   // activations of one step, bf16
    size_t proj0, proj, x_conv, qg, y, gated, total;
};
static DecodeBuffers decode_buffers(int B, int di, int H, int N) {
    const size_t b = (size_t)B * 2;
    DecodeBuffers o;
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t p = at; at += up256(bytes); return p; };
    const size_t cols = ((size_t)(3 * di + H * N) + 7) & ~(size_t)7;
    o.proj0 = take(b * cols);   // layer 0's, kept: its V is every later layer's v_first
    o.proj = take(b * cols);
    o.x_conv = take(b * di);
    o.qg = take(b * (((size_t)di + (N + 5) * H + 7) & ~(size_t)7));
    o.y = take(b * H * N);
    o.gated = take(b * di);
    o.total = at;
    return o;
}

extern "C" size_t cdssm_b200_lm_decode_workspace_bytes(int B, int d_model, int state_dim, int groups, int vocab, int dtype) {
    const int di = 2 * d_model, H = di / 64, N = state_dim;
    if (dtype != CDSSM_BF16 || B <= 0 || d_model <= 0 || N <= 0 || (N & 1) || N > kMaxStateDim || groups <= 0 || vocab <= 0) return 0;
    if (!lmstep::lm_decode_takes(B, d_model, di, H, N, groups)) return 0;
    return decode_buffers(B, di, H, N).total;
}

extern "C" int cdssm_b200_lm_decode(const cdssm_lm_layer* layers, int n_layers, void* x, const void* final_norm_w,
                                    const void* head_w, void* logits, void* workspace, size_t workspace_bytes, float eps_norm,
                                    float eps_group, float eps_final, float gating_c, float omega_thresh, float adt_delta,
                                    float adt_smoothness, float adt_eps, int B, int d_model, int state_dim, int groups,
                                    int vocab, int pos, const int* pos_dev, int dtype, void* stream) {
    using namespace lmstep;
    if (!layers || n_layers <= 0 || !x || !final_norm_w || !head_w || !logits) return CDSSM_ERR_BAD_ARG;
    const size_t need = cdssm_b200_lm_decode_workspace_bytes(B, d_model, state_dim, groups, vocab, dtype);
    if (need == 0) return CDSSM_ERR_UNSUPPORTED;
    if (!workspace || workspace_bytes < need || ((uintptr_t)workspace & 255)) return CDSSM_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    const int di = 2 * d_model, H = di / 64, N = state_dim, G = (N + 5) * H;
    const DecodeBuffers off = decode_buffers(B, di, H, N);
    char* ws = static_cast<char*>(workspace);
    auto at = [&](size_t o) { return reinterpret_cast<bf16*>(ws + o); };
    int dev = 0, sms = 0;
    if (int rc = check_cuda(cudaGetDevice(&dev))) return rc;
    if (int rc = check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev))) return rc;
    Args a = {};
    a.x = (bf16*)x;
    a.x_conv = at(off.x_conv); a.qg = at(off.qg); a.y = at(off.y); a.gated = at(off.gated);
    a.final_norm_w = (const bf16*)final_norm_w;
    a.eps_norm = eps_norm; a.eps_group = eps_group; a.eps_final = eps_final;
    a.dc = DynConsts{gating_c, omega_thresh, adt_delta, adt_smoothness, adt_eps};
    a.B = B; a.d = d_model; a.di = di; a.H = H; a.N = N; a.vocab = vocab;
    a.pos = pos; a.pos_dev = pos_dev;
    a.proj_stride = ((long long)(3 * di + H * N) + 7) & ~7LL;
    a.qg_stride = ((long long)(di + G) + 7) & ~7LL;
    const unsigned step_blocks = (unsigned)(((long long)B * H * (N / 2) + 15) / 16);
    for (int l = 0; l < n_layers; l++) {
        const cdssm_lm_layer& w = layers[l];
        a.proj = at(l == 0 ? off.proj0 : off.proj);
        a.v_first = l == 0 ? nullptr : at(off.proj0) + 3 * di;
        if (l > 0 && !w.mix) return CDSSM_ERR_BAD_ARG;
        const Product in = {(const bf16*)w.w_in, a.x, d_model, 3 * di + H * N, d_model, 0};
        const Product qg = {(const bf16*)w.w_qg, a.x_conv, di, di + G, di, 0};
        const Product ro = {(const bf16*)w.w_readout, a.y, (long long)H * N, di, H * N, 0};
        const Product op = {(const bf16*)w.w_out, a.gated, di, d_model, di, 0};
        auto ahead = [&](const void* w0, size_t b0, const void* w1, size_t b1) {
            a.ahead[0] = w0; a.ahead_bytes[0] = w0 ? (unsigned)b0 & ~15u : 0;
            a.ahead[1] = w1; a.ahead_bytes[1] = w1 ? (unsigned)b1 & ~15u : 0;
        };
        auto bytes = [](const Product& x) { return (size_t)x.M * x.K * 2; };
        const bool last = l + 1 == n_layers;
        a.first = l == 0;
        ahead(qg.w, bytes(qg), nullptr, 0);
        if (int rc = launch_batch<2, kInProj>(a, w, in, a.proj, a.proj_stride, 0, st)) return rc;
        ahead(op.w, bytes(op), ro.w, bytes(ro));
        if (int rc = launch_batch<1, kQGates>(a, w, qg, a.qg, a.qg_stride, 0, st)) return rc;
        if (last) ahead(head_w, std::min<size_t>((size_t)vocab * d_model * 2, 48u << 20), nullptr, 0);
        else ahead(layers[l + 1].w_in, bytes(in), nullptr, 0);
        if (int rc = launch_overlapped(lm_step_kernel, dim3(step_blocks), dim3(128), 0, st, a, w)) return rc;
        ahead(nullptr, 0, nullptr, 0);
        int rc = CDSSM_ERR_UNSUPPORTED;
        switch (di / groups) {
            case 16: rc = launch_batch<1, kReadout>(a, w, ro, a.gated, di, 0, st); break;
            case 32: rc = launch_batch<2, kReadout>(a, w, ro, a.gated, di, 0, st); break;
            case 48: rc = launch_batch<3, kReadout>(a, w, ro, a.gated, di, 0, st); break;
            case 64: rc = launch_batch<4, kReadout>(a, w, ro, a.gated, di, 0, st); break;
        }
        if (rc) return rc;
        if (int rc2 = launch_batch<1, kOutProj>(a, w, op, a.x, d_model, 0, st)) return rc2;
    }
    const Product head = {(const bf16*)head_w, a.x, d_model, vocab, d_model, 0};
    return launch_batch<2, kHead>(a, layers[0], head, (bf16*)logits, vocab, 2 * sms, st);
}
