// Per-token records of the tensor-core scans: dynamics (dynamics_fused.cu:64-139) and the vp scale of block.py:194-195, every
// result rounded to bf16 like the reference's stores (the transition optionally not).
//
// The gates lie heads-fastest, the scans want a head's tokens side by side.  A block takes 32 tokens of 8 or 16 heads, reads
// the gates with the heads across the lanes, and turns its results around in shared memory, so that both sides move whole
// sectors; a thread has the loads of all its values in flight before the first transcendental.  Bounded by issue slots and the
// special-function unit (a pair takes some hundred instructions, nine of them special functions).
// Instructions a pair at N 16: 209 -> 160 without divisions by what is known before and without the special functions' ways for subnormal
// numbers (cdssm_math.cuh), 31.7 -> 26.3 us cold; N 2 328 -> 287 a token-head.
// Measured on B200: 393 216 token-heads, N 16: 58 -> 27 us against one pair at a time with two barriers each; N 2, 7.7 -> 7.5,
// and 2.1 M token-heads 27 -> 26 us against a thread per token-head that wrote its 16-byte record straight to memory.
#include "cdssm_common.cuh"
#include <algorithm>

namespace cdssm {
namespace records {

constexpr int kTokens = 32, kThreads = 256;

struct Args {
    const __nv_bfloat16 *v, *gate_raw;
    const float *log_dt_scale, *rope_freqs;
    uint4* rec;                    // kWa: {a_re, a_im | v pair | beta, sel_C} (B, 32-token blocks, H, 32)
    float2* rec_a;                 // else: transition (B,NC,H,NP,C)
    uint32_t *rec_v, *rec_g;       // vp-scaled v (B,NC,H,NP,C); beta and sel_C (B,NC,H,C), bf16 pairs
    const __nv_bfloat16 *v_first, *mix;   // or nullptr: v <- lerp(v_first, v, mix[head])
    long long v_rs, vf_rs, g_rs;   // elements between token rows
    int *clear, *clear2;           // words cleared here for the passes that follow (16-byte aligned; the second: a multiple of four)
    size_t clear_words, clear2_words;
    DynConsts dc;
    int B, L, H, N, C, NC, pos0, segs, fp32_decay, tiles;   // tiles: 32-token tiles per batch row, chunks padded to full length
    uint32_t tiles_inv;            // 2^32 / tiles, rounded up (at least two tiles): a division is twenty instructions of every thread
};

__device__ __forceinline__ float bfr(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// (Resident blocks that the registers are cut for.  Left to itself the compiler takes 32 registers for the N = 2 form and has loads wait
// for each other: 3 x 777 tokens of 24 heads 27.3 us a scan, so 26.5.)
template <int kNP, int kHg, bool kResidual, bool kWa>
constexpr int kMinBlocks = kHg == 16 ? 2 : kNP <= 2 ? (kWa ? 5 : 1) : kNP == 8 && kResidual ? 3 : 4;

// kNP: pairs per thread, from kNP * blockIdx.z on; kHg: heads per block.
template <int kNP, int kHg, bool kWa, bool kResidual>
__global__ void __launch_bounds__(kThreads, kMinBlocks<kNP, kHg, kResidual, kWa>) records_kernel(const Args a) {
    using T = __nv_bfloat16;
    constexpr int kItems = kTokens * kHg / kThreads, kRow = kTokens + 1;
    extern __shared__ __align__(16) unsigned char smem[];
    uint4* sr = reinterpret_cast<uint4*>(smem);                        // kWa: [head][token]
    float2* sa = reinterpret_cast<float2*>(smem);                      // else [pair][head][token]
    uint32_t* sv = reinterpret_cast<uint32_t*>(sa + kNP * kHg * kRow);
    uint32_t* sg = sv + kNP * kHg * kRow;
    __shared__ int old_ticket;   // (read by nobody: the wait for it is what counts)
    grid_dependency_wait();
    const size_t first = ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * kThreads + threadIdx.x, step = (size_t)gridDim.x * gridDim.y * kThreads;
    if (kWa) {   // a few words
        for (size_t i = first; i < a.clear_words; i += step) a.clear[i] = 0;
    } else if (blockIdx.z == 0) {
        for (size_t i = first; i < a.clear_words / 4; i += step) reinterpret_cast<uint4*>(a.clear)[i] = make_uint4(0u, 0u, 0u, 0u);
        if (first < a.clear_words % 4) a.clear[a.clear_words / 4 * 4 + first] = 0;
        for (size_t i = first; i < a.clear2_words / 4; i += step) reinterpret_cast<uint4*>(a.clear2)[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    // The whole-chunk scan's wide blocks draw tickets from clear[1] before this kernel is done (scan_tile.cu): the word is zero in the L2 cache
    // when the exchange is back, and nothing else of this launch touches it afterwards (the store above is the same thread's).
    const bool clears_ticket = !kWa && first == 0 && blockIdx.z == 0 && a.clear_words > 1;
    int ticket = 0;
    if (clears_ticket) ticket = atomicExch(a.clear + 1, 0);
    const int H = a.H, N = a.N, NP = N >> 1, p0 = kWa ? 0 : kNP * (int)blockIdx.z, pairs = min(kNP, NP - p0);
    // (One or two pairs a thread are for short inputs, a layer's scan of which takes 15 us whatever these instructions: with the quick
    // division and cut registers the kernel alone took 3.7 us instead of 4.3, but 8 layers of 300 tokens, N 4, 403 us, without 387; 12 of 60,
    // N 8, 545 / 536.  Why is not shown; the moment at which the next kernel's blocks start moves with these instructions.)
    constexpr bool kQuick = kWa || kNP >= 4;
    uint32_t row_of;
    if (kQuick) {
        row_of = __umulhi(blockIdx.x, a.tiles_inv);   // (the quotient, or one more)
        if (row_of * (uint32_t)a.tiles > blockIdx.x) row_of--;
    } else {
        row_of = blockIdx.x / (unsigned)a.tiles;
    }
    const int b = (int)row_of, tile = (int)(blockIdx.x - row_of * (uint32_t)a.tiles), l0 = tile * kTokens;
    // position of the row's first token
    const int before = a.pos0 + (kQuick ? (a.segs > 1 ? (b % a.segs) * a.L : 0) : (b % a.segs) * a.L);
    const int head0 = blockIdx.y * kHg, heads = min(kHg, H - head0);
    const int head = threadIdx.x & (kHg - 1), hd = head0 + min(head, heads - 1);
    const float lds = a.log_dt_scale[hd], freq = a.rope_freqs[hd];
    T x[kItems][7], ga[kItems][kNP], gw[kItems][kNP];
    uint32_t vv[kItems][kNP], vf[kResidual ? kItems : 1][kNP];
#pragma unroll
    for (int i = 0; i < kItems; i++) {
        const int l = min(l0 + (int)(threadIdx.x / kHg) + i * (kThreads / kHg), a.L - 1);
        const size_t row = (size_t)b * a.L + l;
        const T* g = a.gate_raw + row * a.g_rs + hd;
        const uint32_t* v = reinterpret_cast<const uint32_t*>(a.v + row * a.v_rs + hd * N);
#pragma unroll
        for (int s = 0; s < 5; s++) x[i][s] = g[(N + s) * H];
        x[i][5] = g[0];             // (the first pair's: part of what the pairs share)
        x[i][6] = g[NP * H];
#pragma unroll
        for (int p = 0; p < kNP; p++) {
            const int pp = p < pairs ? p0 + p : p0;
            ga[i][p] = g[pp * H];
            gw[i][p] = g[(NP + pp) * H];
            vv[i][p] = v[pp];
        }
        if (kResidual) {
            const uint32_t* f = reinterpret_cast<const uint32_t*>(a.v_first + row * a.vf_rs + hd * N);
#pragma unroll
            for (int p = 0; p < kNP; p++) vf[i][p] = f[p < pairs ? p0 + p : p0];
        }
    }
    const float mix = kResidual ? __bfloat162float(a.mix[hd]) : 0.f;
#pragma unroll
    for (int i = 0; i < kItems; i++) {
        const int t = (int)(threadIdx.x / kHg) + i * (kThreads / kHg), l = l0 + t;
        const bool on = l < a.L;                                       // behind the end a = 1, beta = v = 0: the state stands still
        const float pos = (float)(l + before);
        auto f = [](T y) { return __bfloat162float(y); };
        const DynShared ds = dyn_shared<true, kWa>(f(x[i][5]), f(x[i][6]), f(x[i][0]), f(x[i][1]), f(x[i][2]), f(x[i][3]), f(x[i][4]),
                                              lds, freq, pos, a.dc);
        const uint32_t bs = on ? pack2(ds.beta, ds.sel_c) : 0u;
        if (!kWa) sg[head * kRow + t] = bs;
#pragma unroll
        for (int p = 0; p < kNP; p++) {
            if (p >= pairs) break;
            float ar, ai, vp;
            dyn_pair<true, kWa>(f(ga[i][p]), f(gw[i][p]), freq, pos, ds, ar, ai, vp);
            if (!a.fp32_decay) { ar = bfr(ar); ai = bfr(ai); }
            vp = bfr(vp);
            float v0 = __uint_as_float(vv[i][p] << 16), v1 = __uint_as_float(vv[i][p] & 0xffff0000u);
            if (kResidual) {
                v0 = value_residual<T>(__uint_as_float(vf[i][p] << 16), v0, mix);
                v1 = value_residual<T>(__uint_as_float(vf[i][p] & 0xffff0000u), v1, mix);
            }
            const uint32_t vg = on ? pack2(v0 * vp, v1 * vp) : 0u;
            if (!on) { ar = 1.f; ai = 0.f; }
            if (kWa) {
                sr[head * kRow + t] = make_uint4(__float_as_uint(ar), __float_as_uint(ai), vg, bs);
            } else {
                sa[(p * kHg + head) * kRow + t] = make_float2(ar, ai);
                sv[(p * kHg + head) * kRow + t] = vg;
            }
        }
    }
    if (clears_ticket) *reinterpret_cast<volatile int*>(&old_ticket) = ticket;   // (it is back)
    __syncthreads();
    grid_launch_dependents();   // (not earlier: blocks that start while these fill the SMs are packed onto the few with room)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (kWa) {
#pragma unroll 1
        for (int h = warp; h < heads; h += kThreads / 32)
            a.rec[(((size_t)b * a.tiles + tile) * H + head0 + h) * kTokens + lane] = sr[h * kRow + lane];
    } else {
        const int c = kQuick ? l0 >> (a.C == 64 ? 6 : 7) : l0 / a.C, in_chunk = l0 - c * a.C;
        const size_t unit0 = ((size_t)b * a.NC + c) * H + head0;
        if constexpr (kNP >= 4) {   // a warp has a head and its pairs: no division an item
#pragma unroll 1
            for (int h = warp; h < heads; h += kThreads / 32) {
                const size_t o = ((unit0 + h) * NP + p0) * a.C + in_chunk + lane;
                const float2* fa = sa + h * kRow + lane;
                const uint32_t* fv = sv + h * kRow + lane;
#pragma unroll
                for (int p = 0; p < kNP; p++) {
                    if (p >= pairs) break;
                    a.rec_a[o + p * a.C] = fa[p * kHg * kRow];
                    a.rec_v[o + p * a.C] = fv[p * kHg * kRow];
                }
            }
        } else {                    // (12 layers of a 523-token prompt, two pairs a thread: 796 us, 823 in the other order)
            for (int i = warp; i < heads * pairs; i += kThreads / 32) {
                const int h = i / pairs, p = i - h * pairs, s = (p * kHg + h) * kRow + lane;
                const size_t o = ((unit0 + h) * NP + p0 + p) * a.C + in_chunk + lane;
                a.rec_a[o] = sa[s];
                a.rec_v[o] = sv[s];
            }
        }
        for (int h = warp; h < heads && p0 == 0; h += kThreads / 32) a.rec_g[(unit0 + h) * a.C + in_chunk + lane] = sg[h * kRow + lane];
    }
}

template <int kNP, int kHg, bool kWa, bool kResidual> struct KernelTag {};
template <int kNP, int kHg, bool kWa, bool kResidual>
static int launch(const Args& a, cudaStream_t st) {
    const size_t smem = kWa ? (size_t)kHg * (kTokens + 1) * 16 : (size_t)kHg * (kTokens + 1) * (kNP * 12 + 4);
    if (smem > 48 * 1024)
        if (int rc = allow_smem<KernelTag<kNP, kHg, kWa, kResidual>>((const void*)records_kernel<kNP, kHg, kWa, kResidual>, smem)) return rc;
    return launch_overlapped(records_kernel<kNP, kHg, kWa, kResidual>,
                             dim3((unsigned)(a.B * a.tiles), (a.H + kHg - 1) / kHg, kWa ? 1 : (a.N / 2 + kNP - 1) / kNP), dim3(kThreads),
                             smem, st, a);
}
// 16 heads fill the sectors of the gate rows; 8 where that leaves fewer lanes empty (24 heads) or more blocks are wanted.
template <int kNP, bool kWa>
static int launch_group(const Args& a, cudaStream_t st) {
    const bool eight = (a.H + 15) / 16 * 16 > (a.H + 7) / 8 * 8 || (long long)a.B * a.tiles * a.H < 148 * 64;
    if (a.v_first) return eight ? launch<kNP, 8, kWa, true>(a, st) : launch<kNP, 16, kWa, true>(a, st);
    return eight ? launch<kNP, 8, kWa, false>(a, st) : launch<kNP, 16, kWa, false>(a, st);
}

}  // namespace records

// Bytes of the records: transition and scaled v per pair, beta and sel_C (both layouts).
size_t scan_record_bytes(int B, int L, int H, int N, int C) {
    return (size_t)B * (((size_t)L + C - 1) / C) * H * C * ((size_t)(N / 2) * 12 + 4);
}

// The three arrays of the layout of scan_tile.cu inside the record buffer.
void scan_record_arrays(void* rec, int B, int L, int H, int N, int C, float2** a, uint32_t** v, uint32_t** g) {
    const size_t n = (size_t)B * (((size_t)L + C - 1) / C) * H * C;
    *a = static_cast<float2*>(rec);
    *v = reinterpret_cast<uint32_t*>(*a + n * (N / 2));
    *g = *v + n * (N / 2);
}

// Fills the records every pass over the same inputs reads.  wa: the layout of scan_wa.cu (N = 2), else of scan_tile.cu.
int scan_records(bool wa, const void* v, long long v_rs, const void* v_first, long long vf_rs, const void* mix,
                 const void* gate_raw, long long g_rs, const float* log_dt_scale, const float* rope_freqs, void* rec,
                 int* clear, size_t clear_words, int* clear2, size_t clear2_words, const DynConsts& dc, int B, int L, int H, int N, int C, int pos0, int segs,
                 int fp32_decay, cudaStream_t st) {
    using namespace records;
    Args a;
    a.v = static_cast<const __nv_bfloat16*>(v);
    a.gate_raw = static_cast<const __nv_bfloat16*>(gate_raw);
    a.log_dt_scale = log_dt_scale; a.rope_freqs = rope_freqs;
    a.rec = static_cast<uint4*>(rec);
    scan_record_arrays(rec, B, L, H, N, C, &a.rec_a, &a.rec_v, &a.rec_g);
    a.v_first = static_cast<const __nv_bfloat16*>(v_first); a.mix = static_cast<const __nv_bfloat16*>(mix);
    a.v_rs = v_rs; a.vf_rs = vf_rs; a.g_rs = g_rs;
    a.clear = clear; a.clear_words = clear_words;
    a.clear2 = clear2; a.clear2_words = clear2_words;
    a.dc = dc;
    a.B = B; a.L = L; a.H = H; a.N = N; a.C = C; a.NC = (L + C - 1) / C; a.pos0 = pos0; a.segs = segs; a.fp32_decay = fp32_decay;
    a.tiles = a.NC * (C / kTokens);
    a.tiles_inv = (uint32_t)(((1ull << 32) + a.tiles - 1) / a.tiles);
    if ((long long)B * a.tiles > 0x7fffffff || H > 8 * 65535) return CDSSM_ERR_UNSUPPORTED;
    if (wa) return launch_group<1, true>(a, st);
    if (N <= 2) return launch_group<1, false>(a, st);
    // Short inputs: one pair per thread up to two blocks per SM, two up to four; each computes what the pairs share.  us of a
    // whole scan call, 24 heads, N 16, one / two / all pairs per thread: 128 tokens 17.4 / 17.7 / 20.9, 523 30.6 / 31.4 / 32.5,
    // 1046 37.2 / 37.3 / 40.4, 2092 61.1 / 59.0 / 61.0, 4 x 2092 227 / 214 / 203.
    const long long blocks = (long long)B * a.tiles * ((H + 7) / 8);
    if (blocks * (N / 2) <= 296) return launch_group<1, false>(a, st);
    if (N > 4 && blocks * ((N / 2 + 1) / 2) <= 592) return launch_group<2, false>(a, st);
    if (N <= 4) return launch_group<2, false>(a, st);
    if (N <= 8) return launch_group<4, false>(a, st);
    return launch_group<8, false>(a, st);
}

}  // namespace cdssm
