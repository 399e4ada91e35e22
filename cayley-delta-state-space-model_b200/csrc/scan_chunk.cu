// The scan on tensor cores: bf16 storage, head_dim D = chunk C in {64, 128}, any even state_dim 2 < N <= 16, any
// head count.
//
// One thread block owns one chunk of one head; a warp (head_dim 64 and N > 4: two warps, half of the pairs each) its 32-token
// block.  With g_t the coefficient that the step at
// token t adds along k_t (raw keys; n_t = 1/|k_t|, c_t = beta_t n_t^2, W_t = a_0 ... a_t),
//     local state     z_t = W_t sum_{i<=t} (g_i / W_i) k_i,   g_t = beta_t n_t v_t - c_t W_t sum_{i<t} (g_i / W_i) G[t,i]
//     correction      r_t = W_t (r_0 - sum_{i<=t} h_i k_i),   h_t = c_t (k_t.r_0) - c_t sum_{i<t} h_i G[t,i]
//     read-out        y_t ~ W_t sum_{i<=t} (g_i / W_i) P[t,i]  +  W_{t-1} (q_t.r_0 - sum_{i<t} h_i P[t,i])
// with G = K K^T, P = Q K^T.  In the scaled unknowns g_i / W_i and h_i both systems have the same REAL unit lower
// triangular matrix I + M, M[t,i] = c_t G[t,i], for every complex pair of the head: the pairs are right-hand sides.  So
//   - G and P are products of the chunk's tiles (mma.sync on ldmatrix fragments of the swizzled TMA tiles, lower triangle
//     only), computed once per head and chunk whatever N is;
//   - the two 16 x 16 diagonal blocks of 32 tokens are inverted by substitution, a row per lane, all rows at once and
//     independent of any state (as 8 x 8 halves: seven dependent steps instead of fifteen);
//   - what is left of the serial chain is three 16-wide products per 32 tokens, passed from warp to warp;
//   - everything with a right-hand side (cross-block terms, read-outs, K^T g, K r_0, Q r_0) is a product with n = 8
//     columns {pair 2q: re p1, re p2, im p1, im p2, pair 2q+1: ...} and a second set for p3: a float32 value enters as the
//     exact sum of three bf16 parts, on the matrix side too; terms below 2^-24 are left out, accumulation is fp32.
// So the state is as precise as that of a walk in float32 (one chunk: 1.4e-7 of it, the walk 1.1e-7; two parts, 16 bits, left
// 1.7e-5).  Bounded by issue slots and the latency of its dependent steps at 16 warps per SM (registers); a tensor-core
// generation with tiles of 128 rows has no use for 16-wide products.  Measured on B200, D 64, N 16, B 8, H 24, 6144 chunks, the
// whole call: 279 us, 183 with two parts, the walk 540; 216 chunks: 32 us, 26 with two parts, the walk 55.
// The division by W_i only spans a 32-token block, relative to its middle (|W ratio| of 16 tokens >= 1e-30); values cross
// blocks relative to the block ends, where all factors are plain products.  A (block, pair) that decays further is walked
// step by step (slow_walk).
//
// The reference's carry s_{c+1} = gamma_c s_c + z_{C-1} (inter_chunk_scan.cu:73-83) is handed from block to block inside
// the kernel: blocks take (chunk, batch, head) work in chunk-major order from a ticket counter, so the chunk a block waits
// for is held by a block that started before it.  kLocal / kOutput are the two halves with the carry pass of scan_simt.cu
// between them (summaries, and shapes whose chain of chunks is longer than their work: one_kernel_pays() there).
//
// Reference semantics (intra_chunk_scan.cu:100-195, exact_correction.cu:89-150): z starts at zero at the chunk start, r
// from the bf16-rounded carry, the correction is read before its step.
#include "cdssm_common.cuh"
#include "sm100_ptx.cuh"
#include "tile_map.cuh"

namespace cdssm {
using namespace sm100;

namespace chunk {

enum Mode { kLocal, kOutput, kFused };

struct Args {
    const float2* rec_a;         // (B,NC,H,NP,C): transition a_t
    const uint32_t* rec_v;       // (B,NC,H,NP,C): vp-scaled v_t, bf16 pair
    const uint32_t* rec_g;       // (B,NC,H,C): beta_t, sel_C, bf16 pair
    const float* h0;
    __nv_bfloat16* y;
    float *final_state, *tail_state;
    float* ws_gamma;             // (B,NC,H,NP,2): chunk decays (kLocal); kFused: first word of a unit = "carry is there"
    float* ws_state;             // (B,NC,H,NP,2,D): z_{C-1} (kLocal), carry into the chunk (kOutput: rounded, kFused: not)
    int *status, *ticket;
    unsigned long long wait_ns;  // limit of every device-side wait
    int withhold;                // test hook: nothing is loaded, so the first wait runs out
    float shortcut_scale;
    int from_chunks;             // kOutput: the carry from the local results of the chunks before (no carry pass has run)
    int B, L, H, N, NC;
    int groups;                  // blocks that share a chunk of a head: kPairs pairs each
};

#define kNotANumber __int_as_float(0x7fffffff)

struct cplx { float r, i; };
__device__ __forceinline__ cplx cmul(cplx a, cplx b) { return {a.r * b.r - a.i * b.i, a.r * b.i + a.i * b.r}; }
__device__ __forceinline__ cplx cshfl(cplx v, int src) {
    return {__shfl_sync(0xffffffffu, v.r, src), __shfl_sync(0xffffffffu, v.i, src)};
}
__device__ __forceinline__ float bfr(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// x = p1 + p2 + p3, each part the next eight significant bits cut off as a bf16: exact, a float has 24.  Integer and FMA pipes
// only.  pair_hi: the first parts of two values; rest: what is left behind the first part.
__device__ __forceinline__ uint32_t pair_hi(float x0, float x1) { return __byte_perm(__float_as_uint(x0), __float_as_uint(x1), 0x7632); }
__device__ __forceinline__ float rest(float x) { return x - __uint_as_float(__float_as_uint(x) & 0xffff0000u); }
__device__ __forceinline__ uint32_t movmatrix(uint32_t x) {   // 8 x 8 bf16 matrix, one row a quad, transposed
    uint32_t y;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
    return y;
}
__device__ __forceinline__ float bits_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ float bits_lo(uint32_t w) { return __uint_as_float(w << 16); }

// A 16 x 16 operand in float32, in the order of two 16 x 8 accumulators, and as A fragments of its three bf16 parts.
struct Frag { float x[8]; };
__device__ __forceinline__ Frag frag_of(const float (&n0)[4], const float (&n1)[4]) {
    return {{n0[0], n0[1], n0[2], n0[3], n1[0], n1[1], n1[2], n1[3]}};
}
struct Split { uint32_t p1[4], p2[4], p3[4]; };
__device__ __forceinline__ Split split(const Frag& f) {
    Split s;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float r0 = rest(f.x[2 * i]), r1 = rest(f.x[2 * i + 1]);
        s.p1[i] = pair_hi(f.x[2 * i], f.x[2 * i + 1]);
        s.p2[i] = pair_hi(r0, r1);
        s.p3[i] = pair_hi(rest(r0), rest(r1));
    }
    return s;
}
// B fragments of 16 tokens: ab has columns {p1, p2} of the tile's components, c {p3, 0}.
struct Rhs { uint2 ab, c; };
// values of rows g, g + 8 (this lane's complex component)
__device__ __forceinline__ Rhs rhs_frag(float x0, float x1) {
    const float r0 = rest(x0), r1 = rest(x1);
    return {make_uint2(movmatrix(pair_hi(x0, r0)), movmatrix(pair_hi(x1, r1))),
            make_uint2(movmatrix(pair_hi(rest(r0), 0.f)), movmatrix(pair_hi(rest(r1), 0.f)))};
}
// d (+ e) += s f up to 2^-24 of a term; d holds the large terms, e the small ones (may be the same accumulator)
__device__ __forceinline__ void mma_split(float (&d)[4], float (&e)[4], const Split& s, const Rhs& f) {
    mma_bf16_m16n8k16(e, s.p3, f.ab.x, f.ab.y);
    mma_bf16_m16n8k16(e, s.p1, f.c.x, f.c.y);
    mma_bf16_m16n8k16(d, s.p2, f.ab.x, f.ab.y);
    mma_bf16_m16n8k16(d, s.p1, f.ab.x, f.ab.y);
}

template <int kD, int kPairs_>
struct Geo {
    static constexpr int kPairs = kPairs_;               // complex pairs held (>= N / 2)
    static constexpr int kTiles = (kPairs + 1) / 2;      // column tiles of two pairs
    static constexpr int kBlocks = kD / 32;              // warps: one per 32-token block
    static constexpr int kSplit = kD == 64 && kPairs >= 4 ? 2 : 1;   // warps that share the column tiles of a 32-token block
    static constexpr int kThreads = 32 * kBlocks * kSplit;
    static constexpr int kOwn = kTiles / kSplit, kOwnPairs = kPairs / kSplit;   // of a warp
    static constexpr int kSlabs = kD / 64, kKs = kD / 16;
    static constexpr uint32_t kSlab = kD * 128;          // bytes of kD rows x 64 bf16 columns
    static constexpr uint32_t kTile = kSlabs * kSlab;
    // right-hand-side fragments of a 32-token block, published for others: g for every later block (rotated to its
    // start) and for the chunk end, h for every later block and itself
    static constexpr int kCross = kBlocks * (kBlocks - 1) / 2;
    static constexpr int kSlots = kCross + 2 * kBlocks;
    static __device__ __forceinline__ int slot_g(int from, int to) { return to * (to - 1) / 2 + from; }
    static __device__ __forceinline__ int slot_end(int from) { return kCross + from; }
    static __device__ __forceinline__ int slot_h(int from) { return kCross + kBlocks + from; }
};

struct BlockPair {   // of one 32-token block and pair
    cplx A, R, D31;  // product of a over the block; product of its first half (the scaling's reference); D of the last token
};

struct Scratch {   // of one 32-token block, until the Q tile arrives in its place
    union {
        struct {                                         // of the two 16 x 16 diagonal blocks of M, 8 x 8 each
            float tri[4][100];                           // [block, half] diagonal ones: column j, row i at 12 j + i
            float low[2][68], inv[2][68];                // [block] the one below, the first half's inverse: 8 i + j
        };
        float t[32][20];                                 // rows of the inverses
    };
    float4 m21[2][32];                                   // for the block's other warp: M between its halves, |k|^-1
    float nrm[32];
};

// (head_dim 128 with one pair: 74.2 KB, three blocks per SM)
template <int kD, int kPairs, Mode kMode>
struct __align__(1024) Smem {
    using G = Geo<kD, kPairs>;
    uint8_t k[G::kTile];                                 // swizzled rows = tokens
    union {
        uint8_t q[kMode == kLocal ? 1024 : G::kTile];
        Scratch scr[G::kBlocks];
    };
    float frag[G::kSlots][G::kTiles][2][64];             // [slot][tile][16-token half][component, token]
    float2 viw[kPairs][kD], dd[kPairs][kD];              // v / D, D
    float beta[kD], sel[kD];
    BlockPair bp[kPairs][G::kBlocks];
    float s_in[2 * kPairs][kD];                          // carry into the chunk
    __nv_bfloat16 r0[2 * kPairs][kD + 8];                // the same rounded (padded rows: fragment loads hit distinct banks)
    float4 walk[G::kBlocks * G::kSplit][32];             // slow_walk results
    // outputs of a warp on their way to one row a lane, in place of the carry (in bf16 by then)
    __device__ __forceinline__ __nv_bfloat16* y(int token) {
        return reinterpret_cast<__nv_bfloat16*>(s_in) + token * (2 * kPairs + 2);
    }
    uint64_t full_k, full_q;
    int slow[G::kBlocks];                                // pairs that are walked step by step, a bit each
    int abort_flag, item, stop;
    int first_bad;                                       // first token whose key or beta is no number, kD if there is none
    // (the tokens of components 2 and 3 are turned by eight: a store's lanes then hit distinct banks)
    static __device__ __forceinline__ int at(int comp, int token) { return comp * 16 + (token ^ ((comp >> 1) * 8)); }
    // values of tokens g, g + 8 of a half, this lane's component
    __device__ __forceinline__ void put(int slot, int tile, int half, int lane, float x0, float x1) {
        const int g = lane >> 2, comp = lane & 3;
        frag[slot][tile][half][at(comp, g)] = x0;
        frag[slot][tile][half][at(comp, g + 8)] = x1;
    }
    __device__ __forceinline__ Rhs get(int slot, int tile, int half, int lane) const {
        const int g = lane >> 2, comp = g >> 1, token = 2 * (lane & 3);
        const float2 x0 = *reinterpret_cast<const float2*>(&frag[slot][tile][half][at(comp, token)]);
        const float2 x1 = *reinterpret_cast<const float2*>(&frag[slot][tile][half][at(comp, token + 8)]);
        const float2 r0 = make_float2(rest(x0.x), rest(x0.y)), r1 = make_float2(rest(x1.x), rest(x1.y));
        if (g & 1) return {make_uint2(pair_hi(r0.x, r0.y), pair_hi(r1.x, r1.y)), make_uint2(0u, 0u)};
        return {make_uint2(pair_hi(x0.x, x0.y), pair_hi(x1.x, x1.y)),
                make_uint2(pair_hi(rest(r0.x), rest(r0.y)), pair_hi(rest(r1.x), rest(r1.y)))};
    }
};

// ---- fragments ------------------------------------------------------------------------------------------------
// A (16 tokens x 16 columns, row-major) or, with registers {0,2} / {1,3}, two B fragments (8 tokens each)
template <uint32_t kSlab>
__device__ __forceinline__ uint32_t row_frag(uint32_t tile, int row0, int ks, int lane) {
    const int row = row0 + (lane & 7) + ((lane >> 3) & 1) * 8, piece = (ks & 3) * 2 + (lane >> 4);
    return tile + (uint32_t)(ks >> 2) * kSlab + (uint32_t)row * 128u + (uint32_t)((piece ^ (row & 7)) << 4);
}
// A fragment of the transposed tile: 16 columns x 16 tokens (for ldmatrix.trans)
template <uint32_t kSlab>
__device__ __forceinline__ uint32_t col_frag(uint32_t tile, int tok0, int col0, int lane) {
    const int row = tok0 + (lane & 7) + ((lane >> 4) & 1) * 8, piece = ((col0 & 63) >> 3) + ((lane >> 3) & 1);
    return tile + (uint32_t)(col0 >> 6) * kSlab + (uint32_t)row * 128u + (uint32_t)((piece ^ (row & 7)) << 4);
}

// acc[mt][nt] = rows row_a + 16 mt .. of tile A against rows row_b + 8 nt .. of tile B, 32 x 32
template <int kD, int kPairs, bool kSame>
__device__ __forceinline__ void gram_block(float (&acc)[2][4][4], uint32_t ta, int row_a, uint32_t tb, int row_b, int lane,
                                           bool diagonal) {
    using G = Geo<kD, kPairs>;
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int n = 0; n < 4; n++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[m][n][e] = 0.f;
#pragma unroll
    for (int ks = 0; ks < G::kKs; ks++) {
        uint32_t a[2][4], b[2][4];
        ldsm_x4(row_frag<G::kSlab>(ta, row_a, ks, lane), a[0]);
        ldsm_x4(row_frag<G::kSlab>(ta, row_a + 16, ks, lane), a[1]);
        if (!kSame) {
            ldsm_x4(row_frag<G::kSlab>(tb, row_b, ks, lane), b[0]);
            ldsm_x4(row_frag<G::kSlab>(tb, row_b + 16, ks, lane), b[1]);
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t(&bb)[4] = kSame ? a[h] : b[h];
#pragma unroll
            for (int m = 0; m < 2; m++) {
                if (m == 0 && h == 1 && diagonal) continue;   // above the diagonal
                mma_bf16_m16n8k16(acc[m][2 * h], a[m], bb[0], bb[2]);
                mma_bf16_m16n8k16(acc[m][2 * h + 1], a[m], bb[1], bb[3]);
            }
        }
    }
}

// Diagonal elements of a 16 x 16 block held as two 16 x 8 accumulators: rows g and g + 8, handed to the whole quad.
__device__ __forceinline__ void diagonal_of(const float (&n0)[4], const float (&n1)[4], int lane, float& d0, float& d1) {
    const int g = lane >> 2, src = (lane & ~3) | (g >> 1);
    const float x0 = (g & 1) ? n0[1] : n0[0], x1 = (g & 1) ? n1[3] : n1[2];
    d0 = __shfl_sync(0xffffffffu, x0, src);
    d1 = __shfl_sync(0xffffffffu, x1, src);
}

// ---- decay scalings of a 32-token block and pair (lane = token) ---------------------------------------------------
// The scaled unknowns need ratios of the prefix products W_t = a_0 ... a_t only, taken relative to the middle of the
// block, D_t = W_t / W_15: lanes 0-15 hold the suffix product a_{t+1} ... a_15 = 1 / D_t, lanes 16-31 the prefix product
// a_16 ... a_t = D_t, and neither half leaves the float range unless one half alone decays by more than 1e-30.
// kW pairs side by side: one alone waits for its shuffles.  at, vg: a_t, v_t in; D, v_t / D out (a and v of a pair outside the
// range: the walk reads them themselves).  Returns the pairs outside the range, a bit each.
template <int kW>
__device__ __forceinline__ int scalings(cplx (&at)[kW], cplx (&vg)[kW], int tl, BlockPair (&bp)[kW]) {
    const bool lo = tl < 16;
    cplx X[kW];
#pragma unroll
    for (int w = 0; w < kW; w++) X[w] = at[w];
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
        const bool on = lo ? (tl + o < 16) : (tl - o >= 16);
#pragma unroll
        for (int w = 0; w < kW; w++) {
            const cplx other = cshfl(X[w], lo ? tl + o : tl - o);
            if (on) X[w] = cmul(X[w], other);
        }
    }
    int slow = 0;
#pragma unroll
    for (int w = 0; w < kW; w++) {
        const cplx R = cshfl(X[w], 0);           // a_0 ... a_15
        cplx E = cshfl(X[w], tl + 1);            // first half: exclusive suffix = inclusive suffix of lane t + 1
        if (tl == 15) E = {1.f, 0.f};
        if (!lo) E = X[w];
        const float m = fmaxf(fabsf(E.r), fabsf(E.i));
        const float sc1 = __frcp_rn(m);
        const cplx En = {E.r * sc1, E.i * sc1};
        const float q = sc1 * __frcp_rn(En.r * En.r + En.i * En.i);
        const cplx Einv = {En.r * q, -En.i * q};
        const cplx D = lo ? Einv : E, v = cmul(vg[w], lo ? E : Einv);
        const bool in_range = m >= 1e-30f && m <= 1e30f && fabsf(v.r) <= 1e33f && fabsf(v.i) <= 1e33f;   // (false for NaN)
        const cplx D31 = cshfl(D, 31);
        const float mr = fmaxf(fabsf(R.r), fabsf(R.i));
        const bool fast = __all_sync(0xffffffffu, in_range && mr >= 1e-30f && mr <= 1e30f);
        bp[w].A = cmul(D31, R);                  // both factors are plain products of a: valid for any a
        bp[w].R = fast ? R : cplx{1.f, 0.f};
        bp[w].D31 = fast ? D31 : cplx{1.f, 0.f};
        if (!fast) slow |= 1 << w;
        at[w] = fast ? D : at[w];
        vg[w] = fast ? v : vg[w];
    }
    return slow;
}

// Step-by-step walk of pair p over this warp's block, for decays the scaled form cannot hold: state columns over the
// lanes.  First without read-out (walk[t].x = |k_t|^-1 in; out walk[t] = {g_t carried to the block end}, and g_t in place of
// v_t), later with it (walk[t] = {q_t.z_t, W_{t-1} from the block start}; no sums on the way of the state any more).  The
// incoming state is rebuilt from the fragments the earlier blocks published for this one.
template <int kD, int kPairs, Mode kMode, bool kReadout>
__device__ __noinline__ void slow_walk(Smem<kD, kPairs, kMode>& sm, int p, int I, int W, int tl) {
    using G = Geo<kD, kPairs>;
    constexpr int kCols = kD / 32;
    auto column = [&](const uint8_t* tile, int row, int c) {
        const int piece = (c & 63) >> 3;
        const __nv_bfloat16* x = reinterpret_cast<const __nv_bfloat16*>(tile + (c >> 6) * G::kSlab + row * 128 + ((piece ^ (row & 7)) << 4));
        return __bfloat162float(x[c & 7]);
    };
    float zr[kCols], zi[kCols];
#pragma unroll
    for (int i = 0; i < kCols; i++) zr[i] = zi[i] = 0.f;
    for (int J = 0; J < I; J++)
#pragma unroll 4
        for (int t = 0; t < 32; t++) {
            const float* f = sm.frag[G::slot_g(J, I)][p >> 1][t >> 4];
            const int comp = 2 * (p & 1);
            const float wr = f[sm.at(comp, t & 15)], wi = f[sm.at(comp + 1, t & 15)];
#pragma unroll
            for (int i = 0; i < kCols; i++) {
                const float k = column(sm.k, 32 * J + t, tl + 32 * i);
                zr[i] += wr * k;
                zi[i] += wi * k;
            }
        }
    cplx own = {0.f, 0.f};
#pragma unroll 2
    for (int t = 0; t < 32; t++) {
        const int row = 32 * I + t;
        const float2 a = sm.dd[p][row], vg = sm.viw[p][row];
        float k[kCols];
#pragma unroll
        for (int i = 0; i < kCols; i++) k[i] = column(sm.k, row, tl + 32 * i);
        cplx gt = {vg.x, vg.y};               // read-out: g_t as the first walk left it
        if (!kReadout) {
            const float be = sm.beta[row], n = sm.walk[W][t].x;
            float ur = 0.f, ui = 0.f;
#pragma unroll
            for (int i = 0; i < kCols; i++) {
                ur += zr[i] * k[i];
                ui += zi[i] * k[i];
            }
            ur = warp_sum(ur); ui = warp_sum(ui);
            const cplx au = cmul({a.x, a.y}, {n * ur, n * ui});
            gt = {be * n * (vg.x - au.r), be * n * (vg.y - au.i)};
            if (tl == t) own = gt;
        }
#pragma unroll
        for (int i = 0; i < kCols; i++) {
            const cplx z = cmul({a.x, a.y}, {zr[i], zi[i]});
            zr[i] = z.r + gt.r * k[i];
            zi[i] = z.i + gt.i * k[i];
        }
        if (kReadout) {
            float yr = 0.f, yi = 0.f;
#pragma unroll
            for (int i = 0; i < kCols; i++) {
                const float q = column(sm.q, row, tl + 32 * i);
                yr += zr[i] * q;
                yi += zi[i] * q;
            }
            yr = warp_sum(yr); yi = warp_sum(yi);
            if (tl == t) own = {yr, yi};
        }
    }
    __syncwarp();
    if (!kReadout) sm.viw[p][32 * I + tl] = make_float2(own.r, own.i);
    // g carried to the block end: times a_{t+1} ... a_31; W_{t-1} = a_0 ... a_{t-1}
    const float2 a = sm.dd[p][32 * I + tl];
    cplx S = {a.x, a.y};
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int from = kReadout ? tl - o : tl + o;
        const cplx other = cshfl(S, from);
        if (from >= 0 && from < 32) S = cmul(S, other);
    }
    cplx V = cshfl(S, kReadout ? tl - 1 : tl + 1);
    if (tl == (kReadout ? 0 : 31)) V = {1.f, 0.f};
    if (!kReadout) own = cmul(V, own);
    __syncwarp();
    sm.walk[W][tl] = make_float4(own.r, own.i, V.r, V.i);
    __syncwarp();
}

// s <- gamma s + l in the order in which the carry pass (scan_simt.cu) evaluates it, so that the two ways to hand the carry on
// give the same bits: chunk-aligned pieces of a sequence compose exactly whichever of them their lengths choose.
__device__ __forceinline__ float next_re(cplx g, float sr, float si, float l) {
    return __fadd_rn(__fmaf_rn(g.r, sr, -__fmul_rn(g.i, si)), l);
}
__device__ __forceinline__ float next_im(cplx g, float sr, float si, float l) {
    return __fadd_rn(__fmaf_rn(g.r, si, __fmul_rn(g.i, sr)), l);
}

// resident blocks per SM the registers are cut for (N 16, head_dim 64, 4 / 3 blocks: 285 / 284 us with 6144 chunks, 111 / 119
// with 1692, where a chain of chunks waits)
template <int kD, int kPairs>
constexpr int kMinBlocks = kD == 128 ? 2 : (kPairs == 2 ? 6 : 4);

// A key row or a beta that is infinite or no number makes the state no number from its token on, whatever the pair.  In the
// products of a block it would reach the tokens before it too (0 x NaN), so its row is emptied and the outputs from it on are set
// apart at the end.  A finite row whose square overflows has |k|^-1 = 0: it neither erases nor adds.
template <int kD, int kPairs, Mode kMode>
__device__ __noinline__ void empty_bad_rows(Smem<kD, kPairs, kMode>& sm, int I, int tl) {
    using G = Geo<kD, kPairs>;
    const int row = 32 * I + tl;
    bool number = fabsf(sm.beta[row]) <= 3e38f;
    float ss = 0.f;
    for (int c = 0; c < kD; c++) {
        const float k = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(sm.k + (c >> 6) * G::kSlab + row * 128)[c & 63]);
        number = number && fabsf(k) <= 3.4e38f;
        ss += k * k;
    }
    if (!number) atomicMin(&sm.first_bad, row);
    if (!number || !(ss <= 3.4e38f)) {
        for (int s = 0; s < G::kSlabs; s++)
            for (int i = 0; i < 8; i++) *reinterpret_cast<uint4*>(sm.k + s * G::kSlab + row * 128 + 16 * i) = make_uint4(0u, 0u, 0u, 0u);
        sm.beta[row] = 0.f;
    }
    __syncwarp();
}

template <int kD, int kPairs, Mode kMode>
__global__ void __launch_bounds__(Geo<kD, kPairs>::kThreads, kMinBlocks<kD, kPairs>)
scan_chunk_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmQ, const Args a) {
    using G = Geo<kD, kPairs>;
    constexpr int kBlocks = G::kBlocks, kKs = G::kKs;
    constexpr bool kOut = kMode != kLocal, kNeedEnd = kMode != kOutput;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    Smem<kD, kPairs, kMode>& sm = *reinterpret_cast<Smem<kD, kPairs, kMode>*>(smem_raw);
    constexpr int kSplit = G::kSplit, kOwn = G::kOwn;
    // warp W: 32-token block I, column tiles S * kOwn ... (the warps of a block meet at the tiles and the inverses only)
    const int tid = threadIdx.x, W = tid >> 5, I = W % kBlocks, S = W / kBlocks, tl = tid & 31, g = tl >> 2, t4 = tl & 3;
    const int tok = 32 * I + tl;
    const int H = a.H, N = a.N, NP = N >> 1, L = a.L;

    if (kMode == kFused) grid_dependency_wait();   // (the records kernel clears the ticket counter)
    if (tid == 0) {
        mbar_init(&sm.full_k, 1);
        mbar_init(&sm.full_q, 1);
        sm.abort_flag = 0;
        sm.first_bad = kD;
        fence_barrier_init();
        sm.item = kMode == kFused ? atomicAdd(a.ticket, 1) : (int)blockIdx.x;
        sm.stop = kMode == kFused ? *reinterpret_cast<volatile int*>(a.status) : 0;
    }
    __syncthreads();
    if ((smem_u32(smem_raw) & 1023u) != 0) {   // the swizzled tiles need 1024-byte alignment
        if (tid == 0) atomicCAS(a.status, 0, 399);
        return;
    }
    if (sm.stop) return;   // an earlier block gave up
    // chunk-major: every block that a block may wait for has an earlier ticket
    const int group = kD == 128 ? sm.item % a.groups : 0, item = kD == 128 ? sm.item / a.groups : sm.item;
    const int hd = item % H, b = (item / H) % a.B, c = item / (H * a.B);
    const int pair0 = group * kPairs, NPB = min(kPairs, NP - pair0);   // the block's pairs
    const size_t unit = ((size_t)b * a.NC + c) * H + hd;       // workspace slot
    const int Lc = min(kD, L - c * kD);
    if (tid == 0 && !a.withhold) {
        mbar_arrive_expect_tx(&sm.full_k, G::kTile);
#pragma unroll
        for (int s = 0; s < G::kSlabs; s++) tma_load_4d(sm.k + s * G::kSlab, &tmK, &sm.full_k, 64 * s, hd, c * kD, b);
    }

    // a block that gives up stays until its own copy has landed (or a limit has passed again): the next one has its memory then
    auto drain = [&](uint64_t* bar) {
        volatile int never = 0;
        if (tid == 0 && !a.withhold) mbar_wait_ns(bar, 0, &never, a.wait_ns);
    };
    // ---- carry into the chunk: this warp's 32 columns of its state rows.  Early if its producer is done, else polled for
    // behind the products that do not need it (kOutput: the previous pass is waited for there).
    const float* carry_src = a.ws_state + (unit * (size_t)N + 2 * pair0) * kD;
    const int flag_bit = G::kBlocks * kSplit * group + W;
    int* carry_flag = reinterpret_cast<int*>(a.ws_gamma + unit * (size_t)N);   // a bit per warp
    auto flag_set = [&]() {
        int v;
        asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(carry_flag) : "memory");
        return ((v >> flag_bit) & 1) != 0;
    };
    auto load_carry = [&](const float* src) {
        const int col = 32 * I + 4 * (tl & 7);
#pragma unroll
        for (int n0 = 0; n0 < 2 * G::kOwnPairs; n0 += 4) {
            const int n = 2 * G::kOwnPairs * S + n0 + (tl >> 3);
            if (n0 + (tl >> 3) < 2 * G::kOwnPairs) {
                const bool on = src != nullptr && n < 2 * NPB;
                cp_async16(&sm.s_in[n][col], on ? src + (size_t)n * kD + col : a.ws_state, on);
            }
        }
        cp_async_commit();
    };
    bool have_carry = true;
    if (kMode == kFused) {
        if (c == 0) load_carry(a.h0 ? a.h0 + (((size_t)b * H + hd) * N + 2 * pair0) * kD : nullptr);
        else if ((have_carry = __all_sync(0xffffffffu, flag_set()))) load_carry(carry_src);
    }
    // the token's dynamics, parked where the results will go (padding pairs: identity)
    const bool first_warp = kSplit == 1 || S == 0, last_warp = kSplit == 1 || S == kSplit - 1;
    auto load_records = [&]() {
        if (first_warp) cp_async_small<4>(&sm.beta[tok], a.rec_g + unit * kD + tok);
        if (last_warp) {
            const float2* ra = a.rec_a + (unit * (size_t)NP + pair0) * kD + tok;
            const uint32_t* rv = a.rec_v + (unit * (size_t)NP + pair0) * kD + tok;
#pragma unroll
            for (int p = 0; p < kPairs; p++) {
                if (p < NPB) {
                    cp_async_small<8>(&sm.dd[p][tok], ra + p * kD);
                    cp_async_small<4>(&sm.viw[p][tok], rv + p * kD);
                } else {
                    sm.dd[p][tok] = make_float2(1.f, 0.f);
                    sm.viw[p][tok] = make_float2(0.f, 0.f);
                }
            }
        }
        cp_async_commit();
    };
    if (kMode != kLocal) load_records();
    const bool k_here = mbar_wait_suspend(&sm.full_k, 0, &sm.abort_flag, a.wait_ns);
    if (!__syncthreads_and(k_here)) {
        if (tid == 0) atomicCAS(a.status, 0, 201);
        cp_async_wait_all();
        drain(&sm.full_k);
        return;
    }
    const uint32_t kt = smem_u32(sm.k), qt = smem_u32(sm.q);

    // ---- G: diagonal block, |k|^-1, inverses
    float cc[4], bn[4], nrm[4];               // c_t, beta_t n_t, n_t of rows g, g + 8, g + 16, g + 24
    Frag T11, T22, M21;
    Frag M[kBlocks > 1 ? kBlocks - 1 : 1][2][2];
    {
        float acc[2][4][4], kk[4];
        if (first_warp) {
            gram_block<kD, kPairs, true>(acc, kt, 32 * I, kt, 32 * I, tl, true);
            diagonal_of(acc[0][0], acc[0][1], tl, kk[0], kk[1]);
            diagonal_of(acc[1][2], acc[1][3], tl, kk[2], kk[3]);
        }
        // the token's dynamics, from the kernel before this one (its launch let this one start early; no __ldg here: loads
        // that claim the data constant may be moved above the wait)
        if (kMode == kLocal) grid_dependency_wait();
        grid_launch_dependents();
        if (kMode == kLocal) load_records();
        cp_async_wait_all();
        if (first_warp) {
            const uint32_t gg = __float_as_uint(sm.beta[tok]);
            sm.beta[tok] = bits_lo(gg);
            sm.sel[tok] = bits_hi(gg);
            __syncwarp();
            bool number = fabsf(bits_lo(gg)) <= 3e38f;   // (false for NaN)
#pragma unroll
            for (int r = 0; r < 4; r++) number = number && kk[r] <= 3.4e38f;
            if (!__all_sync(0xffffffffu, number)) {
                empty_bad_rows<kD, kPairs, kMode>(sm, I, tl);
                gram_block<kD, kPairs, true>(acc, kt, 32 * I, kt, 32 * I, tl, true);
                diagonal_of(acc[0][0], acc[0][1], tl, kk[0], kk[1]);
                diagonal_of(acc[1][2], acc[1][3], tl, kk[2], kk[3]);
            }
        }
        if (last_warp) {
            constexpr int kW = kPairs < 4 ? kPairs : 4;
            int slow = 0;
#pragma unroll 1
            for (int p0 = 0; p0 < kPairs; p0 += kW) {
                cplx at[kW], vg[kW];
                BlockPair bp[kW];
#pragma unroll
                for (int w = 0; w < kW; w++) {
                    const float2 x = sm.dd[p0 + w][tok];
                    const uint32_t y = __float_as_uint(sm.viw[p0 + w][tok].x);
                    at[w] = {x.x, x.y};
                    vg[w] = {bits_lo(y), bits_hi(y)};
                }
                slow |= scalings<kW>(at, vg, tl, bp) << p0;
#pragma unroll
                for (int w = 0; w < kW; w++) {
                    sm.viw[p0 + w][tok] = make_float2(vg[w].r, vg[w].i);
                    sm.dd[p0 + w][tok] = make_float2(at[w].r, at[w].i);
                    if (tl == 0) sm.bp[p0 + w][I] = bp[w];
                }
            }
            if (tl == 0) sm.slow[I] = slow;
            __syncwarp();
        }
        if (first_warp) {
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const float be = sm.beta[32 * I + 8 * r + g];
                nrm[r] = rsqrtf(kk[r] + kEps);
                bn[r] = be * nrm[r];
                cc[r] = bn[r] * nrm[r];
            }
            // M's diagonal 16 x 16 blocks, as 8 x 8: the strictly lower part of two, and the one below
            auto& sc = sm.scr[I];
#pragma unroll
            for (int m = 0; m < 2; m++) {
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int col = 2 * t4 + e;
                    sc.tri[2 * m][12 * col + g] = g > col ? cc[2 * m] * acc[m][2 * m][e] : 0.f;
                    sc.tri[2 * m + 1][12 * col + g] = g > col ? cc[2 * m + 1] * acc[m][2 * m + 1][2 + e] : 0.f;
                }
                *reinterpret_cast<float2*>(&sc.low[m][8 * g + 2 * t4]) =
                    make_float2(cc[2 * m + 1] * acc[m][2 * m][2], cc[2 * m + 1] * acc[m][2 * m][3]);
            }
#pragma unroll
            for (int n = 0; n < 2; n++)
#pragma unroll
                for (int e = 0; e < 4; e++) acc[1][n][e] *= cc[2 + (e >> 1)];
            M21 = frag_of(acc[1][0], acc[1][1]);
            if (kSplit > 1) {
                sm.scr[I].m21[0][tl] = make_float4(M21.x[0], M21.x[1], M21.x[2], M21.x[3]);
                sm.scr[I].m21[1][tl] = make_float4(M21.x[4], M21.x[5], M21.x[6], M21.x[7]);
                if (t4 == 0) {
#pragma unroll
                    for (int r = 0; r < 4; r++) sm.scr[I].nrm[8 * r + g] = nrm[r];
                }
            }
            __syncwarp();
            // A lane has a row of the inverse.  The halves first, T[r][j] = - sum_{i>j} T[r][i] M[i][j]: seven dependent steps
            // instead of the fifteen of the whole block; then the lower rows' left part, - T_2 M_21 T_1.
            const int r = tl & 7, half = (tl >> 3) & 1, blk = tl >> 4;
            float2 T2[4], U[4], X[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                T2[j] = make_float2(2 * j == r ? 1.f : 0.f, 2 * j + 1 == r ? 1.f : 0.f);
                U[j] = X[j] = make_float2(0.f, 0.f);
            }
            const float* tri = sc.tri[2 * blk + half];
#pragma unroll
            for (int j = 6; j >= 0; j--) {
                float2 sum = make_float2(0.f, 0.f);
                const float4 m1 = *reinterpret_cast<const float4*>(tri + 12 * j + 4);
                if (j < 6) sum = __ffma2_rn(T2[3], make_float2(m1.z, m1.w), sum);
                else sum.y = T2[3].y * m1.w;
                if (j < 5) sum = __ffma2_rn(T2[2], make_float2(m1.x, m1.y), sum);
                if (j < 3) {
                    const float4 m0 = *reinterpret_cast<const float4*>(tri + 12 * j);
                    sum = __ffma2_rn(T2[1], make_float2(m0.z, m0.w), sum);
                    if (j < 1) sum = __ffma2_rn(T2[0], make_float2(m0.x, m0.y), sum);
                }
                if (j & 1) T2[j >> 1].y -= sum.x + sum.y;
                else T2[j >> 1].x -= sum.x + sum.y;
            }
            if (half == 0) {
                float4* inv = reinterpret_cast<float4*>(&sc.inv[blk][8 * r]);
                inv[0] = make_float4(T2[0].x, T2[0].y, T2[1].x, T2[1].y);
                inv[1] = make_float4(T2[2].x, T2[2].y, T2[3].x, T2[3].y);
            }
            auto add_rows = [&](float2 (&to)[4], const float2 (&by)[4], const float* rows) {   // to += by . rows (8 x 8)
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float4 r0 = *reinterpret_cast<const float4*>(rows + 8 * i), r1 = *reinterpret_cast<const float4*>(rows + 8 * i + 4);
                    const float f = (i & 1) ? by[i >> 1].y : by[i >> 1].x;
                    const float2 ff = make_float2(f, f);
                    to[0] = __ffma2_rn(ff, make_float2(r0.x, r0.y), to[0]);
                    to[1] = __ffma2_rn(ff, make_float2(r0.z, r0.w), to[1]);
                    to[2] = __ffma2_rn(ff, make_float2(r1.x, r1.y), to[2]);
                    to[3] = __ffma2_rn(ff, make_float2(r1.z, r1.w), to[3]);
                }
            };
            add_rows(U, T2, sc.low[blk]);
            __syncwarp();
            add_rows(X, U, sc.inv[blk]);
            float2 R[8];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                R[j] = half == 0 ? T2[j] : make_float2(-X[j].x, -X[j].y);
                R[4 + j] = half == 0 ? make_float2(0.f, 0.f) : T2[j];
            }
            __syncwarp();
            float4* row = reinterpret_cast<float4*>(sm.scr[I].t[tl]);
#pragma unroll
            for (int j = 0; j < 4; j++) row[j] = make_float4(R[2 * j].x, R[2 * j].y, R[2 * j + 1].x, R[2 * j + 1].y);
            __syncwarp();
        }
        if (kSplit > 1) {
            __syncthreads();
            if (!first_warp) {
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    nrm[r] = sm.scr[I].nrm[8 * r + g];
                    bn[r] = sm.beta[32 * I + 8 * r + g] * nrm[r];
                    cc[r] = bn[r] * nrm[r];
                }
                const float4 x = sm.scr[I].m21[0][tl], y = sm.scr[I].m21[1][tl];
                M21 = {{x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w}};
            }
        }
        auto half = [&](int r0) {
            Frag f;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 x = *reinterpret_cast<const float2*>(&sm.scr[I].t[r0 + g + 8 * (i & 1)][2 * t4 + 8 * (i >> 1)]);
                f.x[2 * i] = x.x;
                f.x[2 * i + 1] = x.y;
            }
            return f;
        };
        T11 = half(0);
        T22 = half(16);
    }
    // (block decays of all warps are in shared memory; the scratch has been read: the Q tile comes in its place)
    fence_proxy_async();
    __syncthreads();
    if (kOut) {
        if (tid == 0) {
            mbar_arrive_expect_tx(&sm.full_q, G::kTile);
#pragma unroll
            for (int s = 0; s < G::kSlabs; s++) tma_load_4d(sm.q + s * G::kSlab, &tmQ, &sm.full_q, 64 * s, hd, c * kD, b);
        }
    }
    // ---- M against the earlier blocks
#pragma unroll
    for (int J = 0; J < kBlocks - 1; J++)
        if (J < I) {
            float acc[2][4][4];
            gram_block<kD, kPairs, false>(acc, kt, 32 * I, kt, 32 * J, tl, false);
#pragma unroll
            for (int m = 0; m < 2; m++) {
#pragma unroll
                for (int n = 0; n < 4; n++)
#pragma unroll
                    for (int e = 0; e < 4; e++) acc[m][n][e] *= cc[2 * m + (e >> 1)];
                M[J][m][0] = frag_of(acc[m][0], acc[m][1]);
                M[J][m][1] = frag_of(acc[m][2], acc[m][3]);
            }
        }
    auto tile = [&](int q) { return S * kOwn + q; };
    // sums of a tile's accumulators: rows g and g + 8, this lane's component
    auto sum_lo = [](const float (&d)[4], const float (&e)[4]) { return (d[0] + d[1]) + (e[0] + e[1]); };
    auto sum_hi = [](const float (&d)[4], const float (&e)[4]) { return (d[2] + d[3]) + (e[2] + e[3]); };
    // x <- (I + M_own)^-1 x, all column tiles
    auto solve = [&](float (&x)[kOwn][4]) {
        auto apply = [&](const Frag& f, int from, auto&& use) {
            const Split s = split(f);
#pragma unroll
            for (int q = 0; q < kOwn; q++) {
                float d[4] = {0.f, 0.f, 0.f, 0.f}, e[4] = {0.f, 0.f, 0.f, 0.f};
                mma_split(d, e, s, rhs_frag(x[q][from], x[q][from + 1]));
                use(x[q], sum_lo(d, e), sum_hi(d, e));
            }
        };
        apply(T11, 0, [](float (&v)[4], float lo, float hi) { v[0] = lo; v[1] = hi; });
        apply(M21, 0, [](float (&v)[4], float lo, float hi) { v[2] -= lo; v[3] -= hi; });
        apply(T22, 2, [](float (&v)[4], float lo, float hi) { v[2] = lo; v[3] = hi; });
    };
    // sum over the earlier blocks of M times their published fragments, subtracted from the right-hand sides
    auto subtract_earlier = [&](int J, int slot, float (&x)[kOwn][4]) {
#pragma unroll
        for (int m = 0; m < 2; m++) {
            float d[kOwn][4], e[kOwn][4];
#pragma unroll
            for (int q = 0; q < kOwn; q++)
#pragma unroll
                for (int i = 0; i < 4; i++) d[q][i] = e[q][i] = 0.f;
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int JJ = 0; JJ < kBlocks - 1; JJ++)
                    if (JJ == J) {
                        const Split s = split(M[JJ][m][h]);
#pragma unroll
                        for (int q = 0; q < kOwn; q++) mma_split(d[q], e[q], s, sm.get(slot, tile(q), h, tl));
                    }
#pragma unroll
            for (int q = 0; q < kOwn; q++) {
                x[q][2 * m] -= sum_lo(d[q], e[q]);
                x[q][2 * m + 1] -= sum_hi(d[q], e[q]);
            }
        }
    };
    const int comp = t4 & 1;
    // pair of the lane's component / of the fragment column in tile q
    auto pair_of = [&](int q) { return 2 * tile(q) + (t4 >> 1); };
    auto column_pair = [&](int q) { return 2 * tile(q) + (g >> 2); };
    constexpr int kPerTile = 2;
    // complex factor times the lane's component; `other` is the other component of the same value
    auto rotate = [&](cplx f, float own, float other) { return f.r * own + (comp ? f.i : -f.i) * other; };

    const int slow = sm.slow[I] & (((1 << G::kOwnPairs) - 1) << (G::kOwnPairs * S));   // of this warp's pairs
    // ---- g: the chain over the blocks of the chunk
    float gx[kOwn][4];
    {
#pragma unroll
        for (int q = 0; q < kOwn; q++)
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const float2 e = sm.viw[pair_of(q)][32 * I + 8 * r + g];
                gx[q][r] = bn[r] * (comp ? e.y : e.x);
            }
#pragma unroll
        for (int J = 0; J < kBlocks - 1; J++)
            if (J < I) {
                asm volatile("bar.sync %0, %1;" ::"r"(1 + S * (kBlocks - 1) + J), "r"(32 * (kBlocks - J)) : "memory");
                subtract_earlier(J, G::slot_g(J, I), gx);
            }
        solve(gx);
        float w[kOwn][4];                      // g carried to the block end
#pragma unroll
        for (int q = 0; q < kOwn; q++) {
            const cplx d31 = sm.bp[pair_of(q)][I].D31;
#pragma unroll
            for (int r = 0; r < 4; r++) w[q][r] = rotate(d31, gx[q][r], __shfl_xor_sync(0xffffffffu, gx[q][r], 1));
        }
        if (slow != 0) {                       // decays beyond the scaled form: step by step
            if (t4 == 0) {
#pragma unroll
                for (int r = 0; r < 4; r++) sm.walk[W][8 * r + g].x = nrm[r];
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < kOwn; q++)
#pragma unroll 1
                for (int s = 0; s < kPerTile; s++)
                    if ((slow >> (2 * tile(q) + s)) & 1) {
                        slow_walk<kD, kPairs, kMode, false>(sm, 2 * tile(q) + s, I, W, tl);
                        if ((t4 >> 1) == s) {
#pragma unroll
                            for (int r = 0; r < 4; r++) {
                                const float4 x = sm.walk[W][8 * r + g];
                                w[q][r] = comp ? x.y : x.x;
                            }
                        }
                        __syncwarp();
                        if (t4 == 0) {
#pragma unroll
                            for (int r = 0; r < 4; r++) sm.walk[W][8 * r + g].x = nrm[r];
                        }
                        __syncwarp();
                    }
        }
        // to every later block's start (times its reference product), and to the chunk end
#pragma unroll
        for (int q = 0; q < kOwn; q++) {
            const int p = pair_of(q);
            float wo[4];
#pragma unroll
            for (int r = 0; r < 4; r++) wo[r] = __shfl_xor_sync(0xffffffffu, w[q][r], 1);
            cplx f = {1.f, 0.f};
#pragma unroll
            for (int to = 1; to <= kBlocks; to++) {
                const bool end = to == kBlocks;
                if (to > I) {
                    if (!end || kNeedEnd || a.tail_state) {
                        const cplx ff = end ? f : cmul(f, sm.bp[p][to < kBlocks ? to : 0].R);
                        const int slot = end ? G::slot_end(I) : G::slot_g(I, to);
                        sm.put(slot, tile(q), 0, tl, rotate(ff, w[q][0], wo[0]), rotate(ff, w[q][1], wo[1]));
                        sm.put(slot, tile(q), 1, tl, rotate(ff, w[q][2], wo[2]), rotate(ff, w[q][3], wo[3]));
                    }
                    if (!end) f = cmul(f, sm.bp[p][to < kBlocks ? to : 0].A);
                }
            }
        }
        if (I < kBlocks - 1) asm volatile("bar.arrive %0, %1;" ::"r"(1 + S * (kBlocks - 1) + I), "r"(32 * (kBlocks - I)) : "memory");
        if (slow != 0) {                       // a slow pair takes no part in the scaled read-out
#pragma unroll
            for (int q = 0; q < kOwn; q++) {
                const bool mine = (slow >> pair_of(q)) & 1;
#pragma unroll
                for (int r = 0; r < 4; r++) gx[q][r] = mine ? 0.f : gx[q][r];
            }
        }
    }
    __syncthreads();

    // product of K^T (this warp's 32 columns) with the fragments `slot0 + block` of all blocks, one column tile
    auto k_transposed = [&](int slot0, int q, float (&d)[2][4]) {
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int e = 0; e < 4; e++) d[m][e] = 0.f;
#pragma unroll
        for (int J = 0; J < kBlocks; J++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const Rhs f = sm.get(slot0 + J, tile(q), h, tl);
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    uint32_t ka[4];
                    ldsm_x4_trans(col_frag<G::kSlab>(kt, 32 * J + 16 * h, 32 * I + 16 * m, tl), ka);
                    mma_bf16_m16n8k16(d[m], ka, f.c.x, f.c.y);
                    mma_bf16_m16n8k16(d[m], ka, f.ab.x, f.ab.y);
                }
            }
    };
    auto chunk_decay = [&](int p) {
        cplx w = sm.bp[p][0].A;
#pragma unroll
        for (int J = 1; J < kBlocks; J++) w = cmul(w, sm.bp[p][J].A);
        return w;
    };

    // ---- z at the chunk end; the carry
    if (kNeedEnd) {
        float z[kOwn][2][4];
#pragma unroll
        for (int q = 0; q < kOwn; q++) k_transposed(G::slot_end(0), q, z[q]);
        if (kMode == kFused) {
            if (!have_carry) {
                const unsigned long long t0 = global_ns();
                while (!(have_carry = __all_sync(0xffffffffu, flag_set()))) {
                    __nanosleep(20);
                    if (*reinterpret_cast<volatile int*>(a.status) != 0 || global_ns() - t0 > a.wait_ns) break;
                }
                have_carry = __all_sync(0xffffffffu, have_carry);
                if (have_carry) load_carry(carry_src);
            }
            cp_async_wait_all();
            __syncwarp();
        }
        const bool whole = Lc == kD;           // the reference's zero padding wipes state and decay (ssd.py:60-67)
        const bool bad = sm.first_bad < kD;
#pragma unroll
        for (int q = 0; q < kOwn; q++) {
            const int p = pair_of(q);
            if (p < NPB) {
                cplx gam = chunk_decay(p);
                gam = whole ? cplx{bfr(gam.r), bfr(gam.i)} : cplx{0.f, 0.f};
                if (kMode == kLocal && I == 0 && g == 0)
                    a.ws_gamma[unit * N + 2 * (pair0 + p) + comp] = comp ? gam.i : gam.r;
                const int n = 2 * (pair0 + p) + comp;
#pragma unroll
                for (int m = 0; m < 2; m++)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const int d = 32 * I + 16 * m + 8 * e + g;
                        const float l = !whole ? 0.f : bad ? kNotANumber : bfr(z[q][m][2 * e] + z[q][m][2 * e + 1]);
                        if (kMode == kLocal) {
                            a.ws_state[(unit * N + n) * kD + d] = l;
                        } else {
                            const float sr = sm.s_in[2 * p][d], si = sm.s_in[2 * p + 1][d];
                            const float s = comp ? next_im(gam, sr, si, l) : next_re(gam, sr, si, l);
                            if (c + 1 < a.NC) a.ws_state[((unit + H) * N + n) * kD + d] = s;
                            else if (a.final_state) a.final_state[(((size_t)b * H + hd) * N + n) * kD + d] = s;
                        }
                    }
            }
        }
        if (kMode == kLocal) return;
        if (c + 1 < a.NC && have_carry) {      // release this warp's columns to the next chunk
            __syncwarp();
            int* next = reinterpret_cast<int*>(a.ws_gamma + (unit + H) * (size_t)N);
            if (tl == 0) asm volatile("red.release.gpu.global.or.b32 [%0], %1;" ::"l"(next), "r"(1 << flag_bit) : "memory");
        }
    } else {
        grid_dependency_wait();   // the pass before; the records are there: it has waited for them before this launch
        if (!a.from_chunks) {
            load_carry(carry_src);
            cp_async_wait_all();
        } else {
            // s <- gamma s + z over the chunks before, in the carry pass's order; lane = column
            const size_t first = (size_t)b * a.NC * H + hd;
            float sr[G::kOwnPairs], si[G::kOwnPairs];
            const float* h0 = a.h0 ? a.h0 + ((size_t)b * H + hd) * N * kD + tok : nullptr;
            auto row = [&](int i) { return 2 * (pair0 + min(G::kOwnPairs * S + i, NPB - 1)); };
#pragma unroll
            for (int i = 0; i < G::kOwnPairs; i++) {
                sr[i] = h0 ? h0[row(i) * kD] : 0.f;
                si[i] = h0 ? h0[(row(i) + 1) * kD] : 0.f;
            }
            const int chunks = c + (c + 1 == a.NC && a.final_state ? 1 : 0);
            constexpr int kBatch = 8 / G::kOwnPairs < 2 ? 2 : 8 / G::kOwnPairs;
#pragma unroll 1
            for (int c0 = 0; c0 < chunks; c0 += kBatch) {
                float l[kBatch][G::kOwnPairs][2];
                float2 gm[kBatch][G::kOwnPairs];
#pragma unroll
                for (int k = 0; k < kBatch; k++) {
                    const size_t u = first + (size_t)min(c0 + k, chunks - 1) * H;
#pragma unroll
                    for (int i = 0; i < G::kOwnPairs; i++) {
                        const float* z = a.ws_state + (u * N + row(i)) * kD + tok;
                        l[k][i][0] = __ldcg(z);
                        l[k][i][1] = __ldcg(z + kD);
                        gm[k][i] = __ldcg(reinterpret_cast<const float2*>(a.ws_gamma + u * N + row(i)));
                    }
                }
#pragma unroll
                for (int k = 0; k < kBatch; k++) {
                    if (c0 + k == c) {   // (the last chunk's own step, for the final state)
#pragma unroll
                        for (int i = 0; i < G::kOwnPairs; i++) {
                            sm.s_in[2 * (G::kOwnPairs * S + i)][tok] = sr[i];
                            sm.s_in[2 * (G::kOwnPairs * S + i) + 1][tok] = si[i];
                        }
                    }
                    if (c0 + k < chunks) {
#pragma unroll
                        for (int i = 0; i < G::kOwnPairs; i++) {
                            const cplx gam = {gm[k][i].x, gm[k][i].y};
                            const float nr = next_re(gam, sr[i], si[i], l[k][i][0]);
                            si[i] = next_im(gam, sr[i], si[i], l[k][i][1]);
                            sr[i] = nr;
                        }
                    }
                }
            }
            if (chunks == c) {
#pragma unroll
                for (int i = 0; i < G::kOwnPairs; i++) {
                    sm.s_in[2 * (G::kOwnPairs * S + i)][tok] = sr[i];
                    sm.s_in[2 * (G::kOwnPairs * S + i) + 1][tok] = si[i];
                }
            } else {
                float* fs = a.final_state + ((size_t)b * H + hd) * N * kD + tok;
#pragma unroll
                for (int i = 0; i < G::kOwnPairs; i++)
                    if (G::kOwnPairs * S + i < NPB) {
                        fs[row(i) * kD] = sr[i];
                        fs[(row(i) + 1) * kD] = si[i];
                    }
            }
        }
        __syncwarp();
    }
    // r_0: the carry rounded to bf16
#pragma unroll
    for (int i = 0; i < 2 * G::kOwnPairs; i++) {
        const int n = 2 * G::kOwnPairs * S + i;
        sm.r0[n][tok] = __float2bfloat16_rn(sm.s_in[n][tok]);
    }
    const bool q_here = mbar_wait_suspend(&sm.full_q, 0, &sm.abort_flag, a.wait_ns);
    if (!__syncthreads_and(q_here && have_carry)) {
        if (tid == 0) atomicCAS(a.status, 0, 202);
        drain(&sm.full_q);
        return;
    }

    // B fragment of r_0^T: columns in the tiles' order, the lo columns empty (r_0 is bf16)
    auto r0_frag = [&](int q, int ks) {
        const int n = 2 * column_pair(q) + ((g >> 1) & 1);
        const uint32_t* s = reinterpret_cast<const uint32_t*>(&sm.r0[n][16 * ks + 2 * t4]);
        return (g & 1) ? make_uint2(0u, 0u) : make_uint2(s[0], s[4]);
    };
    // ---- h: right-hand sides c_t k_t.r_0, the same chain
    float hx[kOwn][4];
    {
        float d[kOwn][2][4];
#pragma unroll
        for (int q = 0; q < kOwn; q++)
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int e = 0; e < 4; e++) d[q][m][e] = 0.f;
#pragma unroll
        for (int ks = 0; ks < kKs; ks++) {
            uint32_t ka[2][4];
            ldsm_x4(row_frag<G::kSlab>(kt, 32 * I, ks, tl), ka[0]);
            ldsm_x4(row_frag<G::kSlab>(kt, 32 * I + 16, ks, tl), ka[1]);
#pragma unroll
            for (int q = 0; q < kOwn; q++) {
                const uint2 f = r0_frag(q, ks);
                mma_bf16_m16n8k16(d[q][0], ka[0], f.x, f.y);
                mma_bf16_m16n8k16(d[q][1], ka[1], f.x, f.y);
            }
        }
#pragma unroll
        for (int q = 0; q < kOwn; q++)
#pragma unroll
            for (int r = 0; r < 4; r++) hx[q][r] = cc[r] * d[q][r >> 1][2 * (r & 1)];
#pragma unroll
        for (int J = 0; J < kBlocks - 1; J++)
            if (J < I) {
                asm volatile("bar.sync %0, %1;" ::"r"(1 + S * (kBlocks - 1) + J), "r"(32 * (kBlocks - J)) : "memory");
                subtract_earlier(J, G::slot_h(J), hx);
            }
        solve(hx);
#pragma unroll
        for (int q = 0; q < kOwn; q++) {
            sm.put(G::slot_h(I), tile(q), 0, tl, hx[q][0], hx[q][1]);
            sm.put(G::slot_h(I), tile(q), 1, tl, hx[q][2], hx[q][3]);
        }
        if (I < kBlocks - 1) asm volatile("bar.arrive %0, %1;" ::"r"(1 + S * (kBlocks - 1) + I), "r"(32 * (kBlocks - I)) : "memory");
        __syncwarp();
    }

    // ---- |q|^-1 and q.r_0
    float mq[4], rho[kOwn][4];
    {
        float qd[2][2][4], d[kOwn][2][4];
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int e = 0; e < 4; e++) qd[m][0][e] = qd[m][1][e] = 0.f;
#pragma unroll
        for (int q = 0; q < kOwn; q++)
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int e = 0; e < 4; e++) d[q][m][e] = 0.f;
#pragma unroll
        for (int ks = 0; ks < kKs; ks++) {
            uint32_t qa[2][4];
            ldsm_x4(row_frag<G::kSlab>(qt, 32 * I, ks, tl), qa[0]);
            ldsm_x4(row_frag<G::kSlab>(qt, 32 * I + 16, ks, tl), qa[1]);
#pragma unroll
            for (int m = 0; m < 2; m++) {
                mma_bf16_m16n8k16(qd[m][0], qa[m], qa[m][0], qa[m][2]);
                mma_bf16_m16n8k16(qd[m][1], qa[m], qa[m][1], qa[m][3]);
            }
#pragma unroll
            for (int q = 0; q < kOwn; q++) {
                const uint2 f = r0_frag(q, ks);
                mma_bf16_m16n8k16(d[q][0], qa[0], f.x, f.y);
                mma_bf16_m16n8k16(d[q][1], qa[1], f.x, f.y);
            }
        }
        diagonal_of(qd[0][0], qd[0][1], tl, mq[0], mq[1]);
        diagonal_of(qd[1][0], qd[1][1], tl, mq[2], mq[3]);
#pragma unroll
        for (int r = 0; r < 4; r++) mq[r] = rsqrtf(mq[r] + kEps);
#pragma unroll
        for (int q = 0; q < kOwn; q++)
#pragma unroll
            for (int r = 0; r < 4; r++) rho[q][r] = d[q][r >> 1][2 * (r & 1)];
    }
    // ---- read-out: P against the block itself and the earlier ones
    float oz[kOwn][4], pd[4];
#pragma unroll
    for (int q = 0; q < kOwn; q++)
#pragma unroll
        for (int r = 0; r < 4; r++) oz[q][r] = 0.f;
#pragma unroll 1
    for (int J = I; J >= 0; J--) {
        const bool diag = J == I;
        float acc[2][4][4];
        gram_block<kD, kPairs, false>(acc, qt, 32 * I, kt, 32 * J, tl, diag);
        if (diag) {
            diagonal_of(acc[0][0], acc[0][1], tl, pd[0], pd[1]);
            diagonal_of(acc[1][2], acc[1][3], tl, pd[2], pd[3]);
#pragma unroll
            for (int m = 0; m < 2; m++)        // strictly lower (the diagonal enters with g itself below)
#pragma unroll
                for (int n = 0; n < 2; n++)
#pragma unroll
                    for (int e = 0; e < 4; e++)
                        if (g + 8 * (e >> 1) <= 8 * n + 2 * t4 + (e & 1)) acc[m][2 * m + n][e] = 0.f;
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const Split p0 = split(frag_of(acc[0][2 * h], acc[0][2 * h + 1])), p1 = split(frag_of(acc[1][2 * h], acc[1][2 * h + 1]));
#pragma unroll
            for (int q = 0; q < kOwn; q++) {
                const Rhs fg = diag ? rhs_frag(gx[q][2 * h], gx[q][2 * h + 1]) : sm.get(G::slot_g(J, I), tile(q), h, tl);
                const Rhs fh = sm.get(G::slot_h(J), tile(q), h, tl);
                float dz[2][4], dh[2][4];
#pragma unroll
                for (int m = 0; m < 2; m++)
#pragma unroll
                    for (int e = 0; e < 4; e++) dz[m][e] = dh[m][e] = 0.f;
                if (!(diag && h == 1)) {
                    mma_split(dz[0], dz[0], p0, fg);
                    mma_split(dh[0], dh[0], p0, fh);
                }
                mma_split(dz[1], dz[1], p1, fg);
                mma_split(dh[1], dh[1], p1, fh);
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    oz[q][r] += dz[r >> 1][2 * (r & 1)] + dz[r >> 1][2 * (r & 1) + 1];
                    rho[q][r] -= dh[r >> 1][2 * (r & 1)] + dh[r >> 1][2 * (r & 1) + 1];
                }
            }
        }
    }
    // W_{t-1} = D_{t-1} F, F = (decay up to the block) R; the first token of a block takes the decay itself
    auto decay_before = [&](int p) {
        cplx pre = {1.f, 0.f};
#pragma unroll
        for (int J = 0; J < kBlocks - 1; J++)
            if (J < I) pre = cmul(pre, sm.bp[p][J].A);
        return pre;
    };
#pragma unroll
    for (int q = 0; q < kOwn; q++) {
        const int p = pair_of(q);
        const cplx pre = decay_before(p), F = cmul(pre, sm.bp[p][I].R);
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int row = 32 * I + 8 * r + g;
            const float x = oz[q][r] + pd[r] * gx[q][r], xo = __shfl_xor_sync(0xffffffffu, x, 1);
            const float ho = __shfl_xor_sync(0xffffffffu, rho[q][r], 1);
            const float2 D = sm.dd[p][row], D0 = sm.dd[p][row > 0 ? row - 1 : 0];
            const bool first = r == 0 && g == 0;
            const cplx w0 = first ? pre : cmul({D0.x, D0.y}, F);
            oz[q][r] = rotate({D.x, D.y}, x, xo) + rotate(w0, rho[q][r], ho);
        }
    }
    if (slow != 0) {
#pragma unroll
        for (int q = 0; q < kOwn; q++)
#pragma unroll 1
            for (int s = 0; s < kPerTile; s++)
                if ((slow >> (2 * tile(q) + s)) & 1) {
                    const cplx pre = decay_before(2 * tile(q) + s);
                    slow_walk<kD, kPairs, kMode, true>(sm, 2 * tile(q) + s, I, W, tl);
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        const float ho = __shfl_xor_sync(0xffffffffu, rho[q][r], 1);
                        const float4 x = sm.walk[W][8 * r + g];
                        if ((t4 >> 1) == s)
                            oz[q][r] = (comp ? x.y : x.x) + rotate(cmul(pre, {x.z, x.w}), rho[q][r], ho);
                    }
                    __syncwarp();
                }
    }
#pragma unroll
    for (int q = 0; q < kOwn; q++) {
        const int p = pair_of(q);
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int row = 32 * I + 8 * r + g;
            float yy = row >= sm.first_bad ? kNotANumber : mq[r] * oz[q][r];
            if (a.shortcut_scale != 0.f) {   // block.py:202-208; v after the vp scale
                const float qk = mq[r] * nrm[r] * pd[r];
                const float2 e = sm.viw[p][row], D = sm.dd[p][row];
                cplx vg = cmul({e.x, e.y}, {D.x, D.y});
                if ((slow >> p) & 1) {               // (its v has made room for g)
                    const uint32_t w = __ldcg(a.rec_v + (unit * (size_t)NP + pair0 + p) * kD + row);
                    vg = {bits_lo(w), bits_hi(w)};
                }
                yy += a.shortcut_scale * qk * qk * bfr(comp ? vg.i : vg.r);
            }
            sm.y(row)[2 * p + comp] = __float2bfloat16_rn(bfr(yy) * sm.sel[row]);
        }
    }
    __syncwarp();
    if (tok < Lc) {   // lane = token: its row of this warp's values
        constexpr int kOwnPairs = G::kOwnPairs;
        __nv_bfloat16* yo = a.y + (((size_t)b * L + c * kD + tok) * H + hd) * N + 2 * pair0;
        const uint32_t* ys = reinterpret_cast<const uint32_t*>(sm.y(tok));
        const int p0 = kOwnPairs * S;
        if (kOwnPairs >= 4 && NPB == kPairs && N % 8 == 0 && (reinterpret_cast<uintptr_t>(a.y) & 15) == 0) {
#pragma unroll
            for (int i = 0; i < kOwnPairs; i += 4)
                *reinterpret_cast<uint4*>(yo + 2 * (p0 + i)) = make_uint4(ys[p0 + i], ys[p0 + i + 1], ys[p0 + i + 2], ys[p0 + i + 3]);
        } else {
            for (int i = p0; i < min(NPB, p0 + kOwnPairs); i++) reinterpret_cast<uint32_t*>(yo)[i] = ys[i];
        }
    }
    // ---- the recurrent state after the last token
    if (a.tail_state && c == a.NC - 1) {
        __syncthreads();   // every block's h is published
#pragma unroll 1
        for (int q = 0; q < kOwn; q++) {
            float z[2][4], h[2][4];
            k_transposed(G::slot_end(0), q, z);
            k_transposed(G::slot_h(0), q, h);
            const int p = pair_of(q);
            const cplx w = chunk_decay(p);
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int d = 32 * I + 16 * m + 8 * e + g, n = 2 * p + comp;
                    const float r = __bfloat162float(sm.r0[n][d]) - (h[m][2 * e] + h[m][2 * e + 1]);
                    const float o = __shfl_xor_sync(0xffffffffu, r, 1);
                    if (p < NPB)
                        a.tail_state[(((size_t)b * H + hd) * N + 2 * pair0 + n) * kD + d] =
                            sm.first_bad < kD ? kNotANumber : z[m][2 * e] + z[m][2 * e + 1] + rotate(w, r, o);
                }
        }
    }
}

// ------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------
template <int kD, int kPairs, Mode kMode> struct KernelTag {};

template <int kD, int kPairs, Mode kMode>
static int launch_one(const CUtensorMap& tmK, const CUtensorMap& tmQ, const Args& a, cudaStream_t st) {
    const size_t smem = sizeof(Smem<kD, kPairs, kMode>);
    static_assert(sizeof(Smem<kD, kPairs, kMode>) <= 227 * 1024, "shared memory");
    if (int rc = allow_smem<KernelTag<kD, kPairs, kMode>>((const void*)scan_chunk_kernel<kD, kPairs, kMode>, smem)) return rc;
    const long long units = (long long)a.B * a.NC * a.H * a.groups;
    return launch_overlapped(scan_chunk_kernel<kD, kPairs, kMode>, dim3((unsigned)units), dim3(Geo<kD, kPairs>::kThreads), smem, st,
                             tmK, tmQ, a);
}
template <int kD, int kPairs>
static int launch_mode(Mode m, const CUtensorMap& tmK, const CUtensorMap& tmQ, const Args& a, cudaStream_t st) {
    if (m == kLocal) return launch_one<kD, kPairs, kLocal>(tmK, tmQ, a, st);
    if (m == kOutput) return launch_one<kD, kPairs, kOutput>(tmK, tmQ, a, st);
    return launch_one<kD, kPairs, kFused>(tmK, tmQ, a, st);
}
template <int kD>
static int launch_tiles(Mode m, const CUtensorMap& tmK, const CUtensorMap& tmQ, const Args& a, cudaStream_t st) {
    // (head_dim 128, eight pairs in one block: 124 KB, one block per SM, 400 ns a chunk on the full GPU; in two blocks that
    // both form G and P, 218)
    if (a.N <= 4) return launch_mode<kD, 2>(m, tmK, tmQ, a, st);
    if (kD == 128 || a.N <= 8) return launch_mode<kD, 4>(m, tmK, tmQ, a, st);
    return launch_mode<64, 8>(m, tmK, tmQ, a, st);
}

}  // namespace chunk

bool scan_chunk_supported(int D, int N, int C, int dtype) {
    return dtype == CDSSM_BF16 && D == C && (D == 64 || D == 128) && N > 2 && N <= 16;
}

// scan_records.cu
void scan_record_arrays(void* rec, int B, int L, int H, int N, int C, float2** a, uint32_t** v, uint32_t** g);

// mode 0: local pass (fills ws_gamma / ws_state for the carry pass), 1: output pass (reads the carries from ws_state, with
// from_chunks the local results of this call's local pass; writes y, with from_chunks the final state too), 2: both in one kernel with the carry handed on inside it (ws_gamma and *ticket zeroed by the caller).
// status: one int in device memory, set by a bounded wait that ran out (not cleared here).
int scan_chunk_pass(int mode, int from_chunks, const void* q, long long q_rs, const void* k, long long k_rs, void* rec, const float* h0, void* y, float* final_state,
                    float* tail_state, float* ws_gamma, float* ws_state, int* status, int* ticket, float shortcut_scale, int B,
                    int L, int H, int D, int N, unsigned long long wait_ns, int withhold, cudaStream_t st) {
    using namespace chunk;
    CUtensorMap tmK, tmQ;
    if (!make_tile_map(&tmK, k, k_rs, B, L, H, D, D) || !make_tile_map(&tmQ, mode == 0 ? k : q, mode == 0 ? k_rs : q_rs, B, L, H, D, D)) return CDSSM_ERR_CUDA;
    Args a;
    float2* ra;
    uint32_t *rv, *rg;
    scan_record_arrays(rec, B, L, H, N, D, &ra, &rv, &rg);
    a.rec_a = ra; a.rec_v = rv; a.rec_g = rg;
    a.h0 = h0;
    a.y = static_cast<__nv_bfloat16*>(y);
    a.final_state = final_state; a.tail_state = tail_state;
    a.ws_gamma = ws_gamma; a.ws_state = ws_state; a.status = status; a.ticket = ticket;
    a.wait_ns = wait_ns ? wait_ns : 400ull * 1000 * 1000;
    a.withhold = withhold;
    a.from_chunks = from_chunks;
    a.shortcut_scale = shortcut_scale;
    a.B = B; a.L = L; a.H = H; a.N = N; a.NC = (L + D - 1) / D;
    a.groups = D == 128 && N > 8 ? 2 : 1;
    if ((long long)B * a.NC * H * a.groups > 0x7fffffff) return CDSSM_ERR_UNSUPPORTED;
    const Mode m = mode == 0 ? kLocal : mode == 1 ? kOutput : kFused;
    if (mode == 0) a.tail_state = nullptr;
    return D == 128 ? launch_tiles<128>(m, tmK, tmQ, a, st) : launch_tiles<64>(m, tmK, tmQ, a, st);
}

}  // namespace cdssm
