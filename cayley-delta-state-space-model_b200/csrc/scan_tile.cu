// The scan on tensor cores, one pass over k and q: bf16 storage, head_dim D = chunk C in {64, 128}, even state_dim N <= 16,
// any head count.
//
// One thread block owns a tile of 128 tokens: a chunk of one head (D 128) or the same chunk of two heads (D 64); a warp (D 64
// and N > 4: two warps, half of the pairs each) its 32 tokens.  With g_t the coefficient that the step at token t adds along k_t (raw
// keys; n_t = 1/|k_t|, c_t = beta_t n_t^2, W_t = a_0 ... a_t),
//     local state     z_t = W_t sum_{i<=t} (g_i / W_i) k_i,   g_t = beta_t n_t v_t - c_t W_t sum_{i<t} (g_i / W_i) G[t,i]
//     correction      r_t = W_t (r_0 - sum_{i<=t} h_i k_i),   h_t = c_t (k_t.r_0) - c_t sum_{i<t} h_i G[t,i]
//     read-out        y_t ~ W_t sum_{i<=t} (g_i / W_i) P[t,i]  +  W_{t-1} (q_t.r_0 - sum_{i<t} h_i P[t,i])
// with G = K K^T, P = Q K^T.  In the scaled unknowns g_i / W_i and h_i both systems have the same REAL unit lower triangular
// matrix I + M, M[t,i] = c_t G[t,i], for every complex pair of the head: the pairs are right-hand sides.  So
//   - G and P of the whole tile are tcgen05 products of the TMA-staged tiles (M = N = 128, fp32 accumulators in tensor memory,
//     128 columns: P takes G's place), read back as 32 x 32 blocks in the fragment layout of the warp-level mma;
//   - the 16 x 16 diagonal blocks are inverted by substitution, a row per lane, all rows at once and independent of any state
//     (as 8 x 8 halves: seven dependent steps instead of fifteen);
//   - what is left of the serial chain is three 16-wide products per 32 tokens, passed from warp to warp;
//   - everything with a right-hand side is a warp-level tf32 product with n = 8 columns {re hi, re lo, im hi, im lo} of two
//     pairs; a float32 operand enters as hi + lo, 11 significant bits each, on the matrix side too, hi rounded to nearest: the sum
//     is the value to half an ulp (root mean square).  G and P go in as they come from tensor memory: an instruction's split costs
//     three operations a value (three bf16 parts: five and a half, and as many products).  State after one chunk against float64,
//     median, D 64 / 128: 1.6e-7 / 1.8e-7 of it; three bf16 parts 1.6e-7 / 1.9e-7, the walk in float32 1.5e-7 / 1.8e-7, hi cut off
//     instead of rounded 2.5e-7 / 2.4e-7 (test_scan_precision_gpu.py).
// The division by W_i only spans a 32-token block, relative to its middle (|W ratio| of 16 tokens >= 1e-30); between blocks
// all factors are plain products, applied to the sums over a block.  A (block, pair) that decays further is walked step by
// step (slow_walk).
//
// The reference's carry s_{c+1} = gamma_c s_c + z_{C-1} (inter_chunk_scan.cu:73-83) is handed on inside the kernel: blocks take
// (chunk, batch, head) work in chunk-major order from a ticket counter, leave their chunk's (gamma, z) for others as soon as they
// have it, then look back for the nearest chunk whose carry-out is known and add up the chunks in between, in the order of the
// sequence: the bits do not depend on how far anybody had come.  kLocal / kOutput are the two halves with the carry pass of
// scan_simt.cu between them (summaries, callers with little scratch, few long sequences: hands_carry_on() there); while there are
// few chunks the output pass adds them up itself instead, having done all that needs no carry by the time the local pass ends.
//
// Bounded by issue slots (45 % of them busy at 16 warps per SM) and by the chain of barriers and products through a chunk.  us of a
// whole call on B200, before (a block per chunk and head, Gram blocks and three bf16 parts on the warp-level mma, carry behind a
// fence and a flag) / now: D 64, B 8, L 2048, H 24, N 16 291 / 229, N 8 171 / 151, N 4 136 / 113; one sequence of 523, N 16
// 36.7 / 30.1, N 4 22.8 / 19.0; D 128, 4 x 2048, H 12, N 4 76 / 49, 2 x 1000, H 32, N 8 73 / 51, 4000 tokens, H 12, N 16 144 / 74.
// One or two chunks of D 64, N 8, gain nothing: 2 x 41 tokens, H 16 11.5 / 12.3.
//
// Reference semantics (intra_chunk_scan.cu:100-195, exact_correction.cu:89-150): z starts at zero at the chunk start, r
// from the bf16-rounded carry, the correction is read before its step.
#include "cdssm_common.cuh"
#include "sm100_ptx.cuh"
#include "tile_map.cuh"
#include <type_traits>

namespace cdssm {
using namespace sm100;

namespace tile {

enum Mode { kLocal, kOutput, kFused };   // local results only; outputs from given carries; both, the carry handed on inside
enum Vec { kG, kH };             // solutions in shared memory: g (scaled), h

struct Args {
    const float2* rec_a;         // (B,NC,H,NP,C): transition a_t
    const uint32_t* rec_v;       // (B,NC,H,NP,C): vp-scaled v_t, bf16 pair
    const uint32_t* rec_g;       // (B,NC,H,C): beta_t, sel_C, bf16 pair
    const float* h0;
    __nv_bfloat16* y;
    float *final_state, *tail_state;
    float* ws_gamma;             // (B,NC,H,NP,2): chunk decays (kLocal)
    float* ws_state;             // (B,NC,H,NP,2,D): z_{C-1} (kLocal), rounded carry into the chunk (kOutput)
    uint32_t *gammas, *chunks;   // (B,NC,H,NP) gamma, (B,NC,H,NP,D) z of a chunk: words (put_word32()) of bf16 pairs
    uint64_t* carries;           // (B,NC,H,NP,D): carry out of a chunk (kFused: all three zeroed by the records kernel)
    int *status, *ticket;
    unsigned long long wait_ns;  // limit of every device-side wait
    int withhold;                // test hook: nothing is loaded, so the first wait runs out
    float shortcut_scale;
    int B, L, H, N, NC;
    int HG;                      // tiles beside each other: ceil(H / heads of a tile) x blocks that share a tile (kPairs pairs each)
    int groups;
    int from_chunks;             // kOutput: the carry from the local results of the chunks before (no carry pass has run)
    int fixed;                   // kFused: a block per SM at most: narrow blocks have the tiles of their own numbers, not of tickets
};

#define kNotANumber __int_as_float(0x7fffffff)

struct cplx { float r, i; };
// (Which products and sums go together is said here and below, not left to the compiler: the versions of the kernel have the same bits.
// cmul(a, b) and cmul(b, a) differ in the last bit of the imaginary part.)
__device__ __forceinline__ cplx cmul(cplx a, cplx b) {
    return {__fmaf_rn(a.r, b.r, -__fmul_rn(a.i, b.i)), __fmaf_rn(a.r, b.i, __fmul_rn(a.i, b.r))};
}
__device__ __forceinline__ cplx cshfl(cplx v, int src) {
    return {__shfl_sync(0xffffffffu, v.r, src), __shfl_sync(0xffffffffu, v.i, src)};
}
__device__ __forceinline__ float bfr(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ float bits_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ float bits_lo(uint32_t w) { return __uint_as_float(w << 16); }

// 1 / x for normal x in 1e-30 ... 1e30: the approximation and one Newton step, no branch for the values outside.  Its remainder is
// squared by the step (2^-44), so the result is the nearest float but where two are as near to 2^-20 of their distance; __frcp_rn
// gave states off by the same three digits and took 3 % of the call.
__device__ __forceinline__ float reciprocal(float x) {
    const float r = __fdividef(1.f, x);
    return fmaf(r, fmaf(-x, r, 1.f), r);
}

struct BlockPair {   // of one 32-token block and pair
    cplx A, R, D31;  // product of a over the block; product of its first half (the scaling's reference); D of the last token
};

// ---- decay scalings of a 32-token block and pair (lane = token) ---------------------------------------------------
// The scaled unknowns need ratios of the prefix products W_t = a_0 ... a_t only, taken relative to the middle of the
// block, D_t = W_t / W_15: lanes 0-15 hold the suffix product a_{t+1} ... a_15 = 1 / D_t, lanes 16-31 the prefix product
// a_16 ... a_t = D_t, and neither half leaves the float range unless one half alone decays by more than 1e-30.
// kW pairs side by side: one alone waits for its shuffles.  at, vg: a_t, v_t in; D, v_t / D out (a and v of a pair outside the
// range: the walk reads them themselves).  Returns the pairs outside the range, a bit each.
// kSwap: the factors of the prefix products the other way round, for the bits of the pair that a first warp has alone (kD 64, four pairs).
template <int kW, bool kSwap>
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
            if (on) X[w] = kSwap ? cmul(other, X[w]) : cmul(X[w], other);
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
        const float sc1 = reciprocal(m);
        const cplx En = {E.r * sc1, E.i * sc1};
        const float q = sc1 * reciprocal(__fmaf_rn(En.r, En.r, __fmul_rn(En.i, En.i)));
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

// What takes block `from`'s sums, carried to its end, into block `to`'s frame (to = blocks: the chunk end), blocks counted in the
// chunk, bp at the chunk's first block: the decay over the blocks in between and up to `to`'s middle.  To its end a block's scaled
// sums (up to 1e30) are carried by D31 (down to 1e-30), and by that alone: its product with the later block's R (1e-30 as well) would
// be zero in float32 where the value is of order one.
__device__ __forceinline__ cplx behind(const BlockPair* bp, int from, int to, int blocks) {
    cplx f = {1.f, 0.f};
    for (int j = from + 1; j < to; j++) f = cmul(bp[j].A, f);
    return to < blocks ? cmul(bp[to].R, f) : f;
}

// s <- gamma s + l in the order in which the carry pass (scan_simt.cu) evaluates it, so that the two ways to hand the carry on
// give the same bits: chunk-aligned pieces of a sequence compose exactly whichever of them runs.
__device__ __forceinline__ float next_re(cplx g, float sr, float si, float l) {
    return __fadd_rn(__fmaf_rn(g.r, sr, -__fmul_rn(g.i, si)), l);
}
__device__ __forceinline__ float next_im(cplx g, float sr, float si, float l) {
    return __fadd_rn(__fmaf_rn(g.r, si, __fmul_rn(g.i, sr)), l);
}

// ---- the carry from block to block, a column at a time: words that are zero until they are written once, so that a
// reader sees from the word itself whether it is there.  No fence, no flag: a fence of the writer's took 2 000 to 4 000 cycles
// beside the tiles' own traffic, and whoever waited for the flag waited for it too.
// A word holds the complement of its value, which is never all ones: numbers that are none have one pattern.
__device__ __forceinline__ uint64_t word_of(uint32_t lo, uint32_t hi) { return ~((uint64_t)hi << 32 | lo); }
__device__ __forceinline__ uint32_t word_lo(uint64_t w) { return ~(uint32_t)w; }
__device__ __forceinline__ uint32_t word_hi(uint64_t w) { return ~(uint32_t)(w >> 32); }
__device__ __forceinline__ void put_word(uint64_t* p, uint64_t w) { asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(w) : "memory"); }
__device__ __forceinline__ uint64_t get_word(const uint64_t* p) {
    uint64_t w;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    return w;
}
__device__ __forceinline__ void put_word32(uint32_t* p, uint32_t x) { asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(~x) : "memory"); }
__device__ __forceinline__ uint32_t get_word32(const uint32_t* p) {
    uint32_t w;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(w) : "l"(p) : "memory");
    return w;
}
// carry out of a chunk: real, imaginary part
__device__ __forceinline__ uint64_t carry_word(float r, float i) {
    return word_of(r == r ? __float_as_uint(r) : 0x7fffffffu, i == i ? __float_as_uint(i) : 0x7fffffffu);
}
// two values that are bf16 already
__device__ __forceinline__ uint32_t bf16_pair(cplx x) { return pack2(x.r, x.i); }
__device__ __forceinline__ cplx pair_of_word(uint32_t w) { return {bits_lo(~w), bits_hi(~w)}; }

// The nearest value of 11 significant bits, what a tf32 operand holds.  The rest, 12 bits and a sign, goes into another one, which
// drops its last bit: an ulp of x in one value of four, to either side.  (Cut off instead of rounded, the rest had 13 bits and lost
// up to three ulps, always to the same side.)
__device__ __forceinline__ float tf32_hi(float x) { return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u); }

// One k-step of eight columns: x in accumulator order (row g: columns 2 t4, 2 t4 + 1; row g + 8), b the two tokens' values of
// this lane's column.  kFirst: d = x b, else d += x b.
template <bool kFirst>
__device__ __forceinline__ void mma_tf32(float (&d)[4], float x0, float x1, float x2, float x3, float2 b) {
    if (kFirst)
        asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
            : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
            : "r"(__float_as_uint(x0)), "r"(__float_as_uint(x2)), "r"(__float_as_uint(x1)), "r"(__float_as_uint(x3)),
              "r"(__float_as_uint(b.x)), "r"(__float_as_uint(b.y)), "f"(0.f));
    else
        asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(__float_as_uint(x0)), "r"(__float_as_uint(x2)), "r"(__float_as_uint(x1)), "r"(__float_as_uint(x3)),
              "r"(__float_as_uint(b.x)), "r"(__float_as_uint(b.y)));
}
struct Split { float hi[4], lo[4]; };
__device__ __forceinline__ Split split(const float* x) {
    Split s;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float v = x[i];
        asm volatile("" : "+f"(v));   // (a second split of the same value is made anew: parts that were kept spilt, 252 -> 245 us at N 16, 160 -> 157 at N 8)
        s.hi[i] = tf32_hi(v);
        s.lo[i] = v - s.hi[i];
    }
    return s;
}
// d (+)= hi(x) b, e (+)= lo(x) b
template <bool kFirst>
__device__ __forceinline__ void mma_split(float (&d)[4], float (&e)[4], const Split& s, float2 b) {
    mma_tf32<kFirst>(d, s.hi[0], s.hi[1], s.hi[2], s.hi[3], b);
    mma_tf32<kFirst>(e, s.lo[0], s.lo[1], s.lo[2], s.lo[3], b);
}

// kWide: a warp per column tile of a 32-token block, for calls that have an SM per tile: half the chain, half the code
template <int kD, int kPairs_, bool kWide = false>
struct Geo {
    static constexpr int kPairs = kPairs_;               // complex pairs held (>= N / 2)
    static constexpr int kComps = 2 * kPairs;
    static constexpr int kHeads = 128 / kD;              // of a tile
    static constexpr int kBlocks = kD / 32;              // 32-token blocks of a chunk
    static constexpr int kTiles = (kPairs + 1) / 2;      // column tiles of two pairs
    static constexpr int kNarrow = kPairs >= 8 || (kD == 64 && kPairs >= 4) ? 2 : 1;
    static constexpr int kSplit = kWide ? kTiles : kNarrow;   // warps that share the column tiles of a 32-token block
    static constexpr int kThreads = 128 * kSplit;
    static constexpr int kOwn = kTiles / kSplit, kOwnPairs = kPairs / kSplit;   // of a warp
    static constexpr int kSlabs = kD / 64, kKs = kD / 16;
    static constexpr uint32_t kSlab = 128 * 128;         // bytes of 128 rows x 64 bf16 columns
    static constexpr uint32_t kTile = kSlabs * kSlab;
    // solutions as rows of 128 tokens, the hi parts of all components, then the lo parts: the strides keep the eight-byte reads of
    // a fragment (columns {re hi, re lo, im hi, im lo ...} x token pairs) and the writes of a quad on distinct banks
    static constexpr int kRow = 136;
    static constexpr int kPart = kComps * kRow + (kComps * kRow % 32 == 16 ? 0 : 16);
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

// (resident blocks per SM: kMinBlocks below)
template <int kD, int kPairs, Mode kMode, bool kWide>
struct __align__(1024) Smem {
    using G = Geo<kD, kPairs, kWide>;
    uint8_t k[G::kTile];                                 // swizzled rows = tokens
    union {
        uint8_t q[kMode == kLocal ? 1024 : G::kTile];
        Scratch scr[4];
    };
    float vec[kMode == kLocal ? 1 : 2][2 * G::kPart];    // g, h
    float2 viw[kPairs][128], dd[kPairs][128];            // v / D, D
    uint32_t bs[128];                                    // beta, sel_C: bf16 pair
    BlockPair bp[kPairs][4];
    float zl[G::kComps][128];                            // z at the chunk end; later y on its way to one row a lane
    __nv_bfloat16 r0[G::kHeads][G::kComps][kD + 8];      // the carry rounded (padded rows: fragment loads hit distinct banks)
    float4 walk[4 * G::kSplit][32];                      // slow_walk results
    __device__ __forceinline__ __nv_bfloat16* y(int token) {
        return reinterpret_cast<__nv_bfloat16*>(zl) + token * (2 * kPairs + 2);
    }
    uint64_t full_k, full_q, mma_g, mma_p;
    uint32_t tmem;
    int slow[G::kSplit][4];                              // pairs that are walked step by step, a bit each
    int abort_flag, item, stop;
    int bad_rows;                                        // a key row has been emptied: G is formed again
    int first_bad[2];                                    // per head: first token whose key or beta is no number, kD if there is none
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
// A 32 x 32 block of tensor memory in accumulator order: [m][4 n + e] = rows 16 m + g (+ 8), columns 8 n + 2 t4 (+ 1)
__device__ __forceinline__ void load_block(uint32_t t, float (&x)[2][16]) {
    tmem_ld_frag32(t, x[0]);
    tmem_ld_frag32(t + (16u << 16), x[1]);
}

// Diagonal elements of a 16 x 16 block held as two 16 x 8 accumulators: rows g and g + 8, handed to the whole quad.
__device__ __forceinline__ void diagonal_of(const float* n0, const float* n1, int lane, float& d0, float& d1) {
    const int g = lane >> 2, src = (lane & ~3) | (g >> 1);
    const float x0 = (g & 1) ? n0[1] : n0[0], x1 = (g & 1) ? n1[3] : n1[2];
    d0 = __shfl_sync(0xffffffffu, x0, src);
    d1 = __shfl_sync(0xffffffffu, x1, src);
}

// Step-by-step walk of pair p over a warp's block I of the chunk whose rows start at row0, for decays the scaled form cannot
// hold: state columns over the lanes.  First without read-out (walk[t].x = |k_t|^-1 in; out walk[t] = {g_t carried to the block
// end}, and g_t in place of v_t), later with it (walk[t] = {q_t.z_t, W_{t-1} from the block start}; no sums on the way of the
// state any more).  The incoming state is rebuilt from what the earlier blocks published.
template <int kD, int kPairs, Mode kMode, bool kWide, bool kReadout>
__device__ __noinline__ void slow_walk(Smem<kD, kPairs, kMode, kWide>& sm, int p, int row0, int I, int W, int tl) {
    using G = Geo<kD, kPairs, kWide>;
    constexpr int kCols = kD / 32;
    auto column = [&](const uint8_t* tile, int row, int c) {
        const int piece = (c & 63) >> 3;
        const __nv_bfloat16* x = reinterpret_cast<const __nv_bfloat16*>(tile + (c >> 6) * G::kSlab + row * 128 + ((piece ^ (row & 7)) << 4));
        return __bfloat162float(x[c & 7]);
    };
    const BlockPair* bp = &sm.bp[p][row0 / 32];
    float zr[kCols], zi[kCols];
#pragma unroll
    for (int i = 0; i < kCols; i++) zr[i] = zi[i] = 0.f;
    for (int J = 0; J < I; J++) {
        const cplx D31 = bp[J].D31, F = behind(bp, J, I, G::kBlocks);   // (this block's own reference product is one)
        const float* gr = sm.vec[kG] + 2 * p * G::kRow + row0 + 32 * J;
        float ar[kCols], ai[kCols];
#pragma unroll
        for (int i = 0; i < kCols; i++) ar[i] = ai[i] = 0.f;
#pragma unroll 4
        for (int t = 0; t < 32; t++) {
            const cplx w = cmul(D31, {gr[t] + gr[G::kPart + t], gr[G::kRow + t] + gr[G::kRow + G::kPart + t]});
#pragma unroll
            for (int i = 0; i < kCols; i++) {
                const float k = column(sm.k, row0 + 32 * J + t, tl + 32 * i);
                ar[i] += w.r * k;
                ai[i] += w.i * k;
            }
        }
#pragma unroll
        for (int i = 0; i < kCols; i++) {
            const cplx z = cmul(F, {ar[i], ai[i]});
            zr[i] += z.r;
            zi[i] += z.i;
        }
    }
    cplx own = {0.f, 0.f};
#pragma unroll 2
    for (int t = 0; t < 32; t++) {
        const int row = row0 + 32 * I + t;
        const float2 a = sm.dd[p][row], vg = sm.viw[p][row];
        float k[kCols];
#pragma unroll
        for (int i = 0; i < kCols; i++) k[i] = column(sm.k, row, tl + 32 * i);
        cplx gt = {vg.x, vg.y};               // read-out: g_t as the first walk left it
        if (!kReadout) {
            const float be = bits_lo(sm.bs[row]), n = sm.walk[W][t].x;
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
            const cplx z = cmul({zr[i], zi[i]}, {a.x, a.y});
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
    const int row = row0 + 32 * I + tl;
    if (!kReadout) sm.viw[p][row] = make_float2(own.r, own.i);
    // g carried to the block end: times a_{t+1} ... a_31; W_{t-1} = a_0 ... a_{t-1}
    const float2 a = sm.dd[p][row];
    cplx S = {a.x, a.y};
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int from = kReadout ? tl - o : tl + o;
        const cplx other = cshfl(S, from);
        if (from >= 0 && from < 32) S = cmul(other, S);
    }
    cplx V = cshfl(S, kReadout ? tl - 1 : tl + 1);
    if (tl == (kReadout ? 0 : 31)) V = {1.f, 0.f};
    if (!kReadout) own = cmul(V, own);
    __syncwarp();
    sm.walk[W][tl] = make_float4(own.r, own.i, V.r, V.i);
    __syncwarp();
}

// A key row or a beta that is infinite or no number makes the state no number from its token on, whatever the pair.  In the
// products of a block it would reach the tokens before it too (0 x NaN), so its row is emptied and the outputs from it on are set
// apart at the end.  A finite row whose square overflows has |k|^-1 = 0: it neither erases nor adds.  Returns whether this
// lane's row is emptied.
template <int kD, int kPairs, Mode kMode, bool kWide>
__device__ __noinline__ bool empty_bad_rows(Smem<kD, kPairs, kMode, kWide>& sm, int row, int head) {
    using G = Geo<kD, kPairs, kWide>;
    bool number = fabsf(bits_lo(sm.bs[row])) <= 3e38f;
    float ss = 0.f;
    for (int c = 0; c < kD; c++) {
        const float k = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(sm.k + (c >> 6) * G::kSlab + row * 128)[c & 63]);
        number = number && fabsf(k) <= 3.4e38f;
        ss += k * k;
    }
    if (!number) atomicMin(&sm.first_bad[head], row - head * kD);
    const bool empty = !number || !(ss <= 3.4e38f);
    if (empty) {
        for (int s = 0; s < G::kSlabs; s++)
            for (int i = 0; i < 8; i++) *reinterpret_cast<uint4*>(sm.k + s * G::kSlab + row * 128 + 16 * i) = make_uint4(0u, 0u, 0u, 0u);
        sm.bs[row] &= 0xffff0000u;
        sm.bad_rows = 1;
    }
    __syncwarp();
    return empty;
}

// A block runs most of its code once, 100 to 200 KB of straight line, more than an SM's instruction cache: a warp of a call with a block per
// SM spent 44 % of its stalls on waiting for instructions, of a full GPU 13 %.  So what comes at several places, or seldom, is a function
// or a loop: with that and kWide, us before / now: D 64, 523 tokens, H 24, N 16 32.0 / 30.1; B 8, L 2048, H 24, N 4 120 / 112, N 16 245 / 229;
// D 128, 1000 tokens, H 12, N 8 24.5 / 21.5; 12 layers of a 523-token prompt 801 / 751.  (Not faster: the records' loads as a function with a
// loop, or one turn of the look-back for carries and states alike.)
__device__ __noinline__ bool wait_longer(uint64_t* bar, uint32_t parity, int* abort_flag, unsigned long long limit) {
    return mbar_wait_suspend(bar, parity, abort_flag, limit);
}

// A block that gives up stays until its own copies and products have landed (or a limit has passed again): the next one has
// its memory then.  (g_issued, p_issued: warp 0's)
template <typename Smem>
__device__ __noinline__ void leave(Smem& sm, const Args& a, int code, bool q_loaded, int g_issued, bool p_issued, uint32_t tmem) {
    const int W = threadIdx.x >> 5;
    cp_async_wait_all();
    if (W == 0) {
        if ((threadIdx.x & 31) == 0) {
            atomicCAS(a.status, 0, code);
            int never = 0;
            if (!a.withhold) mbar_wait_ns(&sm.full_k, 0, &never, a.wait_ns);
            if (q_loaded && !a.withhold) mbar_wait_ns(&sm.full_q, 0, &never, a.wait_ns);
            if (g_issued) mbar_wait_ns(&sm.mma_g, g_issued - 1, &never, a.wait_ns);
            if (p_issued) mbar_wait_ns(&sm.mma_p, 0, &never, a.wait_ns);
        }
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    if (W == 0) tmem_dealloc(tmem, 128);
}

// resident blocks per SM the registers are cut for
template <int kD, int kPairs, bool kWide = false>
constexpr int kMinBlocks = kWide ? 1 : kPairs >= 4 || kD == 128 ? 2 : 4;

template <int kD, int kPairs, Mode kMode, bool kWide>
__global__ void __launch_bounds__(Geo<kD, kPairs, kWide>::kThreads, kMinBlocks<kD, kPairs, kWide>)
scan_tile_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ Args a) {
    using G = Geo<kD, kPairs, kWide>;
    constexpr int kBlocks = G::kBlocks, kKs = G::kKs, kSplit = G::kSplit, kOwn = G::kOwn, kOwnPairs = G::kOwnPairs;
    constexpr bool kOut = kMode != kLocal, kNeedEnd = kMode != kOutput;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    using S_ = Smem<kD, kPairs, kMode, kWide>;
    S_& sm = *reinterpret_cast<S_*>(smem_raw);
    // warp W: 32-token block W4 of the tile, column tiles S * kOwn ... (the warps of a block meet at the tiles and the inverses only)
    const int tid = threadIdx.x, W = tid >> 5, W4 = W & 3, S = W >> 2, tl = tid & 31, g = tl >> 2, t4 = tl & 3;
    const int hs = W4 / kBlocks, I = W4 % kBlocks, row0 = hs * kD;   // head of the tile, block of the chunk, the chunk's first row
    const int base = 32 * W4, tok = base + tl;
    const int H = a.H, N = a.N, NP = N >> 1, L = a.L;

    if ((smem_u32(smem_raw) & 1023u) != 0) {   // the swizzled tiles need 1024-byte alignment
        if (tid == 0) atomicCAS(a.status, 0, 399);
        return;
    }
    // The records kernel clears the ticket counter.  While there is a block per SM at most the blocks start on their tiles while it is still at
    // work (8 layers of 2 x 41 tokens, N 8: 404 us, 376 so).  Narrow ones need no tickets then (launch_mode()).  Wide ones do, an SM has
    // room for one, and draw them before the records are there: the exchange that clears the counter has come back to its block before that
    // block lets this kernel start, and the additions here take place at the same word of the L2 cache.  It costs 0.1 to 0.5 us
    // of a call (523 tokens, H 24, N 16 29.6 -> 30.1; D 128, 1000 tokens, H 12, N 8 21.4 -> 21.5), the narrow form 30.9 and 23.7.
    const bool early = kMode == kLocal || (kMode == kFused && a.fixed);
    if (kMode == kFused && !early) grid_dependency_wait();
    if (tid == 0) {
        mbar_init(&sm.full_k, 1);
        mbar_init(&sm.full_q, 1);
        mbar_init(&sm.mma_g, 1);
        mbar_init(&sm.mma_p, 1);
        sm.abort_flag = 0;
        sm.bad_rows = 0;
        sm.first_bad[0] = sm.first_bad[1] = kD;
        fence_barrier_init();
        sm.item = kMode == kFused && (kWide || !early) ? atomicAdd(a.ticket, 1) : (int)blockIdx.x;
        sm.stop = kMode == kFused && !early ? *reinterpret_cast<volatile int*>(a.status) : 0;
    }
    __syncthreads();
    if (sm.stop) return;   // an earlier block gave up
    // chunk-major: every block that a block may wait for has an earlier ticket
    const int item = sm.item, hg = item % a.HG, b = (item / a.HG) % a.B, c = item / (a.HG * a.B);
    const int group = kD == 128 ? hg % a.groups : 0, head0 = kD == 128 ? hg / a.groups : 2 * hg;
    const int hd = min(head0 + hs, H - 1);                     // (a tile's second head behind the last one: rows of zeros)
    const bool head_on = head0 + hs < H;
    const int pair0 = group * kPairs, NPB = min(kPairs, NP - pair0);   // the block's pairs
    const size_t unit = ((size_t)b * a.NC + c) * H + hd;       // workspace slot
    const int Lc = min(kD, L - c * kD);
    auto load_tile = [&](uint8_t* to, const CUtensorMap* map, uint64_t* bar) {
        mbar_arrive_expect_tx(bar, G::kTile);
#pragma unroll
        for (int h = 0; h < G::kHeads; h++)
#pragma unroll
            for (int s = 0; s < G::kSlabs; s++) tma_load_4d(to + s * G::kSlab + h * kD * 128, map, bar, 64 * s, head0 + h, c * kD, b);
    };
    if (tid == 0 && !a.withhold) load_tile(sm.k, &tmK, &sm.full_k);
    // the token's dynamics, parked where the results will go (padding: identity)
    // (two warps: fewer pairs beside the inverses; four: none)
    const bool first_warp = kSplit == 1 || S == 0;
    constexpr int kFirstPairs = kSplit == 1 ? kPairs : kSplit == 4 ? 0 : kPairs == 4 ? 1 : 3;
    constexpr int kOtherPairs = kSplit == 4 ? 3 : kPairs - kFirstPairs;
    const int p_lo = first_warp ? 0 : kFirstPairs + (S - 1) * kOtherPairs, p_hi = first_warp ? kFirstPairs : min(kPairs, p_lo + kOtherPairs);
    auto load_records = [&]() {
        const size_t t = (size_t)(tok - row0);
        if (first_warp) {
            if (head_on) cp_async_small<4>(&sm.bs[tok], a.rec_g + unit * kD + t);
            else sm.bs[tok] = 0u;
        }
        const float2* ra = a.rec_a + (unit * (size_t)NP + pair0) * kD + t;
        const uint32_t* rv = a.rec_v + (unit * (size_t)NP + pair0) * kD + t;
#pragma unroll
        for (int p = 0; p < kPairs; p++) {
            if (p < p_lo || p >= p_hi) continue;
            if (p < NPB && head_on) {
                cp_async_small<8>(&sm.dd[p][tok], ra + p * kD);
                cp_async_small<4>(&sm.viw[p][tok], rv + p * kD);
            } else {
                sm.dd[p][tok] = make_float2(1.f, 0.f);
                sm.viw[p][tok] = make_float2(0.f, 0.f);
            }
        }
        cp_async_commit();
    };
    if (!early) load_records();
    if (W == 0) tmem_alloc(&sm.tmem, 128);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sm.tmem, lane_base = tmem + ((uint32_t)base << 16);
    const uint32_t kt = smem_u32(sm.k), qt = smem_u32(sm.q);
    // warp 0: all 128 rows of tile `rows` against those of K
    auto gram = [&](uint32_t rows, uint64_t* bar) {
        constexpr uint32_t idesc = umma_idesc_bf16(128, 128, false, false);
        uint32_t x = desc_lo_sw128(rows, 16), k = desc_lo_sw128(kt, 16);
        tc_fence_after();
#pragma unroll
        for (int j = 0; j < kKs; j++) {
            umma_bf16_elect(tmem, x, k, idesc, j);
            const uint32_t step = (j & 3) == 3 ? 2 + (G::kSlab >> 4) - 8 : 2;
            x += step;
            k += step;
        }
        umma_commit_elect(bar);
    };
    auto wait = [&](uint64_t* bar, uint32_t parity) {
        return __all_sync(0xffffffffu, mbar_try_wait_nohint(bar, parity) || wait_longer(bar, parity, &sm.abort_flag, a.wait_ns));
    };
    int g_issued = 0;                          // (warp 0) products G: a second one where key rows have been emptied
    bool p_issued = false;
    auto give_up = [&](int code, bool q_loaded) { leave(sm, a, code, q_loaded, g_issued, p_issued, tmem); };

    bool ok = wait(&sm.full_k, 0);
    if (W == 0 && ok) { gram(kt, &sm.mma_g); g_issued = 1; }
    // the token's dynamics, from the kernel before this one (its launch let this one start early; no __ldg here: loads
    // that claim the data constant may be moved above the wait)
    if (early) grid_dependency_wait();
    grid_launch_dependents();
    if (early) load_records();
    cp_async_wait_all();
    {
        auto some = [&](auto count, int p0) {
            constexpr int kW = decltype(count)::value;
            cplx at[kW], vg[kW];
            BlockPair bp[kW];
#pragma unroll
            for (int w = 0; w < kW; w++) {
                const int p = min(p0 + w, p_hi - 1);   // (a warp's last three may be two: it forms one twice)
                const float2 x = sm.dd[p][tok];
                const uint32_t y = __float_as_uint(sm.viw[p][tok].x);
                at[w] = {x.x, x.y};
                vg[w] = {bits_lo(y), bits_hi(y)};
            }
            const int slow = (scalings<kW, kD == 64 && kPairs == 4 && kW == 1>(at, vg, tl, bp) << p0) & ((1 << p_hi) - 1);
#pragma unroll
            for (int w = 0; w < kW; w++) {
                if (p0 + w >= p_hi) break;
                sm.viw[p0 + w][tok] = make_float2(vg[w].r, vg[w].i);
                sm.dd[p0 + w][tok] = make_float2(at[w].r, at[w].i);
                if (tl == 0) sm.bp[p0 + w][W4] = bp[w];
            }
            return slow;
        };
        int slow = 0;
        if constexpr (kSplit == 1) {
            slow = some(std::integral_constant<int, kPairs>(), 0);
        } else if constexpr (kPairs == 8) {    // (three at a time, whoever has how many)
#pragma unroll 1
            for (int p0 = p_lo; p0 < p_hi; p0 += 3) slow |= some(std::integral_constant<int, 3>(), p0);
        } else {
            slow = first_warp ? some(std::integral_constant<int, kFirstPairs>(), 0) : some(std::integral_constant<int, kOtherPairs>(), kFirstPairs);
        }
        if (tl == 0) sm.slow[S][W4] = slow;
        __syncwarp();
    }
    ok = ok && wait(&sm.mma_g, 0);
    tc_fence_after();

    // ---- G: diagonal block, |k|^-1, inverses
    float cc[4], bn[4], nrm[4];               // c_t, beta_t n_t, n_t of rows g, g + 8, g + 16, g + 24
    float T11[8], T22[8], M21[8];
    if (first_warp) {
        float acc[2][16], kk[4];
        load_block(lane_base + base, acc);
        tmem_ld_wait(acc[0]);
        tmem_ld_wait(acc[1]);
        diagonal_of(&acc[0][0], &acc[0][4], tl, kk[0], kk[1]);
        diagonal_of(&acc[1][8], &acc[1][12], tl, kk[2], kk[3]);
        __syncwarp();
        bool number = fabsf(bits_lo(sm.bs[tok])) <= 3e38f;   // (false for NaN)
#pragma unroll
        for (int r = 0; r < 4; r++) number = number && kk[r] <= 3.4e38f;
        if (ok && !__all_sync(0xffffffffu, number)) {   // (not from tensor memory that nothing has been written to)
            const uint32_t bad = __ballot_sync(0xffffffffu, empty_bad_rows<kD, kPairs, kMode, kWide>(sm, tok, hs));
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const int row = 16 * m + g + 8 * ((i >> 1) & 1), col = 8 * (i >> 2) + 2 * t4 + (i & 1);
                    if (((bad >> row) | (bad >> col)) & 1) acc[m][i] = 0.f;
                }
#pragma unroll
            for (int r = 0; r < 4; r++)
                if ((bad >> (8 * r + g)) & 1) kk[r] = 0.f;
        }
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const float be = bits_lo(sm.bs[base + 8 * r + g]);
            nrm[r] = rsqrtf(kk[r] + kEps);
            bn[r] = be * nrm[r];
            cc[r] = bn[r] * nrm[r];
        }
        // M's diagonal 16 x 16 blocks, as 8 x 8: the strictly lower part of two, and the one below
        auto& sc = sm.scr[W4];
#pragma unroll
        for (int m = 0; m < 2; m++) {
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int col = 2 * t4 + e;
                sc.tri[2 * m][12 * col + g] = g > col ? cc[2 * m] * acc[m][8 * m + e] : 0.f;
                sc.tri[2 * m + 1][12 * col + g] = g > col ? cc[2 * m + 1] * acc[m][8 * m + 4 + 2 + e] : 0.f;
            }
            *reinterpret_cast<float2*>(&sc.low[m][8 * g + 2 * t4]) =
                make_float2(cc[2 * m + 1] * acc[m][8 * m + 2], cc[2 * m + 1] * acc[m][8 * m + 3]);
        }
#pragma unroll
        for (int i = 0; i < 8; i++) M21[i] = cc[2 + ((i >> 1) & 1)] * acc[1][i];
        if (kSplit > 1) {
            sc.m21[0][tl] = make_float4(M21[0], M21[1], M21[2], M21[3]);
            sc.m21[1][tl] = make_float4(M21[4], M21[5], M21[6], M21[7]);
            if (t4 == 0) {
#pragma unroll
                for (int r = 0; r < 4; r++) sc.nrm[8 * r + g] = nrm[r];
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
        float4* row = reinterpret_cast<float4*>(sc.t[tl]);
#pragma unroll
        for (int j = 0; j < 4; j++) row[j] = make_float4(R[2 * j].x, R[2 * j].y, R[2 * j + 1].x, R[2 * j + 1].y);
        __syncwarp();
    }
    if (kSplit > 1) {
        __syncthreads();
        if (!first_warp) {
#pragma unroll
            for (int r = 0; r < 4; r++) {
                nrm[r] = sm.scr[W4].nrm[8 * r + g];
                bn[r] = bits_lo(sm.bs[base + 8 * r + g]) * nrm[r];
                cc[r] = bn[r] * nrm[r];
            }
            const float4 x = sm.scr[W4].m21[0][tl], y = sm.scr[W4].m21[1][tl];
            M21[0] = x.x; M21[1] = x.y; M21[2] = x.z; M21[3] = x.w;
            M21[4] = y.x; M21[5] = y.y; M21[6] = y.z; M21[7] = y.w;
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float2 x = *reinterpret_cast<const float2*>(&sm.scr[W4].t[g + 8 * (i & 1)][2 * t4 + 8 * (i >> 1)]);
        const float2 y = *reinterpret_cast<const float2*>(&sm.scr[W4].t[16 + g + 8 * (i & 1)][2 * t4 + 8 * (i >> 1)]);
        T11[2 * i] = x.x; T11[2 * i + 1] = x.y;
        T22[2 * i] = y.x; T22[2 * i + 1] = y.y;
    }
    // (block decays of all warps are in shared memory; the scratch has been read: the Q tile comes in its place)
    fence_proxy_async();
    tc_fence_before();
    if (!__syncthreads_and(ok)) {
        give_up(201, false);
        return;
    }
    tc_fence_after();
    if (kOut && tid == 0 && !a.withhold) load_tile(sm.q, &tmQ, &sm.full_q);
    if (sm.bad_rows) {   // G without the emptied rows
        if (W == 0) { gram(kt, &sm.mma_g); g_issued = 2; }
        ok = wait(&sm.mma_g, 1);
        tc_fence_after();
    }
    // ---- G against the earlier blocks
    constexpr int kEarlier = kBlocks - 1;
    float M[kEarlier][2][16];
#pragma unroll
    for (int J = 0; J < kEarlier; J++)
        if (J < I) load_block(lane_base + row0 + 32 * J, M[J]);
#pragma unroll
    for (int J = 0; J < kEarlier; J++) {
        tmem_ld_wait(M[J][0]);
        tmem_ld_wait(M[J][1]);
    }
    tc_fence_before();   // (P comes in G's place, behind the next barrier)

    const int comp = t4 & 1;
    auto tile = [&](int q) { return S * kOwn + q; };
    // pair of the lane's component in tile q
    auto pair_of = [&](int q) { return 2 * tile(q) + (t4 >> 1); };
    // this lane's component of a row into / a fragment's two tokens out of a solution
    auto put = [&](int v, int q, int r, float x) {
        float* to = sm.vec[v] + (2 * pair_of(q) + comp) * G::kRow + base + 8 * r + g;
        const float hi = tf32_hi(x);
        to[0] = hi;
        to[G::kPart] = x - hi;
    };
    const float* frag_at = sm.vec[0] + (g & 1) * G::kPart + 2 * t4;
    auto get = [&](int v, int q, int row) {
        const int cmp = 4 * tile(q) + (g >> 1);
        return *reinterpret_cast<const float2*>(frag_at + v * (2 * G::kPart) + cmp * G::kRow + row);
    };
    // sums of a tile's accumulators: rows g and g + 8, this lane's component
    auto sum_lo = [](const float (&d)[4], const float (&e)[4]) { return (d[0] + d[1]) + (e[0] + e[1]); };
    auto sum_hi = [](const float (&d)[4], const float (&e)[4]) { return (d[2] + d[3]) + (e[2] + e[3]); };
    // complex factor times the lane's component; `other` is the other component of the same value
    auto rotate = [&](cplx f, float own, float other) { return __fmaf_rn(f.r, own, __fmul_rn(comp ? f.i : -f.i, other)); };
    auto other_of = [](float x) { return __shfl_xor_sync(0xffffffffu, x, 1); };
    // block J's scaled sum times D31, then times f (behind()), this lane's component
    auto carried = [&](cplx d31, cplx f, float own) {
        const float other = other_of(own), i = comp ? d31.i : -d31.i;
        return rotate(f, __fmaf_rn(d31.r, own, __fmul_rn(i, other)), __fmaf_rn(d31.r, other, -__fmul_rn(i, own)));
    };

    // x <- (I + M_own)^-1 x, all column tiles; published as vector v
    auto solve = [&](int v, float (&x)[kOwn][4]) {
        auto apply = [&](const float (&f)[8], int row, float (&lo)[kOwn], float (&hi)[kOwn]) {
            __syncwarp();
            float d[kOwn][4], e[kOwn][4];
#pragma unroll
            for (int n = 0; n < 2; n++) {
                const Split s = split(f + 4 * n);
#pragma unroll
                for (int q = 0; q < kOwn; q++) {
                    if (n == 0) mma_split<true>(d[q], e[q], s, get(v, q, base + row));
                    else mma_split<false>(d[q], e[q], s, get(v, q, base + row + 8));
                }
            }
#pragma unroll
            for (int q = 0; q < kOwn; q++) {
                lo[q] = sum_lo(d[q], e[q]);
                hi[q] = sum_hi(d[q], e[q]);
            }
            __syncwarp();
        };
        auto publish = [&](int r) {
#pragma unroll
            for (int q = 0; q < kOwn; q++) {
                put(v, q, r, x[q][r]);
                put(v, q, r + 1, x[q][r + 1]);
            }
        };
        float lo[kOwn], hi[kOwn];
        publish(0);
        apply(T11, 0, lo, hi);
#pragma unroll
        for (int q = 0; q < kOwn; q++) { x[q][0] = lo[q]; x[q][1] = hi[q]; }
        publish(0);
        apply(M21, 0, lo, hi);
#pragma unroll
        for (int q = 0; q < kOwn; q++) { x[q][2] -= lo[q]; x[q][3] -= hi[q]; }
        publish(2);
        apply(T22, 16, lo, hi);
#pragma unroll
        for (int q = 0; q < kOwn; q++) { x[q][2] = lo[q]; x[q][3] = hi[q]; }
        publish(2);
    };
    // sums over block J's tokens of a 32 x 32 block times the vectors v .. v + kV - 1, rows g + 8 r
    auto times = [&](const float (&x)[2][16], auto kVectors, int v, int J, float* out) {
        constexpr int kV = decltype(kVectors)::value;
        // (accumulators of their own for the lo parts where there are few chains of products beside each other)
        constexpr bool kApart = kV * (G::kTiles / G::kNarrow) < 4;   // (the same sums, and so the same bits, however many warps share the tiles)
        float d[kV][kOwn][2][4], e[kApart ? kV : 1][kOwn][2][4];
#pragma unroll
        for (int n = 0; n < 4; n++) {
            float2 f[kV][kOwn];
#pragma unroll
            for (int w = 0; w < kV; w++)
#pragma unroll
                for (int q = 0; q < kOwn; q++) f[w][q] = get(v + w, q, row0 + 32 * J + 8 * n);
#pragma unroll
            for (int m = 0; m < 2; m++) {
                const Split s = split(&x[m][4 * n]);
#pragma unroll
                for (int w = 0; w < kV; w++)
#pragma unroll
                    for (int q = 0; q < kOwn; q++) {
                        if constexpr (kApart) {
                            if (n == 0) mma_split<true>(d[w][q][m], e[w][q][m], s, f[w][q]);
                            else mma_split<false>(d[w][q][m], e[w][q][m], s, f[w][q]);
                        } else {
                            if (n == 0) mma_tf32<true>(d[w][q][m], s.lo[0], s.lo[1], s.lo[2], s.lo[3], f[w][q]);
                            else mma_tf32<false>(d[w][q][m], s.lo[0], s.lo[1], s.lo[2], s.lo[3], f[w][q]);
                            mma_tf32<false>(d[w][q][m], s.hi[0], s.hi[1], s.hi[2], s.hi[3], f[w][q]);
                        }
                    }
            }
        }
#pragma unroll
        for (int w = 0; w < kV; w++)
#pragma unroll
            for (int q = 0; q < kOwn; q++)
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    const float(&x0)[4] = d[w][q][m];
                    float lo = x0[0] + x0[1], hi = x0[2] + x0[3];
                    if constexpr (kApart) {
                        const float(&x1)[4] = e[w][q][m];
                        lo += x1[0] + x1[1];
                        hi += x1[2] + x1[3];
                    }
                    out[(w * kOwn + q) * 4 + 2 * m] = lo;
                    out[(w * kOwn + q) * 4 + 2 * m + 1] = hi;
                }
    };
    using One = std::integral_constant<int, 1>;
    using Two = std::integral_constant<int, 2>;
    auto chain_wait = [&](int J) {
        asm volatile("bar.sync %0, %1;" ::"r"(1 + (S * G::kHeads + hs) * kEarlier + J), "r"(32 * (kBlocks - J)) : "memory");
    };
    auto chain_pass = [&]() {
        if (I < kEarlier)
            asm volatile("bar.arrive %0, %1;" ::"r"(1 + (S * G::kHeads + hs) * kEarlier + I), "r"(32 * (kBlocks - I)) : "memory");
        __syncwarp();
    };

    int slow = 0;                              // of this warp's pairs
#pragma unroll
    for (int i = 0; i < kSplit; i++) slow |= sm.slow[i][W4];
    slow &= ((1 << kOwnPairs) - 1) << (kOwnPairs * S);
    // ---- g: the chain over the blocks of the chunk
    float gx[kOwn][4];
    {
#pragma unroll
        for (int q = 0; q < kOwn; q++)
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const float2 e = sm.viw[pair_of(q)][base + 8 * r + g];
                gx[q][r] = __fmul_rn(bn[r], comp ? e.y : e.x);
            }
#pragma unroll
        for (int J = 0; J < kEarlier; J++)
            if (J < I) {
                float s[kOwn][4];
                chain_wait(J);
                times(M[J], One(), kG, J, &s[0][0]);
#pragma unroll
                for (int q = 0; q < kOwn; q++) {
                    const BlockPair* bp = &sm.bp[pair_of(q)][row0 / 32];
                    const cplx D31 = bp[J].D31, F = behind(bp, J, I, kBlocks);
#pragma unroll
                    for (int r = 0; r < 4; r++) gx[q][r] = __fmaf_rn(-cc[r], carried(D31, F, s[q][r]), gx[q][r]);
                }
            }
        solve(kG, gx);
        if (slow != 0) {                       // decays beyond the scaled form: step by step
            __syncwarp();
            if (t4 == 0) {
#pragma unroll
                for (int r = 0; r < 4; r++) sm.walk[W][8 * r + g].x = nrm[r];
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < kOwn; q++)
#pragma unroll 1
                for (int s = 0; s < 2; s++)
                    if ((slow >> (2 * tile(q) + s)) & 1) {
                        slow_walk<kD, kPairs, kMode, kWide, false>(sm, 2 * tile(q) + s, row0, I, W, tl);
                        if ((t4 >> 1) == s) {
#pragma unroll
                            for (int r = 0; r < 4; r++) {
                                const float4 x = sm.walk[W][8 * r + g];
                                put(kG, q, r, comp ? x.y : x.x);
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
        chain_pass();
    }
    __syncthreads();
    tc_fence_after();
    bool q_here = true;
    if (kOut && W == 0) {
        q_here = wait(&sm.full_q, 0);
        if (q_here) { gram(qt, &sm.mma_p); p_issued = true; }
    }

    // product of K^T (this warp's 32 columns of its head) with vector v, the blocks' sums carried to the chunk end (g) or as they
    // are (h): rows 16 m + g (+ 8) of component t4 of each tile
    auto k_transposed = [&](int v, float (&z)[kOwn][2][2]) {
#pragma unroll
        for (int q = 0; q < kOwn; q++)
#pragma unroll
            for (int m = 0; m < 2; m++) z[q][m][0] = z[q][m][1] = 0.f;
#pragma unroll
        for (int J = 0; J < kBlocks; J++) {
            float d[kOwn][2][2][4];
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    uint32_t ka[4];
                    ldsm_x4_trans(col_frag<G::kSlab>(kt, row0 + 32 * J + 16 * h, 32 * I + 16 * m, tl), ka);
#pragma unroll
                    for (int q = 0; q < kOwn; q++) {
                        const float2 f0 = get(v, q, row0 + 32 * J + 16 * h), f1 = get(v, q, row0 + 32 * J + 16 * h + 8);
                        if (h == 0) {
                            mma_tf32<true>(d[q][m][0], bits_lo(ka[0]), bits_hi(ka[0]), bits_lo(ka[1]), bits_hi(ka[1]), f0);
                            mma_tf32<true>(d[q][m][1], bits_lo(ka[2]), bits_hi(ka[2]), bits_lo(ka[3]), bits_hi(ka[3]), f1);
                        } else {
                            mma_tf32<false>(d[q][m][0], bits_lo(ka[0]), bits_hi(ka[0]), bits_lo(ka[1]), bits_hi(ka[1]), f0);
                            mma_tf32<false>(d[q][m][1], bits_lo(ka[2]), bits_hi(ka[2]), bits_lo(ka[3]), bits_hi(ka[3]), f1);
                        }
                    }
                }
#pragma unroll
            for (int q = 0; q < kOwn; q++) {
                const BlockPair* bp = &sm.bp[pair_of(q)][row0 / 32];
                const cplx D31 = bp[J].D31, F = behind(bp, J, kBlocks, kBlocks);
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    const float x0 = sum_lo(d[q][m][0], d[q][m][1]), x1 = sum_hi(d[q][m][0], d[q][m][1]);
                    z[q][m][0] += v == kG ? carried(D31, F, x0) : x0;
                    z[q][m][1] += v == kG ? carried(D31, F, x1) : x1;
                }
            }
        }
    };
    auto chunk_decay = [&](int p) {
        const BlockPair* bp = &sm.bp[p][row0 / 32];
        cplx w = bp[0].A;
#pragma unroll
        for (int J = 1; J < kBlocks; J++) w = cmul(bp[J].A, w);
        return w;
    };

    // ---- z at the chunk end; the carry (a thread has a column of its warp's pairs: base + tl = 32 I + tl of head hs)
    const int col = 32 * I + tl;
    auto state_at = [&](const float* s, size_t u, int i) { return s + (u * N + 2 * (pair0 + kOwnPairs * S + i)) * kD + col; };
    const int own_pairs = head_on ? max(0, min(kOwnPairs, NPB - kOwnPairs * S)) : 0;
    if (kNeedEnd) {
        float z[kOwn][2][2];
        k_transposed(kG, z);
#pragma unroll
        for (int q = 0; q < kOwn; q++)
#pragma unroll
            for (int m = 0; m < 2; m++) {
                sm.zl[2 * pair_of(q) + comp][base + 16 * m + g] = z[q][m][0];
                sm.zl[2 * pair_of(q) + comp][base + 16 * m + g + 8] = z[q][m][1];
            }
        __syncwarp();
        const bool whole = Lc == kD;           // the reference's zero padding wipes state and decay (ssd.py:60-67)
        const bool bad = sm.first_bad[hs] < kD;
        float lr[kOwnPairs], li[kOwnPairs];
        cplx gam[kOwnPairs];
#pragma unroll
        for (int i = 0; i < kOwnPairs; i++) {
            const int p = kOwnPairs * S + i;
            gam[i] = chunk_decay(p);
            gam[i] = whole ? cplx{bfr(gam[i].r), bfr(gam[i].i)} : cplx{0.f, 0.f};
            lr[i] = !whole ? 0.f : bad ? kNotANumber : bfr(sm.zl[2 * p][base + tl]);
            li[i] = !whole ? 0.f : bad ? kNotANumber : bfr(sm.zl[2 * p + 1][base + tl]);
            if (kMode == kLocal && i < own_pairs) {
                float* s = a.ws_state + (unit * N + 2 * (pair0 + p)) * kD + col;
                s[0] = lr[i];
                s[kD] = li[i];
                if (col == 0) *reinterpret_cast<float2*>(a.ws_gamma + unit * N + 2 * (pair0 + p)) = make_float2(gam[i].r, gam[i].i);
            }
        }
        if (kMode == kFused) {
            // slots of this column's pairs: word (slot + i) kD, gamma word slot + i; a chunk back: - H NP slots
            const size_t slot = unit * NP + pair0 + kOwnPairs * S, back = (size_t)H * NP;
            uint32_t* zs = a.chunks + slot * kD + col;
            uint64_t* cs = a.carries + slot * kD + col;
            const uint32_t* gs = a.gammas + slot;
            float sr[kOwnPairs], si[kOwnPairs];
            auto from_start = [&]() {
#pragma unroll
                for (int i = 0; i < kOwnPairs; i++) {
                    sr[i] = si[i] = 0.f;
                    if (i < own_pairs && a.h0) {
                        const float* s = state_at(a.h0, (size_t)b * H + hd, i);
                        sr[i] = s[0];
                        si[i] = s[kD];
                    }
                }
            };
            // the carry out of the chunk n back: whether it is there for the whole warp, and then what it is
            auto carry_of = [&](int n) {
                uint64_t w[kOwnPairs];
                bool here = true;
#pragma unroll
                for (int i = 0; i < kOwnPairs; i++) {
                    w[i] = i < own_pairs ? get_word(cs - back * kD * n + i * kD) : 1;
                    here = here && w[i] != 0;
                }
                if (!__all_sync(0xffffffffu, here)) return false;
#pragma unroll
                for (int i = 0; i < kOwnPairs; i++) {
                    sr[i] = __uint_as_float(word_lo(w[i]));
                    si[i] = __uint_as_float(word_hi(w[i]));
                }
                return true;
            };
            bool here = true;
            if (c == 0) {
                from_start();
            } else if (!carry_of(1)) {
                // others may come through this chunk before its own carry does
                if (c + 1 < a.NC) {
#pragma unroll
                    for (int i = 0; i < kOwnPairs; i++)
                        if (i < own_pairs) {
                            put_word32(zs + i * kD, bf16_pair({lr[i], li[i]}));
                            if (col == 0) put_word32(a.gammas + slot + i, bf16_pair(gam[i]));
                        }
                }
                // the nearest chunk before this one whose carry-out is known (there at the latest when all are), ...
                int n = 2;
                while (n <= c) {                  // (a lane asks for one chunk's first word)
                    const uint32_t some = __ballot_sync(0xffffffffu, n + tl <= c && get_word(a.carries + (slot - back * (n + tl)) * kD) != 0);
                    if (some == 0) { n += 32; continue; }
                    n += __ffs(some) - 1;
                    if (carry_of(n)) break;
                    n++;                          // (it is being written)
                }
                if (n > c) { n = c + 1; from_start(); }
                // ... then s <- gamma s + z over the chunks up to this one as they come (or again from a carry that has come
                // meanwhile: the same bits)
                constexpr int kBatch = 16 / kOwnPairs;
                const unsigned long long t0 = global_ns();
#pragma unroll 1
                for (n--; n > 0 && here; n -= kBatch) {
                    uint32_t z[kBatch][kOwnPairs];
                    // (lane: chunk tl / kOwnPairs of the batch, pair tl % kOwnPairs)
                    uint32_t gw = get_word32(gs - back * max(n - min(tl / kOwnPairs, kBatch - 1), 1) + min(tl % kOwnPairs, max(own_pairs, 1) - 1));
#pragma unroll
                    for (int k = 0; k < kBatch; k++)
#pragma unroll
                        for (int i = 0; i < kOwnPairs; i++)
                            z[k][i] = i < own_pairs ? get_word32(zs - back * max(n - k, 1) * kD + i * kD) : 1u;
#pragma unroll
                    for (int k = 0; k < kBatch; k++) {
                        if (n - k <= 0 || !here) break;
                        for (;;) {
                            bool all = true;
                            uint32_t gj[kOwnPairs];
#pragma unroll
                            for (int i = 0; i < kOwnPairs; i++) {
                                gj[i] = __shfl_sync(0xffffffffu, gw, k * kOwnPairs + i);
                                all = all && z[k][i] != 0 && gj[i] != 0;
                            }
                            if (__all_sync(0xffffffffu, all)) {
#pragma unroll
                                for (int i = 0; i < kOwnPairs; i++) {
                                    const cplx zj = pair_of_word(z[k][i]), g1 = pair_of_word(gj[i]);
                                    const float nr = next_re(g1, sr[i], si[i], zj.r);
                                    si[i] = next_im(g1, sr[i], si[i], zj.i);
                                    sr[i] = nr;
                                }
                                break;
                            }
                            if (carry_of(n - k)) break;
                            __nanosleep(20);
                            if (__any_sync(0xffffffffu, global_ns() - t0 > 20000)) {   // (rarely: a trip to memory each)
                                const int gave_up = *reinterpret_cast<volatile int*>(a.status);
                                if (__any_sync(0xffffffffu, gave_up != 0 || global_ns() - t0 > a.wait_ns)) { here = false; break; }
                            }
                            const uint32_t again = get_word32(gs - back * (n - k) + min(tl % kOwnPairs, max(own_pairs, 1) - 1));
                            if (tl / kOwnPairs == k) gw = again;
#pragma unroll
                            for (int i = 0; i < kOwnPairs; i++) z[k][i] = i < own_pairs ? get_word32(zs - back * (n - k) * kD + i * kD) : 1u;
                        }
                    }
                }
            }
            ok = ok && here;
#pragma unroll
            for (int i = 0; i < kOwnPairs; i++) {
                const int p = kOwnPairs * S + i;
                sm.r0[hs][2 * p][col] = __float2bfloat16_rn(sr[i]);
                sm.r0[hs][2 * p + 1][col] = __float2bfloat16_rn(si[i]);
                if (i < own_pairs) {
                    const float nr = next_re(gam[i], sr[i], si[i], lr[i]), ni = next_im(gam[i], sr[i], si[i], li[i]);
                    if (c + 1 < a.NC) {
                        put_word(cs + i * kD, carry_word(nr, ni));
                    } else if (a.final_state) {
                        float* to = a.final_state + (((size_t)b * H + hd) * N + 2 * (pair0 + p)) * kD + col;
                        to[0] = nr;
                        to[kD] = ni;
                    }
                }
            }
            if (!__syncthreads_and(ok)) {
                give_up(203, true);
                return;
            }
        }
    } else {
        grid_dependency_wait();   // the pass before; the records are there: it has waited for them before this launch
        float sr[kOwnPairs], si[kOwnPairs];
#pragma unroll
        for (int i = 0; i < kOwnPairs; i++) {
            sr[i] = si[i] = 0.f;
            if (i < own_pairs && (!a.from_chunks || a.h0)) {
                const float* s = a.from_chunks ? state_at(a.h0, (size_t)b * H + hd, i) : state_at(a.ws_state, unit, i);
                sr[i] = __ldcg(s);
                si[i] = __ldcg(s + kD);
            }
        }
        auto into_chunk = [&]() {
#pragma unroll
            for (int i = 0; i < kOwnPairs; i++) {
                const int p = kOwnPairs * S + i;
                sm.r0[hs][2 * p][col] = __float2bfloat16_rn(sr[i]);
                sm.r0[hs][2 * p + 1][col] = __float2bfloat16_rn(si[i]);
            }
        };
        if (a.from_chunks) {      // s <- gamma s + z over the chunks before, in the carry pass's order
            // (the last chunk's own step too, where the final state is wanted)
            const int chunks = c + (c + 1 == a.NC && a.final_state ? 1 : 0);
            constexpr int kBatch = 8 / kOwnPairs;
#pragma unroll 1
            for (int c0 = 0; c0 < chunks; c0 += kBatch) {
                float l[kBatch][kOwnPairs][2];
                float2 gm[kBatch][kOwnPairs];
#pragma unroll
                for (int k = 0; k < kBatch; k++)
#pragma unroll
                    for (int i = 0; i < kOwnPairs; i++)
                        if (i < own_pairs) {
                            const size_t u = ((size_t)b * a.NC + min(c0 + k, chunks - 1)) * H + hd;
                            const float* z = state_at(a.ws_state, u, i);
                            l[k][i][0] = __ldcg(z);
                            l[k][i][1] = __ldcg(z + kD);
                            gm[k][i] = __ldcg(reinterpret_cast<const float2*>(a.ws_gamma + u * N + 2 * (pair0 + kOwnPairs * S + i)));
                        }
#pragma unroll
                for (int k = 0; k < kBatch; k++) {
                    if (c0 + k >= chunks) break;
                    if (c0 + k == c) into_chunk();
#pragma unroll
                    for (int i = 0; i < kOwnPairs; i++)
                        if (i < own_pairs) {
                            const cplx gam = {gm[k][i].x, gm[k][i].y};
                            const float nr = next_re(gam, sr[i], si[i], l[k][i][0]);
                            si[i] = next_im(gam, sr[i], si[i], l[k][i][1]);
                            sr[i] = nr;
                        }
                }
            }
            if (chunks > c) {
#pragma unroll
                for (int i = 0; i < kOwnPairs; i++)
                    if (i < own_pairs) {
                        float* to = a.final_state + (((size_t)b * H + hd) * N + 2 * (pair0 + kOwnPairs * S + i)) * kD + col;
                        to[0] = sr[i];
                        to[kD] = si[i];
                    }
            } else {
                into_chunk();
            }
        } else {
            into_chunk();
        }
        __syncthreads();
    }
    if (kMode == kLocal) {
        tc_fence_before();
        if (!__syncthreads_and(ok)) give_up(202, false);
        else if (W == 0) tmem_dealloc(tmem, 128);
        return;
    }

    // rows of a tile times r_0: the accumulators of tiles 2 Q (even columns) and 2 Q + 1 (odd ones); with |row|^2 where asked for
    constexpr int kQ = (kOwn + 1) / 2;
    auto times_r0 = [&](uint32_t rows, float (&x)[kOwn][4], float* ss) {
        float d[kQ][2][4], qd[2][2][4];
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                qd[m][0][e] = qd[m][1][e] = 0.f;
#pragma unroll
                for (int Q = 0; Q < kQ; Q++) d[Q][m][e] = 0.f;
            }
        // column g: component (g >> 1) of tile 2 Q + (g & 1)
        const uint32_t* r[kQ];
#pragma unroll
        for (int Q = 0; Q < kQ; Q++) {
            const int q = min(2 * Q + (g & 1), kOwn - 1);
            r[Q] = reinterpret_cast<const uint32_t*>(&sm.r0[hs][4 * tile(q) + (g >> 1)][2 * t4]);
        }
#pragma unroll
        for (int ks = 0; ks < kKs; ks++) {
            uint32_t ra[2][4];
            ldsm_x4(row_frag<G::kSlab>(rows, base, ks, tl), ra[0]);
            ldsm_x4(row_frag<G::kSlab>(rows, base + 16, ks, tl), ra[1]);
#pragma unroll
            for (int m = 0; m < 2; m++) {
#pragma unroll
                for (int Q = 0; Q < kQ; Q++) mma_bf16_m16n8k16(d[Q][m], ra[m], r[Q][8 * ks], r[Q][8 * ks + 4]);
                if (ss) {
                    mma_bf16_m16n8k16(qd[m][0], ra[m], ra[m][0], ra[m][2]);
                    mma_bf16_m16n8k16(qd[m][1], ra[m], ra[m][1], ra[m][3]);
                }
            }
        }
#pragma unroll
        for (int q = 0; q < kOwn; q++)
#pragma unroll
            for (int r4 = 0; r4 < 4; r4++) x[q][r4] = d[q >> 1][r4 >> 1][2 * (r4 & 1) + (q & 1)];
        if (ss) {
            diagonal_of(qd[0][0], qd[0][1], tl, ss[0], ss[1]);
            diagonal_of(qd[1][0], qd[1][1], tl, ss[2], ss[3]);
        }
    };
    // ---- h: right-hand sides c_t k_t.r_0, the same chain
    {
        float hx[kOwn][4];
        times_r0(kt, hx, nullptr);
#pragma unroll
        for (int q = 0; q < kOwn; q++)
#pragma unroll
            for (int r = 0; r < 4; r++) hx[q][r] = __fmul_rn(hx[q][r], cc[r]);
#pragma unroll
        for (int J = 0; J < kEarlier; J++)
            if (J < I) {
                float s[kOwn][4];
                chain_wait(J);
                times(M[J], One(), kH, J, &s[0][0]);
#pragma unroll
                for (int q = 0; q < kOwn; q++)
#pragma unroll
                    for (int r = 0; r < 4; r++) hx[q][r] = __fmaf_rn(-cc[r], s[q][r], hx[q][r]);
            }
        solve(kH, hx);
        chain_pass();
    }

    // ---- |q|^-1, q.r_0; read-out: P against the block itself and the earlier ones
    if (W != 0) q_here = wait(&sm.full_q, 0);
    q_here = q_here && wait(&sm.mma_p, 0);
    tc_fence_after();
    float mq[4], rho[kOwn][4];
    times_r0(qt, rho, mq);
#pragma unroll
    for (int r = 0; r < 4; r++) mq[r] = rsqrtf(mq[r] + kEps);
    float oz[kOwn][4], pd[4];
#pragma unroll
    for (int q = 0; q < kOwn; q++)
#pragma unroll
        for (int r = 0; r < 4; r++) oz[q][r] = 0.f;
#pragma unroll 1
    for (int J = I; J >= 0; J--) {
        const bool diag = J == I;
        float x[2][16];
        load_block(lane_base + row0 + 32 * J, x);
        tmem_ld_wait(x[0]);
        tmem_ld_wait(x[1]);
        if (diag) {
            diagonal_of(&x[0][0], &x[0][4], tl, pd[0], pd[1]);
            diagonal_of(&x[1][8], &x[1][12], tl, pd[2], pd[3]);
#pragma unroll
            for (int m = 0; m < 2; m++)        // strictly lower (the diagonal enters with g itself below)
#pragma unroll
                for (int i = 0; i < 16; i++)
                    if (16 * m + g + 8 * ((i >> 1) & 1) <= 8 * (i >> 2) + 2 * t4 + (i & 1)) x[m][i] = 0.f;
        }
        float s[2][kOwn][4];
        times(x, Two(), kG, J, &s[0][0][0]);
#pragma unroll
        for (int q = 0; q < kOwn; q++) {
            cplx D31 = {1.f, 0.f}, F = {1.f, 0.f};
            if (!diag) {
                const BlockPair* bp = &sm.bp[pair_of(q)][row0 / 32];
                D31 = bp[J].D31;
                F = behind(bp, J, I, kBlocks);
            }
#pragma unroll
            for (int r = 0; r < 4; r++) {
                oz[q][r] += carried(D31, F, s[0][q][r]);
                rho[q][r] -= s[1][q][r];
            }
        }
    }
    // W_{t-1} = D_{t-1} F, F = (decay up to the block) R; the first token of a block takes the decay itself
    auto decay_before = [&](int p) {
        cplx pre = {1.f, 0.f};
#pragma unroll
        for (int J = 0; J < kEarlier; J++)
            if (J < I) pre = cmul(sm.bp[p][row0 / 32 + J].A, pre);
        return pre;
    };
#pragma unroll
    for (int q = 0; q < kOwn; q++) {
        const int p = pair_of(q);
        const cplx pre = decay_before(p), F = cmul(sm.bp[p][W4].R, pre);
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int row = base + 8 * r + g;
            const float x = __fmaf_rn(pd[r], gx[q][r], oz[q][r]), xo = other_of(x), ho = other_of(rho[q][r]);
            const float2 D = sm.dd[p][row], D0 = sm.dd[p][row > 0 ? row - 1 : 0];
            const bool first = r == 0 && g == 0;
            const cplx w0 = first ? pre : cmul(F, {D0.x, D0.y});
            oz[q][r] = rotate({D.x, D.y}, x, xo) + __fmaf_rn(comp ? w0.i : -w0.i, ho, __fmul_rn(w0.r, rho[q][r]));
        }
    }
    if (slow != 0) {
#pragma unroll
        for (int q = 0; q < kOwn; q++)
#pragma unroll 1
            for (int s = 0; s < 2; s++)
                if ((slow >> (2 * tile(q) + s)) & 1) {
                    const cplx pre = decay_before(2 * tile(q) + s);
                    slow_walk<kD, kPairs, kMode, kWide, true>(sm, 2 * tile(q) + s, row0, I, W, tl);
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        const float ho = other_of(rho[q][r]);
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
            const int row = base + 8 * r + g;
            float yy = row - row0 >= sm.first_bad[hs] ? kNotANumber : __fmul_rn(mq[r], oz[q][r]);
            if (a.shortcut_scale != 0.f) {   // block.py:202-208; v after the vp scale
                const float qk = mq[r] * nrm[r] * pd[r];
                const float2 e = sm.viw[p][row], D = sm.dd[p][row];
                cplx vg = cmul({D.x, D.y}, {e.x, e.y});
                if (((slow >> p) & 1) && p < NPB && head_on) {   // (its v has made room for g)
                    const uint32_t w = __ldcg(a.rec_v + (unit * (size_t)NP + pair0 + p) * kD + row - row0);
                    vg = {bits_lo(w), bits_hi(w)};
                }
                yy = __fmaf_rn(a.shortcut_scale * qk * qk, bfr(comp ? vg.i : vg.r), yy);
            }
            sm.y(row)[2 * p + comp] = __float2bfloat16_rn(bfr(yy) * bits_hi(sm.bs[row]));
        }
    }
    __syncwarp();
    if (tok - row0 < Lc && head_on) {   // lane = token: its row of this warp's values
        __nv_bfloat16* yo = a.y + (((size_t)b * L + c * kD + tok - row0) * H + hd) * N + 2 * pair0;
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
        float z[kOwn][2][2], h[kOwn][2][2];
        k_transposed(kG, z);
        k_transposed(kH, h);
#pragma unroll
        for (int q = 0; q < kOwn; q++) {
            const int p = pair_of(q);
            const cplx w = chunk_decay(p);
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int d = 32 * I + 16 * m + 8 * e + g, n = 2 * p + comp;
                    const float r = __bfloat162float(sm.r0[hs][n][d]) - h[q][m][e], o = other_of(r);
                    if (p < NPB && head_on)
                        a.tail_state[(((size_t)b * H + hd) * N + 2 * pair0 + n) * kD + d] =
                            sm.first_bad[hs] < kD ? kNotANumber : z[q][m][e] + rotate(w, r, o);
                }
        }
    }
    tc_fence_before();
    if (!__syncthreads_and(q_here && ok)) give_up(202, true);
    else if (W == 0) tmem_dealloc(tmem, 128);
}

// ------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------
template <int kD, int kPairs, Mode kMode, bool kWide> struct KernelTag {};

template <int kD, int kPairs, Mode kMode, bool kWide = false>
static int launch_one(const CUtensorMap& tmK, const CUtensorMap& tmQ, Args& a, long long items, cudaStream_t st) {
    const size_t smem = sizeof(Smem<kD, kPairs, kMode, kWide>);
    static_assert(sizeof(Smem<kD, kPairs, kMode, kWide>) <= (227 * 1024 + 1024) / kMinBlocks<kD, kPairs, kWide> - 1024, "shared memory");
    static_assert(kMinBlocks<kD, kPairs, kWide> <= 4, "tensor memory: 128 columns a block");
    if (int rc = allow_smem<KernelTag<kD, kPairs, kMode, kWide>>((const void*)scan_tile_kernel<kD, kPairs, kMode, kWide>, smem)) return rc;
    return launch_overlapped(scan_tile_kernel<kD, kPairs, kMode, kWide>, dim3((unsigned)items), dim3(Geo<kD, kPairs, kWide>::kThreads), smem, st,
                             tmK, tmQ, a);
}
template <int kD, int kPairs>
static int launch_mode(Mode m, const CUtensorMap& tmK, const CUtensorMap& tmQ, Args& a, cudaStream_t st) {
    const long long items = (long long)a.B * a.NC * a.HG;
    if (items > 0x7fffffff) return CDSSM_ERR_UNSUPPORTED;
    int sms = 0;
    if (int rc = sm_count(sms)) return rc;
    // Blocks wait for those with smaller numbers, which start first: blocks start in the order of their numbers.  No document says
    // so, hence one block per SM at most: should other streams' kernels hold back an earlier one, the waiting blocks have at most one
    // of two or more places of an SM, and a wait that lasts ends with the status word set.  A wide block has an SM to itself, two calls on two
    // streams would have no place left, so wide blocks draw tickets: whatever a block waits for is done or running.
    a.fixed = items <= sms;
    if (m == kLocal) return launch_one<kD, kPairs, kLocal>(tmK, tmQ, a, items, st);
    if (m == kOutput) return launch_one<kD, kPairs, kOutput>(tmK, tmQ, a, items, st);
    if constexpr (Geo<kD, kPairs>::kOwn > 1)
        if (a.fixed) return launch_one<kD, kPairs, kFused, true>(tmK, tmQ, a, items, st);
    return launch_one<kD, kPairs, kFused>(tmK, tmQ, a, items, st);
}
template <int kD>
static int launch_pairs(Mode m, const CUtensorMap& tmK, const CUtensorMap& tmQ, Args& a, cudaStream_t st) {
    if (a.N <= 4) return launch_mode<kD, 2>(m, tmK, tmQ, a, st);
    if (kD == 128 || a.N <= 8) return launch_mode<kD, 4>(m, tmK, tmQ, a, st);
    return launch_mode<64, 8>(m, tmK, tmQ, a, st);
}
// blocks that share a tile, tiles beside each other
static int groups_of(int D, int N) { return D == 128 && N > 8 ? 2 : 1; }
static int tiles_of(int H, int D, int N) { return D == 128 ? H * groups_of(D, N) : (H + 1) / 2; }

}  // namespace tile

bool scan_tile_supported(int D, int N, int C, int dtype) {
    return dtype == CDSSM_BF16 && D == C && (D == 64 || D == 128) && N > 2 && N <= 16;
}
// Words of the chunks' gammas and states that the one-kernel form hands on, in the places of the chunk decays and states; the gammas
// before the states (from a multiple of 64 words on).
static size_t gamma_words(int B, int L, int H, int D, int N) {
    return ((size_t)B * (((size_t)L + D - 1) / D) * H * (N / 2) + 63) & ~(size_t)63;
}
size_t scan_tile_words(int B, int L, int H, int D, int N) {
    return gamma_words(B, L, H, D, N) + (size_t)B * (((size_t)L + D - 1) / D) * H * (N / 2) * D;
}
// Bytes of the carries that it hands on beside them.
size_t scan_tile_extra_bytes(int B, int L, int H, int D, int N) {
    return (size_t)B * (((size_t)L + D - 1) / D) * H * (N / 2) * D * sizeof(uint64_t);
}

// scan_records.cu
void scan_record_arrays(void* rec, int B, int L, int H, int N, int C, float2** a, uint32_t** v, uint32_t** g);

// mode 0: local pass (fills ws_gamma / ws_state for the carry pass), 1: output pass (reads the rounded carries from ws_state, with
// from_chunks the local results of this call's local pass; writes y, with from_chunks the final state too), 2: both in one kernel
// with the carry handed on inside it (extra: scan_tile_extra_bytes() of scratch; it, scan_tile_words() words from ws_gamma on and
// *ticket zeroed by the caller).
// status: one int in device memory, set by a bounded wait that ran out (not cleared here).
int scan_tile_pass(int mode, int from_chunks, const void* q, long long q_rs, const void* k, long long k_rs, void* rec, const float* h0, void* y,
                   float* final_state, float* tail_state, float* ws_gamma, float* ws_state, void* extra, int* status, int* ticket,
                   float shortcut_scale, int B, int L, int H, int D, int N, unsigned long long wait_ns, int withhold, cudaStream_t st) {
    using namespace tile;
    CUtensorMap tmK, tmQ;
    if (!make_tile_map(&tmK, k, k_rs, B, L, H, D, D) || !make_tile_map(&tmQ, mode == 0 ? k : q, mode == 0 ? k_rs : q_rs, B, L, H, D, D)) return CDSSM_ERR_CUDA;
    Args a;
    float2* ra;
    uint32_t *rv, *rg;
    scan_record_arrays(rec, B, L, H, N, D, &ra, &rv, &rg);
    a.rec_a = ra; a.rec_v = rv; a.rec_g = rg;
    a.h0 = h0;
    a.y = static_cast<__nv_bfloat16*>(y);
    a.final_state = final_state; a.tail_state = mode == 0 ? nullptr : tail_state;
    a.ws_gamma = ws_gamma; a.ws_state = ws_state; a.status = status; a.ticket = ticket;
    a.gammas = reinterpret_cast<uint32_t*>(ws_gamma);
    a.chunks = a.gammas + gamma_words(B, L, H, D, N);
    a.carries = static_cast<uint64_t*>(extra);
    a.wait_ns = wait_ns ? wait_ns : 400ull * 1000 * 1000;
    a.withhold = withhold;
    a.from_chunks = from_chunks;
    a.shortcut_scale = shortcut_scale;
    a.B = B; a.L = L; a.H = H; a.N = N; a.NC = (L + D - 1) / D;
    a.groups = groups_of(D, N);
    a.HG = tiles_of(H, D, N);
    const Mode m = mode == 0 ? kLocal : mode == 1 ? kOutput : kFused;
    return D == 128 ? launch_pairs<128>(m, tmK, tmQ, a, st) : launch_pairs<64>(m, tmK, tmQ, a, st);
}

}  // namespace cdssm
