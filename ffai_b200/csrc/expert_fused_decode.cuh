// One forward of the whole block in ONE launch, for the smallest batches (up to 8 tokens).
//
// Replaces, for those batches, the launch chain router -> gate/up -> down -> combine (and the shared expert's
// launches), that is the reference's per-token decode (MoELayer.decode, FFAI MoELayer.swift:530-634;
// GPTOSSMoELayer.decode, GPTOSSText.swift:1340-1445; Qwen35MoEFFN.forward, Qwen3xText.swift:928-1035).
//
// Why: at one token the weights of the selected experts take 3 to 9 us at the HBM rate, and the chain took 41 us.
// Every launch costs about 3.5 us of its own even as a dependent launch, while a grid-wide barrier inside a
// cooperative launch costs 1.2 us; and inside one launch the next phase's weights can be in flight across the
// barrier.  So:
//   phase 1  router logits (one expert row per CTA, the fixed chunk order), the token rows into shared memory,
//            and the shared expert's gate/up, which needs no routing
//   barrier  every logit is visible
//   phase 2  every CTA routes all tokens for itself (one warp per token) and builds the list of distinct experts
//   phase 3  gate/up + activation: items of 16 gate and 16 up rows, the 16 warps of a CTA split the reduction axis
//   barrier  (the first weights of phase 4 are on their way into L2)
//   phase 4  down: items of 16 output rows over ALL selected experts (and the shared one), each expert's product
//            scaled by its combine weight, so the sum over warps is the block's output: no y buffer, no combine
// Operands: cells of 16 weight rows x 64 k, loaded straight into registers: every cell is used once, by one warp, so shared
// memory would only add instructions (bulk copies into per-warp rings measured the same at one token and 10 % slower at
// eight).  4-bit experts of group 64 and 128 are read from the streams that expert_stream_decode.cuh keeps anyway; all others
// from the packed rows as they are: no further copy of the experts.
// mma.sync m16n8k16 has 8 columns: the tokens.  Bound: at one to four tokens latency (launch, two barriers, the cold
// instruction fetches of code that runs once), at eight the issue slots of unpack and fold (about 105 instructions per
// 16 x 64 cell; packed rows 12 more than streams).  Measured against the launch chain: 32 experts of 2880 x 2880, top 4, one
// token 42.7 -> 30.8 us, group 32, one token 47.1 -> 37.3, six 101 -> 92; 128 experts of 2048 x 768, top 8, one token
// 41.8 -> 21; 8-bit codes, four tokens 196 -> 63; 256 experts and a shared one, three tokens 102 -> 37.
// fp32 accumulation throughout.  The activation's result is held as the launch chain holds it: rounded to bf16 for 4-bit
// routed experts, in fp32 for 8-bit ones and for the shared expert.  The MMA reads the latter as three bf16 terms whose sum is
// the fp32 value (split3): three times the MMAs of down, no bit lost.
//
// The waits at the grid barriers are bounded; a CTA that gives up raises the error word and leaves.  The barrier word then holds a
// partial count, so it also marks the barrier broken: later launches leave before they write an output, until the host, which
// reads the error word, has reset both.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "expert_stream_decode.cuh"
#include "router.cuh"

namespace ffai {
namespace fdec {

constexpr int WARPS = 16;
constexpr int THREADS = WARPS * 32;
constexpr int MAX_T = 8;            // tokens: the columns of one MMA
constexpr int MAX_ROWS = 64;        // routed rows, and so distinct experts
constexpr int SHARED_U = MAX_ROWS;  // table slot of the shared expert
constexpr int RED_PITCH = 20;       // floats per activation column of a 16-row partial: lanes (g, t) hit distinct banks
constexpr int RED_BYTES = 56 * 1024;           // partial sums; also router and routing scratch
constexpr int MAX_DOWN_ITEMS = 12;             // down items a CTA's range may touch
constexpr uint32_t BARRIER_POLLS = 1u << 21;   // of about half a microsecond each
enum : uint32_t { ERR_GRID_BARRIER = 64 };

// Where the weights of a cell lie.  STREAM: one run in MMA fragment order, words first (lane l's at l * 16), then the
// (scale | bias << 16) words of rows g and g+8, 8 bytes per g.  ROWS: the packed rows, scales and biases as the layer has
// them.  ROWS_SB: the packed rows, and the (scale | bias << 16) words re-tiled as [16-row block][32-run][16 rows].
// Lane (g, t) holds the 8-runs 2t and 2t+1 of the cell's k in rows g and g+8 (group 32: runs t and t+4, so that a run's two
// MMAs stay in one half).
enum Source { STREAM, ROWS, ROWS_SB };
template <int BITS, bool G32>
constexpr Source SOURCE = BITS == 8 ? ROWS : (G32 ? ROWS_SB : STREAM);
// loads in flight per warp (1 in gate/up: 9.3 -> 11.4 us at one token of the 32-expert layer; 3 and 5: no gain, and the
// longer unrolled loop costs instruction fetches)
constexpr int PAIRS_AHEAD = 2;   // gate/up: (gate cell, up cell) pairs
constexpr int CELLS_AHEAD = 3;   // down (2 with activations of three terms)

// One stacked projection.  STREAM: w alone (gate/up: gate and up cells of a 64-run alternate).
struct Proj {
    const uint8_t* w;
    const uint8_t* s;   // scales (ROWS_SB: the re-tiled words)
    const uint8_t* b;   // biases
};

struct Params {
    RouterParams rp;
    const uint16_t* x;          // [T, H]
    const uint16_t* xr;         // the router's rows (x unless split)
    int T, H, I;
    Proj gate, up, down;        // routed experts
    int gshift;                 // log2 of the group size
    const uint16_t *rb_gate, *rb_up, *rb_down;   // nullable row biases
    int activation;
    float limit, alpha;
    int Is;                     // shared expert: 0 = none
    Proj sh_gate, sh_up, sh_down;
    int sh_gshift;
    int sh_gate_kind;           // 0 none, 1 fp32, 2 bf16, 3 affine
    const void* sh_gate_w;      // [H]
    const uint16_t *sh_gate_s, *sh_gate_b;
    int sh_gate_bits, sh_gate_group;
    float* sh_gate_logit;       // [T]
    float* logits;              // [T, E]
    uint32_t* indices;          // [T, k]
    float* rweights;            // [T, k]
    PlanOut plan;
    uint16_t* inner;            // [INNER_TERMS planes][T*k, I] bf16, 8-run permuted
    uint16_t* sh_inner;         // [3 planes][T, Is]
    uint32_t inner_plane, sh_plane;   // elements between planes
    const uint16_t* residual;   // nullable
    uint16_t* out;
    float* split;               // [2 * CTAs][16 * MAX_T] partial sums of down items that two or more CTAs share
    uint32_t* tickets;          // [H/16] zero before the first launch, zero again after each
    uint32_t* barrier;          // one word, zero before the first launch
    uint32_t* broken;           // non-zero after a wait that was given up
    uint32_t polls;             // limit of a wait
    uint32_t* error_word;
};

struct Tables {
    uint32_t idx[MAX_ROWS];             // [token * k + slot] selected experts, selection order
    uint32_t first[MAX_ROWS];           // the same where it is the expert's first entry, else all ones
    float w[MAX_ROWS];                  // combine weights
    float colw[MAX_ROWS + 1][MAX_T];    // combine weight of (distinct expert, token), 0 where not selected
    int16_t pos[MAX_ROWS + 1][MAX_T];   // row of (distinct expert, token) in `inner`, -1 where not selected
    uint8_t tok[MAX_ROWS + 1][MAX_T];   // tokens of a distinct expert, ascending
    uint16_t expert[MAX_ROWS + 1], base[MAX_ROWS + 1], cnt[MAX_ROWS + 1];
    int n_distinct;
    int failed;
    uint32_t ticket[2];
};

// Dynamic shared memory.  A 64-run of a token row takes 144 bytes: 128 of values, then its sum (4 bytes), a gap, and the sums of its halves (2 x 4).  The odd
// stride lets 8 threads read the same piece of 8 runs from distinct banks (router), the row pitch does so for the MMA
// fragments of neighbouring rows.
constexpr int RUN = 144, RUN_SUM = 128, RUN_HALF_SUMS = 136;
// Gate/up items of a CTA whose partial sums fit the area at a time (a slot has 2 * T * RED_PITCH floats, an item up to WARPS slots).
__host__ __device__ constexpr int gate_up_batch(int T) { return RED_BYTES / 4 / (2 * T * RED_PITCH) - (WARPS - 1); }

template <int BITS, bool G32>
struct Layout {
    static constexpr int STAGE_BYTES = 56 * 1024;
    __host__ __device__ static int x_pitch(int H) {
        const int n = H / 64 * RUN, want = G32 ? 64 : 16;
        return n + ((want - n % 128 + 128) % 128);
    }
    __host__ __device__ static int stage() { return ((int)sizeof(Tables) + 127) & ~127; }
    __host__ __device__ static int red() { return stage() + STAGE_BYTES; }
    __host__ __device__ static int x() { return red() + RED_BYTES; }
    __host__ __device__ static int total(int T, int H) { return x() + T * x_pitch(H); }
    // the router's rows are staged in an area of their own, its chunk sums and the routing tables in the partial-sum area
    static bool fits(int T, int M, int E, int H, int I, int Is, int weight_bytes, int grid) {
        if (SOURCE<BITS, G32> != STREAM && (double)E * H * I * BITS / 8 >= 4e9) return false;   // 32-bit byte offsets
        // Packed rows of group 32 take 12 instructions a cell more than a stream; once a CTA's gate/up items need a second batch
        // of partial sums, the launch chain is faster: 32 experts of 2880, 5 / 6 / 7 / 8 tokens 86 / 94 / 98 / 117 us here, 95 / 101 / 103 /
        // 109 there (the eighth needs two); 128 experts of 2048 x 768, always one, 1 / 4 / 8 tokens 24 / 46 / 68 and 39 / 53 / 72.
        if (SOURCE<BITS, G32> == ROWS_SB && (M < E ? M : E) * (I / 16) > gate_up_batch(T) * grid) return false;
        const int rows = (E + grid - 1) / grid;
        return rows * H * weight_bytes <= STAGE_BYTES && rows * T * (H / 64) * 4 <= RED_BYTES && T * 2 * E * 4 <= RED_BYTES &&
               H / 16 <= (MAX_DOWN_ITEMS - 2) * grid &&
               (double)(H / 16) * (M * (I / 64) + Is / 64) * grid < 4e9;   // flat positions of the down phase times CTAs in 32 bits
    }
};

// (Plain shared-memory loads and MMAs without side effects: the compiler interleaves the chains of neighbouring cells.)
FFAI_DEVINL uint4 ld_s16(uint32_t a) { return *reinterpret_cast<const uint4*>(__cvta_shared_to_generic(a)); }
FFAI_DEVINL float ld_s4(uint32_t a) { return *reinterpret_cast<const float*>(__cvta_shared_to_generic(a)); }
FFAI_DEVINL uint2 ld_s8(uint32_t a) { return *reinterpret_cast<const uint2*>(__cvta_shared_to_generic(a)); }
FFAI_DEVINL void mma16816(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
FFAI_DEVINL void mma16816_zero(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}
// A lane's part of a cell as it comes from memory.
template <int BITS, bool G32, Source SRC>
struct Raw {
    uint4 w[BITS == 4 ? 1 : 2];            // 4 bits: rows g (x, y) and g+8 (z, w); 8 bits: row g, row g+8
    uint32_t s[SRC == ROWS_SB ? 4 : 2];    // ROWS: scales of rows g, g+8 (group 32: both halves); else scale | bias << 16 ...
    uint32_t b[2];                         // ROWS: biases
    // of half h of the cell (group 32) and row half i
    FFAI_DEVINL float scale(int h, int i) const {
        if (SRC == ROWS) return __uint_as_float(G32 && h ? s[i] & 0xFFFF0000u : s[i] << 16);
        return __uint_as_float(s[SRC == ROWS_SB ? 2 * h + i : i] << 16);
    }
    FFAI_DEVINL float bias(int h, int i) const {
        if (SRC == ROWS) return __uint_as_float(G32 && h ? b[i] & 0xFFFF0000u : b[i] << 16);
        return __uint_as_float(s[SRC == ROWS_SB ? 2 * h + i : i] & 0xFFFF0000u);
    }
};
// Loads under a predicate, the registers keeping what they hold otherwise.  (With the load in a branch the compiler
// loads into other registers and moves: the move waits for the load, and nothing is ahead any more.)
FFAI_DEVINL void ldg16_if(bool on, const uint8_t* p, uint4& v) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t@p ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n\t}"
                 : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w) : "l"(p), "r"((int)on));
}
FFAI_DEVINL void ldg8_if(bool on, const uint8_t* p, uint32_t& a, uint32_t& b) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t@p ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];\n\t}"
                 : "+r"(a), "+r"(b) : "l"(p), "r"((int)on));
}
FFAI_DEVINL void ldcg16_if(bool on, const uint16_t* p, uint4& v) {   // written by other CTAs of this launch: L2
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t@p ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];\n\t}"
                 : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w) : "l"(p), "r"((int)on));
}
// Pieces that do not fill a sector, or share it with the next cells': kept in L1.
FFAI_DEVINL void ldg4_if(bool on, const uint8_t* p, uint32_t& v) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p ld.global.nc.u32 %0, [%1];\n\t}" : "+r"(v) : "l"(p), "r"((int)on));
}
FFAI_DEVINL void ldg2_if(bool on, const uint8_t* p, uint32_t& v) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .u16 h;\n\tsetp.ne.b32 p, %2, 0;\n\t@p ld.global.nc.u16 h, [%1];\n\t@p cvt.u32.u16 %0, h;\n\t}"
                 : "+r"(v) : "l"(p), "r"((int)on));
}
// Where a lane reads the cells of an item (16 rows of n_cells cells) from.  STREAM: addresses.  ROWS: 32-bit byte offsets into
// a projection's words and scales (gate and up have the same shape, so the same ones), which an instruction adds to the
// base by itself; `Layout::fits` keeps larger projections out.
template <int BITS, bool G32, Source SRC>
struct Cursor {
    static constexpr int NB = BITS * 8;          // ROWS: bytes of a row per cell
    uint32_t w, s, k;                            // k: of the cell (groups of 64 and 128)
    // row block `rb` = expert * row blocks + row block of the expert; cell c
    FFAI_DEVINL void seek(const Proj&, uint32_t rb, int n_cells, int c, int, int gshift, int lane) {
        const uint32_t g = lane >> 2, t = lane & 3;
        w = ((rb * 16 + g) * n_cells + c) * NB + t * (BITS == 8 ? (G32 ? 8 : 16) : (G32 ? 4 : 8));
        if (SRC == ROWS_SB) s = ((rb * n_cells + c) * 32 + g) * 4;
        else if (G32) s = ((rb * 16 + g) * n_cells + c) * 4;
        else s = (rb * 16 + g) * ((uint32_t)(n_cells * 64) >> gshift) * 2;
        k = c * 64;
    }
    FFAI_DEVINL void next(int) {
        w += NB;
        if (SRC == ROWS_SB) s += 128;
        else if (G32) s += 4;
        else k += 64;
    }
    FFAI_DEVINL void load(bool on, const Proj& p, int, int n_cells, int gshift, Raw<BITS, G32, SRC>& r) const {
        const uint32_t w8 = w + (uint32_t)n_cells * NB * 8;
        if (BITS == 8) {
            uint4& far = r.w[1 % (BITS / 4)];
            if (G32) {
                ldg8_if(on, p.w + w, r.w[0].x, r.w[0].y); ldg8_if(on, p.w + w + 32, r.w[0].z, r.w[0].w);
                ldg8_if(on, p.w + w8, far.x, far.y); ldg8_if(on, p.w + w8 + 32, far.z, far.w);
            } else {
                ldg16_if(on, p.w + w, r.w[0]); ldg16_if(on, p.w + w8, far);
            }
        } else if (G32) {
            ldg4_if(on, p.w + w, r.w[0].x); ldg4_if(on, p.w + w + 16, r.w[0].y);
            ldg4_if(on, p.w + w8, r.w[0].z); ldg4_if(on, p.w + w8 + 16, r.w[0].w);
        } else {
            ldg8_if(on, p.w + w, r.w[0].x, r.w[0].y); ldg8_if(on, p.w + w8, r.w[0].z, r.w[0].w);
        }
        if (SRC == ROWS_SB) {
#pragma unroll
            for (int i = 0; i < 4; ++i) ldg4_if(on, p.s + s + 32 * i, r.s[i % (SRC == ROWS_SB ? 4 : 2)]);
            return;
        }
        const uint32_t s0 = G32 ? s : s + (k >> gshift) * 2, s8 = s0 + ((uint32_t)(n_cells * 64) >> gshift) * 16;
        if (G32) {
            ldg4_if(on, p.s + s0, r.s[0]); ldg4_if(on, p.s + s8, r.s[1]); ldg4_if(on, p.b + s0, r.b[0]); ldg4_if(on, p.b + s8, r.b[1]);
        } else {
            ldg2_if(on, p.s + s0, r.s[0]); ldg2_if(on, p.s + s8, r.s[1]); ldg2_if(on, p.b + s0, r.b[0]); ldg2_if(on, p.b + s8, r.b[1]);
        }
    }
};
template <int BITS, bool G32>
struct Cursor<BITS, G32, STREAM> {
    static constexpr int CELL_BYTES = 576;
    const uint8_t *w, *s;
    FFAI_DEVINL void seek(const Proj& p, size_t rb, int n_cells, int c, int projections, int, int lane) {   // projections alternate
        w = p.w + (rb * n_cells + c) * (CELL_BYTES * projections) + lane * 16;
        s = p.w + (rb * n_cells + c) * (CELL_BYTES * projections) + 512 + (lane >> 2) * 8;
    }
    FFAI_DEVINL void next(int projections) { w += CELL_BYTES * projections; s += CELL_BYTES * projections; }
    FFAI_DEVINL void load(bool on, const Proj&, int projection, int, int, Raw<BITS, G32, STREAM>& r) const {
        ldg16_if(on, w + CELL_BYTES * projection, r.w[0]);
        ldg8_if(on, s + CELL_BYTES * projection, r.s[0], r.s[1]);
    }
};
// The first bytes (at most `budget`) of n cells of an item on their way into L2; returns the bytes asked for.
template <int BITS, bool G32, Source SRC>
FFAI_DEVINL int prefetch_cells(const Proj& p, size_t rb, int n_cells, int c, int n, int gshift, int budget, int lane) {
    auto ask = [](const uint8_t* a) { asm volatile("prefetch.global.L2 [%0];" ::"l"(a)); };
    if (SRC == STREAM) {
        const int bytes = min(n * 576, budget);
        for (int o = lane * 128; o < bytes; o += 32 * 128) ask(p.w + (rb * n_cells + c) * 576 + o);
        return bytes;
    }
    constexpr int NB = BITS * 8;
    const int cells = min(n, budget / (16 * NB) + 1), row = lane & 15;
    const uint8_t* from = p.w + ((rb * 16 + row) * n_cells + c) * NB;
    const uint8_t* to = from + cells * NB;
    // whole lines, the first one from the row's own bytes on
    for (const uint8_t* a = from + 128 * (lane >> 4); a < to; a += 256) ask(a);
    if (lane >= 16) ask(to - NB);
    if (SRC == ROWS_SB) {
        if (lane < cells) ask(p.s + (rb * n_cells + c + lane) * 128);
    } else {
        ask((lane < 16 ? p.s : p.b) + ((rb * 16 + row) * ((size_t)(n_cells * 64) >> gshift) + ((c * 64) >> gshift)) * 2);
    }
    return cells * 16 * NB;
}
// Two bytes of codes (low and high half) -> the bf16 pair of their values: q = 16 * hi + lo, exact.
FFAI_DEVINL uint32_t byte_pair(uint32_t w, uint32_t mask, uint32_t expo) {
    const __nv_bfloat162 k128 = __floats2bfloat162_rn(128.0f, 128.0f), k16 = __floats2bfloat162_rn(16.0f, 16.0f);
    const uint32_t l = dmma::and_or(w, mask, expo), h = dmma::and_or(w >> 4, mask, expo);
    const __nv_bfloat162 lo = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&l), k128), hi = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&h), k128);
    const __nv_bfloat162 q = __hfma2(hi, k16, lo);
    return *reinterpret_cast<const uint32_t*>(&q);
}
// The A fragment of MMA hp of 8-run w: the pairs (0, 4), (1, 5) or (2, 6), (3, 7) of its k, the order the activations have.
// 4 bits: pairs are 128 + q (the offset goes into the bias term).
template <int BITS, bool G32, Source SRC>
FFAI_DEVINL void a_fragment(const Raw<BITS, G32, SRC>& r, int w, int hp, uint32_t mask, uint32_t expo, uint32_t* a) {
    if (BITS == 4) {
        const uint32_t lo = w ? r.w[0].y : r.w[0].x, hi = w ? r.w[0].w : r.w[0].z;   // rows g, g+8
        a[0] = dmma::and_or(lo >> (8 * hp), mask, expo);
        a[1] = dmma::and_or(hi >> (8 * hp), mask, expo);
        a[2] = dmma::and_or(lo >> (8 * hp + 4), mask, expo);
        a[3] = dmma::and_or(hi >> (8 * hp + 4), mask, expo);
    } else {
        const uint4 &x = r.w[0], &y = r.w[BITS == 4 ? 0 : 1];
        const uint32_t sel = hp ? 0x7632 : 0x5410;   // bytes k0 k1 k4 k5 | k2 k3 k6 k7
        const uint32_t lo = w ? __byte_perm(x.z, x.w, sel) : __byte_perm(x.x, x.y, sel), hi = w ? __byte_perm(y.z, y.w, sel) : __byte_perm(y.x, y.y, sel);
        a[0] = byte_pair(lo, mask, expo);
        a[1] = byte_pair(hi, mask, expo);
        a[2] = byte_pair(lo >> 8, mask, expo);
        a[3] = byte_pair(hi >> 8, mask, expo);
    }
}

// Terms of an activation result: 1 = rounded to bf16, 3 = fp32 as a sum of bf16 values.
template <int BITS>
constexpr int INNER_TERMS = BITS == 8 ? 3 : 1;
constexpr int SH_TERMS = 3;

// v as three bf16 values whose sum is v: 24 significant bits are cut into 8 + 8 + 8 (the last ones are lost below 2^-133, the
// smallest bf16).  Infinities and NaN stay in the first.
FFAI_DEVINL void split3(float v, uint16_t (&term)[3]) {
    const uint32_t b = __float_as_uint(v);
    term[0] = (uint16_t)(b >> 16);
    term[1] = term[2] = 0;
    if ((b & 0x7F800000u) == 0x7F800000u) {
        if (b & 0x007FFFFFu) term[0] |= 0x40;   // a NaN whose payload lies in the bits cut off
        return;
    }
    const float r1 = __fsub_rn(v, __uint_as_float(b & 0xFFFF0000u));
    const uint32_t m = __float_as_uint(r1);
    term[1] = (uint16_t)(m >> 16);
    term[2] = (uint16_t)(__float_as_uint(__fsub_rn(r1, __uint_as_float(m & 0xFFFF0000u))) >> 16);
}

// Sums over the 64 k (group 32: over each half) of the activation columns 2t and 2t+1: an MMA with a matrix of ones.
template <bool G32, int TERMS>
FFAI_DEVINL void column_sums(const uint4* x0, const uint4* x1, float (*sx)[2]) {
    const uint32_t ones[4] = {0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u};
    float c[4];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
#pragma unroll
        for (int i = TERMS - 1; i >= 0; --i) {
            const uint4& x = w ? x1[i] : x0[i];
            if ((G32 || w == 0) && i == TERMS - 1) mma16816_zero(c, ones, x.x, x.y);
            else mma16816(c, ones, x.x, x.y);
            mma16816(c, ones, x.z, x.w);
        }
        sx[G32 ? w : 0][0] = c[0]; sx[G32 ? w : 0][1] = c[1];
    }
}

// Adds the cell's contribution to rows g, g+8 (tot[0..1], tot[2..3]) and columns 2t, 2t+1, times the columns' weights
// with WEIGHTED.  x0, x1: the TERMS terms of the activations; sx[half][column]: run sums.  WEIGHTED leaves a column whose token
// does not have this expert (`on`) alone: its products are zero, but zero times an infinite scale is not.
template <int BITS, bool G32, Source SRC, bool WEIGHTED, int TERMS>
FFAI_DEVINL void cell_dot(const Raw<BITS, G32, SRC>& r, uint32_t mask, uint32_t expo, const uint4* x0, const uint4* x1, const float (*sx)[2], float w0,
                          float w1, bool on0, bool on1, float* tot) {
    float c[2][4];
#pragma unroll
    for (int w = 0; w < 2; ++w)
#pragma unroll
        for (int hp = 0; hp < 2; ++hp) {
            uint32_t a[4];
            a_fragment<BITS, G32, SRC>(r, w, hp, mask, expo, a);
#pragma unroll
            for (int i = TERMS - 1; i >= 0; --i) {
                const uint4& x = w ? x1[i] : x0[i];
                float* acc = c[G32 ? w : 0];
                if ((G32 || w == 0) && hp == 0 && i == TERMS - 1) mma16816_zero(acc, a, x.x, x.y);
                else mma16816(acc, a, hp ? x.z : x.x, hp ? x.w : x.y);
            }
        }
#pragma unroll
    for (int h = 0; h < (G32 ? 2 : 1); ++h)
#pragma unroll
        for (int i = 0; i < 2; ++i) {   // row half
            const float sc = r.scale(h, i), b = r.bias(h, i);
            const float bm = BITS == 4 ? fmaf(-128.0f, sc, b) : b;
#pragma unroll
            for (int col = 0; col < 2; ++col) {
                float& t = tot[2 * i + col];
                if (WEIGHTED) {
                    const float v = fmaf(col ? w1 : w0, fmaf(bm, sx[h][col], sc * c[h][2 * i + col]), t);
                    if (col ? on1 : on0) t = v;
                } else t = fmaf(bm, sx[h][col], fmaf(sc, c[h][2 * i + col], t));
            }
        }
}

// Grid barrier in two halves (between them a CTA may do work that needs nothing from the others).  Every CTA adds one;
// CTA 0 adds what is missing to 2^31, so the top bit of the word flips when all have arrived, whatever came before.
struct GridBarrier {
    uint32_t* word;
    uint32_t polls;
    uint32_t old;
    FFAI_DEVINL void arrive() {   // all threads of the CTA
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            old = atomicAdd(word, blockIdx.x == 0 ? 0x80000000u - (gridDim.x - 1) : 1u);
        }
    }
    FFAI_DEVINL bool wait(int* failed) {
        if (threadIdx.x == 0 && !*failed) {
            bool ok = false;
            for (uint32_t i = 0; i < polls && !ok; ++i) {
                uint32_t now;
                asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(word) : "memory");
                ok = ((now ^ old) & 0x80000000u) != 0;
            }
            if (!ok) *failed = 1;
            __threadfence();
        }
        __syncthreads();
        return *failed == 0;
    }
};

FFAI_DEVINL void give_up(const Params& p) {
    atomicExch(p.broken, 1u);
    atomicExch(p.error_word, (uint32_t)ERR_GRID_BARRIER);
}

// Where one expert set's gate/up products come from and go to.
struct GateUp {
    Proj gate, up;         // STREAM: gate alone
    int gshift;
    int I;                 // output rows of each projection
    int u0, n_experts;     // table slots
    const uint16_t *rb_gate, *rb_up;
    int activation;
    float limit, alpha;
    uint16_t* inner;       // rows of I
    uint32_t plane;        // elements between the terms of a result
};

// n cells cut into WARPS contiguous ranges: the first cell of a warp's range, and the warp whose range holds a cell.
FFAI_DEVINL int range_begin(int n, int warp) { return (int)((uint32_t)(n * warp) / WARPS); }
FFAI_DEVINL int range_owner(int n, int cell) { return (int)((uint32_t)((cell + 1) * WARPS - 1) / (uint32_t)n); }

// Gate/up.  A CTA takes consecutive whole items (16 gate and 16 up rows of one distinct expert; consecutive items of an
// expert are consecutive in its stream), a batch of them at a time: the batch's cell pairs are one flat axis
// (item, 64-run), cut into 16 equal contiguous ranges, one per warp.  A warp's partial sums of item j go to slot
// warp + j (ranges are contiguous, so the slots are distinct and an item's are consecutive); after ONE __syncthreads per
// batch the items are finished by all threads.  (With a __syncthreads per item and every warp on the same item an item
// took 1.2 us at one token and 2.9 at eight, mostly waiting for the finishing warps.)
template <int BITS, bool G32, Source SRC, int TERMS>
FFAI_DEVINL void gate_up_phase(const GateUp& a, int T, int H, const Tables* tb, uint32_t x_u, int x_pitch, float* red,
                               int warp, int lane, uint32_t mask, uint32_t expo) {
    constexpr int AHEAD = PAIRS_AHEAD;
    const int n_cells = H / 64, n_rb = a.I / 16, n_items = a.n_experts * n_rb;
    const int g = lane >> 2, t = lane & 3;
    const int i_begin = (int)((uint32_t)n_items * blockIdx.x / gridDim.x), i_end = (int)((uint32_t)n_items * (blockIdx.x + 1) / gridDim.x);
    const int tile = 2 * T * RED_PITCH;                                   // floats per slot
    const int batch = gate_up_batch(T);

    for (int i0 = i_begin; i0 < i_end; i0 += batch) {
        const int n_here = min(batch, i_end - i0), flat = n_here * n_cells;
        const int q0 = range_begin(flat, warp), q1 = range_begin(flat, warp + 1);
        // row biases of the batch on their way into L2
        if (a.rb_gate && (int)threadIdx.x < n_here) {
            const int it = i0 + threadIdx.x, u = it / n_rb;
            const size_t rr = (size_t)tb->expert[a.u0 + u] * a.I + (it - u * n_rb) * 16;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(a.rb_gate + rr));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(a.rb_up + rr));
        }
        // loads run AHEAD pairs in front of the arithmetic; a segment is the rest of the range within one item (one expert's stream)
        struct Pair { Raw<BITS, G32, SRC> gate, up; } buf[AHEAD] = {};
        Cursor<BITS, G32, SRC> cur{};
        int p_q = q0, p_left = 0;
        auto fetch = [&](Pair& d) {
            const bool on = p_q < q1;
            if (p_left == 0 && on) {
                const int j = p_q / n_cells, it = i0 + j, u = it / n_rb, rb = it - u * n_rb, c = p_q - j * n_cells;
                cur.seek(a.gate, tb->expert[a.u0 + u] * (uint32_t)n_rb + rb, n_cells, c, 2, a.gshift, lane);
                p_left = SRC == STREAM ? ((u + 1) * n_rb - i0) * n_cells - p_q : n_cells - c;
            }
            cur.load(on, a.gate, 0, n_cells, a.gshift, d.gate);
            cur.load(on, a.up, 1, n_cells, a.gshift, d.up);
            cur.next(2);
            --p_left; ++p_q;
        };
#pragma unroll
        for (int d = 0; d < AHEAD; ++d) fetch(buf[d]);

        int q = q0, j = q0 / n_cells, here = 0, n = 0;
        uint32_t xl = 0, x0 = 0, x1 = 0;
        float tot[2][4];
        auto begin_item = [&](int c) {
            const int u = a.u0 + (i0 + j) / n_rb;
            n = tb->cnt[u];
            // this lane's row of the B fragment, and the rows of its two result columns
            xl = x_u + tb->tok[u][min(g, n - 1)] * x_pitch + c * RUN + 16 * (G32 ? t : 2 * t);
            x0 = x_u + tb->tok[u][min(2 * t, n - 1)] * x_pitch + c * RUN + (G32 ? RUN_HALF_SUMS : RUN_SUM);
            x1 = x_u + tb->tok[u][min(2 * t + 1, n - 1)] * x_pitch + c * RUN + (G32 ? RUN_HALF_SUMS : RUN_SUM);
#pragma unroll
            for (int pr = 0; pr < 2; ++pr)
#pragma unroll
                for (int i = 0; i < 4; ++i) tot[pr][i] = 0.0f;
            here = min(n_cells - c, q1 - q);
            q += here;
        };
        auto step = [&](Pair& b) {
            const uint4 xa = ld_s16(xl), xb = ld_s16(xl + (G32 ? 64 : 16));
            float sx[2][2];
            if (G32) {
                const uint2 h0 = ld_s8(x0), h1 = ld_s8(x1);
                sx[0][0] = __uint_as_float(h0.x); sx[1][0] = __uint_as_float(h0.y);
                sx[0][1] = __uint_as_float(h1.x); sx[1][1] = __uint_as_float(h1.y);
            } else {
                sx[0][0] = ld_s4(x0); sx[0][1] = ld_s4(x1);
            }
            cell_dot<BITS, G32, SRC, false, 1>(b.gate, mask, expo, &xa, &xb, sx, 0.0f, 0.0f, true, true, tot[0]);
            cell_dot<BITS, G32, SRC, false, 1>(b.up, mask, expo, &xa, &xb, sx, 0.0f, 0.0f, true, true, tot[1]);
            fetch(b);
            xl += RUN; x0 += RUN; x1 += RUN;
            if (--here == 0) {
                float* my = red + (warp + j) * tile;
#pragma unroll
                for (int pr = 0; pr < 2; ++pr)
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (2 * t + (i & 1) < n) my[(pr * T + 2 * t + (i & 1)) * RED_PITCH + g + 8 * (i >> 1)] = tot[pr][i];
                ++j;
                if (q < q1) begin_item(0);
            }
        };
        if (q < q1) begin_item(q0 - j * n_cells);
#pragma unroll 1
        while (here > 0) {
#pragma unroll
            for (int d = 0; d < AHEAD; ++d) {
                step(buf[d]);
                if (here == 0) break;
            }
        }
        __syncthreads();
        // a thread finishes one (item, column, row); 16 consecutive lanes hold an item's rows
        const uint32_t inv_T = (1u << 16) / T + 1;
        const int r = threadIdx.x & 15;
#pragma unroll 1
        for (int jc = threadIdx.x >> 4; jc < n_here * T; jc += THREADS / 16) {
            const int jj = (int)((jc * inv_T) >> 16), col = jc - jj * T;
            const int it = i0 + jj, ui = it / n_rb, rb = it - ui * n_rb, u = a.u0 + ui;
            const bool on = col < tb->cnt[u];
            if (on) {
                const size_t rr = (size_t)tb->expert[u] * a.I + rb * 16 + r;
                float sg = a.rb_gate ? bf16_bits_to_f32(a.rb_gate[rr]) : 0.0f, su = a.rb_up ? bf16_bits_to_f32(a.rb_up[rr]) : 0.0f;
                const int w0 = range_owner(flat, jj * n_cells), w1 = range_owner(flat, (jj + 1) * n_cells - 1);
                const float* src = red + (size_t)(w0 + jj) * tile + col * RED_PITCH + r;
                for (int w = w0; w <= w1; ++w, src += tile)
                    if (flat >= WARPS || range_begin(flat, w) < range_begin(flat, w + 1)) { sg += src[0]; su += src[T * RED_PITCH]; }
                const float v = glu_activation(sg, su, a.activation, a.limit, a.alpha);
                uint16_t* to = a.inner + (size_t)(tb->base[u] + col) * a.I + rb * 16 + dmma::permute8_col(r);
                if (TERMS == 1) {
                    *to = f32_to_bf16_bits(v);
                } else {
                    uint16_t term[3];
                    split3(v, term);
#pragma unroll
                    for (int i = 0; i < 3; ++i) to[i * a.plane] = term[i];
                }
            }
        }
        __syncthreads();   // the partial-sum slots are free
    }
}

// The eight values from k on (a multiple of 8) of a quantized row of K: fma(q, scale, bias), any code width.  Eight codes are
// `bits` whole bytes of the LSB-first stream.
FFAI_DEVINL void affine_run8(const uint32_t* w, const uint16_t* scales, const uint16_t* biases, int bits, int group, int k, int K, float* v) {
    const int byte = k / 8 * bits, i = byte >> 2, shift = (byte & 3) * 8, last = K * bits / 32 - 1;
    const uint32_t a = w[i], b = w[min(i + 1, last)], c = w[min(i + 2, last)];   // (codes of words past the end are not used)
    const uint64_t codes = (uint64_t)__funnelshift_r(a, b, shift) | ((uint64_t)__funnelshift_r(b, c, shift) << 32);
    const float s = bf16_bits_to_f32(scales[k / group]), o = bf16_bits_to_f32(biases[k / group]);
    const uint32_t mask = (1u << bits) - 1;
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = fmaf((float)((uint32_t)(codes >> (j * bits)) & mask), s, o);
}

// SBITS: bit width of the shared expert (4 or 8, group 64 or 128), 0 without one.
template <int BITS, bool G32, int SBITS>
__global__ void __launch_bounds__(THREADS, 1)
fused_decode_kernel(const Params p) {
    using L = Layout<BITS, G32>;
    constexpr Source SRC = SOURCE<BITS, G32>;
    constexpr int SB = SBITS == 0 ? 4 : SBITS;
    extern __shared__ __align__(128) uint8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int T = p.T, H = p.H, I = p.I, E = p.rp.n_experts, K = p.rp.top_k;
    const int n_chunks = H / 64;
    Tables* tb = reinterpret_cast<Tables*>(smem);
    float* red = reinterpret_cast<float*>(smem + L::red());
    const uint32_t x_u = dstr::smem_u32(smem + L::x());
    const int x_pitch = L::x_pitch(H);
    GridBarrier bar{p.barrier, p.polls, 0};
    uint32_t mask, expo;
    asm volatile("mov.u32 %0, 0x000F000F;" : "=r"(mask));
    asm volatile("mov.u32 %0, 0x43004300;" : "=r"(expo));

    // ── phase 1: router logits of experts blockIdx.x, + gridDim.x, ... ──
    const uint32_t broken = threadIdx.x == 0 ? __ldcg(p.broken) : 0;
    for (int i = threadIdx.x; i < (MAX_ROWS + 1) * MAX_T; i += THREADS) { tb->colw[i / MAX_T][i % MAX_T] = 0.0f; tb->pos[i / MAX_T][i % MAX_T] = -1; }
    const int my_experts = (int)blockIdx.x < E ? (E - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int wb = p.rp.kind == 1 ? 4 : 2, lsh = p.rp.kind == 1 ? 4 : 3, line16 = 1 << lsh;   // bytes per router weight; 16-byte pieces per 64 of them
    uint8_t* wst = smem + L::stage();                               // [expert][chunk] lines, pieces XOR-swizzled with the line
    const uint32_t wst_u = dstr::smem_u32(wst);
    for (int ex = 0; ex < my_experts; ++ex) {
        const uint8_t* src = (const uint8_t*)p.rp.weight + (size_t)(blockIdx.x + ex * gridDim.x) * H * wb;
        for (int i = threadIdx.x; i < n_chunks * line16; i += THREADS) {
            const int line = ex * n_chunks + (i >> lsh), j = i & (line16 - 1);
            dmma::cp_async16(wst_u + ((line << lsh) + (j ^ (line & 7))) * 16, src + 16 * i);
        }
    }
    dmma::cp_async_commit();
    // the token rows, every 8-run as 0,4,1,5,2,6,3,7, and the sums of their runs; the loads of four rows at a time
    for (int j0 = 0; j0 < H / 8; j0 += THREADS) {
        const int j = j0 + threadIdx.x;
        const bool in = j < H / 8;
#pragma unroll 1
        for (int t0 = 0; t0 < T; t0 += 4) {
            uint4 v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                v[k] = in && t0 + k < T ? *reinterpret_cast<const uint4*>(p.x + (size_t)(t0 + k) * H + 8 * j) : make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (t0 + k >= T) break;
                uint8_t* run = smem + L::x() + (t0 + k) * x_pitch + (j >> 3) * RUN;
                uint4 o;
                o.x = __byte_perm(v[k].x, v[k].z, 0x5410);
                o.y = __byte_perm(v[k].x, v[k].z, 0x7632);
                o.z = __byte_perm(v[k].y, v[k].w, 0x5410);
                o.w = __byte_perm(v[k].y, v[k].w, 0x7632);
                if (in) *reinterpret_cast<uint4*>(run + (j & 7) * 16) = o;
                float s = ((bf16lo(v[k].x) + bf16hi(v[k].x)) + (bf16lo(v[k].y) + bf16hi(v[k].y))) +
                          ((bf16lo(v[k].z) + bf16hi(v[k].z)) + (bf16lo(v[k].w) + bf16hi(v[k].w)));
                s += __shfl_xor_sync(0xFFFFFFFFu, s, 1);
                s += __shfl_xor_sync(0xFFFFFFFFu, s, 2);
                if (G32 && in && (j & 3) == 0) reinterpret_cast<float*>(run + RUN_HALF_SUMS)[(j >> 2) & 1] = s;
                s += __shfl_xor_sync(0xFFFFFFFFu, s, 4);
                if (in && (j & 7) == 0) *reinterpret_cast<float*>(run + RUN_SUM) = s;
            }
        }
    }
    dmma::cp_async_wait<0>();
    __syncthreads();
    // chunk sums: 64 fused multiply-adds in ascending k from 0 (the fixed order of every router kernel)
    float* part = red;   // [expert][token][chunk]
    for (int i = threadIdx.x; i < my_experts * T * n_chunks; i += THREADS) {
        const int et = i / n_chunks, c = i - et * n_chunks, ex = et / T, tok = et - ex * T, line = ex * n_chunks + c;
        float acc = 0.0f;
#pragma unroll 2
        for (int j = 0; j < 8; ++j) {
            float xf[8];
            if (p.xr == p.x) {
                const uint4 v = *reinterpret_cast<const uint4*>(smem + L::x() + tok * x_pitch + c * RUN + 16 * j);
                xf[0] = bf16lo(v.x); xf[4] = bf16hi(v.x); xf[1] = bf16lo(v.y); xf[5] = bf16hi(v.y);
                xf[2] = bf16lo(v.z); xf[6] = bf16hi(v.z); xf[3] = bf16lo(v.w); xf[7] = bf16hi(v.w);
            } else {
                const uint4 v = *reinterpret_cast<const uint4*>(p.xr + (size_t)tok * H + c * 64 + 8 * j);
                xf[0] = bf16lo(v.x); xf[1] = bf16hi(v.x); xf[2] = bf16lo(v.y); xf[3] = bf16hi(v.y);
                xf[4] = bf16lo(v.z); xf[5] = bf16hi(v.z); xf[6] = bf16lo(v.w); xf[7] = bf16hi(v.w);
            }
            float wf[8];
            if (wb == 4) {
                const float4 w0 = *reinterpret_cast<const float4*>(wst + ((line << lsh) + ((2 * j) ^ (line & 7))) * 16);
                const float4 w1 = *reinterpret_cast<const float4*>(wst + ((line << lsh) + ((2 * j + 1) ^ (line & 7))) * 16);
                wf[0] = w0.x; wf[1] = w0.y; wf[2] = w0.z; wf[3] = w0.w; wf[4] = w1.x; wf[5] = w1.y; wf[6] = w1.z; wf[7] = w1.w;
            } else {
                const uint4 w = *reinterpret_cast<const uint4*>(wst + ((line << lsh) + (j ^ (line & 7))) * 16);
                wf[0] = bf16lo(w.x); wf[1] = bf16hi(w.x); wf[2] = bf16lo(w.y); wf[3] = bf16hi(w.y);
                wf[4] = bf16lo(w.z); wf[5] = bf16hi(w.z); wf[6] = bf16lo(w.w); wf[7] = bf16hi(w.w);
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) acc = __fmaf_rn(xf[k], wf[k], acc);
        }
        part[i] = acc;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < my_experts * T; i += THREADS) {
        const int e = blockIdx.x + (i / T) * gridDim.x, tok = i % T;
        float total = 0.0f;
#pragma unroll 8
        for (int c = 0; c < n_chunks; ++c) total = __fadd_rn(total, part[i * n_chunks + c]);
        if (p.rp.logits_bf16) total = bf16_round(total);
        if (p.rp.bias) {
            total = __fadd_rn(total, bf16_bits_to_f32(p.rp.bias[e]));
            if (p.rp.logits_bf16) total = bf16_round(total);
        }
        p.logits[(size_t)tok * E + e] = total;
    }
    if (SBITS != 0 && p.sh_gate_kind != 0 && blockIdx.x == gridDim.x - 1 && warp < T) {
        float acc = 0.0f;
        auto run = [&](int k, const float* wf) {
            const uint4 xv = *reinterpret_cast<const uint4*>(p.x + (size_t)warp * H + k);
            const float xf[8] = {bf16lo(xv.x), bf16hi(xv.x), bf16lo(xv.y), bf16hi(xv.y), bf16lo(xv.z), bf16hi(xv.z), bf16lo(xv.w), bf16hi(xv.w)};
#pragma unroll
            for (int j = 0; j < 8; ++j) acc = fmaf(wf[j], xf[j], acc);
        };
        if (p.sh_gate_kind == 3) {
#pragma unroll 4
            for (int k = lane * 8; k < H; k += 256) {
                float wf[8];
                affine_run8((const uint32_t*)p.sh_gate_w, p.sh_gate_s, p.sh_gate_b, p.sh_gate_bits, p.sh_gate_group, k, H, wf);
                run(k, wf);
            }
        } else if (p.sh_gate_kind == 1) {
            for (int k = lane * 8; k < H; k += 256) {
                const float4 w0 = *reinterpret_cast<const float4*>((const float*)p.sh_gate_w + k), w1 = *reinterpret_cast<const float4*>((const float*)p.sh_gate_w + k + 4);
                const float wf[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
                run(k, wf);
            }
        } else {
            for (int k = lane * 8; k < H; k += 256) {
                const uint4 w = *reinterpret_cast<const uint4*>((const uint16_t*)p.sh_gate_w + k);
                const float wf[8] = {bf16lo(w.x), bf16hi(w.x), bf16lo(w.y), bf16hi(w.y), bf16lo(w.z), bf16hi(w.z), bf16lo(w.w), bf16hi(w.w)};
                run(k, wf);
            }
        }
        acc = warp_sum(acc);
        if (lane == 0) p.sh_gate_logit[warp] = acc;
    }
    if (threadIdx.x == 0) tb->failed = broken != 0;   // the first wait looks at it
    bar.arrive();
    if (SBITS != 0) {
        // the shared expert takes every token
        if (threadIdx.x < MAX_T) {
            tb->tok[SHARED_U][threadIdx.x] = (uint8_t)threadIdx.x;
            if ((int)threadIdx.x < T) tb->pos[SHARED_U][threadIdx.x] = (int16_t)threadIdx.x;
            if (threadIdx.x == 0) { tb->expert[SHARED_U] = 0; tb->base[SHARED_U] = 0; tb->cnt[SHARED_U] = (uint16_t)T; }
        }
        __syncthreads();
        const GateUp a{p.sh_gate, p.sh_up, p.sh_gshift, p.Is, SHARED_U, 1, nullptr, nullptr, 0, 0.0f, 0.0f, p.sh_inner, p.sh_plane};
        gate_up_phase<SB, false, ROWS, SH_TERMS>(a, T, H, tb, x_u, x_pitch, red, warp, lane, mask, expo);
    }
    if (!bar.wait(&tb->failed)) {
        if (threadIdx.x == 0) give_up(p);
        return;
    }

    // ── phase 2: routing, the same in every CTA; the last one also writes it out ──
    const bool writer = blockIdx.x == gridDim.x - 1;
    const int M = T * K;
    {
        float* lg = red + (size_t)warp * 2 * E;
        if (warp < T) {
            for (int e = lane; e < E; e += 32) lg[e] = __ldcg(p.logits + (size_t)warp * E + e);
            __syncwarp();
            route_token_warp(p.rp, lg, lg + E, lane, tb->idx + warp * K, tb->w + warp * K);
        }
        if (SBITS != 0 && warp == MAX_T && lane < T)
            tb->colw[SHARED_U][lane] = p.sh_gate_kind ? 1.0f / (1.0f + __expf(-__ldcg(p.sh_gate_logit + lane))) : 1.0f;
        __syncthreads();
        // Stable order by (expert, token, slot) and the distinct experts: at most 64 entries, so each entry counts the
        // others against itself (two short loops instead of a histogram, a scan over all experts and four barriers).
        if (threadIdx.x < MAX_ROWS) {
            const int i = threadIdx.x;
            const uint32_t e = i < M ? tb->idx[i] : 0xFFFFFFFFu;
            int less = 0, before = 0, same = 0;
#pragma unroll 4
            for (int j = 0; j < M; ++j) {
                const uint32_t o = tb->idx[j];
                less += o < e; same += o == e; before += (o == e) & (j < i);
            }
            tb->first[i] = before == 0 && i < M ? e : 0xFFFFFFFFu;
            dstr::team_barrier(1, MAX_ROWS);
            int u = 0, n_d = 0;
#pragma unroll 4
            for (int j = 0; j < M; ++j) {
                const uint32_t o = tb->first[j];
                u += o < e; n_d += o != 0xFFFFFFFFu;
            }
            if (i < M) {
                const int tok = i / K, pos = less + before;
                if (before == 0) { tb->expert[u] = (uint16_t)e; tb->base[u] = (uint16_t)pos; tb->cnt[u] = (uint16_t)same; }
                tb->tok[u][before] = (uint8_t)tok;
                tb->pos[u][tok] = (int16_t)pos;
                tb->colw[u][tok] = tb->w[i];
                if (i == 0) tb->n_distinct = n_d;
                if (writer) {
                    p.indices[i] = e; p.rweights[i] = tb->w[i];
                    p.plan.perm[pos] = (uint32_t)i; p.plan.inv_perm[i] = (uint32_t)pos;
                }
            }
        }
        __syncthreads();
    }
    const int U = tb->n_distinct;

    // ── phase 3: gate/up of the routed experts ──
    {
        const GateUp a{p.gate, p.up, p.gshift, I, 0, U, p.rb_gate, p.rb_up, p.activation, p.limit, p.alpha, p.inner, p.inner_plane};
        gate_up_phase<BITS, G32, SRC, INNER_TERMS<BITS>>(a, T, H, tb, x_u, x_pitch, red, warp, lane, mask, expo);
    }

    // ── phase 4: down over all experts of a 16-row block ──
    // Flat axis: (item, cell), an item's cells being the routed experts' in table order, then the shared one's.  When the
    // items give most SMs one each, a CTA takes whole items; otherwise the axis is cut into equal ranges, and the CTAs
    // that share an item add their sums through global memory, the last to arrive in CTA order (2880 rows are 180 items:
    // whole items would take two rounds where 1.2 are needed).
    const int ci = I / 64, cs = SBITS != 0 ? p.Is / 64 : 0, n_rb = H / 16;
    const int routed = U * ci, n_flat = routed + cs, G = gridDim.x, total = n_rb * n_flat;
    // Splitting costs about 2 us (a fence, a ticket, the last CTA's reads); it pays when it saves an SM more than 200 cells
    // (2.7 us at an SM's share of the HBM rate).
    const int rounds = (n_rb + G - 1) / G;
    const bool whole = (rounds * G - n_rb) * n_flat < 200 * G || total < G * WARPS;
    auto cta_begin = [&](int b) { return whole ? (int)((uint32_t)n_rb * b / G) * n_flat : (int)((uint32_t)total * b / G); };
    const int F0 = cta_begin(blockIdx.x), F1 = cta_begin(blockIdx.x + 1), flat = F1 - F0;
    const int q0 = F0 + range_begin(flat, warp), q1 = F0 + range_begin(flat, warp + 1);
    struct Walk {       // position on the flat axis: item, expert (table order, then the shared one), cell of the expert
        int item, u, c;
    };
    auto walk_to = [&](int f) {
        Walk w;
        w.item = f / n_flat;
        const int r = f - w.item * n_flat;
        w.u = r < routed ? r / ci : U;
        w.c = r - w.u * ci;
        return w;
    };
    auto cells_of = [&](int u) { return u < U ? ci : cs; };
    auto advance = [&](Walk& w, int n) {   // by at most what is left of the expert's cells
        w.c += n;
        if (w.c == cells_of(w.u)) {
            w.c = 0;
            if (++w.u > U || cells_of(w.u) == 0) { w.u = 0; ++w.item; }
        }
    };
    // the first 8 KB of the warp's weights (all of them at one token) on their way into L2 across the barrier
    {
        Walk w = walk_to(q0);
        int budget = 8192;
        for (int q = q0; q < q1 && budget > 0;) {
            const int n = min(cells_of(w.u) - w.c, q1 - q);
            if (SBITS != 0 && w.u == U) budget -= prefetch_cells<SB, false, ROWS>(p.sh_down, w.item, cs, w.c, n, p.sh_gshift, budget, lane);
            else budget -= prefetch_cells<BITS, G32, SRC>(p.down, (size_t)tb->expert[w.u] * n_rb + w.item, ci, w.c, n, p.gshift, budget, lane);
            q += n;
            advance(w, n);
        }
    }
    bar.arrive();
    if (!bar.wait(&tb->failed)) {
        if (threadIdx.x == 0) give_up(p);
        return;
    }
    const int first_item = F0 / n_flat, n_items = flat > 0 ? (F1 - 1) / n_flat - first_item + 1 : 0;
    if (p.rb_down)
        for (int i = threadIdx.x; i < n_items * U; i += THREADS)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(p.rb_down + (size_t)tb->expert[i % U] * H + (first_item + i / U) * 16));
    const int tile = T * RED_PITCH;
    float tot[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    // the cells [c, c + n) of one expert: weights and activation fragments are loaded CELLS_AHEAD cells in front
    auto run_cells = [&](auto shared_tag, const Walk& w, int n) {
        constexpr bool SH = decltype(shared_tag)::value;
        constexpr int B = SH ? SB : BITS;
        constexpr bool H32 = SH ? false : G32;
        constexpr int TERMS = SH ? SH_TERMS : INNER_TERMS<BITS>;
        constexpr Source S = SH ? ROWS : SRC;
        constexpr int AHEAD = TERMS == 3 ? 2 : CELLS_AHEAD;
        const uint32_t plane = SH ? p.sh_plane : p.inner_plane;
        const int u = SH ? SHARED_U : w.u;
        const int row = tb->pos[u][g], ld = SH ? p.Is : I;
        const float w0 = tb->colw[u][2 * t], w1 = tb->colw[u][2 * t + 1];
        const bool on0 = tb->pos[u][2 * t] >= 0, on1 = tb->pos[u][2 * t + 1] >= 0;
        // columns without this expert: zero fragments
        const uint16_t* xp = (SH ? p.sh_inner : p.inner) + (size_t)max(row, 0) * ld + w.c * 64 + (H32 ? 8 : 16) * t;
        const Proj& proj = SH ? p.sh_down : p.down;
        const int cells = SH ? cs : ci, gshift = SH ? p.sh_gshift : p.gshift;
        Cursor<B, H32, S> cur;
        cur.seek(proj, SH ? (uint32_t)w.item : tb->expert[w.u] * (uint32_t)n_rb + w.item, cells, w.c, 1, gshift, lane);
        struct Ahead { Raw<B, H32, S> raw; uint4 x0[TERMS], x1[TERMS]; } buf[AHEAD] = {};   // (columns without a row keep zeros)
        int p_n = n;
        auto fetch = [&](Ahead& d) {
            const bool on = p_n > 0;
            cur.load(on, proj, 0, cells, gshift, d.raw);
#pragma unroll
            for (int i = 0; i < TERMS; ++i) {
                ldcg16_if(on && row >= 0, xp + i * plane, d.x0[i]);
                ldcg16_if(on && row >= 0, xp + i * plane + (H32 ? 32 : 8), d.x1[i]);
            }
            cur.next(1); xp += 64; --p_n;
        };
#pragma unroll
        for (int d = 0; d < AHEAD; ++d) fetch(buf[d]);
#pragma unroll 1
        while (n > 0) {
#pragma unroll
            for (int d = 0; d < AHEAD; ++d) {
                float sx[2][2];
                column_sums<H32, TERMS>(buf[d].x0, buf[d].x1, sx);
                cell_dot<B, H32, S, true, TERMS>(buf[d].raw, mask, expo, buf[d].x0, buf[d].x1, sx, w0, w1, on0, on1, tot);
                fetch(buf[d]);
                if (--n == 0) break;
            }
        }
    };
    Walk w = walk_to(q0);
#pragma unroll 1
    for (int q = q0; q < q1;) {
        const int n = min(cells_of(w.u) - w.c, q1 - q), item = w.item;
        if (SBITS != 0 && w.u == U) run_cells(std::true_type{}, w, n);
        else run_cells(std::false_type{}, w, n);
        q += n;
        advance(w, n);
        if (w.item != item || q >= q1) {
            float* my = red + (warp + item - first_item) * tile;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (2 * t + (i & 1) < T) my[(2 * t + (i & 1)) * RED_PITCH + g + 8 * (i >> 1)] = tot[i];
                tot[i] = 0.0f;
            }
        }
    }
    __syncthreads();
    // finish: the CTA's items; one that others share goes through `split` and a ticket
    auto cta_of = [&](int f) { return (int)(((uint32_t)(f + 1) * G - 1) / (uint32_t)total); };   // split axis only
    auto finish = [&](int item, int tok, int r, float v) {
        const int row = item * 16 + r;
        if (p.rb_down)
            for (int s = 0; s < K; ++s) v = fmaf(tb->w[tok * K + s], bf16_bits_to_f32(p.rb_down[(size_t)tb->idx[tok * K + s] * H + row]), v);
        if (p.residual) v += bf16_bits_to_f32(p.residual[(size_t)tok * H + row]);
        p.out[(size_t)tok * H + row] = f32_to_bf16_bits(v);
    };
    for (int i = threadIdx.x; i < n_items * 16 * T; i += THREADS) {
        const int jj = i / (16 * T), o = i - jj * 16 * T, tok = o >> 4, r = o & 15, item = first_item + jj;
        const int f0 = max(item * n_flat, F0) - F0, f1 = min((item + 1) * n_flat, F1) - 1 - F0;
        const int wa = range_owner(flat, f0), wz = range_owner(flat, f1);
        const float* src = red + (wa + jj) * tile + tok * RED_PITCH + r;
        float v = 0.0f;
        for (int ww = wa; ww <= wz; ++ww, src += tile)
            if (flat >= WARPS || range_begin(flat, ww) < range_begin(flat, ww + 1)) v += *src;
        if (item * n_flat >= F0 && (item + 1) * n_flat <= F1) finish(item, tok, r, v);
        else p.split[((size_t)2 * blockIdx.x + (item * n_flat < F0 ? 0 : 1)) * (16 * MAX_T) + o] = v;   // 0: the item began in an earlier CTA
    }
    const bool any_split = n_items > 0 && (first_item * n_flat < F0 || (first_item + n_items) * n_flat > F1);   // its first or its last item
    if (any_split) {
        __threadfence();
        __syncthreads();
        if (threadIdx.x < 2 && (int)threadIdx.x < n_items) {
            const int item = threadIdx.x == 0 ? first_item : first_item + n_items - 1;
            const int b0 = cta_of(item * n_flat), b1 = cta_of((item + 1) * n_flat - 1);
            uint32_t last = 0;
            if (b0 != b1) {
                last = atomicAdd(p.tickets + item, 1u) == (uint32_t)(b1 - b0);
                if (last) p.tickets[item] = 0;
            }
            tb->ticket[threadIdx.x] = last;
        }
        __syncthreads();
        __threadfence();
        for (int i = threadIdx.x; i < min(n_items, 2) * 16 * T; i += THREADS) {
            const int jj = i / (16 * T), o = i - jj * 16 * T, item = jj == 0 ? first_item : first_item + n_items - 1;
            if (!tb->ticket[jj]) continue;
            const int b0 = cta_of(item * n_flat), b1 = cta_of((item + 1) * n_flat - 1);
            float v = 0.0f;
            for (int b = b0; b <= b1; ++b) v += __ldcg(p.split + ((size_t)2 * b + (b == b0 ? 1 : 0)) * (16 * MAX_T) + o);
            finish(item, o >> 4, o & 15, v);
        }
    }
    if (writer)
        for (int e = threadIdx.x; e <= E; e += THREADS) {
            uint32_t less = 0, same = 0;
            for (int j = 0; j < M; ++j) { less += tb->idx[j] < (uint32_t)e; same += tb->idx[j] == (uint32_t)e; }
            p.plan.offsets[e] = less;
            if (e < E) p.plan.counts[e] = same;
        }
}

}  // namespace fdec
}  // namespace ffai
