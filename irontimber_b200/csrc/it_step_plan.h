// How the decode step kernel (it_step.cu) is cut up: its phases, which buffer a quantised row goes to, and the runs of matrix chunks
// that the CTAs take.  Plain host code, so that a test can walk the hand-overs between CTAs without a GPU.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstring>
#include <vector>
#include "../../include/irontimber_cuda.h"

#if defined(__CUDACC__)
#define IT_PLAN_HD __host__ __device__ __forceinline__
#else
#define IT_PLAN_HD static inline
#endif

namespace {

constexpr int ST_TPC = 8;                              // tiles per chunk = per ring slot: two per warp of a group, computed side by side (widths are multiples of 1024, eight tiles)
constexpr int ST_CHUNK = ST_TPC * 1088;                // bytes of one ring slot (a tile is IT_TILE_BYTES)
constexpr int ST_TERMS = ST_TPC * 32;                  // terms of one chunk (floats)
constexpr int ST_SMEM = 227 * 1024;                    // dynamic shared memory of the CTA
constexpr int ST_BARS = 1024;                          // bytes reserved for mbarriers, flags and layer descriptions
constexpr int ST_SD = 128;                             // delta-rule state size this kernel is built for
constexpr int ST_RED = 384;                            // bytes: the dense row's eight f64 warp sums, then the transform's [8] sums of squares and [4][2] group maxima
constexpr int ST_DENSE2 = 128;                         // bytes: where in it a second dense row's warp sums are
constexpr int ST_AT_RED = 36;                          // floats of the attention block's reductions: one a warp, at 32 the sum
constexpr int ST_PITCH = 1344;                         // floats of a block of 1024 in the transform's padded layout (IT_HAD_PITCH)

enum { PH_A, PH_B, PH_C, PH_D, PH_E, PH_F, PH_G, PH_H, PH_I, ST_SUBS };       // phases of a layer

// The half of `codes` that a transform phase writes and the matrix phase behind it reads.  D and H start as soon as the values of
// their own block are there, when CTAs that those values do not come from may not have read the row of B (of G) yet: they write where
// nobody reads that row.  What they overwrite was read before the last phase that waits for a whole row (A, F).  With D in A's half a
// CTA late by B and C finds D's tag in the place of A's and waits for good (tests/test_step_protocol.py walks all of them).
IT_PLAN_HD int step_codes_half(int ph) { return ph == PH_D || ph == PH_E || ph == PH_H || ph == PH_I; }

// A CTA's share of one ternary matrix.  The matrix is a sequence of chunks (eight 32 x 128 tiles of one row group, row
// groups in order); every CTA gets an equal run of it, whatever row group the run starts or ends in (5120 rows are 160 row
// groups: whole ones would leave most of 148 CTAs with one and some with two).  A cut row group is finished by the later
// CTA: the earlier one adds its first blocks and hands the running sums over, which is the same order of additions.  It does
// that part first and the later CTA does its own last, so that nobody waits.  Order of a CTA's chunks: hl of the row group it
// starts but does not finish, whole row groups, tl of the row group begun by the CTA before.
struct StepSpan { int n, hl, tl, lead, uh, uf, ut, nb, cpr, parts, units; unsigned magic; };     // uh, uf, ut: row groups of the three parts
enum { SP_IN_GDN, SP_IN_ATT, SP_OUT_GDN, SP_OUT_ATT, SP_GATE_UP, SP_DOWN, SP_HEAD, SP_KINDS };

// The chunks [c0, c1) of a matrix of `units` row groups (pairs of row groups when parts == 2), in the order a CTA takes them.
inline StepSpan step_span(long long c0, long long c1, int nb, int parts, int units) {
    StepSpan s; memset(&s, 0, sizeof s);
    s.nb = nb; s.cpr = nb / ST_TPC; s.parts = parts; s.units = units; s.magic = 0xffffffffu / (unsigned)s.cpr + 1u;
    const long long cpu = (long long)s.cpr * parts;
    s.n = (int)(c1 - c0); s.lead = (int)(c0 % cpu);
    if (s.n == 0) { s.lead = 0; return s; }
    s.tl = s.lead ? (int)(cpu - s.lead) : 0; s.hl = (int)(c1 % cpu);
    s.ut = (int)(c0 / cpu); s.uf = (int)((c0 + s.tl) / cpu); s.uh = (int)(c1 / cpu);
    return s;
}
// Equal runs of chunks when every CTA gets at least one whole row group's worth (then a row group is cut at most once), else whole
// row groups.
inline void step_spans(std::vector<StepSpan>& out, int kind, int grid, int rows, int cols, int parts) {
    const int nb = cols / 128, units = (rows / parts + 31) / 32; const long long cpu = (long long)(nb / ST_TPC) * parts, total = units * cpu;
    for (int b = 0; b < grid; b++) {
        long long c0, c1;
        if (units >= grid) { c0 = total * b / grid; c1 = total * (b + 1) / grid; }
        else { c0 = (long long)units * b / grid * cpu; c1 = (long long)units * (b + 1) / grid * cpu; }
        out[(size_t)b * SP_KINDS + kind] = step_span(c0, c1, nb, parts, units);
    }
}

// ---- shared memory ----------------------------------------------------------------------------------------------------------
// Behind the ring: the phase scratch, ST_BARS, the CTA's spans.  Scratch of a matrix phase of nb blocks a row: ST_RED bytes of sums, the
// q8k row with its scales (a float per 256) and block sums (an int per 128), then the transform's exchange area and, after it, the terms
// [slots][ST_TPC][32] of the ring's chunks.
IT_PLAN_HD int terms_at(int nb) { return ST_RED + ((nb * 134 + 127) & ~127); }
inline int step_widest(const it_model_config& c) { return std::max(std::max(c.n_embd, c.n_ff), std::max(c.ssm_inner, c.n_head * c.head_dim)); }
// the state tile of the delta-net block comes in while the input projection's chunks run: behind their terms
inline size_t step_gdn_off(const it_model_config& c, int slots) { return (size_t)terms_at(c.n_embd / 128) + (size_t)slots * ST_TERMS * 4; }
inline size_t step_w_bytes(const it_model_config& c) { return (size_t)(c.n_embd / 1024) * ST_PITCH * 4; }
// CTAs that share an attention head: four or two when the grid has them and each then owns whole slices of the V tiles.
inline int step_attn_split(const it_model_config& c, int grid) {
    const int slice = c.head_dim & 63 ? c.head_dim : 64;             // it_vc_slice
    for (int g = 4; g > 1; g /= 2) if (c.head_dim % (32 * g) == 0 && (c.head_dim / g) % slice == 0 && g * c.n_head <= grid) return g;
    return 1;
}
inline size_t step_scratch_bytes(const it_model_config& c, int slots, int attn_g) {
    size_t s = (size_t)terms_at(step_widest(c) / 128) + (size_t)slots * ST_TERMS * 4;
    s = std::max(s, (size_t)ST_RED + (size_t)(c.n_embd / 1024) * ST_PITCH * 4 + (size_t)c.n_embd * 4 + step_w_bytes(c));      // a normed row, a dense row, the norm's weights
    s = std::max(s, step_gdn_off(c, slots) + (size_t)ST_SD * ST_SD * 4);
    // a norm's weights and a dense row come in while the widest matrix's chunks run, and stay while their row is transformed
    const size_t below = std::max((size_t)terms_at(step_widest(c) / 128) + (size_t)slots * ST_TERMS * 4, (size_t)terms_at(c.n_embd / 128) + (size_t)(c.n_embd / 1024) * ST_PITCH * 4);
    s = std::max(s, below + (size_t)c.n_embd * 4 + step_w_bytes(c));
    // scores, q, k, this CTA's elements of v and the gate, reduction; at the longest context three K tiles behind them
    s = std::max(s, ((size_t)(c.ctx_len + 3) / 4 * 4 + 2 * c.head_dim + 2 * (c.head_dim / attn_g) + ST_AT_RED) * 4 + 12 + 3 * (size_t)c.head_dim * 64);
    return (s + 15) / 16 * 16;
}
inline size_t step_smem_bytes(const it_model_config& c, int slots, int attn_g) { return (size_t)slots * ST_CHUNK + step_scratch_bytes(c, slots, attn_g) + ST_BARS + SP_KINDS * sizeof(StepSpan); }
// Ring slots: a power of two (slot = chunk index & (slots - 1)), as many of 16 as fit; 0 when not even four do.  64 layers of the 27B widths, us a step with
// 16 (contexts up to 9988) / 8: 2982 / 3090 at position 9, 5737 / 5844 at 8000.
inline int step_ring_slots(const it_model_config& c, int attn_g) {
    int slots = 16;
    while (slots >= 4 && step_smem_bytes(c, slots, attn_g) > (size_t)ST_SMEM) slots /= 2;
    return slots >= 4 ? slots : 0;
}

}  // namespace
