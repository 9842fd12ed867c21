// How the decode step kernel (it_step.cu) is cut up: its phases, which buffer a quantised row goes to, and the runs of matrix chunks
// that the CTAs take.  Plain host code, so that a test can walk the hand-overs between CTAs without a GPU.
#pragma once
#include <cstring>
#include <vector>

#if defined(__CUDACC__)
#define IT_PLAN_HD __host__ __device__ __forceinline__
#else
#define IT_PLAN_HD static inline
#endif

namespace {

constexpr int ST_TPC = 8;                              // tiles per chunk = per ring slot: two per warp of a group, computed side by side (widths are multiples of 1024, eight tiles)

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

}  // namespace
