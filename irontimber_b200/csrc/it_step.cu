// One greedy decode step of the decoder as ONE persistent kernel.
//
// The per-op schedule of a pass (it_engine_run.cu; the reference's run_chunk_v, src/vk/mod.rs:763-892) is a chain of about
// ten dependent kernels per layer.  At one activation row every kernel is a few microseconds long, so most of a step is
// spent draining and refilling the GPU at kernel boundaries, not streaming weights.  This kernel runs the whole step with
// one CTA per SM that stays resident: the ops of the schedule become phases, and a producer warp per CTA streams the CTA's share of
// every ternary matrix of the step, in schedule order, into a ring in shared memory.  Weights never depend on activations, so the
// producer is only ever held back by the ring being full: while the CTAs wait for a phase's input, the ring already holds the
// first 136 KB per SM of the next matrix, and the HBM stream does not drain at op boundaries.
//
// Arithmetic: every phase performs, per output element, the operations of the kernel it replaces in the same order (the
// kernels of it_support.cu, it_hadamard.cuh, it_matvec_t2.cu), so logits, state and picks are bit-identical to the per-op
// schedule; tests run both and compare.  What changes is only which thread does the work and where intermediate values live.
//
// Phases of a layer:
//   A  rmsnorm -> Hadamard -> q8k of the residual row: one CTA per block of 1024; the dense beta / alpha rows of a delta-net layer
//      from the same normed row: one CTA per row
//   B  everyone: the input projection.  The lane that has added up a row finishes it: conv + SiLU or SiLU (delta-net), or as it is
//   C  delta-net: l2norms + delta rule + gated norm, one CTA per value head; attention: four CTAs per head
//   D  Hadamard -> q8k of the block's output row
//   E  everyone: the output projection, into the residual
//   F  as A, with the layer's other norm
//   G  everyone: gate / up, silu(gate) * up by the lane that has both
//   H  Hadamard -> q8k of the activation row
//   I  everyone: the down projection, into the residual
// then output norm + Hadamard + q8k, the LM head with the greedy pick folded into its epilogue, and the pick's hand-over
// to the next step (token slot, position + 1).
//
// What bounds it.  One row leaves 15.5 us of weight stream a layer; a delta-net layer of the 27B shape takes 44 us (61 with a grid
// barrier after each phase), the rest is latency: a value takes about 0.5 us from one SM to another, a block's transform 1.5,
// the first round of tiles 0.6, a row's last terms 0.4 and its tail, the delta rule 3.5.  What follows from that: values travel
// with tags instead of behind barriers (granules, below); a matrix is cut into equal runs of chunks whatever row groups they
// start in; transforms are as parallel as their blocks and no phase is repeated by everyone (every CTA transforming the whole
// row cost 2.3 us where the owners' way costs 1.4 and one more hop).  Code is kept small: measured on this GPU, straight-line code
// runs at one instruction per cycle and scheduler while it fits 32 KB, at half that up to about 100 KB, at a sixth beyond 128 KB.
//
// Every wait (mbarrier, counter, tag) is bounded; when one runs out the CTA raises the context's error flag and an abort word
// that ends every other CTA's waits, publishes nothing more, drains its copies and returns (IT_ETIMEOUT on the host).  What the
// phases before it wrote (state, caches) stays written; no phase computes from values that did not come.
#define IT_PIPE_OUTLINE_WAIT  // one copy of the retry loop of bounded waits
#define IT_MATH_OUTLINE      // one copy of division, square root and the elementary functions: this kernel's code size is its speed
#include "it_math.h"
#include "it_engine.h"
#include "it_support.h"
#include "it_pipe.cuh"
#include "it_hadamard.cuh"
#include "it_step_plan.h"
#include <algorithm>
#include <vector>

namespace {

constexpr int ST_CW = 4;                               // warps per consumer group
constexpr int ST_NG = 3;                               // consumer groups; group j takes the chunks i of a phase with i % ST_NG == j
constexpr int ST_NCONS = ST_CW * ST_NG;                // consumer warps
constexpr int ST_CT = ST_NCONS * 32;                   // consumer threads
static_assert(ST_CHUNK == ST_TPC * IT_TILE_BYTES && ST_PITCH == IT_HAD_PITCH, "it_step_plan.h");
constexpr int ST_NSUM = 2;                             // warps that only add the per-block terms in block order
constexpr int ST_THREADS = ST_CT + (ST_NSUM + 1) * 32; // + the sum warps + the producer warp

struct StepLayer {
    const uint8_t *in_proj, *out_proj, *gate_up, *down;
    const float *attn_norm, *post_norm;
    const float *conv_w, *dt, *a, *beta, *alpha, *ssm_norm;
    float *conv_st, *ssm_st;
    const float *q_norm, *k_norm;
    __half *kc, *vc;
    int recurrent, in_rows;
};

// Values that one CTA hands to others travel as granules: 16 bytes written and read by single 128-bit accesses, three values and
// the tag of the phase that made them (32 rows of a row group: eleven granules).  A reader that finds the tag has the values; no
// fence is involved.  Why: one value crosses between two SMs in about 960 cycles whatever else the memory system does, but a
// release or acquire-release fence takes 840 cycles on an idle GPU and 1900 while weights stream in, on every CTA's way into
// every barrier.  Tags grow from phase to phase and launch to launch, so no granule needs to be cleared.
// What keeps a buffer until its last reader is through, since nobody waits for everyone (a layer's chain: A to I as above):
//   codes      step_codes_half: A (F) needs every row of I (E), whose CTAs have read what it overwrites; D and H have the other half
//   rows       the next input projection follows an A that needed the heads' o through E .. I; every row belongs to a head that has read it
//   o, act     D (H) reads them; the next heads (gate / up) follow an A or F that needed every row behind all of its blocks
//   xe, xi     read by F (A) and, row by row, by I (E), into whose rows they go; the next E (I) follows a row that needed all of those
//   gate       a head reads its pair; the next dense rows follow an A that needed that head's o
//   prefix     the reader finishes a row of the phase, and the next phase's matrix follows a transform that needed all of them
//   scores     read by the head's CTAs before their o
// tests/test_step_protocol.py walks all of it with CTAs as late as they like.
typedef uint4 granule;
constexpr int ST_GPU = 11;                             // granules of a row group (32 rows)
constexpr int ST_COPIES = 4;                           // copies of the quantised row: all SMs read it at once, and its few lines would crowd a few L2 slices

struct StepParams {
    const StepLayer* layers; const StepSpan* spans; int n_layer;
    int e, ff, widest, hd, nh, nkv, cd, inner, nv, nk, qk, conv_k, n_rot, n_vocab;
    float eps, theta_scale; int sec[4]; int v_grouped;
    float* arena; size_t hrow, logits, amx;
    granule *xe, *xi, *rows, *o, *act; // residual row after the output / down projection; input projection's rows; block output; silu(gate) * up
    unsigned long long* o1;            // block output of attention heads whose dimension is no multiple of 32: a value and its tag an element (else null)
    granule* codes; int codes_half;    // the quantised row: 128 granules a block of 1024, ST_COPIES copies; codes_half granules further: the other half (step_codes_half)
    unsigned long long* gate;          // per value head beta, then decay: value and tag
    granule* prefix;                   // [grid][32] running sums of a cut row group (two matrices' worth) and the tag
    granule* partials;                 // one greedy-pick partial per sum warp: value, row, tag
    unsigned long long* att_sc; int att_stride;   // per head: the scores its CTAs exchange [nh][att_stride] (value and tag)
    const uint32_t* sg[4];             // sign bits of the four widths (n_embd, ssm_inner, attention output, n_ff), 32 words a block of 1024
    const float *tok_embd, *output_norm; const uint8_t* output;
    uint32_t* toks; int* pos;
    unsigned* sync;                    // [0] arrivals, [1] arrivals at the end of the last launch, [2] abort word
    int* error_flag;
    unsigned long long* trace;         // optional: clock readings of CTA 0 and of the last CTA at the waits in front of matrix phases (arrive, leave)
    int slots, scratch, w_off;         // ring slots; bytes of the phase scratch that follows the ring; where a norm's weights lie in it (a dense row in front of them)
    int attn_g;                        // CTAs that share an attention head
    int attn_base;                     // first CTA of the attention heads (value heads start at CTA 0; dense rows count down from the last CTA)
    int had_step;                      // the CTAs that transform the activation row's blocks are this far apart
    int gdn_off;                       // where the delta-net block keeps its state tile inside the scratch (clear of the input projection's buffers)
    int flags;                         // bit 0: the token is the previous pick (amx) instead of toks[0]; bit 1: hand the pick over (toks[0], pos + 1); bit 2: logits wanted
};

struct Pick { float v; unsigned i; };
__device__ __forceinline__ Pick pick_better(Pick a, Pick b) { return (b.v > a.v || (b.v == a.v && b.i < a.i)) ? b : a; }

// Per-thread view of the CTA's state that every phase needs.
struct Cta {
    unsigned char* smem; unsigned char* scratch; unsigned bars; volatile int* abort_flag;
    volatile int* verdict;             // thread 0's answer after a wait, so that all consumer warps leave or stay together
    int tid, warp, lane;
    unsigned q;                        // chunks of the CTA's stream passed so far (slot = q % slots, phase = (q / slots) & 1; slots is a power of two)
    unsigned tf, ps, pd, dn;           // mbarriers: terms of a slot's chunk in place [slots], phase started, phase summed, dense row's warp sums in place
    unsigned issued;                   // where the producer says how many chunks of the stream it has issued
    unsigned mph;                      // matrix phases so far
    unsigned at;                       // mbarriers of the attention block: K full / free, V full / free, eight of each
    const StepLayer* lay;              // the two shared-memory copies of layer descriptions (layer il at lay[il & 1])
    const StepSpan* sp;                // this CTA's spans, by matrix kind
    unsigned base, target;             // tags of this launch start here; what the counter reaches when the transforms so far have begun
    int nsync;                         // waits in front of matrix phases passed so far (index into the trace)
    unsigned dense_seq;                // dense rows this sum warp has finished in this launch
    float inv_sqrt_sd, inv_sqrt_hd;    // 1 / sqrt(state size), 1 / sqrt(head dimension): formed once per launch
    int evt_on, evt_base;              // diagnostics: this thread records fine-grained events into slots evt_base ..
};
constexpr int ST_TRACE_MAX = 1024;     // waits recorded per traced CTA
constexpr int ST_EVT_MAX = 2048;       // fine-grained events (diagnostics)
// Diagnostics: slot `id` of the event area receives the nanosecond clock when the chosen thread passes (one store, no read).
// fine-grained events are compiled in only with -DIT_STEP_EVENTS: their two dozen sites cost 2.8 KB of code, about 1 % of a step
#ifndef IT_STEP_EVENTS
#define ST_EV(P, c, id) do { } while (0)
#else
#define ST_EV(P, c, id) do { if ((P).trace && (c).evt_on && (c).lane == 0) { unsigned long long t_; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_)); (P).trace[4 * ST_TRACE_MAX + (id)] = t_; } } while (0)
#endif

__device__ __forceinline__ void cons_sync() { consumer_barrier<ST_CT>(); }
// four u8 x s8 products added to c
__device__ __forceinline__ int dp4a_us(unsigned a, int b, int c) { int d; asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c)); return d; }
__device__ __forceinline__ granule ld_granule(const granule* p) {
    unsigned long long a, b;
    asm volatile("{\n.reg .b128 q;\nld.relaxed.gpu.global.b128 q, [%2];\nmov.b128 {%0, %1}, q;\n}" : "=l"(a), "=l"(b) : "l"(p) : "memory");
    return make_uint4((unsigned)a, (unsigned)(a >> 32), (unsigned)b, (unsigned)(b >> 32));
}
__device__ __forceinline__ void st_granule(granule* p, unsigned x, unsigned y, unsigned z, unsigned tag) {
    const unsigned long long a = (unsigned long long)y << 32 | x, b = (unsigned long long)tag << 32 | z;
    asm volatile("{\n.reg .b128 q;\nmov.b128 q, {%1, %2};\nst.relaxed.gpu.global.b128 [%0], q;\n}" :: "l"(p), "l"(a), "l"(b) : "memory");
}
// A wait ran out: the host is told, the other CTAs (the abort word) and the other roles of this one.  From then on nothing that this CTA
// publishes can be relied on, and none of its roles publishes anything more.
__device__ __noinline__ void give_up(const StepParams& P, volatile int* abort_flag, int site) { atomicExch(P.error_flag, site); atomicExch(P.sync + 2, 1u); *abort_flag = 1; }
// A wait for tagged values has gone round `it` times: true when it has to end without them (the abort flag is up).
__device__ __noinline__ bool tag_late(const StepParams& P, unsigned it, long long t0, volatile int* abort_flag, int site) {
    if (it & 31u) return false;
    if (*abort_flag) return true;
    if (*reinterpret_cast<volatile unsigned*>(P.sync + 2)) { *abort_flag = 1; return true; }       // another CTA has given up
    if (clock64() - t0 > WAIT_CLOCKS) { give_up(P, abort_flag, site); return true; }
    return false;
}
// The granule, with another tag when the wait had to end without it.
__device__ __noinline__ granule wait_granule(const StepParams& P, const granule* p, unsigned tag, volatile int* abort_flag, int site) {
    const long long t0 = clock64();
    granule v;
#pragma unroll 1
    for (unsigned it = 1;; it++) { v = ld_granule(p); if (v.w == tag || tag_late(P, it, t0, abort_flag, site)) return v; }
}
// Granules p, p + stride, ... (n of them, n <= N; the last one again in the places behind it): all requested, then all again until
// each has its tag.  Bounded by a count of round trips (at least 500 cycles each); no call, so that nothing is spilled around it.
constexpr unsigned ST_POLLS = 1u << 22;
template <int N> __device__ __forceinline__ void read_granules(granule (&g)[N], const granule* p, int stride, int n, unsigned tag, const StepParams& P, const Cta& c, int site) {
#pragma unroll 1
    for (unsigned it = 0;; it++) {
#pragma unroll
        for (int u = 0; u < N; u++) g[u] = ld_granule(p + min(u, n - 1) * stride);
        unsigned miss = 0;
#pragma unroll
        for (int u = 0; u < N; u++) miss |= g[u].w ^ tag;
        if (miss == 0) return;
        if (*c.abort_flag) return;
        if ((it & 63u) == 63u && *reinterpret_cast<volatile unsigned*>(P.sync + 2)) { *c.abort_flag = 1; return; }
        if (it == ST_POLLS) { give_up(P, c.abort_flag, site); return; }
    }
}
// value and tag in one 8-byte word
__device__ __forceinline__ void st_tagged(unsigned long long* p, float v, unsigned tag) { asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" :: "l"(p), "l"((unsigned long long)tag << 32 | __float_as_uint(v)) : "memory"); }
__device__ __noinline__ float ld_tagged(const StepParams& P, const unsigned long long* p, unsigned tag, volatile int* abort_flag, int site) {
    const long long t0 = clock64();
#pragma unroll 1
    for (unsigned it = 1;; it++) {
        unsigned long long v; asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
        if ((unsigned)(v >> 32) == tag || tag_late(P, it, t0, abort_flag, site)) return __uint_as_float((unsigned)v);
    }
}
// One value per lane of a warp (32 consecutive rows) as the granules of row group u.
__device__ __forceinline__ void publish(granule* dst, int u, int lane, float v, unsigned tag, bool lost = false) {
    const float b = __shfl_down_sync(0xffffffffu, v, ST_GPU), d = __shfl_down_sync(0xffffffffu, v, 2 * ST_GPU);
    if (lane < ST_GPU && !lost) st_granule(dst + (size_t)u * ST_GPU + lane, __float_as_uint(v), __float_as_uint(b), __float_as_uint(d), tag);
}
// Granule i of a run of row groups holds rows r, r + 11 and (unless it is the last of its row group) r + 22.
__device__ __forceinline__ int granule_row(int i, bool& two) { const int u = i / ST_GPU, l = i - u * ST_GPU; two = l == ST_GPU - 1; return u * 32 + l; }
__device__ __forceinline__ unsigned tag_of(unsigned base, int il, int sub) { return base + 1u + (unsigned)(ST_SUBS * il + sub); }
// Nothing waits for everyone: a phase starts where its granules are, and polls them.  All CTAs polling a row through the whole of
// the phases that lead to it would take bandwidth from the weights, so they wait on a counter until the owners of the row's
// blocks have begun to transform them (a hint: it orders nothing and needs no fence), about 1500 cycles before the codes come.
// A barrier instead costs 3800 cycles from the last arrival with release adds while weights stream in, 1400 with relaxed ones, and
// another round trip for the row behind it.
__device__ __forceinline__ void count_up(unsigned* counter) { asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" :: "l"(counter) : "memory"); }
__device__ __forceinline__ void grid_arrive(const StepParams& P) { count_up(P.sync); }
__device__ __noinline__ void trace_clock(unsigned long long* trace, int nsync, int side) {
    if ((blockIdx.x == 0 || blockIdx.x == gridDim.x - 1) && nsync < ST_TRACE_MAX) {
        unsigned long long t; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        trace[((size_t)(blockIdx.x ? 1 : 0) * ST_TRACE_MAX + nsync) * 2 + side] = t;
    }
}
// Consumer threads only: thread 0 waits until `counter` has reached `target`.  Returns false when the step has been given up (by
// this CTA's own timeout or by another CTA's).
__device__ __forceinline__ bool count_wait(const StepParams& P, Cta& c, const unsigned* counter, unsigned target, int site, bool traced = true) {
    if (c.tid == 0) {
        if (P.trace && traced) trace_clock(P.trace, c.nsync, 0);
        const long long t0 = clock64();
#pragma unroll 1
        for (unsigned it = 0;; it++) {
            unsigned v; asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
            if ((int)(v - target) >= 0) break;
            if ((it & 63u) == 63u) {
                if (*c.abort_flag) break;
                if (*reinterpret_cast<volatile unsigned*>(P.sync + 2)) { *c.abort_flag = 1; break; }
                if (clock64() - t0 > WAIT_CLOCKS) { give_up(P, c.abort_flag, 100 + site); break; }
            }
        }
        const int gone = *c.abort_flag;
        if (gone) atomicExch(P.sync + 2, 1u);                        // a wait inside this CTA ran out (mbarriers do not tell the others)
        *c.verdict = gone;
        if (P.trace && traced) trace_clock(P.trace, c.nsync++, 1);
    }
    cons_sync();
    return !*c.verdict;
}

// The ternary matvecs of a step in order: four per layer (input projection, output projection, gate/up, down), then the
// LM head.  Every role of the CTA (producer, consumers, sum warps) walks this list with ONE copy of its loop in the code.
__device__ __forceinline__ int mat_count(const StepParams& P) { return 4 * P.n_layer + ((P.flags & 4) ? 1 : 0); }
__device__ __forceinline__ int span_kind(int sub, int recurrent) { return sub == 0 ? (recurrent ? SP_IN_GDN : SP_IN_ATT) : sub == 1 ? (recurrent ? SP_OUT_GDN : SP_OUT_ATT) : sub == 2 ? SP_GATE_UP : SP_DOWN; }

// A wait on an mbarrier sees the parity of a phase only, so whoever waits for chunk q of a slot must know that the chunk before it in that
// slot is through: a sum warp that leaves a row group of more chunks than the ring has slots to the other one, or a consumer group
// whose chunk's predecessor was another group's, otherwise takes the phase before for its own - it adds terms that are not there yet, or
// hands a slot back twice.  The producer issues a chunk when its slot has been handed back, so it says how many chunks it has
// issued, and nobody looks at a chunk's barriers before it is among them (the first `slots` of a phase follow chunks of the phase
// before, which everyone knows to be through).
__device__ __forceinline__ void st_issued(unsigned at, unsigned n) { asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" :: "r"(at), "r"(n) : "memory"); }
__device__ __forceinline__ unsigned ld_issued(unsigned at) { unsigned v; asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(at) : "memory"); return v; }
// The chunks issued once chunk q is one of them; fewer when the wait had to end without it.
__device__ __noinline__ unsigned issued_past(unsigned at, unsigned q, volatile int* abort_flag, int* error_flag, int site) {
    const long long t0 = clock64();
#pragma unroll 1
    for (;;) {
        const unsigned v = ld_issued(at);
        if ((int)(v - q) > 0 || *abort_flag) return v;
        if (clock64() - t0 > WAIT_CLOCKS) { if (!*abort_flag) atomicExch(error_flag, site); *abort_flag = 1; return v; }
        __nanosleep(32);
    }
}
// Waits for the chunk's bytes; `issued`: chunks known to have been issued, or to follow a phase that is through.
__device__ __forceinline__ bool chunk_wait(unsigned bar, unsigned parity, unsigned q, unsigned& issued, const StepParams& P, const Cta& c, int site) {
    if ((int)(issued - q) <= 0) {
        issued = issued_past(c.issued, q, c.abort_flag, P.error_flag, site);
        if ((int)(issued - q) <= 0) return false;
    }
    return mbar_wait(bar, parity, c.abort_flag, P.error_flag, site);
}

// Whoever starts bulk copies leaves only when they have landed, also where nobody waits for them any more: the last `issued` copies of
// a ring of `slots` with full barriers at `full` (each wait bounded by the clock limit).
__device__ __noinline__ void drain_copies(unsigned full, unsigned slots, unsigned issued) {
#pragma unroll 1
    for (unsigned k = issued > slots ? issued - slots : 0u; k < issued; k++) {
        const long long t0 = clock64();
        while (!mbar_test(full + 8 * (k % slots), (k / slots) & 1u) && clock64() - t0 < WAIT_CLOCKS) { }
    }
}

// ---------------------------------------------------------------- producer
__device__ __forceinline__ void producer(const StepParams& P, const Cta& c) {
    int s = 0, issued = 0; unsigned ph = 0u;
    bool ok = true;
    const int nmat = mat_count(P);
#pragma unroll 1
    for (int mp = 0; mp < nmat && ok; mp++) {
        const int il = mp >> 2, sub = mp & 3;
        const uint8_t* tiles = P.output; int kind = SP_HEAD;
        if (il < P.n_layer) { const StepLayer& L = P.layers[il]; kind = span_kind(sub, L.recurrent); tiles = sub == 0 ? L.in_proj : sub == 1 ? L.out_proj : sub == 2 ? L.gate_up : L.down; }
        const StepSpan sp = c.sp[kind];
        const int cpu = sp.cpr * sp.parts;
        int unit = sp.uh, cq = 0;
#pragma unroll 1
        for (int i = 0; i < sp.n; i++) {
            if (i == sp.hl) { unit = sp.uf; cq = 0; }
            if (i == sp.n - sp.tl) { unit = sp.ut; cq = sp.lead; }
            if (!mbar_wait(c.bars + 8 * (P.slots + s), ph ^ 1u, c.abort_flag, P.error_flag, 2)) { ok = false; break; }
            st_issued(c.issued, (unsigned)issued + 1u);
            const bool second = cq >= sp.cpr;
            mbar_expect_tx(c.bars + 8 * s, ST_CHUNK);
            bulk_load(smem_u32(c.smem + s * ST_CHUNK), tiles + ((size_t)(second ? unit + sp.units : unit) * sp.cpr + (second ? cq - sp.cpr : cq)) * ST_CHUNK, ST_CHUNK, c.bars + 8 * s);
            issued++;
            if (++s == P.slots) { s = 0; ph ^= 1u; }
            if (++cq == cpu) { cq = 0; unit++; }
        }
    }
    drain_copies(c.bars, (unsigned)P.slots, (unsigned)issued);
}

// Vectors that a later phase reads once: on their way into L2 while the weight stream would make them wait (lines of 128 bytes, a thread each).
__device__ __forceinline__ void warm_l2(const void* p, int bytes, int i) {
    if (i >= 0 && i * 128 < bytes) asm volatile("prefetch.global.L2 [%0];" :: "l"(reinterpret_cast<const char*>(p) + (size_t)i * 128));
}
// The next layer's (or, behind the last layer, the output norm's): by the last CTA; the conv taps and state of a CTA's own rows by that CTA.
__device__ __forceinline__ void warm_layer(const StepParams& P, const Cta& c, const StepLayer& N, int drow) {
    const int tid = c.tid;
    if (blockIdx.x == gridDim.x - 1) {
        warm_l2(N.attn_norm, P.e * 4, tid); warm_l2(N.post_norm, P.e * 4, tid);
        if (N.recurrent) { warm_l2(N.ssm_norm, ST_SD * 4, tid); warm_l2(N.dt, P.nv * 4, tid - 32); warm_l2(N.a, P.nv * 4, tid - 64); }
        else { warm_l2(N.q_norm, P.hd * 4, tid); warm_l2(N.k_norm, P.hd * 4, tid - 32); }
    }
    if (!N.recurrent) return;
    if (drow < 2 * P.nv) warm_l2((drow < P.nv ? N.beta : N.alpha - (size_t)P.nv * P.e) + (size_t)drow * P.e, P.e * 4, tid);
    const StepSpan& sp = c.sp[SP_IN_GDN];
    const int u = (sp.tl ? sp.ut : sp.uf) + (tid >> 4), k = tid & 15, row = u * 32;      // sixteen threads a row group: conv_k - 1 state rows, conv_k lines of taps
    if (row < P.cd && (tid >> 4) * sp.cpr < sp.n + sp.cpr) {
        if (k < P.conv_k - 1) warm_l2(N.conv_st + (size_t)k * P.cd + row, 128, 0);
        else warm_l2(N.conv_w + (size_t)row * P.conv_k, 128 * P.conv_k, k - (P.conv_k - 1));
    }
}

// ---------------------------------------------------------------- row transform
// [rmsnorm ->] signs -> Hadamard -> q8k of one block of 1024 of a row, by the CTA that owns it, in the operation order of
// it_hadamard_block (it_hadamard.cuh).  All consumer warps bring the row in (a normed one whole, else the block) and form the
// norm; two of them transform the block, 16 values a thread.  The row is read in lane order and put into the padded layout
// of the transform (64 bytes a thread straight into registers: 24 KB cost 2000 cycles with all SMs at it, in lane order 560).
// The norm's weights and the dense row do not depend on the step and are in shared memory before the row is.
struct RowIn {
    const granule* x; unsigned tag; const float* plain; const unsigned long long* one;      // the row (norm) or its block, as granules of a phase, as floats (plain), or as tagged values (one)
    const uint32_t* signs; float* normed;                    // normed: where the normed row goes, or null
    granule* codes; unsigned code_tag; int codes_copy;       // where the quantised block goes (copies codes_copy granules apart), or null
    int nblk, blk; bool norm, dense;                         // blocks brought in, the one to transform; dense: multiply the normed row with this CTA's dense row
    const float* dense2;                                     // ... and with this second one (in global memory), or null
};
__device__ __forceinline__ void pair_sync() { asm volatile("bar.sync 5, 64;" ::: "memory"); }
// nblk blocks of 1024 rows (32 row groups, 352 granules: a thread each) from `x` into the padded layout at `ex`
constexpr int ST_GPB = 32 * ST_GPU;
static_assert(ST_GPB <= ST_CT, "a granule of every block per thread");
__device__ __forceinline__ void row_place(const StepParams& P, const Cta& c, float* ex, const granule* x, int nblk, unsigned tag) {
    constexpr int N = 6;
    if (c.tid >= ST_GPB) return;
    bool two; const int r = granule_row(c.tid, two);
    float *p0 = ex + it_had_at(r), *p1 = ex + it_had_at(r + ST_GPU), *p2 = two ? p1 : ex + it_had_at(r + 2 * ST_GPU);
#pragma unroll 1
    for (int b = 0; b < nblk; b += N, p0 += N * IT_HAD_PITCH, p1 += N * IT_HAD_PITCH, p2 += N * IT_HAD_PITCH) {
        granule g[N];
        const int m = min(N, nblk - b);
        read_granules(g, x + b * ST_GPB + c.tid, ST_GPB, m, tag, P, c, 14);
#pragma unroll
        for (int u = 0; u < N; u++) {
            const int o = min(u, m - 1) * IT_HAD_PITCH;
            p2[o] = __uint_as_float(two ? g[u].y : g[u].z); p0[o] = __uint_as_float(g[u].x); p1[o] = __uint_as_float(g[u].y);
        }
    }
}
// Requests a norm's weights (padded layout, at shared-memory address wb) and, for a CTA that has one, a dense row (natural order,
// in front of them); one group per thread.
__device__ __noinline__ void norm_request(float* wb, const float* w, const float* dense, int e) {
    const int tid = threadIdx.x;
#pragma unroll 1
    for (int i = 4 * tid; i < e; i += 4 * ST_CT) {
        cp_async16(wb + (i >> 10) * IT_HAD_PITCH + it_had_at(i & 1023), w + i);
        if (dense) cp_async16(wb - e + i, dense + i);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <bool ANY> __device__ __forceinline__ void block_transform(const StepParams& P, const Cta& c, const RowIn in) {
    const int tid = c.tid, warp = c.warp, lane = c.lane, j = tid & 63;
    const int n = in.nblk * 1024;
    float* ex0 = reinterpret_cast<float*>(c.scratch + ST_RED);
    float* red = reinterpret_cast<float*>(c.scratch + 64);   // [8] warp sums of squares, [4][2] group maxima
    const float* wb = reinterpret_cast<const float*>(c.scratch + P.w_off);
    const unsigned m16 = warp < 2 && in.codes ? reinterpret_cast<const unsigned short*>(in.signs)[j] : 0u;      // the thread's sixteen signs, here long before the row
    cons_sync();                                             // the scratch is nobody's any more (the block before may still have been writing state)
    if (in.plain) {
#pragma unroll 1
        for (int i = 4 * tid; i < n; i += 4 * ST_CT) *reinterpret_cast<float4*>(ex0 + it_had_at(i)) = *reinterpret_cast<const float4*>(in.plain + i);
    } else if (ANY && in.one) {
#pragma unroll 1
        for (int i = tid; i < n; i += ST_CT) ex0[it_had_at(i)] = ld_tagged(P, in.one + i, in.tag, c.abort_flag, 14);
    } else row_place(P, c, ex0, in.x, in.nblk, in.tag);
    asm volatile("cp.async.wait_group 0;" ::: "memory");             // the norm's weights
    cons_sync();
    const bool lost = *c.abort_flag;                                 // the row may not have come
    if (tid == 0 && in.codes && !lost) grid_arrive(P);               // the codes will follow
    float sc = 0.f;
    if (in.norm) {
        // rmsnorm of the whole row in the order of k_rmsnorm_wide: thread i of 256 adds x[i]^2, x[i + 256]^2, ...; warp
        // butterflies; eight warp sums in ascending order
        if (tid < 256) {
            const float* xp = ex0 + it_had_at(tid);
            float s = 0.f, a[4];
#pragma unroll
            for (int u = 0; u < 4; u++) a[u] = xp[336 * u];
#pragma unroll 1
            for (int k = 1; k <= in.nblk; k++) {                     // the next block's four elements are requested before this one's are added
                float b[4];
                xp += k < in.nblk ? IT_HAD_PITCH : 0;
#pragma unroll
                for (int u = 0; u < 4; u++) b[u] = xp[336 * u];
#pragma unroll
                for (int u = 0; u < 4; u++) { s = it_add(s, it_mul(a[u], a[u])); a[u] = b[u]; }
            }
#pragma unroll
            for (int m = 16; m >= 1; m >>= 1) s = it_add(s, __shfl_xor_sync(0xffffffffu, s, m));
            if (lane == 0) red[warp] = s;
        }
        cons_sync();
        float tot = red[0];
#pragma unroll
        for (int k = 1; k < 8; k++) tot = it_add(tot, red[k]);
        sc = __fdiv_rn(1.0f, __fsqrt_rn(it_add(__fdiv_rn(tot, (float)n), P.eps)));
        if (in.normed) {
#pragma unroll 1
            for (int i = tid; i < n; i += ST_CT) { const int o = (i >> 10) * IT_HAD_PITCH + it_had_at(i & 1023); in.normed[i] = it_mul(it_mul(ex0[o], sc), wb[o]); }
            cons_sync();
        }
        if (in.dense) {
            if (tid < 256) {
                // one row of the beta / alpha matrices times the normed row, in the order of k_dense_rows: thread i adds the
                // products i, i + 256, ... in f64, warp butterflies, eight warp sums in ascending order (by sum warp 1)
                const float* xp = ex0 + it_had_at(tid); const float* wp = wb + it_had_at(tid); const float* dp = wb - P.e + tid;
                double d = 0.0;
#pragma unroll 2
                for (int k = 0; k < in.nblk * 4; k++) d += (double)it_mul(dp[256 * k], it_mul(it_mul(xp[336 * k], sc), wp[336 * k]));
#pragma unroll
                for (int m = 16; m >= 1; m >>= 1) d += __shfl_xor_sync(0xffffffffu, d, m);
                if (ANY && in.dense2) {
                    double d2 = 0.0;
                    dp = in.dense2 + tid;
#pragma unroll 1
                    for (int k = 0; k < in.nblk * 4; k++) d2 += (double)it_mul(dp[256 * k], it_mul(it_mul(xp[336 * k], sc), wp[336 * k]));
#pragma unroll
                    for (int m = 16; m >= 1; m >>= 1) d2 += __shfl_xor_sync(0xffffffffu, d2, m);
                    if (lane == 0) reinterpret_cast<double*>(c.scratch + ST_DENSE2)[warp] = d2;
                }
                if (lane == 0 && !lost) { reinterpret_cast<double*>(c.scratch)[warp] = d; mbar_arrive(c.dn); }
            }
            cons_sync();                                     // the row is about to be overwritten
        }
    }
    if (warp < 2 && in.codes) {
        float* ex = ex0 + in.blk * IT_HAD_PITCH;
        {
            float v[16];
            float* p1 = ex + it_had_at(16 * j);
#pragma unroll
            for (int u = 0; u < 4; u++) { const float4 t = *reinterpret_cast<const float4*>(p1 + 4 * u); v[4 * u] = t.x; v[4 * u + 1] = t.y; v[4 * u + 2] = t.z; v[4 * u + 3] = t.w; }
            if (in.norm) {
                const float* wp = wb + in.blk * IT_HAD_PITCH + it_had_at(16 * j);
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const float4 w = *reinterpret_cast<const float4*>(wp + 4 * u);
                    v[4 * u] = it_mul(it_mul(v[4 * u], sc), w.x); v[4 * u + 1] = it_mul(it_mul(v[4 * u + 1], sc), w.y);
                    v[4 * u + 2] = it_mul(it_mul(v[4 * u + 2], sc), w.z); v[4 * u + 3] = it_mul(it_mul(v[4 * u + 3], sc), w.w);
                }
            }
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] = __uint_as_float(__float_as_uint(v[i]) ^ ((m16 << (31 - i)) & 0x80000000u));     // times +-1
            it_had16_rotate(v, ex, j, [] { pair_sync(); });
            const it_had16_codes q = it_had16_quantise(v, red + 8, j, [] { pair_sync(); });
            // thread j: its four words of codes; threads 0..3 of each half also the group's scale and the half's sum
#pragma unroll 1
            for (int k = lost ? ST_COPIES : 0; k < ST_COPIES; k++) {
                granule* to = in.codes + k * in.codes_copy + j;
                st_granule(to, q.packed[0], q.packed[1], q.packed[2], in.code_tag);
                st_granule(to + 64, q.packed[3], __float_as_uint(q.d), (unsigned)q.sum, in.code_tag);
            }
        }
    }
}

// The quantised row of nblk blocks that other CTAs have published, into this CTA's scratch.
__device__ __forceinline__ void codes_place(const StepParams& P, const Cta& c, const granule* codes, int nblk, unsigned tag) {
    constexpr int N = 6, BPT = ST_CT / 128;                          // blocks a turn of all threads covers
    const int n = nblk * 1024, j = c.tid & 63, blk = c.tid >> 7; const bool odd = c.tid & 64;
    int8_t* xs = reinterpret_cast<int8_t*>(c.scratch + ST_RED);
    float* dxs = reinterpret_cast<float*>(xs + n) + blk * 4 + (j & 3);
    int* sss = reinterpret_cast<int*>(xs + n + n / 64) + blk * 8 + 2 * (j & 3) + (j >> 5);
    uint32_t* at = reinterpret_cast<uint32_t*>(xs + blk * 1024 + 4 * j) + (odd ? 192 : 0);
    const granule* src = codes + (blockIdx.x % ST_COPIES) * nblk * 128 + c.tid;
#pragma unroll 1
    for (int b = 0; b < nblk - blk; b += N * BPT, at += N * BPT * 256, dxs += N * BPT * 4, sss += N * BPT * 8, src += N * ST_CT) {
        const int m = min(N, (nblk - blk - b + BPT - 1) / BPT);
        granule g[N];
        read_granules(g, src, ST_CT, m, tag, P, c, 15);
#pragma unroll
        for (int u = 0; u < N; u++) {
            const int o = min(u, m - 1) * BPT;
            at[o * 256] = g[u].x;
            if (!odd) { at[o * 256 + 64] = g[u].y; at[o * 256 + 128] = g[u].z; }
            else if ((j & 31) < 4) { if (j < 4) dxs[o * 4] = __uint_as_float(g[u].y); sss[o * 8] = (int)g[u].z; }
        }
    }
    cons_sync();
}

// ---------------------------------------------------------------- ternary matvec phase (one activation row)
// Same arithmetic as k_matvec_t2<1> (it_matvec_t2.cu): per 32 x 128 tile the exact integer block sums, then the per-block
// terms (d_w * d_x) * float(S - sum128), which the sum warps add in ascending block order.  A chunk passes through one ring
// slot: producer -> consumers (a group of four warps) -> sum warp (terms of the slot), whose arrival frees the slot and its
// terms together.
__device__ __forceinline__ void matvec_phase(const StepParams& P, Cta& c, const StepSpan& sp) {
    const int warp = c.warp, lane = c.lane, nb = sp.nb, n = sp.n, hl = sp.hl, whole = sp.n - sp.tl, lead = sp.lead - whole, cpr = sp.cpr;   // in registers: stores to the terms would make the compiler fetch the span again
    const unsigned magic = sp.magic;
    const int8_t* xs = reinterpret_cast<const int8_t*>(c.scratch + ST_RED);
    const float* dxs = reinterpret_cast<const float*>(xs + nb * 128);
    const int* sss = reinterpret_cast<const int*>(xs + nb * 130);
    float* terms = reinterpret_cast<float*>(c.scratch + terms_at(nb));
    const int t = lane & 3, wi = warp % ST_CW;
    const int trow = (lane >> 2) + 8 * t;                            // the matrix row of a tile whose term this lane forms: g + 8 t
    const unsigned smask = (unsigned)P.slots - 1u; const int sshift = 31 - __clz(P.slots);
    // One activation row: integer dot products on the SIMT pipe (dp4a, u8 x s8).  Lane 4 g + t owns the 32 columns
    // 32 t .. 32 t + 31 of a tile and, per 32-bit word, the four matrix rows g, g + 8, g + 16, g + 24 (bit pairs 0..3 of
    // every byte).  Masks that keep everything up to a bit pair need three operations a word where isolating the pairs needs four;
    // the differences of the four sums are the rows' sums scaled by 1, 4, 16, 64.  The four lanes of a row group g then add
    // their sums (exact integers) in a reduce-scatter that leaves row g + 8 t with lane t, which forms that row's term.
    auto dots = [&](const unsigned char* tile, int b, int (&a)[4]) {
        const uint4 wa = *reinterpret_cast<const uint4*>(tile + 16 * lane);
        const uint4 wb = *reinterpret_cast<const uint4*>(tile + 512 + 16 * lane);
        const uint4* xp = reinterpret_cast<const uint4*>(xs + 128 * b + 32 * t);
        const uint4 xa = xp[0], xb4 = xp[1];
        const uint32_t w[8] = { wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w };
        const int xb[8] = { (int)xa.x, (int)xa.y, (int)xa.z, (int)xa.w, (int)xb4.x, (int)xb4.y, (int)xb4.z, (int)xb4.w };
        a[0] = a[1] = a[2] = a[3] = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            a[0] = dp4a_us(w[k] & 0x03030303u, xb[k], a[0]);
            a[1] = dp4a_us(w[k] & 0x0f0f0f0fu, xb[k], a[1]);
            a[2] = dp4a_us(w[k] & 0x3f3f3f3fu, xb[k], a[2]);
            a[3] = dp4a_us(w[k], xb[k], a[3]);
        }
        a[3] -= a[2]; a[2] -= a[1]; a[1] -= a[0];
    };
    auto term = [&](const unsigned char* tile, int b, const int (&a)[4]) {
        const bool hi2 = t & 2, hi1 = t & 1;
        int k0 = hi2 ? a[2] : a[0], k1 = hi2 ? a[3] : a[1];
        const int s0 = hi2 ? a[0] : a[2], s1 = hi2 ? a[1] : a[3];
        k0 += __shfl_xor_sync(0xffffffffu, s0, 2); k1 += __shfl_xor_sync(0xffffffffu, s1, 2);
        int S = hi1 ? k1 : k0;
        S += __shfl_xor_sync(0xffffffffu, hi1 ? k0 : k1, 1);
        const __half dwh = *reinterpret_cast<const __half*>(tile + 1024 + 2 * lane);   // scale of row g + 8 t: half 4 g + t
        return __fmul_rn(__fmul_rn(__half2float(dwh), dxs[b >> 1]), (float)((S >> (2 * t)) - sss[b]));
    };
    bool ok = !*c.abort_flag;                                        // (the row may not have come) a lane whose wait ran out goes on without waits and arrivals; the CTA leaves at its next wait
    unsigned issued = c.q + (unsigned)P.slots;                       // the slots of these were another phase's
#pragma unroll 1
    for (int i = warp / ST_CW; i < n; i += ST_NG) {
        const unsigned q = c.q + (unsigned)i;
        const int cs = (int)(q & smask);
        const unsigned r = (unsigned)(i < hl ? i : i < whole ? i - hl : i + lead);
        const int b0 = (cpr == 1 ? 0 : (int)(r - __umulhi(r, magic) * (unsigned)cpr)) * ST_TPC + wi, b1 = b0 + ST_CW;      // r modulo cpr: the chunk's index within its row of blocks
        if (ok) ok = chunk_wait(c.bars + 8 * cs, (q >> sshift) & 1u, q, issued, P, c, 3);
        const unsigned char *tile0 = c.smem + cs * ST_CHUNK + wi * IT_TILE_BYTES, *tile1 = tile0 + ST_CW * IT_TILE_BYTES;
        int a0[4], a1[4];
        dots(tile0, b0, a0); dots(tile1, b1, a1);
        const float t0 = term(tile0, b0, a0), t1 = term(tile1, b1, a1);
        float* tb = terms + cs * ST_TERMS + wi * 32 + trow;
        tb[0] = t0; tb[ST_CW * 32] = t1;
        __syncwarp();
        if (lane == 0 && ok) mbar_arrive(c.tf + 8 * cs);
    }
    c.q += (unsigned)n;
}

// The sum warps' side: warp j takes every second row group (in the order of the CTA's chunks), adds its terms in block order
// and finishes the row: into the residual, through conv and SiLU, through silu(gate) * up, or plainly.
template <bool ANY> __device__ __forceinline__ void sum_warps(const StepParams& P, Cta& c) {
    const int jw = c.warp - ST_NCONS, lane = c.lane;
    float* A = P.arena;
    Pick best{ -INFINITY, 0xffffffffu };
    const int nmat = mat_count(P);
    const unsigned smask = (unsigned)P.slots - 1u; const int sshift = 31 - __clz(P.slots);
    const float* xsrc;
    { const uint32_t tok = (P.flags & 1) ? __float_as_uint(*reinterpret_cast<volatile float*>(A + P.amx)) : *reinterpret_cast<volatile uint32_t*>(P.toks); xsrc = P.tok_embd + (size_t)tok * P.e; }
    const unsigned base = *reinterpret_cast<volatile unsigned*>(P.sync + 3);
    bool ok = true;
#pragma unroll 1
    for (int mp = 0; mp < nmat && ok; mp++) {
        const int il = mp >> 2, sub = mp & 3;
        const bool head = il >= P.n_layer;
        const StepLayer& L = P.layers[head ? 0 : il];
        const StepSpan sp = c.sp[head ? SP_HEAD : span_kind(sub, L.recurrent)];
        const int rows = head ? P.n_vocab : sub == 0 ? L.in_rows : sub == 2 ? P.ff : P.e;
        const int n = sp.n, cpu = sp.cpr * sp.parts;
        const float* terms = reinterpret_cast<const float*>(c.scratch + terms_at(sp.nb));
        const bool gdn_in = !head && sub == 0 && L.recurrent, accum = !head && (sub & 1);
        const int ph = head || sub == 0 ? PH_B : sub == 1 ? PH_E : sub == 2 ? PH_G : PH_I;
        const unsigned tag = tag_of(base, il, ph);
        granule* y = sub == 0 ? P.rows : sub == 1 ? P.xe : sub == 2 ? P.act : P.xi;
        // where the residual row comes from: the down projection of the layer before, or this layer's output projection
        const granule* yo = sub == 1 ? P.xi : P.xe; const unsigned old_tag = sub == 1 ? tag_of(base, il - 1, PH_I) : tag_of(base, il, PH_E);
        // not before the consumers have passed the barrier in front of this phase: an arrival of a warp without row groups
        // would count for the wrong barrier
        if (!mbar_wait_warp(c.ps, (unsigned)mp & 1u, c.abort_flag, P.error_flag, 7)) break;
        const int drow = (int)gridDim.x - 1 - (int)blockIdx.x;
        if (gdn_in && jw == 1 && drow < 2 * P.nv) {
            // the dense row of this CTA: beta (sigmoid) or alpha (decay) gate of a value head
            if (!mbar_wait_warp(c.dn, (c.dense_seq++) & 1u, c.abort_flag, P.error_flag, 12)) break;
            if (lane == 0) {
                const double* ws = reinterpret_cast<const double*>(c.scratch);
#pragma unroll 1
                for (int r = drow; r < (ANY ? 2 * P.nv : drow + 1); r += (int)gridDim.x, ws += ST_DENSE2 / 8) {
                    double tt = ws[0];
                    for (int k = 1; k < 8; k++) tt += ws[k];
                    const float tf = (float)tt;
                    const int h = r % P.nv;
                    st_tagged(P.gate + r, r < P.nv ? it_sigmoid(tf) : it_expf(it_mul(it_softplus(it_add(tf, L.dt[h])), L.a[h])), tag);
                }
            }
            __syncwarp();
        }
        unsigned issued = c.q + (unsigned)P.slots;
        int unit = sp.uf;
#pragma unroll 1
        for (int i = 0, ord = 0, len; i < n; i += len, ord++) {
            const bool first = i < sp.hl, last = !first && i >= n - sp.tl;       // begun here and finished by the next CTA / the other way round
            len = first ? sp.hl : last ? sp.tl : cpu;
            const int u = first ? sp.uh : last ? sp.ut : unit++;
            if ((ord & 1) != jw) continue;
            const int row = u * 32 + lane;
            const bool live = row < rows;
            float s = 0.f, sg = 0.f, old = 0.f;
            float st[3]; float4 cw;                                  // the usual conv size, four taps: operands on their way while the terms are added
            const bool conv = gdn_in && row < P.cd && !first;
            if (accum && live && !first) {
                if (sub == 1 && il == 0) old = xsrc[row];
                else { const int k = lane / ST_GPU; const granule og = wait_granule(P, yo + (size_t)u * ST_GPU + lane - k * ST_GPU, old_tag, c.abort_flag, 16); ok = ok && og.w == old_tag; old = __uint_as_float(k == 0 ? og.x : k == 1 ? og.y : og.z); }
            }
            if (conv && P.conv_k == 4) {
#pragma unroll
                for (int k = 0; k < 3; k++) st[k] = L.conv_st[(size_t)k * P.cd + row];
                cw = *reinterpret_cast<const float4*>(L.conv_w + (size_t)row * 4);
            }
            const int turn = last ? sp.cpr - sp.lead : sp.cpr;       // never reached when there is one matrix
            if (last) {
                // running sums of the blocks the CTA before has added (it does them first)
                const granule a = wait_granule(P, P.prefix + (size_t)(blockIdx.x - 1) * 32 + lane, tag, c.abort_flag, 13);
                ok = ok && a.w == tag;
                s = __uint_as_float(a.x); sg = __uint_as_float(a.y);
            }
            // a lane whose wait ran out goes on without waits; the warp leaves by a vote after the row group
            unsigned q = c.q + (unsigned)i;
            // the chunks before this row group's first `slots` in their slots may be the other warp's (behind those come its own): one look a row
            // group is 1 % of a step less than one a chunk
            const unsigned want = q + (unsigned)min(len, P.slots);
            if (ok && (int)(want - issued) > 0) { issued = issued_past(c.issued, want - 1u, c.abort_flag, P.error_flag, 6); ok = (int)(want - issued) <= 0; }
#pragma unroll 1
            for (int k = 0; k < len; k += 2, q += 2) {               // two chunks a turn: this warp has one issue slot in four, and half a turn is overhead
                const int c0 = (int)(q & smask), c1 = (int)((q + 1) & smask);
                const bool two = k + 1 < len;
                if (ok) ok = mbar_wait(c.tf + 8 * c0, (q >> sshift) & 1u, c.abort_flag, P.error_flag, 6);
                if (ok && two) ok = mbar_wait(c.tf + 8 * c1, ((q + 1) >> sshift) & 1u, c.abort_flag, P.error_flag, 6);
                const float *t0 = terms + c0 * ST_TERMS + lane, *t1 = terms + c1 * ST_TERMS + lane;
                float ta[ST_TPC], tb[ST_TPC];
#pragma unroll
                for (int b = 0; b < ST_TPC; b++) ta[b] = t0[32 * b];
#pragma unroll
                for (int b = 0; b < ST_TPC; b++) tb[b] = two ? t1[32 * b] : 0.f;      // + 0 changes no sum
                if (k == turn) { sg = s; s = 0.f; }                  // second matrix of the pair
#pragma unroll
                for (int b = 0; b < ST_TPC; b++) s = __fadd_rn(s, ta[b]);
                if (k + 1 == turn && two) { sg = s; s = 0.f; }
#pragma unroll
                for (int b = 0; b < ST_TPC; b++) s = __fadd_rn(s, tb[b]);
                __syncwarp();
                if (lane < (two ? 2 : 1) && ok) mbar_arrive(c.bars + 8 * (P.slots + (lane ? c1 : c0)));     // the slots may be refilled, their terms overwritten
            }
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            if (first) {
                st_granule(P.prefix + (size_t)blockIdx.x * 32 + lane, __float_as_uint(s), __float_as_uint(sg), 0u, tag);
                continue;
            }
            if (accum) {
                s = __fadd_rn(old, s);
            } else if (sp.parts == 2 || gdn_in) {
                if (conv) {
                    // conv over the row's last inputs (taps in order) and the state's shift by one input
                    const float mx = s;
                    if (P.conv_k == 4) {
                        s = it_add(it_add(it_add(it_add(0.f, it_mul(st[0], cw.x)), it_mul(st[1], cw.y)), it_mul(st[2], cw.z)), it_mul(mx, cw.w));
                        L.conv_st[row] = st[1]; L.conv_st[(size_t)P.cd + row] = st[2]; L.conv_st[2 * (size_t)P.cd + row] = mx;
                    } else {
                        s = 0.f;
#pragma unroll 1
                        for (int k = 0; k < P.conv_k; k++) {
                            float* at = L.conv_st + (size_t)k * P.cd + row;
                            const float x = k < P.conv_k - 1 ? *at : mx;
                            s = it_add(s, it_mul(x, L.conv_w[(size_t)row * P.conv_k + k]));
                            if (k) at[-(ptrdiff_t)P.cd] = x;
                        }
                    }
                }
                // silu(gate) * up; silu of a conv channel, or of a gate row behind them
                const float a = sp.parts == 2 ? sg : s, sl = __fdiv_rn(a, it_add(1.0f, it_expf_inline(-a)));
                s = sp.parts == 2 ? it_mul(sl, s) : sl;
            }
            if (head) { if (live) { __stcg(A + P.logits + row, s); best = pick_better(best, Pick{ s, (unsigned)row }); } }
            else {
                publish(y, u, lane, s, tag);
            }
        }
        c.q += (unsigned)n;
        if (!ok) break;
        if (head) {         // greedy pick (first index of the maximum) over this warp's rows
#pragma unroll
            for (unsigned mm = 16; mm > 0; mm >>= 1) { Pick o{ __shfl_xor_sync(0xffffffffu, best.v, mm), __shfl_xor_sync(0xffffffffu, best.i, mm) }; best = pick_better(best, o); }
            if (lane == 0) st_granule(P.partials + blockIdx.x * ST_NSUM + jw, __float_as_uint(best.v), best.i, 0u, tag);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(c.pd);                            // this phase's terms have been read
    }
    if (ok && lane == 0) grid_arrive(P);
}

// ---------------------------------------------------------------- delta-net block of one value head
// l2norm of q and k, the delta rule and the gated norm for head blockIdx.x, in the operation order of k_conv_l2_dense and
// k_gdn_norm (it_support.cu; src/cpu.rs:199-237); conv, SiLU and the gates come from the input projection's phase.
// Issued by the CTA of value head blockIdx.x while the input projection runs: the head's state tile (64 KB, it does not
// depend on this step's activations) into its place in shared memory.
__device__ __forceinline__ void gdn_prefetch(const StepParams& P, const StepLayer& L, const Cta& c, int h) {
    constexpr int SD = ST_SD, PPR = SD / 4;
    float* tile = reinterpret_cast<float*>(c.scratch + P.gdn_off);
    const float4* m = reinterpret_cast<const float4*>(L.ssm_st + (size_t)h * SD * SD);
#pragma unroll 1
    for (int f = c.tid; f < SD * PPR; f += ST_CT) { const int j = f / PPR, cc = f % PPR; cp_async16(tile + j * SD + ((cc ^ (j & 7)) << 2), m + f); }
    asm volatile("cp.async.commit_group;" ::: "memory");
}
// sum of a[i] * b[i] in index order (one lane); both 16-byte aligned, n a multiple of 16, with ANY of 8 (up to eight elements behind them are read)
template <bool ANY> __device__ __noinline__ float chain_dot(const float* a, const float* b, int n) {
    float s = 0.f;
    float4 x[4], y[4];
#pragma unroll
    for (int u = 0; u < 4; u++) { x[u] = *reinterpret_cast<const float4*>(a + 4 * u); y[u] = *reinterpret_cast<const float4*>(b + 4 * u); }
#pragma unroll 1
    for (int i = 16; i <= n; i += 16) {
        float p[16];                                             // this run's products; the next run on its way while they are added
#pragma unroll
        for (int u = 0; u < 4; u++) { p[4 * u] = it_mul(x[u].x, y[u].x); p[4 * u + 1] = it_mul(x[u].y, y[u].y); p[4 * u + 2] = it_mul(x[u].z, y[u].z); p[4 * u + 3] = it_mul(x[u].w, y[u].w); }
        const int at = i < n ? i : 0;
#pragma unroll
        for (int u = 0; u < 4; u++) { x[u] = *reinterpret_cast<const float4*>(a + at + 4 * u); y[u] = *reinterpret_cast<const float4*>(b + at + 4 * u); }
#pragma unroll
        for (int u = 0; u < 16; u++) s = it_add(s, p[u]);
    }
    if (ANY)
#pragma unroll 1
        for (int i = n & ~15; i < n; i++) s = it_add(s, it_mul(a[i], b[i]));
    return s;
}
__device__ __forceinline__ void gdn_phase(const StepParams& P, const StepLayer& L, const Cta& c, int h, int il) {
    constexpr int SD = ST_SD, PPR = SD / 4;
    const int tid = c.tid, warp = c.warp, lane = c.lane, kh = h % P.nk;
    float* tile = reinterpret_cast<float*>(c.scratch + P.gdn_off);   // [SD][SD], 16-byte pieces of row j stored at piece index ^ (j & 7); requested by gdn_prefetch
    float* qs = reinterpret_cast<float*>(c.scratch);                 // [SD] q, [SD] k
    float* ks = qs + SD;
    float* dl = ks + SD;                                             // [SD] deltas
    float* os = dl + SD;                                             // [SD] delta-rule outputs
    float* scs = os + SD;                                            // [2] l2norm scales, [2] beta, decay
    float* raw = scs + 4;                                            // [4][SD] the head's q, k, v and gate rows
    auto piece = [&](int j, int cc) { return reinterpret_cast<float4*>(tile + j * SD + ((cc ^ (j & 7)) << 2)); };
    float* m = L.ssm_st + (size_t)h * SD * SD;
    const unsigned tag = tag_of(c.base, il, PH_B);
    constexpr int GH = SD / 32 * ST_GPU;                             // granules of a run of SD rows
    static_assert(4 * GH <= ST_CT, "one granule a thread");
    if (tid < 4 * GH) {
        const int r = tid / GH, first = r == 0 ? kh * SD : r == 1 ? P.qk + kh * SD : r == 2 ? 2 * P.qk + h * SD : P.cd + h * SD;
        const granule* gp = P.rows + (size_t)(first / 32) * ST_GPU + (tid - r * GH);
        const granule g = wait_granule(P, gp, tag, c.abort_flag, 17);
        bool two; float* at = raw + r * SD + granule_row(tid - r * GH, two);
        at[0] = __uint_as_float(g.x); at[ST_GPU] = __uint_as_float(g.y); if (!two) at[2 * ST_GPU] = __uint_as_float(g.z);
    } else if (tid >= ST_CT - 2) scs[2 + tid - (ST_CT - 2)] = ld_tagged(P, P.gate + (tid - (ST_CT - 2)) * P.nv + h, tag, c.abort_flag, 18);
    float nw[SD / 32];
    if (warp == 0) {
#pragma unroll
        for (int i = 0; i < SD / 32; i++) nw[i] = L.ssm_norm[lane + 32 * i];
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    cons_sync();
    const bool lost = *c.abort_flag;                                 // the rows or gates may not have come: the state stays, nothing is published
    const float q = raw[tid & (SD - 1)], k = raw[SD + (tid & (SD - 1))], v = raw[2 * SD + (tid & (SD - 1))], bt = scs[2], eg = scs[3];
    if (warp >= 4 && warp < 6 && lane == 0) { const float* r = raw + (warp - 4) * SD; scs[warp - 4] = __fdiv_rn(1.0f, fmaxf(__fsqrt_rn(chain_dot<false>(r, r, SD)), P.eps)); }
    if (warp < 6) asm volatile("bar.sync 3, 192;" ::: "memory");
    if (tid < SD) {
        qs[tid] = it_mul(q, scs[0]); ks[tid] = it_mul(k, scs[1]);
        asm volatile("bar.sync 2, 128;" ::: "memory");
        const float scale = c.inv_sqrt_sd;
        // Two passes over the thread's state row.  The first: s = sum_i (row[i] * eg) * k[i] in index order.  The second forms the new
        // row, row[i] * eg (the same rounded product) + k[i] * delta, and adds the output in index order.  Four 16-byte pieces at a
        // time; while their products are added (the chain), the next four and their factors are on their way.  The rows' stores
        // are the other warps' work (below), after the output: beside the second pass and the norm they cost 2000 cycles.
        float s = 0.f;
        {
            float4 r[4], kk[4];
#pragma unroll
            for (int u = 0; u < 4; u++) { r[u] = *piece(tid, u); kk[u] = *reinterpret_cast<const float4*>(ks + 4 * u); }
#pragma unroll 1
            for (int c0 = 4; c0 <= PPR; c0 += 4) {
                float p[16];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    p[4 * u] = it_mul(it_mul(r[u].x, eg), kk[u].x); p[4 * u + 1] = it_mul(it_mul(r[u].y, eg), kk[u].y);
                    p[4 * u + 2] = it_mul(it_mul(r[u].z, eg), kk[u].z); p[4 * u + 3] = it_mul(it_mul(r[u].w, eg), kk[u].w);
                }
                const int at = c0 & (PPR - 1);
#pragma unroll
                for (int u = 0; u < 4; u++) { r[u] = *piece(tid, at + u); kk[u] = *reinterpret_cast<const float4*>(ks + 4 * (at + u)); }
#pragma unroll
                for (int u = 0; u < 16; u++) s = it_add(s, p[u]);
            }
        }
        const float delta = it_mul(it_sub(v, s), bt);
        dl[tid] = delta;
        float acc = 0.f;
        {
            float4 r[4], kk[4], qq[4];
#pragma unroll
            for (int u = 0; u < 4; u++) { r[u] = *piece(tid, u); kk[u] = *reinterpret_cast<const float4*>(ks + 4 * u); qq[u] = *reinterpret_cast<const float4*>(qs + 4 * u); }
#pragma unroll 1
            for (int c0 = 4; c0 <= PPR; c0 += 4) {
                float p[16];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    p[4 * u] = it_mul(it_add(it_mul(r[u].x, eg), it_mul(kk[u].x, delta)), qq[u].x); p[4 * u + 1] = it_mul(it_add(it_mul(r[u].y, eg), it_mul(kk[u].y, delta)), qq[u].y);
                    p[4 * u + 2] = it_mul(it_add(it_mul(r[u].z, eg), it_mul(kk[u].z, delta)), qq[u].z); p[4 * u + 3] = it_mul(it_add(it_mul(r[u].w, eg), it_mul(kk[u].w, delta)), qq[u].w);
                }
                const int at = c0 & (PPR - 1);
#pragma unroll
                for (int u = 0; u < 4; u++) { r[u] = *piece(tid, at + u); kk[u] = *reinterpret_cast<const float4*>(ks + 4 * (at + u)); qq[u] = *reinterpret_cast<const float4*>(qs + 4 * (at + u)); }
#pragma unroll
                for (int u = 0; u < 16; u++) acc = it_add(acc, p[u]);
            }
        }
        os[tid] = it_mul(acc, scale);
        asm volatile("bar.sync 2, 128;" ::: "memory");
        if (warp > 0) asm volatile("bar.arrive 6, 384;" ::: "memory");
    } else {
        // the new state to global memory, a 16-byte piece a thread at a time (coalesced), once the head's output is out
        asm volatile("bar.sync 6, 384;" ::: "memory");
#pragma unroll 2
        for (int f = lost ? SD * PPR : tid - SD; f < SD * PPR; f += ST_CT - SD) {
            const int j = f / PPR, cc = f % PPR;
            const float4 o = *piece(j, cc), k4 = *reinterpret_cast<const float4*>(ks + 4 * cc);
            const float delta = dl[j];
            reinterpret_cast<float4*>(m)[f] = make_float4(it_add(it_mul(o.x, eg), it_mul(k4.x, delta)), it_add(it_mul(o.y, eg), it_mul(k4.y, delta)), it_add(it_mul(o.z, eg), it_mul(k4.z, delta)), it_add(it_mul(o.w, eg), it_mul(k4.w, delta)));
        }
    }
    if (warp == 0) {
        float sc = 0.f;
        if (lane == 0) sc = __fdiv_rn(1.0f, __fsqrt_rn(it_add(__fdiv_rn(chain_dot<false>(os, os, SD), (float)SD), P.eps)));
        sc = __shfl_sync(0xffffffffu, sc, 0);
        // the output projection's columns may be grouped [rep][key head] where value heads are [key head][rep]
        const int u0 = (P.v_grouped ? h / P.nk + P.nv / P.nk * kh : h) * (SD / 32);
        const unsigned otag = tag_of(c.base, il, PH_C);
#pragma unroll
        for (int i = 0; i < SD / 32; i++) { const int j = lane + 32 * i; publish(P.o, u0 + i, lane, it_mul(it_mul(it_mul(os[j], sc), nw[i]), raw[3 * SD + j]), otag, lost); }
        asm volatile("bar.arrive 6, 384;" ::: "memory");             // the other warps may form the new rows
    }
}

// ---------------------------------------------------------------- attention block of one head
// q / k head norms, rope, the new K / V entries and the causal gated attention of head h in the operation order of
// k_attn_prep and k_attention (it_support.cu; src/cpu.rs:252-272): every score a sequential dot over the head dimension,
// the exponentials added in ascending position order by one thread, every output element accumulating w[p] * v[p][j] in
// ascending position order.  The k and v rows of the new position are recomputed by each of the heads that share the KV
// head and used from shared memory (after the same f16 rounding the cache applies); the CTAs of the first head of the
// group store them into the cache.
// Data movement: both caches are tiled (32 positions x head_dim halves = one contiguous 16 KB block per KV head), so a
// loader warp brings whole tiles into a ring of 16 KB slots with one bulk copy each.  One warp per slot scores its K
// tiles, a position per lane, from shared memory; slices of the V tiles follow through the same ring and a warp per 32 output
// elements (one a thread) walks them in order.  Full / free mbarriers pace both; they are set up afresh by every attention
// block.  The tiles were sent on their way into L2 while the input projection ran (attn_prefetch).
__device__ __forceinline__ void attn_prefetch(const StepParams& P, const StepLayer& L, const Cta& c, int hg) {
    if (c.warp != 0 || hg < 0 || hg >= P.nh * P.attn_g) return;
    const int G = P.attn_g, h = hg / G, g = hg % G;
    const int kh = h / (P.nh / P.nkv), ntiles = (*P.pos + 31) / 32; const unsigned bytes = (unsigned)(P.hd * 64);
    for (int i = g + G * c.lane; i < ntiles; i += G * 32)               // the K tiles this CTA will score
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" :: "l"(L.kc + it_kc_index((size_t)i * 32, kh, 0, P.nkv, P.hd)), "r"(bytes) : "memory");
    for (int i = g + G * c.lane; i < ntiles; i += G * 32)               // a quarter of the V tiles each: every CTA of the head reads a slice of all of them
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" :: "l"(L.vc + it_vc_index((size_t)i * 32, kh, 0, P.nkv, P.hd)), "r"(bytes) : "memory");
}
constexpr int ST_AT_MAXS = 8, ST_AT_LOADER = ST_NCONS - 1, ST_AT_T = (ST_NCONS - 1) * 32;
// the block's own barrier: every consumer warp but the loader, which runs ahead and only joins the next phase
__device__ __forceinline__ void at_sync() { asm volatile("bar.sync 4, %0;" :: "n"(ST_AT_T) : "memory"); }
// G = P.attn_g CTAs share a head (hg = G h + g).  Each forms q and the new position's k for itself, and its elements of v, scores the K
// tiles i with i % G == g, publishes those scores, reads the others' as they come (the tag is the exchange: a
// counter would need a base that nobody's late start can miss), runs the softmax for itself (one thread adds the exponentials in position order) and accumulates the
// head_dim / G output elements [g head_dim / G, ...) over all positions from row slices of the V tiles.  A single SM can
// keep only so many bytes in flight, so a head's cache traffic is spread over G SMs.
template <bool ANY> __device__ __forceinline__ void attn_phase(const StepParams& P, const StepLayer& L, Cta& c, int hg, int il) {
    const int tid = c.tid, warp = c.warp, lane = c.lane, hd = P.hd, nkv = P.nkv, kvd = nkv * hd;
    const int G = P.attn_g, h = hg / G, g = hg % G, epc = hd / G;   // elements of the output this CTA owns
    const int vs = it_vc_slice(hd);                                  // elements per V slice: epc is a multiple of it
    const int rep = P.nh / nkv, kh = h / rep;
    const int pos = *P.pos, n = pos + 1, nold = pos;
    const int ntiles = (nold + 31) / 32;                             // K tiles = V tiles of 32 positions
    const int my_tiles = ntiles > g ? (ntiles - g + G - 1) / G : 0;  // tiles g, g + G, ... are scored here
    const int tile_bytes = hd * 64;                                  // 32 positions x hd halves
    const int vslot_bytes = epc * 64;                                // 32 positions x epc halves: this CTA's slice of a V tile
    float* sc = reinterpret_cast<float*>(c.scratch);                 // [n] scores
    float* qs = sc + ((n + 3) & ~3);                                 // [hd] q head after norm + rope
    float* kl = qs + hd;                                             // [hd] k row of the new position as the cache holds it
    float* vl = kl + hd;                                             // [epc] this CTA's elements of the v row of the new position, as the cache holds them
    float* gs = vl + epc;                                            // [epc] and of the head's gate row
    float* red = gs + epc;                                           // [32] + the sum
    unsigned char* ring = reinterpret_cast<unsigned char*>(red + ST_AT_RED) + (-smem_u32(red + ST_AT_RED) & 15u);
    const int room = (int)((c.scratch + P.scratch) - ring);
    // K: tile j of this CTA goes to slot j % S and is scored by warp j % S, so every slot is filled and emptied by the same two
    // warps in order.  V: slice j goes to slot j % SV; the output warps walk the slices in order.
    const int S = max(1, min(ST_AT_MAXS, room / tile_bytes)), SV = max(1, min(ST_AT_MAXS, room / vslot_bytes));
    const int vwarps = (epc + 31) / 32;                              // output warps: one element per thread
    const unsigned kf = c.at, ke = c.at + 8 * ST_AT_MAXS, vf = c.at + 16 * ST_AT_MAXS, ve = c.at + 24 * ST_AT_MAXS;
    if (tid == 0) {
#pragma unroll 1
        for (int k = 0; k < 4 * ST_AT_MAXS; k++) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" :: "r"(c.at + 8 * k) : "memory");
#pragma unroll 1
        for (int k = 0; k < ST_AT_MAXS; k++) { mbar_init(kf + 8 * k, 1); mbar_init(ke + 8 * k, 1); mbar_init(vf + 8 * k, 1); mbar_init(ve + 8 * k, vwarps); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    ST_EV(P, c, c.evt_base + 4);
    {   // the head's q row and the KV head's k row whole, of the gate and v rows this CTA's elements
        const unsigned tag = tag_of(c.base, il, PH_B);
        const int gh = hd / 32 * ST_GPU, ge = epc / 32 * ST_GPU;      // granules of hd and of epc rows; hd <= 256: at most 88 each
        const int r = tid < 2 * gh ? (tid < gh ? 0 : 1) : tid < 2 * gh + ge ? 2 : 3, k = r < 2 ? tid - r * gh : tid - 2 * gh - (r - 2) * ge;
        if ((!ANY || hd % 32 == 0) && tid < 2 * (gh + ge)) {
            const int first = r == 0 ? 2 * h * hd : r == 1 ? 2 * P.nh * hd + kh * hd : r == 2 ? (2 * h + 1) * hd + g * epc : 2 * P.nh * hd + kvd + kh * hd + g * epc;
            const granule v = wait_granule(P, P.rows + (size_t)(first / 32) * ST_GPU + k, tag, c.abort_flag, 17);
            bool two; float* at = (r == 0 ? qs : r == 1 ? kl : r == 2 ? gs : vl) + granule_row(k, two);
            at[0] = __uint_as_float(v.x); at[ST_GPU] = __uint_as_float(v.y); if (!two) at[2 * ST_GPU] = __uint_as_float(v.z);
        }
        // a head dimension that is no multiple of 32 (then G is 1): heads begin inside row groups, every row is looked up by itself
        if (ANY && hd % 32) for (int i = tid; i < 4 * hd; i += ST_CT) {
            const int r = i / hd, k = i - r * hd, row = (r == 0 ? 2 * h * hd : r == 1 ? 2 * P.nh * hd + kh * hd : r == 2 ? (2 * h + 1) * hd : 2 * P.nh * hd + kvd + kh * hd) + k, l = row & 31;
            const granule v = wait_granule(P, P.rows + (size_t)(row / 32) * ST_GPU + l % ST_GPU, tag, c.abort_flag, 17);
            (r == 0 ? qs : r == 1 ? kl : r == 2 ? gs : vl)[k] = __uint_as_float(l < ST_GPU ? v.x : l < 2 * ST_GPU ? v.y : v.z);
        }
    }
    cons_sync();                                                     // all twelve warps, the loader included
    const bool lost = *c.abort_flag, writer = h % rep == 0 && !lost;      // the group's first head stores the new position: k by its first CTA, v by all, their elements
    ST_EV(P, c, c.evt_base + 5);
    const __half* kc = L.kc; const __half* vc = L.vc;

    if (warp == ST_AT_LOADER) {
        // ---- loader: this CTA's K tiles, then its slice of every V tile, as far ahead as the rings allow
        unsigned kn = 0, vn = 0; bool ok = true;
#pragma unroll 1
        for (int j = 0; j < my_tiles; j++, kn++) {
            const unsigned sl = (unsigned)j % (unsigned)S, u = (unsigned)j / (unsigned)S;
            if (!(ok = mbar_wait(ke + 8 * sl, (u & 1u) ^ 1u, c.abort_flag, P.error_flag, 8))) break;
            if (lane == 0) {
                mbar_expect_tx(kf + 8 * sl, (unsigned)tile_bytes);
                bulk_load(smem_u32(ring + sl * tile_bytes), kc + it_kc_index((size_t)(g + G * j) * 32, kh, 0, nkv, hd), (unsigned)tile_bytes, kf + 8 * sl);
            }
        }
        // the V slices go through the same bytes: not before the last K tile of every slot has been scored
        for (int j = my_tiles > S ? my_tiles - S : 0; j < my_tiles; j++) ok = ok && mbar_wait(ke + 8 * (j % S), (unsigned)(j / S) & 1u, c.abort_flag, P.error_flag, 8);
#pragma unroll 1
        for (int i = 0; i < ntiles && ok; i++, vn++) {
            const unsigned sl = (unsigned)i % (unsigned)SV, u = (unsigned)i / (unsigned)SV;
            if (!mbar_wait(ve + 8 * sl, (u & 1u) ^ 1u, c.abort_flag, P.error_flag, 9)) break;
            if (lane == 0) {
                // the slices of the tile that hold elements g epc .. (g + 1) epc - 1 are consecutive: one copy
                mbar_expect_tx(vf + 8 * sl, (unsigned)vslot_bytes);
                bulk_load(smem_u32(ring + sl * vslot_bytes), vc + it_vc_index((size_t)i * 32, kh, g * epc, nkv, hd), (unsigned)vslot_bytes, vf + 8 * sl);
            }
        }
        if (lane == 0) { drain_copies(kf, (unsigned)S, kn); drain_copies(vf, (unsigned)SV, vn); }
        __syncwarp();
        return;                                                      // the loader meets the others at the next phase
    }
    if (warp < 2) {
        // warp 0: q head; warp 1: k head.  rmsnorm with the squares added by one lane in index order, weight, rope.
        float* buf = warp == 0 ? qs : kl;
        const float* w = warp == 0 ? L.q_norm : L.k_norm;
        float wr[8];                                                  // hd <= 256: the norm weights are requested before the sum needs time
#pragma unroll
        for (int k = 0; k < 8; k++) wr[k] = lane + 32 * k < hd ? w[lane + 32 * k] : 0.f;
        float s = 0.f;
        if (lane == 0) s = chain_dot<ANY>(buf, buf, hd);
        s = __shfl_sync(0xffffffffu, s, 0);
        const float scl = it_div(1.0f, it_sqrt(it_add(it_div(s, (float)hd), P.eps)));
#pragma unroll
        for (int k = 0; k < 8; k++) if (lane + 32 * k < hd) buf[lane + 32 * k] = it_mul(it_mul(buf[lane + 32 * k], scl), wr[k]);
        __syncwarp();
        const int half = P.n_rot / 2, sect = P.sec[0] + P.sec[1] + P.sec[2] + P.sec[3];
#pragma unroll 1
        for (int i = lane; i < half; i += 32) {
            float theta = (float)pos;
            for (int k = 0; k < i; k++) theta = it_mul(theta, P.theta_scale);
            const int sector = sect > 0 ? i % sect : 0;
            const bool use_e = sect > 0 && !((sector % 3 == 1 && sector < 3 * P.sec[1]) || (sector % 3 == 2 && sector < 3 * P.sec[2]) || (sector % 3 == 0 && sector < 3 * P.sec[0]));
            float sn, cs; it_sincosf(use_e ? 0.0f : theta, &sn, &cs);
            const float x0 = buf[i], x1 = buf[i + half];
            buf[i] = it_sub(it_mul(x0, cs), it_mul(x1, sn));
            buf[i + half] = it_add(it_mul(x0, sn), it_mul(x1, cs));
        }
        __syncwarp();
        if (warp == 1) for (int i = lane; i < hd; i += 32) {
            const __half hv = __float2half_rn(buf[i]);
            if (writer && g == 0) const_cast<__half*>(kc)[it_kc_index(pos, kh, i, nkv, hd)] = hv;
            buf[i] = __half2float(hv);
        }
    } else if (warp == 2) {
        for (int i = lane; i < epc; i += 32) {
            const __half hv = __float2half_rn(vl[i]);
            if (writer) const_cast<__half*>(vc)[it_vc_index(pos, kh, g * epc + i, nkv, hd)] = hv;
            vl[i] = __half2float(hv);
        }
    }
    at_sync();                                                       // q, and the new position's k and v, are in shared memory
    ST_EV(P, c, c.evt_base + 6);
    const float scale = c.inv_sqrt_hd;
    const int nvec = hd / 8;
    unsigned long long* shared_sc = P.att_sc + (size_t)h * P.att_stride;      // the head's scores, where its CTAs leave theirs for one another
    const unsigned sc_tag = tag_of(c.base, il, PH_C);
    if (warp < S) {
        // ---- scores: this CTA's tile j by warp j % S, position 32 (g + G j) + lane; piece v of the tile's 32 positions is contiguous
        for (int j = warp; j < my_tiles; j += S) {
            const unsigned sl = (unsigned)j % (unsigned)S, u = (unsigned)j / (unsigned)S;
            if (!mbar_wait(kf + 8 * sl, u & 1u, c.abort_flag, P.error_flag, 10)) break;
            const int p = (g + G * j) * 32 + lane;
            if (p < nold) {
                const uint4* kp = reinterpret_cast<const uint4*>(ring + sl * tile_bytes) + lane;
                float s = 0.f;
#pragma unroll 4
                for (int v = 0; v < nvec; v++) {
                    const uint4 kk = kp[v * 32];
                    const __half2* hh = reinterpret_cast<const __half2*>(&kk);
                    const float4 qa = *reinterpret_cast<const float4*>(qs + v * 8), qb = *reinterpret_cast<const float4*>(qs + v * 8 + 4);
                    float2 f = __half22float2(hh[0]); s = it_add(s, it_mul(qa.x, f.x)); s = it_add(s, it_mul(qa.y, f.y));
                    f = __half22float2(hh[1]); s = it_add(s, it_mul(qa.z, f.x)); s = it_add(s, it_mul(qa.w, f.y));
                    f = __half22float2(hh[2]); s = it_add(s, it_mul(qb.x, f.x)); s = it_add(s, it_mul(qb.y, f.y));
                    f = __half22float2(hh[3]); s = it_add(s, it_mul(qb.z, f.x)); s = it_add(s, it_mul(qb.w, f.y));
                }
                s = it_mul(s, scale); sc[p] = s;
                if (G > 1 && !lost) st_tagged(shared_sc + p, s, sc_tag);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(ke + 8 * sl);
        }
    } else if (warp == ST_AT_MAXS && lane == 0) {
        sc[nold] = it_mul(chain_dot<ANY>(qs, kl, hd), scale);             // the new position, from its row in shared memory (every CTA of the head for itself)
    }
    ST_EV(P, c, c.evt_base + 7);
    if (G > 1) {
        // ---- the other CTAs' scores, as they come: their tags say that they are this layer's
#pragma unroll 1
        for (int i = 0; i < ntiles; i++) {
            if (i % G == g) continue;
            const int p = i * 32 + lane;
            if (warp == i % (ST_NCONS - 1) && p < nold) sc[p] = ld_tagged(P, shared_sc + p, sc_tag, c.abort_flag, 19);
        }
    }
    at_sync();
    ST_EV(P, c, c.evt_base + 8);
    float mx = -INFINITY;
#pragma unroll 1
    for (int p = tid; p < n; p += ST_AT_T) mx = fmaxf(mx, sc[p]);
#pragma unroll
    for (int mm = 16; mm >= 1; mm >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, mm));
    if (lane == 0) red[warp] = mx;
    at_sync();
    mx = red[0];
#pragma unroll
    for (int k = 1; k < ST_NCONS - 1; k++) mx = fmaxf(mx, red[k]);
#pragma unroll 1
    for (int p = tid; p < n; p += ST_AT_T) sc[p] = it_expf(it_sub(sc[p], mx));
    at_sync();
    if (tid == 0) {
        float s = 0.f;
#pragma unroll 8
        for (int p = 0; p < n; p++) s = it_add(s, sc[p]);
        red[32] = s;
    }
    at_sync();
    const float sum = red[32];
#pragma unroll 1
    for (int p = tid; p < n; p += ST_AT_T) sc[p] = it_div(sc[p], sum);
    at_sync();
    ST_EV(P, c, c.evt_base + 9);
    if (warp < vwarps) {
        // ---- output: element j adds w[p] * v[p][j] in ascending p; thread tid owns element g epc + tid of the head.  A whole
        // tile's 32 values are read before the first addition, so that the chain of additions never waits for shared memory.
        const bool live = tid < epc;
        float acc = 0.f;
        const int eoff = (tid / vs) * 32 * vs + tid % vs;             // [slice][32][vs]
        for (int i = 0; i < ntiles; i++) {
            const unsigned sl = (unsigned)i % (unsigned)SV, u = (unsigned)i / (unsigned)SV;
            if (!mbar_wait(vf + 8 * sl, u & 1u, c.abort_flag, P.error_flag, 11)) break;
            const int rows = min(32, nold - i * 32);
            if (live) {
                const __half* src = reinterpret_cast<const __half*>(ring + sl * vslot_bytes) + eoff;
                const float* wp = sc + i * 32;
                if (rows == 32) {
                    float vv[32];
#pragma unroll
                    for (int r = 0; r < 32; r++) vv[r] = __half2float(src[r * vs]);
#pragma unroll
                    for (int r4 = 0; r4 < 8; r4++) {
                        const float4 w4 = *reinterpret_cast<const float4*>(wp + 4 * r4);
                        acc = it_add(acc, it_mul(w4.x, vv[4 * r4])); acc = it_add(acc, it_mul(w4.y, vv[4 * r4 + 1]));
                        acc = it_add(acc, it_mul(w4.z, vv[4 * r4 + 2])); acc = it_add(acc, it_mul(w4.w, vv[4 * r4 + 3]));
                    }
                } else {
                    for (int r = 0; r < rows; r++) acc = it_add(acc, it_mul(wp[r], __half2float(src[r * vs])));
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(ve + 8 * sl);
        }
        if (live) {
            acc = it_add(acc, it_mul(sc[nold], vl[tid]));
            acc = it_mul(acc, it_sigmoid(gs[tid]));
        }
        const bool gone = *c.abort_flag;                             // a wait since the rows came may have run out
        if (!ANY || hd % 32 == 0) publish(P.o, (h * hd + g * epc) / 32 + warp, lane, acc, sc_tag, gone);      // epc is a multiple of 32
        else if (live && !gone) st_tagged(P.o1 + h * hd + tid, acc, sc_tag);
    }
    ST_EV(P, c, c.evt_base + 10);
}

// Dense row `drow` (beta rows, then alpha rows) of a delta-net layer, or null.
__device__ __forceinline__ const float* dense_row(const StepParams& P, const StepLayer& L, int drow) {
    return L.recurrent && drow < 2 * P.nv ? (drow < P.nv ? L.beta : L.alpha - (size_t)P.nv * P.e) + (size_t)drow * P.e : nullptr;
}

// ---------------------------------------------------------------- the step
// ANY: head dimensions that are no multiple of 32, and more dense rows than CTAs, as well.  Their few branches cost the usual step 0.6 % (155.0 instead of 154.0 ms for 48 steps of
// 64 layers behind a 9-token prompt), so that they have a copy of the kernel.
template <bool ANY> __global__ void __launch_bounds__(ST_THREADS, 1) k_decode_step(const __grid_constant__ StepParams P) {
    extern __shared__ __align__(128) unsigned char smem[];
    Cta c;
    c.smem = smem; c.scratch = smem + P.slots * ST_CHUNK;
    unsigned char* tail = c.scratch + P.scratch;
    c.bars = smem_u32(tail);                                         // full[s] at bars + 8 s, empty[s] at bars + 8 (slots + s), terms full[s] at tf + 8 s
    c.tf = c.bars + 16 * P.slots; c.ps = c.tf + 8 * P.slots; c.pd = c.ps + 8; c.dn = c.pd + 8; c.at = c.dn + 8;
    c.lay = reinterpret_cast<const StepLayer*>(tail + 704);         // two layer descriptions
    c.abort_flag = reinterpret_cast<volatile int*>(tail + ST_BARS - 16); c.verdict = c.abort_flag + 1; c.issued = smem_u32(tail + ST_BARS - 8);
    c.sp = reinterpret_cast<const StepSpan*>(tail + ST_BARS);
    c.tid = threadIdx.x; c.warp = c.tid >> 5; c.lane = c.tid & 31;
    c.q = 0u; c.nsync = 0; c.evt_on = 0; c.dense_seq = 0u; c.mph = 0u;
    if (c.tid == 0) {
        st_issued(c.issued, 0u);
        *c.abort_flag = *reinterpret_cast<volatile unsigned*>(P.sync + 2) ? 1 : 0;      // a step that was given up earlier: nothing runs until the host has cleared the words
        for (int s = 0; s < P.slots; s++) { mbar_init(c.bars + 8 * s, 1); mbar_init(c.bars + 8 * (P.slots + s), 1); mbar_init(c.tf + 8 * s, ST_CW); }
        mbar_init(c.ps, 1); mbar_init(c.pd, ST_NSUM); mbar_init(c.dn, 8);
        for (int k = 0; k < 4 * ST_AT_MAXS; k++) mbar_init(c.at + 8 * k, 1);     // set up again, with their counts, by every attention block
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    {   // the first layer's description and this CTA's spans into shared memory (later layers are copied a layer ahead)
        constexpr int words = (int)(sizeof(StepLayer) / 4), sw = (int)(SP_KINDS * sizeof(StepSpan) / 4);
        if (c.tid < words) reinterpret_cast<uint32_t*>(tail + 704)[c.tid] = reinterpret_cast<const uint32_t*>(P.layers)[c.tid];
        if (c.tid < sw) reinterpret_cast<uint32_t*>(tail + ST_BARS)[c.tid] = reinterpret_cast<const uint32_t*>(P.spans + (size_t)blockIdx.x * SP_KINDS)[c.tid];
    }
    __syncthreads();
    if (*c.abort_flag) return;
    if (c.warp == ST_NCONS + ST_NSUM) { if (c.lane == 0) producer(P, c); return; }
    if (c.warp >= ST_NCONS) { sum_warps<ANY>(P, c); return; }

    c.base = *reinterpret_cast<volatile unsigned*>(P.sync + 3); c.target = *reinterpret_cast<volatile unsigned*>(P.sync + 1);
    c.inv_sqrt_sd = it_div(1.0f, it_sqrt((float)ST_SD)); c.inv_sqrt_hd = it_div(1.0f, it_sqrt((float)P.hd));
    float* A = P.arena;
    const int cta = (int)blockIdx.x, grid = (int)gridDim.x, drow = grid - 1 - cta, ah = cta - P.attn_base;
    const int hb = cta % P.had_step == 0 && cta / P.had_step < P.widest / 1024 ? cta / P.had_step : -1;      // the block this CTA transforms, of every row that has as many
    const uint32_t tok = (P.flags & 1) ? __float_as_uint(*reinterpret_cast<volatile float*>(A + P.amx)) : *reinterpret_cast<volatile uint32_t*>(P.toks);
    float* wb = reinterpret_cast<float*>(c.scratch + P.w_off);
    // the norms' weights are wanted where a block of a normed row is transformed and where a dense row is multiplied
    auto want_norm = [&](const float* w, const float* dense) { if (dense || (hb >= 0 && hb * 1024 < P.e)) norm_request(wb, w, dense, P.e); };
    want_norm(c.lay->attn_norm, dense_row(P, *c.lay, drow));
    // Nine phases a layer, then the output norm with the LM head.  One loop, one copy of each kind of phase: transforms (A D F H: the
    // owners of the row's blocks, in A also the owners of dense rows), matrices (B E G I: everyone), the block in between (C).
    const bool logits = (P.flags & 4) != 0;
    int il = 0, ph = PH_A;
#pragma unroll 1
    for (;;) {
        const bool tail_ph = il >= P.n_layer;
        const StepLayer& L = c.lay[il & 1];
        c.evt_on = (il == 1 || il == 3) && c.warp == 0 && (ph == PH_C ? (cta == (il == 1 ? 0 : P.attn_base)) : (ph & 1) == 0 && ph < PH_C || ph == PH_D || ph == PH_F || ph == PH_H ? cta == 0 : (cta == grid - 1)); c.evt_base = (il == 1 ? 0 : 256) + 16 * ph;
        const int row_blocks = (ph < PH_C || ph == PH_F || ph == PH_G ? P.e : ph < PH_F ? (L.recurrent ? P.inner : P.nh * P.hd) : P.ff) / 1024;      // of the row that the phase transforms or reads
        if (ph == PH_C) {
            const int heads = L.recurrent ? P.nv : P.nh * P.attn_g;
            if (L.recurrent) { if (cta < P.nv) { cons_sync(); gdn_phase(P, L, c, cta, il); } }
            else if (ah >= 0 && ah < heads) { cons_sync(); attn_phase<ANY>(P, L, c, ah, il); }
        } else if (ph == PH_A || ph == PH_D || ph == PH_F || ph == PH_H) {
            RowIn in; in.normed = nullptr; in.plain = nullptr; in.one = nullptr; in.norm = ph == PH_A || ph == PH_F; in.dense = ph == PH_A && !tail_ph && L.recurrent && drow < 2 * P.nv;
            const bool owner = hb >= 0 && hb < row_blocks && (!tail_ph || logits || cta == 0);
            if (owner || in.dense) {
                in.codes = owner && (!tail_ph || logits) ? P.codes + step_codes_half(ph) * P.codes_half + hb * 128 : nullptr; in.codes_copy = row_blocks * 128; in.code_tag = tag_of(c.base, il, ph);
                in.nblk = row_blocks; in.blk = hb; in.dense2 = ANY && in.dense ? dense_row(P, L, drow + grid) : nullptr;
                in.signs = P.sg[ph == PH_D ? (L.recurrent ? 1 : 2) : ph == PH_H ? 3 : 0] + (hb >= 0 ? 32 * hb : 0);
                if (ph == PH_A) {
                    in.x = P.xi; in.tag = tag_of(c.base, il - 1, PH_I);
                    if (il == 0) in.plain = P.tok_embd + (size_t)tok * P.e;      // the residual row of layer 0 is the embedding row (Model::embed, src/cpu.rs:118-122)
                    if (tail_ph && cta == 0) in.normed = A + P.hrow;
                } else if (ph == PH_F) { in.x = P.xe; in.tag = tag_of(c.base, il, PH_E); }
                else {
                    in.x = (ph == PH_D ? P.o : P.act) + (size_t)hb * ST_GPB; in.tag = tag_of(c.base, il, ph == PH_D ? PH_C : PH_G); in.nblk = 1; in.blk = 0;
                    if (ANY && ph == PH_D && !L.recurrent && P.o1) in.one = P.o1 + (size_t)hb * 1024;
                }
                if (!owner && !count_wait(P, c, P.sync, c.target + (unsigned)row_blocks, 1 + ph, false)) goto leave;      // a dense row's owner follows the blocks' owners
                ST_EV(P, c, c.evt_base + 0);
                block_transform<ANY>(P, c, in);
                ST_EV(P, c, c.evt_base + 1);
            }
            if (tail_ph && !logits) { if (cta != 0) goto leave; break; }
            c.target += (unsigned)row_blocks;
        } else {
            const int sub = ph == PH_B ? 0 : ph == PH_E ? 1 : ph == PH_G ? 2 : 3;
            const int kind = tail_ph ? SP_HEAD : span_kind(sub, L.recurrent);
            if (!count_wait(P, c, P.sync, c.target, 1 + ph)) goto leave;
            ST_EV(P, c, c.evt_base + 0);
            if (c.tid == 0) mbar_arrive(c.ps);                       // the sum warps may enter this phase
            // (a CTA without row groups does not read the codes: nobody waits for it, so nothing would keep them)
            if (c.sp[kind].n) codes_place(P, c, P.codes + step_codes_half(ph) * P.codes_half, row_blocks, tag_of(c.base, il, ph - 1));
            ST_EV(P, c, c.evt_base + 1);
            if (ph == PH_B && !tail_ph) {
                if (il + 1 < P.n_layer && c.warp == ST_NCONS - 1) {          // the next layer's description, long before it is needed
                    constexpr int words = (int)(sizeof(StepLayer) / 4);
                    uint32_t* dst = reinterpret_cast<uint32_t*>(const_cast<StepLayer*>(c.lay + ((il + 1) & 1)));
#pragma unroll 1
                    for (int i = c.lane; i < words; i += 32) dst[i] = reinterpret_cast<const uint32_t*>(P.layers + il + 1)[i];
                }
                if (L.recurrent) { if (cta < P.nv) gdn_prefetch(P, L, c, cta); }
                else attn_prefetch(P, L, c, ah);
            }
            if (ph == PH_G) { if (il + 1 < P.n_layer) warm_layer(P, c, c.lay[(il + 1) & 1], drow); else if (cta == grid - 1) warm_l2(P.output_norm, P.e * 4, c.tid); }
            matvec_phase(P, c, c.sp[kind]);
            ST_EV(P, c, c.evt_base + 2);
            // the next norm's weights (and dense row) while the other CTAs finish
            if (ph == PH_E) want_norm(L.post_norm, nullptr);
            if (ph == PH_I) {
                const bool more = il + 1 < P.n_layer; const StepLayer& N = c.lay[(il + 1) & 1];
                want_norm(more ? N.attn_norm : P.output_norm, more ? dense_row(P, N, drow) : nullptr);
            }
            if (tail_ph) { if (cta != 0) goto leave; break; }
            // the scratch is the next phase's once this CTA's sum warps are through (they are before anything the next phase needs has arrived)
            mbar_wait(c.pd, c.mph & 1u, c.abort_flag, P.error_flag, 5);
            c.mph++;
        }
        if (++ph == ST_SUBS) { ph = PH_A; il++; }
    }
    // every sum warp counts when it is through: nobody is left who could still read the words written below
    c.target += ST_NSUM * (unsigned)grid;
    if (!count_wait(P, c, P.sync, c.target, 10, false)) goto leave;
    if (logits && c.warp == 0) {
        Pick q{ -INFINITY, 0xffffffffu };
        bool ok = true;
#pragma unroll 1
        for (unsigned b = c.lane; b < gridDim.x * ST_NSUM; b += 32) {
            const unsigned tag = tag_of(c.base, P.n_layer, PH_B);
            const granule u = wait_granule(P, P.partials + b, tag, c.abort_flag, 20);
            ok = ok && u.w == tag;
            q = pick_better(q, Pick{ __uint_as_float(u.x), u.y });
        }
#pragma unroll
        for (unsigned mm = 16; mm > 0; mm >>= 1) { Pick o{ __shfl_xor_sync(0xffffffffu, q.v, mm), __shfl_xor_sync(0xffffffffu, q.i, mm) }; q = pick_better(q, o); }
        if (!__all_sync(0xffffffffu, ok)) goto leave;
        if (c.lane == 0) {
            const unsigned pick = q.i == 0xffffffffu ? 0u : q.i;
            A[P.amx] = __uint_as_float(pick);
            if (P.flags & 2) { P.toks[0] = pick; *P.pos += 1; }
        }
    }
    if (c.tid == 0) { P.sync[1] = c.target; P.sync[3] = c.base + (unsigned)(ST_SUBS * (P.n_layer + 1) + 1); }
leave:
    asm volatile("cp.async.wait_all;" ::: "memory");                 // a norm's weights, a state tile that nobody waited for
}

}  // namespace

// ---------------------------------------------------------------- host side
struct it_step_state {
    StepLayer* layers_dev;
    StepSpan* spans_dev;
    unsigned long long* trace;
    granule *xe, *xi, *rows, *o, *act, *codes, *prefix, *partials;
    unsigned long long *gate, *o1;
    int had_step;
    int grid, slots, scratch, gdn_off, attn_base, attn_g, att_stride;
    unsigned long long* att_sc;
    bool cooperative, any;
};

// Whether this engine's decode step can run as the persistent kernel, and with which geometry.
int it_step_prepare(it_engine* e) {
    const it_model_config& c = e->cfg; it_ctx* cx = e->ctx;
    e->step = nullptr;
    { const char* v = getenv("IT_STEP_KERNEL"); if (v && atoi(v) == 0) return IT_OK; }
    if (e->world != 1) return IT_OK;                                  // row shards exchange results inside the per-op kernels
    if (c.ssm_state != ST_SD || c.conv_k > 8 || c.head_dim > 256 || c.head_dim % 8 || c.n_embd > 8192 || c.n_embd % 1024 || c.n_ff % 1024 || c.ssm_inner % 1024 || (c.n_head * c.head_dim) % 1024) return IT_OK;
    if (c.ssm_vheads > cx->sm_count || c.n_head > cx->sm_count || step_widest(c) / 1024 > cx->sm_count || c.n_embd % 32 || c.ssm_vheads % c.ssm_groups) return IT_OK;
    // several CTAs per attention head when the grid has them: each takes a share of the K tiles and of the output elements
    int attn_g = step_attn_split(c, cx->sm_count);
    { const char* v = getenv("IT_STEP_ATTN_G"); if (v && (atoi(v) == 1 || atoi(v) == 2) && atoi(v) < attn_g) attn_g = atoi(v); }
    const int slots = step_ring_slots(c, attn_g);
    if (!slots) return IT_OK;
    IT_CUDA(cudaSetDevice(cx->device));
    static bool attr_set[16] = {};
    if (!attr_set[cx->device & 15]) {
        IT_CUDA(cudaFuncSetAttribute(k_decode_step<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, ST_SMEM));
        IT_CUDA(cudaFuncSetAttribute(k_decode_step<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, ST_SMEM));
        attr_set[cx->device & 15] = true;
    }
    const bool any = c.head_dim % 32 != 0 || 2 * c.ssm_vheads > cx->sm_count;
    int per_sm = 0;
    IT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, any ? k_decode_step<true> : k_decode_step<false>, ST_THREADS, step_smem_bytes(c, slots, attn_g)));
    if (per_sm < 1) return IT_OK;
    it_step_state* st = new it_step_state();
    st->any = any; st->grid = cx->sm_count; st->slots = slots; st->scratch = (int)step_scratch_bytes(c, slots, attn_g); st->gdn_off = (int)step_gdn_off(c, slots);
    st->attn_g = attn_g;                                              // attention heads sit behind the value heads when they all fit side by side
    st->attn_base = (c.ssm_vheads + st->attn_g * c.n_head <= st->grid) ? c.ssm_vheads : 0;
    st->layers_dev = nullptr; st->spans_dev = nullptr; st->partials = nullptr; st->gate = nullptr; st->o1 = nullptr; st->trace = nullptr; st->had_step = st->grid / (step_widest(c) / 1024); st->att_sc = nullptr;
    st->att_stride = (c.ctx_len + 32 + 3) / 4 * 4;
    { const char* v = getenv("IT_STEP_COOP"); st->cooperative = !v || atoi(v) != 0; }
    std::vector<StepLayer> hl(c.n_layer);
    for (int il = 0; il < c.n_layer; il++) {
        const it_layer& l = e->layers[il]; StepLayer& s = hl[il]; memset(&s, 0, sizeof s);
        s.recurrent = l.recurrent ? 1 : 0; s.in_proj = l.in_proj->tiles; s.in_rows = (int)l.in_proj->rows;
        s.out_proj = (l.recurrent ? l.ssm_out : l.o)->tiles; s.gate_up = l.gate_up->tiles; s.down = l.ffn_down->tiles;
        s.attn_norm = l.attn_norm; s.post_norm = l.post_norm;
        s.conv_w = l.conv_w; s.dt = l.dt; s.a = l.a; s.beta = l.beta; s.alpha = l.alpha; s.ssm_norm = l.ssm_norm; s.conv_st = l.conv_st; s.ssm_st = l.ssm_st;
        s.q_norm = l.q_norm; s.k_norm = l.k_norm; s.kc = l.kc; s.vc = l.vc;
    }
    std::vector<StepSpan> sp((size_t)st->grid * SP_KINDS);
    step_spans(sp, SP_IN_GDN, st->grid, it_cfg_conv_dim(c) + c.ssm_inner, c.n_embd, 1);
    {   // tests drop one CTA's share here, so that the rows it should publish never come and the waits for them run out
        const char* v = getenv("IT_STEP_DROP_CTA"); const int b = v ? atoi(v) : -1;
        if (b >= 0 && b < st->grid) sp[(size_t)b * SP_KINDS + SP_IN_GDN] = step_span(0, 0, c.n_embd / 128, 1, 0);
    }
    step_spans(sp, SP_IN_ATT, st->grid, (2 * c.n_head + 2 * c.n_head_kv) * c.head_dim, c.n_embd, 1);
    step_spans(sp, SP_OUT_GDN, st->grid, c.n_embd, c.ssm_inner, 1);
    step_spans(sp, SP_OUT_ATT, st->grid, c.n_embd, c.n_head * c.head_dim, 1);
    step_spans(sp, SP_GATE_UP, st->grid, 2 * c.n_ff, c.n_embd, 2);
    step_spans(sp, SP_DOWN, st->grid, c.n_embd, c.n_ff, 1);
    step_spans(sp, SP_HEAD, st->grid, c.n_vocab, c.n_embd, 1);
    int r = it_engine_dev_alloc(e, (void**)&st->layers_dev, hl.size() * sizeof(StepLayer), false);
    if (r == IT_OK) r = it_engine_dev_alloc(e, (void**)&st->spans_dev, sp.size() * sizeof(StepSpan), false);
    auto granules = [&](granule** p, size_t n) { if (r == IT_OK) r = it_engine_dev_alloc(e, (void**)p, n * sizeof(granule), true); };
    auto row_of = [&](granule** p, size_t rows) { granules(p, (rows + 31) / 32 * ST_GPU); };
    row_of(&st->xe, c.n_embd); row_of(&st->xi, c.n_embd); row_of(&st->rows, std::max((size_t)it_cfg_conv_dim(c) + c.ssm_inner, (size_t)(2 * c.n_head + 2 * c.n_head_kv) * c.head_dim));
    row_of(&st->o, std::max(c.ssm_inner, c.n_head * c.head_dim)); row_of(&st->act, c.n_ff);
    granules(&st->codes, (size_t)(step_widest(c) / 1024) * 128 * ST_COPIES * 2); granules(&st->prefix, (size_t)st->grid * 32); granules(&st->partials, (size_t)st->grid * ST_NSUM);
    if (r == IT_OK) r = it_engine_dev_alloc(e, (void**)&st->gate, 2 * (size_t)c.ssm_vheads * sizeof(unsigned long long), true);
    if (r == IT_OK && c.head_dim % 32) r = it_engine_dev_alloc(e, (void**)&st->o1, (size_t)c.n_head * c.head_dim * sizeof(unsigned long long), true);
    if (r == IT_OK) r = it_engine_dev_alloc(e, (void**)&st->att_sc, (size_t)c.n_head * st->att_stride * sizeof(unsigned long long), true);
    { const char* v = getenv("IT_STEP_TRACE"); if (r == IT_OK && v && atoi(v) != 0) r = it_engine_dev_alloc(e, (void**)&st->trace, (2 * ST_TRACE_MAX * 2 + ST_EVT_MAX) * sizeof(unsigned long long), true); }
    if (r) { delete st; return r; }
    IT_CUDA(cudaMemcpyAsync(st->layers_dev, hl.data(), hl.size() * sizeof(StepLayer), cudaMemcpyHostToDevice, cx->stream));
    IT_CUDA(cudaMemcpyAsync(st->spans_dev, sp.data(), sp.size() * sizeof(StepSpan), cudaMemcpyHostToDevice, cx->stream));
    IT_CUDA(cudaStreamSynchronize(cx->stream));
    e->step = st;
    return IT_OK;
}
void it_step_release(it_engine* e) { delete e->step; e->step = nullptr; }

// Enqueues one step.  flags: 1 the token is the previous pick, 2 hand the pick over to the next step, 4 logits and pick wanted.
int it_step_launch(it_engine* e, int flags) {
    it_step_state* st = e->step; it_ctx* cx = e->ctx; const it_model_config& c = e->cfg; const it_arena_layout& L = e->lay;
    StepParams P; memset(&P, 0, sizeof P);
    P.layers = st->layers_dev; P.spans = st->spans_dev; P.n_layer = c.n_layer;
    P.e = c.n_embd; P.ff = c.n_ff; P.widest = step_widest(c); P.hd = c.head_dim; P.nh = c.n_head; P.nkv = c.n_head_kv; P.cd = it_cfg_conv_dim(c); P.inner = c.ssm_inner; P.nv = c.ssm_vheads;
    P.nk = c.ssm_groups; P.qk = it_cfg_qk(c); P.conv_k = c.conv_k; P.n_rot = c.n_rot; P.n_vocab = c.n_vocab;
    P.eps = c.eps; P.theta_scale = e->theta_scale; for (int i = 0; i < 4; i++) P.sec[i] = c.rope_sections[i]; P.v_grouped = c.gdn_v_grouped;
    P.arena = cx->arena; P.xe = st->xe; P.xi = st->xi; P.rows = st->rows; P.o = st->o; P.o1 = st->o1; P.act = st->act; P.codes = st->codes; P.codes_half = step_widest(c) / 1024 * 128 * ST_COPIES; P.prefix = st->prefix; P.had_step = st->had_step; P.hrow = L.hrow; P.logits = L.logits; P.amx = L.amx; P.gate = st->gate;
    { const size_t w[4] = { (size_t)c.n_embd, (size_t)c.ssm_inner, (size_t)c.n_head * c.head_dim, (size_t)c.n_ff }; for (int k = 0; k < 4; k++) P.sg[k] = reinterpret_cast<const uint32_t*>(cx->signs[w[k]] + w[k]); }
    P.tok_embd = e->tok_embd; P.output_norm = e->output_norm; P.output = e->output->tiles;
    P.toks = e->toks_dev; P.pos = e->pos_dev;
    P.sync = cx->grid_sync; P.partials = st->partials; P.error_flag = cx->error_flag_dev;
    P.slots = st->slots; P.scratch = st->scratch; P.w_off = st->scratch - (int)step_w_bytes(c); P.flags = flags; P.trace = st->trace; P.gdn_off = st->gdn_off; P.attn_base = st->attn_base; P.attn_g = st->attn_g; P.att_sc = st->att_sc; P.att_stride = st->att_stride;
    it_note_op(cx);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)st->grid); cfg.blockDim = dim3(ST_THREADS); cfg.dynamicSmemBytes = step_smem_bytes(c, st->slots, st->attn_g); cfg.stream = cx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative; attr[0].val.cooperative = 1;
    cfg.attrs = attr; cfg.numAttrs = st->cooperative ? 1 : 0;
    IT_CUDA(cudaLaunchKernelEx(&cfg, st->any ? k_decode_step<true> : k_decode_step<false>, P));
    return IT_OK;
}

// Diagnostics (IT_STEP_TRACE=1 when the engine is built): the nanosecond clock of CTA 0 and of the last CTA when they arrive
// at and leave each wait in front of a matrix phase of the most recent step: out[(cta * max + barrier) * 2 + {0, 1}], cta in {0, 1}.
IT_API int it_engine_step_trace(it_engine* e, uint64_t* out, size_t max_barriers) {
    IT_CHECK_ARG(e && out, "it_engine_step_trace: null argument");
    if (!e->step || !e->step->trace) return it_fail(IT_ESTATE, "it_engine_step_trace: the engine was not built with IT_STEP_TRACE=1, or does not run the step kernel");
    IT_CHECK_ARG(max_barriers == ST_TRACE_MAX || max_barriers == ST_TRACE_MAX + ST_EVT_MAX / 4, "it_engine_step_trace: pass room for %d barriers per CTA", ST_TRACE_MAX);
    IT_CUDA(cudaMemcpyAsync(out, e->step->trace, (2 * ST_TRACE_MAX * 2 + (max_barriers > ST_TRACE_MAX ? ST_EVT_MAX : 0)) * sizeof(unsigned long long), cudaMemcpyDeviceToHost, e->ctx->stream));
    IT_CUDA(cudaStreamSynchronize(e->ctx->stream));
    return IT_OK;
}
