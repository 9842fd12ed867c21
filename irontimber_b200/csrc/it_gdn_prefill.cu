// Gated delta rule of a prompt pass (src/cpu.rs:215-232): many rows of the pass, every state row on its own.
//
// k_gdn_norm (it_support.cu) gives a head one CTA, which suits passes of a few rows: 48 CTAs, one warp per scheduler with two chains and seven
// operations per element and token, and 100 SMs idle: 264 us per 256 rows of the 27B shape.
// Here a CTA has 64 state rows of a head: 96 CTAs at the 27B shape.  A row has two threads, one in each of two warps, that both keep the
// row in registers and update it alike; thread A carries the chain of additions of s (and so the next token's delta, which it
// hands over through shared memory), thread B the chain of acc.  Per element that is five rounded operations a warp instead of seven.
// Four busy warps and a loader: every scheduler of the SM has one.  What bounds it is one warp's issue, about 800 instructions in 1260 cycles a token (173 us per 256 rows).
// The gated norm that follows needs all of a head's rows and is k_norm_head's.
//
// Arithmetic per state row is k_gdn_norm's, operation for operation: x[] holds the row already multiplied by the decay of the token
// about to use it; the two ordered sums of a token, s = sum_i x[i] * k[i] and acc = sum_i st[i] * q[i], are kept in index order.
#include "it_math.h"
#include "it_support.h"
#include "it_pipe.cuh"
#include "it_route.h"

namespace {

constexpr int GP_SD = 128, GP_ROWS = 64, GP_TOK = 16, GP_RING = 3;        // state size; state rows per CTA; tokens per stage; stages
struct GpStage { float k[GP_TOK][GP_SD], q[GP_TOK][GP_SD], v[GP_TOK][GP_ROWS], bt[GP_TOK], eg[GP_TOK]; };

template <bool V> struct GpBool { static constexpr bool value = V; };
__device__ __forceinline__ void bar_sync(int id) { asm volatile("bar.sync %0, 64;" :: "r"(id) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id) { asm volatile("bar.arrive %0, 64;" :: "r"(id) : "memory"); }

__global__ void __launch_bounds__(160) k_gdn_rows(const float* co, size_t co_ts, const float* beta, const float* alpha, size_t ba_ts, const float* __restrict__ dt, const float* __restrict__ a,
                                                 float* state, float* o, size_t o_ts, int nk, int qk, int nt, int* error_flag) {
    IT_PDL_TRIGGER(); IT_PDL_WAIT();
    extern __shared__ __align__(16) unsigned char gp_smem[];
    GpStage* st = reinterpret_cast<GpStage*>(gp_smem);
    __shared__ __align__(8) unsigned long long bars[2 * GP_RING];
    __shared__ int abort_word;
    __shared__ float deltas[2][GP_ROWS];
    volatile int* abort_flag = &abort_word;
    const int h = blockIdx.x, j0 = blockIdx.y * GP_ROWS, lane = threadIdx.x & 31, kh = h % nk, ns = (nt + GP_TOK - 1) / GP_TOK;
    const unsigned full0 = smem_u32(bars), empty0 = full0 + 8 * GP_RING;
    if (threadIdx.x == 0) {
        abort_word = 0;
        for (int s = 0; s < GP_RING; s++) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 4); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5;       // A and B of rows 0..31, A and B of rows 32..63, loader
    if (warp == 4) {
        // ---- loader warp: q, k, v rows of a stage of tokens and the tokens' gates (sigmoid(beta), exp(softplus(alpha + dt) * a)), which depend on no state
        for (int c = 0; c < ns; c++) {
            const int s = c % GP_RING, t0 = c * GP_TOK, n = min(GP_TOK, nt - t0);
            if (!__all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, ((unsigned)(c / GP_RING) & 1u) ^ 1u, abort_flag, error_flag, 31))) break;
            for (int t = 0; t < n; t++) {
                const float* src = co + (size_t)(t0 + t) * co_ts;
                cp_async16(&st[s].q[t][4 * lane], src + kh * GP_SD + 4 * lane);
                cp_async16(&st[s].k[t][4 * lane], src + qk + kh * GP_SD + 4 * lane);
                if (lane < GP_ROWS / 4) cp_async16(&st[s].v[t][4 * lane], src + 2 * qk + h * GP_SD + j0 + 4 * lane);
            }
            if (lane < n) {
                const size_t i = (size_t)(t0 + lane) * ba_ts + h;
                st[s].bt[lane] = it_sigmoid(beta[i]);
                st[s].eg[lane] = it_expf(it_mul(it_softplus(it_add(alpha[i], dt[h])), a[h]));
            }
            cp_async_wait_all();
            __syncwarp();
            if (lane == 0) mbar_arrive(full0 + 8 * s);
        }
        return;
    }
    // ---- one state row per thread, in registers for the whole pass.  Named barriers, four per pair of warps: 1 + b = "the delta is in
    // deltas[b]" (A arrives, B waits), 3 + b = "deltas[b] has been read" (B arrives, A waits before it writes it again two tokens later).
    const bool is_a = !(warp & 1);
    const int r = (warp >> 1) * 32 + lane;                  // this thread's row of the CTA
    const int b0 = (warp >> 1) * 4;
    float x[GP_SD];
    float4* row = reinterpret_cast<float4*>(state + ((size_t)h * GP_SD + j0 + r) * GP_SD);
#pragma unroll
    for (int c = 0; c < GP_SD / 4; c++) { const float4 r = row[c]; x[4 * c] = r.x; x[4 * c + 1] = r.y; x[4 * c + 2] = r.z; x[4 * c + 3] = r.w; }
    bool ok = mbar_wait(full0, 0u, abort_flag, error_flag, 32);
    const float eg0 = st[0].eg[0];
#pragma unroll
    for (int i = 0; i < GP_SD; i++) x[i] = it_mul(x[i], eg0);
    int sl = 0, tt = 0; unsigned ph = 0;                    // stage, token inside it, phase of the stage
    int old = 0; bool leave = false, last = false;
    // to the token after t: from the next stage at the end of this one.  After the last token the factor 1 leaves the state itself in x, bit for bit
    auto advance = [&](int t) {
        old = sl; leave = tt + 1 == GP_TOK; last = t + 1 == nt;
        if (leave) { tt = 0; if (++sl == GP_RING) { sl = 0; ph ^= 1u; } } else tt++;
        if (ok && leave && !last) ok = mbar_wait(full0 + 8 * sl, ph, abort_flag, error_flag, 33);
    };
    auto release = [&]() { if (leave) { __syncwarp(); if (lane == 0) mbar_arrive(empty0 + 8 * old); } };
    // A row is worked through in blocks of GP_B elements.  The terms of the ordered sum wait in pr[] for one block, and their additions,
    // four cycles apart at best, stand between the independent operations of the next block; the operands of the next
    // block are loaded meanwhile.  (Left to the compiler's order the same operations take twice as long.)
    constexpr int GP_B = 16, NB = GP_SD / GP_B;
    float4 ka[2][GP_B / 4], wa[2][GP_B / 4];
    float pr[GP_B];
    auto load = [&](float4 (&d)[GP_B / 4], const float* src) {
#pragma unroll
        for (int c = 0; c < GP_B / 4; c++) d[c] = *reinterpret_cast<const float4*>(src + 4 * c);
    };
    float sum;
    // one block: x <- (x + k * delta) * eg; term = (A ? the new x : x + k * delta) * w.  Adds the block before's terms to the sum unless FIRST.
    auto block = [&](auto is_a_c, auto first_c, float* xb, const float4 (&kb)[GP_B / 4], const float4 (&wb)[GP_B / 4], float delta, float eg) {
        constexpr bool IS_A = decltype(is_a_c)::value, FIRST = decltype(first_c)::value;
#pragma unroll
        for (int c = 0; c < GP_B / 4; c++) {
            const float k[4] = { kb[c].x, kb[c].y, kb[c].z, kb[c].w }, w[4] = { wb[c].x, wb[c].y, wb[c].z, wb[c].w };
            float u[4], v[4];
#pragma unroll
            for (int e = 0; e < 4; e++) u[e] = it_mul(k[e], delta);
            if (!FIRST) sum = it_add(sum, pr[4 * c]);
#pragma unroll
            for (int e = 0; e < 4; e++) u[e] = it_add(xb[4 * c + e], u[e]);
            if (!FIRST) sum = it_add(sum, pr[4 * c + 1]);
#pragma unroll
            for (int e = 0; e < 4; e++) xb[4 * c + e] = it_mul(u[e], eg);
            if (!FIRST) sum = it_add(sum, pr[4 * c + 2]);
#pragma unroll
            for (int e = 0; e < 4; e++) v[e] = it_mul(IS_A ? xb[4 * c + e] : u[e], w[e]);
            if (!FIRST) sum = it_add(sum, pr[4 * c + 3]);
#pragma unroll
            for (int e = 0; e < 4; e++) pr[4 * c + e] = v[e];
        }
    };
    auto flush = [&]() {
#pragma unroll
        for (int e = 0; e < GP_B; e++) sum = it_add(sum, pr[e]);
    };
    using T = GpBool<true>; using F = GpBool<false>;
    if (is_a) {
        sum = 0.f;
#pragma unroll
        for (int c = 0; c < GP_SD / 4; c++) {
            const float4 k4 = *reinterpret_cast<const float4*>(&st[0].k[0][4 * c]);
            const float m[4] = { it_mul(x[4 * c], k4.x), it_mul(x[4 * c + 1], k4.y), it_mul(x[4 * c + 2], k4.z), it_mul(x[4 * c + 3], k4.w) };
#pragma unroll
            for (int e = 0; e < 4; e++) { if (4 * c + e < GP_SD - GP_B) sum = it_add(sum, m[e]); else pr[4 * c + e - (GP_SD - GP_B)] = m[e]; }
        }
        for (int t = 0; t < nt; t++) {
            const float* kt = st[sl].k[tt];
            const float v = st[sl].v[tt][r], bt = st[sl].bt[tt];
            load(ka[0], kt);
            advance(t);
            const float* kn = last ? kt : st[sl].k[tt];      // after the last token the sum is not used
            const float egn = last ? 1.0f : st[sl].eg[tt];
            load(wa[0], kn);
            if (t >= 2) bar_sync(b0 + 3 + (t & 1));
            flush();
            const float delta = it_mul(it_sub(v, sum), bt);
            deltas[t & 1][r] = delta;
            bar_arrive(b0 + 1 + (t & 1));
            sum = 0.f;
#pragma unroll
            for (int b = 0; b < NB; b++) {
                if (b + 1 < NB) { load(ka[(b + 1) & 1], kt + (b + 1) * GP_B); load(wa[(b + 1) & 1], kn + (b + 1) * GP_B); }
                if (b == 0) block(T{}, T{}, x, ka[0], wa[0], delta, egn);
                else block(T{}, F{}, x + b * GP_B, ka[b & 1], wa[b & 1], delta, egn);
            }
            release();
        }
#pragma unroll
        for (int c = 0; c < GP_SD / 4; c++) row[c] = make_float4(x[4 * c], x[4 * c + 1], x[4 * c + 2], x[4 * c + 3]);
    } else {
        const float scale = it_div(1.0f, it_sqrt((float)GP_SD));
        float* op = o + (size_t)h * GP_SD + j0 + r;
        for (int t = 0; t < nt; t++, op += o_ts) {
            const float* kt = st[sl].k[tt]; const float* qt = st[sl].q[tt];
            load(ka[0], kt); load(wa[0], qt);
            bar_sync(b0 + 1 + (t & 1));
            const float delta = deltas[t & 1][r];
            bar_arrive(b0 + 3 + (t & 1));
            advance(t);
            const float egn = last ? 1.0f : st[sl].eg[tt];
            sum = 0.f;
#pragma unroll
            for (int b = 0; b < NB; b++) {
                if (b + 1 < NB) { load(ka[(b + 1) & 1], kt + (b + 1) * GP_B); load(wa[(b + 1) & 1], qt + (b + 1) * GP_B); }
                if (b == 0) block(F{}, T{}, x, ka[0], wa[0], delta, egn);
                else block(F{}, F{}, x + b * GP_B, ka[b & 1], wa[b & 1], delta, egn);
            }
            flush();
            *op = it_mul(sum, scale);
            release();
        }
    }
}

}  // namespace

// Delta rule of nt rows without the norm behind it.  Returns 1 (nothing launched) when the shape does not suit this kernel.
int it_sup_gdn_rows(it_ctx* c, const float* co, size_t co_ts, const float* beta, const float* alpha, size_t ba_ts, const float* dt, const float* a, float* state, float* o, size_t o_ts,
                    int nv, int nk, int sd, int qk, int nt) {
    static_assert(GP_SD == 128, "it_gdn_rows_takes");
    if (!it_gdn_rows_takes(sd, nt) || ((reinterpret_cast<uintptr_t>(co) | reinterpret_cast<uintptr_t>(state)) & 15) || co_ts % 4 || qk % 4) return 1;
    it_note_op(c);
    const size_t smem = GP_RING * sizeof(GpStage);
    static bool set[16] = {};       // the attribute is per device
    if (!set[c->device & 15]) { IT_CUDA(cudaFuncSetAttribute(k_gdn_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); set[c->device & 15] = true; }
    it_pdl(k_gdn_rows, dim3(nv, GP_SD / GP_ROWS), dim3(160), smem, c->stream, co, co_ts, beta, alpha, ba_ts, dt, a, state, o, o_ts, nk, qk, nt, c->error_flag_dev);
    IT_LAUNCH_CHECK("gdn_rows");
    return IT_OK;
}
