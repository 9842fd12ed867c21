// Fused Hadamard rotation + q8k activation quantisation, and the plain f32 transform.
//
// k_hadamard: one CTA of 256 threads per (1024-element block, activation row).  Thread `tid` owns elements
// 4*tid .. 4*tid+3.  The ten radix-2 stages run in the reference's order h = 1, 2, ..., 512 on the
// pairs (j, j+h) with new[j] = a + b, new[j+h] = a - b (src/hadamard.rs:12-17; shaders/hadamard.comp:20-25):
// stages 1-2 inside the thread, 4-64 by lane exchange, 128-512 through shared memory.  Every
// output is produced by the same sequence of rounded additions as on the CPU, so the f32 result
// is bit-identical; the scale 1/32 is exact.
//
// Quantisation follows quantize_row_q8_K_ref as restated in src/quant.rs:75-90: per 256 elements
// (two warps) the signed value of the FIRST element of maximum magnitude gives iscale = -127/max;
// q = min(round_half_even(iscale*x), 127); d = 1/iscale; per-128 sums of q (one warp each).
// Algorithmic traffic per row: 4n bytes in, n + 4n/256 + 4n/128 bytes out.
#include "it_hadamard.cuh"

namespace {

template <bool QUANT>
__global__ void __launch_bounds__(256)
k_hadamard(const float* arena_in, size_t in_off, size_t in_stride,
           float* f32_out, size_t out_off, size_t out_stride,
           const float* __restrict__ signs, int rotate, int inverse,
           unsigned perm_hd, unsigned perm_nk, unsigned perm_rep,
           int8_t* __restrict__ qs, float* __restrict__ qd, int32_t* __restrict__ qsum, size_t q_stride, it_had_prologue pro) {
    IT_PDL_TRIGGER(); IT_PDL_WAIT();
    __shared__ it_had_smem sm;
    it_hadamard_block<QUANT>(sm, threadIdx.x, blockIdx.x, blockIdx.y, arena_in, in_off, in_stride, f32_out, out_off, out_stride, signs, rotate, inverse,
                             perm_hd, perm_nk, perm_rep, qs, qd, qsum, q_stride, pro);
}

// silu(a) * b of four elements, the operations of it_silu.  CUDA's division branches, which puts sixteen of them behind one another; where every
// lane's operands suit it (it_quot_fits), the quotient is formed without branches, four side by side; else the warp takes the division.
__device__ __forceinline__ float4 silu_mul4(const float4 a4, const float4 b4) {
    const float a[4] = { a4.x, a4.y, a4.z, a4.w }, b[4] = { b4.x, b4.y, b4.z, b4.w };
    float d[4], q[4]; bool plain = true;
#pragma unroll
    for (int i = 0; i < 4; i++) { d[i] = it_add(1.0f, it_expf_inline(-a[i])); plain = plain && it_quot_fits(a[i], d[i]); }
    if (__all_sync(0xffffffffu, plain)) {
#pragma unroll
        for (int i = 0; i < 4; i++) { float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d[i])); q[i] = it_quot(a[i], d[i], r); }
    } else {
#pragma unroll 1
        for (int i = 0; i < 4; i++) { const float x = i == 0 ? a[0] : i == 1 ? a[1] : i == 2 ? a[2] : a[3], y = i == 0 ? d[0] : i == 1 ? d[1] : i == 2 ? d[2] : d[3], z = it_div(x, y); if (i == 0) q[0] = z; else if (i == 1) q[1] = z; else if (i == 2) q[2] = z; else q[3] = z; }
    }
    return make_float4(it_mul(q[0], b[0]), it_mul(q[1], b[1]), it_mul(q[2], b[2]), it_mul(q[3], b[3]));
}

// Hadamard + q8k, 64 threads a block (it_had16_*).  ROW: a norm first, formed once by a CTA that takes the whole row, a pair of warps per block (at
// most eight); else a CTA of 64 threads takes one block.
struct Had16In {
    const float* x; size_t stride; const float* signs; int rotate, nblk;
    unsigned hd, nk, rep;
    int8_t* qs; float* qd; int32_t* qsum; size_t q_stride;
};
template <bool ROW>
__global__ void __launch_bounds__(ROW ? 512 : 64) k_hadamard16(const Had16In in, const it_had_prologue pro) {
    IT_PDL_TRIGGER(); IT_PDL_WAIT();
    extern __shared__ __align__(16) float sm[];                  // [pairs][IT_HAD_PITCH], [pairs][8] group maxima; ROW: [8] warp sums of squares
    const int tid = threadIdx.x, j = tid & 63, pair = ROW ? tid >> 6 : 0, pairs = ROW ? (int)blockDim.x >> 6 : 1, lane = tid & 31;
    const int blk = ROW ? pair : (int)blockIdx.x; const size_t tok = ROW ? blockIdx.x : blockIdx.y;
    float* ex = sm + pair * IT_HAD_PITCH; float* mx = sm + pairs * IT_HAD_PITCH + pair * 8;
    auto sync = [&] { if (ROW) asm volatile("bar.sync %0, 64;" :: "r"(1 + pair) : "memory"); else __syncthreads(); };
    const float* x = in.x + tok * in.stride;
    const int g0 = blk * 1024 + 4 * j;                           // thread j comes in with elements g0 + 256 u .. + 3 (16-byte pieces in lane order)
    float4 r[4], sg[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        size_t at = (size_t)(g0 + 256 * u);
        if (in.hd && in.hd % 4 == 0) {                           // grouped [hd, rep, nk] position reads tiled [hd, nk, rep] source
            const unsigned g = (unsigned)at, i0 = g % in.hd, q = g / in.hd, rr = q % in.rep, k = q / in.rep;
            at = i0 + in.hd * (k + in.nk * rr);
        } else if (in.hd) {
            float t[4];
            for (int e = 0; e < 4; e++) { const unsigned g = (unsigned)at + e, i0 = g % in.hd, q = g / in.hd, rr = q % in.rep, k = q / in.rep; t[e] = x[i0 + in.hd * (k + in.nk * rr)]; }
            r[u] = make_float4(t[0], t[1], t[2], t[3]);
        }
        if (!in.hd || in.hd % 4 == 0) r[u] = *reinterpret_cast<const float4*>(x + at);
        sg[u] = in.signs ? *reinterpret_cast<const float4*>(in.signs + g0 + 256 * u) : make_float4(1.f, 1.f, 1.f, 1.f);
    }
    if (!ROW && pro.mode == 1) {
        // silu(a) * b on the way in (src/cpu.rs:183)
        const float* b = pro.b + tok * pro.b_stride + g0;
#pragma unroll
        for (int u = 0; u < 4; u++) r[u] = silu_mul4(r[u], *reinterpret_cast<const float4*>(b + 256 * u));
    }
    if constexpr (ROW) {
        // rmsnorm of the whole row first (src/cpu.rs:14-18), in the order of k_rmsnorm_wide: thread i of 256 adds x[i]^2,
        // x[i + 256]^2, ...; warp butterflies; eight warp sums in ascending order
        float* ws = sm + pairs * (IT_HAD_PITCH + 8);
        float4 w[4];
#pragma unroll
        for (int u = 0; u < 4; u++) w[u] = *reinterpret_cast<const float4*>(pro.w + g0 + 256 * u);
#pragma unroll
        for (int u = 0; u < 4; u++) *reinterpret_cast<float4*>(ex + it_had_at(4 * j) + 336 * u) = r[u];
        __syncthreads();
        if (tid < 64) {
            // four neighbours of the 256 at a time: their butterflies over lanes 16, 8, 4 are this thread's over 4, 2, 1
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
            const float* xp = sm + it_had_at(4 * tid);
#pragma unroll 4
            for (int k = 0; k < in.nblk * 4; k++) {
                const float4 t = *reinterpret_cast<const float4*>(xp + 336 * k);
                s.x = it_add(s.x, it_mul(t.x, t.x)); s.y = it_add(s.y, it_mul(t.y, t.y)); s.z = it_add(s.z, it_mul(t.z, t.z)); s.w = it_add(s.w, it_mul(t.w, t.w));
            }
#pragma unroll
            for (int m = 4; m >= 1; m >>= 1) {
                s.x = it_add(s.x, __shfl_xor_sync(0xffffffffu, s.x, m)); s.y = it_add(s.y, __shfl_xor_sync(0xffffffffu, s.y, m));
                s.z = it_add(s.z, __shfl_xor_sync(0xffffffffu, s.z, m)); s.w = it_add(s.w, __shfl_xor_sync(0xffffffffu, s.w, m));
            }
            if ((lane & 7) == 0) ws[tid >> 3] = it_add(it_add(s.x, s.z), it_add(s.y, s.w));
        }
        __syncthreads();
        float tot = ws[0];
#pragma unroll
        for (int k = 1; k < 8; k++) tot = it_add(tot, ws[k]);
        const float sc = it_div(1.0f, it_sqrt(it_add(it_div(tot, (float)pro.n), pro.eps)));
#pragma unroll
        for (int u = 0; u < 4; u++) {
            r[u].x = it_mul(it_mul(r[u].x, sc), w[u].x); r[u].y = it_mul(it_mul(r[u].y, sc), w[u].y); r[u].z = it_mul(it_mul(r[u].z, sc), w[u].z); r[u].w = it_mul(it_mul(r[u].w, sc), w[u].w);
            if (pro.xn_out) *reinterpret_cast<float4*>(pro.xn_out + tok * pro.xn_stride + g0 + 256 * u) = r[u];
        }
    }
    float v[16];
#pragma unroll
    for (int u = 0; u < 4; u++) { v[4 * u] = it_mul(r[u].x, sg[u].x); v[4 * u + 1] = it_mul(r[u].y, sg[u].y); v[4 * u + 2] = it_mul(r[u].z, sg[u].z); v[4 * u + 3] = it_mul(r[u].w, sg[u].w); }
    if (in.rotate) {
#pragma unroll
        for (int u = 0; u < 4; u++) *reinterpret_cast<float4*>(ex + it_had_at(4 * j) + 336 * u) = make_float4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
        sync();
        const float* p1 = ex + it_had_at(16 * j);
#pragma unroll
        for (int u = 0; u < 4; u++) { const float4 t = *reinterpret_cast<const float4*>(p1 + 4 * u); v[4 * u] = t.x; v[4 * u + 1] = t.y; v[4 * u + 2] = t.z; v[4 * u + 3] = t.w; }
        it_had16_rotate(v, ex, j, sync);
    }
    const it_had16_codes q = it_had16_quantise(v, mx, j, sync);
    int8_t* qs = in.qs + tok * in.q_stride + g0;
#pragma unroll
    for (int g = 0; g < 4; g++) *reinterpret_cast<uint32_t*>(qs + 256 * g) = q.packed[g];
    if (lane < 4) {
        in.qsum[tok * (in.q_stride / 128) + blk * 8 + 2 * lane + (j >> 5)] = q.sum;
        if (j < 4) in.qd[tok * (in.q_stride / 256) + blk * 4 + lane] = q.d;
    }
}

// One CTA of 256 threads a block has the shorter way through one block (4.2 us a launch of a few blocks whatever the prologue, against 4.2
// to 6.2), 64 threads a block the fewer instructions.  They meet at two blocks an SM, with a norm (a CTA a row) between two and four:
// 61 rows of 5120 with norm 6.2 / 6.2 us, 133 rows 8.3 / 6.2; 61 rows plain 5.2 / 4.2, 61 x 17408 with silu 9.3 / 8.3; 777 rows: 26.7 / 17.4 (norm), 24.6 / 15.3 (value heads regrouped, 6144), 71.7 / 48.8
// (silu, 17408; 19 would be HBM's share, the rest is the exponential and the division).
void launch_q8(it_ctx* c, size_t n, size_t ntok, size_t x_off, size_t x_stride, int rotate, const float* signs, size_t hd, size_t nk, size_t rep, it_q8* out, const it_had_prologue& pro) {
    const size_t nblk = n / 1024;
    if (nblk * ntok < (pro.mode == 2 ? 4 : 2) * (size_t)c->sm_count) {
        it_pdl(k_hadamard<true>, dim3((unsigned)nblk, (unsigned)ntok), dim3(256), 0, c->stream, c->arena, x_off, x_stride, nullptr, 0, 0, signs, rotate, 0,
               (unsigned)hd, (unsigned)nk, (unsigned)rep, out->qs, out->d, out->sum128, out->max_n, pro);
        return;
    }
    const Had16In in{ c->arena + x_off, x_stride, signs, rotate, (int)nblk, (unsigned)hd, (unsigned)nk, (unsigned)rep, out->qs, out->d, out->sum128, out->max_n };
    const size_t per = (IT_HAD_PITCH + 8) * sizeof(float);
    if (pro.mode == 2) it_pdl(k_hadamard16<true>, dim3((unsigned)ntok), dim3((unsigned)(64 * nblk)), nblk * per + 32, c->stream, in, pro);      // normed rows are at most 8192 wide: 43.3 KB
    else it_pdl(k_hadamard16<false>, dim3((unsigned)nblk, (unsigned)ntok), dim3(64), per, c->stream, in, pro);
}

int check_common(it_ctx* c, size_t n, size_t ntok, size_t in_off, size_t in_stride, int use_signs,
                 size_t hd, size_t nk, size_t rep, const float** signs, const char* who) {
    IT_CHECK_ARG(c, "%s: null context", who);
    IT_CHECK_ARG(n > 0 && n % 1024 == 0, "%s: width %zu is not a multiple of the 1024 Hadamard block", who, n);
    IT_CHECK_ARG(ntok > 0 && ntok <= 65535, "%s: bad row count %zu", who, ntok);
    IT_CHECK_ARG(in_off % 4 == 0 && (ntok == 1 || in_stride % 4 == 0), "%s: activation offsets must be 4-float aligned", who);
    IT_CHECK_ARG(in_off <= c->arena_floats && (ntok - 1) * in_stride + n <= c->arena_floats - in_off, "%s: input rows fall outside the arena", who);
    if (hd) IT_CHECK_ARG(nk > 0 && rep > 0 && hd * nk * rep == n, "%s: permutation (%zu,%zu,%zu) does not cover width %zu", who, hd, nk, rep, n);
    *signs = nullptr;
    if (use_signs) {
        auto it = c->signs.find(n);
        IT_CHECK_ARG(it != c->signs.end(), "%s: no sign vector registered for width %zu", who, n);
        *signs = it->second;
    }
    return IT_OK;
}

}  // namespace

IT_API int it_hadamard_q8(it_ctx* c, size_t n, size_t ntok, size_t x_off, size_t x_stride, int rotate, int use_signs,
                          size_t hd, size_t nk, size_t rep, it_q8* out) {
    const float* signs; int r = check_common(c, n, ntok, x_off, x_stride, use_signs, hd, nk, rep, &signs, "it_hadamard_q8"); if (r) return r;
    IT_CHECK_ARG(out && out->ctx == c, "it_hadamard_q8: q8 buffer is null or belongs to another context");
    IT_CHECK_ARG(n <= out->max_n && ntok <= out->max_tok, "it_hadamard_q8: %zu rows of %zu do not fit the q8 buffer (%zu x %zu)", ntok, n, out->max_tok, out->max_n);
    it_note_op(c);
    launch_q8(c, n, ntok, x_off, x_stride, rotate, signs, hd, nk, rep, out, it_had_prologue{});
    IT_LAUNCH_CHECK("hadamard_q8");
    out->n = n;
    return IT_OK;
}

IT_API int it_hadamard_f32(it_ctx* c, size_t n, size_t ntok, size_t in_off, size_t in_stride, size_t out_off, size_t out_stride,
                           int use_signs, size_t hd, size_t nk, size_t rep, int inverse) {
    const float* signs; int r = check_common(c, n, ntok, in_off, in_stride, use_signs, hd, nk, rep, &signs, "it_hadamard_f32"); if (r) return r;
    IT_CHECK_ARG(!(inverse && hd), "it_hadamard_f32: the inverse transform takes no permutation");
    IT_CHECK_ARG(!(hd && in_off == out_off), "it_hadamard_f32: a permuted transform cannot run in place");
    IT_CHECK_ARG(out_off % 4 == 0 && (ntok == 1 || out_stride % 4 == 0), "it_hadamard_f32: output offsets must be 4-float aligned");
    IT_CHECK_ARG(out_off <= c->arena_floats && (ntok - 1) * out_stride + n <= c->arena_floats - out_off, "it_hadamard_f32: output rows fall outside the arena");
    it_note_op(c);
    dim3 grid((unsigned)(n / 1024), (unsigned)ntok);
    it_pdl(k_hadamard<false>, dim3(grid), dim3(256), 0, c->stream, c->arena, in_off, in_stride, c->arena, out_off, out_stride, signs, 1, inverse,
        (unsigned)hd, (unsigned)nk, (unsigned)rep, nullptr, nullptr, nullptr, 0, it_had_prologue{});
    IT_LAUNCH_CHECK("hadamard_f32");
    return IT_OK;
}

// Engine-internal: the forward transform + q8k with an elementwise prologue (see it_had_prologue in it_support.h).
int it_sup_hadamard_q8_fused(it_ctx* c, size_t n, size_t ntok, size_t x_off, size_t x_stride, it_q8* out, const it_had_prologue& pro) {
    const float* signs; int r = check_common(c, n, ntok, x_off, x_stride, 1, 0, 0, 0, &signs, "hadamard_q8_fused"); if (r) return r;
    IT_CHECK_ARG(out && out->ctx == c && n <= out->max_n && ntok <= out->max_tok && (pro.mode != 2 || (n <= 8192 && pro.n == n)), "hadamard_q8_fused: bad q8 buffer or width");
    it_note_op(c);
    launch_q8(c, n, ntok, x_off, x_stride, 1, signs, 0, 0, 0, out, pro);
    IT_LAUNCH_CHECK("hadamard_q8_fused");
    out->n = n;
    return IT_OK;
}
