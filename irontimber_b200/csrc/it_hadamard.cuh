// The Hadamard + q8k block transform as a device function (one 1024-element block by 256 threads), used by k_hadamard.
#pragma once
#include "it_internal.h"
#include "it_math.h"
#include "it_support.h"

namespace {

// Shared memory of one Hadamard block (one CTA of 256 threads).
struct it_had_smem { float4 xch[256]; float wsum[8]; float s_amax[8]; float s_val[8]; unsigned s_idx[8]; };

// The 256 threads of a block synchronise on named barrier 2, so callers may have other warps that do not take part.
__device__ __forceinline__ void it_had_sync() { asm volatile("bar.sync 2, 256;" ::: "memory"); }

struct Best { float amax; float val; unsigned idx; };
__device__ __forceinline__ Best better(Best a, Best b) {
    // b replaces a when strictly larger, or equal magnitude with a lower index
    bool take = (b.amax > a.amax) || (b.amax == a.amax && b.idx < a.idx);
    return take ? b : a;
}

// One 1024-element block of one activation row by 256 threads (tid = 0..255): optional prologue, signs, the ten
// butterfly stages, and either the f32 store or q8k quantisation.  Called by k_hadamard (one CTA per block); the
// barriers are named so that a caller with more warps can use it too.
template <bool QUANT>
__device__ __forceinline__ void it_hadamard_block(it_had_smem& sm, const unsigned tid, const unsigned blk, const size_t tok,
           const float* arena_in, size_t in_off, size_t in_stride,
           float* f32_out, size_t out_off, size_t out_stride,
           const float* __restrict__ signs, int rotate, int inverse,
           unsigned perm_hd, unsigned perm_nk, unsigned perm_rep,
           int8_t* __restrict__ qs, float* __restrict__ qd, int32_t* __restrict__ qsum, size_t q_stride, const it_had_prologue& pro) {
    float4* xch = sm.xch; float* wsum = sm.wsum; float* s_amax = sm.s_amax; float* s_val = sm.s_val; unsigned* s_idx = sm.s_idx;
    const unsigned lane = tid & 31, warp = tid >> 5;
    const unsigned g0 = blk * 1024u + 4u * tid;      // index of this thread's first element inside the row
    const float* x = arena_in + in_off + tok * in_stride;

    // loads that depend on nothing computed here are issued first, so that their latency overlaps the row reduction
    float4 sg = make_float4(1.f, 1.f, 1.f, 1.f);
    if (signs) sg = *reinterpret_cast<const float4*>(signs + g0);
    float4 own = make_float4(0.f, 0.f, 0.f, 0.f), w4 = own;
    if (pro.mode == 2) { own = *reinterpret_cast<const float4*>(x + g0); w4 = *reinterpret_cast<const float4*>(pro.w + g0); }
    float v[4];
    if (pro.mode == 2) {
        // rmsnorm of the whole row first (src/cpu.rs:14-18), in the order of k_rmsnorm_wide: thread i adds x[i]^2,
        // x[i+256]^2, ...; warp butterflies; eight warp sums in ascending order.  Every CTA of the row repeats it.
        float xv[32];
#pragma unroll
        for (int k = 0; k < 32; k++) { const unsigned j = tid + 256u * k; xv[k] = j < pro.n ? x[j] : 0.f; }
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 32; k++) if (tid + 256u * k < pro.n) s = it_add(s, it_mul(xv[k], xv[k]));
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) s = it_add(s, __shfl_xor_sync(0xffffffffu, s, m));
        if (lane == 0) wsum[warp] = s;
        it_had_sync();
        float tot = wsum[0];
#pragma unroll
        for (int k = 1; k < 8; k++) tot = it_add(tot, wsum[k]);
        const float sc = it_div(1.0f, it_sqrt(it_add(it_div(tot, (float)pro.n), pro.eps)));
        const float4 t = own;
        v[0] = it_mul(it_mul(t.x, sc), w4.x); v[1] = it_mul(it_mul(t.y, sc), w4.y); v[2] = it_mul(it_mul(t.z, sc), w4.z); v[3] = it_mul(it_mul(t.w, sc), w4.w);
        if (pro.xn_out) *reinterpret_cast<float4*>(pro.xn_out + tok * pro.xn_stride + g0) = make_float4(v[0], v[1], v[2], v[3]);
    } else if (pro.mode == 1) {
        // silu(a) * b (src/cpu.rs:183) computed on the way in
        const float4 a = *reinterpret_cast<const float4*>(x + g0), b = *reinterpret_cast<const float4*>(pro.b + tok * pro.b_stride + g0);
        v[0] = it_mul(it_silu(a.x), b.x); v[1] = it_mul(it_silu(a.y), b.y); v[2] = it_mul(it_silu(a.z), b.z); v[3] = it_mul(it_silu(a.w), b.w);
    } else if (perm_hd == 0) {
        float4 t = *reinterpret_cast<const float4*>(x + g0);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else {
#pragma unroll
        for (int e = 0; e < 4; e++) {   // grouped [hd, rep, nk] position g reads tiled [hd, nk, rep] source
            unsigned g = g0 + e, i0 = g % perm_hd, q = g / perm_hd, r = q % perm_rep, k = q / perm_rep;
            v[e] = x[i0 + perm_hd * (k + perm_nk * r)];
        }
    }
    if (signs && !inverse) { v[0] *= sg.x; v[1] *= sg.y; v[2] *= sg.z; v[3] *= sg.w; }
    if (rotate) {
        float a, b;
        a = v[0]; b = v[1]; v[0] = a + b; v[1] = a - b;      // h = 1
        a = v[2]; b = v[3]; v[2] = a + b; v[3] = a - b;
        a = v[0]; b = v[2]; v[0] = a + b; v[2] = a - b;      // h = 2
        a = v[1]; b = v[3]; v[1] = a + b; v[3] = a - b;
#pragma unroll
        for (unsigned m = 1; m < 32; m <<= 1) {              // h = 4*m: partner lane differs in bit m
            const bool upper = lane & m;
#pragma unroll
            for (int e = 0; e < 4; e++) {
                float o = __shfl_xor_sync(0xffffffffu, v[e], m);
                v[e] = upper ? (o - v[e]) : (v[e] + o);
            }
        }
#pragma unroll
        for (unsigned m = 32; m < 256; m <<= 1) {            // h = 4*m: partner thread differs in bit m
            xch[tid] = make_float4(v[0], v[1], v[2], v[3]);
            it_had_sync();
            float4 o = xch[tid ^ m];
            it_had_sync();
            if (tid & m) { v[0] = o.x - v[0]; v[1] = o.y - v[1]; v[2] = o.z - v[2]; v[3] = o.w - v[3]; }
            else         { v[0] = v[0] + o.x; v[1] = v[1] + o.y; v[2] = v[2] + o.z; v[3] = v[3] + o.w; }
        }
#pragma unroll
        for (int e = 0; e < 4; e++) v[e] *= 0.03125f;
    }
    if (signs && inverse) { v[0] *= sg.x; v[1] *= sg.y; v[2] *= sg.z; v[3] *= sg.w; }
    if (!QUANT) {
        *reinterpret_cast<float4*>(f32_out + out_off + tok * out_stride + g0) = make_float4(v[0], v[1], v[2], v[3]);
        return;
    }
    // ---- q8k: first element of maximum magnitude in each 256-element block (threads 64*q .. 64*q+63)
    Best best{0.f, 0.f, 0xffffffffu};
#pragma unroll
    for (int e = 0; e < 4; e++) { float a = fabsf(v[e]); if (a > best.amax) { best.amax = a; best.val = v[e]; best.idx = 4 * tid + e; } }
#pragma unroll
    for (unsigned m = 1; m < 32; m <<= 1) {
        Best o{ __shfl_xor_sync(0xffffffffu, best.amax, m), __shfl_xor_sync(0xffffffffu, best.val, m), __shfl_xor_sync(0xffffffffu, best.idx, m) };
        best = better(best, o);
    }
    if (lane == 0) { s_amax[warp] = best.amax; s_val[warp] = best.val; s_idx[warp] = best.idx; }
    it_had_sync();
    { Best o{ s_amax[warp ^ 1], s_val[warp ^ 1], s_idx[warp ^ 1] }; best = better(best, o); }

    int q[4] = {0, 0, 0, 0}; float d = 0.f;
    if (best.amax != 0.f) {
        const float iscale = __fdiv_rn(-127.0f, best.val);
#pragma unroll
        for (int e = 0; e < 4; e++) q[e] = min(__float2int_rn(__fmul_rn(iscale, v[e])), 127);
        d = __fdiv_rn(1.0f, iscale);
    }
    const size_t row_q = tok * q_stride;
    uint32_t packed = (uint32_t)(uint8_t)q[0] | ((uint32_t)(uint8_t)q[1] << 8) | ((uint32_t)(uint8_t)q[2] << 16) | ((uint32_t)(uint8_t)q[3] << 24);
    *reinterpret_cast<uint32_t*>(qs + row_q + g0) = packed;
    int s = q[0] + q[1] + q[2] + q[3];
#pragma unroll
    for (unsigned m = 16; m > 0; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
    if (lane == 0) qsum[tok * (q_stride / 128) + blk * 8 + warp] = s;
    if ((tid & 63) == 0) qd[tok * (q_stride / 256) + blk * 4 + (tid >> 6)] = d;
}

// ---- the same transform, 64 threads a block and 16 values a thread ---------------------------------------------------------
// Bit-identical to it_hadamard_block (the same pairs in the same stage order).  Thread j (0..63, two warps) passes through three
// layouts: elements 16 j .. (strides 1..8), every 16th of a run of 256 (16..128), four neighbours of each of the block's four
// q8k groups (256, 512).  Between them the block goes through shared memory in a padded layout: a run of 16 is 20 floats apart
// from the next, a run of 256 336 floats, so that neither the 16-byte accesses of the first and last layout nor the 4-byte
// ones of the second meet in a bank.  About 430 instructions a thread and three barriers of 64 threads; the 256-thread form
// has 150 and eleven barriers of 256, i.e. 1.4 times the instructions a block.
constexpr int IT_HAD_PITCH = 1344;                     // floats of a block in the padded layout
__device__ __forceinline__ int it_had_at(int e) { return e + 4 * (e >> 4) + 16 * (e >> 8); }
__device__ __forceinline__ void it_had16_stage(float (&v)[16], int h) {
#pragma unroll
    for (int i = 0; i < 16; i++) if (!(i & h)) { const float a = v[i], b = v[i | h]; v[i] = it_add(a, b); v[i | h] = it_sub(a, b); }
}
// v: elements 16 j + i in, element 256 g + 4 j + u at 4 g + u out, scaled by 1/32.  ex: the block's IT_HAD_PITCH floats; `sync`
// joins the block's 64 threads.
template <typename Sync> __device__ __forceinline__ void it_had16_rotate(float (&v)[16], float* ex, int j, Sync&& sync) {
    const int lane = j & 31;
    it_had16_stage(v, 1); it_had16_stage(v, 2); it_had16_stage(v, 4); it_had16_stage(v, 8);
    float* p1 = ex + it_had_at(16 * j);
#pragma unroll
    for (int u = 0; u < 4; u++) *reinterpret_cast<float4*>(p1 + 4 * u) = make_float4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
    sync();
    float* p2 = ex + 336 * ((lane >> 4) + 2 * (j >> 5)) + (lane & 15);
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = p2[20 * i];
    it_had16_stage(v, 1); it_had16_stage(v, 2); it_had16_stage(v, 4); it_had16_stage(v, 8);
#pragma unroll
    for (int i = 0; i < 16; i++) p2[20 * i] = v[i];
    sync();
    const float* p3 = ex + it_had_at(4 * j);
#pragma unroll
    for (int g = 0; g < 4; g++) { const float4 t = *reinterpret_cast<const float4*>(p3 + 336 * g); v[4 * g] = t.x; v[4 * g + 1] = t.y; v[4 * g + 2] = t.z; v[4 * g + 3] = t.w; }
    it_had16_stage(v, 4); it_had16_stage(v, 8);
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = it_mul(v[i], 0.03125f);
}
// q8k codes of v (element 256 g + 4 j + u at 4 g + u): word g holds the thread's four codes of group g; in lane l < 4, d is the
// scale of group l and sum the sum of group l's codes over the lane's warp (128 elements).  mx: 8 floats of shared memory.
struct it_had16_codes { uint32_t packed[4]; float d; int sum; };
template <typename Sync> __device__ __forceinline__ it_had16_codes it_had16_quantise(const float (&v)[16], float* mx, int j, Sync&& sync) {
    const int lane = j & 31;
    it_had16_codes r;
    // the first element of largest magnitude of each group; b stands for higher indices than a, a NaN is never taken
    auto larger = [](float a, float b, bool tie) { return fabsf(b) > fabsf(a) || (tie && fabsf(b) == fabsf(a)) ? b : a; };
    float any = 0.f, best[4];
#pragma unroll
    for (int i = 0; i < 16; i++) any += v[i];
#pragma unroll
    for (int g = 0; g < 4; g++) {
        best[g] = 0.f;
#pragma unroll
        for (int u = 0; u < 4; u++) best[g] = larger(best[g], v[4 * g + u], false);
    }
    const bool odd = __any_sync(0xffffffffu, !(fabsf(any) <= 3.4e38f));
    // lanes in ranges that double; the first two steps also share the groups out: lane l keeps group 2 (l & 1) + (l >> 1 & 1)
    float k0 = lane & 1 ? best[2] : best[0], k1 = lane & 1 ? best[3] : best[1];
    const float g0 = __shfl_xor_sync(0xffffffffu, lane & 1 ? best[0] : best[2], 1), g1 = __shfl_xor_sync(0xffffffffu, lane & 1 ? best[1] : best[3], 1);
    k0 = larger(k0, g0, lane & 1); k1 = larger(k1, g1, lane & 1);
    const float g2 = __shfl_xor_sync(0xffffffffu, lane & 2 ? k0 : k1, 2);
    k0 = larger(lane & 2 ? k1 : k0, g2, lane & 2);
#pragma unroll
    for (int m = 4; m <= 16; m <<= 1) k0 = larger(k0, __shfl_xor_sync(0xffffffffu, k0, m), lane & m);
    if (lane < 4) mx[2 * (2 * (lane & 1) + (lane >> 1)) + (j >> 5)] = k0;
    sync();
    const float2 ab = *reinterpret_cast<const float2*>(mx + 2 * (lane & 3));     // lane g (and g + 4, ...): group g's two halves
    const float val = fabsf(ab.y) > fabsf(ab.x) ? ab.y : ab.x;           // equal magnitudes: the lower index
    const float isc = val != 0.f ? __fdiv_rn(-127.0f, val) : 0.f;        // a group of zeros keeps 0, and so codes of 0
    // 1 / scale by a Newton step and a corrected quotient in f64, rounded once: exact to more than twice f32's digits, so the
    // rounding is the division's; without branches, it overlaps the codes
    {
        float r0f; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0f) : "f"(isc));
        const double b = isc, r0 = r0f, r1 = fma(r0, fma(-b, r0, 1.0), r0);
        r.d = __double2float_rn(fma(fma(-b, r1, 1.0), r1, r1));
    }
    if (!(fabsf(isc) >= 3.7e-37f && fabsf(isc) < 1e37f)) r.d = val != 0.f ? __fdiv_rn(1.0f, isc) : 0.f;
    // codes: round to nearest even by adding 1.5 * 2^23 (|is * v| <= 127, and a conversion takes eight cycles of the sub-core where
    // an addition takes one); a scale that overflowed (a group below 4e-37) and values that are not finite go through the
    // conversion and its saturation
    const bool convert = odd || __any_sync(0xffffffffu, fabsf(isc) > 3.4e38f);
    int total[4];
#pragma unroll
    for (int g = 0; g < 4; g++) {
        const float is = __shfl_sync(0xffffffffu, isc, g);
        unsigned q[4];
#pragma unroll
        for (int u = 0; u < 4; u++) q[u] = __float_as_uint(__fadd_rn(it_mul(is, v[4 * g + u]), 12582912.0f));
        if (convert) {
#pragma unroll
            for (int u = 0; u < 4; u++) q[u] = is == 0.f ? 0u : (unsigned)min(__float2int_rn(it_mul(is, v[4 * g + u])), 127);
            total[g] = (int)(q[0] + q[1] + q[2] + q[3]);             // saturated below, a code is its low byte and still counts whole
        }
        r.packed[g] = __byte_perm(__byte_perm(q[0], q[1], 0x0040), __byte_perm(q[2], q[3], 0x0040), 0x5410);
        if (is == 0.f) r.packed[g] = 0;                              // a group of zeros, or one whose maximum is infinite
    }
    const int t0 = __reduce_add_sync(0xffffffffu, __dp4a((int)r.packed[0], 0x01010101, __dp4a((int)r.packed[1], 0x01010101, 0) << 16));   // two groups' sums
    const int t1 = __reduce_add_sync(0xffffffffu, __dp4a((int)r.packed[2], 0x01010101, __dp4a((int)r.packed[3], 0x01010101, 0) << 16));   // (below 2^15) to a word
    const int t = lane & 2 ? t1 : t0, lo = (short)t;
    r.sum = lane & 1 ? (t - lo) >> 16 : lo;
    if (convert) {
#pragma unroll
        for (int g = 0; g < 4; g++) { const int t4 = __reduce_add_sync(0xffffffffu, total[g]); if (lane == g) r.sum = t4; }
    }
    return r;
}

}  // namespace
