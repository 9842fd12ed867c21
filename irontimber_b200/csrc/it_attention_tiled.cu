// Causal gated attention of a long prompt pass as three kernels: scores, softmax, weighted sums of V.
//
// k_attention_group (it_attention_prefill.cu) keeps a row's scores in shared memory from the first product to the last, so a CTA
// can hold six rows only, and every multiply-add of its two products costs a shared-memory operand: at position 2000 of the 27B
// shape it spends 1386 us per layer and 256-row pass on 13 G separate f32 multiplies and adds whose issue floor is 370 us.
// Here the scores go through a scratch buffer (a block of rows at a time, sized to stay in L2), which makes both products
// plain tiled ones: a thread owns an 8 x 8 block of results, so that sixteen loaded values feed 64 multiply-adds.
//
// Arithmetic per (head, row) is that of k_attention, operation for operation (src/cpu.rs:262-272): every score a
// sequential dot over the head dimension in index order, scaled; the exponentials of (score - max) added in ascending
// position order by one thread; every weight divided by that sum; every output element accumulating w[p] * v[p][j] in
// ascending position order, then * sigmoid(gate).  Every product and every sum is rounded by itself.  Results are bit-identical to k_attention's.
//
// Rows: for one KV head, row m = t * rep + g is query head g of the group at row t of the block, so a tile of consecutive
// rows spans few positions of the causal diagonal.
#include "it_math.h"
#include "it_support.h"
#include "it_route.h"

namespace {

constexpr int AT_M = 128, AT_N = 128, AT_K = 16;   // scores: tile of 128 rows x 128 positions, 16 elements of the head dimension a step
constexpr int AT_J = 64;                            // weighted sums: tile of 128 rows x 64 elements, 16 positions a step

struct AtBlock { int slot0, nt, rep, npad; };      // block of rows: first position, rows, query heads per KV head, stride of a row of scores

__device__ __forceinline__ void at_half8(const uint4& u, float (&f)[8]) {
    const __half2* h = reinterpret_cast<const __half2*>(&u);
#pragma unroll
    for (int i = 0; i < 4; i++) { const float2 t = __half22float2(h[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
}

// scores[kvh][m][p] = (q . k) * scale.  256 threads, thread (ty, tx) owns rows ty * 4 + {0..3}, 64 + ..., positions tx * 4 + {0..3}, 64 + ...
// Tiles beyond the last position their rows see are skipped; values above the diagonal are written and never read.
__global__ void __launch_bounds__(256, 2) k_attn_scores(const float* q, size_t q_hs, size_t q_ts, const __half* __restrict__ kc, int hd, int nkv, AtBlock b, float* __restrict__ scores) {
    IT_PDL_TRIGGER(); IT_PDL_WAIT();
    const int p0 = blockIdx.x * AT_N, m0 = blockIdx.y * AT_M, kvh = blockIdx.z, nm = b.nt * b.rep;
    if (p0 > b.slot0 + min(nm - 1, m0 + AT_M - 1) / b.rep) return;
    __shared__ __align__(16) float as[2][AT_K][AT_M], bs[2][AT_K][AT_N];
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    // loads: thread = one row (position) and half of the step's elements
    const int lr = tid & 127, lh = tid >> 7, m = min(m0 + lr, nm - 1);
    const float* qp = q + (size_t)(m / b.rep) * q_ts + (size_t)(kvh * b.rep + m % b.rep) * q_hs + lh * 8;
    const int last = b.slot0 + b.nt - 1;           // positions past the block's last are not read
    const uint4* kp = reinterpret_cast<const uint4*>(kc + it_kc_index((size_t)min(p0 + lr, last), kvh, 0, nkv, hd)) + lh * 32;   // piece v of this position: kp[32 v]
    float4 qa, qb; uint4 kk;
    auto fetch = [&](int s) { qa = *reinterpret_cast<const float4*>(qp + s * AT_K); qb = *reinterpret_cast<const float4*>(qp + s * AT_K + 4); kk = kp[s * 64]; };
    auto store = [&](int buf) {
        const float qv[8] = { qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w };
        float kf[8]; at_half8(kk, kf);
#pragma unroll
        for (int i = 0; i < 8; i++) { as[buf][lh * 8 + i][lr] = qv[i]; bs[buf][lh * 8 + i][lr] = kf[i]; }
    };
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = 0.f;
    const int steps = hd / AT_K;
    fetch(0); store(0); __syncthreads();
    for (int s = 0; s < steps; s++) {
        const int buf = s & 1;
        if (s + 1 < steps) fetch(s + 1);
#pragma unroll
        for (int k = 0; k < AT_K; k++) {
            const float4 a0 = *reinterpret_cast<const float4*>(&as[buf][k][ty * 4]), a1 = *reinterpret_cast<const float4*>(&as[buf][k][64 + ty * 4]);
            const float4 b0 = *reinterpret_cast<const float4*>(&bs[buf][k][tx * 4]), b1 = *reinterpret_cast<const float4*>(&bs[buf][k][64 + tx * 4]);
            const float av[8] = { a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w }, bv[8] = { b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w };
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[i][j] = it_add(acc[i][j], it_mul(av[i], bv[j]));
        }
        if (s + 1 < steps) store(buf ^ 1);          // read last before the barrier at the end of the step before this one
        __syncthreads();
    }
    const float scale = it_div(1.0f, it_sqrt((float)hd));
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int mi = m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + i - 4);
        if (mi >= nm) continue;
        float* o = scores + ((size_t)kvh * nm + mi) * b.npad + p0 + tx * 4;
        *reinterpret_cast<float4*>(o) = make_float4(it_mul(acc[i][0], scale), it_mul(acc[i][1], scale), it_mul(acc[i][2], scale), it_mul(acc[i][3], scale));
        *reinterpret_cast<float4*>(o + 64) = make_float4(it_mul(acc[i][4], scale), it_mul(acc[i][5], scale), it_mul(acc[i][6], scale), it_mul(acc[i][7], scale));
    }
}

// Softmax of 16 rows of scores in place.  The sum of a row's exponentials is one thread's ordered chain (4 cycles a term): warp 0
// runs the 16 chains side by side on one chunk of positions while the other seven warps form the exponentials of the next.
// Bounded by that chain at a few hundred positions and by its passes over the scores behind that.  24 heads of 256, 777 rows: 98 us
// with two integer divisions an element; 75 with a row's count formed once; 64 with chunks of 128, which let eight CTAs share an SM and
// 777 rows be one wave (chunks of 256: six CTAs), and the chain's terms loaded eight ahead.
constexpr int SM_ROWS = 16, SM_CHUNK = 128;
__global__ void __launch_bounds__(256) k_attn_softmax(float* scores, AtBlock b, int rows) {
    IT_PDL_TRIGGER(); IT_PDL_WAIT();
    __shared__ float e[2][SM_ROWS][SM_CHUNK + 1];
    __shared__ float mxs[SM_ROWS], sums[SM_ROWS];
    __shared__ int ns[SM_ROWS];                    // positions a row sees (itself included); the divisions once a row, not once an element
    const int r0 = blockIdx.x * SM_ROWS, nr = min(SM_ROWS, rows - r0), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid < SM_ROWS) ns[tid] = tid < nr ? b.slot0 + (r0 + tid) % (b.nt * b.rep) / b.rep + 1 : 0;
    __syncthreads();
    for (int r = warp; r < nr; r += 8) {
        const float* s = scores + (size_t)(r0 + r) * b.npad; const int n = ns[r];
        float m = -INFINITY;
#pragma unroll 4
        for (int p = lane; p < n; p += 32) m = fmaxf(m, s[p]);
#pragma unroll
        for (int k = 16; k >= 1; k >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, k));
        if (lane == 0) mxs[r] = m;
    }
    __syncthreads();
    int nmax = 0;
#pragma unroll
    for (int r = 0; r < SM_ROWS; r++) nmax = max(nmax, ns[r]);
    const int chunks = (nmax + SM_CHUNK - 1) / SM_CHUNK, myn = ns[lane % SM_ROWS];
    float sum = 0.f;
    for (int c = 0; c <= chunks; c++) {
        if (warp > 0 && c < chunks) {
#pragma unroll 4
            for (int i = tid - 32; i < SM_ROWS * SM_CHUNK; i += 224) {
                const int r = i / SM_CHUNK, j = i % SM_CHUNK, p = c * SM_CHUNK + j;
                if (p < ns[r]) { float* s = scores + (size_t)(r0 + r) * b.npad + p; const float v = it_expf(it_sub(*s, mxs[r])); *s = v; e[c & 1][r][j] = v; }
            }
        } else if (warp == 0 && c > 0 && lane < nr) {
            const int k = min(SM_CHUNK, myn - (c - 1) * SM_CHUNK); const float* ec = e[(c - 1) & 1][lane];
            int j = 0;
            float t[2][8];                         // the next eight are on their way while eight are added
            if (k >= 8)
#pragma unroll
                for (int u = 0; u < 8; u++) t[0][u] = ec[u];
            for (; j + 16 <= k; j += 16) {
#pragma unroll
                for (int u = 0; u < 8; u++) t[1][u] = ec[j + 8 + u];
#pragma unroll
                for (int u = 0; u < 8; u++) sum = it_add(sum, t[0][u]);
#pragma unroll
                for (int u = 0; u < 8; u++) t[0][u] = ec[min(j + 16, SM_CHUNK - 8) + u];
#pragma unroll
                for (int u = 0; u < 8; u++) sum = it_add(sum, t[1][u]);
            }
            if (j + 8 <= k) {
#pragma unroll
                for (int u = 0; u < 8; u++) sum = it_add(sum, t[0][u]);
                j += 8;
            }
            for (; j < k; j++) sum = it_add(sum, ec[j]);
        }
        __syncthreads();
    }
    if (warp == 0 && lane < nr) sums[lane] = sum;
    __syncthreads();
    for (int r = warp; r < nr; r += 8) {
        float* s = scores + (size_t)(r0 + r) * b.npad; const int n = ns[r]; const float d = sums[r];
#pragma unroll 4
        for (int p = lane; p < n; p += 32) s[p] = it_div(s[p], d);
    }
}

// out[t][head][j] = (sum over p of w[p] * v[p][j]) * sigmoid(gate).  128 threads, thread (ty, tx) owns rows ty * 4 + {0..3}, 64 + ..., elements
// tx * 4 + {0..3}, 32 + ...  Positions every row of the tile sees run unguarded; the few behind them are added row by row.
// CTAs start in the order of their length over all heads (777 rows: 592 CTAs, three to an SM; with the longest of one KV head after the shortest
// of another 264 us, now 187; the multiplies and adds alone are 101).
__global__ void __launch_bounds__(128, 3) k_attn_values(const float* __restrict__ w, const __half* __restrict__ vc, const float* gate, size_t q_hs, size_t q_ts, int hd, int nkv, AtBlock b,
                                                        float* out, size_t o_ts) {
    IT_PDL_TRIGGER(); IT_PDL_WAIT();
    __shared__ __align__(16) float as[2][AT_K][AT_M], bs[2][AT_K][AT_J];
    const int slices = hd / AT_J, slice = blockIdx.x % slices, kvh = blockIdx.x / slices, nm = b.nt * b.rep;
    const int m0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * AT_M;             // the longest rows of all heads first
    const int tid = threadIdx.x, ty = tid >> 3, tx = tid & 7;
    const int n_all = b.slot0 + m0 / b.rep + 1, n_any = b.slot0 + min(nm - 1, m0 + AT_M - 1) / b.rep + 1;    // positions seen by every / by some row of the tile
    const float* wp = w + ((size_t)kvh * nm + min(m0 + tid, nm - 1)) * b.npad;
    const int lp = tid >> 3, lc = tid & 7;
    float4 wa[4]; uint4 vv;
    auto fetch = [&](int s) {
#pragma unroll
        for (int i = 0; i < 4; i++) wa[i] = *reinterpret_cast<const float4*>(wp + s * AT_K + 4 * i);
        vv = *reinterpret_cast<const uint4*>(vc + it_vc_index((size_t)min(s * AT_K + lp, n_any - 1), kvh, slice * AT_J + lc * 8, nkv, hd));
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int i = 0; i < 4; i++) { as[buf][4 * i][tid] = wa[i].x; as[buf][4 * i + 1][tid] = wa[i].y; as[buf][4 * i + 2][tid] = wa[i].z; as[buf][4 * i + 3][tid] = wa[i].w; }
        float f[8]; at_half8(vv, f);
        *reinterpret_cast<float4*>(&bs[buf][lp][lc * 8]) = make_float4(f[0], f[1], f[2], f[3]);
        *reinterpret_cast<float4*>(&bs[buf][lp][lc * 8 + 4]) = make_float4(f[4], f[5], f[6], f[7]);
    };
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = 0.f;
    const int full = n_all / AT_K, steps = (n_any + AT_K - 1) / AT_K;
    fetch(0); store(0); __syncthreads();
    for (int s = 0; s < steps; s++) {
        const int buf = s & 1;
        if (s + 1 < steps) fetch(s + 1);
        if (s < full) {
#pragma unroll
            for (int k = 0; k < AT_K; k++) {
                const float4 a0 = *reinterpret_cast<const float4*>(&as[buf][k][ty * 4]), a1 = *reinterpret_cast<const float4*>(&as[buf][k][64 + ty * 4]);
                const float4 b0 = *reinterpret_cast<const float4*>(&bs[buf][k][tx * 4]), b1 = *reinterpret_cast<const float4*>(&bs[buf][k][32 + tx * 4]);
                const float av[8] = { a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w }, bv[8] = { b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w };
#pragma unroll
                for (int i = 0; i < 8; i++)
#pragma unroll
                    for (int j = 0; j < 8; j++) acc[i][j] = it_add(acc[i][j], it_mul(av[i], bv[j]));
            }
        } else {
            for (int k = 0; k < AT_K; k++) {
                const float4 b0 = *reinterpret_cast<const float4*>(&bs[buf][k][tx * 4]), b1 = *reinterpret_cast<const float4*>(&bs[buf][k][32 + tx * 4]);
                const float bv[8] = { b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w };
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const int r = i < 4 ? ty * 4 + i : 64 + ty * 4 + i - 4;
                    if (s * AT_K + k <= b.slot0 + (m0 + r) / b.rep) {          // row r sees this position
                        const float a = as[buf][k][r];
#pragma unroll
                        for (int j = 0; j < 8; j++) acc[i][j] = it_add(acc[i][j], it_mul(a, bv[j]));
                    }
                }
            }
        }
        if (s + 1 < steps) store(buf ^ 1);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int mi = m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + i - 4);
        if (mi >= nm) continue;
        const int t = mi / b.rep, h = kvh * b.rep + mi % b.rep;
#pragma unroll
        for (int jj = 0; jj < 2; jj++) {
            const int j = slice * AT_J + jj * 32 + tx * 4;
            const float4 gv = *reinterpret_cast<const float4*>(gate + (size_t)t * q_ts + (size_t)h * q_hs + j);
            *reinterpret_cast<float4*>(out + (size_t)t * o_ts + (size_t)h * hd + j) =
                make_float4(it_mul(acc[i][4 * jj], it_sigmoid(gv.x)), it_mul(acc[i][4 * jj + 1], it_sigmoid(gv.y)), it_mul(acc[i][4 * jj + 2], it_sigmoid(gv.z)), it_mul(acc[i][4 * jj + 3], it_sigmoid(gv.w)));
        }
    }
}

}  // namespace

// Same results as it_sup_attention for the rows of one pass at known positions.  scratch: scores of a block of rows; rows are taken in blocks
// that fit it.  Returns 1 (nothing launched) when the shape or the scratch does not suit: the caller then uses it_sup_attention_prefill.
int it_sup_attention_tiled(it_ctx* c, const float* q, size_t q_hs, size_t q_ts, const float* gate, const void* kc, const void* vc, int hd, int nh, int nkv, int slot0,
                           float* out, size_t o_ts, int nt, float* scratch, size_t scratch_floats, int choice) {
    if (choice == 0 || hd % 64 || nh % nkv || ((q_hs | q_ts | o_ts) & 3) || ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(out)) & 15)) return 1;
    const int rep = nh / nkv, npad = (slot0 + nt + AT_N - 1) / AT_N * AT_N;
    const size_t fit = scratch_floats / ((size_t)nh * npad);
    const int blk = (int)(fit < (size_t)nt ? fit : (size_t)nt);
    if (blk < 1 || (choice < 0 && !it_attn_takes_tiled(hd, nh, nkv, slot0, nt, blk, c->sm_count))) return 1;
    it_note_op(c);
    const int nblk = (nt + blk - 1) / blk, per = (nt + nblk - 1) / nblk;       // blocks of equal size
    for (int t0 = 0; t0 < nt; t0 += per) {
        AtBlock b; b.slot0 = slot0 + t0; b.nt = nt - t0 < per ? nt - t0 : per; b.rep = rep; b.npad = npad;
        const int nm = b.nt * rep, mt = (nm + AT_M - 1) / AT_M, pt = (b.slot0 + b.nt + AT_N - 1) / AT_N;
        it_pdl(k_attn_scores, dim3(pt, mt, nkv), dim3(256), 0, c->stream, q + (size_t)t0 * q_ts, q_hs, q_ts, (const __half*)kc, hd, nkv, b, scratch);
        it_pdl(k_attn_softmax, dim3((nm * nkv + SM_ROWS - 1) / SM_ROWS), dim3(256), 0, c->stream, scratch, b, nm * nkv);
        it_pdl(k_attn_values, dim3(hd / AT_J * nkv, mt), dim3(128), 0, c->stream, scratch, (const __half*)vc, gate + (size_t)t0 * q_ts, q_hs, q_ts, hd, nkv, b, out + (size_t)t0 * o_ts, o_ts);
        IT_LAUNCH_CHECK("attention_tiled");
    }
    return IT_OK;
}
