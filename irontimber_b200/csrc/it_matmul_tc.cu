// Ternary GEMM on q8k activations with the 5th-generation tensor cores: tcgen05.mma kind::i8, accumulators in tensor
// memory.  Same function and the same bits as k_matmul_t2 (it_matmul_t2.cu) and cpu::matvec's ternary arm
// (src/cpu.rs:48-63); it takes the place of the 64x64 tile kernels VkEngine::mv selects for prompt chunks
// (src/vk/mod.rs:655-677).
//
// A CTA owns 128 matrix rows (four 32-row groups) x 64 activation rows (x 128 when the launch has more than 64: one
// expanded tile and one issue sequence then feed twice the columns) and walks the 128-column blocks in order.
//   warp 24  producer: per block one stage = four weight tiles (bulk copies) + the 64 x 128 int8 activations as one
//            box of a tiled tensor map with the 128-byte swizzle, i.e. already in the K-major layout the MMA reads
//   warps 16-23 expanders (two sets of four, alternating blocks): turn the packed 2-bit codes of a stage into a 128 x 128 tile of unsigned bytes (codes 0..3)
//            in the same K-major 128-byte-swizzled layout (row r at 128 r, 16-byte piece p at (p ^ (r & 7)) * 16),
//            and the f16 block scales of the 128 rows into f32
//   warp 25  one thread issues four tcgen05.mma (M 128, N 64, K 32, u8 x s8 -> s32) per block into one of eight
//            64-column accumulators in tensor memory and commits them to mbarriers (accumulator ready; A tile and
//            stage free again)
//   warps 0-15 epilogue, four groups of four warps: group q owns activation rows 16 q .. 16 q + 15, its thread r reads
//            those columns of row r of the accumulator (tcgen05.ld 32x32b; warp w may touch lanes 32 (w % 4) ..), forms
//            (d_w * d_x) * float(S - sum128) for each and adds it to an f32 accumulator it keeps in registers for the
//            whole row of blocks: ascending block order, one thread per (row, activation row) pair - the CPU's order,
//            bit for bit.  The MMA of block b + 1 runs while block b is folded.
// Integer block sums are exact whatever the hardware's summation order, so only the f32 epilogue decides the bits.
//
// Every wait is bounded; when one runs out the CTA raises the context's error flag (IT_ETIMEOUT), every role leaves
// its loop, the producer waits (bounded) for its copies in flight, and the tensor memory is released before the CTA exits.
#include "it_internal.h"
#include "it_pipe.cuh"

namespace {

constexpr int TC_ROWS = 128;                     // matrix rows per CTA (M of the MMA)
constexpr int TC_A_BYTES = TC_ROWS * 128;        // one expanded weight tile
constexpr int TC_KB = 4;                         // blocks per weight stage: one bulk copy per row group and stage (issuing a bulk copy costs a
                                                 // thread some 250 cycles, so four small copies per block made the producer the bottleneck)
constexpr int TC_W_BYTES = 4 * TC_KB * IT_TILE_BYTES;   // four row groups x TC_KB consecutive tiles
constexpr int TC_NA = 2;                         // steps of expanded tiles in flight
constexpr int TC_SMEM_MAX = 226 * 1024;
constexpr unsigned TC_TMEM_COLS = 512;           // all of it: 2 * ND accumulators x TOK columns
constexpr int TC_EPI_WARPS = 8, TC_EXP_WARPS = 8, TC_THREADS = (TC_EPI_WARPS + TC_EXP_WARPS + 4) * 32;
// The launch's even share of registers (96 x 640 threads) is dealt out again: 168 x 256 + 48 x 384 = 61,440.
constexpr int TC_EPI_REGS = 168, TC_OTHER_REGS = 48;
// NH: 64-row halves of the CTA's activation tile.  NH = 1: 64 activation rows per CTA (prompt passes of up to 64 rows).
// NH = 2: 128 rows: one expanded weight tile and one issue sequence feed twice the columns.
template <int NH> struct Tc {
    static constexpr int TOK = 64 * NH;                  // activation rows per CTA (N of the MMA)
    static constexpr int X_BYTES = TOK * 128;            // the activation tile of one block: NH boxes of the tensor map, one under the other
    static constexpr int XS = NH == 1 ? 3 : 2;           // steps of activation tiles in flight (they come from L2)
    static constexpr int ND = 256 / TOK;                 // steps of accumulators in tensor memory
    static constexpr int EPI_TOK = TOK / 2;              // activation rows per epilogue warp
    static constexpr int CG = EPI_TOK / 8;               // 8-column groups per epilogue warp
    static constexpr int NDW = 2 * (TC_NA + ND);         // ring of per-block row scales: the expanders run at most NA + ND steps ahead of the epilogue
    // kind::i8 instruction descriptor: D s32, A signed 8 bit, B signed 8 bit, both K-major, N = TOK, M = 128
    static constexpr unsigned IDESC = (2u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(TOK >> 3) << 17) | ((unsigned)(TC_ROWS >> 4) << 24);
};

// Weight stages and activation boxes have rings of their own: the weights come from HBM, the boxes from L2.
struct TcSmem { int x, a, w, dx, dx_bytes, dw, bars, tmem, flag, total; };
template <int NH> __host__ __device__ inline TcSmem tc_layout(int nb, int wstages, int dxbufs) {
    TcSmem L; int o = 0;
    L.x = o; o += Tc<NH>::XS * 2 * Tc<NH>::X_BYTES;    // 1024-byte aligned (128-byte swizzle)
    L.a = o; o += TC_NA * 2 * TC_A_BYTES;              // 1024-byte aligned
    L.w = o; o += wstages * TC_W_BYTES;
    L.dx = o; L.dx_bytes = (nb / 2) * Tc<NH>::TOK * 4; o += dxbufs * L.dx_bytes;
    L.dw = o; o += Tc<NH>::NDW * TC_ROWS * 8;
    L.bars = o; o += (2 * wstages + Tc<NH>::XS + TC_NA + 2 * Tc<NH>::ND + 4) * 8;
    o = (o + 15) & ~15;
    L.tmem = o; o += 16;
    L.flag = o; o += 16;
    L.total = o;
    return L;
}

// K-major operand tile with 128-byte rows and the 128-byte swizzle: start address in 16-byte units, 8-row groups 1024
// bytes apart (stride byte offset), descriptor version 1, layout type 2 (128-byte swizzle).
__device__ __forceinline__ unsigned long long tc_smem_desc(unsigned addr) {
    return (unsigned long long)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((unsigned long long)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
template <bool ACC>
__device__ __forceinline__ void tc_mma(unsigned d_tmem, unsigned long long adesc, unsigned long long bdesc, unsigned idesc) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}"
                 :: "r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "n"(ACC ? 1 : 0), "r"(0u) : "memory");
}
__device__ __forceinline__ void tc_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar) : "memory");
}
// Accumulator read-out in the fragment shape 16x256b: of 16 lanes (matrix rows) x 32 columns (activation rows) thread 4 g + t gets, for
// each of the four column groups c, rows g and g + 8, columns 8 c + 2 t and 8 c + 2 t + 1.
__device__ __forceinline__ void tc_ld_frag(unsigned taddr, int (&v)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]),
                   "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(taddr) : "memory");
}
// Waits for the loads; the values pass through it so that nothing that uses them moves in front.
__device__ __forceinline__ void tc_ld_wait(int (&v)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]),
                   "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]) :: "memory");
}
__device__ __forceinline__ void mbar_arrive_n(unsigned bar, unsigned n) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(n) : "memory"); }

// Two values per instruction; every lane of the pair is rounded as the scalar instruction rounds it.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk(unsigned lo, unsigned hi) { f32x2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi)); return r; }
__device__ __forceinline__ f32x2 pkf(float lo, float hi) { return pk(__float_as_uint(lo), __float_as_uint(hi)); }
__device__ __forceinline__ float2 upk(f32x2 v) { unsigned a, b; asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(v)); return make_float2(__uint_as_float(a), __uint_as_float(b)); }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) { f32x2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
// A product that an addition follows.  The assembler joins mul.rn.f32x2 and add.rn.f32x2 into one fused operation (the scalar
// forms with .rn it leaves alone; -fmad=false changes nothing), which drops the rounding of the product.  a * b + (-0.0) rounds
// once, to the rounded product with its sign of zero, and an addition cannot be joined to it; mz is a launch argument so that
// the constant is not known at compile time.
__device__ __forceinline__ f32x2 mul2_rounded(f32x2 a, f32x2 b, f32x2 mz) { f32x2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(mz)); return r; }

// Place of activation row m's scale inside a step's TOK of them: the 2 * CG rows of one epilogue thread (8 c + 2 t + e) lie side by side.
template <int NH> __device__ __forceinline__ int tc_dx_slot(int m) {
    constexpr int E = Tc<NH>::EPI_TOK;
    return m / E * E + ((m & 7) >> 1) * (E / 4) + 2 * ((m % E) >> 3) + (m & 1);
}
template <int N> __device__ __forceinline__ void reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" :: "n"(N)); }
template <int N> __device__ __forceinline__ void reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" :: "n"(N)); }

template <int NH>
__global__ void __launch_bounds__(TC_THREADS, 1)
k_matmul_tc(const __grid_constant__ CUtensorMap xmap, const uint8_t* __restrict__ tiles, int nb, int rows, int row_groups, int wstages, int ntiles, int tok_tiles, int dxbufs,
            const float* __restrict__ xd, int x_stride, int ntok,
            float* arena, size_t y_off, size_t y_stride, int accum, int* error_flag, const it_peers* peers, const it_rowmap map, float minus_zero) {
    constexpr int TC_TOK = Tc<NH>::TOK, TC_X_BYTES = Tc<NH>::X_BYTES, TC_XS = Tc<NH>::XS, TC_ND = Tc<NH>::ND, TC_EPI_TOK = Tc<NH>::EPI_TOK, CG = Tc<NH>::CG, NDW = Tc<NH>::NDW;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const TcSmem L = tc_layout<NH>(nb, wstages, dxbufs);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, np = nb / 2;      // np: steps (pairs of blocks) of a tile
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L.flag);
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(smem + L.tmem);
    const unsigned bars = smem_u32(smem + L.bars);
    // barrier addresses: weight stages (full / empty), activation boxes of a step landed, tiles of a step expanded, accumulators of a
    // step (full / empty), activation scales (full / empty).  "Accumulators d full" is the one commit of a step: it also tells the
    // expanders and the activation producer that the tiles and boxes the step read may be reused.
    const unsigned wfull0 = bars, wempty0 = wfull0 + 8 * wstages, xfull0 = wempty0 + 8 * wstages,
                   afull0 = xfull0 + 8 * TC_XS, dfull0 = afull0 + 8 * TC_NA, dempty0 = dfull0 + 8 * TC_ND, sfull0 = dempty0 + 8 * TC_ND, sempty0 = sfull0 + 16;
    // The CTA's tiles: blockIdx.x, + gridDim.x, ...; the activation tiles of one group of matrix rows are neighbours.  Every role walks
    // the same tiles with its ring positions running on, so the next tile's weights, boxes and products are under way while
    // the epilogue still stores the last one's results.
    const int tile0 = (int)blockIdx.x, tstep = (int)gridDim.x;

    if (tid == 0) {
        *abort_flag = 0;
        for (int s = 0; s < wstages; s++) { mbar_init(wfull0 + 8 * s, 1); mbar_init(wempty0 + 8 * s, 8); }
        for (int s = 0; s < TC_XS; s++) mbar_init(xfull0 + 8 * s, 1);
        for (int a = 0; a < TC_NA; a++) mbar_init(afull0 + 8 * a, 4);
        for (int d = 0; d < TC_ND; d++) { mbar_init(dfull0 + 8 * d, 1); mbar_init(dempty0 + 8 * d, TC_EPI_WARPS); }
        for (int k = 0; k < 2; k++) { mbar_init(sfull0 + 8 * k, 1); mbar_init(sempty0 + 8 * k, TC_EPI_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {   // tensor memory for the accumulators
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(tmem_slot)), "r"(TC_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem_base = *tmem_slot;

    if (warp >= TC_EPI_WARPS) reg_dec<TC_OTHER_REGS>();
    if (warp == TC_EPI_WARPS + TC_EXP_WARPS) {
        // ---------------- weight producer: the weights depend on no earlier kernel, so it neither waits for one nor triggers.
        // Lane i < 4 copies the TC_KB consecutive tiles of row group i; lane 0 announces the bytes of the stage first.
        const int nst = (nb + TC_KB - 1) / TC_KB;
        int s = 0, issued = 0; unsigned ph = 0; bool ok = true;
        for (int tile = tile0; ok && tile < ntiles; tile += tstep) {
            const int rg0 = tile / tok_tiles * 4, nrg = min(4, row_groups - rg0);
            for (int q = 0; q < nst; q++) {
                if (lane == 0) ok = mbar_wait(wempty0 + 8 * s, ph ^ 1u, abort_flag, error_flag, 11);
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (!ok) break;
                const int kb = min(TC_KB, nb - q * TC_KB);
                unsigned char* st = smem + L.w + s * TC_W_BYTES;
                if (lane == 0) mbar_expect_tx(wfull0 + 8 * s, (unsigned)(nrg * kb * IT_TILE_BYTES));
                __syncwarp();
                if (lane < nrg) bulk_load(smem_u32(st + lane * TC_KB * IT_TILE_BYTES), tiles + ((size_t)(rg0 + lane) * nb + (size_t)q * TC_KB) * IT_TILE_BYTES,
                                          (unsigned)(kb * IT_TILE_BYTES), wfull0 + 8 * s);
                issued++;
                if (++s == wstages) { s = 0; ph ^= 1u; }
            }
        }
        if (*abort_flag && lane == 0) {   // leave only after every copy this warp started has landed (bounded)
            const int first = issued > wstages ? issued - wstages : 0;
            for (int k = first; k < issued; k++) {
                const long long t0 = clock64();
                while (!mbar_test(wfull0 + 8 * (k % wstages), (unsigned)(k / wstages) & 1u) && clock64() - t0 < WAIT_CLOCKS) { }
            }
        }
    } else if (warp == TC_EPI_WARPS + TC_EXP_WARPS + 2) {
        // ---------------- activation producer: the rows come from the kernel before this one
        if (lane == 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            int s = 0, issued = 0, dp = 0; unsigned dpp = 0; bool ok = true;
            for (int tile = tile0; ok && tile < ntiles; tile += tstep) {
                const int tok0 = tile % tok_tiles * TC_TOK;
                for (int p = 0; p < np; p++) {
                    // the slot was last read TC_XS steps ago: wait for that step's commit
                    if (issued >= TC_XS) {
                        if (!mbar_wait(dfull0 + 8 * dp, dpp, abort_flag, error_flag, 19)) { ok = false; break; }
                        if (++dp == TC_ND) { dp = 0; dpp ^= 1u; }
                    }
                    mbar_expect_tx(xfull0 + 8 * s, (unsigned)(2 * TC_X_BYTES));
#pragma unroll
                    for (int k = 0; k < 2 * NH; k++)     // 64 rows per box; the boxes of a block lie one under the other like one box of TOK rows
                        tma_load_2d(smem_u32(smem + L.x + s * 2 * TC_X_BYTES + k * 64 * 128), &xmap, (2 * p + k / NH) * 128, tok0 + 64 * (k % NH), xfull0 + 8 * s);
                    issued++;
                    if (++s == TC_XS) s = 0;
                }
            }
            if (*abort_flag) {
                const int first = issued > TC_XS ? issued - TC_XS : 0;
                for (int k = first; k < issued; k++) {
                    const long long t0 = clock64();
                    while (!mbar_test(xfull0 + 8 * (k % TC_XS), (unsigned)(k / TC_XS) & 1u) && clock64() - t0 < WAIT_CLOCKS) { }
                }
            }
        }
    } else if (warp == TC_EPI_WARPS + TC_EXP_WARPS + 1) {
        // ---------------- MMA issuer
        if (lane == 0) {
            int s = 0, a = 0, d = 0; unsigned xph = 0, aph = 0, dph = 0; bool ok = true;
            const unsigned long long adesc0 = tc_smem_desc(smem_u32(smem + L.a)), bdesc0 = tc_smem_desc(smem_u32(smem + L.x));
            for (int tile = tile0; ok && tile < ntiles; tile += tstep)
            for (int p = 0; p < np; p++) {
                // accumulators read out; boxes landed; tiles expanded (the condition that is met last)
                if (!mbar_wait(dempty0 + 8 * d, dph ^ 1u, abort_flag, error_flag, 14) || !mbar_wait(xfull0 + 8 * s, xph, abort_flag, error_flag, 13) ||
                    !mbar_wait(afull0 + 8 * a, aph, abort_flag, error_flag, 12)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                // descriptors differ from the first tile's only in the start-address field (16-byte units): + tile index, + 2 per K step of 32
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const unsigned long long ad = adesc0 + (unsigned)((2 * a + h) * (TC_A_BYTES >> 4)), bd = bdesc0 + (unsigned)((2 * s + h) * (TC_X_BYTES >> 4));
                    const unsigned dt = tmem_base + (unsigned)((2 * d + h) * TC_TOK);
                    tc_mma<false>(dt, ad, bd, Tc<NH>::IDESC);
                    tc_mma<true>(dt, ad + 2, bd + 2, Tc<NH>::IDESC);
                    tc_mma<true>(dt, ad + 4, bd + 4, Tc<NH>::IDESC);
                    tc_mma<true>(dt, ad + 6, bd + 6, Tc<NH>::IDESC);
                }
                tc_commit(dfull0 + 8 * d);        // accumulators complete; tiles and boxes of this step may be reused
                if (++s == TC_XS) { s = 0; xph ^= 1u; }
                if (++a == TC_NA) { a = 0; aph ^= 1u; }
                if (++d == TC_ND) { d = 0; dph ^= 1u; }
            }
        }
    } else if (warp == TC_EPI_WARPS + TC_EXP_WARPS + 3) {
        // ---------------- activation scales of every tile but the first (which the epilogue warps fetch together), one tile ahead
        asm volatile("griddepcontrol.wait;" ::: "memory");
        int j = 1;                                                    // the CTA's j-th tile uses buffer j % 2
        for (int tile = tile0 + tstep; tile < ntiles; tile += tstep, j++) {
            const int k = j & 1;
            const int tok0 = tile % tok_tiles * TC_TOK, ntv = min(TC_TOK, ntok - tok0);
            const bool ok = mbar_wait(sempty0 + 8 * k, ((unsigned)(j >> 1) & 1u) ^ 1u, abort_flag, error_flag, 20);     // tile j - 2 is done with it
            if (!__all_sync(0xffffffffu, ok)) break;
            float* dxs = reinterpret_cast<float*>(smem + L.dx + k * L.dx_bytes);
            for (int m = lane; m < TC_TOK; m += 32) {
                const float* src = xd + (size_t)(tok0 + m) * (x_stride / 256);
                float* dst = dxs + tc_dx_slot<NH>(m);
#pragma unroll 8
                for (int bb = 0; bb < np; bb++) dst[bb * TC_TOK] = m < ntv ? src[bb] : 0.f;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(sfull0 + 8 * k);
        }
    } else if (warp >= TC_EPI_WARPS) {
        // ---------------- expanders: warp 8 + 4 e + i expands row group i of the steps with number % 2 == e into tile pair e
        static_assert(TC_NA == 2 && TC_EXP_WARPS == 8, "set e fills tile pair e");
        const int eset = (warp - TC_EPI_WARPS) >> 2, rgl = (warp - TC_EPI_WARPS) & 3, g = lane >> 2, t = lane & 3;
        unsigned char* const at = smem + L.a + 2 * eset * TC_A_BYTES + (rgl * 32 + g) * 128;
        unsigned char* const plo = at + (((2 * t) ^ g) << 4);          // columns 32 t .. 32 t + 15 of row g; the other rows 1024 bytes apart
        unsigned char* const phi = at + (((2 * t + 1) ^ g) << 4);      // columns 32 t + 16 .. 32 t + 31
        float* const dws = reinterpret_cast<float*>(smem + L.dw) + rgl * 64 + 8 * g;
        const unsigned char* const src0 = smem + L.w + rgl * TC_KB * IT_TILE_BYTES;
        int s = 0, dp = eset, r = 0, gp = 0; unsigned sph = 0, dpp = 0; bool ok = true;
        for (int tile = tile0; ok && tile < ntiles; tile += tstep)
        for (int p = 0; p < np; p++, gp++) {
            const bool last = (p & 1) || p + 1 == np;         // last step of the weight stage
            if ((gp & 1) == eset) {
                if (!mbar_wait(wfull0 + 8 * s, sph, abort_flag, error_flag, 15)) { ok = false; break; }
                // the tile pair was last read two steps ago: wait for that step's commit
                if (gp >= 2) {
                    if (!mbar_wait(dfull0 + 8 * dp, dpp, abort_flag, error_flag, 16)) { ok = false; break; }
                    dp += 2;
                    if (dp >= TC_ND) { dp -= TC_ND; dpp ^= 1u; }
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const unsigned char* src = src0 + s * TC_W_BYTES + (2 * (p & 1) + h) * IT_TILE_BYTES;
                    const uint4 wa = *reinterpret_cast<const uint4*>(src + 16 * lane);
                    const uint4 wb = *reinterpret_cast<const uint4*>(src + 512 + 16 * lane);
#pragma unroll
                    for (int i = 0; i < 4; i++) {         // bit pair i of every byte: matrix row g + 8 i of the group
                        auto sgn = [&](unsigned w) { return (((w >> (2 * i)) & 0x03030303u) + 0x7f7f7f7fu) ^ 0x80808080u; };   // code - 1 in every byte; no carry crosses a byte
                        *reinterpret_cast<uint4*>(plo + h * TC_A_BYTES + i * 1024) = make_uint4(sgn(wa.x), sgn(wa.y), sgn(wa.z), sgn(wa.w));
                        *reinterpret_cast<uint4*>(phi + h * TC_A_BYTES + i * 1024) = make_uint4(sgn(wb.x), sgn(wb.y), sgn(wb.z), sgn(wb.w));
                    }
                    if (t == 0) {                         // row scales, each one twice (the operand pair of the epilogue's two-value products)
                        const uint2 sc = *reinterpret_cast<const uint2*>(src + 1024 + 8 * g);
                        const __half2 h01 = *reinterpret_cast<const __half2*>(&sc.x), h23 = *reinterpret_cast<const __half2*>(&sc.y);
                        const float d0 = __low2float(h01), d1 = __high2float(h01), d2 = __low2float(h23), d3 = __high2float(h23);
                        float4* dw = reinterpret_cast<float4*>(dws + (r + h) * 2 * TC_ROWS);
                        dw[0] = make_float4(d0, d0, d1, d1); dw[1] = make_float4(d2, d2, d3, d3);      // rows g, g + 8, g + 16, g + 24: the rows of one epilogue thread
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // generic-proxy stores before the MMA's async-proxy reads
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(afull0 + 8 * eset);
                    mbar_arrive_n(wempty0 + 8 * s, last && !(p & 1) ? 2u : 1u);  // read its tiles; a stage of one step counts them twice
                }
            }
            r = r + 2 == NDW ? 0 : r + 2;
            if (last) { if (++s == wstages) { s = 0; sph ^= 1u; } }
        }
    } else {
        // ---------------- epilogue: warp 4 q + i owns row group i x activation rows EPI_TOK q ..; its thread 4 g + t owns rows
        // g, g + 8, g + 16, g + 24 of the group and, of every eight activation rows, the two at 2 t.  Two 16-byte loads of row
        // scales and EPI_TOK / 16 of activation scales then serve EPI_TOK results per block: with a row per thread and all columns
        // (one broadcast 16-byte load per four results) the shared-memory read port was what bounded the kernel.
        constexpr int NEPI = TC_EPI_WARPS * 32;
        reg_inc<TC_EPI_REGS>();
        const int grp = warp >> 2, rgl = warp & 3, g = lane >> 2, t = lane & 3, m0 = grp * TC_EPI_TOK;
        const unsigned tquad = tmem_base + ((unsigned)(rgl * 32) << 16) + (unsigned)m0;
        const ulonglong2* const dws = reinterpret_cast<const ulonglong2*>(smem + L.dw) + rgl * 16 + 2 * g;
        asm volatile("griddepcontrol.wait;" ::: "memory");            // q8 scales and (when accumulating) y come from earlier kernels
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        {
            float* dxs = reinterpret_cast<float*>(smem + L.dx);
            const int tok0 = tile0 % tok_tiles * TC_TOK, ntv = min(TC_TOK, ntok - tok0);
#pragma unroll 4
            for (int i = tid; i < np * TC_TOK; i += NEPI) {
                const int m = i % TC_TOK, bb = i / TC_TOK;
                dxs[bb * TC_TOK + tc_dx_slot<NH>(m)] = m < ntv ? xd[(size_t)(tok0 + m) * (x_stride / 256) + bb] : 0.f;
            }
            asm volatile("bar.sync 1, %0;" :: "n"(NEPI) : "memory");
        }
        const f32x2 mz = pkf(minus_zero, minus_zero);
        int d = 0, r = 0, j = 0; unsigned dph = 0;
        bool ok = true;
        for (int tile = tile0; tile < ntiles; tile += tstep, j++) {
            const int k = j & 1;
            const int rg0 = tile / tok_tiles * 4, tok0 = tile % tok_tiles * TC_TOK, ntv = min(TC_TOK, ntok - tok0);
            const bool active = m0 < ntv;              // groups past the last activation row only release the accumulators
            if (j > 0 && !mbar_wait(sfull0 + 8 * k, (unsigned)((j - 1) >> 1) & 1u, abort_flag, error_flag, 18)) break;
            const ulonglong2* dx2 = reinterpret_cast<const ulonglong2*>(smem + L.dx + k * L.dx_bytes + (m0 + t * 2 * CG) * 4);
            f32x2 acc[4][CG];                          // [row g + 8 i][column pair of group c]
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int c = 0; c < CG; c++) acc[i][c] = 0ull;
            for (int p = 0; p < np; p++) {             // two blocks at a time: they share the activation scale, the wait and the release
                if (!mbar_wait(dfull0 + 8 * d, dph, abort_flag, error_flag, 17)) { ok = false; break; }
                __syncwarp();
                if (active) {
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    // chunks of 16 lanes x 32 columns; the next one is on its way while one is folded
                    constexpr int NCC = CG / 4, NCH = 4 * NCC;
                    const unsigned ta = tquad + (unsigned)(2 * d * TC_TOK);
                    auto chunk = [&](int ch) { return ta + (unsigned)(ch / (2 * NCC) * TC_TOK) + ((unsigned)(ch / NCC % 2) << 20) + (unsigned)(32 * (ch % NCC)); };
                    int S[2][16];
                    tc_ld_frag(chunk(0), S[0]);
                    f32x2 dx[CG];
#pragma unroll
                    for (int c = 0; c < CG / 2; c++) { const ulonglong2 v = dx2[c]; dx[2 * c] = v.x; dx[2 * c + 1] = v.y; }
                    ulonglong2 dw[2];
#pragma unroll
                    for (int ch = 0; ch < NCH; ch++) {
                        const int h = ch / (2 * NCC), hf = ch / NCC % 2, cc = ch % NCC;
                        // row scales of this block: stored by the expanders before they released the tile to the MMA whose completion we just saw
                        if (ch % (2 * NCC) == 0) { dw[0] = dws[(r + h) * TC_ROWS / 2]; dw[1] = dws[(r + h) * TC_ROWS / 2 + 1]; }
                        int (&v)[16] = S[ch & 1];
                        tc_ld_wait(v);
                        if (ch + 1 < NCH) tc_ld_frag(chunk(ch + 1), S[(ch + 1) & 1]);
                        else {
                            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                            __syncwarp();
                            if (lane == 0) mbar_arrive(dempty0 + 8 * d);      // the MMAs of step p + ND may use the accumulators
                        }
#pragma unroll
                        for (int c = 0; c < 4; c++) {
                            f32x2 (&a0)[CG] = acc[2 * hf], (&a1)[CG] = acc[2 * hf + 1];
                            const f32x2 x = dx[4 * cc + c];
                            a0[4 * cc + c] = add2(a0[4 * cc + c], mul2_rounded(mul2(dw[hf].x, x), pkf((float)v[4 * c], (float)v[4 * c + 1]), mz));
                            a1[4 * cc + c] = add2(a1[4 * cc + c], mul2_rounded(mul2(dw[hf].y, x), pkf((float)v[4 * c + 2], (float)v[4 * c + 3]), mz));
                        }
                    }
                } else if (lane == 0) mbar_arrive(dempty0 + 8 * d);
                dx2 += TC_TOK / 4;
                if (++d == TC_ND) { d = 0; dph ^= 1u; }
                r = r + 2 == NDW ? 0 : r + 2;
            }
            if (!ok || *abort_flag) break;
            __syncwarp();
            if (lane == 0) mbar_arrive(sempty0 + 8 * k);          // the tile's activation scales have been read
            if (!active) continue;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int row = (rg0 + rgl) * 32 + g + 8 * i;
                if (row >= rows) continue;
                const int grow = it_map_row(map, row);
                const size_t off = y_off + (size_t)(tok0 + m0 + 2 * t) * y_stride + grow;     // first of this thread's activation rows
                if (!peers) {
                    float* y = arena + off;
                    float old[2 * CG];
#pragma unroll
                    for (int c = 0; c < CG; c++)
#pragma unroll
                        for (int e = 0; e < 2; e++) old[2 * c + e] = accum && m0 + 8 * c + 2 * t + e < ntv ? __ldcg(y + (size_t)(8 * c + e) * y_stride) : 0.f;
#pragma unroll
                    for (int c = 0; c < CG; c++) {
                        const float2 v = upk(acc[i][c]);
                        const int m = m0 + 8 * c + 2 * t;
                        if (m < ntv) y[(size_t)(8 * c) * y_stride] = accum ? __fadd_rn(old[2 * c], v.x) : v.x;
                        if (m + 1 < ntv) y[(size_t)(8 * c + 1) * y_stride] = accum ? __fadd_rn(old[2 * c + 1], v.y) : v.y;
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < CG; c++) {
                        const float2 v = upk(acc[i][c]);
                        const int m = m0 + 8 * c + 2 * t;
                        if (m < ntv) it_result_store(peers, arena, off + (size_t)(8 * c) * y_stride, v.x, accum);
                        if (m + 1 < ntv) it_result_store(peers, arena, off + (size_t)(8 * c + 1) * y_stride, v.y, accum);
                    }
                }
            }
        }
        if (peers) __threadfence_system();
    }
    // ---------------- common end: every role arrives here, also after a wait that ran out
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(TC_TMEM_COLS) : "memory");
    }
    if (peers && tid == 0) it_shard_finish(peers, gridDim.x, error_flag);
}

}  // namespace

template <int NH>
static int tc_launch(it_ctx* c, const it_mat* w, int ntok, const it_q8* x, float* y, size_t y_stride, int accum) {
    const int nb = (int)(w->cols / 128);
    const int tok_tiles = (ntok + Tc<NH>::TOK - 1) / Tc<NH>::TOK, ntiles = (int)((w->row_groups + 3) / 4) * tok_tiles;
    // one CTA per SM walks its tiles, with two buffers of activation scales; where those do not fit (wide rows), a CTA per tile
    int grid = ntiles < c->sm_count ? ntiles : c->sm_count, dxbufs = ntiles > grid ? 2 : 1;
    if (tc_layout<NH>(nb, 2, dxbufs).total + 1024 > TC_SMEM_MAX) { grid = ntiles; dxbufs = 1; }
    int stages = 5;                        // weight stages of TC_KB blocks: as deep as shared memory allows
    while (stages > 2 && tc_layout<NH>(nb, stages, dxbufs).total + 1024 > TC_SMEM_MAX) stages--;
    const TcSmem L = tc_layout<NH>(nb, stages, dxbufs);
    if (L.total + 1024 > TC_SMEM_MAX) return 1;
    static bool attr_set[16] = {};
    if (!attr_set[c->device & 15]) { IT_CUDA(cudaFuncSetAttribute(k_matmul_tc<NH>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM_MAX)); attr_set[c->device & 15] = true; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(TC_THREADS); cfg.dynamicSmemBytes = (size_t)L.total + 1024; cfg.stream = c->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    IT_CUDA(cudaLaunchKernelEx(&cfg, k_matmul_tc<NH>, x->tmap, (const uint8_t*)w->tiles, nb, (int)w->rows, (int)w->row_groups, stages, ntiles, tok_tiles, dxbufs,
        (const float*)x->d, (int)x->max_n, ntok, c->arena, (size_t)(y - c->arena), y_stride, accum, c->error_flag_dev,
        (const it_peers*)(w->sharded ? c->peers_dev : nullptr), w->map, -0.0f));
    c->pdl_safe_q8 = x;
    return IT_OK;
}

// Returns IT_OK after launching, or a positive value when the shape does not suit this kernel (the caller then uses k_matmul_t2).
// More than 64 activation rows go to the 128-row variant when its buffers fit (rows of up to about 12,000 columns).
int it_matmul_tc_launch(it_ctx* c, const it_mat* w, int ntok, const it_q8* x, float* y, size_t y_stride, int accum) {
    static const bool wide = []{ const char* v = getenv("IT_MATMUL_WIDE"); return !v || atoi(v) != 0; }();
    if (wide && ntok > 64) { const int r = tc_launch<2>(c, w, ntok, x, y, y_stride, accum); if (r != 1) return r; }
    return tc_launch<1>(c, w, ntok, x, y, y_stride, accum);
}
