// Ternary GEMM on q8k activations with the 5th-generation tensor cores: tcgen05.mma kind::i8, accumulators in tensor
// memory.  Same function and the same bits as k_matmul_t2 (it_matmul_t2.cu) and cpu::matvec's ternary arm
// (src/cpu.rs:48-63); it takes the place of the 64x64 tile kernels VkEngine::mv selects for prompt chunks
// (src/vk/mod.rs:655-677).
//
// A CTA walks tiles of 128 matrix rows (four 32-row groups; two, where that gives idle SMs a tile) x 64 activation rows (x 128 in larger
// launches: one expanded tile and one issue sequence then feed twice the columns); one CTA per SM, a tile's 128-column blocks in order, two
// blocks (the 256 columns of a q8k scale) a step.
//   warp 16  weight producer: per stage four weight tiles of each of the four row groups (bulk copies)
//   warp 18  activation producer: per step the int8 activations as boxes of a tiled tensor map with the 128-byte swizzle,
//            i.e. already in the K-major layout the MMA reads
//   warps 8-15 expanders (two sets of four, alternating steps): turn the packed 2-bit codes into 128 x 128 tiles of signed bytes
//            code - 1 in the same K-major 128-byte-swizzled layout (row r at 128 r, 16-byte piece p at (p ^ (r & 7)) * 16), so that
//            the accumulator is S - sum128 at once, and the f16 block scales of the 128 rows into f32
//   warp 17  one thread issues eight tcgen05.mma (M 128, K 32, s8 x s8 -> s32) per step into the step's two accumulators in tensor
//            memory and commits them to one mbarrier (accumulators ready; tiles and boxes free again)
//   warp 19  fetches the next tile's activation scales
//   warps 0-7 epilogue: reads the accumulators (a thread gets four rows x every fourth column), forms
//            (d_w * d_x) * float(S - sum128) for each and adds it to an f32 accumulator it keeps in registers for the
//            whole row of blocks: ascending block order, one thread per (row, activation row) pair - the CPU's order, bit for bit.
// What bounds it: per block and SM sub-core the epilogue's 64 pairs of values cost about 6.5 cycles each (conversion, two products, one
// addition, every one rounded; a two-value instruction takes two cycles of the f32 pipe) = 420 cycles, the MMAs 256 plus their
// operands' share of the shared-memory port; with everything running a block takes 740 cycles at 64 activation rows and 970 at 128
// (the epilogue alone 510 and 810, the expanders alone 530 and 660: the roles share the issue slots of their sub-core).  What the steps
// gave, 34816 x 5120 x 512 rows: 310 us with a row per epilogue thread (256 broadcast loads of scales a block: 1024 cycles of the
// shared-memory port); 251 with the fragment layout and two-value arithmetic; 242 with conversions instead of biased accumulators; 217 with
// CTAs that walk several tiles (7 us of 31 per tile were fill and drain); 202 with two blocks a step and eight epilogue warps; 197 with
// the 16x128b read-out; 180 with an issuer whose descriptors stay in uniform registers (elect.sync) and whose three waits a step are one look
// ahead, taken over from the expanders' loop (5120 x 17408 x 64 rows: 59.6 us before, 52.2 now).  What gave nothing: 16 epilogue warps
// of half the columns, the next step's accumulators on their way across steps, conversions by addition of 1.5 x 2^23.
// Integer block sums are exact whatever the hardware's summation order, so only the f32 epilogue decides the bits.
//
// Every wait is bounded; when one runs out the CTA raises the context's error flag (IT_ETIMEOUT), every role leaves
// its loop (expanders and epilogue by going on without waits or arrivals, the epilogue to the end of its tile and without storing
// it: a lane that left alone would leave the rest of its warp in a warp-wide instruction), the producer waits (bounded) for its copies in flight, and the tensor memory is released before the CTA exits.
#include "it_internal.h"
#include "it_pipe.cuh"
#include "it_route.h"

namespace {

constexpr int TC_KB = 4;                         // blocks per weight stage: one bulk copy per row group and stage (issuing a bulk copy costs a
                                                 // thread some 250 cycles, so four small copies per block made the producer the bottleneck)
constexpr int TC_NA_MAX = 3;                     // steps of expanded tiles in flight where they fit, else two: with two, an expander waits for the commit of its
                                                 // own last step and the chain commit - expand - issue - commit sets the pace (14336 x 5120 x 64: 19.9 us, with three 19.2)
constexpr int TC_NC = 4;                         // barriers the steps commit to in turn; at least the steps of boxes in flight, see the barrier list
constexpr int TC_SMEM_MAX = 226 * 1024;
constexpr unsigned TC_TMEM_COLS = 512;           // all of it: 2 * ND accumulators x TOK columns
constexpr int TC_EPI_WARPS = 8, TC_EXP_WARPS = 8, TC_THREADS = (TC_EPI_WARPS + TC_EXP_WARPS + 4) * 32;
// The launch's even share of registers (96 x 640 threads) is dealt out again: 168 x 256 + 48 x 384 = 61,440.
constexpr int TC_EPI_REGS = 168, TC_OTHER_REGS = 48;
// NH: 64-row halves of the CTA's activation tile.  NH = 1: 64 activation rows per CTA (prompt passes of up to 64 rows).
// NH = 2: 128 rows: one expanded weight tile and one issue sequence feed twice the columns.
// RG: row groups of the CTA's weight tile.  RG = 4: 128 matrix rows.  RG = 2: 64 rows, where that gives idle SMs a tile: every warp then has
// half of a step's work (an expander one block of a row group, an epilogue warp 16 rows).
template <int NH, int RG> struct Tc {
    static constexpr int ROWS = 32 * RG;                 // matrix rows per CTA (M of the MMA)
    static constexpr int A_BYTES = ROWS * 128;           // one expanded weight tile
    static constexpr int W_BYTES = RG * TC_KB * IT_TILE_BYTES;   // RG row groups x TC_KB consecutive tiles
    static constexpr int TOK = 64 * NH;                  // activation rows per CTA (N of the MMA)
    static constexpr int X_BYTES = TOK * 128;            // the activation tile of one block: NH boxes of the tensor map, one under the other
    static constexpr int ND = 256 / TOK;                 // steps of accumulators in tensor memory
    static constexpr int EPI_TOK = TOK / 2;              // activation rows per epilogue warp
    static constexpr int CC = EPI_TOK / 32;              // 32-column chunks per epilogue warp
    static constexpr int NDW = 2 * (TC_NA_MAX + ND);     // ring of per-block row scales: the expanders run at most NA + ND steps ahead of the epilogue
    // kind::i8 instruction descriptor: D s32, A signed 8 bit, B signed 8 bit, both K-major, N = TOK, M = ROWS
    static constexpr unsigned IDESC = (2u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(TOK >> 3) << 17) | ((unsigned)(ROWS >> 4) << 24);
};

// Weight stages and activation boxes have rings of their own: the weights come from HBM, the boxes from L2.
struct TcSmem { int x, a, w, dx, dx_bytes, dw, bars, tmem, flag, total; };
template <int NH, int RG> __host__ __device__ inline TcSmem tc_layout(int nb, int wstages, int dxbufs, int xsteps, int na) {
    using T = Tc<NH, RG>;
    TcSmem L; int o = 0;
    L.x = o; o += xsteps * 2 * T::X_BYTES;    // 1024-byte aligned (128-byte swizzle)
    L.a = o; o += na * 2 * T::A_BYTES;              // 1024-byte aligned
    L.w = o; o += wstages * T::W_BYTES;
    L.dx = o; L.dx_bytes = (nb / 2) * T::TOK * 4; o += dxbufs * L.dx_bytes;
    L.dw = o; o += T::NDW * T::ROWS * 4;
    L.bars = o; o += (2 * wstages + xsteps + na + TC_NC + T::ND + 4) * 8;
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
// One lane of the warp, chosen by the hardware's own instruction: the compiler then knows that what follows runs once, and keeps descriptors
// and barrier addresses in the warp's uniform registers (under `lane == 0` it moved them there for every instruction).
__device__ __forceinline__ bool tc_elect() {
    unsigned e;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(e));
    return e != 0;
}
// Non-blocking probe of three phases at once: their answers are under way together.
__device__ __forceinline__ bool mbar_poll3(unsigned a, unsigned pa, unsigned b, unsigned pb, unsigned c, unsigned pc) {
    unsigned ok;
    asm volatile("{\n.reg .pred p, q, r;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nmbarrier.test_wait.parity.shared::cta.b64 q, [%3], %4;\n"
                 "mbarrier.test_wait.parity.shared::cta.b64 r, [%5], %6;\nand.pred p, p, q;\nand.pred p, p, r;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(a), "r"(pa), "r"(b), "r"(pb), "r"(c), "r"(pc) : "memory");
    return ok != 0;
}
__device__ __forceinline__ void tc_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar) : "memory");
}
// Accumulator read-out of 32 lanes (matrix rows) x 32 columns (activation rows) in the fragment shape 16x128b: of 16 lanes x 4 columns
// thread 4 g + t gets rows g and g + 8 of column t, side by side.  v[16 hf + 2 c + e]: row g + 16 hf + 8 e, column 4 c + t.
// Measured per register and warp: 1.0 cycle, against 2.0 for the shape 16x256b and 0.6 for 32x32b, whose threads would need
// the scales of 32 columns each.
__device__ __forceinline__ void tc_ld_chunk(unsigned taddr, int (&v)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.16x128b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%32];\n\t"
                 "tcgen05.ld.sync.aligned.16x128b.x8.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%33];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                 : "r"(taddr), "r"(taddr + (16u << 16)) : "memory");
}
// The same of 16 lanes: v[2 c + e]: row g + 8 e.
__device__ __forceinline__ void tc_ld_chunk(unsigned taddr, int (&v)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.16x128b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(taddr) : "memory");
}
// Waits for the loads; the values pass through it so that nothing that uses them moves in front.
__device__ __forceinline__ void tc_ld_wait(int (&v)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]) :: "memory");
}
__device__ __forceinline__ void tc_ld_wait(int (&v)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]), "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]), "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]), "+r"(v[30]), "+r"(v[31]) :: "memory");
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

// Place of activation row m's scale inside a step's TOK of them: of every 16 rows the four of one epilogue thread (4 c + t) lie side by side.
__device__ __forceinline__ int tc_dx_slot(int m) { return (m & ~15) + (m & 3) * 4 + ((m >> 2) & 3); }
template <int N> __device__ __forceinline__ void reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" :: "n"(N)); }
template <int N> __device__ __forceinline__ void reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" :: "n"(N)); }

template <int NH, int RG>
__global__ void __launch_bounds__(TC_THREADS, 1)
k_matmul_tc(const __grid_constant__ CUtensorMap xmap, const uint8_t* __restrict__ tiles, int nb, int rows, int row_groups, int wstages, int ntiles, int tok_tiles, int dxbufs, int xsteps, int na,
            const float* __restrict__ xd, int x_stride, int ntok,
            float* arena, size_t y_off, size_t y_stride, int accum, int* error_flag, const it_peers* peers, const it_rowmap map, float minus_zero) {
    using T = Tc<NH, RG>;
    constexpr int TC_TOK = T::TOK, TC_X_BYTES = T::X_BYTES, TC_ND = T::ND, TC_EPI_TOK = T::EPI_TOK, CC = T::CC, NDW = T::NDW, TC_ROWS = T::ROWS, TC_A_BYTES = T::A_BYTES, TC_W_BYTES = T::W_BYTES;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const TcSmem L = tc_layout<NH, RG>(nb, wstages, dxbufs, xsteps, na);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, np = nb / 2;      // np: steps (pairs of blocks) of a tile
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L.flag);
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(smem + L.tmem);
    const unsigned bars = smem_u32(smem + L.bars);
    // barrier addresses: weight stages (full / empty), activation boxes of a step landed, tiles of a step expanded, steps committed, accumulators
    // of a step empty, activation scales (full / empty).  "Committed" is the one commit of a step: accumulators full, and the
    // tiles and boxes that the step read may be reused.  TC_NC barriers take turns whatever the number of accumulators: a wait sees
    // one bit, and with a barrier per accumulator (two) and three steps of boxes the box of step n - 1 is in place while the producer
    // waits for step n - 3 on the barrier that n - 1 commits to as well, so that the parity could flip twice before it looks.
    const unsigned wfull0 = bars, wempty0 = wfull0 + 8 * wstages, xfull0 = wempty0 + 8 * wstages,
                   afull0 = xfull0 + 8 * xsteps, dfull0 = afull0 + 8 * na, dempty0 = dfull0 + 8 * TC_NC, sfull0 = dempty0 + 8 * TC_ND, sempty0 = sfull0 + 16;
    // The CTA's tiles: blockIdx.x, + gridDim.x, ...; the activation tiles of one group of matrix rows are neighbours.  Every role walks
    // the same tiles with its ring positions running on, so the next tile's weights, boxes and products are under way while
    // the epilogue still stores the last one's results.
    const int tile0 = (int)blockIdx.x, tstep = (int)gridDim.x;

    if (tid == 0) {
        *abort_flag = 0;
        for (int s = 0; s < wstages; s++) { mbar_init(wfull0 + 8 * s, 1); mbar_init(wempty0 + 8 * s, 8); }
        for (int s = 0; s < xsteps; s++) mbar_init(xfull0 + 8 * s, 1);
        for (int a = 0; a < na; a++) mbar_init(afull0 + 8 * a, 4);
        for (int k = 0; k < TC_NC; k++) mbar_init(dfull0 + 8 * k, 1);
        for (int d = 0; d < TC_ND; d++) mbar_init(dempty0 + 8 * d, TC_EPI_WARPS);
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
            const int rg0 = tile / tok_tiles * RG, nrg = min(RG, row_groups - rg0);
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
            int s = 0, issued = 0, k0 = 0; unsigned kph = 0; bool ok = true;
            for (int tile = tile0; ok && tile < ntiles; tile += tstep) {
                const int tok0 = tile % tok_tiles * TC_TOK;
                for (int p = 0; p < np; p++) {
                    // the slot was last read xsteps steps ago: wait for that step's commit
                    if (issued >= xsteps) {
                        if (!mbar_wait(dfull0 + 8 * k0, kph, abort_flag, error_flag, 19)) { ok = false; break; }
                        if (++k0 == TC_NC) { k0 = 0; kph ^= 1u; }
                    }
                    mbar_expect_tx(xfull0 + 8 * s, (unsigned)(2 * TC_X_BYTES));
#pragma unroll
                    for (int k = 0; k < 2 * NH; k++)     // 64 rows per box; the boxes of a block lie one under the other like one box of TOK rows
                        tma_load_2d(smem_u32(smem + L.x + s * 2 * TC_X_BYTES + k * 64 * 128), &xmap, (2 * p + k / NH) * 128, tok0 + 64 * (k % NH), xfull0 + 8 * s);
                    issued++;
                    if (++s == xsteps) s = 0;
                }
            }
            if (*abort_flag) {
                const int first = issued > xsteps ? issued - xsteps : 0;
                for (int k = first; k < issued; k++) {
                    const long long t0 = clock64();
                    while (!mbar_test(xfull0 + 8 * (k % xsteps), (unsigned)(k / xsteps) & 1u) && clock64() - t0 < WAIT_CLOCKS) { }
                }
            }
        }
    } else if (warp == TC_EPI_WARPS + TC_EXP_WARPS + 1) {
        // ---------------- MMA issuer
        if (tc_elect()) {
            int s = 0, a = 0, d = 0, k = 0; unsigned sph = 0, aph = 0, dph = 1, kph = 0, last = 0, last_ph = 0; bool ok = true, ready = false;
            const unsigned long long adesc0 = tc_smem_desc(smem_u32(smem + L.a)), bdesc0 = tc_smem_desc(smem_u32(smem + L.x));
            for (int tile = tile0; ok && tile < ntiles; tile += tstep)
            for (int p = 0; p < np; p++) {
                // A wait costs this thread some 200 cycles even when it is met, and the tensor pipe idles meanwhile (three of them were 640
                // of a step's 1650 cycles at 64 activation rows): the next step's three are looked at together, while this one's MMAs run.
                if (!ready) {
                    ok = ok && mbar_wait(xfull0 + 8 * s, sph, abort_flag, error_flag, 13);
                    ok = ok && mbar_wait(dempty0 + 8 * d, dph, abort_flag, error_flag, 14);
                    ok = ok && mbar_wait(afull0 + 8 * a, aph, abort_flag, error_flag, 12);
                    if (!ok) break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned long long ad0 = adesc0 + (unsigned)(2 * a * (TC_A_BYTES >> 4)), bd0 = bdesc0 + (unsigned)(2 * s * (TC_X_BYTES >> 4));
                const unsigned dt0 = tmem_base + (unsigned)(2 * d * TC_TOK), commit = dfull0 + 8 * k;
                last = commit; last_ph = kph;
                if (++k == TC_NC) { k = 0; kph ^= 1u; }
                if (++s == xsteps) { s = 0; sph ^= 1u; }
                if (++a == na) { a = 0; aph ^= 1u; }
                if (++d == TC_ND) { d = 0; dph ^= 1u; }
                // descriptors differ from the first tile's only in the start-address field (16-byte units): + tile index, + 2 per K step of 32
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const unsigned long long ad = ad0 + (unsigned)(h * (TC_A_BYTES >> 4)), bd = bd0 + (unsigned)(h * (TC_X_BYTES >> 4));
                    const unsigned dt = dt0 + (unsigned)(h * TC_TOK);
                    tc_mma<false>(dt, ad, bd, T::IDESC);
                    tc_mma<true>(dt, ad + 2, bd + 2, T::IDESC);
                    tc_mma<true>(dt, ad + 4, bd + 4, T::IDESC);
                    tc_mma<true>(dt, ad + 6, bd + 6, T::IDESC);
                }
                tc_commit(commit);                // accumulators complete; tiles and boxes of this step may be reused
                ready = mbar_poll3(xfull0 + 8 * s, sph, dempty0 + 8 * d, dph, afull0 + 8 * a, aph);
            }
            // the last commit's arrival must find the CTA's shared memory still its own (bounded)
            const long long t0 = clock64();
            while (last && !mbar_test(last, last_ph) && clock64() - t0 < WAIT_CLOCKS) { }
        }
    } else if (warp == TC_EPI_WARPS + TC_EXP_WARPS + 3) {
        // ---------------- activation scales of every tile but the first (which the epilogue warps fetch together), one tile ahead
        asm volatile("griddepcontrol.wait;" ::: "memory");
        int j = 1;                                                    // the CTA's j-th tile uses buffer j % 2
        for (int tile = tile0 + tstep; tile < ntiles; tile += tstep, j++) {
            const int k = j & 1;
            const int tok0 = tile % tok_tiles * TC_TOK, ntv = min(TC_TOK, ntok - tok0);
            if (!mbar_wait_warp(sempty0 + 8 * k, ((unsigned)(j >> 1) & 1u) ^ 1u, abort_flag, error_flag, 20)) break;     // tile j - 2 is done with it
            float* dxs = reinterpret_cast<float*>(smem + L.dx + k * L.dx_bytes);
            for (int m = lane; m < TC_TOK; m += 32) {
                const float* src = xd + (size_t)(tok0 + m) * (x_stride / 256);
                float* dst = dxs + tc_dx_slot(m);
#pragma unroll 8
                for (int bb = 0; bb < np; bb++) dst[bb * TC_TOK] = m < ntv ? src[bb] : 0.f;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(sfull0 + 8 * k);
        }
    } else if (warp >= TC_EPI_WARPS) {
        // ---------------- expanders: warp 8 + 4 e + i expands row group i of the steps with number % 2 == e (with two row groups: block i / 2 of
        // group i % 2); step n goes into tile pair n % na
        static_assert(TC_NA_MAX <= TC_NC && TC_EXP_WARPS == 8, "step n commits after it is expanded: a wait for step n - na is at most one phase behind");
        const int eset = (warp - TC_EPI_WARPS) >> 2, rgl = (warp - TC_EPI_WARPS) & (RG - 1), h0 = RG == 4 ? 0 : ((warp - TC_EPI_WARPS) >> 1) & 1, g = lane >> 2, t = lane & 3;
        unsigned char* const at = smem + L.a + (rgl * 32 + g) * 128;
        unsigned char* const plo = at + (((2 * t) ^ g) << 4);          // columns 32 t .. 32 t + 15 of row g; the other rows 1024 bytes apart
        unsigned char* const phi = at + (((2 * t + 1) ^ g) << 4);      // columns 32 t + 16 .. 32 t + 31
        float* const dws = reinterpret_cast<float*>(smem + L.dw) + rgl * 32 + 4 * g;
        const unsigned char* const src0 = smem + L.w + rgl * TC_KB * IT_TILE_BYTES;
        int s = 0, dp = TC_NC - na, r = 0, gp = 0, pair = 0; unsigned sph = 0, dpp = 1; bool ok = true;        // dp, dpp: the barrier and parity of step gp - na
        for (int tile = tile0; tile < ntiles; tile += tstep)
        for (int p = 0; p < np; p++, gp++) {
            const bool last = (p & 1) || p + 1 == np;         // last step of the weight stage
            if ((gp & 1) == eset) {
                ok = ok && mbar_wait(wfull0 + 8 * s, sph, abort_flag, error_flag, 15);
                // the tile pair was last read na steps ago: wait for that step's commit
                if (gp >= na) ok = ok && mbar_wait(dfull0 + 8 * dp, dpp, abort_flag, error_flag, 16);
                unsigned char *const lo = plo + 2 * pair * TC_A_BYTES, *const hi = phi + 2 * pair * TC_A_BYTES;
#pragma unroll
                for (int hh = 0; hh < RG / 2; hh++) {
                    const int h = hh + h0;
                    const unsigned char* src = src0 + s * TC_W_BYTES + (2 * (p & 1) + h) * IT_TILE_BYTES;
                    const uint4 wa = *reinterpret_cast<const uint4*>(src + 16 * lane);
                    const uint4 wb = *reinterpret_cast<const uint4*>(src + 512 + 16 * lane);
#pragma unroll
                    for (int i = 0; i < 4; i++) {         // bit pair i of every byte: matrix row g + 8 i of the group
                        auto sgn = [&](unsigned w) { return (((w >> (2 * i)) & 0x03030303u) + 0x7f7f7f7fu) ^ 0x80808080u; };   // code - 1 in every byte; no carry crosses a byte
                        *reinterpret_cast<uint4*>(lo + h * TC_A_BYTES + i * 1024) = make_uint4(sgn(wa.x), sgn(wa.y), sgn(wa.z), sgn(wa.w));
                        *reinterpret_cast<uint4*>(hi + h * TC_A_BYTES + i * 1024) = make_uint4(sgn(wb.x), sgn(wb.y), sgn(wb.z), sgn(wb.w));
                    }
                    if (t == 0) {
                        const uint2 sc = *reinterpret_cast<const uint2*>(src + 1024 + 8 * g);
                        const __half2 h01 = *reinterpret_cast<const __half2*>(&sc.x), h23 = *reinterpret_cast<const __half2*>(&sc.y);
                        *reinterpret_cast<float4*>(dws + (r + h) * TC_ROWS) =      // rows g, g + 8, g + 16, g + 24: the rows of one epilogue thread
                            make_float4(__low2float(h01), __high2float(h01), __low2float(h23), __high2float(h23));
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // generic-proxy stores before the MMA's async-proxy reads
                __syncwarp();
                if (lane == 0 && ok) {
                    mbar_arrive(afull0 + 8 * pair);
                    mbar_arrive_n(wempty0 + 8 * s, last && !(p & 1) ? 2u : 1u);  // read its tiles; a stage of one step counts them twice
                }
            }
            r = r + 2 == NDW ? 0 : r + 2;
            if (++pair == na) pair = 0;
            dp++;
            if (dp >= TC_NC) { dp = 0; dpp ^= 1u; }
            if (last) { if (++s == wstages) { s = 0; sph ^= 1u; } }
        }
    } else {
        // ---------------- epilogue: warp 4 q + i owns row group i x activation rows EPI_TOK q ..; its thread 4 g + t owns rows
        // g, g + 8, g + 16, g + 24 of the group (with two row groups warp 4 q + i half i % 2 of group i / 2, and two rows) and every fourth activation row.  One 16-byte load of row scales per block and one of
        // activation scales per 16 columns and step then serve all of a thread's results: with a row per thread and all columns
        // (one broadcast 16-byte load per four results) the shared-memory read port was what bounded the kernel.
        constexpr int NEPI = TC_EPI_WARPS * 32;
        reg_inc<TC_EPI_REGS>();
        constexpr int HF = RG / 2;                     // pairs of rows of a thread
        const int grp = warp >> 2, quad = warp & 3, row0 = quad * 8 * RG, g = lane >> 2, t = lane & 3, m0 = grp * TC_EPI_TOK;     // row0: this warp's first row of the tile
        const unsigned tquad = tmem_base + ((unsigned)(quad * 32) << 16) + (unsigned)m0;
        // scales: four rows of a group side by side (g, g + 8, g + 16, g + 24), two of them this thread's when it has two
        const f32x2* const dws = reinterpret_cast<const f32x2*>(smem + L.dw) + (row0 & ~31) / 2 + 2 * g + (RG == 2 ? quad & 1 : 0);
        asm volatile("griddepcontrol.wait;" ::: "memory");            // q8 scales and (when accumulating) y come from earlier kernels
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        {
            float* dxs = reinterpret_cast<float*>(smem + L.dx);
            const int tok0 = tile0 % tok_tiles * TC_TOK, ntv = min(TC_TOK, ntok - tok0);
#pragma unroll 4
            for (int i = tid; i < np * TC_TOK; i += NEPI) {
                const int m = i % TC_TOK, bb = i / TC_TOK;
                dxs[bb * TC_TOK + tc_dx_slot(m)] = m < ntv ? xd[(size_t)(tok0 + m) * (x_stride / 256) + bb] : 0.f;
            }
            asm volatile("bar.sync 1, %0;" :: "n"(NEPI) : "memory");
        }
        const f32x2 mz = pkf(minus_zero, minus_zero);
        int d = 0, r = 0, j = 0, kc = 0; unsigned kph = 0;
        bool ok = true;
        for (int tile = tile0; tile < ntiles; tile += tstep, j++) {
            const int k = j & 1;
            const int rg0 = tile / tok_tiles * RG, tok0 = tile % tok_tiles * TC_TOK, ntv = min(TC_TOK, ntok - tok0);
            const bool active = m0 < ntv;              // groups past the last activation row only release the accumulators
            if (j > 0) ok = ok && mbar_wait(sfull0 + 8 * k, (unsigned)((j - 1) >> 1) & 1u, abort_flag, error_flag, 18);
            const float4* dxs = reinterpret_cast<const float4*>(smem + L.dx + k * L.dx_bytes) + m0 / 4 + t;
            f32x2 acc[HF][8 * CC];                     // rows g + 16 hf and g + 8 + 16 hf of column 4 c + t
#pragma unroll
            for (int hf = 0; hf < HF; hf++)
#pragma unroll
                for (int c = 0; c < 8 * CC; c++) acc[hf][c] = 0ull;
            for (int p = 0; p < np; p++) {             // two blocks at a time: they share the activation scale, the wait and the release
                ok = ok && mbar_wait(dfull0 + 8 * kc, kph, abort_flag, error_flag, 17);
                __syncwarp();
                if (active) {
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    // chunks of 32 columns of one block; the next one is on its way while one is folded
                    const unsigned ta = tquad + (unsigned)(2 * d * TC_TOK);
                    auto chunk = [&](int ch) { return ta + (unsigned)((ch & 1) * TC_TOK + (ch >> 1) * 32); };
                    int S[2][16 * HF];
                    tc_ld_chunk(chunk(0), S[0]);
                    // row scales of both blocks: stored by the expanders before they released the tiles to the MMAs whose completion we just saw
                    f32x2 dwb[2][HF];
#pragma unroll
                    for (int bk = 0; bk < 2; bk++) {
                        const f32x2* p = dws + (r + bk) * (TC_ROWS / 2);
                        if constexpr (HF == 2) { const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p); dwb[bk][0] = v.x; dwb[bk][HF - 1] = v.y; }
                        else dwb[bk][0] = *p;
                    }
                    f32x2 dx[8];
#pragma unroll
                    for (int ch = 0; ch < 2 * CC; ch++) {
                        if (!(ch & 1)) {                                      // both blocks of these columns share the activation scales
                            const float4 xa = dxs[(ch >> 1) * 8], xb = dxs[(ch >> 1) * 8 + 4];
                            dx[0] = pkf(xa.x, xa.x); dx[1] = pkf(xa.y, xa.y); dx[2] = pkf(xa.z, xa.z); dx[3] = pkf(xa.w, xa.w);
                            dx[4] = pkf(xb.x, xb.x); dx[5] = pkf(xb.y, xb.y); dx[6] = pkf(xb.z, xb.z); dx[7] = pkf(xb.w, xb.w);
                        }
                        int (&v)[16 * HF] = S[ch & 1];
                        tc_ld_wait(v);
                        if (ch + 1 < 2 * CC) tc_ld_chunk(chunk(ch + 1), S[(ch + 1) & 1]);
                        else {
                            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                            __syncwarp();
                            if (lane == 0 && ok) mbar_arrive(dempty0 + 8 * d);      // the MMAs of step p + ND may use the accumulators
                        }
#pragma unroll
                        for (int c = 0; c < 8; c++) {
                            const int cc = (ch >> 1) * 8 + c;
#pragma unroll
                            for (int hf = 0; hf < HF; hf++)
                                acc[hf][cc] = add2(acc[hf][cc], mul2_rounded(mul2(dwb[ch & 1][hf], dx[c]), pkf((float)v[16 * hf + 2 * c], (float)v[16 * hf + 2 * c + 1]), mz));
                        }
                    }
                } else if (lane == 0 && ok) mbar_arrive(dempty0 + 8 * d);
                dxs += TC_TOK / 4;
                if (++kc == TC_NC) { kc = 0; kph ^= 1u; }
                if (++d == TC_ND) d = 0;
                r = r + 2 == NDW ? 0 : r + 2;
            }
            if (!__all_sync(0xffffffffu, ok && !*abort_flag)) break;
            __syncwarp();
            if (lane == 0) mbar_arrive(sempty0 + 8 * k);          // the tile's activation scales have been read
            if (!active) continue;
#pragma unroll
            for (int i = 0; i < 2 * HF; i++) {
                const int row = rg0 * 32 + row0 + g + 8 * i;
                if (row >= rows) continue;
                const int grow = it_map_row(map, row);
                const size_t off = y_off + (size_t)(tok0 + m0 + t) * y_stride + grow;     // first of this thread's activation rows
                float old[8 * CC];
                if (!peers) {
                    float* y = arena + off;
#pragma unroll
                    for (int c = 0; c < 8 * CC; c++) old[c] = accum && m0 + 4 * c + t < ntv ? __ldcg(y + (size_t)(4 * c) * y_stride) : 0.f;
#pragma unroll
                    for (int c = 0; c < 8 * CC; c++) {
                        const float2 v2 = upk(acc[i >> 1][c]); const float v = i & 1 ? v2.y : v2.x;
                        if (m0 + 4 * c + t < ntv) y[(size_t)(4 * c) * y_stride] = accum ? __fadd_rn(old[c], v) : v;
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < 8 * CC; c++) {
                        const float2 v2 = upk(acc[i >> 1][c]); const float v = i & 1 ? v2.y : v2.x;
                        if (m0 + 4 * c + t < ntv) it_result_store(peers, arena, off + (size_t)(4 * c) * y_stride, v, accum);
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

template <int NH, int RG>
static int tc_launch(it_ctx* c, const it_mat* w, int ntok, const it_q8* x, float* y, size_t y_stride, int accum) {
    const int nb = (int)(w->cols / 128);
    const int tok_tiles = (ntok + Tc<NH, RG>::TOK - 1) / Tc<NH, RG>::TOK, ntiles = (int)((w->row_groups + RG - 1) / RG) * tok_tiles;
    // One CTA per SM walks its tiles, with two buffers of activation scales; where those do not fit (wide rows), a CTA per tile.
    int grid = ntiles < c->sm_count ? ntiles : c->sm_count, dxbufs = ntiles > grid ? 2 : 1;
    int na = 2;
    auto fits = [&](int wst, int xst) { return tc_layout<NH, RG>(nb, wst, dxbufs, xst, na).total + 1024 <= TC_SMEM_MAX; };
    if (!fits(2, 2)) { grid = ntiles; dxbufs = 1; }
    if (!fits(2, 2)) return 1;
    na = TC_NA_MAX;
    if (!fits(2, 2)) na = 2;
    // Activation boxes three steps deep where they fit (two left the MMA waiting 375 cycles a step), then weight stages of TC_KB blocks
    const int xsteps = fits(2, 3) ? 3 : 2;       // no more than TC_NC
    int stages = 5;
    while (!fits(stages, xsteps)) stages--;
    const TcSmem L = tc_layout<NH, RG>(nb, stages, dxbufs, xsteps, na);
    static bool attr_set[16] = {};
    if (!attr_set[c->device & 15]) { IT_CUDA(cudaFuncSetAttribute(k_matmul_tc<NH, RG>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM_MAX)); attr_set[c->device & 15] = true; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(TC_THREADS); cfg.dynamicSmemBytes = (size_t)L.total + 1024; cfg.stream = c->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    IT_CUDA(cudaLaunchKernelEx(&cfg, k_matmul_tc<NH, RG>, x->tmap, (const uint8_t*)w->tiles, nb, (int)w->rows, (int)w->row_groups, stages, ntiles, tok_tiles, dxbufs, xsteps, na,
        (const float*)x->d, (int)x->max_n, ntok, c->arena, (size_t)(y - c->arena), y_stride, accum, c->error_flag_dev,
        (const it_peers*)(w->sharded ? c->peers_dev : nullptr), w->map, -0.0f));
    c->pdl_safe_q8 = x;
    return IT_OK;
}

// Returns IT_OK after launching, or a positive value when the shape does not suit this kernel (the caller then uses k_matmul_t2).
// Tiles by it_tc_tile (it_route.h); 128 activation rows only when their buffers fit (rows of up to about 28,000 columns).
int it_matmul_tc_launch(it_ctx* c, const it_mat* w, int ntok, const it_q8* x, float* y, size_t y_stride, int accum) {
    static const bool wide = []{ const char* v = getenv("IT_MATMUL_WIDE"); return !v || atoi(v) != 0; }();
    const int best = it_tc_tile((long)w->row_groups, ntok, c->sm_count);
    if (best == IT_TC_128X128 && wide) { const int r = tc_launch<2, 4>(c, w, ntok, x, y, y_stride, accum); if (r != 1) return r; }
    if (best == IT_TC_64X64) return tc_launch<1, 2>(c, w, ntok, x, y, y_stride, accum);
    return tc_launch<1, 4>(c, w, ntok, x, y, y_stride, accum);
}
