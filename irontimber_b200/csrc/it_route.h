// Which kernel takes a launch, as functions of sizes alone: plain host code, so that a test holds the rules to their edges without a GPU.
#pragma once
#include <cstddef>

// ---- ternary products of up to eight rows -----------------------------------------------------------------------------------
// Ring slots of a CTA of k_matvec_t2 (it_matvec_t2.cu) whose chunks `groups` groups of warps take in turn: a multiple of them, so that a slot
// is always the same group's.  A wait on an mbarrier sees a parity: in a ring of another size a group's chunk follows another group's in
// its slot, and a copy that lands that much late would let the group take the phase before for its own.
static inline int it_mv_ring(int slots, int groups) { return slots - slots % groups; }

// ---- ternary products of more than eight rows -----------------------------------------------------------------------------
// Row groups (of 32 matrix rows) a CTA of the mma.sync kernel owns: 128-row tiles with sixteen consumer warps when that still gives
// the grid at least 0.6 CTAs per SM, else 64-row tiles (eight warps, two CTAs per SM), else 32-row tiles.
static inline int it_mm_groups(long row_groups, long ntok, int sm_count) {
    const long tok_tiles = (ntok + 63) / 64, want = (long)sm_count * 6 / 10;
    return (row_groups + 3) / 4 * tok_tiles >= want ? 4 : (row_groups + 1) / 2 * tok_tiles >= want ? 2 : 1;
}
// Whether the tensor-memory kernel (it_matmul_tc.cu, one CTA per SM) goes first: for everything but short rows and few of them, where both kernels
// are all start-up and the mma.sync kernel's is shorter.
// us, mma.sync / tensor memory:
//   5120 x 17408 at 9 rows 44.1 / 34.7, at 33 58.9 / 37.9, at 64 67.5 / 38.1, at 128 103.5 / 53.8;  1024 x 17408 at 9 rows 33.9 / 33.3, at 64 44.5 / 36.8
//   5120 x 5120 at 9 rows 15.0 / 12.4, at 64 22.0 / 13.6;  4736 x 5120 at 9 12.2 / 11.8, at 64 15.2 / 13.0;  96 x 5120 at 9 11.5 / 11.2, at 64 14.5 / 12.5
//   9000 x 5120 at 9 rows 20.8 / 13.1, at 64 21.7 / 14.2;  2560 x 3072 at 9 8.3 / 8.0;  5120 x 2048 at 9 7.4 / 6.9;  640 x 2048 at 9 to 32 6.0 / 6.0
//   2560 x 2048 at 9 rows 6.1 / 6.2, at 33 7.3 / 6.7;  5000 x 1024 at 9 4.9 / 5.0, at 33 5.7 / 5.4;  512 x 1024 at 9 4.2 / 4.3, at 32 4.2 / 4.4, at 33 4.7 / 4.6
static inline bool it_mm_takes_tc(long row_groups, long cols, long ntok, int sm_count) {
    return ntok > 32 || cols > 2048 || (row_groups > sm_count && cols > 1024) || it_mm_groups(row_groups, ntok, sm_count) > 1;
}
// Which tiles it cuts a product into, matrix rows x activation rows: what the busiest SM's tiles take, a step of theirs some 1980, 1480 and 1080
// cycles.  us, 128 x 128 / 128 x 64 / 64 x 64: 5120 x 17408 at 64 rows - / 52.2 / 38.1, at 128 69.5 / 53.3 / - ; 34816 x 5120 at 128 48.2 / 63 / -
enum it_tc_tiles { IT_TC_128X128, IT_TC_128X64, IT_TC_64X64 };
static inline it_tc_tiles it_tc_tile(long row_groups, long ntok, int sm_count) {
    auto rounds = [&](long groups, long tok) { return ((row_groups + groups - 1) / groups * ((ntok + tok - 1) / tok) + sm_count - 1) / sm_count; };
    const long a = 20 * rounds(4, 128), b = 15 * rounds(4, 64), d = 11 * rounds(2, 64);
    return a < b && a < d ? IT_TC_128X128 : b <= d ? IT_TC_128X64 : IT_TC_64X64;
}

// ---- attention of a prompt pass ---------------------------------------------------------------------------------------------
// What a CTA of k_attention_group (it_attention_prefill.cu) takes: query heads of one KV head x rows of the pass.  rows 0: the scores of no
// grouping fit its shared memory (from about 13,000 positions on at three heads of 256), and k_attention's CTAs of one head and row run.
struct it_attn_group { int heads, rows; };
#define IT_ATTN_THREADS 1024
#define IT_ATTN_CHUNK_POS 64                       // positions per V chunk (two cache tiles)
#define IT_ATTN_RING 2                             // V chunks in flight
#define IT_ATTN_SMEM ((size_t)220 * 1024)
static inline size_t it_attn_group_smem(it_attn_group g, int hd, int npos) {
    const size_t npad = (size_t)(npos + 3) / 4 * 4;
    return (size_t)g.heads * g.rows * (npad + hd) * 4 + (size_t)IT_ATTN_RING * IT_ATTN_CHUNK_POS * hd * 2;
}
static inline it_attn_group it_attn_grouping(int hd, int nh, int nkv, int npos) {
    it_attn_group g = { 0, 0 };
    if (hd % 8 || nh % nkv || hd > IT_ATTN_THREADS) return g;
    const int rep = nh / nkv;
    g.heads = rep % 3 == 0 && 3 * hd <= IT_ATTN_THREADS ? 3 : rep % 2 == 0 && 2 * hd <= IT_ATTN_THREADS ? 2 : 1;
    for (g.rows = 2; g.rows > 0; g.rows--) if (it_attn_group_smem(g, hd, npos) <= IT_ATTN_SMEM && (g.rows == 2 || g.heads > 1)) break;
    return g;
}
// Whether the tiled kernels (it_attention_tiled.cu) take the pass, blk rows at a time (what their scratch holds): by the time either side needs, in
// ns per position that the pass sees on average.  The other side pays by waves of CTAs, so a few rows far into a context are its own; the tiled
// kernels' ordered sums walk all positions once per block of rows, however few the rows, and they are three launches.  The constants are
// those of 24 heads over 4 of dimension 256: a wave of grouped CTAs 83 ns a position (3 heads x 2 rows) or 50 (x 1 row), one of
// k_attention's two CTAs per SM 83; tiled 200 a block and 0.7 a row, 0.95 once the scores of a block are past 100 MB and leave L2, and 40 us.
// They are scaled with the chains of a CTA and the width of a row.  us a layer of an attention-only stack, other / tiled (taken when the tiled
// kernels' three launches were 540 us at 777 rows from position 0; they are 435 now, so the line errs towards the other side):
//   at    0:   9 rows 186 / 248, 256 518 / 522, 257 588 / 632, 300 648 / 652, 384 744 / 704, 512 1106 / 966, 777 1776 / 1482
//   at 1024:  32 rows 276 / 464, 64 404 / 504, 96 556 / 604, 128 665 / 635, 256 1091 / 899
//   at 4096:  24 rows 515 / 1092, 64 899 / 1184, 96 1299 / 1346, 128 1653 / 1434, 256 2817 / 2086
//   at 7000:  24 rows 894 / 1728, 64 1640 / 1867, 96 2413 / 2090, 128 2790 / 2258      (one row a CTA from 6400 positions on)
//   in several blocks: 1024 rows at 8800 27,576 / 24,772, at 10,800 33,222 / 33,085; 512 at 9000 13,839 / 12,323, at 12,000 18,063 / 19,137; 256 at
//   9000 6866 / 6067, at 11,000 8252 / 9519
//   at 14,000 (k_attention): 9 rows 1359 / 2969, 32 3725 / 3190, 64 6788 / 3820
static inline bool it_attn_takes_tiled(int hd, int nh, int nkv, int slot0, int nt, int blk, int sm_count) {
    const it_attn_group g = it_attn_grouping(hd, nh, nkv, slot0 + nt);
    const double p = slot0 + 0.5 * nt, width = nh * hd / 6144.0;
    const long ctas = g.rows ? (long)(nh / g.heads) * ((nt + g.rows - 1) / g.rows) : ((long)nh * nt + 1) / 2;
    const double other = (double)((ctas + sm_count - 1) / sm_count) * (g.rows ? 17 + 11 * g.heads * g.rows : 83);
    const int blocks = (nt + blk - 1) / blk;
    const double scores = 4.0 * nh * (slot0 + nt) * ((nt + blocks - 1) / blocks);
    const double tiled = 200.0 * blocks + (scores > 1e8 ? 0.95 : 0.7) * width * nt;
    return other * p > tiled * p + 40000;
}

// ---- delta rule of a prompt pass --------------------------------------------------------------------------------------------
// k_gdn_rows (it_gdn_prefill.cu) is built for a state size of 128 and for three tokens or more: the warp that stores a state row first waits for
// the other warp's read of it at the third token.
static inline bool it_gdn_rows_takes(int sd, int nt) { return sd == 128 && nt >= 3; }
