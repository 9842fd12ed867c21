// Which kernel takes a launch, as functions of sizes alone: plain host code, so that a test holds the rules to their edges without a GPU.
#pragma once

// ---- ternary products of more than eight rows -----------------------------------------------------------------------------
// Row groups (of 32 matrix rows) a CTA of the mma.sync kernel owns: 128-row tiles with sixteen consumer warps when that still gives
// the grid at least 0.6 CTAs per SM, else 64-row tiles (eight warps, two CTAs per SM), else 32-row tiles.
static inline int it_mm_groups(long row_groups, long ntok, int sm_count) {
    const long tok_tiles = (ntok + 63) / 64, want = (long)sm_count * 6 / 10;
    return (row_groups + 3) / 4 * tok_tiles >= want ? 4 : (row_groups + 1) / 2 * tok_tiles >= want ? 2 : 1;
}
// Whether the tensor-memory kernel (it_matmul_tc.cu, one CTA per SM and 128-row tiles) goes first.  Matrices that give such tiles to most SMs
// do.  So do smaller ones of more row groups than SMs, whose 32-row tiles are one wave and a few CTAs, from 41 activation rows on (the mma.sync
// kernel's time steps every eight), and those it would give 64-row tiles, from 33 on.  us, mma.sync / tensor memory:
//   5120 x 5120 at 33-40 rows 18.8 / 20.1, at 41-48 21.5 / 20.2, at 64 21.9 / 20.3, at 65-128 32 / 27; at 17-24 15.2 / 18.1
//   5120 x 17408 at 40 rows 59.4 / 59.4, at 48 65.6 / 59.4, at 64 68.1 / 59.6, at 65 99.2 / 78.3, at 128 102.3 / 78.8
//   6144 and 8192 x 5120 at 33 rows 21.0 / 20.2 and 21.4 / 20.3, at 64 21.4 / 20.4 and 21.5 / 20.5; 9600 and 11136 x 5120 at 33 to 64 rows 32 / 21
//   no more row groups than SMs: 4736 x 5120 at 33 rows 14.7 / 20.2, at 64 15.1 / 20.5; 2560 x 5120 at 64 14.7 / 20.3
static inline bool it_mm_takes_tc(long row_groups, long ntok, int sm_count) {
    const int wr = it_mm_groups(row_groups, ntok, sm_count);
    return wr == 4 || (row_groups > sm_count && ntok > (wr == 2 ? 32 : 40));
}
