// The split (integer tensor core) form of the Gram product, between
// fb_ozaki_gram.cu, which computes it, and fb_gram.cu, which chooses it,
// reads its sums and falls back to FP64 where its verdict says so.
#pragma once

#include <algorithm>

#include "fb_common.cuh"

namespace fb {

constexpr int SPLIT_STAGE_ROWS = 16;              // complex rows per stage; chunks are whole stages
constexpr int SPLIT_TILE_DOUBLES = 128 * 64;      // a partial or summed tile, column n of it contiguous
constexpr int SPLIT_SCREEN_PARTS = 4;             // blocks a column of the screen
constexpr int SPLIT_E_UNSET = -4000;              // scale of a column that has only zeros so far
constexpr int SPLIT_E_TINY = -3999;               // and of one that has nothing above the subnormals
constexpr int SPLIT_INVALID = 1;                  // Inf, NaN or a wait that gave up: the sums mean nothing
constexpr int SPLIT_INACCURATE = 2;               // the slices may leave out more than FP64 rounding would

struct SplitShape {
    int nt_a, nt_b;      // 64-column tiles of A and of B
    int hermitian;       // folded diagonal tiles first, then the tiles above the diagonal
    int ntiles;
    int screened;        // columns the screen looks at: A's, and B's if it is another matrix
    int64_t chunk_rows;
    int nchunks;
};

// What a CTA reports about its chunk: per input column (A's 64, then B's) the
// last scale exponent and the sum of squares, and what is wrong with it.
struct SplitStat {
    double sumsq[128];
    int E[128];
    int flags;           // SPLIT_INVALID, SPLIT_INACCURATE
    int pad[3];
};

struct SplitLayout {
    size_t verdict, refused, sums, stats, partial, total;  // byte offsets in the workspace
};

// Tile `x` of a launch over the folded or the full tiles.
__host__ __device__ inline void split_tile_of(const SplitShape& sh, bool full, int x, int& ti, int& tj, int& tile) {
    if (!full) {
        ti = tj = tile = x;
    } else if (sh.hermitian) {
        ti = 0;
        tile = sh.nt_a + x;
        while (x >= sh.nt_a - 1 - ti) { x -= sh.nt_a - 1 - ti; ++ti; }
        tj = ti + 1 + x;
    } else {
        ti = x / sh.nt_b;
        tj = x - ti * sh.nt_b;
        tile = x;
    }
}

SplitShape split_shape(int64_t rows, int kA, int kB, bool hermitian);
SplitLayout split_layout(const SplitShape& sh);
// The screen over a sample of all rows: which columns go to the FP64 kernels.
int split_screen_enqueue(const z64* A, int64_t lda, const z64* B, int64_t ldb, int64_t rows, int kA,
                         const SplitShape& sh, void* workspace, cudaStream_t stream, const ChainStatus* st, int gate);
// The partial tiles of chunks [chunk0, chunk1); each depends on its rows alone.
// screened: nothing, where a screen that ran before refused a column. strict:
// no FP64 kernels stand behind the sums.
int split_partials_enqueue(const z64* A, int64_t lda, const z64* B, int64_t ldb, int64_t rows, int kA, int kB,
                           const SplitShape& sh, void* workspace, cudaStream_t stream, const ChainStatus* st, int gate,
                           int chunk0, int chunk1, bool screened, bool strict);
// Sums the partial tiles of every chunk and writes each tile's verdict.
int split_sum_enqueue(int64_t rows, const SplitShape& sh, void* workspace, cudaStream_t stream, const ChainStatus* st,
                      int gate, bool screened);

}  // namespace fb
