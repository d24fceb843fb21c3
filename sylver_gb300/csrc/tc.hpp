// Tensor-core (tcgen05) Schur-complement update: descriptors and launchers.
#pragma once

#include <cuda.h>

#include "device.hpp"

namespace sylver_gb300 {

// One 128 x 128 tile of C -= P_a P_b^T for a contribution block:
// C(i, j) = arena[c_off + j*ldc + i] for i in [row0, row0+128) < rowEnd,
// j in [col0, col0+128) < colEnd, only i >= j written.  A rows start at
// stacked panel row a_row, B rows at b_row; nk chunks of TC_KCHUNK along k
// starting at chunk kc0.
struct TcTask {
  int64_t c_off;
  int ldc, row0, col0, rowEnd, colEnd, a_row, b_row, nk;
  int kc0;
};

// Transposed 3xBF16 copy of front rows [n, m) x columns [c0, c0 + K) into
// stacked panel rows [base, base + m - n) of the three planes.
struct TcSplit {
  int64_t off;
  int ld, m, n, K, base, c0;
};

size_t tc_smem_bytes();
void prepare_tc_kernels();
// Tensor map of one BF16 plane: rows x pitch elements (pitch a multiple of
// TC_KCHUNK), boxes of TC_KCHUNK x 128.
void make_panel_map(CUtensorMap* map, const uint16_t* base, int64_t rows, int pitch);
// planes: three BF16 planes, plane q at planes + q * pstride.
void launch_split_t(const float* arena, const TcSplit* sp, int nsplit, int64_t max_rows,
                    uint16_t* planes, int64_t pstride, int pitch, cudaStream_t s);
// maps: the tensor maps of the three planes.
void launch_update_tc(const CUtensorMap* maps, float* arena, const TcTask* t, int ntask,
                      unsigned* err, cudaStream_t s);

// FP64 fronts (kernels_tc64.cu): C -= P P^T on the BF16 tensor cores with
// operands cut into eight signed 9-bit digits of a per-row fixed-point scaling,
// and on the FP64 pipe for the entries that this would not hold to FP64's bound.
constexpr int OZ_KC = 32;  // columns of a k chunk
constexpr int OZ_DIGITS = 8;
constexpr int OZ_TILE_COLS = 64;  // tiles are 128 x 64 or narrower
constexpr int OZ_GW = 256;  // fully-summed columns per trailing update
// Columns of a front per contribution-block update, each with row scales of its
// own: 56^3 13.8 ms of updates, 14.1 with 256, 13.9 with 1024 columns (all K columns
// at once: more rows far below their scale, 20 ms when their warps redid them).
constexpr int OZ_KB = 512;
// Operand entries an update launch cuts at most (16 bytes of digit planes each): an
// eighth of the front storage's, within these limits (64 MiB to 2 GiB of planes).
// Level and front sizes do not set the size of the planes: what does not fit goes
// in several launches, each still of thousands of tile columns.
constexpr int64_t OZ_MIN_ENTRIES = 1 << 22, OZ_MAX_ENTRIES = 1 << 27;
constexpr int OZ_FEW_TILES = 2 * NUM_SMS;  // launches below this many CTAs take smaller tiles
// Digits of front rows [r0, r0 + rows) x columns [c0, c0 + K): stacked rows
// [base, base + rows) of the planes (zeros from K to K rounded up to
// OZ_KC), and each row's scale exponent in sexp[base ..].
struct OzSplit {
  int64_t off;
  int ld, r0, rows, c0, K, base;
};
// One tile (128 rows, OZ_TILE_COLS columns or fewer) of an update of a front at
// off by its own columns [k0, k0 + K): rows [row0, row0 + 128) < rowEnd, columns
// [col0, colEnd), only row >= column written; a_row, b_row: stacked rows of row0
// and col0.
struct OzTask {
  int64_t off;
  int ld, row0, col0, rowEnd, colEnd, a_row, b_row, k0, K, pad;
};
// Panel step of an FP64 front (kernels_panel64.cu): the w x w diagonal block at
// (k0, k0), w <= 32, and rows [r0, r1) below it; base >= 0: stacked row of
// r0 in the digit planes; didx >= 0: this CTA stores the factorised block as
// block didx of the level's store.
struct P64Task {
  int64_t off;
  int ld, k0, w, r0, r1, base, didx, pad;
};
// rows: most rows of a task (16 or fewer take the kernel for short tasks)
void launch_panel64(double* arena, const P64Task* t, int ntask, int rows, double* dstore,
                    uint16_t* planes, int64_t pstride, int pitch, int* sexp, unsigned* status,
                    cudaStream_t s);
void launch_diag_store64(double* arena, const P64Task* t, int ntask, const double* dstore,
                         cudaStream_t s);
void prepare_tc64_kernels();
// Maps of all planes (plane q at planes + q * pstride) with the boxes
// of the A (128 rows) and the B operand (64 rows).
void make_digit_maps(CUtensorMap* maps, const uint16_t* planes, int64_t pstride, int64_t rows,
                     int pitch);
void launch_oz_split(const double* arena, const OzSplit* sp, int nsplit, int64_t max_rows,
                     uint16_t* planes, int64_t pstride, int pitch, int* sexp, cudaStream_t s);
// redo: update_tc64_redo_words(ntask) words of scratch
void launch_update_tc64(const CUtensorMap* maps, double* arena, const int* sexp, const OzTask* t,
                        int ntask, unsigned* redo, unsigned* err, cudaStream_t s);
size_t update_tc64_redo_words(int64_t ntask);

}  // namespace sylver_gb300
