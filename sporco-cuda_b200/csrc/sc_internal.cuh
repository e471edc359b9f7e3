// Internal structures shared by the solver kernels and the host driver.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/sporco_b200.h"
#include "sc_fft.cuh"

// Elements one thread holds during an FFT pass (see sc_fft.cuh).
#define SC_MAXE 16
// Threads per CTA of the row-pass kernels.
#define SC_ROW_THREADS 256
// Image columns (spectrum columns) per column-pass CTA.
#define SC_COL_TILE 4
// Largest column-pass CTA (SC_COL_TILE transforms of length <= 2048).
#define SC_COL_MAX_THREADS 512
// Row pass: radix-16 plans (16 elements per thread, 3 passes) for rows of
// 1024 and 2048, radix-8 plans for the other compile-time lengths.
__host__ __device__ constexpr int row_radix(int W) { return W == 1024 || W == 2048 ? 16 : 8; }
// Resident row-pass CTAs per SM the kernel is compiled for (register cap).
__host__ __device__ constexpr int row_min_blocks(int W) { return row_radix(W) == 16 ? 2 : 3; }
// Barrier scope of a row transform (group_sync): its own threads where they
// are whole warps or lie within one, else the CTA.
__host__ __device__ constexpr int row_barrier(int W) {
  if (W == 0) return 0;
  const int g = ct_threads(W, row_radix(W));
  if (g <= 32) return 32 % g == 0 ? 32 : 0;
  return g % 32 == 0 && 2 * g <= SC_ROW_THREADS ? g : 0;
}
// The row pass from the state V with register hand-over (sc_row.cuh): threads
// per CTA, resident CTAs per SM it is compiled for, barrier scope and shared
// memory of a transform group (its transform and one staging buffer for the
// pair's two spectrum rows or two state rows).  Measured at 2048 x 2048, 256
// maps: 4 / 5 / 6 CTAs of 128 threads per SM 4.12 / 4.0 / 3.93 ms (6: 80
// registers, 198 KB of shared memory); at 512 x 512, 100 maps: 6 / 7 / 8 / 9
// / 10 CTAs 114 / 108 / 101 / 114 / 116 us (8: 64 registers, more spill).
#define SC_ROWV_THREADS 128
__host__ __device__ constexpr bool rowv_len(int W) { return W >= 64 && ct_reg_edges(W, row_radix(W)); }
__host__ __device__ constexpr int rowv_min_blocks(int W) { return row_radix(W) == 16 ? 6 : 8; }
__host__ __device__ constexpr int rowv_barrier(int W) {
  const int g = ct_threads(W, row_radix(W));
  return g <= 32 ? 32 : g < SC_ROWV_THREADS ? g : 0;
}
__host__ __device__ constexpr int rowv_slot_bytes(int W) {
  return W * 8 + 2 * ((W / 2 + 1 + 3) & ~3) * 8;
}
// Shared memory of a transform group of the row pass at any other length.
__host__ __device__ inline size_t rowg_slot_bytes(int W, int Wp) {
  const size_t f = (size_t)2 * Wp * 8, v = ((size_t)2 * W * 4 + 15) / 16 * 16;
  return (size_t)((W + 1) & ~1) * 8 + (f > v ? f : v);
}
// Column pass: radix-16 plans (16 elements per thread) for long columns,
// radix-8 plans (8 per thread, twice the threads) for short ones.
__host__ __device__ constexpr int col_radix(int H) { return H >= 512 ? 16 : 8; }
// Shared memory that one CTA can have on sm_100a.
#define SC_SMEM_MAX (227 * 1024)
// Largest transform length this build supports along a row or a column.
#define SC_MAX_N 4096

// Float index of the real part of column k in a spectrum row in the paired
// layout, which F has between the convolution column pass and the row pass:
// columns 2 j and 2 j + 1 as (Re, Re, Im, Im), in every other group of eight
// pairs as (Im, Im, Re, Re), so that the real (imaginary) parts of 32
// consecutive columns lie in different banks.  The imaginary part is at index
// ^ 2.
__host__ __device__ constexpr int spec_re(int k) {
  return 4 * (k >> 1) + (k & 1) + ((k >> 3) & 2);
}

// Per-image ADMM scalar state, kept on the device for the whole solve.
struct ImgState {
  double rho;      // rho used by the next iteration
  double rho_prev; // rho of the last iteration (its Y: shrinkage of V at lambda / rho_prev)
  double rsf;    // scale factor chosen by the last adaptive-rho step (1: none)
  double uscale; // the next row pass reads U scaled by this (1 / rsf)
  double r, s;   // last residuals (normalised unless StdResiduals)
  double epri, edua;
  double nX, nY, nU;
  int k;         // iterations completed (over all solves of a warm-started state)
  int done;      // 1: converged, iteration cap reached, or failed
  int status;    // sc_status of this image
  int k0;        // k at the start of the current solve call (its cap counts from here)
  int paired;    // layout of F (RowParams::paired)
  int relay;     // F is in the other layout still (a warm start with another column
                 // pass): the fix-up at the start of the call writes it afresh
};

// What the workspace holds of the dictionary besides what every set-up leaves
// there (a flag word on the device; a solve that reuses the spectra, warm_start
// 2, makes what it needs and an earlier one did not): its 2-D spectrum, and
// Psum of map 0 and of the others apart.
enum { HELD_DICT = 1, HELD_SPLIT = 2 };

// Scalar options the finalize kernel needs.
struct FinParams {
  int max_iter;
  int auto_rho, period, auto_scaling, std_residuals;
  double rho_scaling, rsdl_ratio, abs_tol, rel_tol;
  double nelem;          // coefficients per image (M H W)
  const double* xi;      // (B,) residual ratio target per image
  double* itstat;        // (B, max_iter, SC_ITSTAT_FIELDS) or NULL
  int* ndone;            // images finished
};

// Geometry of one batch of equal-sized images.
struct Geom {
  int B;       // images
  int M;       // coefficient maps per image
  int H, W;
  int Wf;      // W/2 + 1 spectrum columns
  int Wp;      // spectrum row pitch (elements)
};

struct RowParams {
  Geom g;
  FftPlan pw;
  const float2* twW;
  int gsz;                 // threads per transform
  int nblk;                // CTAs per image (grid.x)
  float2* F;               // (B, M, H, Wp) spectra
  int paired;              // F in the paired layout (spec_re)
  int plain;               // ROW_ITER by row_kernel at every length (the unrolled solve)
  float* Y;                // (B, M, H, W)
  float* U;                // (B, M, H, W): U, or V = Y + U for ROW_ITER
  int vstate;              // ROW_FIXUP: P.U holds V (1) or U (0)
  float* Yo;               // ROW_ITER writes Y here (== Y unless a trace is kept)
  // epilogue
  const float* lam;        // (B,)
  int l1_kind;
  float l1_scalar;
  const float* l1w;
  const int32_t* mask;     // (B, H, W) or NULL
  int nonneg;              // NonNegCoef: Y >= 0
  int bnd_r, bnd_c;        // NoBndryCross: rows >= bnd_r and columns >= bnd_c
                           // of every map are zero (H, W: none)
  float relax;
  float invN;              // 1 / (H W)
  int delta;               // ROW_ITER*: F holds the column pass's correction only,
                           // X = (Y - U) + IFFTrow(F) / (H W) (CONV_DELTA)
  double* partials;        // (B, nblk, 5)
  ImgState* st;            // (B,)
  // setup / tool modes
  const float* src;        // real rows (B, M, H, W) for ROW_FWD_REAL
  const float* D;          // (M, Kr, Kc) for ROW_FWD_DICT
  int Kr, Kc;
  const int* held;         // ROW_FWD_DICT: nothing to do if *held has HELD_DICT (or NULL)
  float* dst;              // real rows out for ROW_INV_REAL
  // adjoint (ROW_ADJ)
  float* gV;               // (B, M, H, W) gradient w.r.t. V of the step, in place
  const float* Ymask;      // (B, M, H, W) Y the step produced (nonzero: shrinkage active),
                           // or with vmask its V (active: the shrinkage of V is nonzero)
  int vmask;
  float* Vo;               // ROW_ITER: V written here (NULL: in place, into U)
  int first;               // 1: gV holds dLoss/dY of the last iterate, no Q yet
};

struct ColParams {
  Geom g;
  FftPlan ph;
  const float2* twH;
  const float2* twW;
  int gsz;                 // threads per transform (column)
  int G;                   // CTAs (cluster ranks) sharing one column tile
  int Hs;                  // shared-memory column stride (elements)
  int tile0;               // column tile of blockIdx.y = 0 (a launch over part of the tiles)
  float2* F;               // (B, M, H, Wp)
  const float2* Dh;        // (M, H, Wp)
  const float2* Sh;        // (B, H, Wp)
  int grd;
  float mu;
  const float* wgrd;       // (M,)
  const float* Psum;       // (H, Wp) sum_m |Df_m|^2 (solve with one d for all maps)
  const float* E;          // (M, Ep, Wp / 2, 8): row spectra e of the filter rows, zero rows
                           // from Kr on, as column pairs (Re e, Re e + Im e, Im e - Re e,
                           // Im e) x 2
  int Kr;                  // filter rows
  int Ep;                  // rows of E per map (conv_pad_taps(Kr))
  int two;                 // CONV_GRAD: the gradient weight of map 0 is zero
  const double2* twHd;     // column twiddles in double precision (COL_CONV, any length)
  const float* Psum0;      // (H, Wp) |Df_0|^2 (two; Psum is then over the other maps)
  const int* held;         // COL_FWD: nothing to do if *held has HELD_DICT (or NULL)
  ImgState* st;
  float2* Xtr;             // COL_SOLVE_X: x^ also written here (B, M, H, Wp); COL_SOLVE_C*T:
                           // the row spectra of X (or NULL)
  // adjoint (COL_ADJ)
  const float2* Xh;        // (B, M, H, Wp) x^ of the step (COL_ADJ_C*: the row spectra of X)
  float2* gDh;             // (B, M, H, Wp) dictionary-gradient spectra, accumulated
  float2* gSh;             // (B, H, Wp) signal-gradient spectra, accumulated
  // convolution-form adjoint
  float2* SCtr;            // (B, H, Wp) IFFTcol(S^ - cb) / rho of the step (written by
                           // COL_SOLVE_C*T unless NULL, read by COL_ADJ_C*)
  float2* gE;              // (B, M, Kr, Wp) dictionary gradient as filter-row spectra
};

enum RowMode {
  ROW_ITER = 0, ROW_FWD_REAL = 1, ROW_FWD_DICT = 2, ROW_INV_REAL = 3, ROW_FIXUP = 4,
  ROW_FWD_YU = 5, // row spectra of Y - U (start from given iterates)
  ROW_ADJ = 6,    // adjoint step: Q = row IFFT, gV update, row FFT of relax * gV
  ROW_ITER_D = 8, // ROW_ITER with F the column pass's correction to Y - U (CONV_DELTA)
  ROW_ITER_YU = 7 // ROW_ITER with Y and U stored separately (warm starts, the
                  // adjoint's recomputation, which keeps Y of every step)
};
// COL_SOLVE: all maps share d (cbpdn, or cbpdngrd with one GradWeight), so
// sum_m |Df_m|^2 / d comes from the precomputed Psum; COL_SOLVE_W: per-map
// d_m = mu w_m |G|^2 + rho, the sum is accumulated over the maps.
// COL_SOLVE_P: the solve with d = rho for every map and frequency (cbpdn,
// cbpdnmsk), without the write-back of the column spectra between its two
// passes.  COL_CONV: the convolution column pass (colc_kernel, sc_col.cuh; its
// kinds are ConvKind), for filters of at most 16 rows.  COL_SOLVE_G16: the
// gradient term with one weight of unknown or negative sign, in convolution
// form with two transforms per map.  COL_SOLVE_X: COL_SOLVE that also writes
// x^ to ColParams::Xtr (the recomputation inside the adjoint).  COL_ADJ:
// adjoint of the plain cbpdn solve (one d = rho): column FFT, Q^ = A^{-1} G^,
// gradient accumulation, inverse column FFT.  COL_ADJ_C8 / COL_ADJ_C16: the
// same in convolution form (the dictionary gradient accumulated as
// correlations over the Kr filter rows, ColParams::gE).  COL_SOLVE_C8T /
// COL_SOLVE_C16T: the plain solve in convolution form of the unrolled solve,
// which can keep ColParams::Xtr (the row spectra of X) and SCtr.  The unrolled
// solve keeps to these kernels and to row_kernel: the gradients jump where a
// coefficient lies within rounding of its threshold, so that kernels with
// another order of the same sums (a last-bit change of the iterates, 5e-7 of X)
// moved them by 1e-4 to 5e-3 on one training problem in three.
enum ColMode {
  COL_SOLVE = 0, COL_FWD = 1, COL_INV = 2, COL_SOLVE_W = 3, COL_ADJ = 4, COL_SOLVE_X = 5,
  COL_SOLVE_P = 6, COL_CONV = 7, COL_SOLVE_G16 = 9, COL_SOLVE_C8T = 10, COL_SOLVE_C16T = 11,
  COL_ADJ_C8 = 12, COL_ADJ_C16 = 13
};
// Filter rows (taps) of the convolution modes of col_kernel.
__host__ __device__ constexpr int col_taps(int mode) {
  return mode == COL_ADJ_C8 || mode == COL_SOLVE_C8T ? 8
         : mode == COL_SOLVE_G16 || mode == COL_ADJ_C16 || mode == COL_SOLVE_C16T ? 16
                                                                                  : 0;
}
// The convolution-form adjoint.
__host__ __device__ constexpr bool col_adj_conv(int mode) {
  return mode == COL_ADJ_C8 || mode == COL_ADJ_C16;
}
// Modes that launch as a cluster over the maps of one column tile.
__host__ __device__ constexpr bool col_clustered(int mode) {
  return mode == COL_SOLVE || mode == COL_SOLVE_W || mode == COL_SOLVE_X || mode == COL_ADJ ||
         mode == COL_SOLVE_P || col_taps(mode) > 0;
}

// ------------------------------------------- convolution column pass (sc_col.cuh)
enum ConvKind { CONV_DELTA = 0, CONV_FULL = 1, CONV_GRAD = 2 };
// Rows per thread at column lengths without a compiled transform: odd, so that
// the tile needs no padding; up to SC_CONV_ANY_H rows.
#define SC_CONV_ANY_L 9
#define SC_CONV_ANY_H 1024
// Taps a filter of Kr <= 16 rows is padded to.
__host__ __device__ constexpr int conv_pad_taps(int Kr) { return Kr <= 8 ? 8 : Kr <= 12 ? 12 : 16; }
// Rows per thread at the compiled length n: the default, and the alternative
// the autotuner tries (0: none).
__host__ __device__ constexpr int conv_rows(int n) {
  return n == 0 ? SC_CONV_ANY_L : n == 48 ? 6 : n <= 128 ? 4 : n >= 1536 ? 16 : 8;
}
__host__ __device__ constexpr int conv_rows_alt(int n) {
  return n == 512 || n == 768 || n == 1024 ? 16 : 0;
}
__host__ __device__ constexpr int conv_threads(int n, int L) { return n > 0 ? 2 * n / L : 256; }
// Threads at a length without a compiled transform: two per block of rows, and
// at least a sixteenth of the column for each of its four transforms.
inline int conv_threads_any(int H) {
  const int a = 2 * ((H + SC_CONV_ANY_L - 1) / SC_CONV_ANY_L), b = (H + 3) / 4;
  return ((a > b ? a : b) + 31) & ~31;
}
// Radix of the tile's column transforms.
__host__ __device__ constexpr int conv_radix(int n) { return n >= 192 ? 16 : 8; }
// Taps per sweep over the window (their entries stay in registers).
__host__ __device__ constexpr int conv_sweep(int KR, int L) { return KR == 16 ? 8 : KR; }
// Complex products in Gauss's form (three packed FMAs) or plainly (four); both
// measured: 256 x 256, 8 taps 17.7 / 18.5 us, 512 x 512, 12 taps 99 / 108 us,
// 2048 x 2048, 16 taps 2.95 / 3.25 ms, 64 x 64, 8 taps 8.0 / 7.5 us, 320 rows
// (not compiled) 78.3 / 78.6 us.
__host__ __device__ constexpr bool conv_gauss(int n) { return n > 128; }
// Resident CTAs per SM the kernel is compiled for: as many as its registers
// (three packed sums per row, three packed entries per tap; two of each without
// Gauss's form) leave room for.
// (At a length without a compiled transform two, with the gradient term's
// recursions one: 320 rows 78 us with two, 109 with one.)
__host__ __device__ constexpr int conv_min_blocks(int kind, int n, int L, int KR) {
  if (n == 0) return kind == CONV_GRAD ? 1 : 2;
  const int nt = (conv_threads(n, L) + 31) / 32 * 32;
  const int regs = (conv_gauss(n) ? 6 : 4) * (L + conv_sweep(KR, L)) + 56;
  const int b = 65536 / (nt * (regs < 255 ? regs : 255));
  return b < 1 ? 1 : b > 16 ? 16 : b;
}
__host__ __device__ constexpr int conv_slots(int H, int L) { return L & 1 ? H : H + H / L; }
// Shared memory of one CTA: three tiles of four columns (at least one map's
// filter rows each), three maps' filter rows, the gradient term's carries
// and their weights, and map 0's tile.
__host__ __device__ inline size_t conv_tile_entries(int H, int L, int KR) {
  const size_t a = (size_t)4 * conv_slots(H, L), b = (size_t)KR * 8;
  return a > b ? a : b;
}
__host__ __device__ inline size_t conv_smem_bytes(int kind, int H, int L, int KR, int NT, int two) {
  const size_t tl = conv_tile_entries(H, L, KR) * 8;
  return 3 * tl + (size_t)3 * KR * 64 +
         (kind == CONV_GRAD ? (size_t)NT * (4 * 16 + (L & 1 ? 16 : 8)) : 0) + (two ? tl : 0);
}

// Whether the convolution column pass of that kind fits (its default variant):
// every length does but 2048 rows with map 0 apart, whose four tiles take 296 KB.
inline bool conv_fits(int kind, int H, bool compiled, int Kr, bool two) {
  const int n = compiled ? H : 0, L = conv_rows(n);
  const int NT = compiled ? conv_threads(n, L) : conv_threads_any(H);
  return conv_smem_bytes(kind, H, L, conv_pad_taps(Kr), NT, two) <= SC_SMEM_MAX;
}

__host__ __device__ inline size_t sc_align16(size_t x) { return (x + 15) & ~(size_t)15; }

// Shared memory of one row-pass slot (one row pair in flight); zlen is the
// (padded) number of shared-memory slots of one row transform.  The
// iteration mode stages the next pair's two spectrum rows and the pair's Y
// and U rows: [z: zlen complex][F: 2Wp complex][Y: 2W][U: 2W]; the adjoint
// step stages gV and the shrinkage mask source in the Y and U places, the
// rho fix-up the pair's U rows and spectrum rows.
__host__ __device__ inline size_t row_slot_bytes(int mode, int zlen, int W, int Wp) {
  size_t z = sc_align16((size_t)zlen * 8);
  if (mode != ROW_ITER && mode != ROW_ITER_YU && mode != ROW_ADJ && mode != ROW_FIXUP) return z;
  // staged spectrum rows, then one staged real row pair (V for ROW_ITER, the
  // state for ROW_FIXUP) or two (Y and U, gV and the mask source)
  const int nreal = mode == ROW_ITER || mode == ROW_FIXUP ? 1 : 2;
  return z + (size_t)(2 * Wp) * 8 + nreal * sc_align16((size_t)(2 * W) * 4);
}

// Shared memory of one column-pass CTA; hlen is the (padded) number of
// shared-memory slots of one column transform.  A tile is SC_COL_TILE
// interleaved columns.  The solve double-buffers the spectrum
// tile and stages the dictionary tile: [F0][F1][D]; the cluster reduction
// reuses [F1][D].  The convolution modes use three tiles and three staged
// filter-row tiles (16 bytes an entry); the convolution adjoint two more tiles (the forward's
// SC trace and row spectra of X) and per-warp partial sums of the
// dictionary gradient for its nt threads (two maps).
__host__ __device__ inline size_t col_smem_bytes(int mode, int hlen, int nt = SC_COL_MAX_THREADS) {
  const int tw = SC_COL_TILE;
  const size_t tile = (size_t)tw * hlen * 8;
  return (col_clustered(mode) ? (col_adj_conv(mode) ? 5 : 3) * tile : tile) +
         (size_t)3 * col_taps(mode) * tw * 16 +
         (col_adj_conv(mode) ? (size_t)2 * (nt / 32) * col_taps(mode) * tw * 8 : 0);
}
