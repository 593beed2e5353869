// Sliced contractions on tcgen05 (FP16 fixed-point slices, the Ozaki scheme):
// operand images, work descriptors and launchers.
//
// A contraction (P0 or Sigma) is a chain of three block GEMMs per V block:
//   stage 1   X1[(tau, L)][(x, y)] = sum_k  G[(tau, L)][k]   V1[(x, y)][k]
//   stage 2   X2[tau][(x, L)][z]   = sum_y  X1[tau][(x, L)][y]  B2[tau][z][y]
//   stage 3   C[(tau, x)][n]       = sum_(c, L, z) X2[(tau, x)][(c, L, z)]  V3[n][(c, L, z)]
// with, for P0:     L = m, x = P, y = t, z = p, n = Q, k = n',  B2 = G(k1, beta - tau)
//      for Sigma:   L = n, x = i, y = Q, z = P, n = j, k = m,   B2 = P~(tau).
//
// Every operand lives in memory as the image the tensor core reads: the row's
// value as NS FP16 slices (planes), K interleaved (re, im) in 32-byte steps of
// 8 complex ("octets"), 128 rows (A) or 16 rows per 8 complex columns (B, the
// real embedding) per step, in the 32-byte swizzle of the shared-memory matrix
// descriptors.  One image ("blob") covers at most OCT octets of K (one round:
// one exponent per row) and carries one scale per row behind the planes (NS = 3:
// an FP32 factor, NS = 6: an int32 exponent, so that the range is that of FP64):
//   A blob: [step][plane][128 rows][32 B], scale[128]
//   B blob: [step][plane][16 noct rows][32 B], scale[8 noct]
// so the GEMM moves blobs with bulk copies and does no work on its operands.
#pragma once

#include "common.h"

namespace gwgb {

constexpr int OZ_M = 128;   // rows per tile (TMEM lanes)
// X1 + X2 of one chunk, when that is at most an eighth of the free memory.
constexpr int64_t OZ_CHUNK_BYTES = 16ll << 30;

// Geometry of one slicing: NS planes; OCT octets (of 8 complex) per round and per column tile; NACC
// accumulators of slice products up to class CMAX, SETS sets of them in TMEM, each with a copy and an MMA warp
// and operand rings of its own; HO octets per drain thread;
// SEG K steps per operand copy (SEG3: in stage 3).
template <int NS> struct OzCfg;
template <> struct OzCfg<3> {  // 33-bit operands: the split-precision path
  static constexpr int OCT = 4, NACC = 4, CMAX = 3, SETS = 2, HO = 2, SEG = 2, SEG3 = 2;
};
template <> struct OzCfg<6> {  // 57-bit operands: the FP64 contractions
  static constexpr int OCT = 4, NACC = 7, CMAX = 6, SETS = 1, HO = 1, SEG = 1, SEG3 = 1;
};
constexpr int OZ_OCT = 4;

__host__ __device__ constexpr int64_t oz_abytes(int ns, int nks) { return (int64_t)ns * nks * 4096 + 512; }
// B blob bytes per octet of columns
__host__ __device__ constexpr int64_t oz_bbytes1(int ns, int nks) { return (int64_t)ns * nks * 512 + 32; }

// Stage 1: the images of one G block (all tau), row tile mt, round r at
// a + mt * (bytes of all rounds) + r * oz_abytes(full round).
struct OzS1 {
  int64_t a;
  int32_t M, nL;   // rows = n_tau * nL, row = tau * nL + L
  int32_t kos;     // octets of K
  int32_t pad;
};
// Stage-1 column tile: ngrp consecutive x of one contribution, gs octets of y each.
struct OzCol1 {
  int64_t b;       // its B blobs, rounds consecutive
  int32_t dst;     // OzDst1
  int32_t yoff;    // byte offset of the stage-2 round these columns are in
  int16_t x0;
  int8_t ngrp, gs;
  int32_t ny;      // valid y of this round
};
// Where the stage-1 output of a contribution goes: row slots of stage 2.  Blocks of four L, in each the x, in each x the
// L of the block: with Lq = L & ~3 and n = min(4, nLp - Lq),
//   slot = slot0 + Lq * nx + x * n + (L & 3)
// (slot0 a multiple of 4, nLp = nL padded to 2^glog), tile slot / 128 of base + (tau * nt2 + tile) * t2bytes.  A warp
// of the stage-1 drain (consecutive L) then writes whole 128-byte lines of four rows, and one of the stage-2 drain
// holds 8 x of 4 L, which are 8 neighbouring rows of 4 images; with the L of an x next to one another its 32 rows
// were 32 lines (stage 2 of Sigma, hexagonal 8 k: three slices 15.4 ms, with blocks of four 13.1; six slices, 4 k: 7.4, 5.95).
struct OzDst1 {
  int64_t base, t2bytes;
  int32_t nt2, slot0, nLp, nx;
};
// Stage 2: one pack (contributions that share the B2 operand and glog).
struct OzS2 {
  int64_t a, t2bytes;      // X1 images of the pack
  int64_t b, bt, bz;       // B2 images: b + tau * bt + (column tile) * bz
  int32_t nt2, kos, zos, glog;
  int32_t rows;            // first entry of the row map
  int32_t nz;              // valid z
};
// A row slot of stage 2: row tau * nx + x of the stage-3 image at base + (row / 128) * f16 * 16, octets of K from ks
// on; nks: octets of the image (glog > 0).
struct OzRow {
  int64_t base;
  int32_t f16;
  uint32_t pk;  // x | nx << 8 | ks << 16 | nks << 24; OZ_NOROW: empty
};
constexpr uint32_t OZ_NOROW = 0xffffffffu;
// Stage 3: one unit (a K slice of an output block).
struct OzS3 {
  int64_t a, fbytes;       // X2 images: a + f * fbytes + round offset
  int64_t b, bz;           // V3 images: b + (column tile) * bz + round offset * octets
  int64_t part;            // FP64 partial: part + tau * elems + n * sn + x * sx
  int32_t rt, nkr;         // rounds [rt, rt + nkr) of the round table
  int32_t M, N, nx, elems, sn, sx;
  int32_t oct, pad;        // octets per column tile
};
struct OzRnd { int32_t a16, b16, nks, pad; };  // byte offsets / 16 in the row tile and per octet of the column tile

// One CTA work item.  Stage 1: OzS1 d, column tile i, row tiles [m0, m0 + n);
// stage 2: pack d, i = tau | ztile << 16, row tiles [m0, m0 + n);
// stage 3: unit d, i = first row tile | column tile << 16, n row tiles (at most OCT / octets of the column tile).
struct OzTask { int32_t d, i, m0, n; };

// One operand image built from FP64 data: row r (r0 + local) at (r / rd) * rs1 + (r % rd) * rs0,
// valid when r % rd < rv and r / rd < rn; K index k at (k / kd) * ks1 + (k % kd) * ks0, valid likewise;
// kx >= 0: element k is multiplied by scale[kx + k] (powers of two).
struct OzBuild {
  int64_t src, dst;
  int64_t rs1, ks1;
  int32_t rs0, ks0, rd, kd, rv, kv, rn, kn, r0;
  int16_t rows, nks;       // rows of the image (complex), K octets
  int8_t isb, conj;
  int16_t pad;
  int32_t kx, pad2;
};

struct OzArgs {
  const void *desc;
  const OzTask *tasks;
  int ntasks;
  const void *aux1, *aux2;   // stage 1: OzCol1, OzDst1; stage 2: OzRow; stage 3: OzRnd
  const char *A, *B;
  char *X;                   // stages 1, 2: output images
  double2 *part;             // stage 3
  int nA, nB;                // operand rings of a set (segments of K steps); stages 1, 2: nB K steps of B per task,
  int tasksB;                // for one or two tasks
  int *err;
};

void set_oz_kernel_attributes();
// Ring sizes of a launch; max_kos: most octets of K of its tasks (stages 1 and 2).
void oz_rings(int ns, int stage, int max_kos, OzArgs *a);
// multi (stages 1 and 2): the tasks have more than one round of K.
void launch_oz_gemm(int ns, int stage, bool multi, const OzArgs &a, int nsm, cudaStream_t st);
// scale[i] = 2^-e and scale[nin + i] = 2^e with 2^(e-1) <= the largest finite component of row row0 + i over all slabs <
// 2^e, |e| at most 500; 1 and 0 for a row without one, so that its matrix elements do not set the scale of theirs.
void launch_oz_row_scale(const TSlab *slabs, int nslabs, const double2 *X, int row0, int nin, double *scale,
                         cudaStream_t st);
void launch_oz_build(int ns, const OzBuild *tasks, int64_t ntasks, const double2 *src, char *dst, cudaStream_t st,
                     const double *scale = nullptr);

}  // namespace gwgb
