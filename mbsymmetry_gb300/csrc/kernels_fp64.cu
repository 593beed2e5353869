// FP64 kernels of the GW engine: block rotations, the P0 and Sigma
// contractions, the tau <-> omega transforms and the batched block inverses.
//
// GB300's FP64 rate is a small fraction of its tensor rate, so these kernels
// are FP64-pipe bound: they keep the reference's three-GEMM contraction
// order (no redundant flops), keep every SM busy with owner-computes tiles
// (one CTA owns an output block for a tau range and sums all its (k, q, s)
// contributions, so no atomics and bitwise run-to-run reproducibility), and
// stage the per-contribution intermediates in shared memory.
#include "common.h"
#include "kernels.h"

#include <algorithm>

namespace gwgb {

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// c + a * b
__device__ __forceinline__ double2 cfma(double2 a, double2 b, double2 c) {
  c.x = fma(a.x, b.x, c.x);
  c.x = fma(-a.y, b.y, c.x);
  c.y = fma(a.x, b.y, c.y);
  c.y = fma(a.y, b.x, c.y);
  return c;
}
// c + conj(a) * b
__device__ __forceinline__ double2 cfma_conja(double2 a, double2 b, double2 c) {
  c.x = fma(a.x, b.x, c.x);
  c.x = fma(a.y, b.y, c.x);
  c.y = fma(a.x, b.y, c.y);
  c.y = fma(-a.y, b.x, c.y);
  return c;
}
// c - a * b, the product first: three instructions a component.  Two, fma(-a.x, b.x, fma(a.y, b.y, c.x)), round twice at
// the size of c; in the eliminations below that makes the error of the inverses 12 to 26% larger.
__device__ __forceinline__ double2 csub(double2 c, double2 a, double2 b) {
  return make_double2(c.x - fma(a.x, b.x, -(a.y * b.y)), c.y - fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }

// ---------------------------------------------------------------------------
// P0 contraction (restates gw_block.cpp:52-75 / cugw_qkpt_block.cu:195-267):
//   X1[t,m][Q] = sum_p G^{k1}(beta - tau)[t][p] V[Q][p][m]
//   X2[P][t,m] = sum_n conj(V[P][t][n]) G^{k2}(tau)[m][n]
//   P0(tau)[Q][P] += sum_{t,m} X1[t,m][Q] X2[P][t,m]
// The t (row of the k1 block) range is processed in chunks so the
// intermediates of any block size fit in shared memory.  A tile sums one
// slice of the block's contributions into its own partial block; the slices
// are added in a fixed order by reduce_slices_kernel.
// ---------------------------------------------------------------------------
template <int MAXO>
__global__ void __launch_bounds__(256, 2) p0_fp64_kernel(const P0Tile *__restrict__ tiles,
                                                         const P0Contrib *__restrict__ contribs,
                                                         const double2 *__restrict__ V,
                                                         const double2 *__restrict__ G,
                                                         double2 *__restrict__ Part, int ns, int nts,
                                                         int smem_cap) {
  extern __shared__ double2 sm[];
  const P0Tile tile = tiles[blockIdx.x];
  const int qb = tile.qb, nt = tile.nt;
  const int nout = nt * qb * qb;
  double2 acc[MAXO];
#pragma unroll
  for (int i = 0; i < MAXO; ++i) acc[i] = make_double2(0.0, 0.0);

  for (int c = tile.c0; c < tile.c1; ++c) {
    const P0Contrib cb = contribs[c];
    const int b1 = cb.b1, b2 = cb.b2;
    const double2 *Vb = V + cb.v;
    int TT = smem_cap / (2 * qb * b2 * nt);
    TT = TT < b1 ? TT : b1;
    for (int s = 0; s < ns; ++s) {
      for (int r0 = 0; r0 < b1; r0 += TT) {
        const int tn = (b1 - r0) < TT ? (b1 - r0) : TT;
        const int K = tn * b2;
        double2 *X1 = sm;
        double2 *X2 = sm + (size_t)nt * qb * K;
        __syncthreads();
        for (int e = threadIdx.x; e < nt * qb * K; e += blockDim.x) {
          const int it = e / (qb * K);
          const int rem = e - it * qb * K;
          const int Q = rem / K, k = rem - Q * K;
          const int tt = k / b2, m = k - tt * b2;
          const int tau = tile.t0 + it;
          const double2 *Gm = G + cb.ga + ((size_t)(nts - 1 - tau) * ns + s) * cb.sa + (size_t)(r0 + tt) * b1;
          const double2 *Vq = Vb + (size_t)Q * b1 * b2 + m;
          double2 a = make_double2(0.0, 0.0);
          for (int p = 0; p < b1; ++p) a = cfma(Gm[p], Vq[(size_t)p * b2], a);
          X1[(size_t)(it * qb + Q) * K + k] = a;
        }
        for (int e = threadIdx.x; e < nt * qb * K; e += blockDim.x) {
          const int it = e / (qb * K);
          const int rem = e - it * qb * K;
          const int P = rem / K, k = rem - P * K;
          const int tt = k / b2, m = k - tt * b2;
          const int tau = tile.t0 + it;
          const double2 *G2 = G + cb.gb + ((size_t)tau * ns + s) * cb.sb + (size_t)m * b2;
          const double2 *Vr = Vb + ((size_t)P * b1 + r0 + tt) * b2;
          double2 a = make_double2(0.0, 0.0);
          for (int n = 0; n < b2; ++n) a = cfma_conja(Vr[n], G2[n], a);
          X2[(size_t)(it * qb + P) * K + k] = a;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < MAXO; ++i) {
          const int o = threadIdx.x + i * blockDim.x;
          if (o < nout) {
            const int it = o / (qb * qb);
            const int rem = o - it * qb * qb;
            const int Q = rem / qb, P = rem - Q * qb;
            const double2 *x1 = X1 + (size_t)(it * qb + Q) * K;
            const double2 *x2 = X2 + (size_t)(it * qb + P) * K;
            double2 a = acc[i];
            for (int k = 0; k < K; ++k) a = cfma(x1[k], x2[k], a);
            acc[i] = a;
          }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < MAXO; ++i) {
    const int o = threadIdx.x + i * blockDim.x;
    if (o < nout) Part[tile.part + o] = acc[i];
  }
}

// ---------------------------------------------------------------------------
// Sigma contraction (restates gw_block.cpp:128-151 / cugw_qkpt_block.cu:343-412):
//   Y1[Q][i][n] = sum_m V[Q][i][m] G^{k2}(tau)[m][n]
//   Y2[i][n][P] = sum_Q Y1[Q][i][n] P(tau)[Q][P]
//   Sigma(tau)[i][j] += sum_{n,P} Y2[i][n][P] conj(V[P][j][n])
// The n range is processed in chunks so the intermediates fit in shared memory.
// Like P0, a tile writes the partial sum of one slice of the contributions.
// ---------------------------------------------------------------------------
template <int MAXO>
__global__ void __launch_bounds__(256, 2) sigma_fp64_kernel(const SigTile *__restrict__ tiles,
                                                            const SigContrib *__restrict__ contribs,
                                                            const double2 *__restrict__ V,
                                                            const double2 *__restrict__ G,
                                                            const double2 *__restrict__ P,
                                                            double2 *__restrict__ Part, int ns, int smem_cap) {
  extern __shared__ double2 sm[];
  const SigTile tile = tiles[blockIdx.x];
  const int b1 = tile.b1, nt = tile.nt, s = tile.s;
  const int nout = nt * b1 * b1;
  double2 acc[MAXO];
#pragma unroll
  for (int i = 0; i < MAXO; ++i) acc[i] = make_double2(0.0, 0.0);

  for (int c = tile.c0; c < tile.c1; ++c) {
    const SigContrib cb = contribs[c];
    const int qb = cb.qb, b2 = cb.b2;
    const double2 *Vb = V + cb.v;
    int NT = smem_cap / (2 * qb * b1 * nt);
    NT = NT < b2 ? NT : b2;
    for (int n0 = 0; n0 < b2; n0 += NT) {
      const int nn_n = (b2 - n0) < NT ? (b2 - n0) : NT;
      double2 *Y1 = sm;                                  // [nt][qb][b1][nn]
      double2 *Y2 = sm + (size_t)nt * qb * b1 * nn_n;    // [nt][b1][nn][qb]
      __syncthreads();
      for (int e = threadIdx.x; e < nt * qb * b1 * nn_n; e += blockDim.x) {
        const int it = e / (qb * b1 * nn_n);
        int rem = e - it * qb * b1 * nn_n;
        const int Q = rem / (b1 * nn_n);
        rem -= Q * b1 * nn_n;
        const int i = rem / nn_n, nn = rem - i * nn_n;
        const int tau = tile.t0 + it;
        const double2 *G2 = G + cb.gb + ((size_t)tau * ns + s) * cb.sb + n0 + nn;
        const double2 *Vr = Vb + ((size_t)Q * b1 + i) * b2;
        double2 a = make_double2(0.0, 0.0);
        for (int m = 0; m < b2; ++m) a = cfma(Vr[m], G2[(size_t)m * b2], a);
        Y1[e] = a;
      }
      __syncthreads();
      for (int e = threadIdx.x; e < nt * b1 * nn_n * qb; e += blockDim.x) {
        const int it = e / (b1 * nn_n * qb);
        int rem = e - it * b1 * nn_n * qb;
        const int i = rem / (nn_n * qb);
        rem -= i * nn_n * qb;
        const int nn = rem / qb, Pi = rem - nn * qb;
        const int tau = tile.t0 + it;
        const double2 *Pt = P + cb.pq + (size_t)tau * cb.pstride + Pi;
        const double2 *y1 = Y1 + ((size_t)it * qb * b1 + i) * nn_n + nn;
        double2 a = make_double2(0.0, 0.0);
        if (cb.pconj)  // P~(q) of a time-reversal partner: conj(P~(q'))
          for (int Q = 0; Q < qb; ++Q) a = cfma(y1[(size_t)Q * b1 * nn_n], cconj(Pt[(size_t)Q * qb]), a);
        else
          for (int Q = 0; Q < qb; ++Q) a = cfma(y1[(size_t)Q * b1 * nn_n], Pt[(size_t)Q * qb], a);
        Y2[e] = a;
      }
      __syncthreads();
#pragma unroll
      for (int ii = 0; ii < MAXO; ++ii) {
        const int o = threadIdx.x + ii * blockDim.x;
        if (o < nout) {
          const int it = o / (b1 * b1);
          const int rem = o - it * b1 * b1;
          const int i = rem / b1, j = rem - i * b1;
          const double2 *y2 = Y2 + ((size_t)it * b1 + i) * nn_n * qb;
          double2 a = acc[ii];
          for (int nn = 0; nn < nn_n; ++nn) {
            const double2 *vc = Vb + (size_t)j * b2 + n0 + nn;
            for (int Pi = 0; Pi < qb; ++Pi)
              a = cfma(y2[nn * qb + Pi], cconj(vc[(size_t)Pi * b1 * b2]), a);
          }
          acc[ii] = a;
        }
      }
    }
  }
#pragma unroll
  for (int ii = 0; ii < MAXO; ++ii) {
    const int o = threadIdx.x + ii * blockDim.x;
    if (o < nout) Part[tile.part + o] = acc[ii];
  }
}

// Fixed-order sum of the slices (deterministic), scaled, into P0 or Sigma.
__global__ void reduce_slices_kernel(const RedTask *__restrict__ tasks, const double2 *__restrict__ part,
                                     double2 *__restrict__ out, int nts, double scale, int mirror) {
  const RedTask tk = tasks[blockIdx.x];
  const int n = tk.nt * tk.elems;
  for (int o = blockIdx.y * blockDim.x + threadIdx.x; o < n; o += gridDim.y * blockDim.x) {
    double2 a = part[tk.part + o];
    for (int sl = 1; sl < tk.nslice; ++sl) a = cadd(a, part[tk.part + (int64_t)sl * n + o]);
    const int it = o / tk.elems, e = o - it * tk.elems;
    const int tau = tk.t0 + it;
    const double2 v = cscale(a, scale);
    out[tk.out + (int64_t)tau * tk.ostride + e] = v;
    if (mirror) out[tk.out + (int64_t)(nts - 1 - tau) * tk.ostride + e] = v;
  }
}

// ---------------------------------------------------------------------------
// Pre-rotated V of the Sigma contributions: Vt[Q'][x] = sum_Q op(O[Q][Q']) V[Q][x]
// (op = conj for a time-reversal partner; o < 0: a copy), once per V / rep
// upload.  One CTA per contribution block.
// ---------------------------------------------------------------------------
__global__ void vrot_kernel(const VrTask *__restrict__ tasks, const double2 *__restrict__ V,
                            const double2 *__restrict__ O, double2 *__restrict__ Vt) {
  const VrTask t = tasks[blockIdx.x];
  const int qb = t.qb, n = t.b1b2;
  const double2 *v = V + t.v;
  double2 *out = Vt + t.vt;
  if (t.o < 0) {
    for (int e = threadIdx.x; e < qb * n; e += blockDim.x) out[e] = v[e];
    return;
  }
  const double2 *o = O + t.o;
  for (int e = threadIdx.x; e < qb * n; e += blockDim.x) {
    const int Qp = e / n, x = e - Qp * n;
    double2 a = make_double2(0.0, 0.0);
    if (t.conj)
      for (int Q = 0; Q < qb; ++Q) a = cfma(cconj(o[Q * qb + Qp]), v[(size_t)Q * n + x], a);
    else
      for (int Q = 0; Q < qb; ++Q) a = cfma(o[Q * qb + Qp], v[(size_t)Q * n + x], a);
    out[e] = a;
  }
}

// ---------------------------------------------------------------------------
// Block rotation dst = O src O^H (+conj), or slice copy (+conj); restates
// cugw_routines_block.cu:134-186 (G) and cugw_qkpt_block.cu:288-340 (P).
// grid = (tasks, batch)
// ---------------------------------------------------------------------------
__global__ void rotate_kernel(const RotTask *__restrict__ tasks, const double2 *__restrict__ src,
                              const double2 *__restrict__ O, double2 *__restrict__ dst) {
  extern __shared__ double2 sm[];
  const RotTask t = tasks[blockIdx.x];
  const double2 *s = src + t.src + (size_t)blockIdx.y * t.sstride;
  double2 *d = dst + t.dst + (size_t)blockIdx.y * t.dstride;
  if (!t.rotate) {
    for (int i = threadIdx.x; i < t.m; i += blockDim.x) d[i] = t.conj ? cconj(s[i]) : s[i];
    return;
  }
  const int m = t.m, n = t.n;
  double2 *Os = sm;               // m x n
  double2 *X = sm + m * n;        // n x n
  double2 *T = X + n * n;         // m x n
  const double2 *Og = O + t.o;
  for (int i = threadIdx.x; i < m * n; i += blockDim.x) Os[i] = Og[i];
  for (int i = threadIdx.x; i < n * n; i += blockDim.x) X[i] = s[i];
  __syncthreads();
  for (int e = threadIdx.x; e < m * n; e += blockDim.x) {
    const int i = e / n, j = e - i * n;
    double2 a = make_double2(0.0, 0.0);
    for (int p = 0; p < n; ++p) a = cfma(Os[i * n + p], X[p * n + j], a);
    T[e] = a;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < m * m; e += blockDim.x) {
    const int i = e / m, j = e - i * m;
    double2 a = make_double2(0.0, 0.0);
    for (int p = 0; p < n; ++p) a = cfma(T[i * n + p], cconj(Os[j * n + p]), a);
    d[e] = t.conj ? cconj(a) : a;
  }
}

// P0(beta - t) = P0(t) (cugw_solver_block.cpp:441-456); grid over q, threads over elements.
__global__ void mirror_kernel(double2 *__restrict__ P, const int64_t *__restrict__ qoff,
                              const int32_t *__restrict__ qsz, int nts) {
  const int q = blockIdx.x;
  const int64_t base = (int64_t)nts * qoff[q];
  const int sz = qsz[q];
  const int half = nts / 2;
  for (int64_t e = (int64_t)blockIdx.y * blockDim.x + threadIdx.x; e < (int64_t)half * sz;
       e += (int64_t)gridDim.y * blockDim.x) {
    const int t = (int)(e / sz);
    const int i = (int)(e - (int64_t)t * sz);
    P[base + (int64_t)(nts - 1 - t) * sz + i] = P[base + (int64_t)t * sz + i];
  }
}

// Zero rows t >= nts/2 of every P0 slice (state left by solve_P0).
__global__ void zero_upper_kernel(double2 *__restrict__ P, const int64_t *__restrict__ qoff,
                                  const int32_t *__restrict__ qsz, int nts) {
  const int q = blockIdx.x;
  const int64_t base = (int64_t)nts * qoff[q];
  const int sz = qsz[q];
  const int half = nts / 2;
  for (int64_t e = (int64_t)blockIdx.y * blockDim.x + threadIdx.x; e < (int64_t)(nts - half) * sz;
       e += (int64_t)gridDim.y * blockDim.x)
    P[base + (int64_t)half * sz + e] = make_double2(0.0, 0.0);
}

// ---------------------------------------------------------------------------
// tau <-> omega transform (transformer_t.h:66-99, 226-308):
//   Y[slab][r][c] = sum_i T[r][i] X[slab][row0 + i][c],  r < nout, i < nin.
// One CTA = 32 columns x 8R output rows (R per warp, rows r0 + warp*R + j),
// grid = (slab, column tile, row tile).  The T rows of the tile are staged
// through shared memory in 32-wide chunks of i.  Warps whose rows all lie
// beyond nout skip the arithmetic (the FP64 pipe is the bound).
// ---------------------------------------------------------------------------
constexpr int TR_MAXOUT = 160;  // nout limit of the engine's grids
template <int R>
__global__ void __launch_bounds__(256) transform_kernel(const TSlab *__restrict__ slabs,
                                                        const double2 *__restrict__ T, int nout,
                                                        int nin, int row0,
                                                        const double2 *__restrict__ X,
                                                        double2 *__restrict__ Y) {
  __shared__ double2 Ts[8 * R][33];
  const TSlab sl = slabs[blockIdx.x];
  const int cl = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int c = blockIdx.y * 32 + cl;
  const int r0 = blockIdx.z * 8 * R;
  const int nr = min(8 * R, nout - r0);
  const bool active = c < sl.ncols && w * R < nr;
  double2 acc[R];
#pragma unroll
  for (int j = 0; j < R; ++j) acc[j] = make_double2(0.0, 0.0);
  const double2 *x = X + sl.x + (int64_t)row0 * sl.ldx + c;
  for (int i0 = 0; i0 < nin; i0 += 32) {
    const int ni = (nin - i0) < 32 ? (nin - i0) : 32;
    __syncthreads();
    for (int e = threadIdx.x; e < nr * 32; e += 256) {
      const int r = e >> 5, ii = e & 31;
      Ts[r][ii] = (ii < ni) ? T[(int64_t)(r0 + r) * nin + i0 + ii] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    if (active) {
      for (int ii = 0; ii < ni; ++ii) {
        const double2 xv = x[(int64_t)(i0 + ii) * sl.ldx];
#pragma unroll
        for (int j = 0; j < R; ++j) acc[j] = cfma(Ts[w * R + j][ii], xv, acc[j]);
      }
    }
  }
  if (active) {
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int rl = w * R + j;
      if (rl < nr) Y[sl.y + (int64_t)(r0 + rl) * sl.ldy + c] = acc[j];
    }
  }
}

// ---------------------------------------------------------------------------
// Batched block inverses.  An exactly singular block sets *bad and leaves its
// output untouched.
//   mode 0 (W~ solve, cugw_solver_block.cpp:412-424):
//     A = I - (P + P^H)/2 ; A^-1 ; R = (A^-1 + A^-H)/2 ; P <- R P
//   mode 1 (Dyson, sc_type_block.cpp:48-57):
//     A = (i w_n + mu) S - F - Sigma(i w_n) ; G = A^-1   (in place)
// Bound: the FP64 pipe (2 FMA per cycle and SM; a DFMA of one warp takes 64 cycles
// of its scheduler), so what counts is the number of FP64 instructions:
//  - the A of mode 0 is Hermitian and, at bosonic frequencies, positive definite: symmetric sweeps over its
//    lower triangle, no pivot search (3 n^3 instructions against 6 n^3 and the search).  A pivot that is not clearly
//    positive sends the block to the general elimination;
//  - the general one is Gauss-Jordan with full pivoting (the strategy of Eigen::FullPivLU,
//    sc_type_block.cpp:55), 6 instructions per element and step; the pivot is the element of
//    largest modulus to 20 bits, found in integers and FP32 while the elimination writes the elements (the largest
//    component instead made Dyson's error up to 12% larger).
// One warp per matrix up to n = 16, a CTA of 128 threads up to 32, of 256 above (NT), elements spread over the threads.
// Measured, with one general elimination per warp or CTA of 128 and now: W~ s+p+d+4 (aux 9-46) 3.36 and 1.53 ms,
// hexagonal 8 k (aux 2-30) 3.15 and 0.95; Dyson there (AO 2-30) 0.61 and 0.26; s+p (n up to 12), both solves, 0.17 and 0.075.
// With 4 instead of 6 instructions per element (csub) 1.33, 0.83, 0.20 and 0.071, at an error 12 to 26% larger.  Tried
// and slower: the product R P from one triangle (R commutes with the Hermitian part of P), the rest in FP32.
// ---------------------------------------------------------------------------
template <int NT> __device__ __forceinline__ void inv_sync() {
  if constexpr (NT == 32)
    __syncwarp();
  else
    __syncthreads();
}

// Size of an element for the pivot choice: |v|^2 to 20 bits as an ordered integer, from the upper words in FP32 (the
// FP64 pipe bounds the elimination).  0 for NaN and for what underflows when squared.
__device__ __forceinline__ unsigned inv_key(double2 v) {
  const unsigned x = (unsigned)__double2hiint(v.x) & 0x7fffffffu, y = (unsigned)__double2hiint(v.y) & 0x7fffffffu;
  const unsigned k = max(x, y), s = min(x, y), e = k >> 20, d = e - (s >> 20);
  if (k >= 0x7ff00000u) return k == 0x7ff00000u ? 0xffffffffu : 0u;
  if (k < (unsigned)(1023 - 537) << 20) return 0u;
  const float fk = __uint_as_float(0x3f800000u | (k & 0xfffffu) << 3);                             // [1, 2)
  const float fs = d < 16u ? __uint_as_float((127u - d) << 23 | (s & 0xfffffu) << 3) : 0.f;  // on the scale of fk
  return (e << 21) + ((__float_as_uint(fmaf(fk, fk, fs * fs)) - 0x3f800000u) >> 3);          // fk^2 + fs^2 < 8
}

// Inverse of the n x n matrix A of NT threads, in place, columns permuted: column m of A is column perm[m] of the
// inverse.  rowk, old, fcol: n complex each; used, perm: n ints; red: NT / 32 pairs.  False if singular.
template <int NT>
__device__ __forceinline__ bool gauss_jordan(double2 *A, int n, double2 *rowk, double2 *old, double2 *fcol, int *used,
                                             int *perm, unsigned (*red)[2], int tid) {
  const int lane = tid & 31, warp = tid >> 5, nn = n * n;
  for (int j = tid; j < n; j += NT) {
    used[j] = 0;
    perm[j] = j;
  }
  unsigned best = 0u;
  int bidx = 0x7fffffff;
  for (int e = tid; e < nn; e += NT) {
    const unsigned k = inv_key(A[e]);
    if (k > best) { best = k; bidx = e; }
  }
  for (int it = 0; it < n; ++it) {
    {  // largest key, first in row-major order
      const unsigned wb = __reduce_max_sync(0xffffffffu, best);
      const unsigned wi = __reduce_min_sync(0xffffffffu, best == wb ? (unsigned)bidx : 0x7fffffffu);
      best = wb;
      bidx = (int)wi;
    }
    if constexpr (NT > 32) {
      if (lane == 0) {
        red[warp][0] = best;
        red[warp][1] = (unsigned)bidx;
      }
    }
    inv_sync<NT>();
    if constexpr (NT > 32) {
      best = red[0][0];
      bidx = (int)red[0][1];
#pragma unroll
      for (int w = 1; w < NT / 32; ++w)
        if (red[w][0] > best || (red[w][0] == best && (int)red[w][1] < bidx)) {
          best = red[w][0];
          bidx = (int)red[w][1];
        }
    }
    if (best == 0u) return false;  // uniform
    const int irow = bidx / n, icol = bidx - irow * n;
    // scaled pivot row, the row it trades places with, the pivot's column after that
    if ((tid & ~31) < n) {  // whole warps
      // The reciprocal as two divisions, one for even and one for odd lanes, not as 1 / den and two products: m times m / (m m)
      // rounds to one far more often, which is what leaves the exact zero of a singular block, and 1 / den overflows
      // below 2^-512.  (A pass of Dyson, hexagonal 8 k: one division 0.662 ms, this
      // 0.667, both in every lane 0.690.)
      const double2 pv = A[irow * n + icol];
      const double den = pv.x * pv.x + pv.y * pv.y;
      const double mine = ((tid & 1) ? -pv.y : pv.x) / den, other = __shfl_xor_sync(0xffffffffu, mine, 1);
      const double2 pinv = (tid & 1) ? make_double2(other, mine) : make_double2(mine, other);
      for (int l = tid; l < n; l += NT) {
        rowk[l] = l == icol ? pinv : cmul(A[irow * n + l], pinv);
        old[l] = A[icol * n + l];
        fcol[l] = A[(l == irow ? icol : l) * n + icol];
      }
    }
    if (tid == 0) {
      used[icol] = 1;
      const int t = perm[irow];
      perm[irow] = perm[icol];
      perm[icol] = t;
    }
    inv_sync<NT>();
    best = 0u;
    bidx = 0x7fffffff;
    for (int e = tid; e < nn; e += NT) {
      const int i = e / n, j = e - i * n;
      const double2 r = rowk[j];
      double2 a = r;
      if (i != icol) {
        const double2 f = fcol[i];
        a = csub(j == icol ? make_double2(0.0, 0.0) : i == irow ? old[j] : A[e], r, f);
        if (!used[i] && !used[j]) {
          const unsigned k = inv_key(a);
          if (k > best) { best = k; bidx = e; }
        }
      }
      A[e] = a;
    }
  }
  inv_sync<NT>();
  return true;
}

// -A^-1 of a positive definite A (lower triangle, in place) by symmetric sweeps.  c, w: n complex each.  False (A
// overwritten) where a pivot is not clearly positive: below 2^-40 of its diagonal element 1 - Re P.
template <int NT>
__device__ __forceinline__ bool sweep_inverse(double2 *A, const double2 *P, int n, double2 *c, double2 *w, int tid) {
  const int half = (n + 1) / 2, ne = half * (n + 1);
  for (int k = 0; k < n; ++k) {
    const double p = A[k * n + k].x;
    const double p0 = 1.0 - P[k * n + k].x;
    if (!(p > 0x1p-40 * p0) || !(p0 > 0.0) || isinf(p)) return false;  // uniform
    for (int i = tid; i < n; i += NT) {  // column k, and its conjugate over the pivot
      const double d = 1.0 / p;
      const double2 v = i >= k ? A[i * n + k] : cconj(A[k * n + i]);
      c[i] = v;
      w[i] = i == k ? make_double2(-d, 0.0) : make_double2(v.x * d, -v.y * d);
    }
    inv_sync<NT>();
    // rows q and n - 1 - q of the triangle together have n + 1 elements
    for (int e = tid; e < ne; e += NT) {
      const int q = e / (n + 1), r = e - q * (n + 1), lng = n - q;
      const int i = r < lng ? n - 1 - q : q, j = r < lng ? r : r - lng;
      if (r >= lng && n - 1 - q == q) continue;
      double2 a;
      if (i == k) {
        a = w[j];
      } else if (j == k) {
        a = cconj(w[i]);
      } else {
        a = csub(A[i * n + j], c[i], w[j]);
      }
      A[i * n + j] = a;
    }
    inv_sync<NT>();
  }
  return true;
}

// nm = largest block of the launch.  Shared, per matrix: A [nm^2] | P [nm^2] (mode 0) | three rows [nm] (complex) |
// 2 nm ints.
template <int NT>
__global__ void __launch_bounds__(NT == 32 ? 256 : NT) inverse_kernel(
    const InvTask *__restrict__ tasks, int ntasks, double2 *__restrict__ W, const double2 *__restrict__ S,
    const double2 *__restrict__ F, const int64_t *__restrict__ wsample, double beta, double mu, int mode,
    int *__restrict__ bad, int nm, const double *__restrict__ mu_ptr, double2 *__restrict__ Wout,
    const int *__restrict__ skip) {
  if (skip && *skip) return;  // the mu search has converged (uniform over the grid)
  extern __shared__ double2 smem_inv[];
  __shared__ unsigned red[NT / 32][2];
  const int per = NT == 32 ? blockDim.x / 32 : 1, mat = NT == 32 ? threadIdx.x >> 5 : 0, tid = threadIdx.x % NT;
  const int ti = blockIdx.x * per + mat;
  if (ti >= ntasks) return;
  const int na = (mode == 0 ? 2 : 1) * nm * nm + 3 * nm;
  double2 *A = smem_inv + (size_t)mat * na;
  double2 *B = A + (mode == 0 ? nm * nm : 0);
  double2 *rowk = A + na - 3 * nm, *old = rowk + nm, *fcol = old + nm;
  int *used = reinterpret_cast<int *>(smem_inv + (size_t)per * na) + mat * 2 * nm, *perm = used + nm;
  const InvTask tk = tasks[ti];
  const int n = tk.n, nn = n * n;
  double2 *g = W + tk.a;
  auto hermitian = [&]() {  // A = I - (P + P^H)/2
    for (int e = tid; e < nn; e += NT) {
      const int i = e / n, j = e - i * n;
      const double2 pij = B[e], pji = B[j * n + i];
      A[e] = make_double2((i == j ? 1.0 : 0.0) - 0.5 * (pij.x + pji.x), -0.5 * (pij.y - pji.y));
    }
    inv_sync<NT>();
  };
  if (mode == 1) {
    if (mu_ptr) mu = *mu_ptr;
    const double wn = (2.0 * (double)wsample[tk.w] + 1.0) * 3.14159265358979323846 / beta;
    for (int e = tid; e < nn; e += NT) {
      const double2 sv = S[tk.s + e], fv = F[tk.f + e], sg = g[e];
      // (mu + i wn) * S - F - Sigma
      A[e] = make_double2(mu * sv.x - wn * sv.y - fv.x - sg.x, mu * sv.y + wn * sv.x - fv.y - sg.y);
    }
    inv_sync<NT>();
    if (!gauss_jordan<NT>(A, n, rowk, old, fcol, used, perm, red, tid)) {
      if (tid == 0) atomicExch(bad, 1);
      return;
    }
    double2 *o = Wout ? Wout + tk.a : g;
    for (int e = tid; e < nn; e += NT) {
      const int i = e / n, j = e - i * n;
      o[i * n + perm[j]] = A[e];
    }
    return;
  }
  for (int e = tid; e < nn; e += NT) B[e] = g[e];
  inv_sync<NT>();
  hermitian();
  if (sweep_inverse<NT>(A, B, n, rowk, old, tid)) {
    // R = -A, both triangles
    for (int e = tid; e < nn; e += NT) {
      const int i = e / n, j = e - i * n;
      if (j > i) continue;
      const double2 v = A[e];
      A[e] = make_double2(-v.x, i == j ? 0.0 : -v.y);
      if (j < i) A[j * n + i] = make_double2(-v.x, v.y);
    }
  } else {
    inv_sync<NT>();
    hermitian();
    if (!gauss_jordan<NT>(A, n, rowk, old, fcol, used, perm, red, tid)) {
      if (tid == 0) atomicExch(bad, 1);
      return;
    }
    for (int e = tid; e < nn; e += NT) {  // columns in order, by way of B
      const int i = e / n, j = e - i * n;
      B[i * n + perm[j]] = A[e];
    }
    inv_sync<NT>();
    for (int e = tid; e < nn; e += NT) {  // R = (A^-1 + A^-H)/2
      const int i = e / n, j = e - i * n;
      const double2 aij = B[e], aji = B[j * n + i];
      A[e] = make_double2(0.5 * (aij.x + aji.x), 0.5 * (aij.y - aji.y));
    }
    inv_sync<NT>();
    for (int e = tid; e < nn; e += NT) B[e] = g[e];
  }
  inv_sync<NT>();
  for (int e = tid; e < nn; e += NT) {
    const int i = e / n, j = e - i * n;
    double2 a = make_double2(0.0, 0.0);
    for (int l = 0; l < n; ++l) a = cfma(A[i * n + l], B[l * n + j], a);
    g[e] = a;
  }
}

// Leakage check of G (sc_type_block.cpp:66-71): max over elements of
// |sum_t tct[t] G(tau_{t+1})| for the first and last IR coefficient.
__global__ void leakage_kernel(const TSlab *__restrict__ slabs, const double2 *__restrict__ G,
                               const double *__restrict__ tct_first, const double *__restrict__ tct_last,
                               int ncheb, unsigned long long *__restrict__ out) {
  const TSlab sl = slabs[blockIdx.x];
  double mf = 0.0, ml = 0.0;
  for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < sl.ncols; c += gridDim.y * blockDim.x) {
    double2 a = make_double2(0.0, 0.0), b = make_double2(0.0, 0.0);
    for (int t = 0; t < ncheb; ++t) {
      const double2 g = G[sl.y + (int64_t)(t + 1) * sl.ldy + c];
      a.x += tct_first[t] * g.x; a.y += tct_first[t] * g.y;
      b.x += tct_last[t] * g.x;  b.y += tct_last[t] * g.y;
    }
    mf = fmax(mf, sqrt(a.x * a.x + a.y * a.y));
    ml = fmax(ml, sqrt(b.x * b.x + b.y * b.y));
  }
  for (int off = 16; off > 0; off >>= 1) {
    mf = fmax(mf, __shfl_down_sync(0xffffffffu, mf, off));
    ml = fmax(ml, __shfl_down_sync(0xffffffffu, ml, off));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(out, (unsigned long long)__double_as_longlong(mf));
    atomicMax(out + 1, (unsigned long long)__double_as_longlong(ml));
  }
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
void launch_p0_fp64(const P0Tile *tiles, int ntiles, int maxo, const P0Contrib *contribs,
                    const double2 *V, const double2 *G, double2 *Part, int ns, int nts, int smem_bytes,
                    cudaStream_t st) {
  if (ntiles == 0) return;
  const int cap = smem_bytes / (int)sizeof(double2);
  if (maxo <= 8) {
    p0_fp64_kernel<8><<<ntiles, 256, smem_bytes, st>>>(tiles, contribs, V, G, Part, ns, nts, cap);
  } else {
    p0_fp64_kernel<16><<<ntiles, 256, smem_bytes, st>>>(tiles, contribs, V, G, Part, ns, nts, cap);
  }
  GWGB_CUDA(cudaGetLastError());
}

// Hartree term (HF on the block layout; the reference's HF solver is a stub,
// cuhf_solver_block.h:36-39).  One thread per aux index Q (c) or per element of
// an AO block (J); every sum runs over its items in list order (deterministic).
__global__ void hartree_c_kernel(const HcTask *__restrict__ tasks, const HcItem *__restrict__ items,
                                 const double2 *__restrict__ V, const double2 *__restrict__ G, int ns,
                                 double scale, double2 *__restrict__ c) {
  const HcTask t = tasks[blockIdx.x];
  for (int Q = threadIdx.x; Q < t.qb; Q += blockDim.x) {
    double2 acc = make_double2(0.0, 0.0);
    for (int it = t.i0; it < t.i1; ++it) {
      const HcItem x = items[it];
      const double2 *vq = V + x.v + (int64_t)Q * x.b * x.b;
      for (int s = 0; s < ns; ++s) {
        const double2 *r = G + x.g + (int64_t)s * x.gstride;
        for (int a = 0; a < x.b; ++a)
          for (int b = 0; b < x.b; ++b) acc = cfma(vq[a * x.b + b], r[b * x.b + a], acc);
      }
    }
    c[t.cout + Q] = make_double2(acc.x * scale, acc.y * scale);
  }
}

__global__ void hartree_j_kernel(const HjTask *__restrict__ tasks, const HjItem *__restrict__ items,
                                 const double2 *__restrict__ V, const double2 *__restrict__ c,
                                 double2 *__restrict__ J) {
  const HjTask t = tasks[blockIdx.x];
  const int bb = t.b * t.b;
  for (int e = threadIdx.x; e < bb; e += blockDim.x) {
    double2 acc = make_double2(0.0, 0.0);
    for (int it = t.i0; it < t.i1; ++it) {
      const HjItem x = items[it];
      for (int Q = 0; Q < x.qb; ++Q) acc = cfma(V[x.v + (int64_t)Q * bb + e], c[x.c + Q], acc);
    }
    J[t.out + e] = acc;
  }
}

void launch_hartree(const HcTask *ct, int nct, const HcItem *ci, const HjTask *jt, int njt, const HjItem *ji,
                    const double2 *V, const double2 *G, int ns, double scale, double2 *c, double2 *J,
                    cudaStream_t st) {
  if (nct > 0) {
    hartree_c_kernel<<<nct, 128, 0, st>>>(ct, ci, V, G, ns, scale, c);
    GWGB_CUDA(cudaGetLastError());
  }
  if (njt > 0) {
    hartree_j_kernel<<<njt, 128, 0, st>>>(jt, ji, V, c, J);
    GWGB_CUDA(cudaGetLastError());
  }
}

void launch_reduce_slices(const RedTask *tasks, int ntasks, const double2 *part, double2 *out, int nts,
                          double scale, int mirror, cudaStream_t st, int ny) {
  if (ntasks == 0) return;
  reduce_slices_kernel<<<dim3(ntasks, std::max(1, std::min(ny, 65535))), 256, 0, st>>>(tasks, part, out, nts, scale,
                                                                                       mirror);
  GWGB_CUDA(cudaGetLastError());
}

void launch_sigma_fp64(const SigTile *tiles, int ntiles, int maxo, const SigContrib *contribs,
                       const double2 *V, const double2 *G, const double2 *P, double2 *Part, int ns,
                       int smem_bytes, cudaStream_t st) {
  if (ntiles == 0) return;
  const int cap = smem_bytes / (int)sizeof(double2);
  if (maxo <= 8) {
    sigma_fp64_kernel<8><<<ntiles, 256, smem_bytes, st>>>(tiles, contribs, V, G, P, Part, ns, cap);
  } else {
    sigma_fp64_kernel<16><<<ntiles, 256, smem_bytes, st>>>(tiles, contribs, V, G, P, Part, ns, cap);
  }
  GWGB_CUDA(cudaGetLastError());
}

void launch_rotate(const RotTask *tasks, int ntasks, int nbatch, int smem_bytes, const double2 *src,
                   const double2 *O, double2 *dst, cudaStream_t st) {
  if (ntasks == 0 || nbatch == 0) return;
  rotate_kernel<<<dim3(ntasks, nbatch), 128, smem_bytes, st>>>(tasks, src, O, dst);
  GWGB_CUDA(cudaGetLastError());
}

void launch_vrot(const VrTask *tasks, int ntasks, const double2 *V, const double2 *O, double2 *Vt, cudaStream_t st) {
  if (ntasks == 0) return;
  vrot_kernel<<<ntasks, 256, 0, st>>>(tasks, V, O, Vt);
  GWGB_CUDA(cudaGetLastError());
}

void launch_mirror(double2 *P, const int64_t *qoff, const int32_t *qsz, int nq, int nts, cudaStream_t st) {
  mirror_kernel<<<dim3(nq, 8), 256, 0, st>>>(P, qoff, qsz, nts);
  GWGB_CUDA(cudaGetLastError());
}

void launch_zero_upper(double2 *P, const int64_t *qoff, const int32_t *qsz, int nq, int nts, cudaStream_t st) {
  zero_upper_kernel<<<dim3(nq, 8), 256, 0, st>>>(P, qoff, qsz, nts);
  GWGB_CUDA(cudaGetLastError());
}

void launch_transform(const TSlab *slabs, int nslabs, int max_cols, const double2 *T, int nout, int nin,
                      int row0, const double2 *X, double2 *Y, cudaStream_t st) {
  if (nslabs == 0 || nout == 0) return;
  GWGB_REQUIRE(nout <= TR_MAXOUT, GWGB_E_UNSUPPORTED, "transform output longer than 160 rows");
  const int ct = (max_cols + 31) / 32;
  // the largest rows-per-warp that still gives about two CTAs per SM
  auto ctas = [&](int R) { return (int64_t)nslabs * ct * ((nout + 8 * R - 1) / (8 * R)); };
  if (nout > 8 && ctas(4) >= 304) {
    transform_kernel<4><<<dim3(nslabs, ct, (nout + 31) / 32), 256, 0, st>>>(slabs, T, nout, nin, row0, X, Y);
  } else if (nout > 8 && ctas(2) >= 304) {
    transform_kernel<2><<<dim3(nslabs, ct, (nout + 15) / 16), 256, 0, st>>>(slabs, T, nout, nin, row0, X, Y);
  } else {
    transform_kernel<1><<<dim3(nslabs, ct, (nout + 7) / 8), 256, 0, st>>>(slabs, T, nout, nin, row0, X, Y);
  }
  GWGB_CUDA(cudaGetLastError());
}

std::vector<InvClass> inv_classes(std::vector<InvTask> &tasks) {
  std::stable_sort(tasks.begin(), tasks.end(), [](const InvTask &x, const InvTask &y) { return x.n > y.n; });
  std::vector<InvClass> c;
  auto kind = [](int n) { return n > 32 ? 2 : n > 16 ? 1 : 0; };
  for (size_t i = 0; i < tasks.size(); ++i) {
    if (i == 0 || kind(tasks[i].n) != kind(tasks[i - 1].n)) c.push_back({(int)i, 0, tasks[i].n});
    ++c.back().count;
  }
  return c;
}

void launch_inverse(const InvTask *tasks, const std::vector<InvClass> &classes, double2 *W, const double2 *S,
                    const double2 *F, const int64_t *wsample, double beta, double mu, int mode, int *bad,
                    cudaStream_t st, const double *mu_ptr, double2 *Wout, const int *skip) {
  for (const InvClass &c : classes) {
    const int bytes = inv_bytes(c.nmax, mode);
    auto run = [&](auto kernel, int per, int threads) {
      kernel<<<(c.count + per - 1) / per, per * threads, per * bytes, st>>>(
          tasks + c.first, c.count, W, S, F, wsample, beta, mu, mode, bad, c.nmax, mu_ptr, Wout, skip);
    };
    if (c.nmax > 32)
      run(inverse_kernel<256>, 1, 256);
    else if (c.nmax > 16)
      run(inverse_kernel<128>, 1, 128);
    else  // one warp per block
      run(inverse_kernel<32>, inv_warps_per_block(c.nmax, mode), 32);
    GWGB_CUDA(cudaGetLastError());
  }
}

void launch_leakage(const TSlab *slabs, int nslabs, const double2 *G, const double *tf, const double *tl,
                    int ncheb, unsigned long long *out, cudaStream_t st) {
  if (nslabs == 0) return;
  leakage_kernel<<<dim3(nslabs, 4), 256, 0, st>>>(slabs, G, tf, tl, ncheb, out);
  GWGB_CUDA(cudaGetLastError());
}

void set_fp64_kernel_attributes(int smem_bytes) {
  GWGB_CUDA(cudaFuncSetAttribute(p0_fp64_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
  GWGB_CUDA(cudaFuncSetAttribute(p0_fp64_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
  GWGB_CUDA(cudaFuncSetAttribute(sigma_fp64_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
  GWGB_CUDA(cudaFuncSetAttribute(sigma_fp64_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
  GWGB_CUDA(cudaFuncSetAttribute(rotate_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, rotate_smem_bytes(MAX_BLOCK)));
  set_inverse_kernel_attributes();
}

void set_inverse_kernel_attributes() {
  GWGB_CUDA(cudaFuncSetAttribute(inverse_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, inv_bytes(MAX_BLOCK, 0)));
  GWGB_CUDA(cudaFuncSetAttribute(inverse_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, inv_bytes(32, 0)));
}

}  // namespace gwgb
