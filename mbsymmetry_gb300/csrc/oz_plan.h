// Work lists and buffers of one sliced contraction (P0 or Sigma).
#pragma once

#include <algorithm>
#include <vector>

#include "dbuf.h"
#include "kernels_oz.h"

namespace gwgb {

// One V block (and spin) of a contraction, in the names of kernels_oz.h.
// Offsets and strides in complex elements of the source buffers.
struct OzContrib {
  int32_t nL, nx, ny, nz, N, K1;
  int32_t vid;                 // V block id: contributions with the same id share their V images
  int64_t v;                   // V block in the V source
  int32_t sx, sy, sk;          // stage 1: V1[(x, y)][k]
  int32_t sn, sL, sz;          // stage 3: V3[n][(L, z)]
  int8_t conj1, conj3;
  int64_t ga, gt;              // stage 1 operand G[(tau, L)][k]: ga + tau * gt + L * gL + k * gk
  int32_t gL, gk;
  int64_t b2, b2t;             // stage 2 operand B2[tau][z][y]: b2 + tau * b2t + z * b2z + y * b2y
  int32_t b2z, b2y;
  int8_t b2conj;
};

// One output block and its contributions [c0, c1) in K order.
struct OzOwner {
  int64_t out;                 // block at tau = 0
  int32_t ostride, N, nx;
  int32_t sn, sx;              // element (n, x) at n * sn + x * sx
  int32_t c0, c1;
};

// One launch; kind as in gwgb_launch_stat.kernel.
struct OzLaunch {
  int kind = 0, stage = 0;     // 0 oz_gemm_kernel, 2 reduce_slices_kernel, 3 oz_build_kernel
  int64_t t0 = 0, n = 0;       // tasks
  int64_t d0 = 0;              // descriptors / auxiliary lists of the launch
  int src = 0, dst = 0;        // builds: source (0 V, 1 G, 2 B2 source) and image buffer
  OzArgs args{};               // rings (pointers are filled in when it runs)
  bool multi = false;          // stages 1, 2: tasks of more than one round of K
  int ny = 1;                  // reductions: CTAs per task
  double flops = 0, ops = 0, bytes = 0;
};

// Buffers that the plans of one handle share (they run one after the other).
struct OzShared {  // one allocation (a first pass waits for it)
  template <typename T> struct Part {
    T *p = nullptr;
    size_t n = 0;
  };
  Part<char> A1, B2, X1, X2;
  Part<double2> part;
  DBuf<char> pool;
  // At least these sizes (the contents are lost when that means a new allocation).
  void grow(int64_t a1, int64_t b2, int64_t x1, int64_t x2, int64_t np) {
    auto fits = [](const auto &x, int64_t n) { return n <= (int64_t)x.n; };
    if (fits(A1, a1) && fits(B2, b2) && fits(X1, x1) && fits(X2, x2) && fits(part, np)) return;
    size_t at = 0;
    auto place = [&](auto &x, int64_t n, auto *q) {
      x.n = std::max(x.n, (size_t)n);
      x.p = reinterpret_cast<decltype(q)>(at);
      at = (at + x.n * sizeof(*q) + 1023) / 1024 * 1024;
    };
    auto all = [&](auto &&f) { f(A1); f(B2); f(X1); f(X2); };
    pool.free();
    place(A1, a1, (char *)nullptr); place(B2, b2, (char *)nullptr);
    place(X1, x1, (char *)nullptr); place(X2, x2, (char *)nullptr);
    place(part, np, (double2 *)nullptr);
    pool.alloc(at);
    all([&](auto &x) { x.p = pool.p + reinterpret_cast<size_t>(x.p); });
    part.p = reinterpret_cast<double2 *>(pool.p + reinterpret_cast<size_t>(part.p));
  }
  void free() {
    pool.free();
    A1 = B2 = X1 = X2 = {};
    part = {};
  }
};

// A tau <-> omega transform Y[slab][r][c] = sum_i T[r][i] X[slab][row0 + i][c] as a stage-3
// GEMM in six slices: rows c, K = i, columns r.  Scaled: X[i] by the power of two below its largest
// element over all columns and T[.][i] by the inverse, in every run, so that the slices of a row of T follow its terms.
// The transforms to tau need that: their terms fall off with frequency in X and, towards the middle of the tau axis, in T,
// where the result is a small rest of them.  Errors against extended precision, relative to the FP64 kernel's, over the
// committed grids, G and P~ of s+p+d crystals, geometric mean and worst: 2-norm 0.1 and 0.2, largest of a row r relative to that
// row 0.08 and 0.3; scaled by the columns of T alone 0.39 and 0.64, but rows 12 and 900.  The transforms from tau
// are as good without (0.05 and 0.2, rows 0.05 and 0.15).
class OzTransform {
 public:
  void build(const std::vector<TSlab> &slabs, int nout, int nin, int row0, bool scaled, int64_t nX, int64_t nY, int nsm,
             cudaStream_t st);
  int64_t bytes_A() const { return a_; }
  bool built() const { return gemm_.n > 0; }
  bool ready = false;           // the matrix has been set
  int launches() const { return scaled_ ? 4 : 2; }
  // T: [nout][nin] on the device; may be set again, the buffers stay where they are
  void set_matrix(const double2 *T, cudaStream_t st);
  // slabs: those of build(), on the device; A: bytes_A() bytes of scratch
  void run(const TSlab *slabs, int nslabs, const double2 *T, const double2 *X, double2 *Y, char *A, int nsm, int *err,
           cudaStream_t st) const;
  void free();

 private:
  int64_t a_ = 0, nbuild_ = 0, nT_ = 0;
  int nin_ = 0, row0_ = 0;
  bool scaled_ = false;
  OzLaunch gemm_;
  DBuf<OzBuild> builds_;        // images of X, then those of T
  DBuf<OzTask> tasks_;
  DBuf<OzS3> s3_;
  DBuf<OzRnd> rnd_;
  DBuf<char> T_;
  DBuf<double> scale_;          // [nin] of X, [nin] of T, of the last run
};

class OzPlan {
 public:
  enum { IMG_V, IMG_A1, IMG_B2 };
  // stage0: gwgb_launch_stat.stage of stage 1; budget: bytes of X1 + X2 per chunk; persist_bytes: the
  // V images are kept (built once per upload) when they take at most this, else built per chunk; tau_bytes: the images
  // of G and of the stage-2 operand, for a range of tau if those of all take more.
  // Host side only (no CUDA calls); upload() then moves the lists to the device.
  void build(int ns, const std::vector<OzContrib> &cs, const std::vector<OzOwner> &own, int ntau, int stage0,
             int64_t budget, int64_t persist_bytes, int64_t tau_bytes, int nsm, int64_t nV, int64_t nG, int64_t nB2,
             int64_t nout);
  void upload(cudaStream_t st);
  int64_t bytes_lists() const { return (int64_t)host_.size(); }  // until upload()
  int64_t bytes_V() const { return vimg_; }
  int64_t bytes_A1() const { return a1_; }
  int64_t bytes_B2() const { return b2_; }
  int64_t bytes_X1() const { return x1_; }
  int64_t bytes_X2() const { return x2_; }
  int64_t part_elems() const { return part_; }
  void alloc_images() { V_.alloc((size_t)vimg_); }
  void free_images() { V_.free(); }
  // the operand images that do not change between iterations (after a V / rotation upload)
  void build_static(const double2 *V, cudaStream_t st);
  void run_one(const OzLaunch &l, OzShared &sh, const double2 *V, const double2 *G, const double2 *B2, double2 *out,
               int nts, double scale, int nsm, int *err, cudaStream_t st) const;
  const std::vector<OzLaunch> &launches() const { return launches_; }
  void free();

 private:
  int ns_ = 3;
  int64_t vimg_ = 0, a1_ = 0, b2_ = 0, x1_ = 0, x2_ = 0, part_ = 0;
  std::vector<OzLaunch> launches_, static_;
  DBuf<char> V_;
  // the work lists, one allocation
  template <typename T> struct List {
    T *p = nullptr;
    size_t n = 0;
  };
  std::vector<char> host_;      // the lists until they are uploaded
  DBuf<char> lists_;
  List<OzBuild> builds_;
  List<OzTask> tasks_;
  List<OzS1> s1_;
  List<OzCol1> col1_;
  List<OzDst1> dst1_;
  List<OzS2> s2_;
  List<OzRow> rows_;
  List<OzS3> s3_;
  List<OzRnd> rnd_;
  List<RedTask> red_;
};

}  // namespace gwgb
