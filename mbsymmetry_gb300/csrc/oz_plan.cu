// Host side of the sliced contractions: cuts a contraction into units and
// chunks, lays out the operand images and builds the task lists of the three
// stages (kernels_oz.h).
//
// Unit: a consecutive range of an output block's contributions (a K slice of
// stage 3, with an FP64 partial of its own; the partials are summed in order
// at the end).  Units depend on the block alone, so no result bit depends on
// the chunking.  Chunk: consecutive units whose intermediates X1 and X2 fit
// the budget; each chunk is one launch per stage.  Where the images of G and of
// the stage-2 operand at every tau exceed their limit, the chunks are those of one
// tau range after the other.
#include "oz_plan.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <tuple>

#include "kernels.h"

namespace gwgb {

namespace {

int cdiv(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }

// L rows per stage-3 round (2^glog * zos <= oct octets of K): a round costs its stage-2 rows and one
// accumulator drain of stage 3, about 1.5 rows' worth.
int choose_glog(int zos, int nL, int oct) {
  int best = 0;
  double cost = 1e30;
  for (int gl = 0; (zos << gl) <= oct; ++gl) {
    const int g = 1 << gl;
    const double c = (double)cdiv(nL, g) * (g + 1.5);
    if (c < cost - 1e-9) {
      cost = c;
      best = gl;
    }
  }
  return best;
}

}  // namespace

void OzPlan::build(int ns, const std::vector<OzContrib> &cs, const std::vector<OzOwner> &own, int ntau, int stage0,
                   int64_t budget, int64_t persist_bytes, int64_t tau_bytes, int nsm, int64_t nV, int64_t nG, int64_t nB2,
                   int64_t nout) {
  ns_ = ns;
  const int OCT = OZ_OCT, NS = ns;
  const int FK = 8 * OCT;  // complex K of a full round
  const double nprod = ns == 3 ? 8 : 26;  // slice products per K step
  const int64_t fullA = oz_abytes(NS, OCT);
  launches_.clear();
  static_.clear();
  vimg_ = a1_ = b2_ = x1_ = x2_ = part_ = 0;
  std::vector<OzBuild> builds;
  std::vector<OzTask> tasks;
  std::vector<OzS1> s1;
  std::vector<OzCol1> col1;
  std::vector<OzDst1> dst1;
  std::vector<OzS2> s2;
  std::vector<OzRow> rows;
  std::vector<OzS3> s3;
  std::vector<OzRnd> rnd;
  std::vector<RedTask> red;

  auto geom_ok = [&](const OzContrib &c) {
    GWGB_REQUIRE(c.nL > 0 && c.nx > 0 && c.ny > 0 && c.nz > 0 && c.N > 0 && c.K1 > 0 && c.nL <= MAX_BLOCK &&
                     c.nx <= MAX_BLOCK && c.ny <= MAX_BLOCK && c.nz <= MAX_BLOCK && c.N <= MAX_BLOCK &&
                     c.K1 <= MAX_BLOCK,
                 GWGB_E_INVALID, "internal work list out of bounds: sliced block size");
  };
  for (const OzContrib &c : cs) {
    geom_ok(c);
    const int64_t ext = (int64_t)(c.nx - 1) * c.sx + (int64_t)(c.ny - 1) * c.sy + (int64_t)(c.K1 - 1) * c.sk + 1;
    check_range(c.v, ext, nV, "sliced V block (stage 1)");
    check_range(c.v, (int64_t)(c.N - 1) * c.sn + (int64_t)(c.nL - 1) * c.sL + (int64_t)(c.nz - 1) * c.sz + 1, nV,
                "sliced V block (stage 3)");
    check_range(c.ga + std::min<int64_t>(0, c.gt * (ntau - 1)),
                std::abs(c.gt) * (ntau - 1) + (int64_t)(c.nL - 1) * c.gL + (int64_t)(c.K1 - 1) * c.gk + 1, nG,
                "sliced G block");
    check_range(c.b2 + std::min<int64_t>(0, c.b2t * (ntau - 1)),
                std::abs(c.b2t) * (ntau - 1) + (int64_t)(c.nz - 1) * c.b2z + (int64_t)(c.ny - 1) * c.b2y + 1, nB2,
                "sliced stage-2 operand");
  }

  // --- distinct operands of stage 1 and of stage 2 (their first contribution), and the tau ranges
  struct B2 { int64_t b, bt, bz; };
  std::map<int64_t, int> s1_of;                       // G block -> OzS1 of the tau range
  std::map<std::pair<int64_t, int>, B2> b2_of;        // (block, conj) -> images of the tau range
  std::vector<int> s1_first, b2_first;
  for (size_t c = 0; c < cs.size(); ++c) {
    if (s1_of.emplace(cs[c].ga, 0).second) s1_first.push_back((int)c);
    if (b2_of.emplace(std::make_pair(cs[c].b2, (int)cs[c].b2conj), B2{}).second) b2_first.push_back((int)c);
  }
  auto b2_bytes = [&](const OzContrib &c) {  // of one tau and octet of columns
    const int kos = cdiv(c.ny, 8);
    return (int64_t)NS * kos * 512 + 32 * cdiv(kos, OCT);
  };
  auto image_bytes = [&](int nt) {
    int64_t n = 0;
    for (int i : s1_first) {
      const int kos = cdiv(cs[i].K1, 8);
      n += cdiv((int64_t)nt * cs[i].nL, OZ_M) * ((int64_t)NS * kos * 4096 + 512 * cdiv(kos, OCT));
    }
    for (int i : b2_first) n += (int64_t)nt * cdiv(cs[i].nz, 8) * b2_bytes(cs[i]);
    return n;
  };
  int ntr = ntau;  // tau of a range
  while (ntr > 1 && image_bytes(ntr) > tau_bytes) ntr = (ntr + 1) / 2;
  auto add_build = [&](std::vector<OzLaunch> &v, size_t lo, size_t hi, int src, int dst, int stage) {
    if (lo == hi) return;
    OzLaunch l;
    l.kind = 3;
    l.stage = stage;
    l.t0 = (int64_t)lo;
    l.n = (int64_t)(hi - lo);
    l.src = src;
    l.dst = dst;
    for (size_t i = lo; i < hi; ++i) {
      const OzBuild &b = builds[i];
      l.bytes += 16.0 * 8 * b.nks * b.rows + (b.isb ? (double)(b.rows / 8) * oz_bbytes1(NS, b.nks) : (double)oz_abytes(NS, b.nks));
    }
    v.push_back(l);
  };
  // images of G rows (tau, L) and of the stage-2 operand, tau in [t0, t0 + nt)
  auto add_images = [&](int t0, int nt) {
    const size_t ga0 = builds.size();
    int64_t a1 = 0, b2 = 0;
    for (int i : s1_first) {
      const OzContrib &c = cs[i];
      const int kos = cdiv(c.K1, 8), R = cdiv(kos, OCT), M = nt * c.nL;
      s1_of[c.ga] = (int)s1.size();
      s1.push_back({a1, M, c.nL, kos, 0});
      for (int mt = 0; mt * OZ_M < M; ++mt)
        for (int r = 0; r < R; ++r) {
          const int nks = std::min(OCT, kos - r * OCT);
          builds.push_back({c.ga + t0 * c.gt + (int64_t)r * FK * c.gk, a1, c.gt, 0, c.gL, c.gk, c.nL, 1 << 20, c.nL,
                            c.K1 - r * FK, nt, 1, mt * OZ_M, OZ_M, (int16_t)nks, 0, 0, 0, -1, 0});
          a1 += oz_abytes(NS, nks);
        }
    }
    const size_t gb0 = builds.size();
    for (int i : b2_first) {
      const OzContrib &c = cs[i];
      const int kos = cdiv(c.ny, 8), R = cdiv(kos, OCT), zos = cdiv(c.nz, 8);
      const int64_t per = b2_bytes(c);
      b2_of[std::make_pair(c.b2, (int)c.b2conj)] = {b2, zos * per, OCT * per};
      for (int t = t0; t < t0 + nt; ++t)
        for (int z0 = 0; z0 < zos; z0 += OCT) {
          const int noct = std::min(OCT, zos - z0);
          for (int r = 0; r < R; ++r) {
            const int nks = std::min(OCT, kos - r * OCT);
            builds.push_back({c.b2 + t * c.b2t + (int64_t)z0 * 8 * c.b2z + (int64_t)r * FK * c.b2y, b2, 0, 0, c.b2z,
                              c.b2y, 1 << 20, 1 << 20, c.nz - 8 * z0, c.ny - r * FK, 1, 1, 0, (int16_t)(8 * noct),
                              (int16_t)nks, 1, c.b2conj, 0, -1, 0});
            b2 += noct * oz_bbytes1(NS, nks);
          }
        }
    }
    a1_ = std::max(a1_, a1);
    b2_ = std::max(b2_, b2);
    add_build(launches_, ga0, gb0, 1, IMG_A1, stage0);
    add_build(launches_, gb0, builds.size(), 2, IMG_B2, stage0 + 1);
  };

  // --- units
  struct Unit { int own, c0, c1, idx, nunits; int64_t bytes; };
  std::vector<Unit> units;
  std::vector<int> glog(cs.size());
  auto rounds_of = [&](int c) { return cdiv(cs[c].nL, 1 << glog[c]) * cdiv(cdiv(cs[c].nz, 8), OCT); };
  auto x_bytes = [&](int c) {
    const OzContrib &x = cs[c];
    const int yos = cdiv(x.ny, 8), zos = cdiv(x.nz, 8), nLg = cdiv(x.nL, 1 << glog[c]);
    const int64_t r1 = (int64_t)x.nx * (nLg << glog[c]) * (NS * 32 * yos + 4 * cdiv(yos, OCT));
    const int64_t r2 = (int64_t)x.nx * (NS * 32 * (int64_t)x.nL * zos + 4 * rounds_of(c));
    return ntr * (r1 + r2);
  };
  for (size_t o = 0; o < own.size(); ++o) {
    const OzOwner &ow = own[o];
    if (ow.c1 == ow.c0) continue;
    int64_t rounds = 0;
    for (int c = ow.c0; c < ow.c1; ++c) {
      glog[c] = choose_glog(cdiv(cs[c].nz, 8), cs[c].nL, OCT);
      rounds += rounds_of(c);
    }
    // about four waves of stage-3 tasks (G row tiles each) for this block alone, at least 16 / G rounds each
    const int nos = cdiv(ow.N, 8), G = OCT / std::min(OCT, nos);
    const int64_t tiles = (int64_t)cdiv(cdiv((int64_t)ntau * ow.nx, OZ_M), G) * cdiv(nos, OCT);
    const int64_t want = (4 * (int64_t)std::max(1, nsm) + tiles - 1) / tiles;
    const int64_t nsl = std::max<int64_t>(1, std::min<int64_t>(want, rounds * G / 16));
    const int64_t per = (rounds + nsl - 1) / nsl;
    const size_t u0 = units.size();
    int a = ow.c0;
    int64_t acc = 0;
    for (int c = ow.c0; c <= ow.c1; ++c) {
      if (c == ow.c1 || (c > a && acc + rounds_of(c) > per)) {
        int64_t b = 0;
        for (int k = a; k < c; ++k) b += x_bytes(k);
        units.push_back({(int)o, a, c, (int)(units.size() - u0), 0, b});
        a = c;
        acc = 0;
      }
      if (c < ow.c1) acc += rounds_of(c);
    }
    for (size_t u = u0; u < units.size(); ++u) units[u].nunits = (int)(units.size() - u0);
  }

  // --- V images (shared by the spins): sizes first, to decide whether they are kept
  auto v1_bytes = [&](const OzContrib &c) {
    const int kos = cdiv(c.K1, 8), yos = cdiv(c.ny, 8);
    return (int64_t)c.nx * yos * (NS * kos * 512 + 32 * cdiv(kos, OCT));
  };
  auto v3_bytes = [&](int c) {
    const OzContrib &x = cs[c];
    return (int64_t)cdiv(x.N, 8) * (NS * 512 * (int64_t)x.nL * cdiv(x.nz, 8) + 32 * rounds_of(c));
  };
  bool persist;
  {
    std::map<int, int> seen;
    int64_t tot = 0;
    for (size_t c = 0; c < cs.size(); ++c)
      if (!seen[cs[c].vid]++) tot += v1_bytes(cs[c]) + v3_bytes((int)c);
    persist = tot <= persist_bytes;
  }

  // --- chunks
  struct V1 { size_t col0; std::vector<OzCol1> cols; };
  std::map<int, V1> v1_of;                                     // vid -> column tiles (dst filled per use)
  std::map<std::tuple<int, int, int>, std::pair<int64_t, std::vector<OzRnd>>> v3_of;  // (first vid, last vid, n) -> images
  // FP64 partials held before a reduction: the chunk's budget, at most 1 GB
  const int64_t PART_MAX = std::min<int64_t>((int64_t)1 << 26, budget / 16);
  int64_t part = 0, vbase = 0;
  size_t red0 = 0;
  auto flush_red = [&]() {
    if (red.size() == red0) return;
    OzLaunch l;
    l.kind = 2;
    l.stage = stage0 + 2;
    l.t0 = (int64_t)red0;
    l.n = (int64_t)(red.size() - red0);
    int64_t maxn = 1;
    for (size_t r = red0; r < red.size(); ++r) {
      l.bytes += 16.0 * red[r].nt * red[r].elems * (red[r].nslice + 1);
      maxn = std::max<int64_t>(maxn, (int64_t)red[r].nt * red[r].elems);
    }
    // about four waves of 256-thread CTAs, none with under 256 elements
    const int64_t wantc = (4 * 8 * (int64_t)std::max(1, nsm) + l.n - 1) / l.n;
    l.ny = (int)std::max<int64_t>(1, std::min<int64_t>({wantc, (maxn + 255) / 256, 4096}));
    launches_.push_back(l);
    red0 = red.size();
    part = 0;
  };
  GWGB_REQUIRE(ntau < 65536, GWGB_E_UNSUPPORTED, "too many tau points");
  size_t u0 = 0;  // the next chunk's first unit, in the tau range from t0 on
  for (int t0 = 0; t0 < ntau && !units.empty();) {
    const int nt = std::min(ntr, ntau - t0);
    if (u0 == 0) add_images(t0, nt);
    size_t u1 = u0;
    int64_t tot = 0;
    while (u1 < units.size() && (u1 == u0 || tot + units[u1].bytes <= budget)) {
      if (u1 > u0 && units[u1].idx == 0 && part >= PART_MAX) break;
      tot += units[u1].bytes;
      const OzOwner &ow = own[units[u1].own];
      part += (int64_t)nt * ow.N * ow.nx;
      ++u1;
    }
    for (size_t u = u0; u < u1; ++u) part -= (int64_t)nt * own[units[u].own].N * own[units[u].own].nx;
    if (!persist) {
      v1_of.clear();
      v3_of.clear();
      vbase = 0;
    }
    int64_t voff = vbase;
    const size_t bv0 = builds.size();
    struct Pack { std::vector<int> cs; int64_t slots = 0; };
    std::map<std::tuple<int64_t, int, int>, Pack> packs;  // (B2 block, conj, glog)
    struct Use { int c, d1; int64_t slot, x2, fb, kbase, lgb; };
    std::vector<Use> uses;
    const size_t s3_0 = s3.size();
    int64_t x2 = 0;
    std::vector<OzTask> t3;
    std::vector<std::pair<int64_t, int64_t>> s3_cost;  // of the chunk's units: drains, K steps
    OzLaunch l1, l2, l3;
    l1.stage = stage0; l2.stage = stage0 + 1; l3.stage = stage0 + 2;
    // stage 3: X2 and V3 layout of every unit
    for (size_t u = u0; u < u1; ++u) {
      const Unit &un = units[u];
      const OzOwner &ow = own[un.own];
      const int nf = cdiv((int64_t)nt * ow.nx, OZ_M), nos = cdiv(ow.N, 8), nct = cdiv(nos, OCT);
      const auto vkey = std::make_tuple(cs[un.c0].vid, cs[un.c1 - 1].vid, un.c1 - un.c0);
      auto hit = v3_of.find(vkey);
      const bool fresh = hit == v3_of.end();
      if (fresh) hit = v3_of.emplace(vkey, std::make_pair(voff, std::vector<OzRnd>())).first;
      std::vector<OzRnd> rr;
      int64_t fb = 0, vb = 0;
      std::map<int, size_t> in_unit;  // vid -> first round (the spins of P0 share V3)
      std::vector<int64_t> kbase(un.c1 - un.c0);
      struct VB { int c, Lg, zt, nks; int64_t b16; };
      std::vector<VB> vbs;
      for (int c = un.c0; c < un.c1; ++c) {
        const OzContrib &x = cs[c];
        const int g = 1 << glog[c], nLg = cdiv(x.nL, g), zos = cdiv(x.nz, 8), nzt = cdiv(zos, OCT);
        kbase[c - un.c0] = fb;
        auto iu = in_unit.find(x.vid);
        const bool again = iu != in_unit.end();
        size_t from = again ? iu->second : rr.size();
        if (!again) in_unit[x.vid] = rr.size();
        for (int Lg = 0; Lg < nLg; ++Lg)
          for (int zt = 0; zt < nzt; ++zt) {
            const int nks = nzt > 1 ? std::min(OCT, zos - zt * OCT) : std::min(g, x.nL - Lg * g) * zos;
            OzRnd q{(int32_t)(fb / 16), 0, nks, 0};
            if (again) {
              q.b16 = rr[from++].b16;
            } else {
              q.b16 = (int32_t)(vb / 16);
              if (fresh) vbs.push_back({c, Lg, zt, nks, vb / 16});
              vb += oz_bbytes1(NS, nks);
            }
            rr.push_back(q);
            fb += oz_abytes(NS, nks);
          }
      }
      GWGB_REQUIRE(fb / 16 < INT32_MAX && vb / 16 < INT32_MAX, GWGB_E_UNSUPPORTED, "sliced unit too large");
      const int64_t bz = (int64_t)OCT * vb;
      if (fresh) {
        hit->second.second = rr;
        for (int ct = 0; ct < nct; ++ct) {
          const int noct = std::min(OCT, nos - ct * OCT);
          for (const VB &w : vbs) {
            const OzContrib &x = cs[w.c];
            const int zos = cdiv(x.nz, 8), nzt = cdiv(zos, OCT), g = 1 << glog[w.c];
            const int zr = nzt > 1 ? w.nks : zos;
            builds.push_back({x.v + (int64_t)ct * FK * x.sn + (int64_t)w.Lg * g * x.sL + (int64_t)w.zt * FK * x.sz,
                              voff + ct * bz + w.b16 * 16 * noct, 0, x.sL, x.sn, x.sz, 1 << 20, 8 * zr,
                              x.N - ct * FK, std::min(8 * zr, x.nz - w.zt * FK), 1, w.nks / zr, 0,
                              (int16_t)(8 * noct), (int16_t)w.nks, 1, x.conj3, 0, -1, 0});
          }
        }
        voff += (int64_t)nos * vb;
      }
      const int id = (int)s3.size();
      s3.push_back({x2, fb, hit->second.first, bz, part, (int32_t)rnd.size(), (int32_t)rr.size(), nt * ow.nx, ow.N,
                    ow.nx, ow.N * ow.nx, ow.sn, ow.sx, OCT, 0});
      rnd.insert(rnd.end(), rr.begin(), rr.end());
      int64_t steps = 0;
      for (const OzRnd &q : rr) steps += q.nks;
      s3_cost.push_back({3 * (int64_t)rr.size(), steps});
      for (int ct = 0; ct < nct; ++ct)
        for (int f = 0, G = OCT / std::min(OCT, nos - ct * OCT); f < nf; f += G)
          t3.push_back({id, f | ct << 16, 0, std::min(G, nf - f)});
      for (int c = un.c0; c < un.c1; ++c) {
        const OzContrib &x = cs[c];
        const int g = 1 << glog[c], zos = cdiv(x.nz, 8), R = cdiv(zos, OCT), nLg = cdiv(x.nL, g);
        const int64_t lgb = R > 1 ? (int64_t)NS * zos * 4096 + 512 * R : oz_abytes(NS, g * zos);
        Pack &p = packs[std::make_tuple(x.b2, (int)x.b2conj, glog[c])];
        uses.push_back({c, 0, p.slots, x2, fb, kbase[c - un.c0], lgb});
        p.cs.push_back((int)uses.size() - 1);
        p.slots += ((int64_t)x.nx * nLg * g + 3) / 4 * 4;
        const double rowsx = (double)nt * x.nx * x.nL;
        l1.flops += 8.0 * rowsx * x.ny * x.K1;
        l2.flops += 8.0 * rowsx * x.ny * x.nz;
        l3.flops += 8.0 * rowsx * x.nz * x.N;
      }
      for (const OzRnd &q : rr) l3.ops += nprod * 2.0 * OZ_M * 16.0 * nos * 16.0 * q.nks * nf;
      // partials
      if (un.idx == 0)
        red.push_back({part, ow.out, ow.ostride, ow.N * ow.nx, t0, nt, un.nunits, 0});
      part += (int64_t)nt * ow.N * ow.nx;
      part_ = std::max(part_, part);
      x2 += (int64_t)nf * fb;
    }
    x2_ = std::max(x2_, x2);
    // stage 2: packs
    int64_t x1 = 0;
    std::vector<OzTask> t2;
    int m_kos2 = 1;
    int64_t npk_tiles = 0;
    int64_t nrow = (int64_t)rows.size();
    for (auto &kv : packs) {
      npk_tiles += (int64_t)nt * cdiv(kv.second.slots, OZ_M);
      nrow += (int64_t)cdiv(kv.second.slots, OZ_M) * OZ_M;
    }
    if (nrow > (int64_t)rows.capacity()) rows.reserve(std::max<int64_t>(nrow, 2 * (int64_t)rows.capacity()));
    // row tiles per task: enough tasks for about eight waves, at most 16 tiles
    const int per2 = (int)std::max<int64_t>(1, std::min<int64_t>(16, npk_tiles / (8 * (int64_t)std::max(1, nsm))));
    for (auto &kv : packs) {
      Pack &p = kv.second;
      const int gl = std::get<2>(kv.first);
      const OzContrib &x0 = cs[uses[p.cs[0]].c];
      const int kos = cdiv(x0.ny, 8), R = cdiv(kos, OCT), zos = cdiv(x0.nz, 8), nzt = cdiv(zos, OCT);
      const int nt2 = cdiv(p.slots, OZ_M);
      const int64_t t2b = (int64_t)NS * kos * 4096 + 512 * R;
      const B2 &b2 = b2_of[std::make_pair(x0.b2, (int)x0.b2conj)];
      const int id = (int)s2.size();
      s2.push_back({x1, t2b, b2.b, b2.bt, b2.bz, nt2, kos, zos, gl, (int32_t)rows.size(), x0.nz});
      const size_t r0 = rows.size();
      rows.resize(r0 + (size_t)nt2 * OZ_M, OzRow{0, 0, OZ_NOROW});
      for (int ui : p.cs) {
        Use &us = uses[ui];
        const OzContrib &x = cs[us.c];
        GWGB_REQUIRE(x.ny == x0.ny && x.nz == x0.nz && x.b2z == x0.b2z && x.b2y == x0.b2y && x.b2t == x0.b2t,
                     GWGB_E_INVALID, "sliced pack of unequal blocks");
        const int g = 1 << gl, nLp = cdiv(x.nL, g) * g;
        us.d1 = (int)dst1.size();
        dst1.push_back({x1, t2b, nt2, (int32_t)us.slot, nLp, x.nx});
        check_range(us.slot, (int64_t)x.nx * nLp, (int64_t)nt2 * OZ_M, "sliced stage-2 rows");
        for (int L = 0; L < x.nL; ++L) {
          const int Lq = L & ~3, Lg = L >> gl, step = std::min(4, nLp - Lq);
          OzRow row{us.x2 + us.kbase + Lg * us.lgb, (int32_t)(us.fb / 16),
                    (uint32_t)x.nx << 8 | (uint32_t)((L & (g - 1)) * zos) << 16 |
                        (uint32_t)(gl ? std::min(g, x.nL - Lg * g) * zos : 0) << 24};
          OzRow *to = rows.data() + r0 + us.slot + (int64_t)Lq * x.nx + (L & 3);
          for (int xx = 0; xx < x.nx; ++xx, ++row.pk) to[(int64_t)xx * step] = row;
        }
      }
      x1 += (int64_t)nt * nt2 * t2b;
      m_kos2 = std::max(m_kos2, kos);
      for (int t = 0; t < nt; ++t)
        for (int zt = 0; zt < nzt; ++zt)
          for (int m = 0; m < nt2; m += per2) t2.push_back({id, t | zt << 16, m, std::min(per2, nt2 - m)});
      l2.ops += nprod * 2.0 * OZ_M * 16.0 * zos * 16.0 * kos * nt2 * nt;
    }
    x1_ = std::max(x1_, x1);
    // stage 1: column tiles of every use
    std::vector<OzTask> t1;
    int m_kos1 = 1;
    for (const Use &us : uses) {
      const OzContrib &x = cs[us.c];
      const int kos = cdiv(x.K1, 8), R = cdiv(kos, OCT), yos = cdiv(x.ny, 8);
      auto hit = v1_of.find(x.vid);
      if (hit == v1_of.end()) {
        V1 v;
        for (int yr = 0; yr * OCT < yos; ++yr) {
          const int gs = std::min(OCT, yos - yr * OCT), ng = OCT / gs;
          for (int xa = 0; xa < x.nx; xa += ng) {
            const int n = std::min(ng, x.nx - xa), noct = n * gs;
            v.cols.push_back({voff, 0, (int32_t)(yr * fullA), (int16_t)xa, (int8_t)n, (int8_t)gs,
                              std::min(8 * gs, x.ny - yr * FK)});
            for (int r = 0; r < R; ++r) {
              const int nks = std::min(OCT, kos - r * OCT);
              builds.push_back({x.v + (int64_t)xa * x.sx + (int64_t)yr * FK * x.sy + (int64_t)r * FK * x.sk, voff, x.sx,
                                0, x.sy, x.sk, 8 * gs, 1 << 20, std::min(8 * gs, x.ny - yr * FK), x.K1 - r * FK, n, 1,
                                0, (int16_t)(8 * noct), (int16_t)nks, 1, x.conj1, 0, -1, 0});
              voff += noct * oz_bbytes1(NS, nks);
            }
          }
        }
        hit = v1_of.emplace(x.vid, std::move(v)).first;
      }
      const int d = s1_of[x.ga], nmt = cdiv(s1[d].M, OZ_M);
      GWGB_REQUIRE(s1[d].nL == x.nL && s1[d].kos == kos, GWGB_E_INVALID, "sliced G operand of unequal blocks");
      for (OzCol1 cl : hit->second.cols) {
        cl.dst = us.d1;
        t1.push_back({d, (int32_t)col1.size(), 0, nmt});
        col1.push_back(cl);
        l1.ops += nprod * 2.0 * OZ_M * 16.0 * cl.ngrp * cl.gs * 16.0 * kos * nmt;
      }
      m_kos1 = std::max(m_kos1, kos);
    }
    // few column tiles: split their row tiles over more CTAs
    if ((int64_t)t1.size() < 8 * (int64_t)nsm) {
      const int per1 = (int)std::max<int64_t>(1, (int64_t)t1.size() / std::max(1, nsm));
      std::vector<OzTask> t;
      for (const OzTask &k : t1)
        for (int m = 0; m < k.n; m += per1) t.push_back({k.d, k.i, m, std::min(per1, k.n - m)});
      t1.swap(t);
    }
    vimg_ = std::max(vimg_, voff);
    add_build(persist ? static_ : launches_, bv0, builds.size(), 0, IMG_V, stage0);
    if (persist) vbase = voff;
    // Longest tasks first: CTA c takes tasks c, c + grid, ..., so the loads differ by one task at most.  Cost in K
    // steps of MMAs: a drain of the accumulators takes about eight in stages 1 and 2, three in stage 3.
    auto cost = [&](const OzTask &k, int stage) -> int64_t {
      if (stage == 0) return (int64_t)k.n * (8 * cdiv(s1[k.d].kos, OCT) + s1[k.d].kos);
      if (stage == 1) {
        const int G = OCT / std::min(OCT, s2[k.d].zos - (k.i >> 16) * OCT);
        return (int64_t)cdiv(k.n, G) * 8 * cdiv(s2[k.d].kos, OCT) + (int64_t)k.n * s2[k.d].kos;
      }
      return s3_cost[k.d - s3_0].first + k.n * s3_cost[k.d - s3_0].second;
    };
    auto add_gemm = [&](OzLaunch l, const std::vector<OzTask> &t, int stage, int kos) {
      l.kind = 0;
      l.t0 = (int64_t)tasks.size();
      l.n = (int64_t)t.size();
      if (t.empty()) return;
      std::vector<uint64_t> order(t.size());  // cost, then list order (one word each: a third of the time of pairs)
      for (size_t i = 0; i < t.size(); ++i)
        order[i] = (uint64_t)(UINT32_MAX - std::min<int64_t>(cost(t[i], stage), UINT32_MAX)) << 32 | (uint32_t)i;
      std::sort(order.begin(), order.end());
      tasks.reserve(tasks.size() + t.size());
      for (uint64_t o : order) tasks.push_back(t[(uint32_t)o]);
      oz_rings(NS, stage, kos, &l.args);
      l.d0 = stage;
      launches_.push_back(l);
    };
    // tasks of one round of K, then those of more; the launch statistics go with the larger list
    auto split = [&](OzLaunch l, std::vector<OzTask> &t, int stage, int kos, auto &&kos_of) {
      auto mid = std::stable_partition(t.begin(), t.end(), [&](const OzTask &k) { return kos_of(k) <= OCT; });
      const std::vector<OzTask> one(t.begin(), mid), more(mid, t.end());
      OzLaunch lm = l;
      lm.multi = true;
      OzLaunch &rest = one.size() >= more.size() ? lm : l;
      rest.flops = rest.ops = 0;
      add_gemm(l, one, stage, std::min(kos, OCT));
      add_gemm(lm, more, stage, kos);
    };
    split(l1, t1, 0, m_kos1, [&](const OzTask &k) { return s1[k.d].kos; });
    split(l2, t2, 1, m_kos2, [&](const OzTask &k) { return s2[k.d].kos; });
    add_gemm(l3, t3, 2, 1);
    for (size_t s = s3_0; s < s3.size(); ++s) {
      check_range(s3[s].a, (int64_t)cdiv(s3[s].M, OZ_M) * s3[s].fbytes, x2, "sliced X2 unit");
      check_range(s3[s].b, 0, voff, "sliced V3 images");
    }
    const bool owner_end = u1 == units.size() || units[u1].idx == 0;
    if (u1 == units.size() || (owner_end && part >= PART_MAX)) flush_red();
    u0 = u1;
    if (u0 == units.size()) {
      u0 = 0;
      t0 += ntr;
    }
  }
  for (const RedTask &r : red) {
    check_range(r.part, (int64_t)r.nslice * r.nt * r.elems, std::max<int64_t>(1, part_), "sliced partials");
    check_range(r.out, (int64_t)(r.t0 + r.nt - 1) * r.ostride + r.elems, nout, "sliced output block");
  }
  for (const OzBuild &b : builds)
    check_range(b.dst, b.isb ? (int64_t)(b.rows / 8) * oz_bbytes1(NS, b.nks) : oz_abytes(NS, b.nks),
                std::max({vimg_, a1_, b2_}), "sliced operand image");
  GWGB_REQUIRE(tasks.size() < (size_t)INT32_MAX && rows.size() < (size_t)INT32_MAX && rnd.size() < (size_t)INT32_MAX &&
                   col1.size() < (size_t)INT32_MAX,
               GWGB_E_UNSUPPORTED, "too many sliced GEMM tasks");
  // one allocation for all lists: each separate one cost about as much as building it
  size_t total = 0;
  auto place = [&](const auto &v, auto &l) {
    total = (total + 255) / 256 * 256;
    l.n = v.size();
    l.p = reinterpret_cast<decltype(l.p)>(total);  // its offset, until the buffer exists
    total += v.size() * sizeof(v[0]);
  };
  auto each = [&](auto &&f) {
    f(builds, builds_); f(tasks, tasks_); f(s1, s1_); f(col1, col1_); f(dst1, dst1_); f(s2, s2_); f(rows, rows_);
    f(s3, s3_); f(rnd, rnd_); f(red, red_);
  };
  each(place);
  host_.resize(total);
  each([&](const auto &v, auto &l) {
    if (!v.empty()) std::memcpy(host_.data() + reinterpret_cast<size_t>(l.p), v.data(), v.size() * sizeof(v[0]));
  });
}

void OzPlan::upload(cudaStream_t st) {
  lists_.alloc(host_.size());
  auto at = [&](auto &l) { l.p = reinterpret_cast<decltype(l.p)>(lists_.p + reinterpret_cast<size_t>(l.p)); };
  at(builds_); at(tasks_); at(s1_); at(col1_); at(dst1_); at(s2_); at(rows_); at(s3_); at(rnd_); at(red_);
  if (!host_.empty()) GWGB_CUDA(cudaMemcpyAsync(lists_.p, host_.data(), host_.size(), cudaMemcpyHostToDevice, st));
  GWGB_CUDA(cudaStreamSynchronize(st));
  host_ = std::vector<char>();
}

void OzPlan::build_static(const double2 *V, cudaStream_t st) {
  for (const OzLaunch &l : static_) launch_oz_build(ns_, builds_.p + l.t0, l.n, V, V_.p, st);
}

void OzPlan::run_one(const OzLaunch &l, OzShared &sh, const double2 *V, const double2 *G, const double2 *B2,
                     double2 *out, int nts, double scale, int nsm, int *err, cudaStream_t st) const {
  if (l.kind == 3) {
    char *dst = l.dst == IMG_V ? V_.p : l.dst == IMG_A1 ? sh.A1.p : sh.B2.p;
    launch_oz_build(ns_, builds_.p + l.t0, l.n, l.src == 0 ? V : l.src == 1 ? G : B2, dst, st);
    return;
  }
  if (l.kind == 2) {
    launch_reduce_slices(red_.p + l.t0, (int)l.n, sh.part.p, out, nts, scale, 0, st, l.ny);
    return;
  }
  OzArgs a = l.args;
  a.tasks = tasks_.p + l.t0;
  a.ntasks = (int)l.n;
  a.part = sh.part.p;
  a.err = err;
  if (l.d0 == 0) {
    a.desc = s1_.p;
    a.aux1 = col1_.p;
    a.aux2 = dst1_.p;
    a.A = sh.A1.p;
    a.B = V_.p;
    a.X = sh.X1.p;
  } else if (l.d0 == 1) {
    a.desc = s2_.p;
    a.aux1 = rows_.p;
    a.A = sh.X1.p;
    a.B = sh.B2.p;
    a.X = sh.X2.p;
  } else {
    a.desc = s3_.p;
    a.aux1 = rnd_.p;
    a.aux2 = nullptr;
    a.A = sh.X2.p;
    a.B = V_.p;
    a.X = nullptr;
  }
  launch_oz_gemm(ns_, (int)l.d0, l.multi, a, nsm, st);
}

void OzTransform::build(const std::vector<TSlab> &slabs, int nout, int nin, int row0, bool scaled, int64_t nX, int64_t nY,
                        int nsm, cudaStream_t st) {
  const int NS = 6, OCT = OZ_OCT, FK = 8 * OCT;
  const int kos = cdiv(nin, 8), R = cdiv(kos, OCT), nos = cdiv(nout, 8);
  nin_ = nin;
  row0_ = row0;
  scaled_ = scaled;
  const int64_t fb = (int64_t)NS * kos * 4096 + 512 * R, vb = (int64_t)NS * kos * 512 + 32 * R;
  std::vector<OzBuild> builds;
  std::vector<OzTask> tasks;
  std::vector<OzS3> s3;
  std::vector<OzRnd> rnd;
  int64_t tiles = 0;
  for (const TSlab &x : slabs) tiles += cdiv(x.ncols, OZ_M);
  // the widest column tile (octets) that gives every SM a task: wide tiles read X's images less often
  int oct = OCT;
  while (oct > 1 && tiles * cdiv(nos, oct) < nsm) oct >>= 1;
  for (int r = 0; r < R; ++r)
    rnd.push_back({(int32_t)(r * oz_abytes(NS, OCT) / 16), (int32_t)(r * oz_bbytes1(NS, OCT) / 16),
                   std::min(OCT, kos - r * OCT), 0});
  a_ = 0;
  for (size_t i = 0; i < slabs.size(); ++i) {
    const TSlab &x = slabs[i];
    check_range(x.x, (int64_t)(row0 + nin - 1) * x.ldx + x.ncols, nX, "transform input");
    check_range(x.y, (int64_t)(nout - 1) * x.ldy + x.ncols, nY, "transform output");
    s3.push_back({a_, fb, 0, oct * vb, x.y, 0, R, x.ncols, nout, 1 << 30, 0, x.ldy, 1, oct, 0});
    for (int f = 0; f * OZ_M < x.ncols; ++f) {
      for (int r = 0; r < R; ++r) {
        const int nks = std::min(OCT, kos - r * OCT);
        builds.push_back({x.x + (int64_t)(row0 + r * FK) * x.ldx, a_, 0, 0, 1, x.ldx, 1 << 30, 1 << 20, x.ncols,
                          nin - r * FK, 1, 1, f * OZ_M, OZ_M, (int16_t)nks, 0, 0, 0, scaled ? r * FK : -1, 0});
        a_ += oz_abytes(NS, nks);
      }
      GWGB_REQUIRE(f < 65536, GWGB_E_UNSUPPORTED, "transform slab too large");
      for (int ct = 0; ct * oct < nos; ++ct) tasks.push_back({(int32_t)i, f | ct << 16, 0, 1});
    }
  }
  nbuild_ = (int64_t)builds.size();
  int64_t tb = 0;
  for (int ct = 0; ct * oct < nos; ++ct) {
    const int noct = std::min(oct, nos - ct * oct);
    for (int r = 0; r < R; ++r) {
      const int nks = std::min(OCT, kos - r * OCT);
      builds.push_back({(int64_t)ct * oct * 8 * nin + r * FK, tb, 0, 0, nin, 1, 1 << 20, 1 << 20, nout - ct * oct * 8,
                        nin - r * FK, 1, 1, 0, (int16_t)(8 * noct), (int16_t)nks, 1, 0, 0, scaled ? nin + r * FK : -1, 0});
      tb += noct * oz_bbytes1(NS, nks);
    }
  }
  nT_ = (int64_t)builds.size() - nbuild_;
  gemm_ = OzLaunch{};
  gemm_.n = (int64_t)tasks.size();
  if (tasks.empty()) return;
  oz_rings(NS, 2, 1, &gemm_.args);
  builds_.upload(builds, st);
  tasks_.upload(tasks, st);
  s3_.upload(s3, st);
  rnd_.upload(rnd, st);
  T_.alloc((size_t)tb);
  if (scaled) scale_.alloc(2 * (size_t)nin);
  GWGB_CUDA(cudaStreamSynchronize(st));
}

// In place: a captured graph holds the address of T_ (and, scaled, of T).
void OzTransform::set_matrix(const double2 *T, cudaStream_t st) {
  ready = false;
  if (!scaled_) launch_oz_build(6, builds_.p + nbuild_, nT_, T, T_.p, st);
  GWGB_CUDA(cudaStreamSynchronize(st));
  ready = true;
}

void OzTransform::run(const TSlab *slabs, int nslabs, const double2 *T, const double2 *X, double2 *Y, char *A, int nsm,
                      int *err, cudaStream_t st) const {
  if (scaled_) {
    launch_oz_row_scale(slabs, nslabs, X, row0_, nin_, scale_.p, st);
    launch_oz_build(6, builds_.p + nbuild_, nT_, T, T_.p, st, scale_.p);
  }
  launch_oz_build(6, builds_.p, nbuild_, X, A, st, scale_.p);
  OzArgs a = gemm_.args;
  a.desc = s3_.p;
  a.tasks = tasks_.p;
  a.ntasks = (int)gemm_.n;
  a.aux1 = rnd_.p;
  a.aux2 = nullptr;
  a.A = A;
  a.B = T_.p;
  a.X = nullptr;
  a.part = Y;
  a.err = err;
  launch_oz_gemm(6, 2, false, a, nsm, st);
}

void OzTransform::free() {
  builds_.free(); tasks_.free(); s3_.free(); rnd_.free(); T_.free(); scale_.free();
  gemm_.n = 0;
  ready = false;
}

void OzPlan::free() {
  V_.free();
  lists_.free();
  host_ = std::vector<char>();
  launches_.clear();
  static_.clear();
  vimg_ = a1_ = b2_ = x1_ = x2_ = part_ = 0;
}

}  // namespace gwgb
