// Planner: from a parsed expression + extents to the launch description.
//
// This replaces the reference's offline search
// (cogent/src/generators/configurations.py:15-289 -> enumeration.py:15-278 ->
// cost_models.py:11-39), which enumerates thread-block / register-tile index
// groups and ranks them by estimated DRAM transactions.  The B200 kernels tile
// the FLATTENED external index spaces instead of per-index boxes, so the search
// collapses to: classify and order the indices, fuse what is contiguous, pick
// the loader per operand, pick a CTA tile and (for small outputs) a K split.
//
//   M  = external indices of X, ordered by their stride in the output
//   N  = external indices of Y, ordered by their stride in the output
//   K  = contraction indices, ordered by their stride in whichever operand has
//        a contraction index as its fastest index
// where X is the operand that carries the output's fastest index (operands are
// swapped if that is the right one; the product is commutative).  The reference
// makes the same choice when it maps the input holding the output's fastest
// index to the thread-block X dimension (enumeration.py:72-100).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <sstream>

#include "tc_internal.h"

namespace {

struct Dim {
  int64_t extent, s_in, s_out;  // for K: s_in = stride in X, s_out = stride in Y
};

int find(const std::vector<std::string>& v, const std::string& s) {
  for (size_t i = 0; i < v.size(); ++i)
    if (v[i] == s) return (int)i;
  return -1;
}

std::vector<int64_t> compact_strides(const std::vector<std::string>& idx, const tc_plan& p) {
  std::vector<int64_t> s(idx.size());
  int64_t acc = 1;
  for (size_t i = 0; i < idx.size(); ++i) {
    s[i] = acc;
    acc *= p.idx_extent[find(p.idx_names, idx[i])];
  }
  return s;
}

// Drops unit extents and merges neighbours that are contiguous in both tensors.
std::vector<Dim> fuse(std::vector<Dim> d) {
  std::vector<Dim> out;
  for (const Dim& x : d) {
    if (x.extent == 1) continue;
    if (!out.empty()) {
      Dim& b = out.back();
      if (x.s_in == b.s_in * b.extent && x.s_out == b.s_out * b.extent) {
        b.extent *= x.extent;
        continue;
      }
    }
    out.push_back(x);
  }
  return out;
}

bool to_dims(const std::vector<Dim>& d, TcDims* t, int64_t* flat) {
  if ((int)d.size() > TC_MAX_DIMS) return false;
  std::memset(t, 0, sizeof(*t));
  t->n = (int)d.size();
  int64_t f = 1;
  for (size_t i = 0; i < d.size(); ++i) {
    t->extent[i] = (uint32_t)d[i].extent;
    t->s_in[i] = d[i].s_in;
    t->s_out[i] = d[i].s_out;
    f *= d[i].extent;
    if (f >= (int64_t(1) << 31)) return false;
  }
  *flat = f;
  return true;
}

int64_t span(const std::vector<int64_t>& ext, const std::vector<int64_t>& str) {
  int64_t s = 1;
  for (size_t i = 0; i < ext.size(); ++i) s += (ext[i] - 1) * str[i];
  return s;
}

// A consumer warp's batch of 8 output rows (n = base + 2g + parity, WM consecutive m) of the persistent fp64
// kernels is one box of a rank-5 view of C when, with each class's dimensions fused as far as they are
// contiguous IN C (the flattened index does not change by that),
//   * the warp's WM outputs of a row sit inside one contiguous run: the fastest fused M dimension has
//     stride 1 and is the only one, or a multiple of the tile,
//   * the 16 rows of two batches stay inside N's fastest fused dimension (the only one, or a multiple of
//     16), which must be even so that n splits into (parity, n / 2),
//   * what is left of both classes fits the two remaining tensor dimensions, and every stride keeps
//     16-byte alignment.
// Then one tiled TMA reduce-add (or store) replaces eight per-row bulk copies (*per_warp); a whole bm x bn tile
// is a box too when its bn rows stay inside N's fastest fused dimension (*per_tile).
void out_box_view(const TcKernelArgs& a, int es, int bm, int bn, TcOutMap* map, bool* per_warp, bool* per_tile) {
  *per_warp = false;
  *per_tile = false;
  *map = TcOutMap{};
  if (!(es == 8 && a.vec_c == 4 && a.M.n >= 1 && a.N.n >= 1 && a.M.s_out[0] == 1)) return;
  auto fuse_out = [](const TcDims& cls, std::vector<int64_t>* ext, std::vector<int64_t>* str) {
    for (int d = 0; d < cls.n; ++d) {
      if (!ext->empty() && cls.s_out[d] == str->back() * ext->back()) ext->back() *= cls.extent[d];
      else { ext->push_back(cls.extent[d]); str->push_back(cls.s_out[d]); }
    }
  };
  std::vector<int64_t> me, ms, ne, ns;
  fuse_out(a.M, &me, &ms);
  fuse_out(a.N, &ne, &ns);
  bool ok = (me.size() == 1 || me[0] % bm == 0) && ne[0] % 2 == 0 && (ne.size() == 1 || ne[0] % 16 == 0) &&
            (me.size() - 1) + (ne.size() - 1) <= 2;
  for (size_t d = 0; d < ne.size(); ++d) ok = ok && ns[d] % 2 == 0 && ns[d] > 0 && ns[d] < (int64_t(1) << 36) && ne[d] < (int64_t(1) << 31);
  for (size_t d = 1; d < me.size(); ++d) ok = ok && ms[d] % 2 == 0 && ms[d] > 0 && ms[d] < (int64_t(1) << 36) && me[d] < (int64_t(1) << 31);
  ok = ok && me[0] < (int64_t(1) << 31);
  if (!ok) return;
  TcOutMap& o = *map;
  o.e0 = (uint32_t)me[0];
  o.f0 = (uint32_t)ne[0];
  o.stride_n = ns[0];
  o.ne = (int32_t)ne.size() - 1;
  o.me = (int32_t)me.size() - 1;
  int r = 0;
  for (size_t d = 1; d < ne.size(); ++d, ++r) { o.ext[r] = (uint32_t)ne[d]; o.stride[r] = ns[d]; }
  for (size_t d = 1; d < me.size(); ++d, ++r) { o.ext[r] = (uint32_t)me[d]; o.stride[r] = ms[d]; }
  *per_warp = true;
  *per_tile = ne.size() == 1 || ne[0] % bn == 0;
}

// Cut tiles of the output-resident kernel: how its bm x bn tile is laid over the output so that it is one box of a
// rank-<=5 view of C.  Per class either the dimensions fused as far as they are contiguous in C, of which a tile takes a
// range of the first, or the planner's own dimensions, of which it takes ranges of the first two -- what an output with
// short runs needs (24-element runs: 5 of them make 120 of 128 rows: triples term 24/16, K = 24, 155 us on one B200, 211
// on the best flat tile of the other kernels, 261 on the 128 x 64 one).  Every even b0 and every c0 is tried; the score is
// the number of tiles (rows that a tile leaves unused cost as much as used ones) times a penalty for short pieces: of C
// (b0 elements, or b0 * c0 where the next index of C is N's first) and of an operand whose fastest index is external.
struct BoxPlan {
  bool ok = false;
  double score = 0, tiles = 0;
  TcCut m{}, n{};
  TcBoxMap map{};
  int across_x = 0, across_y = 0;
};
BoxPlan plan_boxes(const std::vector<Dim>& dm, const std::vector<Dim>& dn, uint32_t bm, uint32_t bn) {
  BoxPlan best;
  if (dm.empty() || dm[0].s_out != 1 || dm[0].extent % 2 != 0) return best;
  for (const std::vector<Dim>* l : {&dm, &dn})
    for (const Dim& d : *l)
      if ((d.s_out != 1 && d.s_out % 2 != 0) || d.s_out <= 0 || d.s_out >= (int64_t(1) << 36) || d.extent >= (int64_t(1) << 31)) return best;
  auto fuse_out = [](const std::vector<Dim>& l) {
    std::vector<Dim> r;
    for (const Dim& d : l) {
      if (!r.empty() && d.s_out == r.back().s_out * r.back().extent) r.back().extent *= d.extent;
      else r.push_back(d);
    }
    return r;
  };
  auto unit_at = [](const std::vector<Dim>& l) {
    for (size_t i = 0; i < l.size(); ++i)
      if (l[i].extent > 1 && l[i].s_in == 1) return (int)i;
    return -1;
  };
  auto product = [](const std::vector<Dim>& l, size_t from) {
    int64_t r = 1;
    for (size_t i = from; i < l.size(); ++i) r *= l[i].extent;
    return r;
  };
  auto piece = [](double bytes) { return bytes >= 256 ? 1.0 : bytes >= 128 ? 1.02 : bytes >= 64 ? 1.08 : bytes >= 32 ? 1.25 : 1.7; };
  auto gather = [](int64_t run) { return run >= 4 ? 1.0 : run >= 2 ? 1.15 : 1.4; };
  const int ux = unit_at(dm), uy = unit_at(dn);
  const std::vector<Dim> fm = fuse_out(dm), fn = fuse_out(dn);
  for (int two_m = 0; two_m < 2; ++two_m)
    for (int two_n = 0; two_n < 2; ++two_n) {
      const std::vector<Dim>&lm = two_m ? dm : fm, &ln = two_n ? dn : fn;
      if ((two_m && dm.size() < 2) || (two_n && dn.size() < 2)) continue;
      const size_t m_rest = two_m ? 2 : 1, n_rest = two_n ? 2 : 1;
      if (lm.size() > m_rest + 2 || ln.size() > n_rest + 2) continue;
      // six dimensions fit where the one left of each class are neighbours in C and share a dimension of the map
      const bool shared = lm.size() + ln.size() == 6 && lm.size() == m_rest + 1 && ln.size() == n_rest + 1 &&
                          lm.back().extent * ln.back().extent < (int64_t(1) << 31) &&
                          (lm.back().s_out == ln.back().s_out * ln.back().extent || ln.back().s_out == lm.back().s_out * lm.back().extent);
      if (lm.size() + ln.size() > 5 && !shared) continue;
      const int64_t e0 = lm[0].extent, e1 = two_m ? lm[1].extent : 1, f0 = ln.empty() ? 1 : ln[0].extent, f1 = two_n ? ln[1].extent : 1;
      const int64_t rest = product(lm, m_rest) * product(ln, ln.empty() ? 0 : n_rest);
      // N's cuts, the one of fewest tiles first in line (its choice depends on M's only where a run and its n are one piece)
      struct NCut { uint32_t c0, c1; int64_t s0, s1; double cost; };
      std::vector<NCut> ncuts;
      size_t fewest = 0;
      for (uint32_t c0 = std::min<int64_t>(bn, f0); c0 >= 1; --c0) {
        // (an input read in pairs along N's first index: pairs lie in one run and tiles start on 16 bytes)
        if (uy == 0 && dn[0].extent % 2 == 0 && c0 % 2 != 0) continue;
        const int64_t s0 = (f0 + c0 - 1) / c0;
        const int64_t s1 = two_n ? (f1 + bn / c0 - 1) / (bn / c0) : 1;
        const uint32_t c1 = two_n ? (uint32_t)((f1 + s1 - 1) / s1) : 1;
        const double cost = (double)(s0 * s1) * (uy >= 0 ? gather(uy == 0 ? c0 : uy == 1 && two_n ? c1 : 1) : 1.0);
        if (!ncuts.empty() && cost < ncuts[fewest].cost) fewest = ncuts.size();
        ncuts.push_back({c0, c1, s0, s1, cost});
      }
      for (uint32_t b0 = std::min<int64_t>(bm, e0); b0 >= 2; b0 -= 2) {
        const int64_t t0 = (e0 + b0 - 1) / b0;
        const int64_t t1 = two_m ? (e1 + bm / b0 - 1) / (bm / b0) : 1;
        const uint32_t b1 = two_m ? (uint32_t)((e1 + t1 - 1) / t1) : 1;
        const bool adjacent = b0 == e0 && !ln.empty() && ln[0].s_out == e0;
        for (size_t nc = adjacent ? 0 : fewest; nc < (adjacent ? ncuts.size() : std::min(fewest + 1, ncuts.size())); ++nc) {
          const uint32_t c0 = ncuts[nc].c0, c1 = ncuts[nc].c1;
          const int64_t s0 = ncuts[nc].s0, s1 = ncuts[nc].s1;
          const double tiles = (double)(t0 * t1) * (double)(s0 * s1) * (double)rest;
          if (tiles >= 2.0e9) continue;
          double score = (double)(t0 * t1) * ncuts[nc].cost * (double)rest * piece(8.0 * b0 * (adjacent ? c0 : 1));
          if (ux >= 0) score *= gather(ux == 0 ? b0 : ux == 1 && two_m ? b1 : 1);
          if (best.ok && score >= best.score) continue;
          best.ok = true;
          best.score = score;
          best.tiles = tiles;
          best.m = {b0, b1, (uint32_t)e0, (uint32_t)e1, (uint32_t)t0, (uint32_t)t1};
          best.n = {c0, c1, (uint32_t)f0, (uint32_t)f1, (uint32_t)s0, (uint32_t)s1};
          best.across_x = ux == 1 && two_m && b1 > 1 ? (int)b1 : 0;
          best.across_y = uy == 1 && two_n && c1 > 1 ? (int)c1 : 0;
          TcBoxMap& o = best.map;
          o = TcBoxMap{};
          o.mr = o.nr = 1;
          auto add = [&](const Dim& d, uint32_t box) {
            o.ext[o.rank] = (uint32_t)d.extent;
            o.stride[o.rank] = d.s_out;
            o.box[o.rank] = box;
            return (int8_t)o.rank++;
          };
          add(lm[0], b0);
          if (!ln.empty()) o.n0 = add(ln[0], c0);
          if (two_n) o.n1 = add(ln[1], c1);
          if (two_m) o.m1 = add(lm[1], b1);
          if (shared) {
            const bool m_first = lm.back().s_out < ln.back().s_out;
            Dim both = m_first ? lm.back() : ln.back();
            o.m_step = m_first ? 1 : (uint32_t)both.extent;
            o.n_step = m_first ? (uint32_t)both.extent : 1;
            both.extent *= m_first ? ln.back().extent : lm.back().extent;
            o.mr0 = o.nr0 = add(both, 1);
            continue;
          }
          if (lm.size() > m_rest) { o.mr0 = add(lm[m_rest], 1); o.mr = (uint32_t)lm[m_rest].extent; }
          if (lm.size() > m_rest + 1) o.mr1 = add(lm[m_rest + 1], 1);
          if (ln.size() > n_rest) { o.nr0 = add(ln[n_rest], 1); o.nr = (uint32_t)ln[n_rest].extent; }
          if (ln.size() > n_rest + 1) o.nr1 = add(ln[n_rest + 1], 1);
        }
      }
    }
  return best;
}

// The staged output layout of the fp32 kernels: a tile's rows split into runs of E0 elements that are contiguous in
// the output (E0 a multiple of 4, tiles 16-byte aligned); `n_adjacent`: consecutive n are adjacent in the output
// inside blocks of N's fastest extent, so a run and its n leave as one chunk.  Returns E0, or 0 where bulk copies do
// not pay (chunks under 256 bytes) or are not possible.
int64_t staged_run(const TcKernelArgs& a, int bm, int bn, int es, bool* n_adjacent) {
  const int V = 16 / es;
  *n_adjacent = false;
  if (!(a.M.n > 0 && a.M.s_out[0] == 1 && a.vec_c >= V)) return 0;
  const int64_t e = a.M.extent[0];
  const int64_t e0 = e % bm == 0 ? bm : (bm % e == 0 ? e : std::gcd<int64_t>(bm, e));
  if (e0 % V != 0 || e0 < V) return 0;
  *n_adjacent = e0 == e && a.N.n > 0 && a.N.s_out[0] == e && (int64_t)a.N.extent[0] >= bn;
  return (*n_adjacent || e0 * es >= 256) ? e0 : 0;
}
bool wt_eligible(const TcKernelArgs& a, int bm, int es) {
  bool adj;
  return es == 4 && staged_run(a, bm, 128, es, &adj) > 0;
}

}  // namespace

int tc_plan_build(tc_plan* p, std::string* why) {
  std::string dummy;
  if (!why) why = &dummy;
  const TcExpr& e = p->expr;
  const int es = p->dtype == TC_F64 ? 8 : 4;
  auto ext_of = [&](const std::string& n) { return p->idx_extent[find(p->idx_names, n)]; };

  // Per-tensor extents and strides in written order.
  const std::vector<std::string>* tidx[3] = {&e.out_idx, &e.left_idx, &e.right_idx};
  std::vector<int64_t> text[3], tstr[3];
  for (int t = 0; t < 3; ++t) {
    for (const std::string& n : *tidx[t]) text[t].push_back(ext_of(n));
    if (p->custom_strides[t]) {
      if (p->strides[t].size() != tidx[t]->size()) { *why = "stride count does not match tensor rank"; return TC_ERR_INVALID_ARG; }
      tstr[t] = p->strides[t];
      for (int64_t s : tstr[t])
        if (s <= 0) { *why = "strides must be positive"; return TC_ERR_EXTENT; }
      // strides that merely restate the compact layout keep the plan eligible for everything compact plans get
      if (tstr[t] == compact_strides(*tidx[t], *p)) p->custom_strides[t] = false;
    } else {
      tstr[t] = compact_strides(*tidx[t], *p);
    }
  }
  // The output must not alias itself: sorted by stride, each stride must clear the previous extent.
  {
    std::vector<std::pair<int64_t, int64_t>> se;
    for (size_t i = 0; i < text[0].size(); ++i)
      if (text[0][i] > 1) se.push_back({tstr[0][i], text[0][i]});
    std::sort(se.begin(), se.end());
    int64_t need = 1;
    for (auto& x : se) {
      if (x.first < need) { *why = "output strides make elements alias"; return TC_ERR_EXTENT; }
      need = x.first * x.second;
    }
  }
  p->count_c = std::accumulate(text[0].begin(), text[0].end(), int64_t(1), std::multiplies<int64_t>());
  p->count_a = std::accumulate(text[1].begin(), text[1].end(), int64_t(1), std::multiplies<int64_t>());
  p->count_b = std::accumulate(text[2].begin(), text[2].end(), int64_t(1), std::multiplies<int64_t>());
  p->size_c = span(text[0], tstr[0]);
  p->size_a = span(text[1], tstr[1]);
  p->size_b = span(text[2], tstr[2]);

  // Which operand carries the output's fastest (non-unit) index?
  int fvi = -1;
  for (size_t i = 0; i < e.out_idx.size(); ++i)
    if (text[0][i] > 1 && (fvi < 0 || tstr[0][i] < tstr[0][fvi])) fvi = (int)i;
  p->swapped = fvi >= 0 && find(e.left_idx, e.out_idx[fvi]) < 0;
  const int X = p->swapped ? 2 : 1, Y = p->swapped ? 1 : 2;

  std::vector<Dim> dm, dn, dk;
  for (size_t i = 0; i < e.out_idx.size(); ++i) {
    const std::string& n = e.out_idx[i];
    const int ix = find(*tidx[X], n), iy = find(*tidx[Y], n);
    if (ix >= 0) dm.push_back({text[0][i], tstr[X][ix], tstr[0][i]});
    else dn.push_back({text[0][i], tstr[Y][iy], tstr[0][i]});
  }
  for (const std::string& n : e.sum_idx) {
    const int ix = find(*tidx[X], n), iy = find(*tidx[Y], n);
    dk.push_back({ext_of(n), tstr[X][ix], tstr[Y][iy]});
  }
  auto by_out = [](const Dim& a, const Dim& b) { return a.s_out < b.s_out; };
  std::stable_sort(dm.begin(), dm.end(), by_out);
  std::stable_sort(dn.begin(), dn.end(), by_out);
  bool x_k_unit = false, y_k_unit = false;
  for (const Dim& d : dk) {
    if (d.extent > 1 && d.s_in == 1) x_k_unit = true;
    if (d.extent > 1 && d.s_out == 1) y_k_unit = true;
  }
  if (!x_k_unit && y_k_unit)
    std::stable_sort(dk.begin(), dk.end(), [](const Dim& a, const Dim& b) { return a.s_out < b.s_out; });
  else
    std::stable_sort(dk.begin(), dk.end(), [](const Dim& a, const Dim& b) { return a.s_in < b.s_in; });
  dm = fuse(dm);
  dn = fuse(dn);
  dk = fuse(dk);

  // Operand-friendly orders.  By output stride alone, an operand whose own fastest index is an external one that
  // comes late in the output would be gathered 8 bytes per sector (the reference's mapping search blocks two
  // indices in that situation, cogent/src/algs/bases/enumeration.py:72-278).  Tiles here are ranges of the
  // flattened class, so the same effect comes from the ORDER of the class's dimensions:
  //   * N, fp64 (never holds the output's fastest index): ordered by stride in Y when Y's fastest index is external;
  //   * M, fp64: the output's fastest index a and X's fastest external index x are both split by 4 and the digits
  //     ordered (a_lo, x_lo, a_hi, ..., x_hi): a thread still owns 4 consecutive output elements (32 bytes), and
  //     the 4 lanes that share an a_lo fetch 4 consecutive x, one whole sector of X.  (Putting x_lo first made
  //     the loads 16-byte vectors but sent the output through the element-wise epilogue: measured slower.)
  if (p->dtype == TC_F64 && !y_k_unit && dn.size() > 1) {  // (the fp32 epilogues lean on N's order in the output)
    bool y_ext_unit = false;
    for (const Dim& d : dn) y_ext_unit = y_ext_unit || (d.extent > 1 && d.s_in == 1);
    if (y_ext_unit && dn[0].s_in != 1) {
      std::stable_sort(dn.begin(), dn.end(), [](const Dim& a, const Dim& b) { return a.s_in < b.s_in; });
      dn = fuse(dn);
    }
  }
  // The output-resident kernel's tiles are cut over two of M's dimensions instead (plan_boxes): for it the dimensions stay
  // whole, the one that comes second chosen by the cost model below.
  const std::vector<Dim> dm_whole = dm;
  auto box_dims = [&](int second) {
    std::vector<Dim> r = dm_whole;
    if (second > 1) std::rotate(r.begin() + 1, r.begin() + second, r.begin() + second + 1);
    return r;
  };
  auto best_boxes = [&](uint32_t bm, uint32_t bn, int* order) {
    BoxPlan best;
    for (int second = 1; second < std::max<int>(2, (int)dm_whole.size()); ++second) {
      if (p->box_order >= 0 && second != p->box_order) continue;
      const BoxPlan q = plan_boxes(box_dims(second), dn, bm, bn);
      if (q.ok && (!best.ok || q.score < best.score)) { best = q; *order = second; }
    }
    return best;
  };
  if (p->box_order >= 0) dm = box_dims(p->box_order);
  else if (p->dtype == TC_F64 && !x_k_unit && dm.size() > 1 && dm[0].s_in != 1 && dm[0].s_out == 1 && dm[0].extent % 4 == 0) {
    for (size_t j = 1; j < dm.size(); ++j) {
      if (dm[j].s_in != 1 || dm[j].extent < 4 || dm[j].extent % 4 != 0) continue;
      if (dm.size() + 2 > (size_t)TC_MAX_DIMS) break;
      // only when a 128-row tile in output order would hold at most two values of x: with short faster
      // dimensions the tile reaches x by itself and keeps the cheaper row-wise output
      int64_t before = 1;
      for (size_t i = 0; i < j; ++i) before *= dm[i].extent;
      if (before < 64) break;
      const Dim o = dm[0], x = dm[j];
      std::vector<Dim> r;
      r.push_back({4, o.s_in, o.s_out});            // 4 consecutive output elements: 32 bytes of C per thread
      r.push_back({4, x.s_in, x.s_out});            // 4 consecutive x: one whole sector of X per 4 lanes
      if (o.extent / 4 > 1) r.push_back({o.extent / 4, o.s_in * 4, o.s_out * 4});
      for (size_t i = 1; i < dm.size(); ++i) {
        if (i != j) r.push_back(dm[i]);
        else if (x.extent / 4 > 1) r.push_back({x.extent / 4, x.s_in * 4, x.s_out * 4});
      }
      dm = r;
      break;
    }
  }

  // K, fp64: where each input's fastest index is a contraction index, but not the same one, either order of the
  // flattened contraction walks one of the two in 8-byte pieces of different sectors.  Both digits are cut by four and
  // the low parts put first -- (4 of X's, 4 of Y's, the rest): a K step of sixteen is then a 4 x 4 block of which both
  // inputs read whole sectors.  Extents that four does not divide are rounded up; positions beyond them have offset -1
  // in the tables, which the loaders of the persistent fp64 kernels (and only they) turn into zeros.
  // What is rounded up costs products, so blocks are taken only where they add few.  In plain order a sector of Y is met
  // again only after all positions of the contraction indices before Y's: while Y stays in L2 that costs little, beyond
  // that memory is read up to four times.  Measured on one B200, 14 000 random sums, time in plain order over time in
  // blocks, per product (10 % / half of them are above): Y over 32 MB 1.15 / 1.36 to 2.4 where X's extent is even (plain
  // order reads X 16 bytes at a time), 1.14 / 1.39 to 2.2 where it is odd; up to 32 MB 1.02 / 1.08 to 1.16 even, and odd
  // 1.18 / 1.39 with fewer than 8 positions before Y's index, 0.98 / 1.19 with fewer than 32, beyond 0.9 / 1.11 (Y over
  // 16 MB) and 0.76 / 0.9.  With the limits below the choice is 1.4 % slower than the better of the two throughout;
  // blocks always 5.8 %, never 24 %.
  int64_t kcut_x = 0, kcut_y = 0;  // extents of the two digits that were cut (0: none)
  if (p->dtype == TC_F64 && p->block_k && x_k_unit && y_k_unit && !dk.empty() && dk[0].s_in == 1 && dk[0].s_out != 1 &&
      dk.size() + 2 <= (size_t)TC_MAX_DIMS) {
    for (size_t j = 1; j < dk.size(); ++j) {
      if (dk[j].s_out != 1) continue;
      const Dim x = dk[0], y = dk[j];
      const double given = (double)x.extent * (double)y.extent;
      const double rounded = 16.0 * (double)((x.extent + 3) / 4) * (double)((y.extent + 3) / 4);
      double before = 1.0;
      for (size_t i = 0; i < j; ++i) before *= (double)dk[i].extent;
      const bool even = x.extent % 2 == 0;
      const double y_bytes = (double)(p->swapped ? p->count_a : p->count_b) * es;
      const double limit = y_bytes > 32.0e6 ? (even ? 1.35 : 1.5)
                           : even           ? 1.1
                                            : before < 8.0 ? 1.34 : before < 32.0 ? 1.15 : y_bytes > 16.0e6 ? 1.1 : 0.0;
      if (rounded > given * limit) break;
      kcut_x = x.extent;
      kcut_y = y.extent;
      std::vector<Dim> r = {{4, x.s_in, x.s_out}, {4, y.s_in, y.s_out}};
      r.push_back({(x.extent + 3) / 4, x.s_in * 4, x.s_out * 4});
      r.push_back({(y.extent + 3) / 4, y.s_in * 4, y.s_out * 4});
      for (size_t i = 1; i < dk.size(); ++i)
        if (i != j) r.push_back(dk[i]);
      dk = r;
      break;
    }
  }

  TcKernelArgs& a = p->args;
  std::memset(&a, 0, sizeof(a));
  int64_t mf = 1, nf = 1, kf = 1;
  TcDims kd;
  if (!to_dims(dm, &a.M, &mf) || !to_dims(dn, &a.N, &nf) || !to_dims(dk, &kd, &kf)) {
    *why = "a fused index class has more than 8 dimensions or 2^31 elements";
    return TC_ERR_UNSUPPORTED;
  }
  a.Mflat = (uint32_t)mf;
  a.Nflat = (uint32_t)nf;
  a.Kflat = (uint32_t)kf;
  p->kdims = kd;
  // Rules on the length of the contraction go by its true length: a sum is not long enough to be sliced, and does not
  // need scratch, because its positions were rounded up.
  const int64_t k_true = kcut_x > 0 ? kf / (16 * ((kcut_x + 3) / 4) * ((kcut_y + 3) / 4)) * kcut_x * kcut_y : kf;

  // Contraction offset tables (one entry per flattened k), digits carried along as on an odometer.
  p->h_koff_x.assign(kf, 0);
  p->h_koff_y.assign(kf, 0);
  {
    int64_t digit[TC_MAX_DIMS] = {}, ox = 0, oy = 0;
    for (int64_t k = 0; k < kf; ++k) {
      const bool hole = kcut_x > 0 && (digit[0] + 4 * digit[2] >= kcut_x || digit[1] + 4 * digit[3] >= kcut_y);
      p->h_koff_x[k] = hole ? -1 : ox;
      p->h_koff_y[k] = hole ? -1 : oy;
      for (int d = 0; d < kd.n; ++d) {
        ox += kd.s_in[d];
        oy += kd.s_out[d];
        if (++digit[d] < (int64_t)kd.extent[d]) break;
        ox -= (int64_t)kd.extent[d] * kd.s_in[d];
        oy -= (int64_t)kd.extent[d] * kd.s_out[d];
        digit[d] = 0;
      }
    }
  }

  // Kernel family.
  TcKernelChoice& c = p->choice;
  c.dtype = p->dtype;
  const int path = p->opt.path;
  if (p->dtype == TC_F64) {
    if (path == TC_PATH_FFMA || path == TC_PATH_3XTF32 || path == TC_PATH_TCGEN05) { *why = "fp32 path requested for an fp64 plan"; return TC_ERR_INVALID_ARG; }
    c.math = path == TC_PATH_DFMA ? TC_MATH_SIMT : TC_MATH_DMMA;
  } else {
    if (path == TC_PATH_DMMA || path == TC_PATH_DFMA) { *why = "fp64 path requested for an fp32 plan"; return TC_ERR_INVALID_ARG; }
    // AUTO: three TF32 tensor-core products per fp32 product measured faster than FFMA on B200 (the
    // vector-pipe kernel is issue-bound on short contractions) at the same observed error (~3e-7).
    // The tcgen05 form of the same arithmetic (TMEM accumulators) is opt-in: measured beside the mma.sync one.
    c.math = path == TC_PATH_FFMA ? TC_MATH_SIMT : path == TC_PATH_TCGEN05 ? TC_MATH_TF32TC : TC_MATH_TF32X3;
  }

  // Loader per operand.
  const int V = 16 / es;
  auto loader = [&](const TcDims& ext, bool k_is_in, bool* vec, bool* kvec, int32_t* lanes_k) {
    *vec = false;
    *kvec = false;
    *lanes_k = 1;
    auto ks = [&](int d) { return k_is_in ? kd.s_in[d] : kd.s_out[d]; };
    if (ext.n > 0 && ext.s_in[0] == 1) {
      bool ok = ext.extent[0] % V == 0;
      for (int d = 1; d < ext.n; ++d) ok = ok && ext.s_in[d] % V == 0;
      for (int d = 0; d < kd.n; ++d) ok = ok && ks(d) % V == 0;
      *vec = ok;
    } else if (kd.n > 0 && ks(0) == 1) {
      *lanes_k = 32 / es;
      bool ok = kd.extent[0] % V == 0;
      for (int d = 1; d < kd.n; ++d) ok = ok && ks(d) % V == 0;
      for (int d = 0; d < ext.n; ++d) ok = ok && ext.s_in[d] % V == 0;
      *kvec = ok;
    }
  };
  loader(a.M, true, &c.vec_x, &c.kvec_x, &a.lanes_k_x);
  loader(a.N, false, &c.vec_y, &c.kvec_y, &a.lanes_k_y);
  a.kstep_x = a.kstep_y = 1;
  if (kcut_x > 0) {
    // Y's unit stride is the second digit: its lanes walk every fourth position; pairs of k along X must not straddle its end
    a.lanes_k_y = 32 / es;
    a.kstep_y = 4;
    if (kcut_x % V != 0) c.kvec_x = false;
  }
  // An operand is a plain 2-D matrix (k fastest, then the flattened external index at a constant pitch)
  // when it has one fused contraction dimension of stride 1 and its external dimensions are contiguous
  // among themselves: then a tile of the flattened class is a box, which TMA can fetch (rows 16 bytes apart or more).
  auto affine = [&](const TcDims& ext, bool k_is_in) {
    if (kd.n != 1 || (k_is_in ? kd.s_in[0] : kd.s_out[0]) != 1 || ext.n < 1) return false;
    for (int d = 1; d < ext.n; ++d)
      if (ext.s_in[d] != ext.s_in[d - 1] * (int64_t)ext.extent[d - 1]) return false;
    return ext.s_in[0] % (16 / es) == 0 && ext.s_in[0] >= (int64_t)kd.extent[0];
  };
  c.tma_x = affine(a.M, true);
  c.tma_y = affine(a.N, false);
  // The transposed case: the whole external class is one contiguous run and the single contraction dimension lies
  // at a constant pitch (rows of the box are then k, 16 bytes apart or more).
  auto affine_ext = [&](const TcDims& ext, bool k_is_in) {
    if (kd.n != 1 || ext.n < 1 || ext.s_in[0] != 1) return false;
    int64_t run = 1;
    for (int d = 0; d < ext.n; ++d) {
      if (ext.s_in[d] != run) return false;
      run *= (int64_t)ext.extent[d];
    }
    const int64_t pitch = k_is_in ? kd.s_in[0] : kd.s_out[0];
    return pitch % (16 / es) == 0 && pitch >= run;
  };
  c.tma_xe = es == 4 && affine_ext(a.M, true);
  c.tma_ye = es == 4 && affine_ext(a.N, false);

  // Contiguous output elements per thread access.
  a.vec_c = 1;
  if (a.M.n > 0 && a.M.s_out[0] == 1) {
    for (int v : {4, 2}) {
      bool ok = a.M.extent[0] % v == 0;
      for (int d = 1; d < a.M.n; ++d) ok = ok && a.M.s_out[d] % v == 0;
      for (int d = 0; d < a.N.n; ++d) ok = ok && a.N.s_out[d] % v == 0;
      if (ok && v * es >= 8) { a.vec_c = v; break; }
    }
  }
  a.alpha = e.op < 0 ? -1.0 : 1.0;
  a.beta = e.op == 0 ? 0 : 1;

  // CTA tile and kernel variant.  Rules distilled from tile sweeps on B200 over the
  // benchmark configurations (they replace the reference's transaction-count
  // cost model, cogent/src/algs/bases/cost_models.py:191-574):
  //   * fp64 tensor pipe: the persistent warp-specialised kernel (variant 2), N tile
  //     64 or 96, whichever wastes less of Nflat (128 x 64 or 64 x 96 per consumer group);
  //   * vector pipe: 128 x 128;
  //   * anything that would leave most SMs without a tile: 64 x 64, one CTA per tile.
  const int64_t sms = p->sm_count > 0 ? p->sm_count : TC_DEFAULT_SMS;
  int bm = 128, bn = 128, variant = 0, fill_bm = 0, fill_bn = 0;
  // fp32 on pairs of CTAs (tc_wd_kernel.cuh): both operands in tiled boxes that hold few k beyond the contraction, a
  // contraction long enough for the products to be what takes the time, and an output of which 32 columns from a multiple
  // of 32 on are neighbours.  Its time and that of the kernels it takes the place of, in us (measured on one B200, 720
  // x 2064 to 4096 x 4096, K = 400 to 3664): a round of tiles takes 1.4 us per 32 k on the pairs (for four times the
  // products) and 1.23 on 128 x 128 tiles; the mma.sync kernels, which take problems of fewer tiles, reach 25 to 33 TFLOP/s
  // of products on whole tiles.
  c.pair = false;
  bool unaligned = false;  // fp32 without any alignment on the one-tile tcgen05 kernel
  const bool boxes_pay = (uint64_t)kf * 5 >= (uint64_t)((kf + TC_BK - 1) / TC_BK * TC_BK) * 4;
  // (a caller that names a tile or a variant gets that kernel)
  const bool named = p->opt.tile_m > 0 || p->opt.tile_n > 0 || p->opt.variant > 0;
  const bool pair_shape = p->dtype == TC_F32 && !named && p->opt.tma != 1 && p->opt.tma != 3 && p->opt.c_path == 0 && boxes_pay && kf >= 16 * TC_BK &&
                          (c.tma_x || c.tma_xe) && (c.tma_y || c.tma_ye) && a.vec_c == 4 && (a.M.n == 1 || a.M.extent[0] % 32 == 0);
  auto rounds_of = [](int64_t tiles, int64_t at_once) { return (double)((tiles + at_once - 1) / at_once); };
  const int64_t pairs = std::max<int64_t>(1, sms / 2), pair_tiles = ((mf + 255) / 256) * ((nf + 255) / 256), pair_left = pair_tiles % pairs;
  const double pair_rounds = (double)(pair_tiles / pairs) + (pair_left == 0 ? 0.0 : 2 * pair_left <= pairs ? 0.7 : 1.0);
  const double pair_us = pair_rounds * (1.38 * (double)((kf + 31) / 32) + 4.0);
  const double single_us = rounds_of(((mf + 127) / 128) * ((nf + 127) / 128), sms) * (0.0385 * (double)kf + 2.0);
  const double sync_us = 2.0 * (double)((mf + 63) / 64 * 64) * (double)((nf + 63) / 64 * 64) * (double)kf / 32.0e6 + 5.0;
  bool slice_persistent = false;  // the persistent reduce-add kernel with K slices (few tiles, long contraction)
  if (p->box_order >= 0) {  // second pass: the tile is the first pass's
    bm = p->box_bm;
    bn = p->box_bn;
    variant = 3;
  } else if (p->opt.tile_m > 0 || p->opt.tile_n > 0) {
    bm = p->opt.tile_m;
    bn = p->opt.tile_n;
    variant = p->opt.variant > 0 ? p->opt.variant - 1 : 0;
  } else {
    if (c.math == TC_MATH_DMMA) {
      // fp64 on the tensor pipe: the persistent kernels, chosen by a small cost model (this takes the place of the
      // reference's ranking of mappings by estimated DRAM transactions, cogent/src/algs/bases/cost_models.py:191-574).
      // Per candidate (tile, kernel) the time of one SM is
      //   tiles per SM  x  max(products + idle, output bytes / rate, least):
      //   products   2 bm bn K / (DMMA rate of one SM x the share of it the kernel's main loop reaches), K rounded up to 4;
      //              the share depends on which operands are copied element by element (medians, K from 120 to 400);
      //   idle       cycles per tile during which the pipe waits (epilogue, hand-overs), measured per kernel;
      //   rate       what the kernel's way of reaching C sustains: reduce-adds of the copy engine 0.76 of the
      //              measured copy bandwidth, tiled loads + stores of a resident tile 0.92;
      //   least      cycles that a tile takes however little is in it: the chain of its copies and hand-overs (medians of
      //              tiles of 32 to 1024 elements with up to 16 products each; a resident tile of 120 elements takes as
      //              long as one of 1000, which made a 20 x 6 x 6 x 95 x 2 x 23 output 358 us instead of 60);
      //   tiles per SM is rounded up (wave quantisation), edge tiles count in full.
      // Constants come from the B200 measurements recorded beside the kernels; the device's SM count is the plan's.  On
      // 8 212 random one-index contractions the choice is 5 % slower than the best of the five, and 0.4 % of them run
      // 30 % slower than on the tiles of before cut tiles.  (One share per kernel, no `least` and 9000 cycles for any
      // element epilogue: 9 and 4 %.)
      struct Cand { int bm, bn, variant; double idle, rate, eff, least, share[4]; };  // share: neither, X, Y, both by element
      const Cand cands[] = {{128, 64, 2, 2100.0, 0.76, 0.90, 4000.0, {0.88, 0.65, 0.80, 0.65}},
                            {64, 96, 2, 800.0, 0.76, 0.86, 3500.0, {0.85, 0.78, 0.73, 0.72}},
                            {128, 32, 2, 1500.0, 0.76, 0.84, 3600.0, {0.78, 0.45, 0.60, 0.40}},
                            {128, 64, 3, 1450.0, 0.92, 0.92, 4400.0, {0.81, 0.67, 0.80, 0.66}},
                            {128, 32, 3, 1200.0, 0.92, 0.84, 3800.0, {0.60, 0.55, 0.61, 0.54}}};
      const bool boxes_in = p->opt.tma == 0 || p->opt.tma == 2 || p->opt.tma == 4;
      const int by_element = (c.vec_x || c.kvec_x || (boxes_in && c.tma_x) ? 0 : 1) + (c.vec_y || c.kvec_y || (boxes_in && c.tma_y) ? 0 : 2);
      const double clk = 1.9e9, flop_per_clk = 37.0e12 / 148.0 / clk, byte_per_clk = 6.5e12 / 148.0 / clk;
      const double kpad = (double)((k_true + 3) / 4 * 4);
      // Outputs whose rows are shorter than a consumer warp's leave the reduce-add kernels element by element (their
      // epilogue reads and writes C through registers, a round trip per batch): 1.25 cycles an element where C is read,
      // 0.55 where it is overwritten (full tiles, K up to 16: 13 800 against 8 300 cycles of the bulk epilogue on
      // 128 x 64, 9 700 against 6 100 on 64 x 96, 7 500 against 5 000 on 128 x 32; overwritten 7 300 / 5 700, 5 200 /
      // 4 500, 4 950 / 4 300).  The resident tile takes them as boxes.
      int64_t run_c = 0;
      if (a.M.n > 0 && a.M.s_out[0] == 1) {
        run_c = a.M.extent[0];
        for (int d = 1; d < a.M.n && a.M.s_out[d] == run_c; ++d) run_c *= a.M.extent[d];
      }
      p->why.clear();
      // The plain model (`eff` for the share, no `least`, no cut tiles) speaks first.  Its tile is final where the caller
      // names the variant: the full model's could be one that the variant is not compiled for.  And its tile says, below,
      // whether there are too few tiles to fill the GPU: which sums are sliced and need scratch does not move with the rest.
      struct Pick { int bm, bn, variant; double t; };
      auto choose = [&](bool plain) {
        Pick best = {bm, bn, variant, 0};
        const bool short_runs = !plain && (a.vec_c < 4 || run_c < 64);
        for (const Cand& k : cands) {
          if (!tc_kernel_exists(TC_F64, TC_MATH_DMMA, k.bm, k.bn, k.variant)) continue;
          double tiles_c = (double)((mf + k.bm - 1) / k.bm) * (double)((nf + k.bn - 1) / k.bn);
          if (plain && k.variant == 3 && k.bn == 32) continue;
          double out_elems = plain ? (double)k.bm * k.bn : (double)mf * (double)nf / tiles_c, idle = k.idle;
          int order = -1;  // M's dimension that comes second
          if (k.variant == 3) {  // needs tiles that are boxes of a rank-5 view of C, and nothing that pins the epilogue
            if (p->opt.tma == 1 || p->opt.tma == 2 || p->opt.c_path != 0) continue;
            // ... and pays only where the output traffic is the longer side: per output element the memory system moves
            // 16 bytes while the pipe does 2 K flops, equal near K = 46.  On long contractions its single consumer group
            // and two producer warps measured a third slower than the two-group kernel (21 against 31 TFLOP/s).
            const double limit = short_runs ? 3.0 : 1.0;
            if (limit * 2.0 * es / 6.5e12 < 0.85 * 2.0 * (double)k_true / 37.0e12) continue;
            if (plain) {
              TcOutMap view;
              bool per_warp = false, per_tile = false;
              out_box_view(a, es, k.bm, k.bn, &view, &per_warp, &per_tile);
              if (!per_tile) continue;
            } else {
              const BoxPlan bp = best_boxes(k.bm, k.bn, &order);
              if (!bp.ok) continue;
              tiles_c = bp.tiles;
              out_elems = (double)mf * (double)nf / bp.tiles;
            }
          } else if (short_runs) {
            idle += (e.op == 0 ? 0.55 : 1.25) * out_elems;
          }
          const double products = 2.0 * k.bm * k.bn * kpad / (flop_per_clk * (plain ? k.eff : k.share[by_element]));
          const double out_bytes = (e.op == 0 ? 1.0 : 2.0) * out_elems * es;
          const double per_tile = std::max(std::max(products + idle, out_bytes / (byte_per_clk * k.rate)), plain ? 0.0 : k.least);
          const double t = std::ceil(tiles_c / (double)sms) * per_tile / clk;
          // an earlier candidate stays unless a later one is estimated a twentieth faster (a tenth in the plain model): the
          // models know tiles, waste and waves, not how well each loader shape feeds each tile
          // (the output-resident kernel has its own gate above and the same tile: any estimated gain counts)
          if (best.t == 0 || t < best.t * (k.variant == 3 ? 0.98 : plain ? 0.90 : 0.95)) best = {k.bm, k.bn, k.variant, t};
        }
        return best;
      };
      const Pick first = choose(true), pick = p->opt.variant > 0 ? first : choose(false);
      bm = pick.bm;
      bn = pick.bn;
      variant = pick.variant;
      fill_bm = first.bm;
      fill_bn = first.bn;
      p->estimate_s = pick.t;
    }
    if (c.math != TC_MATH_DMMA && c.dtype == TC_F32) {
      // fp32: 96 rows instead of 128 when that makes the tile a whole number of the output's contiguous
      // runs (e.g. a fastest output index of extent 24), which the bulk epilogue wants.
      const int64_t e0 = (a.M.n > 0 && a.M.s_out[0] == 1) ? a.M.extent[0] : 0;
      if (e0 > 0 && e0 % 128 != 0 && 128 % e0 != 0 && (96 % e0 == 0 || e0 % 96 == 0)) bm = 96;
    }
    if (c.math == TC_MATH_TF32X3 && path == TC_PATH_AUTO && p->opt.split_k <= 1) {
      // The same three products as tcgen05.mma with the accumulators in tensor memory measured 10 % (K = 24)
      // to 80 % (K = 2048) faster than the mma.sync form on B200.  Its tiles are bm x 128; it is chosen when
      // they fill the GPU, almost all of them are whole (ragged tiles leave row by row through shared memory) and whole
      // tiles can leave through the staged bulk epilogue.
      auto mostly_whole = [](int64_t n, int64_t b) { return n % b == 0 || n >= 16 * b; };
      bool bulk_ok = false;
      if (a.M.n > 0 && a.M.s_out[0] == 1 && a.vec_c >= 4) {
        const int64_t e = a.M.extent[0];
        const int64_t e0 = e % bm == 0 ? bm : (bm % e == 0 ? e : std::gcd<int64_t>(bm, e));
        const bool n_adjacent = e0 == e && a.N.n > 0 && a.N.s_out[0] == e && (int64_t)a.N.extent[0] >= 128;
        bulk_ok = e0 % 4 == 0 && (n_adjacent || e0 * es >= 256);
      }
      const int64_t ctas_tc = ((mf + bm - 1) / bm) * ((nf + 127) / 128);
      if (bulk_ok && ctas_tc >= 2 * sms && mostly_whole(mf, bm) && mostly_whole(nf, 128) &&
          tc_kernel_exists(TC_F32, TC_MATH_TF32TC, bm, 128, 0)) {
        c.math = TC_MATH_TF32TC;
        bn = 128;
      }
    }
    // Nothing aligned: both operands element by element and an output of odd extents.  The one-tile tcgen05 kernel is 1.2 to
    // 2 times as fast as the mma.sync ones there (nineteen products of 39 to 180 565 rows, K = 10 to 3 795; one of K = 10
    // 2 % slower); with 16-byte loads or stores somewhere they win as often as they lose.
    if (c.math == TC_MATH_TF32X3 && path == TC_PATH_AUTO && p->opt.split_k == 0 && p->opt.c_path == 0 && a.vec_c == 1 && !c.vec_x && !c.kvec_x && !c.vec_y &&
        !c.kvec_y && ((mf + 127) / 128) * ((nf + 127) / 128) >= 96) {
      // (up to 64 columns, of which it would compute 128, the small mma.sync tile: four sums, 1.2 to 1.3 times the 128-wide
      // one, level with or up to 14 % ahead of tcgen05)
      // (up to 64 rows likewise, level with or up to 16 % ahead with 35 000 and 76 000 columns, five heights and three sums
      // each; with 309 000 5 % ahead to 6 % behind: 57 x 35 061 sum 63 20.5 -> 18.5 us, 45 x 75 999 sum 33 37.0 -> 32.9)
      const bool small = nf <= 64 || (mf <= 64 && nf <= 80000);
      if (!small) c.math = TC_MATH_TF32TC;
      bm = bn = small ? 64 : 128;
      unaligned = !small;
    }
    if (c.math != TC_MATH_SIMT && pair_shape && path == TC_PATH_AUTO && p->opt.split_k == 0 &&
        pair_us < 0.8 * (c.math == TC_MATH_TF32TC ? single_us : sync_us)) {
      c.math = TC_MATH_TF32TC;
      bm = bn = 128;
      c.pair = true;
    }
    if (c.math == TC_MATH_TF32TC && p->opt.split_k == 0 && p->opt.c_path != 2) {
      // ... as the persistent kernel (two accumulators in tensor memory, output tile staged in shared memory)
      // wherever its tile buffers can hold the output in runs that leave as bulk copies and both operands are
      // fetched 16 bytes at a time: its four loader warps issue element gathers slower than the 24 warps of three
      // resident one-tile CTAs do (measured on the fp32 items of the reference's benchmark list, one operand
      // gathered by element: 12.0-14.7 against 15.5-16.7 TFLOP/s; with vector loads on both sides it is 8-27 % ahead).
      const int tbm = (bm == 96 || bm == 128) ? bm : 128;
      const bool vector_loads = (c.vec_x || c.kvec_x) && (c.vec_y || c.kvec_y);
      if (vector_loads && wt_eligible(a, tbm, es) && tc_kernel_exists(TC_F32, TC_MATH_TF32TC, tbm, 128, 1)) { bm = tbm; bn = 128; variant = 1; }
    }
    if (fill_bm == 0) { fill_bm = bm; fill_bn = bn; }
    const int64_t ctas = ((mf + fill_bm - 1) / fill_bm) * ((nf + fill_bn - 1) / fill_bn);
    if (ctas < 2 * sms && !c.pair && !unaligned) {
      // Too few tiles to fill the GPU.  fp64 with a long contraction stays on the persistent 128 x 64 kernel and
      // slices K over its CTAs instead (16-byte loads along k, tiled TMA operands and two consumer groups are worth
      // more than small tiles: measured 3-4 x on few-tile, long-K items of the reference's list); everything else
      // runs one CTA per 64 x 64 tile, with K slices where K is long.
      const int64_t t128 = ((mf + 127) / 128) * ((nf + 63) / 64), t64 = ((mf + 63) / 64) * ((nf + 63) / 64);
      // ... unless its 128-row tiles pad the problem much more than 64-row ones would while the small kernel can
      // at least load one operand by vector (measured on 312 x 296 outputs: 20 % more padded work cost 20 %)
      const bool padding_ok = 2 * t128 * 100 <= t64 * 112 || (!c.vec_x && !c.vec_y);
      const int64_t steps = (k_true + TC_BK - 1) / TC_BK;
      if (c.math == TC_MATH_DMMA && p->opt.split_k == 0 && steps >= 64 && t128 * (steps / 16) >= 2 * sms && padding_ok && tc_kernel_exists(TC_F64, TC_MATH_DMMA, 128, 64, 2)) {
        bm = 128; bn = 64; variant = 2;
        slice_persistent = true;
      } else {
        bm = 64; bn = 64; variant = 0;
        // fp64 again, where K is not sliced (too short, or enough tiles): the one-tile kernel waits for memory once per K
        // step, 1.2 us a step where both operands load by vector and 2 to 5 where one is gathered, however little of the
        // GPU its tiles fill; the persistent 128 x 32 kernels run ahead (two tiles per SM at 1.15 us a step, 1.35 where
        // both have one and twice that where X is gathered across its sectors; the resident form, one per SM, 0.8).
        // From five steps and 32 tiles on and up to one round of them: 195 sums, 1.0 to 2.5 times as fast (1088 x 688 x 436
        // 62 -> 40 us; 19800 x 19 x 120, gathered, 42 -> 19); below that within 15 % either way, beyond 8 % slower (374).
        // Up to a hundred tiles of five to seven steps the one-tile kernel has as little to wait for where both operands and C
        // are read by 16 bytes (6400 x 22 x 68 8.0 against 10.2 us) or where an odd X is read along its fastest index and C only
        // written (1121 x 219 x 68 12.7 against 16.4).
        const int64_t t32 = ((mf + 127) / 128) * ((nf + 31) / 32);
        const bool short_waits = t32 * 3 < 2 * sms && ((steps < 7 && c.vec_x && c.vec_y && a.vec_c == 4) ||
                                                       (steps < 8 && e.op == 0 && a.lanes_k_x == 1 && !c.vec_x && a.M.s_in[0] == 1));
        if (c.math == TC_MATH_DMMA && p->opt.split_k == 0 && p->opt.variant == 0 && p->opt.c_path == 0 && p->opt.tma == 0 && steps >= 5 && t32 >= 32 && t32 <= 2 * sms &&
            !short_waits && !(t64 * 2 <= sms && steps >= 16)) {
          // (lanes on M's first index read neighbours where that is X's fastest too, only an odd one: 979 x 1032 x 263
          // 47 -> 40 us, 617 x 1840 x 281 49 -> 42)
          const bool across = a.lanes_k_x == 1 && !c.vec_x && a.M.s_in[0] != 1;
          const double ws_us = (rounds_of(t32, 2 * sms) * (double)steps * (t32 > sms ? 1.35 : 1.15) + 6.0) * (across ? 2.0 : 1.0);
          int order = -1;
          const BoxPlan bp = best_boxes(128, 32, &order);
          if (bp.ok && rounds_of((int64_t)bp.tiles, sms) * (double)steps * 0.8 + 5.0 < ws_us) { bm = 128; bn = 32; variant = 3; }
          else if (!across || nf <= 32) { bm = 128; bn = 32; variant = 2; }  // (more than once across its sectors: 61 -> 71 us)
        }
        if (c.math == TC_MATH_TF32TC) c.math = TC_MATH_TF32X3;  // no 64-wide tcgen05 tile: same arithmetic on mma.sync
      }
    }
    if (p->opt.variant > 0) variant = p->opt.variant - 1;
  }
  // (tma 1 and 2 keep the copy engine away from C: such a plan runs on the stand-in and keeps its plain tiles)
  int box_order = -1;
  const bool boxes_allowed = p->opt.tma != 1 && p->opt.tma != 2;
  if (variant == 3 && c.math == TC_MATH_DMMA && boxes_allowed && p->box_order < 0 && best_boxes((uint32_t)bm, (uint32_t)bn, &box_order).ok) {
    p->box_order = box_order;  // plan again with M's dimensions whole and in that order
    p->box_bm = bm;
    p->box_bn = bn;
    const int st = tc_plan_build(p, why);
    p->box_order = -1;
    return st;
  }
  c.bm = bm;
  c.bn = bn;
  c.variant = variant;
  if (tc_kernel_is_tmem_persistent(c) && pair_shape && bm == 128 && p->opt.split_k == 0) c.pair = pair_us < single_us;
  if (tc_kernel_is_tmem_persistent(c) && !wt_eligible(a, bm, es)) {
    *why = "the persistent tcgen05 kernel needs an output whose tile rows are 16-byte aligned contiguous runs";
    return TC_ERR_UNSUPPORTED;
  }
  if (!tc_kernel_exists(c.dtype, c.math, bm, bn, c.variant)) { *why = "requested CTA tile / variant is not compiled in"; return TC_ERR_UNSUPPORTED; }
  a.bm = bm;
  a.bn = bn;
  a.tiles_m = (uint32_t)((mf + bm - 1) / bm);
  a.tiles_n = (uint32_t)((nf + bn - 1) / bn);
  a.mcut = {(uint32_t)bm, 1, (uint32_t)mf, 1, a.tiles_m, 1};
  a.ncut = {(uint32_t)bn, 1, (uint32_t)nf, 1, a.tiles_n, 1};
  a.rows_across_x = a.rows_across_y = 0;
  c.box_c = false;
  a.panel = 0;
  bool plain_m = true, plain_n = true;  // tiles are plain ranges of the flattened index
  a.standin_vec_c = a.vec_c;
  if (tc_kernel_is_c_resident(c) && boxes_allowed) {
    const BoxPlan bp = plan_boxes(dm, dn, (uint32_t)bm, (uint32_t)bn);
    if (bp.ok) {
      c.box_c = true;
      a.mcut = bp.m;
      a.ncut = bp.n;
      a.cbox = bp.map;
      // The stand-in's epilogue takes four consecutive rows as four neighbours in C: true inside a cut tile only where
      // its runs are whole fours.  Else it goes element by element.
      if (bp.m.b0 % 4 != 0) a.standin_vec_c = std::min(a.vec_c, 2);
      a.rows_across_x = bp.across_x;
      a.rows_across_y = bp.across_y;
      const int64_t tm = mf / ((int64_t)bp.m.e0 * bp.m.e1) * bp.m.t0 * bp.m.t1, tn = nf / ((int64_t)bp.n.e0 * bp.n.e1) * bp.n.t0 * bp.n.t1;
      auto plain = [](const TcCut& k, int64_t flat, int b) { return k.b0 == (uint32_t)b && k.b1 == 1 && (k.e0 == flat || k.e0 % b == 0); };
      plain_m = plain(bp.m, mf, bm);
      plain_n = plain(bp.n, nf, bn);
      a.tiles_m = (uint32_t)tm;
      a.tiles_n = (uint32_t)tn;
      // Panels (tc_wp_kernel.cuh): X's tile is kept for a whole row of tiles, and a CTA has to have enough tiles to hide its
      // first one (three tiles 14.4 -> 17.2 us, six 26.6 either way).  They save fetching X again and again and give up the
      // ring kernel's order of tiles -- neighbours in M at the same time -- in which short runs of C share sectors and rows
      // of memory.  Times as fast as the ring kernel, on 570 shapes of three to six indices, K = 8 to 48:
      //   * tiles that cut M's first digit into short runs 0.50 to 1.3, 0.87 in the mean (22 x 16 x 19 x 16 x 24 x 16, K = 38,
      //     199 -> 387 us);
      //   * X gathered across its sectors, from K = 17 on 0.97 to 1.7, mean 1.24 (24 x 16 x 16 x 24 x 16 x 16, K = 24, 156 ->
      //     129 us) but for the shortest runs (80 bytes 0.92 to 1.1); where C is only written 0.97 to 1.7 with any K; below
      //     K = 16 C's traffic is the longer side, 0.80 to 1.08 where Y loads by vector (K = 12 54 -> 64 us), 0.99 to 1.2 else;
      //   * else, three K steps: 0.91 to 0.99 where X comes in tiled boxes, which it is cheap to fetch again; 0.96 to 1.4, mean
      //     1.12, otherwise, but for runs that are not whole sectors (0.77 to 1.25);
      //   * runs of 64 and more, three K steps: 0.98 to 1.29 with a panel for every CTA (40^6 slab, K = 40, 1 736 -> 1 633 us),
      //     where C's slower indices belong to M too, or X is gathered; else 0.81 to 1.02.
      // A caller that names tile and variant gets panels wherever X takes three K steps or is gathered.
      const bool across = a.lanes_k_x == 1 && !c.vec_x && a.M.s_in[0] != 1, whole = bp.m.b0 == bp.m.e0, sectors = bp.m.b0 % 4 == 0;
      const bool three = kf > 2 * TC_BK;
      bool pays = false;
      if (p->opt.variant > 0 && p->opt.tile_m > 0) pays = three || across;
      else if (bp.m.b0 >= 64 && (!whole || bp.m.b0 == (uint32_t)bm)) pays = three && tn >= 8 && (tm >= sms || (int64_t)bp.m.e0 < mf || !c.tma_x);
      else if (whole && !across) pays = three && sectors && !c.tma_x;
      else if (whole && (e.op == 0 || three)) pays = true;
      else if (whole) pays = kf >= TC_BK ? bp.m.b0 >= 14 || (sectors && kf > TC_BK) : sectors && !c.vec_y && !c.kvec_y;
      a.panel = bm == 128 && bn == 64 && kf <= 3 * TC_BK && pays && tn >= 2 && tm * tn >= 8 * sms;
      // a tiled TMA box of an operand takes consecutive values of the flattened index
      if (bp.m.b1 > 1 && bp.m.b0 != bp.m.e0) c.tma_x = false;
      if (bp.n.b1 > 1 && bp.n.b0 != bp.n.e0) c.tma_y = false;
    }
  }
  const int64_t tiles = (int64_t)a.tiles_m * a.tiles_n;
  const int bk = TC_BK;
  // Persistent kernels: walk the tiles in column blocks of 32 M tiles when one sweep over all of M would drag more
  // than a few MB of X through L2 per row of tiles (see tile_coords in tc_kernels.cuh).
  a.mblock_w = 0;
  if (tc_kernel_is_persistent(c) && a.tiles_m > 64 && a.tiles_n > 1 && (double)mf * (double)kf * es > 4.0e6) a.mblock_w = 32;

  // K split: only when the tile count cannot fill the GPU and K is long.
  int64_t ksplit = 1, seg_steps = int64_t(1) << 27;  // seg_steps: the longest chain of additions inside a slice
  const int64_t ksteps = (k_true + bk - 1) / bk;
  const bool persistent = tc_kernel_is_persistent(c);
  // Persistent kernels do not split K, except the fp64 reduce-add kernel: on request (forced tile and split_k), or
  // where the planner kept it for a problem of few tiles.
  const bool ws_kernel = c.math == TC_MATH_DMMA && c.variant == 2;
  if (kcut_x > 0 && !(c.math == TC_MATH_DMMA && persistent)) {  // kernels that know no holes in the contraction
    p->block_k = false;
    const int st = tc_plan_build(p, why);
    p->block_k = true;
    return st;
  }
  if (persistent && ws_kernel && p->opt.split_k > 1) ksplit = std::min<int64_t>(p->opt.split_k, ksteps);
  else if (persistent && ws_kernel && slice_persistent) {
    // Work items (slice, tile) are dealt to two groups per SM: as many slices (of at least 16 steps) as fill whole rounds
    // of the groups.  One item more than a round costs a round (312 x 296 outputs summed over 312 x 312, 15 tiles: 40
    // slices are 600 items on 296 groups, three rounds for 2.03 rounds of work, 975 us; 39 are two, 789 us; 19 are one,
    // 806 us).  The first number of rounds that leaves under 5 % of the groups idle, else the best of four.
    const int64_t slots = 2 * sms;
    double best_fill = 0;
    for (int64_t rounds = 1; rounds <= 4 && best_fill < 0.95; ++rounds) {
      const int64_t ks = std::min<int64_t>(rounds * slots / tiles, ksteps / 16);
      if (ks < 2) continue;  // (one slice goes into C by itself and has no partial tile to be added up in)
      const int64_t items = ks * tiles, used = (items + slots - 1) / slots;
      const double fill = (double)items / (double)(used * slots);
      if (fill > best_fill) { best_fill = fill; ksplit = ks; }
    }
    // ... each added up in segments no longer than four items per SM (of at least 16 steps) would make slices, so that
    // few slices do not lengthen the chains of additions: in one chain, 19 slices of that sum are 2.5e-15 from a sum by
    // pairs, 40 slices 1.8e-15.
    const int64_t most = std::max<int64_t>(1, std::min<int64_t>((4 * sms + tiles - 1) / tiles, ksteps / 16));
    seg_steps = (ksteps + most - 1) / most;
  }
  else if (persistent) ksplit = 1;
  else if (p->opt.split_k > 1) ksplit = std::min<int64_t>(p->opt.split_k, ksteps);
  else if (c.pair) ksplit = 1;  // (the pairs cut their chains themselves, what stands in for them runs in passes: no scratch)
  else if (p->opt.split_k == 0 && tiles * 2 <= sms && ksteps >= 16)
  {
    ksplit = std::max<int64_t>(1, std::min<int64_t>((2 * sms) / tiles, ksteps / 8));
    // fp64, 64 x 64: four CTAs fit an SM, and two of them leave its pipe half fed; slices of at least 16 steps fill all
    // four (312 x 296 summed over 312 x 312, an operand loaded by vector: 25 tiles in 11 slices 1080 us, in 23 858 us).
    // Plans whose scratch fits the allocation-free entry's array keep doing so.
    if (c.math == TC_MATH_DMMA && bm == 64 && bn == 64) {
      int64_t wide = std::min<int64_t>((4 * sms) / tiles, ksteps / 16);
      const int64_t fits = (int64_t)TC_NOALLOC_MAX_WORKSPACE_BYTES / (tiles * bm * bn * es);
      if (ksplit <= fits) wide = std::min(wide, fits);
      ksplit = std::max(ksplit, wide);
    }
  }
  // The tensor cores accumulate fp32 with truncation: measured against exact sums on B200 the relative error of
  // one accumulation chain grows linearly with its length (2e-6 at K = 256, 7e-6 at 1024, 3e-5 at 4096), for
  // mma.sync and tcgen05 alike, while FFMA stays at 1e-6.  No tensor-core plan therefore runs a chain longer
  // than TC_TF32_CHAIN products (tc_options.split_k >= 1 overrides this, as does TC_PATH_FFMA):
  //   * where the slices' partial tiles fit 1 GiB of plan-owned scratch, the contraction is K-sliced and the
  //     combine kernel adds the slices in round-to-nearest fp32;
  //   * larger outputs run the contraction as sequential PASSES over consecutive ranges of at most that many
  //     products, every pass accumulating into the output itself (the first with the expression's operator,
  //     the others with `+=`; the additions into C are round-to-nearest).  A pass re-reads and re-writes C,
  //     which at 512 products per element is noise beside the arithmetic.
  p->passes = 1;
  // (the persistent tcgen05 kernel cuts its chains itself: segments of at most 32 K steps that alternate between
  // two accumulators and are added into the output tile in shared memory)
  if ((c.math == TC_MATH_TF32X3 || c.math == TC_MATH_TF32TC) && p->opt.split_k == 0 && !persistent) {
    const int64_t per_slice = tiles * bm * bn * (int64_t)es;
    const int64_t want = std::min<int64_t>((kf + TC_TF32_CHAIN - 1) / TC_TF32_CHAIN, ksteps);
    // What runs in the pairs' place where a tensor is not aligned, without scratch: a plan that reports none may run on several
    // streams at once.  Against the K slices of before, all three tensors shifted: 900 x 900 sum 512 82 -> 49 us, 2048 x 2048 sum
    // 1024 359 -> 205, but few tiles with several chains 900 x 900 sum 2000 174 -> 280, 720 x 2064 sum 3664 450 -> 520.
    if (c.pair) p->passes = (int)want;
    else if (want > 1 && want * per_slice > (int64_t(1) << 30) && ksplit == 1) p->passes = (int)std::min<int64_t>(want, 1 << 20);
    else ksplit = std::max<int64_t>(ksplit, want);
  }
  if (p->passes > 1) {
    const int64_t steps_per_pass = (ksteps + p->passes - 1) / p->passes;
    p->passes = (int)((ksteps + steps_per_pass - 1) / steps_per_pass);
    a.k_chunk = (uint32_t)(steps_per_pass * bk);
    a.ksplit = 1;
  }
  if (p->passes == 1) {
    const int64_t steps = (kf + bk - 1) / bk;  // positions, rounded-up ones among them
    int64_t chunk_steps = (steps + ksplit - 1) / ksplit;
    ksplit = (steps + chunk_steps - 1) / chunk_steps;
    a.ksplit = (uint32_t)ksplit;
    a.k_chunk = (uint32_t)(chunk_steps * bk);
    const int64_t segs = ksplit > 1 ? (chunk_steps + seg_steps - 1) / seg_steps : 1;
    a.k_seg = (uint32_t)((chunk_steps + segs - 1) / segs);
    a.k_segs = (uint32_t)((chunk_steps + a.k_seg - 1) / a.k_seg);
  }
  if (tiles * ksplit >= (int64_t(1) << 31)) { *why = "too many tiles"; return TC_ERR_UNSUPPORTED; }
  p->ws_bytes = ksplit > 1 ? (size_t)(ksplit * tiles * bm * bn) * es : 0;
  p->launches = ksplit > 1 ? 2 : c.pair ? 1 : p->passes;

  // Staged bulk epilogue of the vector-pipe kernels: the tile's rows split into runs of E0 elements
  // contiguous in the output; if the output's next index belongs to the other operand (its stride equals
  // the extent of the fastest one), consecutive n are adjacent too within blocks of that index's extent.
  a.epi_run = 0;
  a.epi_n_span = 0;
  if (c.math != TC_MATH_DMMA && ksplit == 1) {
    // bulk copies pay off from a few hundred bytes per chunk; shorter runs keep the read-modify-write
    bool n_adjacent = false;
    const int64_t e0 = staged_run(a, bm, bn, es, &n_adjacent);
    if (e0 > 0) {
      a.epi_run = (int32_t)e0;
      if (n_adjacent) a.epi_n_span = (int32_t)a.N.extent[0];
    }
  }

  // Persistent fp64 kernels: which output batches / tiles are boxes of a rank-5 view of C (see out_box_view).
  c.tma_c = false;
  c.tma_ct = false;
  a.cmap = TcOutMap{};
  if (persistent && plain_m && plain_n) out_box_view(a, es, bm, bn, &a.cmap, &c.tma_c, &c.tma_ct);

  double prod = 1.0;
  for (int64_t x : p->idx_extent) prod *= (double)x;
  p->flops = 2.0 * prod;
  p->bytes = (double)es * ((e.op == 0 ? 1.0 : 2.0) * p->count_c + p->count_a + p->count_b);
  return TC_OK;
}

// "kernel" in the plan record is the kernel that the plan was made for; this is the one that a route takes.
static std::string route_name(const tc_plan& p, int route) {
  TcKernelChoice c = p.choice;
  if (route == TC_ROUTE_PAIRS) return "tf32wd_256x256";
  if (route == TC_ROUTE_PANELS) return "dmma_wp_128x64";
  if (route == TC_ROUTE_STANDIN) c.variant = tc_kernel_is_c_resident(c) ? 2 : 0;
  return tc_kernel_name(c);
}

std::string tc_plan_to_json(const tc_plan& p) {
  std::ostringstream o;
  o.precision(17);
  const TcKernelArgs& a = p.args;
  auto dims = [&](const TcDims& d) {
    o << "[";
    for (int i = 0; i < d.n; ++i)
      o << (i ? "," : "") << "{\"extent\":" << d.extent[i] << ",\"s_in\":" << d.s_in[i] << ",\"s_out\":" << d.s_out[i] << "}";
    o << "]";
  };
  o << "{\"expr\":" << tc_expr_to_json(p.expr) << ",\"dtype\":\"" << (p.dtype == TC_F64 ? "f64" : "f32")
    << "\",\"committed\":" << (p.committed ? "true" : "false");
  // longest tensor-core accumulation chain of the plan
  uint32_t chain = std::min<uint32_t>(a.k_chunk, a.Kflat);
  if (tc_kernel_is_tmem_persistent(p.choice) || p.choice.pair) {
    const uint32_t steps = (a.Kflat + TC_BK - 1) / TC_BK, segs = (steps + 31) / 32;
    chain = std::min<uint32_t>(a.Kflat, ((steps + segs - 1) / segs) * TC_BK);
  }
  if (p.committed) {
    const int ran = __atomic_load_n(&p.ran, __ATOMIC_RELAXED);
    o << ",\"swapped\":" << (p.swapped ? "true" : "false") << ",\"M\":";
    dims(a.M);
    o << ",\"N\":";
    dims(a.N);
    o << ",\"K\":";
    dims(p.kdims);
    o << ",\"Mflat\":" << a.Mflat << ",\"Nflat\":" << a.Nflat << ",\"Kflat\":" << a.Kflat
      << ",\"math\":\"" << (p.choice.math == TC_MATH_DMMA ? "dmma" : p.choice.math == TC_MATH_TF32X3 ? "tf32x3" : p.choice.math == TC_MATH_TF32TC ? "tf32x3_tcgen05" : (p.dtype == TC_F64 ? "dfma" : "ffma"))
      << "\",\"kernel\":\"" << tc_kernel_name(p.choice) << "\",\"tile\":[" << p.choice.bm << "," << p.choice.bn << "," << TC_BK
      << "],\"runs\":\"" << route_name(p, tc_plan_route(p)) << "\",\"runs_tile\":[" << (p.choice.pair ? 256 : p.choice.bm) << "," << (p.choice.pair ? 256 : p.choice.bn)
      << "],\"ran\":" << (ran < 0 ? "null" : "\"" + route_name(p, ran) + "\"") << ",\"variant\":" << p.choice.variant << ",\"tiles\":[" << a.tiles_m << "," << a.tiles_n << "],\"estimate_us\":" << p.estimate_s * 1e6 << ",\"mblock_w\":" << a.mblock_w << ",\"ksplit\":" << a.ksplit
      << ",\"k_chunk\":" << a.k_chunk << ",\"k_seg\":" << a.k_seg << ",\"passes\":" << p.passes << ",\"chain\":" << chain << ",\"vec_x\":" << (p.choice.vec_x ? "true" : "false")
      << ",\"vec_y\":" << (p.choice.vec_y ? "true" : "false") << ",\"kvec_x\":" << (p.choice.kvec_x ? "true" : "false")
      << ",\"kvec_y\":" << (p.choice.kvec_y ? "true" : "false") << ",\"tma_x\":" << (p.choice.tma_x ? "true" : "false")
      << ",\"tma_y\":" << (p.choice.tma_y ? "true" : "false") << ",\"tma_xe\":" << (p.choice.tma_xe ? "true" : "false")
      << ",\"tma_ye\":" << (p.choice.tma_ye ? "true" : "false") << ",\"tma_c\":" << (p.choice.tma_c ? "true" : "false") << ",\"tma_ct\":" << (p.choice.tma_ct ? "true" : "false")
      << ",\"pair\":" << (p.choice.pair ? "true" : "false") << ",\"lanes_k_x\":" << a.lanes_k_x
      << ",\"lanes_k_y\":" << a.lanes_k_y << ",\"vec_c\":" << a.vec_c << ",\"standin_vec_c\":" << a.standin_vec_c << ",\"epi_run\":" << a.epi_run << ",\"epi_n_span\":" << a.epi_n_span << ",\"beta\":" << a.beta
      << ",\"alpha\":" << a.alpha << ",\"workspace_bytes\":" << p.ws_bytes << ",\"launches\":" << p.launches
      << ",\"flops\":" << p.flops << ",\"bytes\":" << p.bytes;
    if (p.choice.box_c) {
      const TcBoxMap& b = a.cbox;
      auto cut = [&](const TcCut& c) { o << "[" << c.b0 << "," << c.b1 << "," << c.e0 << "," << c.e1 << "," << c.t0 << "," << c.t1 << "]"; };
      o << ",\"panel\":" << (a.panel ? "true" : "false") << ",\"cbox\":{\"m\":";
      cut(a.mcut);
      o << ",\"n\":";
      cut(a.ncut);
      o << ",\"dims\":[";
      for (int d = 0; d < b.rank; ++d) o << (d ? "," : "") << "[" << b.ext[d] << "," << b.box[d] << "," << b.stride[d] << "]";
      o << "],\"slots\":[" << (int)b.n0 << "," << (int)b.n1 << "," << (int)b.m1 << "," << (int)b.mr0 << "," << (int)b.mr1 << "," << (int)b.nr0 << "," << (int)b.nr1
        << "],\"steps\":[" << b.m_step << "," << b.n_step << "],\"rest\":[" << b.mr << "," << b.nr << "],\"across\":[" << a.rows_across_x << "," << a.rows_across_y << "]}";
    }
  }
  o << "}";
  return o.str();
}
