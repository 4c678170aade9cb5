#include "wplan.h"

#include <algorithm>
#include <cmath>
#include <numeric>
#include <stdexcept>
#include <string>

#include "gridding_kernels.h"

namespace pg {
namespace {
constexpr double kPi = 3.14159265358979323846;

double wrap(double x, double y) {
  double r = std::fmod(x, y);
  if (r < 0) r += y;
  return r;
}

// projection_kernels::pixel_to_lambda (projection_kernels.cc:28-30)
double pixel_to_lambda(double cell, int imsize, double os) {
  return 60. * 60. * 180. / cell / std::floor(os * imsize) / kPi;
}

// The zero-padded linear convolution of convolution.h:42-52,
// out(j) = sum_k f(k) g_pad(n_out - 1 - j + k), n_out = Jg + Jf - 1.
void conv1d(const double *f, int Jf, const std::complex<double> *g, int Jg,
            std::complex<double> *out) {
  const int n_out = Jg + Jf - 1;
  for (int j = 0; j < n_out; ++j) {
    std::complex<double> acc = 0;
    for (int k = 0; k < Jf; ++k) {
      const int idx = n_out - 1 - j + k - (Jf - 1);  // index into the unpadded g
      if (idx >= 0 && idx < Jg) acc += f[k] * g[idx];
    }
    out[j] = acc;
  }
}

// Which of the three terms of a row's sample matrix
//   g = (a~ / (w i)) b~^T + (1 - chi_v) 1^T + chi_v (1 - chi_u)^T
// are nonzero (bit r for term r), from the validity masks chi of
// projection_kernels.cc:38-45 at the row's Jw sample offsets.  A term that is
// zero here is exactly zero, so leaving it out changes no tap.
int row_terms(double u, double v, double w, int Jw, double dul, double dvl) {
  const double dwu = u - std::floor(u - Jw * 0.5), dwv = v - std::floor(v - Jw * 0.5);
  bool any_u = false, all_u = true, any_v = false, all_v = true;
  for (int k = 0; k < Jw; ++k) {
    const double U = dwu - k - 1, V = dwv - k - 1;
    const bool ok_u = std::abs(U * dul / w) < 1, ok_v = std::abs(V * dvl / w) < 1;
    any_u |= ok_u;
    all_u &= ok_u;
    any_v |= ok_v;
    all_v &= ok_v;
  }
  return int(any_v && any_u) | int(!all_v) << 1 | int(any_v && !all_u) << 2;
}
}  // namespace

WPlan build_wplan(const WPlanRequest &rq) {
  if (rq.M < 0) throw std::invalid_argument("negative number of visibilities");
  if (rq.M > 0 && (!rq.u || !rq.v || (!rq.w && !rq.plain)))
    throw std::invalid_argument("u, v and w must be given");
  if (rq.J < 1 || rq.Jw < 1) throw std::invalid_argument("kernel supports must be >= 1");
  if (rq.plain && (rq.Ju < 1 || rq.Jv < 1)) throw std::invalid_argument("kernel supports must be >= 1");
  if (rq.M > int64_t(INT32_MAX) - 1) throw std::invalid_argument("too many visibilities");
  for (int64_t m = 0; m < rq.M; ++m)
    if (!std::isfinite(rq.u[m]) || !std::isfinite(rq.v[m]) || (!rq.plain && !std::isfinite(rq.w[m])))
      throw std::invalid_argument("visibility " + std::to_string(m) +
                                  " has a non-finite u, v or w coordinate");
  WPlan P;
  P.M = rq.M;
  P.Nu = rq.Nu;
  P.Nv = rq.Nv;
  P.plain = rq.plain;
  P.Ju = rq.Ju;
  P.Jv = rq.Jv;
  // plain rows: S = max(Ju, Jv) for every row (a w-support of 1 on a support
  // of S cells)
  const int Jrow = rq.plain ? std::max(rq.Ju, rq.Jv) : rq.J;
  P.J = Jrow;
  const int64_t M = rq.M;
  std::vector<int32_t> jw(M);
  int Smax = 1;
  for (int64_t m = 0; m < M; ++m) {
    jw[m] = rq.plain ? 1 : (rq.jw_rows ? rq.jw_rows[m] : rq.Jw);
    if (jw[m] < 1 || jw[m] + Jrow - 1 > 255) throw std::invalid_argument("w-support out of range");
    Smax = std::max(Smax, int(jw[m] + Jrow - 1));
  }
  P.Smax = Smax;
  P.tu = make_tiling(rq.Nu, rq.tile);
  P.tv = make_tiling(rq.Nv, rq.tile);
  if (rq.Nu < Smax || rq.Nv < Smax)
    throw std::invalid_argument("grid is smaller than the largest w-projection support");
  for (int b = 0; b < P.tu.n; ++b)
    if (P.tu.start[b + 1] - P.tu.start[b] < Smax - 1)
      throw std::invalid_argument("grid width is too small for the w-projection support");
  for (int b = 0; b < P.tv.n; ++b)
    if (P.tv.start[b + 1] - P.tv.start[b] < Smax - 1)
      throw std::invalid_argument("grid height is too small for the w-projection support");
  const int ntu = P.tu.n, ntv = P.tv.n, ntiles = ntu * ntv;

  // The kernel sees w - mean(w) (operators.h:323).
  double wmean = 0;
  if (!rq.plain) {
    for (int64_t m = 0; m < M; ++m) wmean += rq.w[m];
    if (M > 0) wmean /= double(M);
  }
  auto w_of = [&](int64_t m) { return rq.plain ? 0.0 : rq.w[m] - wmean; };

  // Placement per row (operators.cc:85-96): kw = floor(u - S/2), taps at
  // kw + 1 .. kw + S (mod N); the phase (-1)^(kw_u + kw_v) goes with the weight.
  std::vector<int32_t> tile(M), local(M);
  std::vector<uint8_t> flip(M);
  for (int64_t m = 0; m < M; ++m) {
    const int S = jw[m] + Jrow - 1;
    const double kwu = std::floor(rq.u[m] - S * 0.5), kwv = std::floor(rq.v[m] - S * 0.5);
    const int q0 = int(wrap(kwu + 1, rq.Nu)), p0 = int(wrap(kwv + 1, rq.Nv));
    const int a = P.tv.of[p0], b = P.tu.of[q0];
    tile[m] = a * ntu + b;
    local[m] = ((p0 - P.tv.start[a]) << 8) | (q0 - P.tu.start[b]);
    flip[m] = uint8_t((int64_t(kwu) + int64_t(kwv)) & 1);
  }
  // Plan order: tile, then support descending (warps take visibilities in
  // turn, so neighbours in this order cost about the same), then caller order.
  std::vector<int32_t> order(M);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int32_t x, int32_t y) {
    if (tile[x] != tile[y]) return tile[x] < tile[y];
    return jw[x] > jw[y];
  });
  P.du_lambda = pixel_to_lambda(rq.cellx, rq.imsizex, rq.oversample_ratio);
  P.dv_lambda = pixel_to_lambda(rq.celly, rq.imsizey, rq.oversample_ratio);
  P.code.resize(M);
  P.factor.resize(M);
  P.weight.resize(M);
  P.slot_user.resize(M);
  P.user_slot.resize(M);
  int64_t off = 0;
  for (int64_t i = 0; i < M; ++i) {
    const int32_t m = order[i];
    const int S = jw[m] + Jrow - 1;
    const int lp = local[m] >> 8, lq = local[m] & 0xff;  // item_pack layout below
    // plain rows: one term (the separable taps)
    const int terms =
        rq.plain ? 1 : row_terms(rq.u[m], rq.v[m], w_of(m), jw[m], P.du_lambda, P.dv_lambda);
    P.code[i] = lp | (lq << 8) | (S << 16) | (terms << 24);
    P.factor[i] = off;
    off += int64_t(2) * wrow_rank(P.code[i]) * S;
    const std::complex<double> wgt = rq.weights ? rq.weights[m] : std::complex<double>(1.0, 0.0);
    P.weight[i] = flip[m] ? -wgt : wgt;
    P.slot_user[i] = m;
    P.user_slot[m] = int32_t(i);
    P.taps += int64_t(S) * S;
  }
  P.factor_count = off;
  P.kernel = rq.kernel;
  P.oversample_ratio = rq.oversample_ratio;
  P.gen_u.resize(M);
  P.gen_v.resize(M);
  P.gen_w.resize(M);
  P.gen_jw.resize(M);
  for (int64_t i = 0; i < M; ++i) {
    const int32_t m = order[i];
    P.gen_u[i] = rq.u[m];
    P.gen_v[i] = rq.v[m];
    P.gen_w[i] = w_of(m);
    P.gen_jw[i] = jw[m];
  }

  // Tasks: consecutive visibilities of one tile, bounded in taps.
  P.tile_tasks.assign(ntiles + 1, 0);
  int64_t i = 0;
  for (int t = 0; t < ntiles; ++t) {
    const int a = t / ntu, b = t % ntu;
    int64_t e = i;
    while (e < M && tile[order[e]] == t) ++e;
    int64_t s = i;
    while (s < e) {
      int64_t k = s, taps = 0;
      while (k < e && (k == s || taps + wrow_taps(P.code[k]) <= rq.max_taps_per_task)) {
        taps += wrow_taps(P.code[k]);
        ++k;
      }
      Task tk{};
      tk.P = P.tv.start[a];
      tk.Q = P.tu.start[b];
      tk.H = P.tv.start[a + 1] - P.tv.start[a];
      tk.W = P.tu.start[b + 1] - P.tu.start[b];
      tk.batch_begin = int32_t(s);
      tk.batch_end = int32_t(k);
      tk.tile = t;
      P.tasks.push_back(tk);
      s = k;
    }
    P.tile_tasks[t + 1] = int32_t(P.tasks.size());
    P.win_rows = std::max(P.win_rows, P.tv.start[a + 1] - P.tv.start[a] + Smax - 1);
    P.win_cols = std::max(P.win_cols, P.tu.start[b + 1] - P.tu.start[b] + Smax - 1);
    i = e;
  }
  // Staging chunks (the factor ranges of consecutive rows are contiguous).
  P.chunk_values = std::max(kWChunkValues, 6 * Smax);
  P.task_chunk.assign(P.tasks.size() + 1, 0);
  for (size_t k = 0; k < P.tasks.size(); ++k) {
    const int32_t b = P.tasks[k].batch_begin, e = P.tasks[k].batch_end;
    auto fend = [&](int32_t r) { return r + 1 < M ? P.factor[r + 1] : P.factor_count; };
    for (int32_t r = b; r < e;) {
      WChunk c{P.factor[r], fend(r), r, r + 1};
      while (c.vis_end < e && c.vis_end - c.vis_begin < kWChunkVis &&
             fend(c.vis_end) - c.fbegin <= P.chunk_values) {
        c.fend = fend(c.vis_end);
        ++c.vis_end;
      }
      P.chunks.push_back(c);
      r = c.vis_end;
    }
    P.task_chunk[k + 1] = int32_t(P.chunks.size());
  }
  // Launch order: longest tasks (in taps) first while the grid stays in L2,
  // else the spatial order (see build_plan).
  P.task_order.resize(P.tasks.size());
  std::iota(P.task_order.begin(), P.task_order.end(), 0);
  if (int64_t(rq.Nu) * rq.Nv * 8 <= kLptGridBytes) {
    std::vector<int64_t> cost(P.tasks.size(), 0);
    for (size_t k = 0; k < P.tasks.size(); ++k)
      for (int i = P.tasks[k].batch_begin; i < P.tasks[k].batch_end; ++i) {
        cost[k] += wrow_taps(P.code[i]);
      }
    std::stable_sort(P.task_order.begin(), P.task_order.end(),
                     [&](int32_t x, int32_t y) { return cost[x] > cost[y]; });
  }
  return P;
}

bool build_wstrips(const WPlan &plan, int64_t max_cells, WStripPlan &out) {
  WStripPlan W;
  const int64_t M = plan.M;
  W.tiles = (plan.Smax + 7 + 7) / 8;
  if (W.tiles > kMaxStripTiles) return false;
  W.rows = plan.Smax + kStripRows - 1;
  W.strips = (plan.Nv + kStripRows - 1) / kStripRows;
  W.cols = (plan.Nu + kStripCols - 1) / kStripCols;
  const int64_t ngroups = int64_t(W.strips) * W.cols;

  // Sort key of a row inside its group: half of the strip, then blocks of 8
  // rows and columns reached, most first.
  std::vector<int32_t> group(M);
  std::vector<uint16_t> key(M), start(M);
  std::vector<int32_t> tile(M);
  for (size_t k = 0; k < plan.tasks.size(); ++k)
    for (int32_t i = plan.tasks[k].batch_begin; i < plan.tasks[k].batch_end; ++i)
      tile[i] = int32_t(k);
#pragma omp parallel for schedule(static)
  for (int64_t i = 0; i < M; ++i) {
    const int32_t code = plan.code[i];
    const int S = wrow_support(code);
    const int p = plan.tasks[tile[i]].P + (code & 0xff), q = plan.tasks[tile[i]].Q + ((code >> 8) & 0xff);
    group[i] = (p / kStripRows) * W.cols + q / kStripCols;
    const int half = (p % kStripRows) / 8, dv = p % 8, du = q % 8;
    const int tv = (dv + S + 7) / 8, tu = (du + S + 7) / 8;
    start[i] = uint16_t(dv | (du << 4));
    key[i] = uint16_t((half << 8) | ((15 - tv) << 4) | (15 - tu));
  }
  // Stable counting sort by group, then a sort of each group by key.
  std::vector<int64_t> first(ngroups + 1, 0);
  for (int64_t i = 0; i < M; ++i) ++first[group[i] + 1];
  for (int64_t g = 0; g < ngroups; ++g) first[g + 1] += first[g];
  std::vector<int32_t> order(M);
  {
    std::vector<int64_t> fill(first.begin(), first.end() - 1);
    for (int64_t i = 0; i < M; ++i) order[fill[group[i]]++] = int32_t(i);
  }
#pragma omp parallel for schedule(dynamic, 256)
  for (int64_t g = 0; g < ngroups; ++g)
    std::stable_sort(order.begin() + first[g], order.begin() + first[g + 1],
                     [&](int32_t x, int32_t y) { return key[x] < key[y]; });

  // Octs of every group: the terms of a row stay together, an oct stays in
  // one half.
  std::vector<int32_t> goct(ngroups + 1, 0);  // first oct of each group
  std::vector<int64_t> cost(ngroups, 0);
  const WTerm none{0, 0, -1, 0.f, 0.f, 0, 0};
  for (int64_t g = 0; g < ngroups; ++g) {
    int used = kOctTerms, half = -1;
    int32_t *oct = nullptr;
    for (int64_t r = first[g]; r < first[g + 1]; ++r) {
      const int32_t i = order[r], code = plan.code[i];
      const int S = wrow_support(code), rank = wrow_rank(code);
      if (used + rank > kOctTerms || half != (key[i] >> 8)) {
        half = key[i] >> 8;
        if (W.octs.size() >= size_t(INT32_MAX) / kOctTerms) return false;
        W.octs.push_back(0);
        W.terms.insert(W.terms.end(), kOctTerms, none);
        oct = &W.octs.back();
        used = 0;
      }
      const int tv = std::max(*oct & 15, 15 - ((key[i] >> 4) & 15));
      const int tu = std::max((*oct >> 4) & 15, 15 - (key[i] & 15));
      for (int e = 0; e < rank; ++e) {
        WTerm &t = W.terms[(W.octs.size() - 1) * kOctTerms + used + e];
        t.a = plan.factor[i] + int64_t(e) * S;
        t.b_off = rank * S;
        t.m = plan.slot_user[i];
        t.wx = float(plan.weight[i].real());
        t.wy = float(plan.weight[i].imag());
        t.first_tap = start[i] | (S << 8) | ((e == 0 ? rank : 0) << 16);
      }
      used += rank;
      *oct = tv | (tu << 4) | (half << 8);
    }
    for (int32_t o = goct[g]; o < int32_t(W.octs.size()); ++o)
      for (int k = 0; k < kOctTerms; ++k)
        W.terms[size_t(o) * kOctTerms + k].blocks = W.octs[o];
    goct[g + 1] = int32_t(W.octs.size());
    for (int32_t o = goct[g]; o < goct[g + 1]; ++o)
      cost[g] += int64_t(W.octs[o] & 15) * ((W.octs[o] >> 4) & 15);
  }

  // Tasks: runs of groups of one strip, cut at gaps (where the columns a
  // window carries past its last group would all be empty) and at a bound on
  // the work (in blocks of an oct); a group above the bound is split.  A
  // task's window is tail columns wider than its groups, which cost about as
  // much as a few octs, so the bound gives kMinWork to a task once that
  // leaves every SM its 7 CTAs, and three tasks to a warp of G^H (12 an SM)
  // beyond that.  It grows until the windows fit.
  int64_t total = 0;
  for (int64_t g = 0; g < ngroups; ++g) total += cost[g] + 4;
  const int tail = kStripCols * (W.tiles - 1);
  auto cut = [&](int64_t bound) {
    W.tasks.clear();
    W.group_oct.clear();
    W.owner.assign(ngroups, int2_t{0, 0});
    W.window_cells = 0;
    auto add = [&](int s, int c, int n, int32_t o0, int32_t o1) {
      WStripTask t{};
      t.P = s * kStripRows;
      t.Q = c * kStripCols;
      t.groups = n;
      t.width = n * kStripCols + tail;
      t.window = W.window_cells;
      t.oct0 = int32_t(W.group_oct.size());
      W.window_cells += int64_t(t.width) * W.rows;
      W.group_oct.push_back(o0);
      for (int k = 0; k < n; ++k)
        W.group_oct.push_back(n == 1 ? o1 : goct[int64_t(s) * W.cols + c + k + 1]);
      const int32_t id = int32_t(W.tasks.size());
      W.tasks.push_back(t);
      for (int k = 0; k < n; ++k) {
        int2_t &w = W.owner[int64_t(s) * W.cols + c + k];
        if (w.x == w.y) w.x = id;
        w.y = id + 1;
      }
    };
    for (int s = 0; s < W.strips; ++s)
      for (int c = 0; c < W.cols;) {
        const int64_t g0 = int64_t(s) * W.cols;
        if (goct[g0 + c] == goct[g0 + c + 1]) {
          ++c;
          continue;
        }
        if (cost[g0 + c] > bound && goct[g0 + c + 1] - goct[g0 + c] > 1) {
          // parts of one group
          const int32_t a = goct[g0 + c], n = goct[g0 + c + 1] - a;
          const int32_t parts = int32_t(std::min<int64_t>(n, (cost[g0 + c] + bound - 1) / bound));
          for (int32_t k = 0; k < parts; ++k)
            add(s, c, 1, a + int32_t(int64_t(n) * k / parts), a + int32_t(int64_t(n) * (k + 1) / parts));
          ++c;
          continue;
        }
        int e = c, gap = 0, last = c;
        int64_t work = 0;
        while (e < W.cols && gap < W.tiles) {
          const int64_t g = g0 + e;
          const bool empty = goct[g] == goct[g + 1];
          if (!empty) {
            if (e > c && (work + cost[g] > bound || cost[g] > bound)) break;
            last = e;
          }
          work += cost[g] + 4;
          gap = empty ? gap + 1 : 0;
          ++e;
        }
        add(s, c, last - c + 1, goct[g0 + c], goct[g0 + last + 1]);
        c = last + 1;
      }
  };
  constexpr int64_t kMinWork = 256;
  const int64_t most = total / (152 * 12 * 3), few = std::min(kMinWork, total / (152 * 7));
  for (int64_t bound = std::max<int64_t>(64, std::max(most, few));; bound += bound / 8 + 1) {
    cut(bound);
    if (W.window_cells <= max_cells) break;
    if (bound > total) return false;
  }
  W.order.resize(W.tasks.size());
  std::iota(W.order.begin(), W.order.end(), 0);
  std::vector<int64_t> &tcost = W.task_cost;
  tcost.assign(W.tasks.size(), 0);
  for (size_t k = 0; k < W.tasks.size(); ++k) {
    const WStripTask &t = W.tasks[k];
    tcost[k] = 4 * t.groups;
    for (int32_t o = W.group_oct[t.oct0]; o < W.group_oct[t.oct0 + t.groups]; ++o)
      tcost[k] += int64_t(W.octs[o] & 15) * ((W.octs[o] >> 4) & 15);
  }
  std::stable_sort(W.order.begin(), W.order.end(),
                   [&](int32_t x, int32_t y) { return tcost[x] > tcost[y]; });

  out = std::move(W);
  return true;
}

// Each launch takes about fixed + max(A, B) + alpha min(A, B) us: A the work of
// all tasks, B the longest task's.  The band kernels' work goes by the steps
// their warps take over a row's taps, as many as 18 of them spent on a row
// besides, and by window cells; the strip kernels' by octets, their blocks,
// groups or window cells: they waste octets that few rows fill and columns that
// no row touches.  Fitted separately below and at four blocks (whose code starts
// slowly) to both kernels' times on 121 coverages: 64^2 to 1024^2 images, also
// 624 x 208 and 150 x 900, 2 x 10^3 to 10^6 rows, uniform and peaked, supports of 4 to
// 24; rms errors of the fits 4 to 12%.  The strip kernels are taken where
// they are expected to win by 3%.  Some of the times, us, band and strip
// kernels: 512^2, 3 x 10^4 rows of 4 to 24 taps: G 24, 30, G^H 48, 45; 10^6: 282, 180 and
// 557, 246; 1024^2, 10^5: 61, 74 and 132, 126; 3 x 10^5: 111, 119 and 219, 152; 624 x 208,
// 8,000: 16, 16 and 23, 33; supports of 9, 400^2, 2,000: 11, 13 and 17, 17; 2 x 10^5: 80,
// 27 and 174, 39.
RowKernels choose_row_kernels(const WPlan &P, const WStripPlan &W) {
  double steps = 0, longest = 0;
  for (const Task &t : P.tasks) {
    double c = 0;
    for (int32_t i = t.batch_begin; i < t.batch_end; ++i) {
      // rows of taps that the 32 lanes take at once
      const int S = wrow_support(P.code[i]), at_once = std::max(1, 32 / S);
      c += 18 + wrow_rank(P.code[i]) * ((S + at_once - 1) / at_once);
    }
    steps += c;
    longest = std::max(longest, c);
  }
  const double windows = double(P.win_rows) * P.win_cols * double(P.tasks.size());
  double blocks = 0, groups = 0, slongest = 0;
  for (int32_t o : W.octs) blocks += (o & 15) * ((o >> 4) & 15);
  for (size_t k = 0; k < W.tasks.size(); ++k) {
    groups += W.tasks[k].groups;
    slongest = std::max(slongest, double(W.task_cost[k]));
  }
  const double octs = double(W.octs.size()), swindows = double(W.window_cells),
               cells = double(P.Nu) * P.Nv;
  auto time = [](double fixed, double a, double b, double alpha) {
    return fixed + std::max(a, b) + alpha * std::min(a, b);
  };
  double band_g, band_gh, strip_g, strip_gh;
  if (W.tiles >= 4) {
    band_g = time(5.9, 8.0e-6 * steps + 1.75e-6 * windows, 3.15e-3 * longest, 0.39);
    band_gh = time(12.3, 1.58e-5 * steps + 3.7e-6 * windows + 1.2e-6 * cells, 7.8e-3 * longest,
                   0.24);
    strip_g = time(8.3, 6.4e-4 * octs + 3.9e-5 * blocks + 6.7e-4 * groups, 0.068 * slongest, 0.36);
    strip_gh = time(17.9, 7.5e-4 * octs + 6.4e-5 * blocks + 1.24e-6 * swindows + 4.2e-6 * cells,
                    0.168 * slongest, 0.19);
  } else {
    band_g = time(4.9, 6.7e-6 * steps + 1.8e-6 * windows, 3.0e-3 * longest, 0.7);
    band_gh = time(11.3, 1.44e-5 * steps + 4.2e-6 * windows + 1.5e-6 * cells, 4.1e-3 * longest, 1);
    strip_g = time(6.1, 4.0e-4 * octs, 0.097 * slongest, 0.96);
    strip_gh = time(0.8, 5.7e-4 * octs + 9.6e-7 * swindows + 1.4e-5 * cells, 0.112 * slongest, 1);
  }
  RowKernels r;
  r.gh = strip_gh < 0.97 * band_gh;
  r.g = r.gh && strip_g < 0.97 * band_g;
  return r;
}

template <typename T>
void wplan_factors(const WPlan &P, int64_t i0, int64_t i1, std::complex<T> *out) {
  const int J = P.J;
  const GriddingKernel kern(P.kernel, J, P.oversample_ratio);
  // plain rows: details::init_gridding_matrix_2d receives (kernelv, kernelu)
  // in its (u, v) slots (operators.h:322-324), so the u-axis taps use the
  // kernel of support Jv and the v-axis taps the kernel of support Ju
  const GriddingKernel kern_uslot(P.kernel, P.plain ? P.Jv : J, P.oversample_ratio);
  const GriddingKernel kern_vslot(P.kernel, P.plain ? P.Ju : J, P.oversample_ratio);
  const double dul = P.du_lambda, dvl = P.dv_lambda;
  const int64_t base = i0 < int64_t(P.factor.size()) ? P.factor[i0] : 0;
#pragma omp parallel
  {
    std::vector<double> fu(J), fv(J);
    std::vector<std::complex<double>> alpha(3 * 256), beta(3 * 256), row(6 * 256);
#pragma omp for schedule(dynamic, 1024)
    for (int64_t i = i0; i < i1; ++i) {
      const double u = P.gen_u[i], v = P.gen_v[i], w = P.gen_w[i];
      if (P.plain) {
        // operators.cc:8-46: taps at k + 1 .. k + Ju with k = floor(u - Ju / 2),
        // which sit at offset k - kw inside the row of S = J cells placed at
        // kw = floor(u - S / 2); zero elsewhere; the phase (-1)^j as below
        const int S = J;
        const double kwu = std::floor(u - S * 0.5), kwv = std::floor(v - S * 0.5);
        const double ku = std::floor(u - P.Ju * 0.5), kv = std::floor(v - P.Jv * 0.5);
        const int ou = int(ku - kwu), ov = int(kv - kwv);
        for (int k = 0; k < 2 * S; ++k) row[k] = 0.0;
        for (int j = 1; j <= P.Jv; ++j) row[ov + j - 1] = kern_vslot.value(v - (kv + j));
        for (int j = 1; j <= P.Ju; ++j) row[S + ou + j - 1] = kern_uslot.value(u - (ku + j));
        std::complex<T> *dst = out + (P.factor[i] - base);
        for (int r = 0; r < 2; ++r)
          for (int k = 0; k < S; ++k) {
            const std::complex<double> z = (k & 1) ? -row[r * S + k] : row[r * S + k];
            dst[r * S + k] = std::complex<T>(T(z.real()), T(z.imag()));
          }
        continue;
      }
      const int Jw = P.gen_jw[i], S = Jw + J - 1;
      // Kaiser-Bessel (or other) taps: projection_kernels.cc:66-75
      const double du = u - std::floor(u - J * 0.5), dv = v - std::floor(v - J * 0.5);
      for (int k = 0; k < J; ++k) {
        fu[k] = kern.value(du - k - 1);
        fv[k] = kern.value(dv - k - 1);
      }
      // w-kernel samples: sample (row jv, column ju) = kernelw(dwu - ju - 1,
      // dwv - jv - 1, w) (projection_kernels.cc:76-82, 31-47)
      const double dwu = u - std::floor(u - Jw * 0.5), dwv = v - std::floor(v - Jw * 0.5);
      std::complex<double> *a1 = &alpha[0], *a2 = &alpha[256], *a3 = &alpha[512];
      std::complex<double> *b1 = &beta[0], *b2 = &beta[256], *b3 = &beta[512];
      const std::complex<double> c = std::complex<double>(1.0 / w, 0.0) / std::complex<double>(0, 1);
      // g = (a~ / (w i)) b~^T + (1 - chi_v) 1^T + chi_v (1 - chi_u)^T: every
      // sample comes from exactly one term, so no term cancels another.
      for (int k = 0; k < Jw; ++k) {
        const double U = dwu - k - 1, V = dwv - k - 1;
        const bool ok_u = std::abs(U * dul / w) < 1, ok_v = std::abs(V * dvl / w) < 1;
        const double uu = U * dul, vv = V * dvl;
        a1[k] = ok_v ? c * std::exp(std::complex<double>(0, -kPi * vv * vv / w)) : 0.0;
        b1[k] = ok_u ? std::exp(std::complex<double>(0, -kPi * uu * uu / w)) : 0.0;
        a2[k] = ok_v ? 0.0 : 1.0;
        b2[k] = 1.0;
        a3[k] = ok_v ? 1.0 : 0.0;
        b3[k] = ok_u ? 0.0 : 1.0;
      }
      // the nonzero terms only (the row code's term mask): A of each, then B
      const int terms = wrow_terms(P.code[i]), rank = wrow_rank(P.code[i]);
      int e = 0;
      for (int r = 0; r < 3; ++r)
        if (terms >> r & 1) {
          conv1d(fv.data(), J, &alpha[256 * r], Jw, &row[e * S]);
          conv1d(fu.data(), J, &beta[256 * r], Jw, &row[(rank + e) * S]);
          ++e;
        }
      std::complex<T> *dst = out + (P.factor[i] - base);
      for (int r = 0; r < 2 * rank; ++r)
        for (int k = 0; k < S; ++k) {
          const std::complex<double> z = (k & 1) ? -row[r * S + k] : row[r * S + k];
          dst[r * S + k] = std::complex<T>(T(z.real()), T(z.imag()));
        }
    }
  }
}

template void wplan_factors<float>(const WPlan &, int64_t, int64_t, std::complex<float> *);
template void wplan_factors<double>(const WPlan &, int64_t, int64_t, std::complex<double> *);

}  // namespace pg
