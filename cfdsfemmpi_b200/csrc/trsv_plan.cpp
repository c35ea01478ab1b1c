// Host-side schedule of the block triangular solves; see trsv_plan.h.
#include "trsv_plan.h"

#include <algorithm>
#include <functional>
#include <queue>
#include <utility>

namespace cfdgpu {

namespace {

// a run of rows in solve order: rows a, a+1, .. b-1 (lower) or b-1, .. a (upper)
struct Run {
  int32_t a, b;
};

}  // namespace

void build_trsv_plan(const IluPattern &f, int nb, bool upper, TrsvPlan &p, bool choose)
{
  p = TrsvPlan();
  const int cap = trsv_cap(nb), nslots = trsv_slots(nb), max_slots = trsv_max_slots(nb);
  const int n = (int)f.diag.size();
  auto q0 = [&](int i) { return upper ? f.diag[i] + 1 : f.rowptr[i]; };
  auto q1 = [&](int i) { return upper ? f.rowptr[i + 1] : f.diag[i]; };
  const std::vector<int32_t> &ch = upper ? f.uchain : f.lchain;
  const int nc = (int)ch.size() / 2;

  // dependency level of every row (rows come to be solved in about this order)
  const std::vector<int32_t> &lev = upper ? f.ulev : f.llev;
  const int levels = upper ? f.nlev_u : f.nlev_l;
  int64_t off = 0;
  for (int i = 0; i < n; i++) off += q1(i) - q0(i);
  const double at_once = (double)n / std::max(levels, 1);

  // segments: runs of consecutive chains (in solve order) each depending on
  // the one before; strands: chains of a segment cut only by the length limit
  std::vector<Run> strands;
  std::vector<int> seg;           // first strand of every segment
  for (int c = 0; c < nc; c++) {
    const int a = ch[2 * c], b = ch[2 * c + 1];
    bool dep = false, cont = false;
    if (c > 0) {
      const int pa = ch[2 * c - 2], pb = ch[2 * c - 1];
      for (int i = a; i < b && !dep; i++)
        for (int q = q0(i); q < q1(i) && !dep; q++) dep = f.colidx[q] >= pa && f.colidx[q] < pb;
      const int first = upper ? b - 1 : a, before = upper ? b : a - 1;
      for (int q = q0(first); q < q1(first); q++) cont |= f.colidx[q] == before;
    }
    if (!dep) seg.push_back((int)strands.size());
    if (dep && cont) {
      if (upper) strands.back().a = a;
      else strands.back().b = b;
    } else {
      strands.push_back({a, b});
    }
  }
  seg.push_back((int)strands.size());

  // groups of rows (listed in solve order), cut until rows and inputs fit into max_slots
  std::vector<int32_t> grow, gptr(1, 0), ginp, giptr(1, 0), minlev, gate;
  std::vector<uint8_t> cyclic, direct;
  std::vector<int32_t> mark(n, -1), own(n, -1), need(n, 0), tmp;
  int stamp = 0;
  // inputs of the listed rows from elsewhere, in the order of the lowest level that needs them
  auto inputs = [&](const int32_t *r0, const int32_t *r1) {
    tmp.clear();
    stamp++;
    for (const int32_t *r = r0; r < r1; r++) own[*r] = stamp;
    for (const int32_t *r = r0; r < r1; r++)
      for (int q = q0(*r); q < q1(*r); q++) {
        const int c = f.colidx[q];
        if (own[c] == stamp) continue;
        if (mark[c] != stamp) { mark[c] = stamp; need[c] = lev[*r]; tmp.push_back(c); }
        else need[c] = std::min(need[c], lev[*r]);
      }
    return (int)tmp.size() + (int)(r1 - r0) <= max_slots;
  };
  auto emit = [&](const int32_t *r0, const int32_t *r1, bool cyc) {
    std::sort(tmp.begin(), tmp.end(), [&](int x, int y) { return need[x] != need[y] ? need[x] < need[y] : x < y; });
    int g = 0;
    while (g + 1 < (int)tmp.size() && need[tmp[g + 1]] == need[tmp[0]]) g++;
    gate.push_back(g);
    ginp.insert(ginp.end(), tmp.begin(), tmp.end());
    giptr.push_back((int32_t)ginp.size());
    int m = lev[*r0];
    for (const int32_t *r = r0; r < r1; r++) m = std::min(m, lev[*r]);
    minlev.push_back(m);
    cyclic.push_back(cyc ? 1 : 0);
    direct.push_back(0);
    grow.insert(grow.end(), r0, r1);
    gptr.push_back((int32_t)grow.size());
  };
  // listed rows as one group, or halved until they fit
  auto cut = [&](auto &&self, const int32_t *r0, const int32_t *r1, bool cyc) -> void {
    const bool fits = inputs(r0, r1);
    if (fits || r1 - r0 == 1) {
      emit(r0, r1, cyc);
      direct.back() = !fits;
      return;
    }
    const int32_t *m = r0 + (r1 - r0) / 2;
    self(self, r0, m, cyc);
    self(self, m, r1, cyc);
  };
  int64_t in_turn = 0;            // rows in groups whose rows go to all warps in turn
  const bool level_order = (int64_t)strands.size() * TRSV_SHORT_STRAND > n;
  if (level_order) {
    p.chains = at_once >= TRSV_LEVEL_P || (double)off / levels >= TRSV_LEVEL_BLOCKS;
    if (p.chains && choose) return;
    // level order: groups small enough that every SM has some
    const std::vector<int32_t> &by_level = upper ? f.uorder : f.lorder;
    const int step = std::max(16, std::min(TRSV_LEVEL_ROWS, n / (2 * 148)));
    for (int x = 0; x < n; x += step) cut(cut, by_level.data() + x, by_level.data() + std::min(n, x + step), true);
  } else {
    std::vector<int32_t> rows;    // solve order
    rows.reserve(n);
    std::vector<int32_t> sp(1, 0);
    for (const Run &s : strands) {
      for (int x = 0; x < s.b - s.a; x++) rows.push_back(upper ? s.b - 1 - x : s.a + x);
      sp.push_back((int32_t)rows.size());
    }
    auto cut_strands = [&](auto &&self, int s0, int s1) -> void {
      const int32_t *r0 = rows.data() + sp[s0], *r1 = rows.data() + sp[s1];
      if (s1 - s0 == 1) { cut(cut, r0, r1, false); return; }
      if (r1 - r0 <= max_slots && inputs(r0, r1)) { emit(r0, r1, false); return; }
      const int m = s0 + (s1 - s0) / 2;
      self(self, s0, m);
      self(self, m, s1);
    };
    for (size_t k = 0; k + 1 < seg.size(); k++) {
      const int s0 = seg[k], s1 = seg[k + 1], m = s1 - s0, len = sp[s1] - sp[s0];
      int64_t blocks = 0;
      for (int x = sp[s0]; x < sp[s1]; x++) blocks += q1(rows[x]) - q0(rows[x]);
      if (blocks > (int64_t)len * TRSV_CYCLIC_BLOCKS) {
        // half the slots for the group's own rows, the other half for its inputs
        const int step = std::max(1, max_slots / 2);
        in_turn += len;
        for (int x = 0; x < len; x += step)
          cut(cut, rows.data() + sp[s0] + x, rows.data() + sp[s0] + std::min(len, x + step), true);
        continue;
      }
      const int parts = (m + TRSV_STRANDS - 1) / TRSV_STRANDS;
      for (int g = 0; g < parts; g++)
        cut_strands(cut_strands, s0 + (int)((int64_t)m * g / parts), s0 + (int)((int64_t)m * (g + 1) / parts));
    }
  }
  const int ng = (int)cyclic.size();
  if (!level_order) {
    if (2 * in_turn > n)
      p.chains = at_once >= TRSV_CYCLIC_P && n >= (int64_t)TRSV_CYCLIC_ROWS * ng;
    else
      p.chains = TRSV_GROUP_US * ng / 148 > levels * (TRSV_LEVEL_US + trsv_block_us(nb) * (double)off / n);
    if (p.chains && choose) return;
  }

  // order of the groups: topological, lowest level first
  std::vector<int32_t> group_of(n), order;
  for (int g = 0; g < ng; g++)
    for (int x = gptr[g]; x < gptr[g + 1]; x++) group_of[grow[x]] = g;
  {
    std::vector<int32_t> indeg(ng, 0), seen(ng, -1);
    std::vector<std::vector<int32_t>> succ(ng);
    for (int g = 0; g < ng; g++)
      for (int x = giptr[g]; x < giptr[g + 1]; x++) {
        const int o = group_of[ginp[x]];
        if (seen[o] != g) { seen[o] = g; succ[o].push_back(g); indeg[g]++; }
      }
    using E = std::pair<int32_t, int32_t>;
    std::priority_queue<E, std::vector<E>, std::greater<E>> ready;
    for (int g = 0; g < ng; g++)
      if (!indeg[g]) ready.push({minlev[g], g});
    order.reserve(ng);
    while (!ready.empty()) {
      const int g = ready.top().second;
      ready.pop();
      order.push_back(g);
      for (int o : succ[g])
        if (--indeg[o] == 0) ready.push({minlev[o], o});
    }
  }

  // pieces, slots and input lists in that order
  for (int g = 0; g < ng; g++)
    p.max_slots = std::max(p.max_slots, gptr[g + 1] - gptr[g] + (direct[g] ? 0 : giptr[g + 1] - giptr[g]));
  p.groups.reserve(ng);
  p.wptr.reserve((size_t)ng * (TRSV_WARPS + 1));
  p.pieces.reserve(n + n / 8);
  p.desc.reserve((size_t)(n + n / 8) * (4 + nslots));
  std::vector<int32_t> slot(n, 0);
  for (int g : order) {
    const int32_t *r = grow.data() + gptr[g];
    const int rows = gptr[g + 1] - gptr[g], next = direct[g] ? 0 : giptr[g + 1] - giptr[g];
    p.groups.push_back({rows, (int32_t)p.ext.size(), next, direct[g] ? 0 : gate[g]});
    for (int k = 0; k < rows; k++) slot[r[k]] = k;
    for (int k = 0; k < next; k++) {
      const int c = ginp[giptr[g] + k];
      slot[c] = rows + k;
      p.ext.push_back(c);
    }
    auto add_row = [&](int i) {
      const int lo = q0(i), hi = q1(i), cnt = hi - lo;
      // the blocks nearest the diagonal come last: their inputs are the last to be known
      int done = 0;
      do {
        const int k = std::min(cap, cnt - done);
        const int s = upper ? hi - done - k : lo + done;
        TrsvPiece t;
        t.q0 = s;
        t.n = k | (done == 0 ? TRSV_FIRST : 0) | (done + k == cnt ? TRSV_LAST : 0) | (direct[g] ? TRSV_DIRECT : 0) | ((s & 3) << TRSV_Q0_SHIFT);
        t.desc = (int32_t)(p.desc.size() / 4);
        const int32_t node = f.perm.empty() ? i : f.perm[i];
        t.at = upper ? i : node;
        const int late = k > 0 && !direct[g] ? slot[f.colidx[upper ? s : s + k - 1]] : p.max_slots;    // nearest the diagonal
        for (int32_t v : {i, node, t.n, slot[i] * nb | late * nb << 16}) p.desc.push_back((uint32_t)v);
        const size_t e = p.desc.size();
        p.desc.resize(e + nslots, (uint32_t)(p.max_slots * nb * 8));
        const int per = nslots / 4;
        for (int q = 0; q < k; q++) {
          const int c = f.colidx[s + q];
          p.desc[e + 4 * (q % per) + q / per] =
              direct[g] ? (uint32_t)(upper && !f.perm.empty() ? f.perm[c] : c) * nb : (uint32_t)(slot[c] * nb * 8);
        }
        p.pieces.push_back(t);
        done += k;
      } while (done < cnt);
    };
    p.wptr.push_back((int32_t)p.pieces.size());
    if (cyclic[g]) {
      for (int w = 0; w < TRSV_WARPS; w++) {
        for (int x = w; x < rows; x += TRSV_WARPS) add_row(r[x]);
        p.wptr.push_back((int32_t)p.pieces.size());
      }
    } else {
      // a strand's rows to four warps in turn
      constexpr int PER = TRSV_WARPS / TRSV_STRANDS;
      int w = 0;
      for (int x0 = 0, x1; x0 < rows; x0 = x1) {
        for (x1 = x0 + 1; x1 < rows; x1++) {
          bool cont = false;
          for (int q = q0(r[x1]); q < q1(r[x1]); q++) cont |= f.colidx[q] == r[x1 - 1];
          if (!cont && w < TRSV_WARPS - PER) break;
        }
        for (int k = 0; k < PER; k++) {
          for (int x = x0 + k; x < x1; x += PER) add_row(r[x]);
          p.wptr.push_back((int32_t)p.pieces.size());
          w++;
        }
      }
      for (; w < TRSV_WARPS; w++) p.wptr.push_back((int32_t)p.pieces.size());
    }
  }
}

}  // namespace cfdgpu
