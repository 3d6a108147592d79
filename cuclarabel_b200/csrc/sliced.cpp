// sliced.cpp -- builds the layouts of sliced.hpp from a prepared instance.
//
// What bounds it: short loops (a row of L has three terms, a level a few dozen
// rows) whose exits the host mispredicts, some 15 k terms and operations an
// instance.  So parts point at their terms where these already lie, lanes are
// written once, to their final place, and the operations of a level are listed
// in one sweep and sorted flat.  The first form, which copied terms, filled pages
// and then copied them into stages, took 430 us an instance of the MPC family
// (4096 of them: 97-104 ms on 16 threads); this takes 290 us (58 ms).
#include "sliced.hpp"

#include <algorithm>
#include <cstring>
#include <type_traits>

namespace clgpu {

namespace {

// A segment's part inside one chunk: its first term in the stream and in its
// source array, terms, lanes; where its sum goes, or the carry it starts from or
// leaves (-1: none).
struct Part {
  int first, src, len, to;
  int carry_in, carry_out;
  int lanes;
  bool scan_last;  // the last lane's run is full
};

// The parts of a stream's segments, chunk length 32 R, by phase: part i of a
// segment is in phase i, which needs phase i - 1's carries.  Carry slots count
// from 0.
struct Splitter {
  std::vector<std::vector<Part>> phase{1};
  int nphase = 0, ncarry = 0;
  void start() {
    for (int i = 0; i < nphase; ++i) phase[i].clear();
    nphase = ncarry = 0;
  }
  // terms [p0, p1) of the stream, at src in their source
  template <int R>
  void add(int to, int src, int p0, int p1) {
    constexpr int chunk = 32 * R;
    if (p0 >= p1) return;
    if (p0 / chunk == (p1 - 1) / chunk) {
      nphase = std::max(nphase, 1);
      phase[0].push_back({p0, src, p1 - p0, to, -1, -1,
                          (p1 - 1) % chunk / R - p0 % chunk / R + 1, (p1 - 1) % R == R - 1});
      return;
    }
    const int carry = ncarry++;
    for (int a = p0, i = 0; a < p1; ++i) {
      const int b = std::min(p1, (a / chunk + 1) * chunk);
      if (i == (int)phase.size()) phase.emplace_back();
      nphase = std::max(nphase, i + 1);
      phase[i].push_back({a, src + (a - p0), b - a, to, i > 0 ? carry : -1, b < p1 ? carry : -1,
                          (b - 1) % chunk / R - a % chunk / R + 1, (b - 1) % R == R - 1});
      a = b;
    }
  }
};

// steps a scan takes to add `reach` lanes back
int scan_steps(int reach) {
  int s = 0;
  for (int d = 1; d <= reach; d <<= 1) ++s;
  return s;
}
// The last lane of a part that ends inside its run is not scanned: it adds the
// previous lane's scanned sum.
bool adds_previous(const Part &q) { return !q.scan_last && q.lanes > 1; }

// Fills pages with whole parts, widest first, so a page's parts need about
// the same scan steps.
struct Packer {
  struct Page {
    int used, steps;  // lanes with a part; the widest part's scan steps
    bool prev, carry;  // some lane adds the previous one's sum; starts from a carry
  };
  std::vector<int> order;
  std::vector<std::pair<int, int>> at;  // per part: page, first lane
  std::vector<Page> pages;
  void pack(const std::vector<Part> &parts) {
    static const struct Steps {
      int of[33];
      Steps() {
        for (int r = 0; r < 33; ++r) of[r] = scan_steps(r);
      }
    } steps;
    const int n = (int)parts.size();
    int cnt[34] = {};
    for (const Part &q : parts) cnt[33 - q.lanes]++;
    for (int i = 1; i < 34; ++i) cnt[i] += cnt[i - 1];
    order.resize(n);
    for (int i = n - 1; i >= 0; --i) order[--cnt[33 - parts[i].lanes]] = i;
    at.resize(n);
    pages.clear();
    int lane = 32;
    for (int i : order) {
      const Part &q = parts[i];
      if (lane + q.lanes > 32) {
        pages.push_back({0, 0, false, false});
        lane = 0;
      }
      Page &pg = pages.back();
      at[i] = {(int)pages.size() - 1, lane};
      lane += q.lanes;
      const bool prev = adds_previous(q);
      pg.used = lane;
      pg.steps = std::max(pg.steps, steps.of[q.lanes - (prev ? 2 : 1)]);
      pg.prev = pg.prev || prev;
      pg.carry = pg.carry || q.carry_in >= 0;
    }
  }
};

struct Op {
  uint16_t a, b, k;
};
struct Place {
  int lane0, in_stage, used;  // first stored lane, lane in the stage, stage's lanes
};
struct Mark {
  int of, at;
};
// A thread's working arrays, kept between instances (taken by reference once: a
// thread_local's address is looked up at every use).
struct Work {
  Splitter split;
  Packer packer;
  std::vector<Place> place;
  std::vector<Mark> mark;
  std::vector<Op> lev, found;
  std::vector<int> nodes, target_of, cnt, segs, target, page_of;
  std::vector<uint32_t> opg[kSlWarps];
};

}  // namespace

bool sl_build(const Prepared &p, int vgroup, SlicedPlan &s) {
  const int N = p.N, nl = (int)p.Li.size(), nlev = (int)p.lvl_ptr.size() - 1;
  s.N = N;
  s.nl = nl;
  s.nlev = nlev;
  thread_local Work own;
  Work &work = own;
  Splitter &split = work.split;
  Packer &packer = work.packer;
  auto &place = work.place;
  s.ncarry = 0;
  s.ent.clear();
  s.lpos.clear();
  s.used.clear();
  s.kslot.resize(p.Kj.size());
  for (int &n : s.nstage) n = 0;
  int nlane = 0, nklane = 0;  // lanes of the factor passes, of the residual
  const uint32_t pad = 8u * (uint32_t)N, none = (uint32_t)N << 16;
  // One pass's level: its split parts into pages, phase by phase, and those into
  // stages.  slot[src]: gathered slot of a term; pos(src): its factor entry.
  auto emit = [&](auto which, const int *slot, auto pos) {
    constexpr int pass = decltype(which)::value;
    s.ncarry = std::max(s.ncarry, split.ncarry);
    int &base = pass < 2 ? nlane : nklane;
    for (int ph = 0; ph < split.nphase; ++ph) {
      const auto &parts = split.phase[ph];
      packer.pack(parts);
      const int np = (int)packer.pages.size(), first = base;
      place.resize(np);
      for (int i = 0; i < np; i += kSlStagePages) {
        const int last = std::min(np, i + kSlStagePages) - 1;
        // every page but the last with all its lanes
        const int used = 32 * (last - i) + packer.pages[last].used;
        s.used.push_back((uint8_t)used);
        s.nstage[pass]++;
        for (int k = i; k <= last; ++k) place[k] = {base + 32 * (k - i), 32 * (k - i), used};
        base += used;
      }
      const size_t e0 = s.ent.size();
      s.ent.resize(e0 + 4 * (size_t)(base - first));
      uint32_t *ent = s.ent.data() + e0;
      if (pass < 2) s.lpos.resize((size_t)base * kSlRun, kSlNone);
      uint16_t *lpos = s.lpos.data();
      int *kslot = s.kslot.data();
      auto control = [&](const Packer::Page &pg) {
        return (uint32_t)(pg.steps | (pg.carry ? 8 : 0) | (pg.prev ? 16 : 0)) << 16;
      };
      for (int k = 0; k < np; ++k) {  // lanes without a part
        const Packer::Page &pg = packer.pages[k];
        const int end = std::min(32, place[k].used - place[k].in_stage);
        for (int l = pg.used; l < end; ++l) {
          uint32_t *w = ent + 4 * (place[k].lane0 - first + l);
          w[0] = w[2] = pad | none;
          w[1] = pad;
          w[3] = pad | control(pg);
        }
      }
      for (int i : packer.order) {  // (parts of equal widths one after the other)
        const Part &q = parts[i];
        const Packer::Page &pg = packer.pages[packer.at[i].first];
        const Place &pl = place[packer.at[i].first];
        const int l0 = packer.at[i].second;
        const uint32_t ctl = control(pg);
        const bool prev = adds_previous(q);
        const int to = q.carry_out >= 0 ? N + 1 + q.carry_out : q.to;
        uint32_t *w = ent + 4 * (pl.lane0 - first + l0);
        int x = q.src, left = q.len, room = kSlRun - q.first % kSlRun;
        for (int r = 0; r < q.lanes; ++r, w += 4) {
          const int n = std::min(left, room), lane = pl.in_stage + l0 + r;
          // positions of the run's terms: sl_at of (0 .. 3, lane)
          const int v = pass < 2 ? vgroup : 2;
          const int v0 = (pl.lane0 - pl.in_stage) * kSlRun + lane * v;
          const int v2 = v0 + (v == 2 ? 2 * pl.used : 2);
          const int at[kSlRun] = {v0, v0 + 1, v2, v2 + 1};
          uint32_t id[kSlRun] = {pad, pad, pad, pad};
          for (int c = 0; c < n; ++c) {
            id[c] = 8u * (uint32_t)slot[x + c];
            if (pass < 2)
              lpos[at[c]] = (uint16_t)pos(x + c);
            else
              kslot[x + c] = at[c];
          }
          const bool last = r == q.lanes - 1;
          w[0] = id[0] | (last ? (uint32_t)to << 16 : none);
          w[1] = id[1] | (uint32_t)(last && prev ? 32 : r) << 16;
          w[2] = id[2] | (r == 0 && q.carry_in >= 0 ? (uint32_t)(N + 1 + q.carry_in) << 16 : none);
          w[3] = id[3] | ctl;
          x += n;
          left -= n;
          room = kSlRun;
        }
      }
    }
  };
  // ---- substitutions: rows of L, leaves first; columns of L, roots first
  for (int dir = 0; dir < 2; ++dir) {
    const bool fwd = dir == 0;
    const int *Xp = fwd ? p.Rp.data() : p.Lp.data();
    for (int ll = 0; ll < nlev; ++ll) {
      const int l = fwd ? ll : nlev - 1 - ll;
      split.start();
      int at = 0;
      for (int t = p.lvl_ptr[l]; t < p.lvl_ptr[l + 1]; ++t) {
        const int j = p.lvl_nodes[t], len = Xp[j + 1] - Xp[j];
        split.add<kSlRun>(j, Xp[j], at, at + len);
        at += len;
      }
      if (fwd)
        emit(std::integral_constant<int, 0>(), p.Rk.data(), [&](int x) { return p.Rpos[x]; });
      else
        emit(std::integral_constant<int, 1>(), p.Li.data(), [](int x) { return x; });
    }
  }
  // ---- residual: the rows of K as one stream
  split.start();
  for (int r = 0; r < N; ++r) split.add<kSlRun>(r, p.Kp[r], p.Kp[r], p.Kp[r + 1]);
  emit(std::integral_constant<int, 2>(), p.Kj.data(), [](int x) { return x; });
  if (8 * (N + 1 + s.ncarry) >= 0xffff) return false;
  // ---- the work position every stored K value initialises
  s.kdst.assign((size_t)nklane * kSlRun, kSlNone);
  work.mark.assign(N, {-1, 0});
  Mark *mark = work.mark.data();
  for (int r = 0; r < N; ++r) {
    for (int t = p.Rp[r]; t < p.Rp[r + 1]; ++t) mark[p.Rk[t]] = {r, p.Rpos[t]};
    for (int t = p.Kp[r]; t < p.Kp[r + 1]; ++t) {
      const int col = p.Kj[t];
      if (col == r) {
        s.kdst[s.kslot[t]] = (uint16_t)r;
      } else if (col < r) {
        if (mark[col].of != r) return false;  // not inside the factor's pattern
        s.kdst[s.kslot[t]] = (uint16_t)(N + mark[col].at);
      }
    }
  }
  // ---- factorisation ops, level by level: the updates of the level's
  // diagonals (M(j,k)^2 / d_k), then of its columns' entries (M(i,k) M(j,k) /
  // d_k), grouped by target, targets in increasing order; the stream is cut
  // into kSlWarps parts of about equal length at segment starts, chunks start
  // anew in each
  auto &nodes = work.nodes, &cnt = work.cnt, &segs = work.segs, &target = work.target,
       &page_of = work.page_of;
  auto &opg = work.opg;
  size_t nops = p.Rk.size();  // every op of the instance, so of any level
  for (size_t r = 0; r < p.Rk.size(); ++r) nops += p.Lp[p.Rk[r] + 1] - p.Rpos[r] - 1;
  if (work.lev.size() < nops) {
    work.lev.resize(nops);
    work.found.resize(nops);
    work.target_of.resize(nops);
  }
  Op *lev = work.lev.data(), *found = work.found.data();
  int *target_of = work.target_of.data();
  int oskip[kSlWarps] = {}, ends[kSlWarps] = {};
  for (auto &o : opg) o.clear();
  s.nopcarry = 0;
  s.olevels = 0;
  s.ecol.resize(nl);
  for (int j = 0; j < N; ++j)
    for (int q = p.Lp[j]; q < p.Lp[j + 1]; ++q) s.ecol[q] = (uint16_t)j;
  s.sign.assign(p.Dsign.begin(), p.Dsign.end());
  s.leaf.assign(p.lvl_nodes.begin() + p.lvl_ptr[0], p.lvl_nodes.begin() + p.lvl_ptr[1]);
  const int zero = N + nl;
  // one lane of an op page (the fields of sliced.hpp)
  auto encode = [](uint32_t *w, const Op &o0, const Op &o1, uint32_t t, uint32_t ini,
                   uint32_t meta) {
    w[0] = o0.a | ((uint32_t)o0.b << 15) | ((uint32_t)o0.k << 30);
    w[1] = ((uint32_t)o0.k >> 2) | ((uint32_t)o1.a << 11) | ((uint32_t)o1.b << 26);
    w[2] = ((uint32_t)o1.b >> 6) | ((uint32_t)o1.k << 9) | (t << 22);
    w[3] = (t >> 10) | (ini << 5) | (meta << 16);
  };
  const Op none_op{(uint16_t)zero, (uint16_t)zero, 0};
  uint32_t padw[4];
  encode(padw, none_op, none_op, (uint32_t)zero, 0u, 0u);
  // the level ends a warp's last page has collected, written with its next page
  auto settle = [&](int w) {
    if (opg[w].empty() || !ends[w]) return;
    uint32_t *e = opg[w].data() + opg[w].size() - kSlOpWords;
    for (int l = 0; l < 32; ++l) e[4 * l + 3] |= (uint32_t)ends[w] << 25;
    ends[w] = 0;
  };
  work.mark.assign(N, {-1, 0});
  const int *Li = p.Li.data(), *Lp = p.Lp.data();
  for (int l = 1; l < nlev; ++l) {
    nodes.assign(p.lvl_nodes.begin() + p.lvl_ptr[l], p.lvl_nodes.begin() + p.lvl_ptr[l + 1]);
    std::sort(nodes.begin(), nodes.end());
    // one sweep lists the diagonals' ops in place and the entries' in the order
    // they are found, each with its entry's place in the level
    segs.clear();
    target.clear();
    int nent = 0, nd = 0, nf = 0;
    for (int j : nodes) {
      const int r0 = p.Rp[j], r1 = p.Rp[j + 1], q0 = Lp[j], len = Lp[j + 1] - q0;
      if (r0 == r1) continue;
      segs.push_back(nd);
      target.push_back(j);
      for (int q = 0; q < len; ++q) mark[Li[q0 + q]] = {j, nent + q};
      bool inside = true;
      for (int r = r0; r < r1; ++r) {
        const int k = p.Rk[r], pjk = p.Rpos[r], pe = Lp[k + 1];
        const uint16_t b = (uint16_t)(N + pjk), kk = (uint16_t)k;
        lev[nd++] = {b, b, kk};
        for (int pp = pjk + 1; pp < pe; ++pp, ++nf) {
          const Mark m = mark[Li[pp]];
          inside &= m.of == j;
          target_of[nf] = m.at;
          found[nf] = {(uint16_t)(N + pp), b, kk};
        }
      }
      if (!inside) return false;  // fill outside the pattern
      nent += len;
    }
    // sorted by entry, in the order found (columns of L lie in node order)
    cnt.assign(nent + 1, 0);
    for (int t = 0; t < nf; ++t) cnt[target_of[t]]++;
    const int f = nd + nf;
    {
      int at = nd, e = 0;
      for (int j : nodes) {
        if (p.Rp[j] == p.Rp[j + 1]) continue;
        for (int q = Lp[j]; q < Lp[j + 1]; ++q, ++e) {
          const int n = cnt[e];
          cnt[e] = at;
          if (!n) continue;
          segs.push_back(at);
          target.push_back(N + q);
          at += n;
        }
      }
    }
    for (int t = 0; t < nf; ++t) lev[cnt[target_of[t]]++] = found[t];
    const int nseg = (int)segs.size();
    segs.push_back(f);
    int sb[kSlWarps + 1];
    sb[0] = 0;
    sb[kSlWarps] = nseg;
    for (int w = 1; w < kSlWarps; ++w) {
      const int ideal = (int)((size_t)f * w / kSlWarps);
      const int g = (int)(std::lower_bound(segs.begin(), segs.end(), ideal) - segs.begin());
      sb[w] = std::min(nseg, std::max(sb[w - 1], g));
    }
    // every stream part starts a chunk of the common stream
    split.start();
    constexpr int chunk = 32 * kSlOpRun;
    for (int w = 0, at = 0; w < kSlWarps; ++w) {
      const int s0 = segs[sb[w]];
      for (int g = sb[w]; g < sb[w + 1]; ++g)
        split.add<kSlOpRun>(target[g], segs[g], segs[g] - s0 + at, segs[g + 1] - s0 + at);
      at += (segs[sb[w + 1]] - s0 + chunk - 1) / chunk * chunk;
    }
    s.nopcarry = std::max(s.nopcarry, split.ncarry);
    if (zero + s.nopcarry >= 1 << kSlOpT.width || s.nopcarry >= 1 << kSlOpIni.width) return false;
    for (int ph = 0; ph < split.nphase; ++ph) {
      const auto &parts = split.phase[ph];
      packer.pack(parts);
      int rank[kSlWarps];
      for (int w = 0; w < kSlWarps; ++w) rank[w] = w;
      std::stable_sort(rank, rank + kSlWarps,
                       [&](int a, int b) { return opg[a].size() < opg[b].size(); });
      const int np = (int)packer.pages.size();
      page_of.resize(np);
      for (int i = 0; i < np; ++i) {
        const int w = rank[i % kSlWarps];
        settle(w);
        auto &O = opg[w];
        page_of[i] = (int)O.size();
        O.resize(O.size() + kSlOpWords);
        uint32_t *e = O.data() + page_of[i];
        const Packer::Page &pg = packer.pages[i];
        for (int l2 = pg.used; l2 < 32; ++l2) {
          std::copy_n(padw, 4, e + 4 * l2);
          e[4 * l2 + 3] |= (uint32_t)pg.steps << 22;
        }
      }
      for (int i : packer.order) {
        const Part &q = parts[i];
        const int pgi = packer.at[i].first, l0 = packer.at[i].second;
        uint32_t *e = opg[rank[pgi % kSlWarps]].data() + page_of[pgi] + 4 * l0;
        const uint32_t steps = (uint32_t)packer.pages[pgi].steps << 6;
        const bool prev = adds_previous(q);
        const uint32_t to = (uint32_t)(q.carry_out >= 0 ? zero + 1 + q.carry_out : q.to);
        const Op *o = lev + q.src;
        int t = q.first;
        const int end = q.first + q.len;
        for (int r = 0; r < q.lanes; ++r, e += 4) {
          const bool two = t % kSlOpRun == 0 && t + 1 < end, last = r == q.lanes - 1;
          Op o1 = o[two ? 1 : 0];
          if (!two) o1.a = o1.b = (uint16_t)zero;
          encode(e, o[0], o1, last ? to : (uint32_t)zero,
                 r == 0 && q.carry_in >= 0 ? 1u + (uint32_t)q.carry_in : 0u,
                 steps | (last && prev ? 32u : (uint32_t)r));
          t += two ? 2 : 1;
          o += two ? 2 : 1;
        }
      }
      // the phase's end (the last one is the level's)
      ++s.olevels;
      for (int w = 0; w < kSlWarps; ++w) {
        if (opg[w].empty())
          ++oskip[w];
        else if (++ends[w] > kSlOpMaxWait)
          return false;
      }
    }
  }
  s.ops.clear();
  size_t nop_words = 0;
  for (const auto &o : opg) nop_words += o.size();
  s.ops.reserve(nop_words);
  for (int w = 0; w < kSlWarps; ++w) {
    settle(w);
    s.op.first[w] = (int)(s.ops.size() / kSlOpWords);
    s.op.count[w] = (int)(opg[w].size() / kSlOpWords);
    s.op.skip[w] = oskip[w];
    s.ops.insert(s.ops.end(), opg[w].begin(), opg[w].end());
  }
  const SlNeed need = sl_need(s);
  return std::max({need.solve[0], need.solve[1], need.factor[0]}) <= kSlSmemMax;
}

SlNeed sl_need(const SlicedPlan &p) {
  const long long ring = (long long)kSlRing * kSlStage * (8 * kSlRun + 16) +
                         (((long long)p.used.size() + 15) & ~15LL);
  const long long slots = 2LL * p.N + 1 + p.ncarry;
  const long long tab = (long long)kSlWarps * kSlOpRing * 512 + ((p.N + 15) & ~15LL);
  const long long V = (long long)p.N + p.nl + 1 + p.nopcarry;
  return {{ring + 8 * slots, ring + 16 * slots}, {tab + 8 * V, tab + 4 * V}};
}

}  // namespace clgpu
