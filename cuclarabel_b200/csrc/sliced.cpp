// sliced.cpp -- builds the layouts of sliced.hpp from a prepared instance.
#include "sliced.hpp"

#include <algorithm>
#include <cstring>

namespace clgpu {

namespace {

// A segment's part inside one chunk: its first term in the stream, terms, and
// which part of the segment it is.
struct Part {
  int first, len, seg, lanes;
  bool more, scan_last;  // continued in the next chunk; last lane's run is full
  int carry_in, carry_out;
};

// The parts of a stream's segments (ends[s] = one past segment s's last term,
// from `begin`), chunk length 32 R, by phase: part i of a segment is in phase
// i, which needs phase i - 1's carries.  Carry slots count from 0.
struct Splitter {
  std::vector<std::vector<Part>> phase;
  int nphase = 0, ncarry = 0;
  void start() {
    for (int i = 0; i < nphase; ++i) phase[i].clear();
    nphase = ncarry = 0;
  }
  // terms [p0, p1) of the stream, which starts at position 0 of a chunk
  void add(int seg, int p0, int p1, int R) {
    const int chunk = 32 * R;
    int carry = -1;
    for (int a = p0, i = 0; a < p1; ++i) {
      const int b = std::min(p1, (a / chunk + 1) * chunk);
      if (i == (int)phase.size()) phase.emplace_back();
      nphase = std::max(nphase, i + 1);
      const int la = a % chunk / R, lb = (b - 1) % chunk / R;
      Part q{a, b - a, seg, lb - la + 1, b < p1, (b - 1) % R == R - 1, i > 0 ? carry : -1, -1};
      if (b < p1) {
        if (carry < 0) carry = ncarry++;
        q.carry_out = carry;
      }
      phase[i].push_back(q);
      a = b;
    }
  }
};

// Fills pages with whole parts, widest first, so a page's parts need about
// the same scan steps.
struct Packer {
  std::vector<int> order, cnt;
  std::vector<std::pair<int, int>> at;  // per part: page, first lane
  int npages = 0;
  void pack(const std::vector<Part> &parts) {
    const int n = (int)parts.size();
    cnt.assign(34, 0);
    for (const Part &q : parts) cnt[33 - q.lanes]++;
    for (int i = 1; i < 34; ++i) cnt[i] += cnt[i - 1];
    order.resize(n);
    for (int i = n - 1; i >= 0; --i) order[--cnt[33 - parts[i].lanes]] = i;
    at.resize(n);
    npages = 0;
    int lane = 32;
    for (int i : order) {
      if (lane + parts[i].lanes > 32) {
        ++npages;
        lane = 0;
      }
      at[i] = {npages - 1, lane};
      lane += parts[i].lanes;
    }
  }
};

int scan_steps(int reach) {
  int s = 0;
  for (int d = 1; d <= reach; d <<= 1) ++s;
  return s;
}

}  // namespace

bool sl_build(const Prepared &p, int vgroup, SlicedPlan &s) {
  const int N = p.N, nl = (int)p.Li.size(), nlev = (int)p.lvl_ptr.size() - 1;
  s.N = N;
  s.nl = nl;
  s.nlev = nlev;
  thread_local Splitter split;
  thread_local Packer packer;
  // one pass's pages, and the first page of every stage
  struct Pages {
    std::vector<uint32_t> ent;
    std::vector<int> pos;    // value position of every term, -1: none
    std::vector<int> used;   // lanes of every page
    std::vector<int> stage;
    void clear() {
      ent.clear();
      pos.clear();
      used.clear();
      stage.clear();
    }
  };
  thread_local Pages pass[3];
  thread_local std::vector<int> term_slot, term_pos, seg_target;
  s.ncarry = 0;
  const uint32_t pad = 8u * (uint32_t)N | ((uint32_t)N << 16);
  // The level's split parts into pages, phase by phase, and those into stages.
  // Terms are term_slot / term_pos, targets seg_target.
  auto emit = [&](Pages &P) {
    s.ncarry = std::max(s.ncarry, split.ncarry);
    for (int ph = 0; ph < split.nphase; ++ph) {
      const auto &parts = split.phase[ph];
      packer.pack(parts);
      const int p0 = (int)P.used.size();
      for (int i = 0; i < packer.npages; i += kSlStagePages) P.stage.push_back(p0 + i);
      P.used.resize(p0 + packer.npages, 0);
      P.ent.resize((size_t)(p0 + packer.npages) * kSlPage, pad);
      P.pos.resize((size_t)(p0 + packer.npages) * kSlPage, -1);
      for (int i = p0; i < p0 + packer.npages; ++i)
        for (int l = 0; l < 32; ++l) {
          P.ent[(size_t)i * kSlPage + 4 * l + 1] = pad & 0xffffu;
          P.ent[(size_t)i * kSlPage + 4 * l + 3] = pad & 0xffffu;
        }
      for (size_t i = 0; i < parts.size(); ++i) {
        const Part &q = parts[i];
        const int pgi = p0 + packer.at[i].first, l0 = packer.at[i].second;
        uint32_t *e = P.ent.data() + (size_t)pgi * kSlPage;
        int *pos = P.pos.data() + (size_t)pgi * kSlPage;
        P.used[pgi] = std::max(P.used[pgi], l0 + q.lanes);
        int reach = 0;
        int t = q.first;
        const int end = q.first + q.len;
        for (int r = 0; r < q.lanes; ++r) {
          uint32_t *el = e + 4 * (l0 + r);
          for (int c = 0; t < end && (c == 0 || t % kSlRun != 0); ++c, ++t) {
            el[c] = (el[c] & 0xffff0000u) | (uint32_t)(8 * term_slot[t]);
            pos[4 * (l0 + r) + c] = term_pos[t];
          }
          const bool last = r == q.lanes - 1;
          const bool prev = last && !q.scan_last && r > 0;
          el[1] = (el[1] & 0xffffu) | ((uint32_t)(prev ? 32 : r) << 16);
          if (!prev)
            reach = std::max(reach, r);
          else if (!(e[3] & (16u << 16)))
            for (int l = 0; l < 32; ++l) e[4 * l + 3] |= 16u << 16;
          if (last) {
            const int to = q.more ? N + 1 + q.carry_out : seg_target[q.seg];
            el[0] = (el[0] & 0xffffu) | ((uint32_t)to << 16);
          }
          if (r == 0 && q.carry_in >= 0) {
            el[2] = (el[2] & 0xffffu) | ((uint32_t)(N + 1 + q.carry_in) << 16);
            if (!(e[3] & (8u << 16)))
              for (int l = 0; l < 32; ++l) e[4 * l + 3] |= 8u << 16;
          }
        }
        const uint32_t steps = (uint32_t)scan_steps(reach);
        if (((e[3] >> 16) & 7u) < steps)
          for (int l = 0; l < 32; ++l) e[4 * l + 3] = (e[4 * l + 3] & ~(7u << 16)) | (steps << 16);
      }
    }
  };
  // ---- substitutions: rows of L, leaves first; columns of L, roots first
  for (int dir = 0; dir < 2; ++dir) {
    const bool fwd = dir == 0;
    const auto &Xp = fwd ? p.Rp : p.Lp;
    const auto &Xi = fwd ? p.Rk : p.Li;
    Pages &pg = pass[dir];
    pg.clear();
    for (int ll = 0; ll < nlev; ++ll) {
      const int l = fwd ? ll : nlev - 1 - ll;
      split.start();
      term_slot.clear();
      term_pos.clear();
      seg_target.clear();
      for (int t = p.lvl_ptr[l]; t < p.lvl_ptr[l + 1]; ++t) {
        const int j = p.lvl_nodes[t], p0 = (int)term_slot.size();
        for (int x = Xp[j]; x < Xp[j + 1]; ++x) {
          term_slot.push_back(Xi[x]);
          term_pos.push_back(fwd ? p.Rpos[x] : x);
        }
        if ((int)term_slot.size() == p0) continue;
        split.add((int)seg_target.size(), p0, (int)term_slot.size(), kSlRun);
        seg_target.push_back(j);
      }
      if (seg_target.empty()) continue;
      emit(pg);
    }
  }
  // ---- residual: the rows of K as one stream
  {
    pass[2].clear();
    split.start();
    const int nk = (int)p.Kj.size();
    term_slot.assign(p.Kj.begin(), p.Kj.end());
    term_pos.resize(nk);
    for (int t = 0; t < nk; ++t) term_pos[t] = t;
    seg_target.resize(N);
    for (int r = 0; r < N; ++r) {
      seg_target[r] = r;
      split.add(r, p.Kp[r], p.Kp[r + 1], kSlRun);
    }
    emit(pass[2]);
  }
  if (8 * (N + 1 + s.ncarry) >= 0xffff) return false;
  // ---- stage arrays, pass by pass
  s.ent.clear();
  s.lpos.clear();
  s.used.clear();
  s.kslot.resize(p.Kj.size());
  int nklane = 0;
  for (int ps = 0; ps < 3; ++ps) {
    Pages &P = pass[ps];
    s.nstage[ps] = (int)P.stage.size();
    P.stage.push_back((int)P.used.size());
    for (int st = 0; st < s.nstage[ps]; ++st) {
      const int pa = P.stage[st], pb = P.stage[st + 1];
      // every page but the last with all its lanes
      const int used = 32 * (pb - pa - 1) + P.used[pb - 1];
      const uint32_t *e = P.ent.data() + (size_t)pa * kSlPage;
      const int *pos = P.pos.data() + (size_t)pa * kSlPage;
      s.used.push_back((uint8_t)used);
      s.ent.insert(s.ent.end(), e, e + 4 * used);
      const size_t v0 = s.lpos.size();
      if (ps < 2) s.lpos.resize(v0 + (size_t)used * kSlRun, kSlNone);
      for (int l = 0; l < used; ++l)
        for (int c = 0; c < kSlRun; ++c) {
          const int x = pos[4 * l + c];
          if (x < 0) continue;
          if (ps == 2)
            s.kslot[x] = nklane * kSlRun + sl_at(c, l, 2, used);
          else
            s.lpos[v0 + sl_at(c, l, vgroup, used)] = (uint16_t)x;
        }
      if (ps == 2) nklane += used;
    }
  }
  // ---- the work position every stored K value initialises
  s.kdst.assign((size_t)nklane * kSlRun, kSlNone);
  {
    thread_local std::vector<int> mark, at;
    mark.assign(N, -1);
    at.resize(N);
    for (int r = 0; r < N; ++r) {
      for (int t = p.Rp[r]; t < p.Rp[r + 1]; ++t) {
        mark[p.Rk[t]] = r;
        at[p.Rk[t]] = p.Rpos[t];
      }
      for (int t = p.Kp[r]; t < p.Kp[r + 1]; ++t) {
        const int col = p.Kj[t];
        if (col == r) {
          s.kdst[s.kslot[t]] = (uint16_t)r;
        } else if (col < r) {
          if (mark[col] != r) return false;  // not inside the factor's pattern
          s.kdst[s.kslot[t]] = (uint16_t)(N + at[col]);
        }
      }
    }
  }
  // ---- factorisation ops, level by level: the updates of the level's
  // diagonals (M(j,k)^2 / d_k), then of its columns' entries (M(i,k) M(j,k) /
  // d_k), grouped by target, targets in increasing order; the stream is cut
  // into kSlWarps parts of about equal length at segment starts, chunks start
  // anew in each
  struct Op {
    uint16_t a, b, k;
  };
  thread_local std::vector<Op> lev;
  thread_local std::vector<int> nodes, cnt, segs, target, rowpos, rowmark;
  thread_local std::vector<uint32_t> opg[kSlWarps];
  thread_local std::vector<int> page_of;
  if ((int)rowpos.size() < N) rowpos.resize(N);
  rowmark.assign(N, -1);
  int oskip[kSlWarps] = {};
  for (auto &o : opg) o.clear();
  s.nopcarry = 0;
  s.olevels = 0;
  s.ecol.resize(nl);
  for (int j = 0; j < N; ++j)
    for (int q = p.Lp[j]; q < p.Lp[j + 1]; ++q) s.ecol[q] = (uint16_t)j;
  s.sign.assign(p.Dsign.begin(), p.Dsign.end());
  s.leaf.clear();
  const int zero = N + nl;
  // one lane of an op page (the fields of sliced.hpp)
  auto encode = [](uint32_t *w, const Op &o0, const Op &o1, uint32_t t, uint32_t ini,
                   uint32_t meta) {
    w[0] = o0.a | ((uint32_t)o0.b << 15) | ((uint32_t)o0.k << 30);
    w[1] = ((uint32_t)o0.k >> 2) | ((uint32_t)o1.a << 11) | ((uint32_t)o1.b << 26);
    w[2] = ((uint32_t)o1.b >> 6) | ((uint32_t)o1.k << 9) | (t << 22);
    w[3] = (t >> 10) | (ini << 5) | (meta << 16);
  };
  auto none = [&](uint16_t k) { return Op{(uint16_t)zero, (uint16_t)zero, k}; };
  uint32_t padw[4];
  encode(padw, none(0), none(0), (uint32_t)zero, 0u, 0u);
  thread_local std::vector<int> page_reach;
  for (int l = 0; l < nlev; ++l) {
    const int qa = p.lvl_ptr[l], qb = p.lvl_ptr[l + 1];
    if (l == 0) {
      s.leaf.assign(p.lvl_nodes.begin() + qa, p.lvl_nodes.begin() + qb);
      continue;
    }
    nodes.assign(p.lvl_nodes.begin() + qa, p.lvl_nodes.begin() + qb);
    std::sort(nodes.begin(), nodes.end());
    size_t nop = 0;
    for (int j : nodes)
      for (int r = p.Rp[j]; r < p.Rp[j + 1]; ++r) nop += p.Lp[p.Rk[r] + 1] - p.Rpos[r];
    if (lev.size() < nop) lev.resize(nop);
    segs.clear();
    target.clear();
    int f = 0;
    for (int j : nodes) {
      if (p.Rp[j + 1] > p.Rp[j]) {
        segs.push_back(f);
        target.push_back(j);
      }
      for (int r = p.Rp[j]; r < p.Rp[j + 1]; ++r) {
        const uint16_t e = (uint16_t)(N + p.Rpos[r]);
        lev[f++] = {e, e, (uint16_t)p.Rk[r]};
      }
    }
    for (int j : nodes) {
      if (p.Rp[j + 1] == p.Rp[j]) continue;
      const int q0 = p.Lp[j], len = p.Lp[j + 1] - q0;
      cnt.assign(len + 1, 0);
      for (int q = q0; q < q0 + len; ++q) {
        rowpos[p.Li[q]] = q - q0;
        rowmark[p.Li[q]] = j;
      }
      for (int r = p.Rp[j]; r < p.Rp[j + 1]; ++r) {
        const int k = p.Rk[r];
        for (int pp = p.Rpos[r] + 1; pp < p.Lp[k + 1]; ++pp) {
          if (rowmark[p.Li[pp]] != j) return false;  // fill outside the pattern
          cnt[rowpos[p.Li[pp]] + 1]++;
        }
      }
      for (int a = 0; a < len; ++a) {
        if (cnt[a + 1]) {
          segs.push_back(f + cnt[a]);
          target.push_back(N + q0 + a);
        }
        cnt[a + 1] += cnt[a];
      }
      const int total = cnt[len];
      for (int r = p.Rp[j]; r < p.Rp[j + 1]; ++r) {
        const int k = p.Rk[r], pjk = p.Rpos[r];
        for (int pp = pjk + 1; pp < p.Lp[k + 1]; ++pp)
          lev[f + cnt[rowpos[p.Li[pp]]]++] = {(uint16_t)(N + pp), (uint16_t)(N + pjk),
                                              (uint16_t)k};
      }
      f += total;
    }
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
    // split: every stream part starts a chunk; positions in the level are kept
    // by aligning each part's start to a chunk boundary of a common stream
    split.start();
    constexpr int chunk = 32 * kSlOpRun;
    int base[kSlWarps], at0 = 0;
    for (int w = 0; w < kSlWarps; ++w) {
      const int s0 = segs[sb[w]];
      base[w] = s0 - at0;  // stream position -> level position
      for (int g = sb[w]; g < sb[w + 1]; ++g)
        split.add(g, segs[g] - base[w], segs[g + 1] - base[w], kSlOpRun);
      at0 += (segs[sb[w + 1]] - s0 + chunk - 1) / chunk * chunk;
    }
    s.nopcarry = std::max(s.nopcarry, split.ncarry);
    if (zero + s.nopcarry >= 1 << kSlOpT.width || s.nopcarry >= 1 << kSlOpIni.width) return false;
    auto part_of = [&](int g) {
      int w = 0;
      while (g >= sb[w + 1]) ++w;
      return w;
    };
    for (int ph = 0; ph < split.nphase; ++ph) {
      const auto &parts = split.phase[ph];
      packer.pack(parts);
      int rank[kSlWarps];
      for (int w = 0; w < kSlWarps; ++w) rank[w] = w;
      std::stable_sort(rank, rank + kSlWarps,
                       [&](int a, int b) { return opg[a].size() < opg[b].size(); });
      page_of.resize(packer.npages);
      for (int i = 0; i < packer.npages; ++i) {
        auto &O = opg[rank[i % kSlWarps]];
        page_of[i] = (int)(O.size() / kSlOpWords);
        O.resize(O.size() + kSlOpWords);
        uint32_t *w = O.data() + (size_t)page_of[i] * kSlOpWords;
        for (int l2 = 0; l2 < kSlOpWords; l2 += 4) std::copy_n(padw, 4, w + l2);
      }
      page_reach.assign(packer.npages, 0);
      for (size_t i = 0; i < parts.size(); ++i) {
        const Part &q = parts[i];
        const int pgi = packer.at[i].first, l0 = packer.at[i].second;
        auto &O = opg[rank[pgi % kSlWarps]];
        uint32_t *e = O.data() + (size_t)page_of[pgi] * kSlOpWords;
        const int off = base[part_of(q.seg)];
        int t = q.first;
        const int end = q.first + q.len;
        for (int r = 0; r < q.lanes; ++r) {
          const Op &o0 = lev[t + off];
          const bool two = t % kSlOpRun == 0 && t + 1 < end;
          const Op o1 = two ? lev[t + 1 + off] : none(o0.k);
          t += two ? 2 : 1;
          const bool last = r == q.lanes - 1;
          const bool prev = last && !q.scan_last && r > 0;
          if (!prev) page_reach[pgi] = std::max(page_reach[pgi], r);
          const int to = !last ? zero : (q.more ? zero + 1 + q.carry_out : target[q.seg]);
          const int ini = r == 0 && q.carry_in >= 0 ? 1 + q.carry_in : 0;
          encode(e + 4 * (l0 + r), o0, o1, (uint32_t)to, (uint32_t)ini,
                 prev ? 32u : (uint32_t)r);
        }
      }
      for (int i = 0; i < packer.npages; ++i) {
        const uint32_t steps = (uint32_t)scan_steps(page_reach[i]) << 22;
        uint32_t *w = opg[rank[i % kSlWarps]].data() + (size_t)page_of[i] * kSlOpWords;
        for (int l2 = 0; steps && l2 < 32; ++l2) w[4 * l2 + 3] |= steps;
      }
      // the phase's end (the last one is the level's)
      ++s.olevels;
      for (int w = 0; w < kSlWarps; ++w) {
        if (opg[w].empty()) {
          ++oskip[w];
          continue;
        }
        uint32_t *e = opg[w].data() + opg[w].size() - kSlOpWords;
        if ((e[3] >> 25) == (uint32_t)kSlOpMaxWait) return false;
        for (int l2 = 0; l2 < 32; ++l2) e[4 * l2 + 3] += 1u << 25;
      }
    }
  }
  s.ops.clear();
  for (int w = 0; w < kSlWarps; ++w) {
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
