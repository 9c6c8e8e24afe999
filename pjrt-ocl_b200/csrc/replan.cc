// See replan.h.
#include "replan.h"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <set>

#include "loader.h"
#include "plan_format.h"

namespace b2 {

bool IsPlannedOp(uint32_t op) { return op >= kTopFuseRows && op <= kTopPlanLast; }

void PlannedLists(const VmProgram &p, const VmTask &t, const int32_t **reads, int *n_reads, const int32_t **writes, int *n_writes,
                  const int32_t **payload) {
  const int32_t *x = &p.aux[t.p2];
  *n_reads = x[0];
  *n_writes = x[1];
  *reads = x + 2;
  *writes = x + 2 + x[0];
  *payload = x + 2 + x[0] + x[1];
}

namespace {

float BitsF(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }
int32_t FBits(float f) { int32_t i; std::memcpy(&i, &f, 4); return i; }
bool IsFloatDt(uint32_t dt) { return dt == kF32 || dt == kF16 || dt == kBF16; }
bool Half(uint32_t dt) { return dt == kF16 || dt == kBF16; }
bool BinSub(uint32_t s) { return s <= kPow || s == kAtan2 || s == kRemainder; }

struct Step { uint32_t code = 0, dt = 0; float s = 0, t = 0; int64_t id = -1; uint32_t reg = 0; };

struct Node {
  VmTask t{};
  uint32_t op = 0, dt = 0, adt = 0;
  int region = 0;            // 0 root before the loop, 1 its body, 2 root after it
  int phase = 0;             // the schedule's
  int order = 0;             // program order inside the whole walk
  uint32_t tiles = 0;
  double cost = 1.0;         // of one tile, relative
  bool planned = false;      // one of this file's own ops
  std::vector<uint32_t> rd, wr;
  std::vector<int32_t> payload;
  std::vector<int> members;  // of a planned op: the tasks it is made of
  int carry_slot = -1;       // full sum counter it uses
  bool by_slot = false;      // entries name {lane slot, slots} instead of a tile range (matmuls)
  size_t owner_word = 0;     // payload word that takes the number of owner lanes (carry_slot >= 0)
};

struct View { bool ok = false; DView v; };

class Planner {
 public:
  Planner(const VmProgram &p, uint32_t lanes) : p_(p), L_(lanes) {}
  bool Run(VmProgram *q, ReplanStats *st);

 private:
  struct Chain;
  const VmProgram &p_;
  const uint32_t L_;
  std::vector<Node> n_;                      // original tasks in program order, then planned ops
  std::vector<std::set<int>> pred_;          // original data dependences,
  std::vector<std::vector<int>> succ_;       // ... the other way
  std::vector<int> rep_;                     // node -> the node it is now part of
  int n_orig_ = 0;
  int loop_trip_ = -1;
  bool has_loop_ = false;
  std::set<uint32_t> in_, out_, const_, written_;
  std::map<uint32_t, std::vector<int>> defs_, uses_;   // by original nodes

  bool Extract();
  bool TaskTiles(const VmTask &t, uint32_t *tiles) const;
  int PhasesMerged(const Chain &c) const;
  double MoveCost(const Node &nd) const;
  void Lists(const VmTask &t, std::vector<uint32_t> *rd, std::vector<uint32_t> *wr) const;
  void Dependences();
  bool Cyclic(int id) const;
  uint64_t Count(uint32_t id) const { return p_.buffers[id].bytes / DtypeSize(p_.buffers[id].dtype); }
  uint32_t Dt(uint32_t id) const { return p_.buffers[id].dtype; }
  bool Pinned(uint32_t id) const { return in_.count(id) || out_.count(id) || const_.count(id); }
  int Def(uint32_t id) const {               // its only writer, if it is an ordinary intermediate or result
    auto it = defs_.find(id);
    return it == defs_.end() || it->second.size() != 1 || in_.count(id) || const_.count(id) ? -1 : it->second[0];
  }
  const std::vector<int> &Uses(uint32_t id) const {
    static const std::vector<int> none;
    auto it = uses_.find(id);
    return it == uses_.end() ? none : it->second;
  }
  bool Free(int i) const { return rep_[i] == i && !n_[i].planned; }      // still a task of its own
  View ViewAt(uint32_t field) const {
    View r;
    if (!field || field - 1 >= p_.aux.size()) return r;
    const int32_t *x = &p_.aux[field - 1];
    r.ok = CollapseView(x + 1, x + 1 + x[0], x[0], x[1 + 2 * x[0]], &r.v);
    return r;
  }
  int AddPlanned(Node nd, const std::vector<int> &members);

  bool FusePairs(int seed);
  bool FuseGemm(int seed);
  void SgShape(uint32_t op, uint64_t M, uint64_t N, uint64_t K, uint32_t lanes, int *shape, uint32_t *tiles, double *cost) const;
  bool GemmEpilogue(const Chain &c, uint32_t dst, std::vector<int32_t> *w) const;
  void GroupGemms(std::vector<int> *live, std::map<std::pair<int, int>, std::vector<int>> *phases, std::vector<std::vector<int>> *of);
  void NormIntoProducts(std::vector<int> *live, std::vector<std::set<int>> *pred);
  bool FuseRows(int seed);
  bool FuseFlat(int seed);
  Node RowsNode(const Chain &c, uint32_t start, const std::vector<uint32_t> &writes, uint64_t R, uint64_t C, uint64_t n) const;
  bool Assemble(VmProgram *q, ReplanStats *st);
};

bool Planner::TaskTiles(const VmTask &t, uint32_t *tiles) const {
  auto div = [](uint64_t a, uint64_t b) { return static_cast<uint32_t>((a + b - 1) / b); };
  switch (t.tile_op & 0xFFu) {
    case kTopEw: case kTopMapRegion: case kTopGather: case kTopScatter: case kTopDynGather: case kTopDynScatter: case kTopIotaDim:
      *tiles = div(t.p1, kEwTs); return t.p1 > 0;
    case kTopMma: *tiles = std::max(1u, t.p3) * div(t.p0, kMmaT) * div(t.p1, kMmaT); return *tiles > 0;
    case kTopRedPart: if (!t.p1) return false; *tiles = div(t.p0, t.p1); return true;
    case kTopRedComb: *tiles = 1; return true;
    case kTopRedSeg: case kTopSoftmaxSeg: case kTopLayernormSeg: *tiles = t.p0; return t.p0 > 0;
    case kTopRedStrided: *tiles = div(t.p0, kEwTs); return t.p0 > 0;
    case kTopFlashAttn: *tiles = t.p1 * t.p2; return *tiles > 0;
    default: return false;      // window / index / convolution ops: programs with them keep their schedule
  }
}

// A tile of a move by its bytes: 23 per cycle is a lane's share of the copy rate; runs that are not contiguous at the far side
// come at about a quarter of it. (A contiguous 16-bit tile is 0.12 of the unit; taken for 1.5, the copies of a decode step's
// caches left all 96 tiles of the products beside them to one lane: 2.18 ms, 1.22 ms now.)
double Planner::MoveCost(const Node &nd) const {
  const double cycles = 2.0 * kEwTs * static_cast<double>(DtypeSize(nd.dt)) / 23.0;
  bool runs = true;
  if (nd.op == kTopGather) {
    const View v = ViewAt(nd.t.p0 + 1);
    runs = v.ok && v.v.rank > 0 && v.v.stride[v.v.rank - 1] == 1;
  }
  return cycles * (runs ? 1.0 : 4.0) / 6000.0;
}

void Planner::Lists(const VmTask &t, std::vector<uint32_t> *rd, std::vector<uint32_t> *wr) const {
  const uint32_t op = t.tile_op & 0xFFu;
  wr->push_back(t.dst);
  switch (op) {
    case kTopEw: {
      const uint32_t s = t.p0;
      if (!(s == kFill || s == kIotaFlat)) rd->push_back(t.a);
      if (BinSub(s) || s == kCmp || s == kSelect || s == kLts || (s >= kAnd && s <= kXor) || (s >= kShl && s <= kShrA)) rd->push_back(t.b);
      if (s == kSelect) rd->push_back(t.p3);
      if (s == kLts) rd->push_back(t.dst);
      break;
    }
    case kTopMma:
      rd->push_back(t.a); rd->push_back(t.b);
      if (t.p6) rd->push_back(t.p7);
      break;
    case kTopRedSeg:
      rd->push_back(t.a);
      if (t.p3) rd->push_back(t.b);
      break;
    case kTopMapRegion: {
      const uint32_t ids[8] = {t.a, t.b, t.p2, t.p3, t.p4, t.p5, t.p6, t.p7};
      const uint32_t n_in = t.p0 < p_.aux.size() ? static_cast<uint32_t>(p_.aux[t.p0]) : 8u;
      for (uint32_t k = 0; k < std::min(8u, n_in); ++k) rd->push_back(ids[k]);
      break;
    }
    case kTopFlashAttn: rd->push_back(t.a); rd->push_back(t.b); rd->push_back(t.p0); break;
    case kTopDynGather: case kTopDynScatter: {
      rd->push_back(t.a);
      const int32_t rank = p_.aux[t.p0];
      for (int32_t d = 0; d < rank; ++d) rd->push_back(static_cast<uint32_t>(p_.aux[t.p0 + 1 + 4 * rank + d]));
      if (op == kTopDynScatter) rd->push_back(t.dst);
      break;
    }
    case kTopScatter: rd->push_back(t.a); rd->push_back(t.dst); break;
    case kTopIotaDim: break;
    default: rd->push_back(t.a); break;
  }
}

// The task graph out of the lanes' streams. Refuses anything but a root walk with at most one counted loop whose
// tasks each run once per pass, in one phase, over exactly their own tiles.
bool Planner::Extract() {
  const uint32_t lanes = static_cast<uint32_t>(p_.lane_tab.size());
  struct Place { int region = -1, phase = -1; std::vector<std::pair<uint32_t, uint32_t>> ranges; };
  std::vector<Place> at(p_.tasks.size());
  std::map<std::pair<int, int>, std::vector<uint32_t>> order;         // (region, phase) -> tasks
  std::map<std::pair<int, int>, std::set<std::vector<uint32_t>>> seqs;  // ... and the orders that lanes run several of them in
  for (uint32_t l = 0; l < lanes; ++l) {
    const VmLane &ln = p_.lane_tab[l];
    std::vector<uint32_t> seq;                                          // this lane's tasks of the phase
    std::pair<int, int> seq_at{0, 0};
    auto close = [&] {
      if (seq.size() > 1) seqs[seq_at].insert(seq);
      seq.clear();
    };
    auto tile = [&](const VmEntry &e, int region, int phase) {
      if (e.task >= p_.tasks.size()) return false;
      if ((e.wait_flag != 0xFFFFFFFFu && e.wait_flag) || e.wait_count || (e.signal_flag != 0xFFFFFFFFu && e.signal_flag)) return false;
      Place &pl = at[e.task];
      if (pl.region < 0) {
        pl.region = region; pl.phase = phase;
        order[{region, phase}].push_back(e.task);
      }
      if (pl.region != region || pl.phase != phase) return false;
      if (seq_at != std::make_pair(region, phase)) { close(); seq_at = {region, phase}; }
      if (std::find(seq.begin(), seq.end(), e.task) == seq.end()) seq.push_back(e.task);       // (a lane may hold several pieces of a task)
      if (e.tile_hi > e.tile_lo) pl.ranges.push_back({e.tile_lo, e.tile_hi});
      return true;
    };
    int region = 0, phase = 0, trip = -1;
    uint32_t covered = ln.root_len;
    for (uint32_t i = 0; i < ln.root_len; ++i) {
      const VmEntry &e = p_.entries[ln.off + i];
      if (e.task == kEntNop) continue;
      if (e.task == kEntBarrier) { ++phase; continue; }
      if (e.task == kEntWhile || e.task == kEntIf) return false;
      if (e.task == kEntFor) {
        if (trip >= 0 || e.wait_flag == 0u || e.wait_flag > 0x7fffffffu || e.tile_lo != ln.root_len) return false;
        trip = static_cast<int>(e.wait_flag);
        int bp = 0;
        for (uint32_t k = e.tile_lo; k < e.tile_lo + e.tile_hi; ++k) {
          const VmEntry &b = p_.entries[ln.off + k];
          if (b.task == kEntNop) continue;
          if (b.task == kEntBarrier) { ++bp; continue; }
          if (b.task >= p_.tasks.size() || !tile(b, 1, bp)) return false;
        }
        covered += e.tile_hi;
        region = 2;
        ++phase;
        continue;
      }
      if (!tile(e, region, phase)) return false;
    }
    if (covered != ln.count) return false;
    close();
    if (l == 0) { loop_trip_ = trip; has_loop_ = trip >= 0; }
    else if (trip != loop_trip_) return false;
  }
  int seq = 0;
  // Inside a phase only tasks of one lane's chain may touch the same buffer: those keep the lane's order.
  for (auto &kv : order) {
    auto &ts = kv.second;
    std::sort(ts.begin(), ts.end());
    std::set<std::pair<uint32_t, uint32_t>> bf;          // which ran before which on some lane
    const auto sq = seqs.find(kv.first);
    if (sq != seqs.end())
      for (const auto &v : sq->second)
        for (size_t i = 0; i < v.size(); ++i)
          for (size_t j = i + 1; j < v.size(); ++j) bf.insert({v[i], v[j]});
    std::vector<std::vector<uint32_t>> rd(ts.size()), wr(ts.size());
    for (size_t i = 0; i < ts.size(); ++i) Lists(p_.tasks[ts[i]], &rd[i], &wr[i]);
    auto meet = [](const std::vector<uint32_t> &a, const std::vector<uint32_t> &b) {
      for (uint32_t x : a) if (std::find(b.begin(), b.end(), x) != b.end()) return true;
      return false;
    };
    std::vector<std::set<size_t>> pre(ts.size());
    for (size_t i = 0; i < ts.size(); ++i)
      for (size_t j = 0; j < ts.size(); ++j) {
        if (i == j || !(meet(wr[i], wr[j]) || meet(wr[i], rd[j]) || meet(rd[i], wr[j]))) continue;
        const bool ij = bf.count({ts[i], ts[j]}) != 0, ji = bf.count({ts[j], ts[i]}) != 0;
        if (ij && ji) return false;
        if (ij) pre[j].insert(i);
        if (!ij && !ji && (meet(wr[i], rd[j]) || meet(rd[i], wr[j]))) return false;     // on different lanes, unordered
      }
    std::vector<uint32_t> done;
    std::set<size_t> placed;
    while (placed.size() < ts.size()) {
      const size_t had = placed.size();
      for (size_t i = 0; i < ts.size(); ++i) {
        bool ready = !placed.count(i);
        for (size_t k : pre[i]) ready = ready && placed.count(k) != 0;
        if (ready) { placed.insert(i); done.push_back(ts[i]); }
      }
      if (placed.size() == had) return false;
    }
    ts = done;
  }
  for (const auto &kv : order)                        // regions, then phases, ascending
    for (uint32_t ti : kv.second) {
      Node nd;
      nd.t = p_.tasks[ti];
      nd.op = nd.t.tile_op & 0xFFu;
      nd.dt = (nd.t.tile_op >> 8) & 0xFFu;
      nd.adt = (nd.t.tile_op >> 16) & 0xFFu;
      nd.region = kv.first.first;
      nd.phase = kv.first.second;
      nd.order = seq++;
      if (!TaskTiles(nd.t, &nd.tiles)) return false;
      auto &r = at[ti].ranges;
      std::sort(r.begin(), r.end());
      uint32_t pos = 0;
      for (auto &x : r) { if (x.first != pos) return false; pos = x.second; }
      if (pos != nd.tiles) return false;
      Lists(nd.t, &nd.rd, &nd.wr);
      switch (nd.op) {
        case kTopMma: nd.cost = 20.0; break;
        case kTopGather: case kTopScatter: case kTopDynGather: case kTopDynScatter: nd.cost = MoveCost(nd); break;
        case kTopRedSeg: case kTopSoftmaxSeg: case kTopLayernormSeg: nd.cost = std::max(0.02, nd.t.p1 / 4096.0); break;
        case kTopRedPart: nd.cost = nd.t.p1 / 4096.0; break;
        case kTopFlashAttn: nd.cost = 0.5; break;
        case kTopMapRegion: nd.cost = 3.0; break;
        default: break;
      }
      n_.push_back(nd);
    }
  n_orig_ = static_cast<int>(n_.size());
  for (const VmTask &t : p_.tasks) written_.insert(t.dst);
  in_.insert(p_.args.ids.begin(), p_.args.ids.end());
  out_.insert(p_.results.ids.begin(), p_.results.ids.end());
  for (const auto &k : p_.consts) const_.insert(k.buffer);
  for (int i = 0; i < n_orig_; ++i) {
    for (uint32_t b : n_[i].wr) defs_[b].push_back(i);
    std::set<uint32_t> once(n_[i].rd.begin(), n_[i].rd.end());
    for (uint32_t b : once) uses_[b].push_back(i);
    rep_.push_back(i);
  }
  Dependences();
  return n_orig_ > 0;
}

void Planner::Dependences() {
  pred_.assign(n_orig_, {});
  std::map<uint32_t, std::vector<int>> writers, readers;
  for (int i = 0; i < n_orig_; ++i) {
    if (i && n_[i].region != n_[i - 1].region) { writers.clear(); readers.clear(); }      // a barrier separates the regions
    for (uint32_t b : n_[i].rd) for (int w : writers[b]) if (w != i) pred_[i].insert(w);
    for (uint32_t b : n_[i].wr) {
      for (int w : writers[b]) if (w != i) pred_[i].insert(w);
      for (int r : readers[b]) if (r != i) pred_[i].insert(r);
    }
    for (uint32_t b : n_[i].wr) writers[b].push_back(i);
    for (uint32_t b : n_[i].rd) readers[b].push_back(i);
  }
  succ_.assign(n_orig_, {});
  for (int i = 0; i < n_orig_; ++i) for (int j : pred_[i]) succ_[j].push_back(i);
}

// Does anything that node `id` is made of need something that needs the node? (Without it the graph had no cycle.)
bool Planner::Cyclic(int id) const {
  std::vector<char> seen(n_.size(), 0);
  std::vector<int> todo{id};
  while (!todo.empty()) {
    const int g = todo.back();
    todo.pop_back();
    const std::vector<int> own{g};
    for (int m : n_[g].planned ? n_[g].members : own)
      for (int k : succ_[m]) {
        const int r = rep_[k];
        if (r == id && g != id) return true;
        if (r != id && !seen[r]) { seen[r] = 1; todo.push_back(r); }
      }
  }
  return false;
}

// Members become part of the new node, unless that would need something that needs the node itself.
int Planner::AddPlanned(Node nd, const std::vector<int> &members) {
  nd.planned = true;
  nd.region = n_[members[0]].region;
  nd.order = n_[members[0]].order;
  for (int m : members) { if (n_[m].region != nd.region) return -1; nd.order = std::max(nd.order, n_[m].order); }
  const int id = static_cast<int>(n_.size());
  nd.members = members;
  n_.push_back(nd);
  rep_.push_back(id);
  for (int m : members) rep_[m] = id;
  if (!Cyclic(id)) return id;
  for (int m : members) rep_[m] = m;
  rep_.pop_back();
  n_.pop_back();
  return -1;
}

// sum_j m_j (|x_j - x_i|^2 s + t)^-1.5 (x_j - x_i), found from its strided sum backwards:
//   out = RED_STRIDED(d * w[., ., broadcast]); d = x[j] - x[i] (views, or gathers of carried positions);
//   w = POW(AFFINE(RED_SEG(d * d)), -1.5) * m[j]
bool Planner::FusePairs(int seed) {
  const Node sum = n_[seed];
  const int64_t n = sum.t.p1;
  if (sum.dt != kF32 || sum.adt != kF32 || sum.t.p2 != 3 || sum.t.p3 != kSum || n < 2 || sum.t.p0 != 3 * n || n > (1 << 14)) return false;
  std::vector<int> members{seed};
  auto ew = [&](uint32_t id, uint32_t sub, int64_t count) -> int {         // the free elementwise task that makes `id`
    const int i = Def(id);
    if (i < 0 || !Free(i) || n_[i].op != kTopEw || n_[i].t.p0 != sub || n_[i].dt != kF32 || n_[i].adt != kF32 || n_[i].t.p1 != count) return -1;
    return i;
  };
  auto only = [&](uint32_t id, std::set<int> want) {
    if (Pinned(id)) return false;
    const auto &u = Uses(id);
    return std::set<int>(u.begin(), u.end()) == want;
  };
  auto view_is = [&](uint32_t field, std::vector<std::pair<int64_t, int64_t>> want) {   // (dim, stride), outermost first
    const View v = ViewAt(field);
    if (!v.ok || v.v.off != 0 || v.v.rank != static_cast<int>(want.size())) return false;
    for (size_t k = 0; k < want.size(); ++k)
      if (v.v.dim[k] != want[k].first || v.v.stride[k] != want[k].second) return false;
    return true;
  };
  const int fi = ew(sum.t.a, kMul, 3 * n * n);
  if (fi < 0 || !only(sum.t.a, {seed})) return false;
  members.push_back(fi);
  const VmTask &f = n_[fi].t;
  if (f.p2 || !view_is(f.p3, {{n * n, 1}, {3, 0}})) return false;
  const uint32_t d = f.a, w = f.b;
  const int di = ew(d, kSubt, 3 * n * n), wi = ew(w, kMul, n * n);
  if (di < 0 || wi < 0 || !only(w, {fi})) return false;
  // d: both operands the same positions
  const VmTask &dt = n_[di].t;
  uint32_t pos;
  const std::vector<std::pair<int64_t, int64_t>> vj{{n, 0}, {3 * n, 1}}, vi{{n, 3}, {n, 0}, {3, 1}};
  if (dt.p2 || dt.p3) {
    if (dt.a != dt.b || !view_is(dt.p2, vj) || !view_is(dt.p3, vi)) return false;
    pos = dt.a;
  } else {
    const int ga = Def(dt.a), gb = Def(dt.b);
    if (ga < 0 || gb < 0 || !Free(ga) || !Free(gb) || n_[ga].op != kTopGather || n_[gb].op != kTopGather) return false;
    if (n_[ga].t.a != n_[gb].t.a || !view_is(n_[ga].t.p0 + 1, vj) || !view_is(n_[gb].t.p0 + 1, vi)) return false;
    if (!only(dt.a, {di}) || !only(dt.b, {di}) || n_[ga].dt != kF32 || n_[gb].dt != kF32) return false;
    pos = n_[ga].t.a;
    members.push_back(ga);
    members.push_back(gb);
  }
  members.push_back(di);
  // w = pow * m[j]
  const VmTask &wt = n_[wi].t;
  if (wt.p2 || !view_is(wt.p3, {{n, 0}, {n, 1}})) return false;
  members.push_back(wi);
  const uint32_t mass = wt.b;
  const int pi = ew(wt.a, kPow, n * n);
  if (pi < 0 || !only(wt.a, {wi}) || n_[pi].t.p2 || !view_is(n_[pi].t.p3, {{n * n, 0}})) return false;
  members.push_back(pi);
  const VmTask &pt = n_[pi].t;
  bool expo = false;
  for (const auto &k : p_.consts)
    if (k.buffer == pt.b && k.data.size() >= 4 && !written_.count(pt.b)) { uint32_t u; std::memcpy(&u, k.data.data(), 4); expo = BitsF(u) == -1.5f; }
  if (!expo) return false;
  float s = 1.0f, t = 0.0f;
  uint32_t r2 = pt.a;
  int user = pi;
  const int ai = ew(r2, kAffine, n * n);
  if (ai >= 0) {
    if (!only(r2, {pi})) return false;
    s = BitsF(n_[ai].t.p2); t = BitsF(n_[ai].t.p3);
    r2 = n_[ai].t.a;
    user = ai;
    members.push_back(ai);
  }
  if (!(s > 0.0f) || !(t >= 0.0f)) return false;
  const int ri = Def(r2);
  if (ri < 0 || !Free(ri) || n_[ri].op != kTopRedSeg || n_[ri].t.p3 || n_[ri].t.p2 != kSum || n_[ri].t.p1 != 3 || n_[ri].t.p0 != n * n ||
      n_[ri].dt != kF32 || n_[ri].adt != kF32 || !only(r2, {user}))
    return false;
  members.push_back(ri);
  const int qi = ew(n_[ri].t.a, kMul, 3 * n * n);
  if (qi < 0 || n_[qi].t.p2 || n_[qi].t.p3 || n_[qi].t.a != d || n_[qi].t.b != d || !only(n_[ri].t.a, {ri}) || !only(d, {qi, fi})) return false;
  members.push_back(qi);
  for (int m : members) if (!Free(m) || n_[m].region != sum.region) return false;
  if (Dt(pos) != kF32 || Dt(mass) != kF32 || Count(pos) < static_cast<uint64_t>(3 * n) || Count(mass) < static_cast<uint64_t>(n) ||
      Dt(sum.t.dst) != kF32)
    return false;

  Node nd;
  nd.op = kTopPairs; nd.dt = nd.adt = kF32;
  nd.t = VmTask{};
  nd.t.dst = sum.t.dst; nd.t.a = pos;
  nd.tiles = static_cast<uint32_t>(n);
  nd.cost = 0.33 * static_cast<double>(n) / 4096.0;
  const std::set<int> core(members.begin(), members.end());
  std::set<int> in_group = core;
  auto depends = [&](int i) {        // does i need anything of the group (through tasks outside it too)?
    std::vector<int> todo{i};
    std::set<int> seen;
    while (!todo.empty()) {
      const int k = todo.back();
      todo.pop_back();
      for (int j : pred_[k]) {
        if (in_group.count(j)) return true;
        if (seen.insert(j).second) todo.push_back(j);
      }
    }
    return false;
  };
  // Depth of a task: the last evaluation (strided sum, in program order) that it needs. The tail takes what follows
  // from this evaluation and earlier ones, and what only later evaluations' tails want: left alone those would be
  // phases of their own, each dearer than what running two evaluations side by side could save.
  std::vector<int> depth(n_orig_, 0);
  for (int i = 0; i < n_orig_; ++i) {
    for (int j : pred_[i]) depth[i] = std::max(depth[i], depth[j]);
    if (n_[i].op == kTopRedStrided) depth[i] = i + 1;
  }
  auto tail_op = [&](int i) {
    const Node &e = n_[i];
    if (e.region != sum.region || !Free(i) || e.op != kTopEw || e.dt != kF32 || e.adt != kF32 || e.t.p1 != 3 * n) return false;
    const uint32_t sub = e.t.p0;
    const bool bin = sub == kAdd || sub == kSubt || sub == kMul;
    return (bin || sub == kAffine || sub == kCopy) && (sub == kAffine || !(e.t.p2 || e.t.p3));
  };
  // Tasks that need no evaluation and that only other evaluations want, where they read their positions: side by side with this
  // one they would be an op of their own on a few lanes, for which the others wait (8 us of the 88 of a Runge-Kutta step).
  // Only for an evaluation that has nothing to wait for, and so runs in the phase that these would run in: another's positions
  // stand in a phase before it, together, and evaluations that are independent of each other stay so.
  std::set<int> early;
  bool first = true;
  for (int m : core) for (int j : pred_[m]) first = first && core.count(j);
  for (int i = 0; first && i < n_orig_; ++i)
    if (tail_op(i) && depth[i] == 0 && Def(n_[i].t.dst) == i && !out_.count(n_[i].t.dst) && n_[i].t.dst != pos && n_[i].t.dst != mass && !Uses(n_[i].t.dst).empty()) early.insert(i);
  for (bool changed = true; changed;) {
    changed = false;
    for (auto it = early.begin(); it != early.end();) {
      bool keep = true;
      for (int u : Uses(n_[*it].t.dst))
        keep = keep && !core.count(u) && (early.count(u) || (n_[u].region == sum.region && (n_[u].op == kTopEw || n_[u].op == kTopGather) && n_[u].t.p1 == 3 * n * n));
      for (int j : pred_[*it]) keep = keep && early.count(j);
      for (int u : succ_[*it]) keep = keep && !core.count(u);
      if (keep) ++it;
      else { it = early.erase(it); changed = true; }
    }
  }
  // With the early tasks, if the tail has room for them beside its own and nothing of the group then waits for the group.
  for (int with_early = early.empty() ? 0 : 1; with_early >= 0; --with_early) {
    // The elementwise tasks on the n x 3 result that need nothing from elsewhere after this evaluation.
    members.assign(core.begin(), core.end());
    in_group = core;
    std::vector<int32_t> tail;
    int n_tail = 0;
    bool room = true;
    std::map<uint32_t, int32_t> made{{sum.t.dst, 1}};      // buffer -> where the tail finds its value (plan_format.h: DPairTail)
    nd.rd = {pos, mass};
    nd.wr = {sum.t.dst};
    for (int i = 0; i < n_orig_; ++i) {
      const Node &e = n_[i];
      if (!tail_op(i)) continue;
      const uint32_t sub = e.t.p0;
      const bool bin = sub == kAdd || sub == kSubt || sub == kMul;
      bool mine = false, foreign = false;
      for (int j : pred_[i]) {
        if (in_group.count(j)) mine = true;
        else if (depends(j) || depth[j] >= depth[seed]) foreign = true;
      }
      if (!mine && !foreign && depth[i] >= 1 && depth[i] < depth[seed]) {
        mine = !Uses(e.t.dst).empty();
        for (int u : Uses(e.t.dst)) if (!in_group.count(u) && depth[u] <= depth[seed]) mine = false;
      }
      if (with_early && early.count(i)) { mine = true; foreign = false; }
      if (!mine || foreign || e.t.dst == pos || e.t.dst == mass) continue;     // other lanes may still read those
      if (n_tail == kPairTailMax) { room = false; break; }
      // rows of the operands are this lane's own only when they come from the group or from before it
      auto src = [&](uint32_t b) { auto it = made.find(b); return it == made.end() ? 0 : it->second; };
      tail.insert(tail.end(), {static_cast<int32_t>(sub), src(e.t.a), bin ? src(e.t.b) : 0, static_cast<int32_t>(sub == kAffine ? e.t.p2 : 0u),
                               static_cast<int32_t>(sub == kAffine ? e.t.p3 : 0u), static_cast<int32_t>(e.t.dst), static_cast<int32_t>(e.t.a),
                               static_cast<int32_t>(bin ? e.t.b : e.t.a)});
      ++n_tail;
      for (uint32_t b : e.rd) if (!made.count(b)) nd.rd.push_back(b);
      nd.wr.push_back(e.t.dst);
      made[e.t.dst] = 1 + n_tail;
      members.push_back(i);
      in_group.insert(i);
    }
    if (with_early && !room) continue;
    nd.payload = {static_cast<int32_t>(n), FBits(s), FBits(t), static_cast<int32_t>(pos), static_cast<int32_t>(mass),
                  static_cast<int32_t>(sum.t.dst), n_tail};
    nd.payload.insert(nd.payload.end(), tail.begin(), tail.end());
    if (AddPlanned(nd, members) >= 0) return true;
  }
  return false;
}

// A value carried through a list of steps. The builder starts from a value in X and follows it forward: reductions of
// it, then the one elementwise task that takes it on, and so on; whatever else reads a value on the way gets it stored.
struct Planner::Chain {
  Planner &P;
  const uint64_t R, C;
  const bool rows;                       // row reductions and row scalars allowed (else: a store epilogue)
  std::vector<Step> steps;
  std::vector<int> members;
  std::set<int> in;
  std::vector<uint32_t> reads;
  struct Kept { size_t at; uint32_t id; };
  std::vector<Kept> values;              // value `id` is in X just before step `at`
  std::set<int> path;                    // tasks to prefer where a value has several readers
  std::map<uint32_t, uint32_t> scalars;  // [R] buffer -> row scalar register
  int total = -1;                        // buffer of the full sum, if any
  uint32_t cur = 0;
  int n_norms = 0, n_work = 0, n_through = 0;
  int limit = 1 << 30;                   // elementwise tasks to go through at most

  Chain(Planner &p, uint64_t r, uint64_t c, bool rw) : P(p), R(r), C(c), rows(rw) {}

  void Take(int i) { members.push_back(i); in.insert(i); }
  bool Open(int i) const { return i >= 0 && i < P.n_orig_ && P.Free(i) && !in.count(i); }
  void Emit(uint32_t code, int64_t id = -1, uint32_t dt = 0, float s = 0, float t = 0, uint32_t reg = 0) {
    Step st;
    st.code = code; st.id = id; st.dt = dt; st.s = s; st.t = t; st.reg = reg;
    steps.push_back(st);
    if (id >= 0 && code != kFuStore) reads.push_back(static_cast<uint32_t>(id));
  }
  bool SoleUse(uint32_t id, int user) const {
    if (P.Pinned(id) || P.Def(id) < 0) return false;
    for (int u : P.Uses(id)) if (u != user) return false;
    return true;
  }
  // Storage type for a load or store step: 32-bit integers move as they are.
  static uint32_t MoveDt(uint32_t dt) { return dt == kI32 || dt == kU32 ? static_cast<uint32_t>(kF32) : dt; }
  static bool IsInt(uint32_t dt) { return dt == kI32 || dt == kU32; }
  // what a view makes of a buffer over the R x C elements
  enum Kind { kBad, kDense, kRowVec, kColVec, kScalar };
  Kind ViewKind(uint32_t field) const {
    if (!field) return kDense;
    const View v = P.ViewAt(field);
    if (!v.ok || v.v.off != 0) return kBad;
    const DView &d = v.v;
    if (d.rank == 0) return kScalar;
    if (d.rank == 1 && d.stride[0] == 0) return kScalar;
    if (d.rank == 1 && d.stride[0] == 1 && d.dim[0] == R * C) return kDense;
    if (d.rank == 2 && d.dim[0] == R && d.dim[1] == C && d.stride[0] == 0 && d.stride[1] == 1) return kRowVec;
    if (d.rank == 2 && d.dim[0] == R && d.dim[1] == C && d.stride[0] == 1 && d.stride[1] == 0) return kColVec;
    return kBad;
  }
  // the region d/dz tanh-GELU; *s takes its one free constant
  static bool IsGeluGrad(const VmProgram &p, const VmTask &t, float *s) {
    static const int32_t want[14][4] = {{kMul, 1, 0, 0}, {kMul, 2, 1, 0}, {kAffine, 3, 2, 2}, {kAdd, 2, 0, 3}, {kAffine, 3, 2, 2},
                                        {kTanh, 2, 3, 3}, {kMul, 3, 2, 2}, {kAffine, 4, 3, 3}, {kAffine, 3, 1, 1}, {kAffine, 1, 2, 2},
                                        {kAffine, 2, 0, 0}, {kMul, 0, 4, 3}, {kMul, 3, 2, 0}, {kAdd, 0, 1, 3}};
    const size_t x = t.p0;
    if (x + 4 + 6 * 14 > p.aux.size()) return false;
    const int32_t *a = &p.aux[x];
    if (a[0] != 1 || a[1] != 0 || a[2] != 14 || a[3] != 0) return false;
    auto is = [&](int m, float fs, float ft) { return BitsF(a[4 + 6 * m + 4]) == fs && BitsF(a[4 + 6 * m + 5]) == ft; };
    for (int m = 0; m < 14; ++m)
      for (int k = 0; k < 4; ++k)
        if (a[4 + 6 * m + k] != want[m][k]) return false;
    *s = BitsF(a[4 + 6 * 8 + 4]);
    return is(2, 0.044715f, 0.0f) && is(4, 0.7978845608f, 0.0f) && is(7, -1.0f, 1.0f) && BitsF(a[4 + 6 * 8 + 5]) == 0.7978845608f &&
           is(9, 0.5f, 0.5f) && is(10, 0.5f, 0.0f);
  }

  // Was what task `user` reads in buffer `id` made from a value of this chain?
  bool Needs(uint32_t id, int user) const {
    std::vector<int> todo;
    std::set<int> seen;
    for (int j : P.pred_[user])
      if (std::find(P.n_[j].wr.begin(), P.n_[j].wr.end(), id) != P.n_[j].wr.end()) todo.push_back(j);
    while (!todo.empty()) {
      const int k = todo.back();
      todo.pop_back();
      if (in.count(k)) return true;
      if (!seen.insert(k).second) continue;
      for (int j : P.pred_[k]) todo.push_back(j);
    }
    return false;
  }

  // Loads a second operand into Y, through a convert or a region of its own where only `user` wants the result.
  bool LoadY(uint32_t id, uint32_t field, int user) {
    const Kind k = ViewKind(field);
    if (k == kBad) return false;
    const uint64_t need = k == kDense ? R * C : k == kRowVec ? C : k == kColVec ? R : 1;
    std::vector<Step> post;
    std::vector<int> took;
    for (int depth = 0; depth < 3; ++depth) {
      const int d = P.Def(id);
      if (d < 0 || !Open(d) || !SoleUse(id, user) || P.n_[d].region != P.n_[user].region) break;
      const Node &nd = P.n_[d];
      if (nd.op == kTopEw && nd.t.p0 == kConvert && !nd.t.p2 && nd.t.p1 == need && IsFloatDt(nd.dt) && IsFloatDt(nd.adt)) {
        if (Half(nd.dt)) { Step q; q.code = kFuQuantY; q.dt = nd.dt; post.insert(post.begin(), q); }
      } else if (k == kDense && nd.op == kTopMapRegion && nd.t.p1 == need && nd.dt == kF32 && nd.adt == kF32) {
        Step g;
        if (!IsGeluGrad(P.p_, nd.t, &g.s)) break;
        g.code = kFuGeluGradY;
        post.insert(post.begin(), g);
      } else {
        break;
      }
      took.push_back(d);
      user = d;
      id = nd.t.a;
    }
    if (!(IsFloatDt(P.Dt(id)) || IsInt(P.Dt(id))) || P.Count(id) < need || Needs(id, user)) return false;
    for (int i : took) Take(i);
    Emit(k == kDense ? kFuLoadY : k == kRowVec ? kFuRowVecY : k == kColVec ? kFuColVecY : kFuScalarY, id, MoveDt(P.Dt(id)));
    for (const Step &q : post) steps.push_back(q);
    return true;
  }

  // Row reductions of `cur`, and the scalar work on their results.
  void Reductions() {
    for (int u : P.Uses(cur)) {
      if (!Open(u)) continue;
      const Node &nd = P.n_[u];
      int red = u, sq = -1, cv = -1;
      if (nd.op == kTopEw && nd.t.p0 == kMul && nd.t.a == cur && nd.t.b == cur && !nd.t.p2 && !nd.t.p3 && nd.dt == kF32 && nd.adt == kF32) {
        const auto &uu = P.Uses(nd.t.dst);
        if (uu.size() != 1 || !Open(uu[0]) || !SoleUse(nd.t.dst, uu[0])) continue;
        sq = u;
        red = uu[0];
      } else if (nd.op == kTopEw && nd.t.p0 == kConvert && nd.dt == kF32 && Half(nd.adt) && !nd.t.p2) {
        const auto &uu = P.Uses(nd.t.dst);
        if (uu.size() != 1 || !Open(uu[0]) || !SoleUse(nd.t.dst, uu[0]) || P.n_[uu[0]].op != kTopRedPart) continue;
        cv = u;
        red = uu[0];
      }
      const Node &r = P.n_[red];
      if (r.op == kTopRedPart) {           // the full sum: partial sums, then one combine
        if (total >= 0 || r.dt != kF32 || r.t.p2 != kSum || r.t.p0 != R * C || (sq < 0 && cv < 0 && P.Dt(cur) != kF32)) continue;
        const auto &cu = P.Uses(r.t.dst);
        if (cu.size() != 1 || !Open(cu[0]) || P.n_[cu[0]].op != kTopRedComb || !SoleUse(r.t.dst, cu[0]) || P.n_[cu[0]].t.p1 != kSum) continue;
        total = static_cast<int>(P.n_[cu[0]].t.dst);
        Emit(sq >= 0 ? kFuCarrySumSq : kFuCarrySum);
        Take(u);
        if (red != u) Take(red);
        Take(cu[0]);
        ++n_work;
        continue;
      }
      if (!rows || cv >= 0 || r.op != kTopRedSeg || r.t.p3 || r.t.p0 != R || r.t.p1 != C || r.dt != kF32 || r.adt != kF32 ||
          !(r.t.p2 == kSum || (r.t.p2 == kRMax && sq < 0)))
        continue;
      // a register whose scalar nothing reads any more
      uint32_t reg = 0;
      for (; reg < kFuScalars; ++reg) {
        bool used = false;
        for (const auto &kv : scalars) used = used || (kv.second == reg && Wanted(kv.first));
        if (!used) break;
      }
      if (reg == kFuScalars) continue;
      // the scalar tasks on it, to the one whose result the R x C elements read
      std::vector<Step> sc;
      std::vector<int> took;
      uint32_t id = r.t.dst;
      for (;;) {
        const auto &su = P.Uses(id);
        if (su.size() != 1 || !Open(su[0]) || P.Pinned(id)) break;
        const Node &q = P.n_[su[0]];
        Step s;
        s.reg = reg;
        if (q.op == kTopEw && q.t.p1 == R && q.dt == kF32 && q.adt == kF32 && q.t.p0 == kAffine) {
          s.code = kFuSAffine; s.s = BitsF(q.t.p2); s.t = BitsF(q.t.p3);
          sc.push_back(s);
        } else if (q.op == kTopEw && q.t.p1 == R && q.dt == kF32 && q.adt == kF32 && q.t.p0 == kRsqrt && !q.t.p2) {
          s.code = kFuSRsqrt;
          sc.push_back(s);
        } else if (q.op == kTopMapRegion && q.t.p1 == R && q.dt == kF32 && q.adt == kF32 && P.p_.aux[q.t.p0] == 1) {
          const int32_t *a = &P.p_.aux[q.t.p0];
          int slot = a[3];
          bool ok = true;
          for (int m = 0; m < a[2] && ok; ++m) {
            const int32_t *mo = a + 4 + 6 * m;
            Step x;
            x.reg = reg;
            if (mo[2] != slot) ok = false;
            else if (mo[0] == static_cast<int32_t>(kAffine)) { x.code = kFuSAffine; x.s = BitsF(mo[4]); x.t = BitsF(mo[5]); }
            else if (mo[0] == static_cast<int32_t>(kRsqrt)) x.code = kFuSRsqrt;
            else ok = false;
            if (ok) sc.push_back(x);
            slot = mo[1];
          }
          if (!ok || slot != a[1]) break;
        } else {
          break;
        }
        took.push_back(su[0]);
        id = q.t.dst;
      }
      // everything that reads the scalar has to be ours in the end: checked when the chain closes (Unread)
      if (P.Pinned(id) || P.Uses(id).empty()) continue;
      Emit(sq >= 0 ? kFuRedSumSq : r.t.p2 == kSum ? kFuRedSum : kFuRedMax, -1, 0, 0, 0, reg);
      for (const Step &s : sc) steps.push_back(s);
      Take(u);
      if (red != u) Take(red);
      for (int i : took) Take(i);
      scalars[id] = reg;
      ++n_work;
    }
  }

  // Takes the value through elementwise task `i`; false (nothing changed) where it has no steps.
  bool Through(int i) {
    const Node &nd = P.n_[i];
    const bool ints = IsInt(nd.dt) && nd.dt == nd.adt;
    if (!ints && (!IsFloatDt(nd.dt) || !IsFloatDt(nd.adt))) return false;
    const size_t keep = steps.size(), keep_m = members.size(), keep_r = reads.size();
    auto undo = [&] {
      steps.resize(keep);
      while (members.size() > keep_m) { in.erase(members.back()); members.pop_back(); }
      reads.resize(keep_r);
      return false;
    };
    bool exact = false;                 // the result needs no rounding of its own
    if (nd.op == kTopMapRegion) {
      const int32_t *a = &P.p_.aux[nd.t.p0];
      float s;
      if (nd.t.p1 != R * C || nd.dt != kF32 || nd.adt != kF32) return false;
      const uint32_t ids[8] = {nd.t.a, nd.t.b, nd.t.p2, nd.t.p3, nd.t.p4, nd.t.p5, nd.t.p6, nd.t.p7};
      if (IsGeluGrad(P.p_, nd.t, &s) && nd.t.a == cur) {
        Emit(kFuGeluGrad, -1, 0, s);
      } else if (a[0] == 2 && a[2] == 2) {
        // {affine of one input, a difference / sum / product with the other}: an update step
        const int32_t *m0 = a + 5, *m1 = a + 11;
        int mine = ids[0] == cur ? 0 : ids[1] == cur ? 1 : -1;
        if (mine < 0 || ids[0] == ids[1] || m0[0] != static_cast<int32_t>(kAffine) || m0[2] != a[3 + mine] || a[1] != m1[1]) return false;
        const int other = a[3 + (1 - mine)], res = m0[1];
        if (res == other) return false;
        const bool fwd = m1[2] == res && m1[3] == other, bwd = m1[2] == other && m1[3] == res;
        if (!fwd && !bwd) return false;
        uint32_t code;
        if (m1[0] == static_cast<int32_t>(kSubt)) code = fwd ? kFuSub : kFuRSub;
        else if (m1[0] == static_cast<int32_t>(kAdd)) code = kFuAdd;
        else if (m1[0] == static_cast<int32_t>(kMul)) code = kFuMul;
        else return false;
        Emit(kFuAffine, -1, 0, BitsF(m0[4]), BitsF(m0[5]));
        if (!LoadY(ids[1 - mine], 0, i)) return undo();
        Emit(code);
      } else {
        return false;
      }
      Take(i);
      return true;
    }
    if (nd.op != kTopEw || nd.t.p1 != R * C) return false;
    const uint32_t sub = nd.t.p0;
    auto unary = [&](uint32_t code) { Emit(code); };
    if (ints) {
      const bool a_cur = nd.t.a == cur && (!BinSub(sub) || ViewKind(nd.t.p2) == kDense), uns = nd.dt == kU32;
      uint32_t code;
      switch (sub) {
        case kAdd: code = kFuIAdd; break;
        case kMul: code = kFuIMul; break;
        case kSubt: code = a_cur ? kFuISub : kFuIRSub; break;
        case kAnd: code = kFuIAnd; break;
        case kOr: code = kFuIOr; break;
        case kXor: code = kFuIXor; break;
        case kMax: code = uns ? kFuUMax : kFuIMax; break;
        case kMin: code = uns ? kFuUMin : kFuIMin; break;
        case kNot: code = kFuINot; break;
        case kNeg: code = kFuINeg; break;
        case kCopy: code = kFuEnd; break;
        default: return false;
      }
      const bool two = BinSub(sub) || sub == kAnd || sub == kOr || sub == kXor;
      if (!two) {
        if (nd.t.a != cur || nd.t.p2) return false;
        if (code != kFuEnd) Emit(code);
      } else {
        const bool views = BinSub(sub);         // bitwise subops carry no views
        const bool b_cur = nd.t.b == cur && (!views || ViewKind(nd.t.p3) == kDense);
        if (a_cur && b_cur) Emit(kFuMovYX);
        else if (!(a_cur || b_cur) || !LoadY(a_cur ? nd.t.b : nd.t.a, !views ? 0u : a_cur ? nd.t.p3 : nd.t.p2, i)) return undo();
        Emit(code);
      }
      Take(i);
      return true;
    }
    if (sub == kAffine || !BinSub(sub)) {
      if (nd.t.a != cur || (sub != kAffine && nd.t.p2)) return false;
      switch (sub) {
        case kConvert: case kCopy: exact = !Half(nd.dt) || nd.dt == nd.adt; break;
        case kAffine: Emit(kFuAffine, -1, 0, BitsF(nd.t.p2), BitsF(nd.t.p3)); break;
        case kGelu: unary(kFuGelu); break;
        case kExp: unary(kFuExp); break;
        case kTanh: unary(kFuTanh); break;
        case kNeg: unary(kFuNeg); exact = true; break;
        case kAbs: unary(kFuAbs); exact = true; break;
        case kSqrt: unary(kFuSqrt); break;
        case kRsqrt: unary(kFuRsqrt); break;
        case kLog: unary(kFuLog); break;
        default: return false;
      }
    } else {
      if (nd.dt != nd.adt) return false;
      const bool a_cur = nd.t.a == cur && ViewKind(nd.t.p2) == kDense, b_cur = nd.t.b == cur && ViewKind(nd.t.p3) == kDense;
      uint32_t code, code_s = kFuEnd;
      switch (sub) {
        case kAdd: code = kFuAdd; code_s = kFuAddS; break;
        case kMul: code = kFuMul; code_s = kFuMulS; break;
        case kSubt: code = a_cur ? kFuSub : kFuRSub; if (a_cur) code_s = kFuSubS; break;
        case kDiv: code = a_cur ? kFuDiv : kFuRDiv; if (a_cur) code_s = kFuDivS; break;
        case kMax: code = kFuMax; exact = true; break;
        case kMin: code = kFuMin; exact = true; break;
        default: return false;
      }
      if (a_cur && b_cur) {
        Emit(kFuMovYX);
        Emit(code);
      } else if (a_cur || b_cur) {
        const uint32_t other = a_cur ? nd.t.b : nd.t.a, field = a_cur ? nd.t.p3 : nd.t.p2;
        auto it = scalars.find(other);
        if (it != scalars.end()) {
          const Kind kind = ViewKind(field);       // (of one row, a value per row is a scalar)
          if (!(kind == kColVec || (R == 1 && kind == kScalar)) || code_s == kFuEnd) return undo();
          Emit(code_s, -1, 0, 0, 0, it->second);
        } else {
          if (!LoadY(other, field, i)) return undo();
          Emit(code);
        }
      } else {
        return false;
      }
    }
    if (Half(nd.dt) && !exact) Emit(kFuQuant, -1, nd.dt);
    Take(i);
    return true;
  }

  bool Norm(int i) {
    const Node &nd = P.n_[i];
    if (!rows || nd.t.a != cur || nd.t.p0 != R || nd.t.p1 != C || !IsFloatDt(nd.dt) || nd.adt != P.Dt(cur)) return false;
    if (nd.op == kTopLayernormSeg) Emit(kFuLayerNorm, -1, 0, BitsF(nd.t.p2));
    else if (nd.op == kTopSoftmaxSeg) Emit(kFuSoftmax);
    else return false;
    if (Half(nd.dt)) Emit(kFuQuant, -1, nd.dt);
    Take(i);
    ++n_norms;
    ++n_work;
    return true;
  }

  // From the value `id` in X to as far as it goes.
  void Follow(uint32_t id, int region) {
    cur = id;
    for (;;) {
      values.push_back({steps.size(), cur});
      Reductions();
      std::vector<int> cand(P.Uses(cur));
      std::sort(cand.begin(), cand.end(), [&](int x, int y) {
        const bool px = path.count(x) != 0, py = path.count(y) != 0;
        return px != py ? px : x < y;
      });
      bool moved = false;
      for (int i : cand) {
        if (!Open(i) || P.n_[i].region != region || steps.size() + 8 > kFuMaxSteps || n_through >= limit) continue;
        if (!Norm(i) && !Through(i)) continue;
        cur = P.n_[i].t.dst;
        ++n_work;
        ++n_through;
        moved = true;
        break;
      }
      if (!moved) break;
      if (P.Def(cur) < 0) {               // written elsewhere too (a loop's carry): what others read there is not followed
        values.push_back({steps.size(), cur});
        break;
      }
    }
    values.back().at = steps.size();
  }
  bool Wanted(uint32_t id) const {
    if (out_of(id) || P.Def(id) < 0) return true;
    for (int u : P.Uses(id)) if (!in.count(u)) return true;
    return false;
  }
  bool out_of(uint32_t id) const { return P.out_.count(id) != 0; }
  // Drops a trailing widening convert whose input is stored anyway: its readers convert as they load.
  void Trim() {
    while (values.size() >= 2) {
      const int d = P.Def(values.back().id);
      if (d < 0 || !in.count(d) || P.n_[d].op != kTopEw || P.n_[d].t.p0 != kConvert || Half(P.n_[d].dt) || out_of(values.back().id)) break;
      bool reduced = false;
      for (int m : members) for (uint32_t b : P.n_[m].rd) if (b == values.back().id) reduced = true;
      if (reduced) break;
      in.erase(d);
      members.erase(std::find(members.begin(), members.end(), d));
      values.pop_back();            // a widening convert has no steps of its own
    }
    cur = values.back().id;
  }
  // The stores that the rest of the program needs; false when a row scalar has a reader outside.
  bool Close(std::vector<uint32_t> *writes, bool first_is_input) {
    for (const auto &kv : scalars) if (Wanted(kv.first)) return false;
    std::vector<Step> all;
    size_t k = 0;
    for (size_t v = 0; v < values.size(); ++v) {
      // a value is complete in X once the steps of its reductions (which leave X alone) begin; store it first
      const size_t at = v == 0 ? values[0].at : values[v].at;
      while (k < std::min(at, steps.size())) all.push_back(steps[k++]);
      const uint32_t id = values[v].id;
      if (v == 0 && first_is_input) continue;
      if (!Wanted(id)) continue;
      Step st;
      st.code = kFuStore; st.id = id; st.dt = MoveDt(P.Dt(id));
      all.push_back(st);
      writes->push_back(id);
    }
    while (k < steps.size()) all.push_back(steps[k++]);
    steps.swap(all);
    if (total >= 0) writes->push_back(static_cast<uint32_t>(total));
    return steps.size() <= static_cast<size_t>(kFuMaxSteps);
  }
};

// A chain's steps as the store epilogue of the product that makes `dst`: fills words 14 .. 24 of its payload.
bool Planner::GemmEpilogue(const Chain &c, uint32_t dst, std::vector<int32_t> *w) const {
  const auto &st = c.steps;
  const bool half = Half(Dt(dst));
  uint32_t flags = 0, rdt = 0, dt0 = 0, dt1 = 0;
  float s0 = 0, s1 = 0, gg = 0;
  int64_t res = -1, out0 = -1, out1 = -1;
  size_t i = 0;
  const size_t n = st.size();
  auto at = [&](size_t k, uint32_t code) { return k < n && st[k].code == code; };
  auto plain_scale = [&](size_t k) { return at(k, kFuAffine) && st[k].t == 0.0f; };
  // The epilogue works on the accumulator and the last store rounds: a 16-bit product that goes on, or leaves in another type,
  // is rounded first; any later value that the program holds in 16 bits may only be the last, and leave in that type.
  if (half && !(n == 1 && at(0, kFuStore) && st[0].dt == Dt(dst))) flags |= kGeQuant0;
  if (at(0, kFuStore) && n > 1) { out0 = st[0].id; dt0 = st[0].dt; i = 1; }
  int64_t rounded = -1;               // the type that the value in hand has yet to be rounded to
  auto quant = [&] { if (at(i, kFuQuant)) rounded = st[i++].dt; };
  if (at(i, kFuGelu)) {
    flags |= kGeGelu;
    ++i;
    quant();
    if ((rounded >= 0 && rounded != static_cast<int64_t>(Dt(dst))) || i + 1 < n) return false;
  }
  if (plain_scale(i) && (at(i + 1, kFuLoadY))) { flags |= kGeScale0; s0 = st[i].s; ++i; if (at(i, kFuQuant)) return false; }
  if (at(i, kFuScalarY) && at(i + 1, kFuMax)) {
    bool known = false;
    for (const auto &k : p_.consts)
      if (k.buffer == static_cast<uint32_t>(st[i].id) && st[i].dt == kF32 && k.data.size() >= 4 && !written_.count(k.buffer)) {
        uint32_t u;
        std::memcpy(&u, k.data.data(), 4);
        s1 = BitsF(u);
        known = true;
      }
    if (!known) return false;
    flags |= kGeMaxS;
    i += 2;
    quant();
  }
  if (at(i, kFuLoadY)) {
    if (rounded >= 0) return false;
    res = st[i].id;
    rdt = st[i].dt;
    ++i;
    flags |= kGeRes;
    if (at(i, kFuGeluGradY)) { gg = st[i].s; ++i; if (!at(i, kFuMul)) return false; flags |= kGeResGeluGrad; ++i; }
    else if (at(i, kFuAdd)) { flags |= kGeResAdd; ++i; }
    else if (at(i, kFuSub)) { flags |= kGeResSub; ++i; }
    else if (at(i, kFuRSub)) { flags |= kGeResRSub; ++i; }
    else if (at(i, kFuMul)) { flags |= kGeResMul; ++i; }
    else return false;
    if (at(i, kFuCarrySumSq)) { flags |= kGeCarrySq; ++i; }
    if (plain_scale(i) && !(flags & kGeMaxS)) { flags |= kGeScale1; s1 = st[i].s; ++i; }
    quant();
  }
  if (!(i + 1 == n && at(i, kFuStore)) || (rounded >= 0 && rounded != static_cast<int64_t>(st[i].dt))) return false;
  out1 = st[i].id;
  dt1 = st[i].dt;
  *w = {static_cast<int32_t>(flags), static_cast<int32_t>(Dt(dst)), static_cast<int32_t>(rdt), FBits(s0), FBits(s1), FBits(gg),
        static_cast<int32_t>(res + 1), static_cast<int32_t>(out0 + 1), static_cast<int32_t>(dt0), static_cast<int32_t>(out1 + 1), static_cast<int32_t>(dt1)};
  return true;
}

// A matmul and the elementwise tasks on its result that a store epilogue can do: on the tensor cores where both operands are
// 16-bit and lie as TMA can fetch them, else on the CUDA cores.
bool Planner::FuseGemm(int seed) {
  const Node &sd = n_[seed];
  const VmTask t = sd.t;
  if (!IsFloatDt(sd.adt) || !IsFloatDt(sd.dt) || Dt(t.a) != sd.adt || Dt(t.b) != sd.adt || Dt(t.dst) != sd.dt) return false;
  if ((t.p3 ? t.p3 : 1u) != 1u || !t.p0 || !t.p1 || !t.p2) return false;
  MmaLayout lay{};
  bool tensor = Half(sd.adt) && MmaOperandLayout(p_, t, &lay);
  for (int64_t v : {lay.a_ld, lay.b_ld, lay.a_off, lay.b_off}) tensor = tensor && v <= 0x7fffffff;
  if (!tensor && !SgOperandsFit(p_, t)) return false;
  // Up to 32 rows: every lane a few columns (ops_skinny.cuh). Above that re-reading the rows for every lane's columns costs more
  // than 128-row tiles leave idle (a 64-row training step: 132 us against 111). So does a second round of columns, where
  // nothing of it is fetched under the first one's sums: 32 x 1024 by 1024 x 8192 33 us against 23 on the tensor-core tiles (29 as
  // scheduled), 1 x 4096 by 4096 x 32000 147 against 82 (88). Few rows and a long K keep it a little further, with k contiguous to
  // four rounds (1 x 4096, 16000 columns 61 against 70, 32000 94 and 82), else to two of up to 4 rows (8192 columns 53 and 59; a
  // batch 1 step of width 2048 147 and 153).
  const uint64_t rounds = (t.p1 + 32ull * L_ - 1) / (32ull * L_);
  const bool few = rounds <= 1 || (lay.bmn ? rounds <= 2 && t.p0 <= 4 && t.p2 >= 2048 : rounds <= 4 && t.p0 <= 16 && t.p2 >= 4096);
  const bool skinny = tensor && few && t.p0 <= 32 && !lay.amn && t.p2 % 8 == 0 && t.p1 >= 8 && (!lay.bmn || t.p1 % 8 == 0) &&
                      static_cast<uint64_t>(t.p1) * t.p2 < (1ull << 31) && SgOperandsFit(p_, t);
  // as many of the tasks that follow as the epilogue has room for: all that the chain takes, then ever fewer
  for (int limit = 1 << 30; limit >= 0;) {
    Chain c(*this, t.p0, t.p1, false);
    c.Take(seed);
    c.limit = limit;
    std::vector<int32_t> epi;
    std::vector<uint32_t> writes;
    if (t.p6) {
      // its own store epilogue: GELU, or a residual sum, on the accumulator
      const int32_t *e = &p_.aux[t.p6 - 1];
      if (e[0] != 1) return false;
      uint32_t flags;
      int64_t res = -1;
      if (e[1] == static_cast<int32_t>(kGelu)) flags = kGeGelu;
      else if (e[1] == static_cast<int32_t>(kAdd) && e[2] == 1 && IsFloatDt(Dt(t.p7))) { flags = kGeRes | kGeResAdd; res = t.p7; c.reads.push_back(t.p7); }
      else return false;
      epi = {static_cast<int32_t>(flags), static_cast<int32_t>(Dt(t.dst)), res >= 0 ? static_cast<int32_t>(Dt(t.p7)) : 0, 0, 0, 0, static_cast<int32_t>(res + 1), 0, 0,
             static_cast<int32_t>(t.dst + 1), static_cast<int32_t>(Dt(t.dst))};
      writes = {t.dst};
    } else {
      c.Follow(t.dst, sd.region);
      limit = std::min(limit, c.n_through) - 1;
      c.Trim();
      if (!c.Close(&writes, false) || writes.empty() || !GemmEpilogue(c, t.dst, &epi)) continue;
    }
    Node nd;
    nd.op = skinny ? kTopSkinny : tensor ? kTopGemm : kTopSgemm;
    nd.dt = sd.dt; nd.adt = sd.adt;
    nd.t = VmTask{};
    nd.t.dst = writes[0];
    nd.t.a = t.a; nd.t.b = t.b;
    nd.rd = c.reads;
    nd.rd.push_back(t.a);
    nd.rd.push_back(t.b);
    nd.wr = writes;
    nd.tiles = 1;
    nd.by_slot = true;
    nd.carry_slot = c.total >= 0 ? 0 : -1;
    nd.owner_word = 2;
    auto I = [](auto v) { return static_cast<int32_t>(v); };
    if (tensor && !skinny) {
      nd.payload = {1, c.total + 1, 0, I(t.p0), I(t.p1), I(t.p2), 0, 0, lay.amn ? 1 : 0, lay.bmn ? 1 : 0,
                    I(sd.adt), I(t.a), I(t.b), I(lay.a_ld), I(lay.b_ld), I(lay.a_off), I(lay.b_off)};
    } else {
      int shape = 0;
      SgShape(nd.op, t.p0, t.p1, t.p2, L_, &shape, &nd.tiles, &nd.cost);
      nd.payload = {shape, c.total + 1, 0, I(t.p0), I(t.p1), I(t.p2), I(sd.adt), I(t.a), I(t.b), I(t.p4), I(t.p5)};
    }
    nd.payload.insert(nd.payload.end(), epi.begin(), epi.end());
    if (skinny) {
      nd.payload.insert(nd.payload.end(), {0, 0, 0, 0});       // gamma + 1, ns, nt: NormIntoProducts; update + 1 (a node here, a task in the program)
      // a dynamic slice update of nothing but this result takes the store
      const int u = writes.size() == 1 && writes[0] == static_cast<uint32_t>(epi[9] - 1) && Uses(writes[0]).size() == 1 && !Pinned(writes[0]) ? Uses(writes[0])[0] : -1;
      if (u >= 0 && Free(u) && n_[u].op == kTopDynScatter && n_[u].t.a == writes[0] && n_[u].dt == Dt(writes[0]) && n_[u].t.p1 == t.p0 * t.p1 &&
          n_[u].region == sd.region) {
        Node with = nd;
        with.payload[20] = static_cast<int32_t>(n_[u].t.dst + 1);
        with.payload[25] = u + 1;
        with.t.dst = n_[u].t.dst;
        with.wr = {n_[u].t.dst};
        for (uint32_t b : n_[u].rd) if (b != writes[0]) with.rd.push_back(b);
        std::vector<int> members = c.members;
        members.push_back(u);
        if (AddPlanned(with, members) >= 0) return true;
      }
    }
    if (AddPlanned(nd, c.members) >= 0) return true;
    if (t.p6) return false;
  }
  return false;
}

// Tile shape of a CUDA-core product: the one with the least time for the busiest lane. A tile's time is its FMAs at the share of
// the issue rate that the shape's shared-memory reads leave, or the latency of its blocks' loads (16 k each, one ahead,
// the CTA's slices taking turns), plus set-up, the slices' sums and stores.
void Planner::SgShape(uint32_t op, uint64_t M, uint64_t N, uint64_t K, uint32_t lanes, int *shape, uint32_t *tiles, double *cost) const {
  struct S { uint32_t tm, tn, slices; double rate; };
  static const S shapes[5] = {{128, 64, 4, 0.75}, {64, 64, 8, 0.75}, {64, 32, 8, 0.6}, {32, 32, 8, 0.45}, {16, 16, 8, 0.2}};
  double best = 1e300;
  if (op == kTopSkinny) {
    // a tile's time: the bytes of its rows and columns at what a lane draws from L2 (~40 a cycle), and what every tile has to
    // wait for once (a first load, the warps' sums, the stores)
    const int mt = M <= 16 ? 0 : 1;
    for (int nb = 0; nb < 3; ++nb) {
      const uint64_t cols = 8ull << nb, T = (N + cols - 1) / cols;
      const double tile = 3000.0 + static_cast<double>(K) * 2.0 * static_cast<double>((16u << mt) + cols) / 40.0;
      const double time = tile * static_cast<double>((T + lanes - 1) / lanes);
      if (time < best) { best = time; *shape = 3 * mt + nb; *tiles = static_cast<uint32_t>(T); *cost = tile / 6000.0; }
    }
    return;
  }
  for (int i = 0; i < 5; ++i) {
    const S &s = shapes[i];
    const uint64_t T = ((M + s.tm - 1) / s.tm) * ((N + s.tn - 1) / s.tn);
    if (T > 0x7fffffffu) continue;
    const double blocks = std::ceil(static_cast<double>((K + 15) / 16) / s.slices);
    const double tile = std::max(static_cast<double>(K) * s.tm * s.tn / (128.0 * s.rate), blocks * 700.0) + 1500.0 + s.tm * s.tn * 0.15;
    const double time = tile * static_cast<double>((T + lanes - 1) / lanes);
    if (time < best) { best = time; *shape = i; *tiles = static_cast<uint32_t>(T); *cost = tile / 6000.0; }
  }
}

// Matmuls of one phase become one task (deepest first), and every product gets its tile shape. A lane's time for a tile is
// the larger of its tensor cycles (2 per column and half, per 64 k) and what it pulls through L2 (~36 bytes per cycle and SM), plus
// the part of the epilogue that nothing hides. The constants were measured with one copying thread and the general epilogue: absolute times
// come out too long (8192 cubed at least 830 us at the top clock, measured 694 at a lower one); they only rank the shapes.
void Planner::GroupGemms(std::vector<int> *live, std::map<std::pair<int, int>, std::vector<int>> *phases, std::vector<std::vector<int>> *of) {
  for (auto &kv : *phases) {
    std::vector<int> gs, rest;
    for (int u : kv.second) (n_[u].op == kTopGemm && n_[u].planned ? gs : rest).push_back(u);
    // CUDA-core and skinny products side by side share the lanes by cost
    double sg_all = 0;
    for (int u : rest) if (n_[u].op == kTopSgemm || n_[u].op == kTopSkinny) sg_all += n_[u].cost * n_[u].tiles;
    for (int u : rest) {
      Node &x = n_[u];
      if (x.op != kTopSgemm && x.op != kTopSkinny) continue;
      const double share = x.cost * x.tiles / sg_all;
      SgShape(x.op, x.payload[3], x.payload[4], x.payload[5], std::max(1u, static_cast<uint32_t>(L_ * share + 0.5)), &x.payload[0], &x.tiles, &x.cost);
    }
    if (gs.empty()) continue;
    std::sort(gs.begin(), gs.end(), [&](int a, int b) { return n_[a].payload[5] > n_[b].payload[5]; });
    std::vector<int> heads;
    for (int g : gs) {
      int into = -1;
      for (int h : heads)
        if (n_[h].payload[0] < kGemmMaxProbs && !(n_[h].carry_slot >= 0 && n_[g].carry_slot >= 0)) { into = h; break; }
      if (into < 0) { heads.push_back(g); continue; }
      Node &h = n_[into];
      const Node &x = n_[g];
      h.payload[0] += 1;
      if (x.carry_slot >= 0) { h.payload[1] = x.payload[1]; h.carry_slot = 0; }
      h.payload.insert(h.payload.end(), x.payload.begin() + 3, x.payload.end());
      h.rd.insert(h.rd.end(), x.rd.begin(), x.rd.end());
      h.wr.insert(h.wr.end(), x.wr.begin(), x.wr.end());
      live->erase(std::find(live->begin(), live->end(), g));
      for (int &r : rep_) if (r == g) r = into;
      (*of)[g].clear();
    }
    for (int h : heads) {
      Node &nd = n_[h];
      const int np = nd.payload[0];
      static const int shapes[6][2] = {{2, 256}, {1, 256}, {2, 128}, {1, 128}, {2, 64}, {1, 64}};
      auto tile_cost = [&](int p, int s) {
        const int32_t *w = &nd.payload[3 + kGemmWords * p];
        const double kb = (w[2] + 63) / 64, hv = shapes[s][0], bn = std::min<double>(shapes[s][1], (w[1] + 15) / 16 * 16);
        const double rows = std::min<double>(hv * 128, (w[0] + 127) / 128 * 128);
        const double tensor = 2.0 * bn * rows / 128, l2 = (rows + bn) * 128 / 36.0;
        return kb * std::max(tensor, l2) + (hv == 2 && bn > 128 ? 1500 : 900) + (hv * bn) * 1.0;
      };
      auto tiles = [&](int p, int s) {
        const int32_t *w = &nd.payload[3 + kGemmWords * p];
        return static_cast<double>((w[0] + 128 * shapes[s][0] - 1) / (128 * shapes[s][0])) * ((w[1] + shapes[s][1] - 1) / shapes[s][1]);
      };
      std::vector<int> best(np, 0), sh(np);
      double best_t = 1e300, cost[kGemmMaxProbs][6], n_tiles[kGemmMaxProbs][6];
      for (int p = 0; p < np; ++p)
        for (int i = 0; i < 6; ++i) { cost[p][i] = tile_cost(p, i); n_tiles[p][i] = tiles(p, i); }
      std::vector<double> load(L_);
      const int combos = np == 1 ? 6 : np == 2 ? 36 : np == 3 ? 216 : 6;
      for (int k = 0; k < combos; ++k) {
        double all = 0;
        for (int p = 0, q = k; p < np; ++p) {
          sh[p] = np <= 3 ? q % 6 : k;
          if (np <= 3) q /= 6;
          all += cost[p][sh[p]] * n_tiles[p][sh[p]];
        }
        if (all >= best_t * L_) continue;              // even cut perfectly no sooner done
        // the lanes' loads when tiles are dealt out in order
        std::fill(load.begin(), load.end(), 0.0);
        uint32_t next = 0;
        for (int p = 0; p < np; ++p) {
          const double c = cost[p][sh[p]];
          const uint64_t n = static_cast<uint64_t>(n_tiles[p][sh[p]]), whole = n / L_;
          for (double &x : load) x += c * static_cast<double>(whole);
          for (uint64_t i = n - whole * L_; i; --i) { load[next] += c; if (++next == L_) next = 0; }
        }
        const double load_max = *std::max_element(load.begin(), load.end());
        if (load_max < best_t) { best_t = load_max; best = sh; }
      }
      uint64_t total = 0;
      for (int p = 0; p < np; ++p) {
        int32_t *w = &nd.payload[3 + kGemmWords * p];
        w[3] = shapes[best[p]][0];
        w[4] = shapes[best[p]][1];
        total += static_cast<uint64_t>(tiles(p, best[p]));
      }
      nd.tiles = static_cast<uint32_t>(std::min<uint64_t>(total, 0x7fffffffu));
      nd.cost = best_t * L_ / std::max<double>(1.0, static_cast<double>(total)) / 6000.0;      // a 4096-element tile of work ~ 6000 cycles
      rest.push_back(h);
    }
    kv.second = rest;
  }
}

// A row pipeline around a row norm or a row reduction: back along the elementwise tasks that lead to it, then forward.
bool Planner::FuseRows(int seed) {
  const Node &sd = n_[seed];
  const uint64_t R = sd.t.p0, C = sd.t.p1;
  if (C < 32 || C > 16384 || R * C >= (1ull << 32)) return false;
  if (sd.op == kTopRedSeg && (sd.t.p3 || sd.dt != kF32 || sd.adt != kF32)) return false;
  if (!IsFloatDt(sd.dt) || !IsFloatDt(sd.adt)) return false;
  uint32_t id = sd.t.a;
  std::vector<int> back;
  for (;;) {
    const int d = Def(id);
    if (d < 0 || !Free(d) || n_[d].op != kTopEw || n_[d].t.p1 != R * C || n_[d].region != sd.region || !IsFloatDt(n_[d].dt) ||
        !IsFloatDt(n_[d].adt))
      break;
    const VmTask &t = n_[d].t;
    if (t.p0 == kFill || t.p0 == kIotaFlat || t.p0 == kCmp || t.p0 == kSelect || t.p0 == kLts || t.p0 == kBitcast || t.p0 == kPow) break;
    if (t.p0 == kAffine || !BinSub(t.p0)) {
      if (t.p0 != kAffine && t.p2) break;
      id = t.a;
    } else if (!t.p2) {
      id = t.a;
    } else if (!t.p3) {
      id = t.b;
    } else {
      break;
    }
    back.push_back(d);
  }
  for (int attempt = 0; attempt < 2; ++attempt) {
    const uint32_t start = attempt == 0 ? id : sd.t.a;
    if (attempt == 1 && start == id) break;
    if (!IsFloatDt(Dt(start)) || Count(start) != R * C) continue;
    Chain c(*this, R, C, true);
    c.path.insert(back.begin(), back.end());
    c.path.insert(seed);
    c.Emit(kFuLoadX, start, Dt(start));
    c.Follow(start, sd.region);
    c.Trim();
    if (!c.in.count(seed) || (c.members.size() < 2 && !c.n_norms)) continue;
    std::vector<uint32_t> writes;
    if (!c.Close(&writes, true) || writes.empty()) continue;
    if (AddPlanned(RowsNode(c, start, writes, R, C, R * C), c.members) >= 0) return true;
  }
  return false;
}

// Phases of the schedule that a chain's tasks are from: how many passes over memory it is instead of. A full sum is one, with
// its combine and a convert that only feeds it (the wire programs' tables fold those too).
int Planner::PhasesMerged(const Chain &c) const {
  std::set<int> ph;
  for (int m : c.members) {
    const Node &nd = n_[m];
    if (nd.op == kTopRedComb) continue;
    if (nd.op == kTopEw && nd.t.p0 == kConvert && Uses(nd.t.dst).size() == 1 && n_[Uses(nd.t.dst)[0]].op == kTopRedPart) continue;
    ph.insert(nd.phase);
  }
  return static_cast<int>(ph.size());
}

Node Planner::RowsNode(const Chain &c, uint32_t start, const std::vector<uint32_t> &writes, uint64_t R, uint64_t C, uint64_t n) const {
  Node nd;
  nd.op = kTopFuseRows;
  nd.dt = nd.adt = kF32;
  nd.t = VmTask{};
  nd.t.dst = writes[0];
  nd.t.a = start;
  nd.rd = c.reads;
  nd.wr = writes;
  nd.tiles = static_cast<uint32_t>(R);
  nd.cost = std::max(0.02, static_cast<double>(C) / 4096.0);
  nd.payload = {static_cast<int32_t>(R), static_cast<int32_t>(C), static_cast<int32_t>(c.steps.size()), c.total + 1,
                C % 4 == 0 && n % 4 == 0 ? 1 : 0, 0, static_cast<int32_t>(n), PhasesMerged(c)};
  nd.owner_word = 5;
  nd.carry_slot = c.total >= 0 ? 0 : -1;
  for (const Step &s : c.steps)
    nd.payload.insert(nd.payload.end(), {static_cast<int32_t>(s.code), static_cast<int32_t>(s.dt), FBits(s.s), FBits(s.t),
                                         static_cast<int32_t>(s.id + 1), static_cast<int32_t>(s.reg)});
  return nd;
}

// What is left of the elementwise tasks, and full sums: chains over a flat list of elements (or over R x C where an operand
// is a row or column vector), one pass each.
bool Planner::FuseFlat(int seed) {
  const Node &sd = n_[seed];
  uint64_t R = 1, C = sd.op == kTopRedPart ? sd.t.p0 : sd.t.p1;
  const uint64_t n = C;
  uint32_t start = sd.t.a;
  if (n == 0 || n >= (1ull << 31)) return false;
  if (sd.op == kTopEw) {
    const uint32_t s = sd.t.p0;
    if (s == kFill || s == kIotaFlat || s == kCmp || s == kSelect || s == kLts || s == kBitcast || s == kIsFinite) return false;
    if (s != kAffine) {
      for (uint32_t field : {sd.t.p2, BinSub(s) ? sd.t.p3 : 0u}) {
        const View v = ViewAt(field);
        if (!field) continue;
        if (!v.ok) return false;
        if (v.v.rank == 2) { R = v.v.dim[0]; C = v.v.dim[1]; }
      }
      if (sd.t.p2) {
        if (!BinSub(s) || sd.t.p3) return false;
        start = sd.t.b;
      }
    }
  }
  if (R * C != n || C > 16384 * (R == 1 ? n : 1) || DtypeSize(Dt(start)) > 4 || Dt(start) == kBool || Count(start) < n) return false;
  Chain c(*this, R, C, false);
  c.path.insert(seed);
  c.Emit(kFuLoadX, start, c.MoveDt(Dt(start)));
  c.Follow(start, sd.region);
  if (!c.in.count(seed)) return false;
  std::vector<uint32_t> writes;
  if (!c.Close(&writes, true) || writes.empty()) return false;
  if (R == 1) {
    // pieces of one "row": one for every lane, as long as that takes, up to what its threads hold
    for (C = 256; C < 4096 && C * L_ < n;) C *= 2;
    R = (n + C - 1) / C;
  }
  return AddPlanned(RowsNode(c, start, writes, R, C, n), c.members) >= 0;
}

// The RMS norm of a few rows that only skinny products read: every lane norms the rows for itself while its weights are on
// their way, instead of in a phase of its own (which is 8 us of latency in a decode step).
void Planner::NormIntoProducts(std::vector<int> *live, std::vector<std::set<int>> *pred) {
  for (size_t k = 0; k < live->size();) {
    const int r = (*live)[k];
    const Node &nd = n_[r];
    ++k;
    if (!nd.planned || nd.op != kTopFuseRows || nd.wr.size() != 1 || nd.payload[0] > 32 || nd.payload[1] > 1024 || nd.payload[1] % 32 != 0 || nd.payload[2] != 9) continue;
    const int32_t *st = &nd.payload[kFuseWords];
    auto code = [&](int i) { return static_cast<uint32_t>(st[6 * i]); };
    const uint32_t dt = static_cast<uint32_t>(st[1]), h = nd.wr[0];
    if (!Half(dt) || code(0) != kFuLoadX || code(1) != kFuRedSumSq || code(2) != kFuSAffine || code(3) != kFuSRsqrt || code(4) != kFuMulS ||
        !(code(5) == kFuRowVecY || (code(5) == kFuLoadY && nd.payload[0] == 1)) || code(6) != kFuMul || code(7) != kFuQuant || code(8) != kFuStore ||
        static_cast<uint32_t>(st[6 * 5 + 1]) != dt || static_cast<uint32_t>(st[6 * 8 + 1]) != dt || Pinned(h))
      continue;
    std::vector<int> users;
    bool ok = true;
    for (int u : *live)
      if (u != r && (*pred)[u].count(r)) {
        users.push_back(u);
        const Node &s = n_[u];
        ok = ok && s.planned && s.op == kTopSkinny && s.region == nd.region && s.payload[3] == nd.payload[0] && s.payload[5] == nd.payload[1] &&
             s.payload[7] == static_cast<int32_t>(h) && s.payload[8] != static_cast<int32_t>(h) && s.payload[9] == 0 && s.payload[17] != static_cast<int32_t>(h + 1) &&
             s.payload[22] == 0;
      }
    if (!ok || users.empty()) continue;
    const int32_t x = st[4] - 1, gamma = st[6 * 5 + 4] - 1;
    for (int u : users) {
      Node &s = n_[u];
      s.payload[7] = x;
      s.payload[22] = gamma + 1;
      s.payload[23] = st[6 * 2 + 2];
      s.payload[24] = st[6 * 2 + 3];
      s.t.a = static_cast<uint32_t>(x);
      s.rd.erase(std::remove(s.rd.begin(), s.rd.end(), h), s.rd.end());
      s.rd.push_back(static_cast<uint32_t>(x));
      s.rd.push_back(static_cast<uint32_t>(gamma));
      (*pred)[u].erase(r);
      (*pred)[u].insert((*pred)[r].begin(), (*pred)[r].end());
    }
    live->erase(live->begin() + static_cast<long>(--k));
  }
}

// Phases by data dependence, lanes by cost, buffers by liveness.
bool Planner::Assemble(VmProgram *q, ReplanStats *st) {
  const int N = static_cast<int>(n_.size());
  // units: planned ops alone; elementwise tasks that followed each other over the same elements stay one chain
  std::vector<int> live;
  for (int i = 0; i < N; ++i) if (rep_[i] == i) live.push_back(i);
  std::vector<std::set<int>> pred(N);
  for (int i = 0; i < n_orig_; ++i)
    for (int j : pred_[i]) if (rep_[j] != rep_[i]) pred[rep_[i]].insert(rep_[j]);
  NormIntoProducts(&live, &pred);
  std::vector<int> unit(N);
  for (int i : live) unit[i] = i;
  std::vector<std::vector<int>> of(N);
  for (int i : live) of[i] = {i};
  auto reaches = [&](int from, int to) {      // a path from -> to through units other than the two
    std::vector<int> todo;
    std::set<int> seen;
    for (int m : of[to]) for (int j : pred[m]) if (unit[j] != from && unit[j] != to) todo.push_back(unit[j]);
    while (!todo.empty()) {
      const int u = todo.back();
      todo.pop_back();
      if (!seen.insert(u).second) continue;
      if (u == from) return true;
      for (int m : of[u]) for (int j : pred[m]) if (unit[j] != u) todo.push_back(unit[j]);
    }
    return false;
  };
  std::sort(live.begin(), live.end(), [&](int a, int b) { return n_[a].order < n_[b].order; });
  for (int i : live) {
    if (n_[i].planned || n_[i].op != kTopEw) continue;
    for (int j : pred[i]) {
      const int u = unit[j];
      if (n_[j].planned || n_[j].op != kTopEw || n_[j].t.p1 != n_[i].t.p1 || n_[j].region != n_[i].region || of[u].size() >= 8 || unit[i] != i)
        continue;
      // the chain runs element by element: its tasks may read each other only without a view
      bool ok = of[u].back() == j;
      for (int m : of[u]) {
        if (n_[i].t.a == n_[m].t.dst && n_[i].t.p2 && n_[i].t.p0 != kAffine) ok = false;
        if (n_[i].t.b == n_[m].t.dst && n_[i].t.p3 && n_[i].t.p0 != kAffine) ok = false;
        for (uint32_t b : n_[m].rd) if (b == n_[i].t.dst) ok = false;
      }
      if (!ok || reaches(u, i)) continue;
      of[u].push_back(i);
      unit[i] = u;
      break;
    }
  }
  // levels
  std::vector<int> level(N, 0);
  bool moved = true;
  for (int round = 0; moved; ++round) {
    if (round > N + 2) return false;
    moved = false;
    for (int i : live)
      for (int j : pred[i]) {
        if (unit[i] == unit[j] || n_[i].region != n_[j].region) continue;
        const int want = level[unit[j]] + 1;
        if (level[unit[i]] < want) { level[unit[i]] = want; moved = true; }
      }
  }
  std::map<std::pair<int, int>, std::vector<int>> phases;        // (region, level) -> units
  for (int i : live) if (unit[i] == i) phases[{n_[i].region, level[i]}].push_back(i);
  GroupGemms(&live, &phases, &of);

  // ---- the program ----
  *q = VmProgram{};
  q->buffers = p_.buffers;
  q->args = p_.args;
  q->results = p_.results;
  q->aux = p_.aux;
  q->consts = p_.consts;
  q->n_instrs = p_.n_instrs;
  q->root_instrs = p_.root_instrs;
  q->n_flags = p_.n_flags;
  std::vector<uint32_t> task_of(N, 0);
  std::map<int, size_t> payload_at;
  // one full-sum counter per op of a phase
  for (auto &kv : phases) {
    int slot = 0;
    for (int u : kv.second)
      for (int i : of[u])
        if (n_[i].carry_slot >= 0) { if (slot >= 3) return false; n_[i].carry_slot = slot++; }
  }
  // the updates that products store through: tasks that no entry names, for their descriptors
  for (int i : live)
    if (n_[i].op == kTopSkinny && n_[i].payload[25]) {
      q->tasks.push_back(n_[n_[i].payload[25] - 1].t);
      n_[i].payload[25] = static_cast<int32_t>(q->tasks.size());
    }
  for (int i : live) {
    VmTask t = n_[i].t;
    if (n_[i].planned) {
      t.tile_op = n_[i].op | (n_[i].dt << 8) | (n_[i].adt << 16);
      t.p2 = static_cast<uint32_t>(q->aux.size());
      t.p3 = static_cast<uint32_t>(std::max(0, n_[i].carry_slot));
      q->aux.push_back(static_cast<int32_t>(n_[i].rd.size()));
      q->aux.push_back(static_cast<int32_t>(n_[i].wr.size()));
      for (uint32_t b : n_[i].rd) q->aux.push_back(static_cast<int32_t>(b));
      for (uint32_t b : n_[i].wr) q->aux.push_back(static_cast<int32_t>(b));
      payload_at[i] = q->aux.size();
      q->aux.insert(q->aux.end(), n_[i].payload.begin(), n_[i].payload.end());
    }
    task_of[i] = static_cast<uint32_t>(q->tasks.size());
    q->tasks.push_back(t);
  }
  std::vector<std::vector<VmEntry>> root(L_), body(L_);
  VmEntry blank;
  std::memset(&blank, 0, sizeof(blank));
  blank.wait_flag = blank.signal_flag = 0xFFFFFFFFu;
  auto barrier = [&](std::vector<std::vector<VmEntry>> &s) {
    VmEntry b = blank;
    b.task = kEntBarrier;
    for (auto &v : s) v.push_back(b);
  };
  int prev_region = -1;
  bool for_placed = false;
  auto place_for = [&] {
    if (!has_loop_ || for_placed) return;
    if (prev_region >= 0) barrier(root);
    VmEntry f = blank;
    f.task = kEntFor;
    f.wait_flag = static_cast<uint32_t>(loop_trip_);
    for (auto &v : root) v.push_back(f);
    for_placed = true;
  };
  std::map<int, int> seen_in_region;
  for (auto &kv : phases) {
    const int region = kv.first.first;
    auto &stream = region == 1 ? body : root;
    if (region == 2 && !for_placed) place_for();
    if (region == 1) {
      if (seen_in_region[1]++) barrier(body);
    } else if (seen_in_region[region]++) {
      barrier(root);
    }
    prev_region = region;
    if (region == 1 && !for_placed) { prev_region = seen_in_region[0] ? 0 : -1; place_for(); prev_region = 1; }
    const auto &us = kv.second;
    std::vector<std::vector<std::pair<uint32_t, uint32_t>>> cut(us.size(), std::vector<std::pair<uint32_t, uint32_t>>(L_, {0u, 0u}));
    // Units of many tiles are cut evenly over all lanes, whatever they cost. Products with few tiles are dear: beside such units they
    // share all lanes among themselves, as they would without them (`mixed`); else units lie side by side by cost.
    bool plenty = true, mixed = false;
    size_t n_slot = 0;
    for (int u : us) { plenty = plenty && n_[u].tiles >= 2 * L_; n_slot += n_[u].by_slot ? 1 : 0; }
    if (!plenty && n_slot && n_slot < us.size()) {
      mixed = true;
      for (int u : us) mixed = mixed && (n_[u].by_slot || n_[u].tiles >= 2 * L_);
    }
    // Only products, not all of them with tiles for everybody: each has lanes of its own. (Cut like tiles, the lane where one product ends
    // and the next begins had a slot in both, and a slot is a whole share of a product: three f32 products of 512 cubed 84 us, where
    // most lanes had done after 50.) A lane works in whole tiles, so one lane after another goes to the product whose busiest lane is
    // done last (of equal ones the one with more work to a lane), as long as it has a tile for it. (By tiles / lanes, not capped, 777 x
    // 100 by K = 512 beside 1024 x 256 by 64 took 31 us, 19 so, 64 x 640 by 64, 400 x 512 by 1024 and 256 x 640 by 2048 together 88, 51
    // so; 4096 x 4096 by 256 beside 2048 x 2048 by 1024, tiles for everybody, 643 apart and 605 side by side.)
    std::vector<std::vector<uint32_t>> own_lanes(us.size());
    const bool apart = us.size() > 1 && n_slot == us.size() && us.size() <= L_ && !plenty;
    if (apart) {
      std::vector<uint32_t> n(us.size(), 1u);
      auto load = [&](size_t k) -> std::pair<double, double> {
        const uint32_t T = n_[us[k]].tiles;
        if (n[k] >= T) return {0.0, 0.0};
        return {n_[us[k]].cost * ((T + n[k] - 1) / n[k]), n_[us[k]].cost * T / n[k]};
      };
      for (uint32_t left = L_ - static_cast<uint32_t>(us.size()); left; --left) {
        size_t most = 0;
        for (size_t k = 1; k < us.size(); ++k) if (load(k) > load(most)) most = k;
        if (load(most).first == 0.0) break;
        ++n[most];
      }
      // Fewer lanes than there are lie spread over the device: side by side some of its parts would do all the loading (three skinny
      // products of 32 x 1024 by 1024, 96 lanes: 18.8 us, 17.9 so).
      uint32_t used = 0, at = 0;
      for (uint32_t x : n) used += x;
      for (size_t k = 0; k < us.size(); ++k)
        for (uint32_t i = 0; i < n[k]; ++i, ++at) own_lanes[k].push_back(static_cast<uint32_t>(static_cast<uint64_t>(at) * L_ / used));
    }
    auto even = [&](int u) { return us.size() == 1 || plenty || (mixed && !n_[u].by_slot); };
    double total = 0;
    for (int u : us) if (!even(u)) total += n_[u].cost * n_[u].tiles * static_cast<double>(of[u].size());
    double at = 0;
    for (size_t k = 0; k < us.size(); ++k) {
      const uint64_t T = n_[us[k]].tiles;
      if (even(us[k])) {
        for (uint64_t l = 0; l < L_; ++l) cut[k][l] = {static_cast<uint32_t>(T * l / L_), static_cast<uint32_t>(T * (l + 1) / L_)};
      } else {
        // units side by side: lane l takes the tiles whose middle falls in its share of the phase's cost
        const double c = n_[us[k]].cost * static_cast<double>(of[us[k]].size());
        uint32_t lo = 0;
        for (uint32_t l = 0; l < L_; ++l) {
          const double edge = total * (l + 1) / L_;
          double hi_f = (edge - at) / c + 0.5;
          uint32_t hi = hi_f <= 0 ? 0u : hi_f >= static_cast<double>(T) ? static_cast<uint32_t>(T) : static_cast<uint32_t>(hi_f);
          if (l + 1 == L_) hi = static_cast<uint32_t>(T);
          hi = std::max(hi, lo);
          cut[k][l] = {lo, hi};
          lo = hi;
        }
        at += c * static_cast<double>(T);
      }
      uint32_t owners = 0;
      if (n_[us[k]].by_slot) {
        // a share of the lanes, each with a slot number (alone in the phase: all of them, as many as there are tiles)
        std::vector<uint32_t> mine = own_lanes[k];
        for (uint32_t l = 0; l < L_ && !apart; ++l)
          if (us.size() == 1 || (mixed && n_slot == 1) ? l < T : cut[k][l].second > cut[k][l].first) mine.push_back(l);
        owners = static_cast<uint32_t>(mine.size());
        for (uint32_t i = 0; i < owners; ++i) {
          VmEntry e = blank;
          e.task = task_of[us[k]];
          e.tile_lo = i;
          e.tile_hi = owners;
          stream[mine[i]].push_back(e);
        }
        if (n_[us[k]].carry_slot >= 0) q->aux[payload_at[us[k]] + n_[us[k]].owner_word] = static_cast<int32_t>(owners);
        continue;
      }
      for (uint32_t l = 0; l < L_; ++l) {
        if (cut[k][l].second <= cut[k][l].first) continue;
        ++owners;
        for (int i : of[us[k]]) {
          VmEntry e = blank;
          e.task = task_of[i];
          e.tile_lo = cut[k][l].first;
          e.tile_hi = cut[k][l].second;
          stream[l].push_back(e);
        }
      }
      for (int i : of[us[k]])
        if (n_[i].carry_slot >= 0) q->aux[payload_at[i] + n_[i].owner_word] = static_cast<int32_t>(owners);
    }
  }
  place_for();
  st->phases = static_cast<uint32_t>(phases.size());
  q->lane_tab.assign(L_, VmLane{});
  q->n_lanes = L_;
  q->barriers_per_lane = 0;
  for (uint32_t l = 0; l < L_; ++l) {
    VmLane &ln = q->lane_tab[l];
    ln.off = static_cast<uint32_t>(q->entries.size());
    ln.root_len = static_cast<uint32_t>(root[l].size());
    for (VmEntry &e : root[l]) {
      if (e.task == kEntFor) { e.tile_lo = ln.root_len; e.tile_hi = static_cast<uint32_t>(body[l].size()); }
      q->entries.push_back(e);
    }
    q->entries.insert(q->entries.end(), body[l].begin(), body[l].end());
    ln.count = static_cast<uint32_t>(q->entries.size()) - ln.off;
    if (l == 0)
      for (uint32_t i = 0; i < ln.count; ++i) q->barriers_per_lane += q->entries[ln.off + i].task == kEntBarrier;
  }

  // ---- buffers: what no task touches any more takes no room; I/O that is bound by address neither ----
  std::map<uint32_t, std::pair<int, int>> span;                 // buffer -> first and last phase (regions far apart)
  std::set<uint32_t> loop_bufs;
  for (int i : live) {
    const int ph = n_[i].region * 100000 + level[unit[i]];
    for (const auto *v : {&n_[i].rd, &n_[i].wr})
      for (uint32_t b : *v) {
        auto it = span.find(b);
        if (it == span.end()) span[b] = {ph, ph};
        else { it->second.first = std::min(it->second.first, ph); it->second.second = std::max(it->second.second, ph); }
        if (n_[i].region == 1) loop_bufs.insert(b);
      }
  }
  std::set<uint32_t> io(in_);
  io.insert(out_.begin(), out_.end());
  std::set<uint32_t> now_written;
  for (int i : live) now_written.insert(n_[i].wr.begin(), n_[i].wr.end());
  auto times = [](const std::vector<uint32_t> &v, uint32_t id) { return std::count(v.begin(), v.end(), id); };
  auto bound = [&](uint32_t b) {               // certainly an I/O port (loader: assign_port)
    if (io.size() > kMaxIoPorts || const_.count(b)) return false;
    if (in_.count(b) && out_.count(b)) return now_written.count(b) && times(p_.args.ids, b) == 1 && times(p_.results.ids, b) == 1;
    return in_.count(b) ? true : out_.count(b) && now_written.count(b) != 0;
  };
  struct Live { uint64_t lo, hi; int last; };
  std::vector<Live> busy;
  uint64_t end = 0;
  std::vector<std::pair<int, uint32_t>> shared;
  std::vector<uint32_t> own;
  for (uint32_t b = 0; b < p_.buffers.size(); ++b) {
    q->buffers[b].offset = 0;
    if (bound(b)) continue;
    if (io.count(b) || const_.count(b) || loop_bufs.count(b)) own.push_back(b);
    else if (span.count(b)) shared.push_back({span[b].first, b});
  }
  std::sort(shared.begin(), shared.end());
  for (auto &x : shared) {
    const uint64_t size = (p_.buffers[x.second].bytes + 255) / 256 * 256;
    busy.erase(std::remove_if(busy.begin(), busy.end(), [&](const Live &l) { return l.last < x.first; }), busy.end());
    std::sort(busy.begin(), busy.end(), [](const Live &a, const Live &b) { return a.lo < b.lo; });
    uint64_t at = 0;
    for (const Live &l : busy) { if (at + size <= l.lo) break; at = std::max(at, l.hi); }
    q->buffers[x.second].offset = at;
    busy.push_back({at, at + size, span[x.second].second});
    end = std::max(end, at + size);
  }
  for (uint32_t b : own) {
    q->buffers[b].offset = end;
    end += (p_.buffers[b].bytes + 255) / 256 * 256;
  }
  q->arena_bytes = std::max<uint64_t>(end, 256);
  return true;
}

bool Planner::Run(VmProgram *q, ReplanStats *st) {
  if (!Extract()) return false;
  for (int i = 0; i < n_orig_; ++i)
    if (Free(i) && n_[i].op == kTopRedStrided && FusePairs(i)) ++st->pairs;
  for (int i = 0; i < n_orig_; ++i)
    if (Free(i) && n_[i].op == kTopMma && FuseGemm(i)) ++st->gemms;
  for (int i = 0; i < n_orig_; ++i)
    if (Free(i) && (n_[i].op == kTopLayernormSeg || n_[i].op == kTopSoftmaxSeg || n_[i].op == kTopRedSeg) && FuseRows(i)) ++st->fused_rows;
  for (int i = 0; i < n_orig_; ++i)
    if (Free(i) && (n_[i].op == kTopEw || n_[i].op == kTopRedPart) && FuseFlat(i)) ++st->fused_rows;
  for (int i = 0; i < n_orig_; ++i) st->absorbed += rep_[i] != i ? 1u : 0u;
  if (!st->absorbed) return false;
  return Assemble(q, st);
}

}  // namespace

bool Replan(const VmProgram &p, uint32_t device_lanes, VmProgram *q, ReplanStats *st) {
  *st = ReplanStats{};
  // A schedule for half the device or less leaves room for another beside it: it keeps its lanes and its cut.
  if (std::getenv("B2VM_NO_REPLAN") || device_lanes < 4 || p.n_lanes * 2 <= device_lanes || p.lane_tab.size() != p.n_lanes) return false;
  Planner pl(p, device_lanes);
  return pl.Run(q, st);
}

}  // namespace b2
