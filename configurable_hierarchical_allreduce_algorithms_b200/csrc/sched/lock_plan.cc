#include "lock_plan.h"

#include <algorithm>
#include <cstring>
#include <random>

namespace chb {
namespace {

inline bool overlap(int64_t a, int64_t an, int64_t b, int64_t bn) { return a < b + bn && b < a + an; }

// Works on steps in the program's serial order; a step without destinations is dead.
struct Rewriter {
  std::vector<LockStepPlan>& s;
  bool in_place;                    // a rank's input and output are one buffer
  int key(int rank, int buf) const { return rank * 3 + (in_place && buf == P_IN ? (int)P_OUT : buf); }
  bool writes(const LockStepPlan& x, int k, int64_t off, int64_t n) const {
    for (const LockDst& d : x.dsts)
      if (key(d.rank, d.buf) == k && overlap(d.off, x.count, off, n)) return true;
    return false;
  }
  bool reads(const LockStepPlan& x, int k, int64_t off, int64_t n) const {
    if (x.dsts.empty()) return false;
    for (const Src& r : x.srcs)
      if (key(r.peer, r.buf) == k && overlap(r.off, x.count, off, n)) return true;
    return false;
  }
  bool plain(const LockStepPlan& x) const { return x.srcs.size() == 1 && !x.final; }
  // last step before i that writes any of [off, off + n), or -1
  int last_writer(int i, int k, int64_t off, int64_t n) const {
    for (int j = i - 1; j >= 0; --j)
      if (writes(s[(size_t)j], k, off, n)) return j;
    return -1;
  }
  const LockDst* covering(const LockStepPlan& x, int k, int64_t off, int64_t n) const {
    for (const LockDst& d : x.dsts)
      if (key(d.rank, d.buf) == k && d.off <= off && off + n <= d.off + x.count) return &d;
    return nullptr;
  }

  void cut(size_t i, int64_t at) {
    LockStepPlan hi = s[i];
    s[i].count = at;
    hi.count -= at;
    for (Src& r : hi.srcs) r.off += at;
    for (LockDst& d : hi.dsts) d.off += at;
    s.insert(s.begin() + (long)i + 1, std::move(hi));
  }
  // Cut readers at the ends of what an earlier writer produced, and writers at the ends of what a copy takes from
  // them.  False when that makes too many steps (the caller then starts from the uncut ones).
  bool refine() {
    for (size_t i = 0; i < s.size(); ++i)
      for (size_t q = 0; q < s[i].srcs.size(); ++q) {
        bool again = true;
        while (again) {
          again = false;
          if (s.size() > kLockMaxRewrite) return false;
          const Src r = s[i].srcs[q];
          const int k = key(r.peer, r.buf);
          const int64_t n = s[i].count;
          for (size_t j = i; j-- > 0 && !again;) {
            if (!writes(s[j], k, r.off, n)) continue;
            const bool copies = plain(s[i]);
            for (const LockDst& d : s[j].dsts) {
              if (!(copies || plain(s[j])) || key(d.rank, d.buf) != k || !overlap(d.off, s[j].count, r.off, n)) continue;
              const int64_t b = d.off, e = d.off + s[j].count;
              if (b > r.off) { cut(i, b - r.off); again = true; }
              else if (e < r.off + n) { cut(i, e - r.off); again = true; }
              else if (copies && r.off > b) { cut(j, r.off - b); ++i; again = true; }
              else if (copies && r.off + n < e) { cut(j, r.off + n - b); ++i; again = true; }
              break;
            }
            break;                                     // the last writer decides
          }
        }
      }
    return true;
  }

  // The regions [off, off + n) that step i is to read or write early: nobody between the two steps touches them.
  bool quiet(int after, int before, int k, int64_t off, int64_t n, bool reads_count) const {
    for (int j = after + 1; j < before; ++j) {
      const LockStepPlan& x = s[(size_t)j];
      if (writes(x, k, off, n) || (reads_count && reads(x, k, off, n))) return false;
    }
    return true;
  }
  void forward_sources(int i) {
    LockStepPlan& x = s[(size_t)i];
    for (Src& r : x.srcs)
      for (;;) {
        const int k = key(r.peer, r.buf);
        const int c = last_writer(i, k, r.off, x.count);
        if (c < 0 || !plain(s[(size_t)c])) break;
        const LockStepPlan& w = s[(size_t)c];
        const LockDst* d = covering(w, k, r.off, x.count);
        if (!d) break;
        const Src from{w.srcs[0].peer, w.srcs[0].buf, w.srcs[0].off + (r.off - d->off)};
        const int kf = key(from.peer, from.buf);
        // the source still holds what was copied (the copy itself may not have overwritten it either), and this
        // step does not write it
        if (writes(w, kf, from.off, x.count) || !quiet(c, i, kf, from.off, x.count, false)) break;
        if (writes(x, kf, from.off, x.count)) break;
        r = from;
      }
  }
  void fold_copy(int i) {
    LockStepPlan& x = s[(size_t)i];
    if (!plain(x) || x.dsts.size() != 1) return;
    const Src r = x.srcs[0];
    const int a = last_writer(i, key(r.peer, r.buf), r.off, x.count);
    if (a < 0) return;
    LockStepPlan& w = s[(size_t)a];
    const LockDst* d = covering(w, key(r.peer, r.buf), r.off, x.count);
    if (!d || w.count != x.count || (int)w.dsts.size() >= kLockMaxDst) return;   // (equal length: refine() cut both)
    const LockDst to = x.dsts[0];
    const int k = key(to.rank, to.buf);
    if (reads(w, k, to.off, x.count) || writes(w, k, to.off, x.count)) return;
    if (!quiet(a, i, k, to.off, x.count, true)) return;
    w.dsts.push_back(to);
    x.dsts.clear();
  }
  // x = (a op b) op c, where only x reads the a op b that step w stored: x takes w's operands in w's place.
  void join_chain(int i) {
    LockStepPlan& x = s[(size_t)i];
    if (x.dsts.empty() || x.srcs.size() < 2) return;
    const Src r = x.srcs[0];
    const int k = key(r.peer, r.buf);
    const int a = last_writer(i, k, r.off, x.count);
    if (a < 0) return;
    LockStepPlan& w = s[(size_t)a];
    if (w.final || w.count != x.count || w.dsts.size() != 1 || w.srcs.size() + x.srcs.size() - 1 > kLockMaxSrc) return;
    const LockDst d = w.dsts[0];
    if (d.off != r.off) return;
    // nobody else reads what w stored before all of it is replaced (scratch: to the end)
    bool needed = d.buf != P_WORK;
    for (size_t j = (size_t)a + 1; j < s.size(); ++j) {
      if (j != (size_t)i && reads(s[j], k, d.off, w.count)) return;
      if (j >= (size_t)i && covering(s[j], k, d.off, w.count)) { needed = false; break; }
    }
    if (needed) return;
    for (size_t q = 1; q < x.srcs.size(); ++q)
      if (key(x.srcs[q].peer, x.srcs[q].buf) == k && overlap(x.srcs[q].off, x.count, d.off, w.count)) return;
    // w's operands still hold the same values, and x does not write them except element for element
    for (const Src& q : w.srcs) {
      const int kq = key(q.peer, q.buf);
      if (!quiet(a, i, kq, q.off, x.count, false)) return;
      for (const LockDst& y : x.dsts)
        if (key(y.rank, y.buf) == kq && y.off != q.off && overlap(y.off, x.count, q.off, x.count)) return;
    }
    std::vector<Src> all = w.srcs;
    all.insert(all.end(), x.srcs.begin() + 1, x.srcs.end());
    x.srcs = std::move(all);
    w.dsts.clear();
  }
  // Writes that nobody reads: scratch to the end of the program, any memory up to a step that replaces all of it.
  void drop_dead_writes() {
    for (int i = (int)s.size() - 1; i >= 0; --i) {
      auto& d = s[(size_t)i].dsts;
      const int64_t n = s[(size_t)i].count;
      for (size_t q = d.size(); q-- > 0;) {
        const int k = key(d[q].rank, d[q].buf);
        bool used = d[q].buf != P_WORK;
        for (size_t j = (size_t)i + 1; j < s.size(); ++j) {
          if (reads(s[j], k, d[q].off, n)) { used = true; break; }
          if (covering(s[j], k, d[q].off, n)) { used = false; break; }
        }
        if (!used) d.erase(d.begin() + (long)q);
      }
    }
  }
  void assign_rounds() {
    for (size_t i = 0; i < s.size(); ++i) {
      int32_t lvl = 0;
      for (size_t j = 0; j < i; ++j) {
        if (s[j].level < lvl) continue;
        bool dep = false;
        for (const Src& r : s[i].srcs) dep = dep || writes(s[j], key(r.peer, r.buf), r.off, s[i].count);
        for (const LockDst& d : s[i].dsts)
          dep = dep || writes(s[j], key(d.rank, d.buf), d.off, s[i].count) || reads(s[j], key(d.rank, d.buf), d.off, s[i].count);
        if (dep) lvl = s[j].level + 1;
      }
      s[i].level = lvl;
    }
  }
  void merge_copies() {
    for (size_t i = 0; i < s.size(); ++i) {
      if (!plain(s[i]) || s[i].dsts.empty()) continue;
      for (size_t j = i + 1; j < s.size(); ++j) {
        if (s[j].level != s[i].level || !plain(s[j]) || s[j].count != s[i].count) continue;
        const Src &a = s[i].srcs[0], &b = s[j].srcs[0];
        if (a.peer != b.peer || a.buf != b.buf || a.off != b.off) continue;
        if (s[i].dsts.size() + s[j].dsts.size() > (size_t)kLockMaxDst) continue;
        s[i].dsts.insert(s[i].dsts.end(), s[j].dsts.begin(), s[j].dsts.end());
        s[j].dsts.clear();
      }
    }
  }
  void sweep() {
    s.erase(std::remove_if(s.begin(), s.end(), [](const LockStepPlan& x) { return x.dsts.empty(); }), s.end());
  }
};

}  // namespace

LockPlan make_lock_plan(const Program& p, int rewrite) {
  LockPlan out;
  out.P = p.P;
  out.in_elems = p.in_elems;
  out.out_elems = p.out_elems;
  out.work_elems = p.work_elems;
  for (const Op& o : p.ops) {
    if (o.count <= 0) continue;
    LockStepPlan x;
    x.count = o.count;
    x.final = (o.flags & OPF_FINAL) != 0;
    x.level = o.level;
    if (o.acc) x.srcs.push_back(Src{o.rank, o.dst_buf, o.dst_off});
    x.srcs.insert(x.srcs.end(), o.srcs.begin(), o.srcs.end());
    x.dsts.push_back(LockDst{o.rank, o.dst_buf, o.dst_off});
    out.steps.push_back(std::move(x));
  }
  if (rewrite != LOCK_PLAIN && out.steps.size() <= kLockMaxRewrite) {
    Rewriter rw{out.steps, p.in_place};
    const std::vector<LockStepPlan> whole = out.steps;
    if (!rw.refine()) out.steps = whole;
    for (int i = 0; i < (int)out.steps.size(); ++i) {
      rw.forward_sources(i);
      rw.fold_copy(i);
    }
    rw.sweep();
    rw.drop_dead_writes();
    rw.sweep();
    if (rewrite == LOCK_CHAINS)
      for (int i = 0; i < (int)out.steps.size(); ++i) rw.join_chain(i);
    rw.sweep();
    rw.drop_dead_writes();
    rw.sweep();
    rw.assign_rounds();
    rw.merge_copies();
    rw.sweep();
  }
  std::stable_sort(out.steps.begin(), out.steps.end(), [](const LockStepPlan& a, const LockStepPlan& b) { return a.level < b.level; });
  // rounds without steps (an entry handshake) need no place of their own
  int32_t last = -1, n = 0;
  for (LockStepPlan& x : out.steps) {
    if (x.level != last) { last = x.level; ++n; }
    x.level = n - 1;
  }
  out.nrounds = n;
  return out;
}

std::vector<char> make_lock_blob(const LockPlan& p) {
  LockHeader h{};
  h.nrounds = p.nrounds;
  h.nsteps = (int)p.steps.size();
  std::vector<LockRound> rounds((size_t)p.nrounds);
  std::vector<LockStep> steps;
  std::vector<LockRef> refs;
  int cur = -1;
  for (const LockStepPlan& x : p.steps) {
    if (x.level != cur) {
      cur = x.level;
      rounds[(size_t)cur].step_begin = rounds[(size_t)cur].step_end = (int)steps.size();
    }
    LockRound& r = rounds[(size_t)cur];
    LockStep d{};
    d.prefix = r.cost;
    d.elems = r.elems;
    r.elems += x.count;
    d.count = x.count;
    d.ref_begin = (int)refs.size();
    d.nsrc = (int)x.srcs.size();
    d.ndst = (int)x.dsts.size();
    d.final = x.final ? 1 : 0;
    for (const Src& q : x.srcs) refs.push_back(LockRef{q.off, q.peer, q.buf});
    for (const LockDst& q : x.dsts) refs.push_back(LockRef{q.off, q.rank, q.buf});
    r.cost += (x.count + kLockGrain - 1) / kLockGrain * (long long)(d.nsrc + d.ndst);
    steps.push_back(d);
    r.step_end = (int)steps.size();
  }
  h.nrefs = (int)refs.size();
  std::vector<char> blob(sizeof(h) + rounds.size() * sizeof(LockRound) + steps.size() * sizeof(LockStep) + refs.size() * sizeof(LockRef));
  char* at = blob.data();
  auto put = [&](const void* src, size_t n) { if (n) std::memcpy(at, src, n); at += n; };
  put(&h, sizeof(h));
  put(rounds.data(), rounds.size() * sizeof(LockRound));
  put(steps.data(), steps.size() * sizeof(LockStep));
  put(refs.data(), refs.size() * sizeof(LockRef));
  return blob;
}

namespace {

template <typename T>
T combine_host(int op, T a, T b) {
  switch (op) {
    case OP_SUM: return (T)(a + b);
    case OP_MAX: return a > b ? a : b;
    case OP_MIN: return a < b ? a : b;
    default: return (T)(a * b);
  }
}

template <typename T>
int simulate_lock_t(const Program& p, const LockPlan& plan, int rop, void* const* in, void* const* out, uint64_t seed, std::string* err) {
  std::vector<std::vector<T>> work((size_t)p.P, std::vector<T>((size_t)p.work_elems));
  for (auto& w : work)
    if (!w.empty()) std::memset(w.data(), 0xFF, w.size() * sizeof(T));      // scratch that nobody has written stands out
  auto ptr = [&](int rank, int buf, int64_t off) -> T* {
    return buf == P_IN ? (T*)in[rank] + off : buf == P_OUT ? (T*)out[rank] + off : work[(size_t)rank].data() + off;
  };
  std::mt19937_64 rng(seed);
  size_t a = 0;
  while (a < plan.steps.size()) {
    size_t b = a;
    while (b < plan.steps.size() && plan.steps[b].level == plan.steps[a].level) ++b;
    std::vector<LockStepPlan> now(plan.steps.begin() + (long)a, plan.steps.begin() + (long)b);
    Rewriter rw{now, p.in_place};
    for (size_t i = 0; i < now.size(); ++i)
      for (size_t j = 0; j < now.size(); ++j)
        for (size_t q = 0; q < now[i].dsts.size(); ++q) {
          const LockDst& d = now[i].dsts[q];
          const int k = rw.key(d.rank, d.buf);
          bool bad = i != j && (rw.writes(now[j], k, d.off, now[i].count) || rw.reads(now[j], k, d.off, now[i].count));
          for (size_t q2 = 0; i == j && q2 < q; ++q2)
            bad = bad || (rw.key(now[i].dsts[q2].rank, now[i].dsts[q2].buf) == k && overlap(now[i].dsts[q2].off, now[i].count, d.off, now[i].count));
          if (i == j)      // a step may read where it writes only element for element
            for (const Src& r : now[i].srcs)
              bad = bad || (rw.key(r.peer, r.buf) == k && r.off != d.off && overlap(r.off, now[i].count, d.off, now[i].count));
          if (bad) {
            if (err) *err = "two steps of round " + std::to_string(now[i].level) + " of " + p.name + " touch the same memory";
            return -1;
          }
        }
    std::shuffle(now.begin(), now.end(), rng);
    for (const LockStepPlan& x : now) {
      auto combined = [&] {
        const T* first = ptr(x.srcs[0].peer, x.srcs[0].buf, x.srcs[0].off);
        std::vector<T> v(first, first + x.count);
        for (size_t i = 1; i < x.srcs.size(); ++i) {
          const T* y = ptr(x.srcs[i].peer, x.srcs[i].buf, x.srcs[i].off);
          for (int64_t e = 0; e < x.count; ++e) v[(size_t)e] = combine_host<T>(rop, v[(size_t)e], y[e]);
        }
        return v;
      };
      unsigned kept = 0u, sources = 0u;
      bool mixed = false;
      T* to[kLockMaxDst] = {};
      T* slot[kLockMaxDst] = {};
      uintptr_t grid = 0;
      for (size_t q = 0; q < x.dsts.size(); ++q) {
        to[q] = ptr(x.dsts[q].rank, x.dsts[q].buf, x.dsts[q].off);
        if (x.srcs.size() == 1 && !x.final && to[q] == ptr(x.srcs[0].peer, x.srcs[0].buf, x.srcs[0].off)) continue;
        if (kept == 0u) grid = (uintptr_t)to[q] & 15u;
        mixed = mixed || ((uintptr_t)to[q] & 15u) != grid;
        kept |= 1u << q;
        for (const Src& r : x.srcs)
          if (ptr(r.peer, r.buf, r.off) == to[q]) sources |= 1u << q;
      }
      for (size_t q = 0; q < x.dsts.size(); ++q)
        if ((kept >> q) & 1u) slot[lock_slot((int)q, kept, mixed, sources, x.count)] = to[q];
      const int passes = lock_passes(kept, mixed, sources, x.count);
      std::vector<T> v;
      for (int d = 0; d < lock_bits(kept); ++d) {
        if (!slot[d]) {
          if (err) *err = "a step of round " + std::to_string(x.level) + " of " + p.name + " leaves a destination unset";
          return -1;
        }
        if (d == 0 || passes > 1) v = combined();
        std::memcpy(slot[d], v.data(), (size_t)x.count * sizeof(T));
      }
    }
    a = b;
  }
  return 0;
}

int simulate_plan(const Program& p, const LockPlan& plan, int dtype, int op, void* const* in, void* const* out, uint64_t seed, std::string* err) {
  switch (dtype) {
    case DT_F32: return simulate_lock_t<float>(p, plan, op, in, out, seed, err);
    case DT_F64: return simulate_lock_t<double>(p, plan, op, in, out, seed, err);
    case DT_I32: return simulate_lock_t<int32_t>(p, plan, op, in, out, seed, err);
    case DT_I64: return simulate_lock_t<int64_t>(p, plan, op, in, out, seed, err);
    case DT_U8: return simulate_lock_t<uint8_t>(p, plan, op, in, out, seed, err);
  }
  if (err) *err = "simulate: unsupported dtype on the host";
  return -2;
}

}  // namespace

int simulate_lock(const Program& p, int dtype, int op, void* const* in, void* const* out, uint64_t seed, int rewrite, std::string* err) {
  return simulate_plan(p, make_lock_plan(p, rewrite), dtype, op, in, out, seed, err);
}

int simulate_flat(const FlatSpec& f, int P, int dtype, int op, void* const* in, void* const* out, uint64_t seed, std::string* err) {
  std::vector<char> table((size_t)flat_bytes(f.coll, P), (char)0xEE);
  const int stride = 1 + (int)(seed % 7);
  for (int first = stride - 1; first >= 0; --first) flat_write(f, P, table.data(), first, stride);
  const LockHeader* h = reinterpret_cast<const LockHeader*>(table.data());
  const LockRound* rounds = reinterpret_cast<const LockRound*>(h + 1);
  const LockStep* steps = reinterpret_cast<const LockStep*>(rounds + h->nrounds);
  const LockRef* refs = reinterpret_cast<const LockRef*>(steps + h->nsteps);
  LockPlan plan;
  plan.P = P;
  plan.nrounds = h->nrounds;
  for (int i = rounds[0].step_begin; i < rounds[0].step_end; ++i) {
    LockStepPlan x;
    x.count = steps[i].count;
    x.final = steps[i].final != 0;
    const LockRef* r = refs + steps[i].ref_begin;
    for (int q = 0; q < steps[i].nsrc; ++q) x.srcs.push_back(Src{r[q].rank, r[q].buf, r[q].off});
    for (int q = 0; q < steps[i].ndst; ++q) x.dsts.push_back(LockDst{r[steps[i].nsrc + q].rank, r[steps[i].nsrc + q].buf, r[steps[i].nsrc + q].off});
    plan.steps.push_back(x);
  }
  // the places of steps and costs are those that the tables of such a plan have
  const std::vector<char> built = make_lock_blob(plan);
  if (built.size() != table.size() || std::memcmp(built.data(), table.data(), table.size()) != 0) {
    if (err) *err = "the flat schedule's table is not that of its steps";
    return -1;
  }
  Program p;
  p.P = P;
  p.name = "flat";
  return simulate_plan(p, plan, dtype, op, in, out, seed, err);
}

}  // namespace chb
