// The lockstep form of a lowered step program: what kernels/lockstep.cu executes when one launch runs ALL ranks on
// one GPU.
//
// Nobody has to be signalled there: every CTA can execute steps of any rank, one barrier over the whole grid separates
// two rounds, and every buffer is visible to every step.  So the program is rewritten as plain data flow before it is
// laid out:
//   1. a step that reads what an earlier copy wrote (staging, a broadcast hop) reads that copy's source instead;
//   2. a copy of what an earlier step produced becomes one more destination of that step;
//   3. a reduction that only continues another one takes over its operands (a ring or pairwise chain becomes one step):
//      where the accumulator is the stored type, so that no rounding falls out;
//   4. writes that nobody reads any more are dropped (scratch, and what a later step replaces);
//   5. rounds are assigned anew, and copies of one source within a round become one step with several destinations.
// Steps are cut where a reader needs a part of what a writer produced.  Every rewrite keeps the serial meaning of the
// program (it is refused when a step in between touches the memory concerned), the order in which a reduction combines
// its operands, and the rounding between two steps, so results are the pull form's bit for bit.
#pragma once
#include <cstdint>
#include <string>
#include <vector>

#include "program.h"

namespace chb {

constexpr int kLockMaxDst = 16;          // destinations of one step
constexpr size_t kLockMaxSrc = 40;       // sources of one step
constexpr int64_t kLockGrain = 2048;     // elements: the unit in which a round's work is dealt to the CTAs
constexpr size_t kLockMaxRewrite = 512;  // longer programs are laid out as they are (the rewriting compares steps pairwise)

struct LockDst { int32_t rank, buf; int64_t off; };
struct LockStepPlan {
  int64_t count = 0;
  bool final = false;               // the reduction's scale applies here
  int32_t level = 0;
  std::vector<Src> srcs;            // an accumulate operand is the first source
  std::vector<LockDst> dsts;
};
struct LockPlan {
  int P = 0, nrounds = 0;
  int64_t in_elems = 0, out_elems = 0, work_elems = 0;
  std::vector<LockStepPlan> steps;  // ordered by round
};

// rewrite: LOCK_PLAIN only the layout (for comparing), LOCK_COPIES without rewrite 3, LOCK_CHAINS everything.
enum { LOCK_PLAIN = 0, LOCK_COPIES = 1, LOCK_CHAINS = 2 };
// The rewriting for a stored type: the 16-bit floats are rounded and bytes wrap after every step (which a scale would
// show), the others accumulate in themselves.
inline int lock_rewrite_for(int dtype) { return dtype == DT_BF16 || dtype == DT_F16 || dtype == DT_U8 ? LOCK_COPIES : LOCK_CHAINS; }
LockPlan make_lock_plan(const Program& p, int rewrite);
inline int lock_saved_rounds(const Program& p, const LockPlan& plan) { return make_lock_plan(p, LOCK_PLAIN).nrounds - plan.nrounds; }

// How a CTA stores the destinations of a step that it has to write (one bit each in `kept`; a copy onto itself is not
// kept).  mixed: they lie on different 16-byte grids, which the vector loops cannot serve at once; `sources`: those that
// are a source of the step as well (same address), looked at only where mixed.
//   0  nothing to store          1  one span for all
//   n  a span for each of the n, which reads the sources anew, so that the one that is a source has to be the last
//  -1  element by element, every source read before any destination is written: several are sources (an in-place
//      allreduce whose chains were joined), and each pass but the first would read what the one before it has stored;
//      or the span has up to kElementSpan elements, where a pass for each destination costs more than element-wise accesses
//      (8 ranks, skewed, in passes / element by element / by the per-rank kernels: allreduce of 39 KiB fp32 33.5 / 14.3 / 17.1 us,
//      of 3 MiB 79 / 32 / 111 us; allgather of 25 MB, whose spans are ten times as long, 62 / 74 / 369 us)
constexpr long long kElementSpan = 8192;
#ifdef __CUDACC__
#define CHB_HOST_DEVICE __host__ __device__
#else
#define CHB_HOST_DEVICE
#endif
CHB_HOST_DEVICE inline int lock_bits(unsigned m) {
#ifdef __CUDA_ARCH__
  return __popc(m);
#else
  return __builtin_popcount(m);
#endif
}
CHB_HOST_DEVICE inline int lock_passes(unsigned kept, bool mixed, unsigned sources, long long count) {
  if (kept == 0u) return 0;
  if (!mixed) return 1;
  return lock_bits(kept & sources) > 1 || count <= kElementSpan ? -1 : lock_bits(kept);
}
// Place of destination i among the kept ones.
CHB_HOST_DEVICE inline int lock_slot(int i, unsigned kept, bool mixed, unsigned sources, long long count) {
  const unsigned last = lock_passes(kept, mixed, sources, count) > 1 ? kept & sources : 0u;
  return (last >> i) & 1u ? lock_bits(kept) - 1 : lock_bits(kept & ~last & ((1u << i) - 1u));
}

// Device tables: LockHeader, LockRound[nrounds], LockStep[nsteps], LockRef[nrefs] (a step's sources, then its
// destinations).  prefix: cost of the round's earlier steps; the cost of a step is its grains x (sources + destinations).
// elems: elements of the round's earlier steps.
struct LockHeader { int nrounds, nsteps, nrefs, pad; };
struct LockRound { int step_begin, step_end; long long cost, elems, pad; };
struct LockStep { long long prefix, count, elems; int ref_begin, nsrc, ndst, final, pad0, pad1; };
struct LockRef { long long off; int rank, buf; };
static_assert(sizeof(LockHeader) % 16 == 0 && sizeof(LockRound) % 16 == 0 && sizeof(LockStep) % 16 == 0 && sizeof(LockRef) % 16 == 0, "copied as 16-byte words");
std::vector<char> make_lock_blob(const LockPlan& p);
inline long long lock_blob_bytes(long long nrounds, long long nsteps, long long nrefs) {
  return (long long)sizeof(LockHeader) + nrounds * (long long)sizeof(LockRound) + nsteps * (long long)sizeof(LockStep) + nrefs * (long long)sizeof(LockRef);
}

// May one CTA run the schedule?  accesses: element loads + stores in all; vec: everything on the 16-byte grid.
constexpr long long kTinyAccesses = 8192;          // loads + stores a round, on average, up to which one CTA runs the schedule
constexpr long long kLockSmemTables = 40 << 10;    // schedules up to this size are kept in shared memory
inline bool lock_one_cta(long long accesses, int nrounds, long long bytes, long long nrefs, int esz, bool vec) {
  return accesses <= kTinyAccesses * nrounds * (vec ? 16 / esz : 1) && bytes + nrefs * (long long)sizeof(void*) <= kLockSmemTables;
}
// Does a schedule run faster in lockstep than with flagged lines (kernels/llprog.cu), whose rounds have no barrier but whose
// data goes through an inbox?  saved: rounds that the rewriting has taken out; payload: bytes of a rank's longer vector.  One
// round: always, its launch alone is cheaper.  One CTA: a round costs little, but it is one SM.  A cluster or the grid: estimates
// in halves of a microsecond.  A round costs about 3.5 us more than one of lines and every 10 KB of tables 1.5 us; lines cost
// 4.5 us where a round is saved and 1 us for each, 0.5 us for each MB that lockstep moves and 20 us for each MB of payload.
// Made from 6520 schedules timed both ways on one B200 (2 to 16 ranks, 2 B to 4 MiB, all algorithms, any alignment): of those
// sent here 179 are more than a tenth and 53 more than three tenths slower than with lines, of those sent to lines 31 and 9 slower
// than in lockstep (with the rounds saved and 192 KiB as the whole rule: 311 and 134, 24 and 9).
// 16 ranks, in lockstep and with lines: ring reduce-scatter of 1248 bf16 a block 51 and 27 us, recursive doubling of 2.5 KiB fp32
// 16.5 and 10.4 us, all-to-all of 80 B blocks 25 and 12 us; 8 ranks, allreduce of 256 KiB fp32, k = 4, b = 2, 13.7 and 15.8 us.  The
// largest misses: a ring reduce-scatter of 16-bit blocks (whose chains are not joined) around 1 MiB, 8 ranks, 44 and 27 us, and
// hierarchical reduce-scatters of a few hundred bytes a block off the 16-byte grid, 16 ranks, 24 and 12 us.
inline bool lock_beats_push(int nrounds, int saved, long long accesses, long long bytes, long long nrefs, long long payload, int esz, bool vec) {
  if (nrounds < 2) return true;
  if (lock_one_cta(accesses, nrounds, bytes, nrefs, esz, vec)) return (vec ? accesses * esz / 16 : accesses) <= kTinyAccesses / 2 * (3 + 2 * saved + nrounds);
  if (saved <= 0 && payload <= (192 << 10)) return false;      // (recursive doubling, halving: every round is an exchange that reduces)
  return 7 * nrounds + 3 * bytes / 10000 <= 13 + (saved > 0 ? 9 + 2 * saved : 0) + ((accesses * esz + 40 * payload) >> 20);
}

// What the one-shot and two-shot line kernels compute, in these tables: operands in rank order, every rank the same result.
// One round: an allreduce is one step (all inputs, all outputs), a reduce-scatter and an allgather one step per block.  It
// follows from a few numbers, so a CTA writes it into its shared memory (entries first, first + stride, ...) instead of
// reading it from a table that somebody has to allocate and upload: the call needs nothing that lasts.
struct FlatSpec { int coll, pad; long long n; };       // coll: 0 allreduce, 1 reduce-scatter, 2 allgather, -1 none; n: elements (of a block)
CHB_HOST_DEVICE inline int flat_steps(int coll, int P) { return coll == 0 ? 1 : P; }
CHB_HOST_DEVICE inline int flat_nsrc(int coll, int P) { return coll == 2 ? 1 : P; }
CHB_HOST_DEVICE inline int flat_ndst(int coll, int P) { return coll == 1 ? 1 : P; }
CHB_HOST_DEVICE inline int flat_refs(int coll, int P) { return flat_steps(coll, P) * (flat_nsrc(coll, P) + flat_ndst(coll, P)); }
CHB_HOST_DEVICE inline int flat_bytes(int coll, int P) {
  return (int)(sizeof(LockHeader) + sizeof(LockRound)) + flat_steps(coll, P) * (int)sizeof(LockStep) + flat_refs(coll, P) * (int)sizeof(LockRef);
}
CHB_HOST_DEVICE inline void flat_write(const FlatSpec& f, int P, char* table, int first, int stride) {
  LockHeader* h = reinterpret_cast<LockHeader*>(table);
  LockRound* round = reinterpret_cast<LockRound*>(h + 1);
  LockStep* steps = reinterpret_cast<LockStep*>(round + 1);
  const int nsteps = flat_steps(f.coll, P), nsrc = flat_nsrc(f.coll, P), refs_per = nsrc + flat_ndst(f.coll, P);
  LockRef* refs = reinterpret_cast<LockRef*>(steps + nsteps);
  const long long cost = (f.n + kLockGrain - 1) / kLockGrain * refs_per;
  for (int i = first; i < nsteps * refs_per + nsteps + 1; i += stride) {
    if (i < nsteps * refs_per) {
      const int s = i / refs_per, q = i % refs_per;      // the q-th reference of block s
      LockRef r;
      r.buf = q < nsrc ? P_IN : P_OUT;
      if (q < nsrc) { r.rank = f.coll == 2 ? s : q; r.off = f.coll == 1 ? s * f.n : 0; }
      else { r.rank = f.coll == 1 ? s : q - nsrc; r.off = f.coll == 2 ? s * f.n : 0; }
      refs[i] = r;
    } else if (i < nsteps * refs_per + nsteps) {
      const int s = i - nsteps * refs_per;
      steps[s] = LockStep{s * cost, f.n, s * f.n, s * refs_per, nsrc, refs_per - nsrc, f.coll == 2 ? 0 : 1, 0, 0};
    } else {
      *h = LockHeader{1, nsteps, nsteps * refs_per, 0};
      *round = LockRound{0, nsteps, nsteps * cost, nsteps * f.n, 0};
    }
  }
}

// Executes the plan on host memory, the steps of a round in random order and the destinations of a step as lock_passes
// has them stored at these addresses, and checks that no step of a round touches what another one writes.  Returns 0, -1 (err says what) or -2 for a bad argument.
int simulate_lock(const Program& p, int dtype, int op, void* const* in, void* const* out, uint64_t seed,
                  int rewrite, std::string* err);
// The same for the flat schedule, as flat_write lays it out.
int simulate_flat(const FlatSpec& f, int P, int dtype, int op, void* const* in, void* const* out, uint64_t seed, std::string* err);

}  // namespace chb
