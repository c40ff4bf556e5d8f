// All ranks of a step program in one grid: how an emulated world (every rank on this GPU) runs a schedule.
//
// The interpreter (interp.cu) gives each rank P-th part of the CTAs and lets the ranks signal each other, as they do on
// separate GPUs.  On one GPU that leaves most of the chip idle: in the rounds of a hierarchical schedule two to four of
// eight ranks have work, and 18 CTAs a rank move 0.8 - 2.5 TB/s.  Here a round's steps of all ranks are dealt to all
// CTAs, one grid barrier separates two rounds, and the schedule is first rewritten as data flow (sched/lock_plan.h): no
// staging, and a reduced value goes to every destination that later copies would have taken it to.  A flat allreduce is
// one round that reads every input once and writes every output once.
//
// What bounds it is HBM (for small messages: the launch).  The split: a round's cost is counted in grains of 2048
// elements times the step's sources + destinations, and every CTA takes one contiguous range of that cost, so that all
// finish together whatever the steps' sizes; a CTA streams through one or two steps with the loops of span.cuh.
//
// Three launches: up to kTinyAccesses loads and stores a round one CTA runs everything (a round costs 0.6 us); up to
// kClusterGrains grains one cluster of eight with its hardware barrier (2.8 us a round); above that the whole grid, by a
// cooperative launch unless there is one round only (3.5 us a round, 148 CTAs).
// Measured on one B200 with 8 emulated ranks, per-rank kernels -> this: allreduce 4 MiB fp32 k = 4, b = 2 113 -> 30 us
// (67 MB in and out: 2.2 TB/s), 25 MiB fp32 143 (101 with the loops of span.cuh) -> 84 us (419 MB: 5.0 TB/s),
// reduce-scatter of 8 x 1,000,003 bf16 1238 (144) -> 66 us, k = 2, b = 4 of 4 KiB 12.5 -> 6.8 us.
//
// The ranks' epochs and signal pads are left alone (nobody is signalled and nobody waits), so launches of this kernel
// and of the per-rank ones mix freely on one communicator.
#include <algorithm>
#include <cstring>
#include <vector>

#include "../api/chb.h"
#include "../api/program_handle.h"
#include "../sched/lock_plan.h"
#include "../symm/comm.h"
#include "common.cuh"
#include "span.cuh"

namespace chb {

constexpr int kTinyThreads = 1024;
constexpr int kLockCluster = 8;                    // CTAs of a cluster launch
constexpr long long kClusterGrains = 32;           // grains of a round up to which a cluster runs the schedule

// Barrier over the grid in two halves, so that a CTA works out its share of the next round while the others arrive: one
// release, one acquire poll, and the abort word only on the slow path.
__device__ __forceinline__ void lock_arrive(Ctrl* c) {
  __syncthreads();
  if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&c->bar_count) : "memory");
}
__device__ __forceinline__ bool lock_wait(Ctrl* c, unsigned nct, unsigned gen, unsigned long long timeout_ns, int round) {
  __shared__ int s_pass;
  if (threadIdx.x == 0) {
    int ok = 1;
    const unsigned target = (gen + 1u) * nct;
    auto arrived = [&] {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&c->bar_count) : "memory");
      return v;
    };
    unsigned seen = arrived();
    if (seen < target) {
      const unsigned long long t0 = globaltimer_ns();
      unsigned spins = 0;
      while ((seen = arrived()) < target) {
        if ((++spins & 31u) == 0u) {
          if (ld_volatile_u32(&c->abort)) { ok = 0; break; }
          if (globaltimer_ns() - t0 > timeout_ns) {
            record_timeout(c, ST_TIMEOUT_GRID, 0, round, -1, target, seen);
            ok = 0;
            break;
          }
        }
      }
    }
    s_pass = ok;
  }
  __syncthreads();
  return s_pass != 0;
}

// The same for a grid that is one thread-block cluster: the hardware barrier, with release / acquire at cluster scope.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Base address of a reference's buffer.
__device__ __forceinline__ char* lock_base(const World& w, const IoTable& io, int rank, int buf) {
  return buf == 0 ? const_cast<char*>(io.in[rank]) : buf == 1 ? io.out[rank] : w.work[rank];
}

// Small messages: one CTA runs the whole schedule, a thread an element (VEC: a 16-byte vector, where every address and
// length allows it) at a time whatever step it belongs to, so that a round costs one trip to L2 and a CTA barrier, and
// the launch need not be cooperative.
template <typename T, bool VEC>
__global__ void __launch_bounds__(kTinyThreads, 1)
lock_tiny_kernel(World w, const char* __restrict__ blob, int blob_bytes, FlatSpec flat, IoTable io, int op, float scale) {
  using Acc = typename Elem<T>::Acc;
  constexpr int VE = VEC ? Elem<T>::kPerVec : 1;
  extern __shared__ __align__(16) unsigned char lock_tables[];
  __shared__ int s_ok;
  const int tid = threadIdx.x;
  if (tid == 0) s_ok = 1;
  dependent_launch();
  __syncthreads();
  if (tid < w.P && ld_volatile_u32(&w.ctrl[tid]->abort)) s_ok = 0;
  if (flat.coll >= 0) {
    flat_write(flat, w.P, reinterpret_cast<char*>(lock_tables), tid, kTinyThreads);
  } else {
    const uint4* g = reinterpret_cast<const uint4*>(blob);
    uint4* s = reinterpret_cast<uint4*>(lock_tables);
    for (int i = tid; i < blob_bytes / 16; i += kTinyThreads) s[i] = g[i];
  }
  __syncthreads();
  const LockHeader* h = reinterpret_cast<const LockHeader*>(lock_tables);
  const LockRound* rounds = reinterpret_cast<const LockRound*>(lock_tables + sizeof(LockHeader));
  const LockStep* steps = reinterpret_cast<const LockStep*>(rounds + h->nrounds);
  const LockRef* refs = reinterpret_cast<const LockRef*>(steps + h->nsteps);
  char** at = reinterpret_cast<char**>(lock_tables + blob_bytes);      // refs as addresses
  for (int i = tid; i < h->nrefs; i += kTinyThreads) at[i] = lock_base(w, io, refs[i].rank, refs[i].buf) + refs[i].off * (long long)sizeof(T);
  __syncthreads();
  const int nrounds = s_ok ? h->nrounds : 0;
  for (int t = 0; t < nrounds; ++t) {
    const int n = (int)(rounds[t].elems / VE);
    for (int e = tid; e < n; e += kTinyThreads) {
      int lo = rounds[t].step_begin, hi = rounds[t].step_end - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((int)(steps[mid].elems / VE) <= e) lo = mid;
        else hi = mid - 1;
      }
      const LockStep& st = steps[lo];
      const int x = (e - (int)(st.elems / VE)) * VE * (int)sizeof(T);
      char* const* src = at + st.ref_begin;
      char* const* dst = src + st.nsrc;
      const bool scaled = st.final && scale != 1.0f;
      if constexpr (VEC) {
        uint4 v = ld16_cg(src[0] + x);
        if (st.nsrc > 1 || scaled) {                       // (a plain copy keeps the bits)
          Acc a[VE];
          vec_to_acc<T>(v, a);
#pragma unroll 4
          for (int j = 1; j < st.nsrc; ++j) vec_combine<T>(op, ld16_cg(src[j] + x), a);
          if (scaled) acc_scale<T>(a, scale);
          v = acc_to_vec<T>(a);
        }
        for (int j = 0; j < st.ndst; ++j) st16(dst[j] + x, v);
      } else {
        T v = __ldcg(reinterpret_cast<const T*>(src[0] + x));
        if (st.nsrc > 1 || scaled) {
          Acc a = Elem<T>::up(v);
#pragma unroll 4
          for (int j = 1; j < st.nsrc; ++j) a = combine<Acc>(op, a, Elem<T>::up(__ldcg(reinterpret_cast<const T*>(src[j] + x))));
          if (scaled) a = (Acc)(a * scale);
          v = Elem<T>::down(a);
        }
        for (int j = 0; j < st.ndst; ++j) *reinterpret_cast<T*>(dst[j] + x) = v;
      }
    }
    __syncthreads();
  }
  if (tid == 0) {
    for (int r = 0; r < w.P; ++r) w.ctrl[r]->status[6] += 1ull;
  }
}

// A span whose destinations lie on different 16-byte grids and that is short, or several of whose destinations are its sources
// (an in-place allreduce of skewed buffers): every thread reads all sources of its elements, kElementUnroll at a time, before it stores any.
// Bound by the requests of element-wise accesses.  8 ranks in place, fp32 25 MB, k = 4, b = 2: 109 us where all buffers are
// aligned, 223 us here (994 us with the per-rank kernels).
constexpr int kElementUnroll = 4;
template <typename T>
__device__ __forceinline__ void element_span(const SpanArgs* a) {
  using Acc = typename Elem<T>::Acc;
  const long long count = a->count, nt = blockDim.x;
  for (long long e0 = threadIdx.x; e0 < count; e0 += nt * kElementUnroll) {
    Acc v[kElementUnroll];
#pragma unroll
    for (int u = 0; u < kElementUnroll; ++u) v[u] = e0 + u * nt < count ? Elem<T>::up(__ldcg(reinterpret_cast<const T*>(a->src[0]) + e0 + u * nt)) : (Acc)0;
#pragma unroll 2
    for (int s = 1; s < a->nsrc; ++s) {
      const T* src = reinterpret_cast<const T*>(a->src[s]) + e0;
#pragma unroll
      for (int u = 0; u < kElementUnroll; ++u)
        if (e0 + u * nt < count) v[u] = combine<Acc>(a->op, v[u], Elem<T>::up(__ldcg(src + u * nt)));
    }
#pragma unroll
    for (int u = 0; u < kElementUnroll; ++u) {
      if (a->do_scale) v[u] = (Acc)(v[u] * a->scale);
      if (e0 + u * nt < count)
        for (int d = 0; d < a->ndst; ++d) reinterpret_cast<T*>(a->dst[d])[e0 + u * nt] = Elem<T>::down(v[u]);
    }
  }
}

// CLUSTER: the grid is one cluster (small messages), else the CTAs are co-resident by a cooperative launch, or the schedule
// has one round only.
template <typename T, bool CLUSTER, typename Shape>
__global__ void __launch_bounds__(Shape::kThreads, Shape::kPerSm)
lock_kernel(World w, const char* __restrict__ blob, int blob_bytes, int in_smem, FlatSpec flat, IoTable io, int op, float scale) {
  extern __shared__ __align__(16) unsigned char lock_tables[];
  __shared__ SpanArgs s_span;
  __shared__ char* s_dst[kLockMaxDst];
  __shared__ int s_first, s_passes, s_ok;
  const int tid = threadIdx.x;
  const long long nct = gridDim.x, cta = blockIdx.x;
  if (tid == 0) s_ok = 1;
  dependent_launch();
  __syncthreads();
  if (tid < w.P && ld_volatile_u32(&w.ctrl[tid]->abort)) s_ok = 0;
  const char* tab = blob;
  if (flat.coll >= 0) {
    flat_write(flat, w.P, reinterpret_cast<char*>(lock_tables), tid, Shape::kThreads);
    tab = reinterpret_cast<const char*>(lock_tables);
  } else if (in_smem) {      // one latency for the whole schedule instead of a chain of dependent loads a round
    const uint4* g = reinterpret_cast<const uint4*>(blob);
    uint4* s = reinterpret_cast<uint4*>(lock_tables);
    for (int i = tid; i < blob_bytes / 16; i += Shape::kThreads) s[i] = g[i];
    tab = reinterpret_cast<const char*>(lock_tables);
  }
  __syncthreads();
  const bool ok = s_ok != 0;
  const LockHeader* h = reinterpret_cast<const LockHeader*>(tab);
  const LockRound* rounds = reinterpret_cast<const LockRound*>(tab + sizeof(LockHeader));
  const LockStep* steps = reinterpret_cast<const LockStep*>(rounds + h->nrounds);
  const LockRef* refs = reinterpret_cast<const LockRef*>(steps + h->nsteps);
  // Sets s_span to this CTA's next share at or after step i of the round and returns the step, or -1.
  auto next_share = [&](const LockRound& R, int i) -> int {
    const long long lo = R.cost * cta / nct, hi = R.cost * (cta + 1) / nct;
    for (; i < R.step_end && steps[i].prefix < hi; ++i) {
      const LockStep st = steps[i];
      // grains whose cost begins inside [lo, hi)
      const long long wgt = st.nsrc + st.ndst;
      const long long g0 = lo > st.prefix ? (lo - st.prefix + wgt - 1) / wgt : 0;
      const long long g1 = (hi - st.prefix + wgt - 1) / wgt;
      const long long e0 = g0 * kLockGrain;
      const long long e1 = g1 * kLockGrain < st.count ? g1 * kLockGrain : st.count;
      if (e0 >= e1) continue;
      const bool scaled = st.final && scale != 1.0f;
      if (tid < 32) {                        // destinations: without copies of a region to itself
        const LockRef q = refs[st.ref_begin + st.nsrc + (tid < st.ndst ? tid : 0)];
        const LockRef f = refs[st.ref_begin];
        char* p = lock_base(w, io, q.rank, q.buf) + (q.off + e0) * (long long)sizeof(T);
        const char* from = lock_base(w, io, f.rank, f.buf) + (f.off + e0) * (long long)sizeof(T);
        const bool keep = tid < st.ndst && !(st.nsrc == 1 && !scaled && p == from);
        const unsigned kept = __ballot_sync(0xffffffffu, keep);
        const unsigned grid16 = (unsigned)(reinterpret_cast<unsigned long long>(p) & 15ull);
        const unsigned first16 = __shfl_sync(0xffffffffu, grid16, kept ? __ffs((int)kept) - 1 : 0);
        const bool mixed = __any_sync(0xffffffffu, keep && grid16 != first16);
        bool is_src = false;
        if (mixed && keep)
          for (int j = 0; j < st.nsrc; ++j) {
            const LockRef x = refs[st.ref_begin + j];
            is_src = is_src || p == lock_base(w, io, x.rank, x.buf) + (x.off + e0) * (long long)sizeof(T);
          }
        const unsigned sources = __ballot_sync(0xffffffffu, is_src);
        const int n = __popc(kept);
        const int at = lock_slot(tid, kept, mixed, sources, e1 - e0);
        if (keep) { s_dst[at] = p; s_span.dst[at] = p; }
        if (tid == 0) {
          s_passes = lock_passes(kept, mixed, sources, e1 - e0);
          s_span.nsrc = st.nsrc;
          s_span.ndst = n;
          s_span.count = e1 - e0;
          s_span.op = op;
          s_span.do_scale = scaled;
          s_span.plain = st.nsrc == 1 && !scaled;
          s_span.scale = scale;
        }
      } else if (tid - 32 < st.nsrc) {
        const LockRef q = refs[st.ref_begin + tid - 32];
        s_span.src[tid - 32] = lock_base(w, io, q.rank, q.buf) + (q.off + e0) * (long long)sizeof(T);
      }
      return i;
    }
    return -1;
  };
  // The step in which this CTA's share of a round begins (visible after the next barrier of the CTA).
  auto find_first = [&](const LockRound& R) {
    const long long lo = R.cost * cta / nct;
    for (int i = R.step_begin + tid; i < R.step_end; i += Shape::kThreads)
      if (steps[i].prefix <= lo && (i + 1 == R.step_end || steps[i + 1].prefix > lo)) s_first = i;
  };
  const int nrounds = ok ? h->nrounds : 0;
  if (nrounds > 0) find_first(rounds[0]);
  __syncthreads();
  int i = nrounds > 0 ? next_share(rounds[0], s_first) : -1;
  __syncthreads();
  for (int t = 0; t < nrounds; ++t) {
    while (i >= 0) {
      const int passes = s_passes;           // see lock_passes()
      if (passes < 0) element_span<T>(&s_span);
      for (int d = 0; d < passes; ++d) {
        if (passes > 1) {
          __syncthreads();
          if (tid == 0) { s_span.dst[0] = s_dst[d]; s_span.ndst = 1; }
          __syncthreads();
        }
        run_span<T, Shape>(&s_span);
      }
      __syncthreads();                       // the span's arguments are no longer read
      i = next_share(rounds[t], i + 1);
      if (i >= 0) __syncthreads();
    }
    if (t + 1 == nrounds) break;
    if (CLUSTER) cluster_arrive();
    else lock_arrive(w.ctrl[0]);
    find_first(rounds[t + 1]);
    __syncthreads();
    i = next_share(rounds[t + 1], s_first);
    if (CLUSTER) { cluster_wait(); __syncthreads(); }
    else if (!lock_wait(w.ctrl[0], gridDim.x, (unsigned)t, w.timeout_ns, t)) break;
  }
  rank_exit(w.ctrl[0], gridDim.x, [&](Ctrl*) {
    for (int r = 1; r < w.P; ++r) w.ctrl[r]->status[6] += 1ull;      // (rank_exit counts rank 0's launch)
  });
}

struct LockKernels { const void *wide, *wide2, *cluster, *tiny, *tiny_vec; };
template <typename T>
static LockKernels lock_kernels() { return {(const void*)lock_kernel<T, false, OneCta<T>>, (const void*)lock_kernel<T, false, TwoCtas<T>>,
          (const void*)lock_kernel<T, true, OneCta<T>>, (const void*)lock_tiny_kernel<T, false>,
          (const void*)lock_tiny_kernel<T, true>}; }
static LockKernels pick_lock(int dtype) {
  switch (dtype) {
    case DT_F32: return lock_kernels<float>();
    case DT_BF16: return lock_kernels<__nv_bfloat16>();
    case DT_F16: return lock_kernels<__half>();
    case DT_I32: return lock_kernels<int32_t>();
    case DT_F64: return lock_kernels<double>();
    case DT_I64: return lock_kernels<int64_t>();
    case DT_U8: return lock_kernels<uint8_t>();
  }
  return {nullptr, nullptr, nullptr, nullptr, nullptr};
}

}  // namespace chb

using namespace chb;

extern "C" {

// May this call run in lockstep?  All ranks are here, no per-rank stamps are wanted (they describe ranks that signal
// each other), the steps fit the span arguments, and no rank's output overlaps any input or another output except as
// the schedule knows it: the same buffer of one rank (in place), or `slot_bytes` > 0: an input that already lies in its
// slot of its own output (allgather).
static bool lock_buffers_ok(const chb_comm* c, size_t ni, size_t no, bool in_place, const void* const* in, void* const* out, long long slot_bytes) {
  if (c->nlocal != c->P || c->P < 2 || c->trace) return false;
  for (int b = 0; b < c->P; ++b) {
    const char* o = (const char*)out[b];
    for (int a = 0; a < c->P; ++a) {
      const char* i = (const char*)in[a];
      if (i < o + no && o < i + ni) {
        const bool known = a == b && ((in_place && i == o) || (slot_bytes > 0 && i == o + (size_t)slot_bytes * (size_t)a));
        if (!known) return false;
      }
      const char* q = (const char*)out[a];
      if (a != b && q < o + no && o < q + no) return false;
    }
  }
  return true;
}
int chb_lockstep_ok(const chb_comm* c, const chb_program* p, int dtype, const void* const* in, void* const* out, long long slot_bytes) {
  const Program& g = p->prog;
  const size_t esz = (size_t)dtype_size(dtype);
  return g.stats.max_nsrc <= kMaxSrc && lock_buffers_ok(c, (size_t)g.in_elems * esz, (size_t)g.out_elems * esz, g.in_place, in, out, slot_bytes);
}

// The lockstep schedule of a program for a stored type: laid out and uploaded once.
static int get_lock_blob(chb_comm* c, const chb_program* p, int dtype, const chb_comm::LockBlob** out) {
  const Program& g = p->prog;
  const int rewrite = lock_rewrite_for(dtype);
  const uint64_t key = p->uid * 2u + (rewrite == LOCK_CHAINS ? 1u : 0u);
  auto it = c->lock_blobs.find(key);
  if (it == c->lock_blobs.end()) {
    if (!program_ranges_ok(g, &c->last_error)) return CHB_ERR_ARG;
    const LockPlan plan = make_lock_plan(g, rewrite);
    chb_comm::LockBlob b;
    long long grains = 0, cost = 0;
    for (size_t i = 0; i < plan.steps.size(); ++i) {
      if (i == 0 || plan.steps[i].level != plan.steps[i - 1].level) grains = cost = 0;
      const long long refs = (long long)(plan.steps[i].srcs.size() + plan.steps[i].dsts.size());
      cost += (plan.steps[i].count + kLockGrain - 1) / kLockGrain * refs;
      b.max_cost = cost > b.max_cost ? cost : b.max_cost;
      b.accesses += plan.steps[i].count * refs;
      b.nrefs += (int)refs;
      b.grid |= plan.steps[i].count;
      for (const Src& q : plan.steps[i].srcs) b.grid |= q.off;
      for (const LockDst& q : plan.steps[i].dsts) b.grid |= q.off;
      grains += (plan.steps[i].count + kLockGrain - 1) / kLockGrain;
      b.max_grains = grains > b.max_grains ? grains : b.max_grains;
    }
    b.nrounds = plan.nrounds;
    b.saved_rounds = lock_saved_rounds(g, plan);
    const std::vector<char> host = make_lock_blob(plan);
    b.bytes = (int)host.size();
    if (cudaMalloc(&b.dev, host.size()) != cudaSuccess) { c->last_error = "cudaMalloc(lockstep schedule) failed"; return CHB_ERR_NO_MEM; }
    if (upload_table(b.dev, host) != cudaSuccess) {
      cudaFree(b.dev);
      c->last_error = "cudaMemcpy(lockstep schedule) failed";
      return CHB_ERR_CUDA;
    }
    it = c->lock_blobs.emplace(key, b).first;
  }
  *out = &it->second;
  return CHB_SUCCESS;
}

// Does the communicator's scratch hold the program's?
int chb_program_fits(const chb_comm* c, const chb_program* p, int dtype) {
  return (size_t)p->prog.work_elems * (size_t)dtype_size(dtype) <= c->scratch_bytes;
}

// Everything on the 16-byte grid: addresses, offsets and lengths.
static bool lock_on_grid16(const chb_comm* c, const chb_comm::LockBlob& b, size_t esz, const void* const* in, void* const* out) {
  unsigned long long low = (unsigned long long)b.grid * esz;
  for (int l = 0; l < c->P; ++l) low |= (unsigned long long)(uintptr_t)in[l] | (unsigned long long)(uintptr_t)out[l];
  return (low & 15ull) == 0ull;
}
int chb_lockstep_beats_push(chb_comm* c, const chb_program* p, int dtype, const void* const* in, void* const* out, cudaStream_t stream) {
  const chb_comm::LockBlob* b = nullptr;
  if (get_lock_blob(c, p, dtype, &b)) return 1;     // (the launch reports what is wrong)
  const size_t esz = (size_t)dtype_size(dtype);
  if (lock_beats_push(b->nrounds, b->saved_rounds, b->accesses, b->bytes, b->nrefs,
                      (long long)(std::max(p->prog.in_elems, p->prog.out_elems) * (int64_t)esz), (int)esz, lock_on_grid16(c, *b, esz, in, out)))
    return 1;
  // A captured call cannot upload the tables of the lines: one whose alignment would send it there, unlike that of the calls
  // before it, stays in lockstep, whose tables are up.
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  return !c->ll_blobs.count(p->uid * 16u + esz) && cudaStreamIsCapturing(stream, &capturing) == cudaSuccess && capturing != cudaStreamCaptureStatusNone;
}

// One launch for a schedule whose tables are on the device (b.dev) or follow from `flat`.
static int launch_lockstep(chb_comm* c, const chb_comm::LockBlob& b, const FlatSpec& flat_spec, int dtype, int op, const void* const* in,
                           void* const* out, float scale, int nctas, cudaStream_t stream) {
  const LockKernels fn = pick_lock(dtype);
  const size_t esz = (size_t)dtype_size(dtype);
  FlatSpec flat = flat_spec;
  IoTable io{};
  for (int l = 0; l < c->P; ++l) { io.in[l] = (const char*)in[l]; io.out[l] = (char*)out[l]; }
  long long n = nctas > 0 ? (long long)nctas * c->P : b.max_grains;      // one grain is the least a CTA can be given
  // Two CTAs an SM pay where an SM has 512 KiB to move in a round; below that the larger barrier costs more (8 ranks, one
  // and two: reduce-scatter of odd bf16 blocks, 1.3 MiB an SM, 77 and 67 us; allreduce 4 MiB k = 4, b = 2, 0.3 MiB an SM,
  // 21 and 25 us).
  const bool two = nctas <= 0 && b.max_cost * kLockGrain * (long long)esz >= ((long long)c->max_ctas << 19);
  const long long most = (long long)c->max_ctas * (two ? 2 : 1);
  if (n > most) n = most;
  if (n < 1) n = 1;
  World w = c->world;
  const char* bp = (const char*)b.dev;
  int bytes = b.bytes;
  int in_smem = flat.coll >= 0 || (b.bytes <= kLockSmemTables && tables_in_smem_wanted()) ? 1 : 0;
  cudaError_t e;
  const size_t tiny_smem = (size_t)b.bytes + (size_t)b.nrefs * sizeof(void*);
  const bool vec = lock_on_grid16(c, b, esz, in, out);
  void* tiny_args[] = {&w, &bp, &bytes, &flat, &io, &op, &scale};
  void* wide_args[] = {&w, &bp, &bytes, &in_smem, &flat, &io, &op, &scale};
  const size_t smem = in_smem ? (size_t)b.bytes : 0;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[2] = {};
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.dynamicSmemBytes = smem;
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // see dependent_launch()
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 1;
  if (nctas <= 0 && lock_one_cta(b.accesses, b.nrounds, b.bytes, b.nrefs, (int)esz, vec)) {
    cfg.gridDim = dim3(1);
    cfg.blockDim = dim3(kTinyThreads);
    cfg.dynamicSmemBytes = tiny_smem;
    e = cudaLaunchKernelExC(&cfg, vec ? fn.tiny_vec : fn.tiny, tiny_args);
  } else if (b.nrounds > 1 && n > 1 && (n <= kLockCluster || (nctas <= 0 && b.max_grains <= kClusterGrains))) {
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)(n < kLockCluster ? n : kLockCluster);
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
    cfg.gridDim = dim3(attr[1].val.clusterDim.x);
    cfg.blockDim = dim3(OneCta<float>::kThreads);
    e = cudaLaunchKernelExC(&cfg, fn.cluster, wide_args);
  } else {
    cfg.gridDim = dim3((unsigned)n);
    cfg.blockDim = dim3(two ? TwoCtas<float>::kThreads : OneCta<float>::kThreads);
    if (b.nrounds > 1 && n > 1) {      // CTAs that wait for each other
      attr[0].id = cudaLaunchAttributeCooperative;
      attr[0].val.cooperative = 1;
    }
    e = cudaLaunchKernelExC(&cfg, two ? fn.wide2 : fn.wide, wide_args);
  }
  if (e != cudaSuccess) {
    c->last_error = std::string("lockstep launch failed: ") + cudaGetErrorString(e);
    return CHB_ERR_CUDA;
  }
  return CHB_SUCCESS;
}

// Launch a compiled program with all ranks of an emulated world in one grid.  The conditions, refusals and results are
// chb_run_program's; nctas is per rank as there (0: the launch takes what the message can use).
int chb_run_program_lockstep(chb_comm* c, const chb_program* p, int dtype, int op, const void* const* in,
                             void* const* out, float scale, int nctas, cudaStream_t stream) {
  if (!c || !p || !in || !out || c->nlocal != c->P) return CHB_ERR_ARG;
  const Program& g = p->prog;
  if (g.P != c->P) { c->last_error = "program was compiled for a different number of ranks"; return CHB_ERR_ARG; }
  if (!pick_lock(dtype).wide) return CHB_ERR_ARG;
  if ((size_t)g.work_elems * (size_t)dtype_size(dtype) > c->scratch_bytes) {
    c->last_error = "program needs more symmetric scratch than the communicator has";
    return CHB_ERR_NO_MEM;
  }
  if (op == OP_PROD && dtype == DT_U8) return CHB_ERR_OP;
  const chb_comm::LockBlob* found = nullptr;
  const int rc = get_lock_blob(c, p, dtype, &found);
  if (rc) return rc;
  return launch_lockstep(c, *found, FlatSpec{-1, 0, 0}, dtype, op, in, out, scale, nctas, stream);
}

// The flat schedule of an allreduce (coll 0), reduce-scatter (1) or allgather (2) of n elements (of a block), which needs no program and keeps
// nothing: the first call of a length is captured like any other, and costs 55 us where one that compiles and uploads a schedule
// costs 77 (8 ranks, allreduce of 32 KB, until the result is there; repeated 46).
// CHB_ERR_UNSUPPORTED, and nothing launched, where the buffers or the type are not lockstep's.
int chb_run_flat_lockstep(chb_comm* c, int coll, int dtype, int op, const void* const* in, void* const* out, long long n,
                          float scale, cudaStream_t stream) {
  const long long esz = dtype_size(dtype);
  const size_t ni = (size_t)(n * esz) * (coll == 1 ? c->P : 1), no = (size_t)(n * esz) * (coll == 2 ? c->P : 1);
  if (!pick_lock(dtype).wide || !lock_buffers_ok(c, ni, no, false, in, out, coll == 2 ? n * esz : 0)) return CHB_ERR_UNSUPPORTED;
  const FlatSpec flat{coll, 0, n};
  const long long steps = flat_steps(flat.coll, c->P), grains = (n + kLockGrain - 1) / kLockGrain;
  chb_comm::LockBlob b;
  b.bytes = flat_bytes(flat.coll, c->P);
  b.nrefs = flat_refs(flat.coll, c->P);
  b.nrounds = 1;
  b.max_grains = steps * grains;
  b.max_cost = grains * b.nrefs;
  b.accesses = n * b.nrefs;
  b.grid = n;                                            // (the offsets are multiples of it)
  return launch_lockstep(c, b, flat, dtype, op, in, out, scale, 0, stream);
}

}  // extern "C"
