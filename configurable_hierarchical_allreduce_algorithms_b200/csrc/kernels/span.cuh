// The element loops of a pull step: combine `nsrc` sources left to right over `count` elements and store the result
// at one or several destinations, with all threads of the CTA.
//
// What bounds them is bytes in flight: a source is local HBM / L2 or a peer's memory over NVLink, so every thread
// keeps 64 - 128 bytes of loads outstanding before it touches the first value.  Which loop runs depends on how the
// pointers of the span lie to each other:
//   all equal modulo 32  a scalar head up to the 32-byte boundary, then 256-bit accesses
//   all equal modulo 16  the same with 128-bit accesses
//   anything else        destinations on the 16-byte grid, every source read in the aligned 16-byte words that
//                        cover it (each word once: the next word comes from the next lane) and shifted into place.
//                        Blocks of odd length put nearly every pointer of a reduce-scatter here; element-wise
//                        accesses, which were the only way before, moved 2 - 4 bytes per request.
// Measured on one B200 with 8 emulated ranks (18 CTAs each), before -> after this form: reduce-scatter of 8 blocks of
// 1,000,003 bf16 elements 1237 -> 144 us (element-wise before), allreduce of 64 MiB bf16 (k = 2, b = 4) 1378 -> 929 us and
// of a 25 MiB fp32 bucket 143 -> 101 us (the loops spilled 250 - 1100 bytes a thread before).
// No access leaves [source, source + count): the vector part is cut so that the words around it lie inside, the few
// elements at both ends are scalar.
#pragma once
#include "common.cuh"

namespace chb {

// The accumulators start from a value although the first source overwrites it: left undefined, they stay allocated
// through every loop around (24 registers for each of the loops below, 700 - 1900 bytes of spills a thread).
template <typename T>
__device__ __forceinline__ void acc_clear(typename Elem<T>::Acc* a) {
#pragma unroll
  for (int i = 0; i < Elem<T>::kPerVec; ++i) a[i] = (typename Elem<T>::Acc)0;
}
// SUM: the sum has loops of its own (the operator is a run-time value, and a choice inside the unrolled loops keeps
// every converted operand alive: 560 bytes of spills in the 16-bit loop)
template <typename T, bool SUM>
__device__ __forceinline__ void vec_combine_as(int op, const uint4& v, typename Elem<T>::Acc* a) {
  vec_combine<T>(SUM ? (int)OP_SUM : op, v, a);
}

// 256-bit loop over vectors [j0, nw) strided by TT: G sources x UW vectors in flight per thread.
// (all loops here are inlined into their kernel; the callers keep their span and their place in the schedule in shared
// memory, so that little else competes for registers)
template <typename T, bool SUM, int G, int UW>
__device__ __forceinline__ void reduce_loop32(const char* const* src, long long sofs, int nsrc, char* const* dst, int ndst, long long dofs,
                                           int j0, int nw, int TT, int op, bool do_scale, float scale) {
  using Acc = typename Elem<T>::Acc;
  constexpr int VE = Elem<T>::kPerVec;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 1
  for (; j0 < nw; j0 += TT * UW) {
    Acc a[UW][2][VE];
#pragma unroll
    for (int u = 0; u < UW; ++u) { acc_clear<T>(a[u][0]); acc_clear<T>(a[u][1]); }
#pragma unroll 1
    for (int s = 0; s < nsrc; s += G) {
      uint4 x[G][UW][2];
#pragma unroll
      for (int gi = 0; gi < G; ++gi) {
#pragma unroll
        for (int u = 0; u < UW; ++u) x[gi][u][0] = x[gi][u][1] = zero;
        if (s + gi < nsrc) {
          const char* p0 = src[s + gi] + sofs;
#pragma unroll
          for (int u = 0; u < UW; ++u) {
            const int j = j0 + u * TT;
            if (j < nw) ld32_cg(p0 + (long long)j * 32, x[gi][u][0], x[gi][u][1]);
          }
        }
      }
#pragma unroll
      for (int gi = 0; gi < G; ++gi) {
        if (s + gi < nsrc) {
          if (gi == 0 && s == 0) {
#pragma unroll
            for (int u = 0; u < UW; ++u) { vec_to_acc<T>(x[0][u][0], a[u][0]); vec_to_acc<T>(x[0][u][1], a[u][1]); }
          } else {
#pragma unroll
            for (int u = 0; u < UW; ++u) { vec_combine_as<T, SUM>(op, x[gi][u][0], a[u][0]); vec_combine_as<T, SUM>(op, x[gi][u][1], a[u][1]); }
          }
        }
      }
    }
#pragma unroll
    for (int u = 0; u < UW; ++u) {
      const int j = j0 + u * TT;
      if (j < nw) {
        if (do_scale) { acc_scale<T>(a[u][0], scale); acc_scale<T>(a[u][1], scale); }
        const uint4 lo = acc_to_vec<T>(a[u][0]), hi = acc_to_vec<T>(a[u][1]);
#pragma unroll 1
        for (int d = 0; d < ndst; ++d) st32(dst[d] + dofs + (long long)j * 32, lo, hi);
      }
    }
  }
}

// Plain copy of 256-bit vectors (gather / broadcast steps, staging): no arithmetic (the bits stay, whatever they
// encode), UC vectors in flight per thread, what is left one by one.
template <int UC>
__device__ __forceinline__ void copy_loop32(const char* src, char* const* dst, int ndst, long long dofs, int j0, int nw, int TT) {
  const int stride = TT * 32;
#pragma unroll 1
  for (; j0 + (UC - 1) * TT < nw; j0 += TT * UC) {
    uint4 lo[UC], hi[UC];
    const char* p = src + (long long)j0 * 32;
#pragma unroll
    for (int u = 0; u < UC; ++u) ld32_cg(p + u * stride, lo[u], hi[u]);
#pragma unroll 1
    for (int d = 0; d < ndst; ++d) {
      char* q = dst[d] + dofs + (long long)j0 * 32;
#pragma unroll
      for (int u = 0; u < UC; ++u) st32(q + u * stride, lo[u], hi[u]);
    }
  }
#pragma unroll 1
  for (; j0 < nw; j0 += TT) {
    uint4 lo, hi;
    ld32_cg(src + (long long)j0 * 32, lo, hi);
#pragma unroll 1
    for (int d = 0; d < ndst; ++d) st32(dst[d] + dofs + (long long)j0 * 32, lo, hi);
  }
}

// Bytes [sh, sh + 16) of the 32 bytes {lo, hi}, 0 < sh < 16 (the same sh in all lanes).
__device__ __forceinline__ uint4 funnel16(const uint4& lo, const uint4& hi, unsigned sh) {
  unsigned w0 = lo.x, w1 = lo.y, w2 = lo.z, w3 = lo.w, w4 = hi.x, w5 = hi.y, w6 = hi.z;
  if (sh & 8u) { w0 = w2; w1 = w3; w2 = w4; w3 = w5; w4 = w6; w5 = hi.w; }
  if (sh & 4u) { w0 = w1; w1 = w2; w2 = w3; w3 = w4; w4 = w5; }
  const unsigned b = (sh & 3u) * 8u;
  return make_uint4(__funnelshift_r(w0, w1, b), __funnelshift_r(w1, w2, b), __funnelshift_r(w2, w3, b), __funnelshift_r(w3, w4, b));
}

// 128-bit loop for pointers that do not share an alignment.  Vector j covers bytes [pos + 16 j, +16) of every pointer;
// dst[.] + pos is 16-byte aligned, sources need not be.  The caller guarantees that the two aligned words around each
// vector lie inside the source.  A warp takes 32 * U consecutive vectors, so that all but its last word are shared.
template <typename T, bool SUM, int G, int U>
__device__ __forceinline__ void reduce_loop16(const char* const* src, int nsrc, char* const* dst, int ndst, long long pos, long long nv,
                                           int op, bool do_scale, float scale) {
  using Acc = typename Elem<T>::Acc;
  constexpr int VE = Elem<T>::kPerVec;
  const int lane = threadIdx.x & 31;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const long long step = (long long)(blockDim.x >> 5) * 32 * U;
#pragma unroll 1
  for (long long base = (long long)(threadIdx.x >> 5) * 32 * U; base < nv; base += step) {   // uniform per warp
    Acc a[U][VE];
#pragma unroll
    for (int u = 0; u < U; ++u) acc_clear<T>(a[u]);
#pragma unroll 1
    for (int s = 0; s < nsrc; s += G) {
      uint4 x[G][U], tail[G];
      unsigned sh[G];
#pragma unroll
      for (int gi = 0; gi < G; ++gi) {
        sh[gi] = 0u;
        tail[gi] = zero;
#pragma unroll
        for (int u = 0; u < U; ++u) x[gi][u] = zero;
        if (s + gi < nsrc) {
          const char* p = src[s + gi] + pos;
          sh[gi] = (unsigned)(reinterpret_cast<unsigned long long>(p) & 15ull);
          p -= sh[gi];
          const long long words = nv + (sh[gi] ? 1 : 0);
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const long long j = base + u * 32 + lane;
            if (j < words) x[gi][u] = ld16_cg(p + j * 16);
          }
          if (sh[gi] && lane == 31 && base + U * 32 < words) tail[gi] = ld16_cg(p + (base + U * 32) * 16);
        }
      }
#pragma unroll
      for (int gi = 0; gi < G; ++gi) {
        if (s + gi < nsrc) {
#pragma unroll
          for (int u = 0; u < U; ++u) {
            uint4 v = x[gi][u];
            if (sh[gi]) {
              // the word after mine: lane + 1's of this block, for lane 31 the first of the next block
              const uint4 give = (lane == 0 && u + 1 < U) ? x[gi][u + 1 < U ? u + 1 : u] : v;
              const int from = (lane + 1) & 31;
              uint4 next;
              next.x = __shfl_sync(0xffffffffu, give.x, from);
              next.y = __shfl_sync(0xffffffffu, give.y, from);
              next.z = __shfl_sync(0xffffffffu, give.z, from);
              next.w = __shfl_sync(0xffffffffu, give.w, from);
              if (u + 1 == U && lane == 31) next = tail[gi];
              v = funnel16(v, next, sh[gi]);
            }
            if (gi == 0 && s == 0) vec_to_acc<T>(v, a[u]);
            else vec_combine_as<T, SUM>(op, v, a[u]);
          }
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long j = base + u * 32 + lane;
      if (j < nv) {
        if (do_scale) acc_scale<T>(a[u], scale);
        const uint4 v = acc_to_vec<T>(a[u]);
#pragma unroll 1
        for (int d = 0; d < ndst; ++d) st16(dst[d] + pos + j * 16, v);
      }
    }
  }
}

// The same for a plain copy.
template <int U>
__device__ __forceinline__ void copy_loop16(const char* src, char* const* dst, int ndst, long long pos, long long nv) {
  const int lane = threadIdx.x & 31;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const char* p = src + pos;
  const unsigned sh = (unsigned)(reinterpret_cast<unsigned long long>(p) & 15ull);
  p -= sh;
  const long long words = nv + (sh ? 1 : 0);
  const long long step = (long long)(blockDim.x >> 5) * 32 * U;
#pragma unroll 1
  for (long long base = (long long)(threadIdx.x >> 5) * 32 * U; base < nv; base += step) {   // uniform per warp
    uint4 x[U], tail = zero;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long j = base + u * 32 + lane;
      x[u] = zero;
      if (j < words) x[u] = ld16_cg(p + j * 16);
    }
    if (sh && lane == 31 && base + U * 32 < words) tail = ld16_cg(p + (base + U * 32) * 16);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      uint4 v = x[u];
      if (sh) {
        const uint4 give = (lane == 0 && u + 1 < U) ? x[u + 1 < U ? u + 1 : u] : v;
        const int from = (lane + 1) & 31;
        uint4 next;
        next.x = __shfl_sync(0xffffffffu, give.x, from);
        next.y = __shfl_sync(0xffffffffu, give.y, from);
        next.z = __shfl_sync(0xffffffffu, give.z, from);
        next.w = __shfl_sync(0xffffffffu, give.w, from);
        if (u + 1 == U && lane == 31) next = tail;
        v = funnel16(v, next, sh);
      }
      const long long j = base + u * 32 + lane;
      if (j < nv) {
#pragma unroll 1
        for (int d = 0; d < ndst; ++d) st16(dst[d] + pos + j * 16, v);
      }
    }
  }
}

// One span: dst[d][e] = scale * (src[0][e] op src[1][e] op ...) for e < count.  All threads of the CTA; src / dst are
// in shared memory; the destinations are equal modulo 16 (the caller issues one span for each otherwise).
// A source may be a destination as well (same address, same element): every element is loaded by the thread that
// stores it, also in the shifted loop, where such a source lies on the destination's grid and needs no shift.
// Shape: what is in flight per thread, see below.
template <typename T, typename Shape>
__device__ __forceinline__ void reduce_span(const char* const* src, int nsrc, char* const* dst, int ndst, long long count,
                                            int op, bool plain, bool do_scale, float scale) {
  using Acc = typename Elem<T>::Acc;
  const int tid = threadIdx.x, nt = blockDim.x;
  const unsigned long long d0 = reinterpret_cast<unsigned long long>(dst[0]);
  unsigned long long diff = 0ull;            // bits in which any pointer differs from the first destination
  for (int d = 1; d < ndst; ++d) diff |= reinterpret_cast<unsigned long long>(dst[d]) ^ d0;
  for (int s = 0; s < nsrc; ++s) diff |= reinterpret_cast<unsigned long long>(src[s]) ^ d0;
  const long long bytes = count * (long long)sizeof(T);
  long long lo, hi;                          // the vector part, in bytes from the start
  if ((diff & 31ull) == 0ull) {
    lo = (long long)((32ull - (d0 & 31ull)) & 31ull);
    if (lo > bytes) lo = bytes;
    const int nw = (int)((bytes - lo) / 32);       // (a span is far below 2^31 vectors)
    hi = lo + (long long)nw * 32;
    const int j0 = tid;
    if (plain) copy_loop32<Shape::kCopy32>(src[0] + lo, dst, ndst, lo, j0, nw, nt);
    else if (op != OP_SUM) reduce_loop32<T, false, 2, 1>(src, lo, nsrc, dst, ndst, lo, j0, nw, nt, op, do_scale, scale);
    else if (Shape::kUnroll == 1 || nw <= nt) reduce_loop32<T, true, Shape::kShort, 1>(src, lo, nsrc, dst, ndst, lo, j0, nw, nt, op, do_scale, scale);
    else reduce_loop32<T, true, Shape::kLong, Shape::kUnroll>(src, lo, nsrc, dst, ndst, lo, j0, nw, nt, op, do_scale, scale);
  } else {
    lo = (long long)((16ull - (d0 & 15ull)) & 15ull);
    long long room = 0;                      // bytes that have to follow the last vector
    if ((diff & 15ull) != 0ull) { lo += 16; room = 16; }
    if (lo > bytes) lo = bytes;
    const long long left = bytes - lo - room;
    const long long nv = left > 0 ? left / 16 : 0;
    hi = lo + nv * 16;
    if (plain) copy_loop16<Shape::kCopy16>(src[0], dst, ndst, lo, nv);
    else if (op == OP_SUM) reduce_loop16<T, true, 2, Shape::kUnroll16>(src, nsrc, dst, ndst, lo, nv, op, do_scale, scale);
    else reduce_loop16<T, false, 2, 1>(src, nsrc, dst, ndst, lo, nv, op, do_scale, scale);
  }
  // both ends, element by element (by the last threads: in a short span they had no vector and start at once)
  const int head = (int)(lo / (long long)sizeof(T));
  const long long at = hi / (long long)sizeof(T);
  const int edge = head + (int)(count - at);
  for (int i = nt - 1 - tid; i < edge; i += nt) {
    const long long e = i < head ? i : at + (i - head);
    Acc a = Elem<T>::up(__ldcg(reinterpret_cast<const T*>(src[0]) + e));
    for (int s = 1; s < nsrc; ++s) a = combine<Acc>(op, a, Elem<T>::up(__ldcg(reinterpret_cast<const T*>(src[s]) + e)));
    if (do_scale) a = (Acc)(a * scale);
    const T v = plain ? __ldcg(reinterpret_cast<const T*>(src[0]) + e) : Elem<T>::down(a);
    for (int d = 0; d < ndst; ++d) reinterpret_cast<T*>(dst[d])[e] = v;
  }
}

// What a span needs, in shared memory: set by the caller between two barriers, so that nothing of the schedule walk
// stays in registers across the loops.
constexpr int kMaxSrc = 40;     // sources per step (incl. the accumulate operand)
struct SpanArgs {
  const char* src[kMaxSrc];
  char* dst[kMaxRanks];
  long long count;
  int nsrc, ndst;
  int op, plain, do_scale;   // plain: one source and no scale
  float scale;
};
// Loads in flight.  A span with at most one vector per thread is bound by the depth of its chain of round trips: several
// sources at a time; longer ones by bytes in flight: fewer sources, two vectors deep.
// OneCta: 128 registers a thread (512 threads, one CTA an SM): 128 bytes a thread, 64 KiB an SM.
template <typename T> struct OneCta {
  static constexpr int kThreads = 512, kPerSm = 1;
  static constexpr bool kWide = sizeof(T) > 1;                     // (16 accumulators a vector for bytes)
  static constexpr int kShort = kWide ? 4 : 2, kLong = 2, kUnroll = kWide ? 2 : 1, kUnroll16 = kWide ? 2 : 1, kCopy32 = 4, kCopy16 = 4;
};
// TwoCtas: 80 registers (384 threads, two CTAs an SM): one vector of as many sources as fit, up to 96 KiB an SM.
template <typename T> struct TwoCtas {
  static constexpr int kThreads = 384, kPerSm = 2;
  static constexpr int kShort = sizeof(T) > 2 ? 4 : 2, kLong = 2, kUnroll = 1, kUnroll16 = sizeof(T) > 1 ? 2 : 1, kCopy32 = 3, kCopy16 = 3;
};
// FourCtas: the registers of TwoCtas in smaller CTAs (192 threads, four an SM).
template <typename T> struct FourCtas : TwoCtas<T> {
  static constexpr int kThreads = 192, kPerSm = 4;
};
template <typename T, typename Shape>
__device__ __forceinline__ void run_span(const SpanArgs* a) {
  reduce_span<T, Shape>(a->src, a->nsrc, a->dst, a->ndst, a->count, a->op, a->plain != 0, a->do_scale != 0, a->scale);
}

}  // namespace chb
