// Gradient bucket fill for the data-parallel path: one launch per bucket moves
// the gradients of all its parameters (bf16, fp16 or fp32, wherever autograd left
// them) into the bucket's flat fp32 buffer in symmetric memory, either
// overwriting a slot (first micro-batch after zero_grad) or adding to it
// (gradient accumulation).  The bucket is the input of the allreduce kernel
// that follows on the side stream, whose 1/P scale is fused into its last step.
// This replaces one eager cast-and-add per parameter.
// No reference counterpart: the reference stops at the allreduce primitive
// (testing/custom_implementations/work_dir/all_reduce/all_reduce_radix_batch.cpp:202).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../api/chb.h"
#include "common.cuh"

namespace chb {

constexpr int kBucketSlots = 48;      // tensors per launch (the table travels as a kernel argument)
constexpr int kBucketThreads = 256;
constexpr int kBucketBlock = kBucketThreads * 8 * 2;      // elements a CTA moves: two groups of eight a thread

struct BucketTable {
  const void* src[kBucketSlots];
  long long dst_off[kBucketSlots];    // element offset in the bucket
  long long n[kBucketSlots];
  int first[kBucketSlots + 1];        // first CTA of each tensor; [count]: CTAs of the launch
  unsigned char mode[kBucketSlots];   // bit 0: overwrite instead of add; bits 1-2: source type (0 f32, 1 bf16, 2 f16)
  int count;
};

template <typename S>
__device__ __forceinline__ float to_f32(S v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }

// Elements [e0, e0 + kBucketBlock) of one tensor.  Bound by HBM (or L2: the allreduce that follows reads the bucket at
// once), so the loads of both groups of a thread are issued before anything is stored: eight elements a group where both
// sides allow 16-byte accesses (every parameter that starts its allocation) or a 16-bit source 8-byte ones (a view that
// starts at a multiple of four elements: 32 Mi bf16 46 us, 101 us by single elements), else one element at a time.
template <typename S>
__device__ __forceinline__ void fill_block(const S* src, float* dst, long long n, bool overwrite, long long e0) {
  constexpr int W = (int)sizeof(S) / 2;      // 16-byte words of eight source elements
  const unsigned low = (unsigned)(reinterpret_cast<uintptr_t>(src) & 15u);
  const bool vec = (low == 0u || (W == 1 && low == 8u)) && ((reinterpret_cast<uintptr_t>(dst) & 15u) == 0);
  const long long end = n - e0 < kBucketBlock ? n : e0 + kBucketBlock;
  const long long nv = vec ? (end - e0) / 8 : 0;
  const int tid = threadIdx.x;
  uint4 x[2][W];
  float4 a[2][2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int i = tid + u * kBucketThreads;
#pragma unroll
    for (int w = 0; w < W; ++w) x[u][w] = make_uint4(0u, 0u, 0u, 0u);
    a[u][0] = a[u][1] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < nv) {
      const uint4* p = reinterpret_cast<const uint4*>(src + e0) + (long long)i * W;
#pragma unroll
      for (int w = 0; w < W; ++w) {
        if (W > 1 || low == 0u) {
          x[u][w] = __ldcg(p + w);
        } else {
          const uint2 a = __ldcg(reinterpret_cast<const uint2*>(p)), b = __ldcg(reinterpret_cast<const uint2*>(p) + 1);
          x[u][w] = make_uint4(a.x, a.y, b.x, b.y);
        }
      }
      if (!overwrite) {
        const float4* q = reinterpret_cast<const float4*>(dst + e0) + (long long)i * 2;
        a[u][0] = __ldcg(q);
        a[u][1] = __ldcg(q + 1);
      }
    }
  }
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int i = tid + u * kBucketThreads;
    if (i < nv) {
      const S* e = reinterpret_cast<const S*>(x[u]);
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = to_f32<S>(e[j]);
      float4* q = reinterpret_cast<float4*>(dst + e0) + (long long)i * 2;
      if (overwrite) {
        q[0] = make_float4(v[0], v[1], v[2], v[3]);
        q[1] = make_float4(v[4], v[5], v[6], v[7]);
      } else {
        q[0] = make_float4(v[0] + a[u][0].x, v[1] + a[u][0].y, v[2] + a[u][0].z, v[3] + a[u][0].w);
        q[1] = make_float4(v[4] + a[u][1].x, v[5] + a[u][1].y, v[6] + a[u][1].z, v[7] + a[u][1].w);
      }
    }
  }
  for (long long e = e0 + nv * 8 + tid; e < end; e += kBucketThreads) dst[e] = overwrite ? to_f32<S>(__ldcg(src + e)) : dst[e] + to_f32<S>(__ldcg(src + e));
}

// One CTA per kBucketBlock elements of a tensor (a grid of blocks x tensors left most CTAs of a launch to the shortest
// tensors; 5.2 M bf16 gradients in four tensors: a step of fill, allreduce and AdamW 38.8 -> 37.0 us in a graph).
__global__ void __launch_bounds__(kBucketThreads)
bucket_fill_kernel(BucketTable t, float* bucket) {
  int lo = 0, hi = t.count - 1;      // the tensor that owns this CTA
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (t.first[mid] <= (int)blockIdx.x) lo = mid;
    else hi = mid - 1;
  }
  const int k = lo;
  dependent_launch();
  const long long e0 = (long long)((int)blockIdx.x - t.first[k]) * kBucketBlock;
  float* dst = bucket + t.dst_off[k];
  const bool overwrite = (t.mode[k] & 1u) != 0;
  switch ((t.mode[k] >> 1) & 3u) {
    case 0: fill_block<float>(reinterpret_cast<const float*>(t.src[k]), dst, t.n[k], overwrite, e0); break;
    case 1: fill_block<__nv_bfloat16>(reinterpret_cast<const __nv_bfloat16*>(t.src[k]), dst, t.n[k], overwrite, e0); break;
    default: fill_block<__half>(reinterpret_cast<const __half*>(t.src[k]), dst, t.n[k], overwrite, e0); break;
  }
}

}  // namespace chb

using namespace chb;

extern "C" {

// bucket[dst_off[i] .. +n[i]) (+)= src[i] for i < count, any count (launched in groups of 48 tensors).
// src_dtype[i]: CHB_F32 / CHB_BF16 / CHB_F16; overwrite[i] != 0 replaces the slot instead of adding to it.
int chb_bucket_fill(float* bucket, int count, const void* const* src, const long long* dst_off, const long long* n,
                    const int* src_dtype, const unsigned char* overwrite, cudaStream_t stream) {
  if (!bucket || count < 0 || (count && (!src || !dst_off || !n || !src_dtype || !overwrite))) return CHB_ERR_ARG;
  for (int base = 0; base < count; base += kBucketSlots) {
    BucketTable t{};
    t.count = count - base < kBucketSlots ? count - base : kBucketSlots;
    long long ctas = 0;
    for (int i = 0; i < t.count; ++i) {
      const int d = src_dtype[base + i];
      const int code = d == CHB_F32 ? 0 : d == CHB_BF16 ? 1 : d == CHB_F16 ? 2 : -1;
      if (code < 0 || n[base + i] < 0 || dst_off[base + i] < 0) return CHB_ERR_ARG;
      t.src[i] = src[base + i];
      t.dst_off[i] = dst_off[base + i];
      t.n[i] = n[base + i];
      t.mode[i] = (unsigned char)((overwrite[base + i] ? 1 : 0) | (code << 1));
      t.first[i] = (int)ctas;
      ctas += (n[base + i] + kBucketBlock - 1) / kBucketBlock;
      if (ctas > 0x7fffffffll) return CHB_ERR_ARG;      // (beyond 8 Ti elements)
    }
    t.first[t.count] = (int)ctas;
    if (ctas == 0) continue;
    if (launch_overlapped(bucket_fill_kernel, dim3((unsigned)ctas), dim3(kBucketThreads), stream, t, bucket) != cudaSuccess) return CHB_ERR_CUDA;
  }
  return CHB_SUCCESS;
}

}  // extern "C"
