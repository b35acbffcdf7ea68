// Local streaming kernel: out[i] = cast(in[i] * scale).
//
// Used for world_size == 1 (the reference's whole-buffer cudaMemcpy,
// ibcomm/allreduce_cuda_impl.h:40-46, 332-340, with the scale and the type
// conversion fused in) and by the copy_scale entry point.
//
// Bound by HBM (large messages) or by the launch (small ones).  A thread moves
// ONE quantum, 32 bytes of the wider type, with the 256-bit global accesses of
// sm_100; the grid covers the message once, so 2048 resident threads keep 64
// KiB of loads in flight per SM and a finished block is replaced by the next
// one without a drain between them.  Measured on a B200, against the ring of
// bulk copies through shared memory (one 128 KiB block per SM) it replaced:
//   256 MiB fp32            84.0 -> 80.6 us  (6.66 TB/s read + write)
//   25.6 M fp32 -> bf16     30.3 -> 24.7 us  (6.2 TB/s)
// Two and four quanta per thread are 1-5 % slower (a longer last wave), a
// persistent grid of full SMs 14 % (the head of a launch cannot overlap the
// tail of the one before).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "ibcomm/communicator.h"
#include "kernels.h"
#include "vec_ops.cuh"

namespace ibcomm {
namespace dev {

constexpr int kCopyThreads = 256;
constexpr int kCopyElemUnroll = 8;  // elements in flight per thread of the element-wise kernel

template <typename TI, typename TO>
struct CopyQuantum {
  static constexpr int kWide = static_cast<int>(sizeof(TI) > sizeof(TO) ? sizeof(TI) : sizeof(TO));
  static constexpr int kN = 32 / kWide;  // elements
};

// kN elements from an address aligned to their size, as accumulators; and back.
template <typename T, int kN>
__device__ __forceinline__ void LoadQuantum(const T* p, typename Acc<T>::type* a) {
  if constexpr (sizeof(T) * kN == 32) {
    uint4 lo, hi;
    Ld32(p, &lo, &hi);
    VecIO<T>::Load(lo, a);
    VecIO<T>::Load(hi, a + VecIO<T>::kN);
  } else {
    VecIO<T>::Load(Ld16(p), a);
  }
}
template <typename T, int kN>
__device__ __forceinline__ void StoreQuantum(T* p, const typename Acc<T>::type* a) {
  if constexpr (sizeof(T) * kN == 32) {
    St32(p, VecIO<T>::Store(a), VecIO<T>::Store(a + VecIO<T>::kN));
  } else {
    St16(p, VecIO<T>::Store(a));
  }
}

// `head` elements come before the first quantum whose input and output are
// both aligned; block 0 also does them and the ragged end.
template <typename TI, typename TO>
__global__ void __launch_bounds__(kCopyThreads) CopyScaleKernel(const TI* __restrict__ in, TO* __restrict__ out, uint64_t n, uint32_t head,
                                                                double scale) {
  using A = typename Acc<TI>::type;
  using AO = typename Acc<TO>::type;
  constexpr int kN = CopyQuantum<TI, TO>::kN;
  const uint64_t quanta = (n - head) / kN;
  const uint64_t q = static_cast<uint64_t>(blockIdx.x) * kCopyThreads + threadIdx.x;
  const bool do_scale = scale != 1.0;
  if (q < quanta) {
    A a[kN];
    LoadQuantum<TI, kN>(in + head + q * kN, a);
    AO o[kN];
#pragma unroll
    for (int e = 0; e < kN; ++e) o[e] = static_cast<AO>(do_scale ? ScaleAcc<A>(a[e], scale) : a[e]);
    StoreQuantum<TO, kN>(out + head + q * kN, o);
  }
  if (blockIdx.x == 0) {
    const uint64_t tail = head + quanta * kN;
    const uint32_t edges = head + static_cast<uint32_t>(n - tail);  // at most 2 (kN - 1) elements
    if (threadIdx.x < edges) {
      const uint64_t i = threadIdx.x < head ? threadIdx.x : tail + (threadIdx.x - head);
      const A v = ToAcc<A, TI>(in[i]);
      out[i] = FromAcc<TO, A>(do_scale ? ScaleAcc<A>(v, scale) : v);
    }
  }
}

// Element by element, for buffers that no common number of elements brings to
// their boundaries; kCopyElemUnroll coalesced loads in flight per thread.
template <typename TI, typename TO>
__global__ void __launch_bounds__(kCopyThreads) CopyScaleElementsKernel(const TI* __restrict__ in, TO* __restrict__ out, uint64_t n, double scale) {
  using A = typename Acc<TI>::type;
  const uint64_t base = static_cast<uint64_t>(blockIdx.x) * kCopyThreads * kCopyElemUnroll + threadIdx.x;
  TI v[kCopyElemUnroll];
#pragma unroll
  for (int u = 0; u < kCopyElemUnroll; ++u)
    if (base + u * kCopyThreads < n) v[u] = in[base + u * kCopyThreads];
#pragma unroll
  for (int u = 0; u < kCopyElemUnroll; ++u) {
    if (base + u * kCopyThreads < n) {
      const A a = ToAcc<A, TI>(v[u]);
      out[base + u * kCopyThreads] = FromAcc<TO, A>(scale != 1.0 ? ScaleAcc<A>(a, scale) : a);
    }
  }
}

}  // namespace dev

template <typename TI, typename TO>
static cudaError_t LaunchCopyTyped(const CopyParams& p, cudaStream_t stream) {
  const TI* in = static_cast<const TI*>(p.in);
  TO* out = static_cast<TO*>(p.out);
  const uint64_t n = p.len_elements;
  if (n == 0) return cudaSuccess;
  constexpr uint64_t kN = dev::CopyQuantum<TI, TO>::kN;
  // The first element at which both buffers are aligned to a quantum.  Slices
  // of two tensors at the same offset have one; other pairs may not.
  uint64_t head = 0;
  while (head < kN && ((reinterpret_cast<uintptr_t>(in + head) % (kN * sizeof(TI))) != 0 ||
                       (reinterpret_cast<uintptr_t>(out + head) % (kN * sizeof(TO))) != 0))
    ++head;
  if (head < kN && head <= n) {
    const uint64_t blocks = ((n - head) / kN + dev::kCopyThreads - 1) / dev::kCopyThreads;
    dev::CopyScaleKernel<TI, TO><<<static_cast<unsigned>(blocks > 0 ? blocks : 1), dev::kCopyThreads, 0, stream>>>(
        in, out, n, static_cast<uint32_t>(head), p.scale);
  } else {
    constexpr uint64_t kPerBlock = static_cast<uint64_t>(dev::kCopyThreads) * dev::kCopyElemUnroll;
    dev::CopyScaleElementsKernel<TI, TO><<<static_cast<unsigned>((n + kPerBlock - 1) / kPerBlock), dev::kCopyThreads, 0, stream>>>(
        in, out, n, p.scale);
  }
  return cudaGetLastError();
}

cudaError_t LaunchCopyKernel(const CopyParams& p, cudaStream_t stream) {
  const DType ti = static_cast<DType>(p.dtype_in), to = static_cast<DType>(p.dtype_out);
  if (ti == DType::kFloat32 && to == DType::kFloat32) return LaunchCopyTyped<float, float>(p, stream);
  if (ti == DType::kFloat32 && to == DType::kBFloat16) return LaunchCopyTyped<float, __nv_bfloat16>(p, stream);
  if (ti == DType::kFloat32 && to == DType::kFloat16) return LaunchCopyTyped<float, __half>(p, stream);
  if (ti == DType::kBFloat16 && to == DType::kFloat32) return LaunchCopyTyped<__nv_bfloat16, float>(p, stream);
  if (ti == DType::kFloat16 && to == DType::kFloat32) return LaunchCopyTyped<__half, float>(p, stream);
  if (ti == DType::kFloat64 && to == ti) return LaunchCopyTyped<double, double>(p, stream);
  if (ti == DType::kInt32 && to == ti) return LaunchCopyTyped<int, int>(p, stream);
  if (ti == DType::kInt64 && to == ti) return LaunchCopyTyped<long long, long long>(p, stream);
  if (ti == DType::kFloat16 && to == ti) return LaunchCopyTyped<__half, __half>(p, stream);
  if (ti == DType::kBFloat16 && to == ti) return LaunchCopyTyped<__nv_bfloat16, __nv_bfloat16>(p, stream);
  return cudaErrorInvalidValue;
}

}  // namespace ibcomm
