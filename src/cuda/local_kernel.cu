// Direct collectives of ranks that share a GPU, on buffers used in place: the
// two-shot allreduce and its halves, and the one-shot allreduce, whose sums are the
// same.  One launch runs all ranks, so the inputs
// are there when it starts, its end is everybody's, and a result is stored by
// the thread that has read everything it replaces: no barrier, flag, call
// number or scratch memory, and an ordinary launch.  Between GPUs these are
// nvls_kernel.cu (peer loads and stores) and rsag_kernel.cu.
//
//   allreduce       element i of every rank's output = scale * sum over the ranks' inputs
//   reduce-scatter  rank s's output = scale * sum over the ranks of block s of their inputs
//   all-gather      block s of every rank's output = rank s's input
//
// Sums run in rank order.  With a 16-bit wire type, fp32 values are rounded to it
// where they would travel: every contribution, and the result.  There is no link to
// save bytes on, so nothing is stored in 16 bits.
//
// Bound by HBM, so as many small blocks as there are vectors, each a round of loads:
// B200, 8 ranks x 16 MiB of bf16 44.2 us (6.1 TB/s) against 55 by the kernel with two
// barriers and blocks that stay, 47 by that one without them; 8 x 25 MiB of fp32 with a
// bf16 wire 66 us against 156 through the pool.  32-byte accesses give another 1 %.
// One-shot, 8 x 64 KiB: 4.1 us, a launch, against 6.2 with a push into every rank's slot
// and a flag (and 8.2 with pushes that carry their flags).
#include <cstdint>

#include "ibcomm/communicator.h"
#include "kernels.h"
#include "vec_ops.cuh"

namespace ibcomm {
namespace dev {

// A thread per vector: blocks of 64 to 256 are within 1 % of each other.
constexpr int kLocalThreads = 128;

// kR: ranks at most (2, 4 or 8), so that all their loads are in flight and in registers.
template <typename T, typename W, LocalOp kOp, int kR>
__global__ void __launch_bounds__(kLocalThreads) LocalKernel(const __grid_constant__ LocalParams p) {
  using A = typename Acc<T>::type;
  constexpr bool kRounds = sizeof(W) != sizeof(T);
  constexpr bool kSums = kOp != LocalOp::kAllGather;
  constexpr bool kToAll = kOp != LocalOp::kReduceScatter;
  constexpr int kN = 16 / static_cast<int>(sizeof(T));
  const int ws = p.world_size, s = blockIdx.y;  // the block, for the halves
  const uint64_t in_at = kOp == LocalOp::kReduceScatter ? static_cast<uint64_t>(s) * p.len_elements : 0;
  const uint64_t out_at = kOp == LocalOp::kAllGather ? static_cast<uint64_t>(s) * p.len_elements : 0;
  const T* src[kR];
  T* dst[kR];
#pragma unroll
  for (int q = 0; q < kR; ++q) {
    src[q] = q < ws ? static_cast<const T*>(p.in[q]) + in_at : nullptr;
    dst[q] = q < ws ? static_cast<T*>(p.out[q]) + out_at : nullptr;
  }
  // The sides of which there is one per rank share their 16-byte boundaries; the vectors are theirs.
  // The other side of a half may be off them.
  const T* const one_src = static_cast<const T*>(p.in[kSums ? 0 : s]);
  T* const one_dst = static_cast<T*>(p.out[kToAll ? 0 : s]);
  const uintptr_t side = reinterpret_cast<uintptr_t>(kSums ? src[0] : dst[0]);
  uint64_t head = ((16u - (side & 15u)) & 15u) / sizeof(T);
  if (head > p.len_elements) head = p.len_elements;
  const uint64_t nvec = (p.len_elements - head) / kN;
  const uint64_t i = static_cast<uint64_t>(blockIdx.x) * kLocalThreads + threadIdx.x;
  const bool do_scale = kSums && p.scale != 1.0;

  auto finish = [&](A v) -> A {
    if (do_scale) v = ScaleAcc<A>(v, p.scale);
    return kRounds ? ThroughWire<W, A>(v) : v;
  };
  if (i < nvec) {
    const uint64_t at = head + i * kN;
    uint4 r;
    if constexpr (kSums) {
      uint4 v[kR];
#pragma unroll
      for (int q = 0; q < kR; ++q)
        if (q < ws) v[q] = Ld16(src[q] + at);
      A acc[kN];
      VecIO<T>::Load(v[0], acc);
      if constexpr (kRounds) {
#pragma unroll
        for (int e = 0; e < kN; ++e) acc[e] = ThroughWire<W, A>(acc[e]);
      }
#pragma unroll
      for (int q = 1; q < kR; ++q)
        if (q < ws) {
          if constexpr (kRounds) {
            A more[kN];
            VecIO<T>::Load(v[q], more);
#pragma unroll
            for (int e = 0; e < kN; ++e) acc[e] += ThroughWire<W, A>(more[e]);
          } else {
            VecIO<T>::Add(v[q], acc);
          }
        }
#pragma unroll
      for (int e = 0; e < kN; ++e) acc[e] = finish(acc[e]);
      r = VecIO<T>::Store(acc);
    } else {
      r = LdUser16<T>(reinterpret_cast<const unsigned char*>(one_src + at), (reinterpret_cast<uintptr_t>(one_src + head) & 15u) == 0);
    }
    if constexpr (kToAll) {
#pragma unroll
      for (int q = 0; q < kR; ++q)
        if (q < ws) St16(dst[q] + at, r);
    } else {
      StUser16<T>(reinterpret_cast<unsigned char*>(one_dst + at), r, (reinterpret_cast<uintptr_t>(one_dst + head) & 15u) == 0);
    }
    return;
  }
  // The elements before the first vector, then those behind the last.
  uint64_t at = i - nvec;
  if (at >= head) at += nvec * kN;
  if (at >= p.len_elements) return;
  T r;
  if constexpr (kSums) {
    A acc = A(0);
#pragma unroll
    for (int q = 0; q < kR; ++q)
      if (q < ws) acc += kRounds ? ThroughWire<W, A>(ToAcc<A, T>(src[q][at])) : ToAcc<A, T>(src[q][at]);
    r = FromAcc<T, A>(finish(acc));
  } else {
    r = one_src[at];
  }
  if constexpr (kToAll) {
#pragma unroll
    for (int q = 0; q < kR; ++q)
      if (q < ws) dst[q][at] = r;
  } else {
    one_dst[at] = r;
  }
}

}  // namespace dev

template <typename T, typename W, LocalOp kOp>
static cudaError_t Launch(const LocalParams& p, cudaStream_t stream) {
  // Every thread has a vector, or one of the elements outside of them; at most 2 * 16 / sizeof(T) of those.
  const uint64_t items = p.len_elements / (16 / sizeof(T)) + 32 / sizeof(T);
  const uint64_t blocks = (items + dev::kLocalThreads - 1) / dev::kLocalThreads;
  if (blocks > 0x7fffffffu) return cudaErrorInvalidValue;
  const dim3 grid(static_cast<unsigned>(blocks), kOp == LocalOp::kAllreduce ? 1u : static_cast<unsigned>(p.world_size));
  if (p.world_size <= 2) dev::LocalKernel<T, W, kOp, 2><<<grid, dev::kLocalThreads, 0, stream>>>(p);
  else if (p.world_size <= 4) dev::LocalKernel<T, W, kOp, 4><<<grid, dev::kLocalThreads, 0, stream>>>(p);
  else dev::LocalKernel<T, W, kOp, kMaxRanks><<<grid, dev::kLocalThreads, 0, stream>>>(p);
  return cudaGetLastError();
}

template <typename T>
static cudaError_t LaunchTyped(const LocalParams& p, cudaStream_t stream) {
  switch (p.op) {
    case LocalOp::kAllreduce: return Launch<T, T, LocalOp::kAllreduce>(p, stream);
    case LocalOp::kReduceScatter: return Launch<T, T, LocalOp::kReduceScatter>(p, stream);
    case LocalOp::kAllGather: return Launch<T, T, LocalOp::kAllGather>(p, stream);
  }
  return cudaErrorInvalidValue;
}

bool LocalKernelTakes(const LocalParams& p) {
  // Where every rank has one, the buffers have to miss their 16-byte boundaries alike.
  bool alike = true;
  auto differ = [](const void* a, const void* b) { return ((reinterpret_cast<uintptr_t>(a) ^ reinterpret_cast<uintptr_t>(b)) & 15u) != 0; };
  for (int q = 0; q < p.world_size; ++q) {
    if (p.op != LocalOp::kAllGather && differ(p.in[0], p.in[q])) alike = false;
    if (p.op != LocalOp::kReduceScatter && differ(p.out[0], p.out[q])) alike = false;
  }
  return alike && (p.op != LocalOp::kAllreduce || !differ(p.in[0], p.out[0]));
}

cudaError_t LaunchLocalKernel(const LocalParams& p, cudaStream_t stream) {
  if (p.world_size < 1 || p.world_size > kMaxRanks || !LocalKernelTakes(p)) return cudaErrorInvalidValue;
  if (p.len_elements == 0) return cudaSuccess;
  const DType t = static_cast<DType>(p.dtype), w = static_cast<DType>(p.wire);
  if (t == DType::kFloat32 && w != t && p.op == LocalOp::kAllreduce) {
    if (w == DType::kBFloat16) return Launch<float, __nv_bfloat16, LocalOp::kAllreduce>(p, stream);
    if (w == DType::kFloat16) return Launch<float, __half, LocalOp::kAllreduce>(p, stream);
  }
  if (w != t) return cudaErrorInvalidValue;
  switch (t) {
    case DType::kFloat32: return LaunchTyped<float>(p, stream);
    case DType::kFloat16: return LaunchTyped<__half>(p, stream);
    case DType::kBFloat16: return LaunchTyped<__nv_bfloat16>(p, stream);
    case DType::kFloat64: return LaunchTyped<double>(p, stream);
    case DType::kInt32: return LaunchTyped<int>(p, stream);
    case DType::kInt64: return LaunchTyped<long long>(p, stream);
  }
  return cudaErrorInvalidValue;
}

}  // namespace ibcomm
