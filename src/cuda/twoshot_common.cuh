// Helpers of the two-shot allreduce kernel (nvls_kernel.cu): multimem accessors, vector copies, range splitting and
// the per-CTA cross-rank barrier.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdint>

#include "flags.cuh"
#include "kernels.h"
#include "vec_ops.cuh"

namespace ibcomm {
namespace dev {

constexpr int kNvlsThreads = 512;

template <typename T> struct Multimem {
  // Types without a multimem form (integers, fp64) only run the direct variant.
  __device__ __forceinline__ static uint4 LdReduce(const void*) { return make_uint4(0, 0, 0, 0); }
  __device__ __forceinline__ static void St(void*, uint4) {}
};

template <> struct Multimem<float> {
  __device__ __forceinline__ static uint4 LdReduce(const void* mc) {
    uint4 v;
    asm volatile("multimem.ld_reduce.relaxed.sys.global.add.v4.f32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(mc) : "memory");
    return v;
  }
  __device__ __forceinline__ static void St(void* mc, uint4 v) {
    asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(mc), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
  }
};
template <> struct Multimem<__half> {
  __device__ __forceinline__ static uint4 LdReduce(const void* mc) {
    uint4 v;
    asm volatile("multimem.ld_reduce.relaxed.sys.global.add.acc::f32.v4.f16x2 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(mc) : "memory");
    return v;
  }
  __device__ __forceinline__ static void St(void* mc, uint4 v) {
    asm volatile("multimem.st.relaxed.sys.global.v4.f16x2 [%0], {%1,%2,%3,%4};" ::"l"(mc), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
  }
};
template <> struct Multimem<__nv_bfloat16> {
  __device__ __forceinline__ static uint4 LdReduce(const void* mc) {
    uint4 v;
    asm volatile("multimem.ld_reduce.relaxed.sys.global.add.acc::f32.v4.bf16x2 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(mc) : "memory");
    return v;
  }
  __device__ __forceinline__ static void St(void* mc, uint4 v) {
    asm volatile("multimem.st.relaxed.sys.global.v4.bf16x2 [%0], {%1,%2,%3,%4};" ::"l"(mc), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
  }
};

// dst[b..e) = src[b..e) in 16-byte vectors, eight loads in flight per thread.
template <bool kStrongSrc>
__device__ __forceinline__ void CopyVectors(uint4* dst, const uint4* src, uint64_t b, uint64_t e) {
  constexpr int kU = 8;
  for (uint64_t i = b + threadIdx.x; i < e; i += static_cast<uint64_t>(blockDim.x) * kU) {
    uint4 v[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint64_t idx = i + static_cast<uint64_t>(u) * blockDim.x;
      if (idx < e) v[u] = kStrongSrc ? Ld16Strong(src + idx) : Ld16(src + idx);
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint64_t idx = i + static_cast<uint64_t>(u) * blockDim.x;
      if (idx < e) St16(dst + idx, v[u]);
    }
  }
}

// Units [b, e) of 16 bytes at `off` in every rank's buffer, summed in rank
// order (so the bits do not depend on who reduces), scaled, and handed to
// `store(index, value)`.  Peer loads are latency-bound: kU vectors per rank
// are in flight per thread, for at most kR ranks (kU * kR <= 8 keeps the
// loads in registers).
template <typename T, int kU, int kR, typename Store>
__device__ __forceinline__ void PeerReduceUnits(unsigned char* const* peer, int ws, uint64_t off, uint64_t b, uint64_t e,
                                                bool do_scale, double scale, Store store, unsigned tid, unsigned nthr) {
  using A = typename Acc<T>::type;
  constexpr int kVecElems = 16 / static_cast<int>(sizeof(T));
  for (uint64_t i = b + tid; i < e; i += static_cast<uint64_t>(nthr) * kU) {
    uint4 v[kU][kR];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint64_t idx = i + static_cast<uint64_t>(u) * nthr;
#pragma unroll
      for (int q = 0; q < kR; ++q)
        if (q < ws && idx < e) v[u][q] = Ld16Strong(peer[q] + off + idx * 16);
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint64_t idx = i + static_cast<uint64_t>(u) * nthr;
      if (idx < e) {
        A acc[kVecElems];
        VecIO<T>::Load(v[u][0], acc);
#pragma unroll
        for (int q = 1; q < kR; ++q)
          if (q < ws) VecIO<T>::Add(v[u][q], acc);
        if (do_scale) {
#pragma unroll
          for (int k = 0; k < kVecElems; ++k) acc[k] = ScaleAcc<A>(acc[k], scale);
        }
        store(idx, VecIO<T>::Store(acc));
      }
    }
  }
}

// ---- loads several rounds deep ----
// With one round of loads in registers a CTA waits a memory round trip per 64
// KiB, and more in registers spills, whether as a second buffer or as a second
// CTA per SM (8 ranks x 16 MiB of bf16: 68 us, 123 and more when spilling).
// Instead a thread's vectors of the coming rounds go to slots of its own in
// shared memory (`cp.async`, 16 bytes through L2): nothing but the thread's own
// wait orders them, and the depth costs no registers.  B200, in place: 8 ranks x
// 32 MiB fp32 113 -> 102 us, 2 x 64 MiB 76 -> 53 us (5.1 TB/s).
constexpr int kRoundVecs = 8;   // 16-byte vectors per thread and round
constexpr int kRoundDepth = 3;  // rounds in flight
constexpr size_t kRoundSmemPerThread = static_cast<size_t>(kRoundDepth) * kRoundVecs * 16;

__device__ __forceinline__ void CpAsync16(uint32_t smem_dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_dst), "l"(src) : "memory");
}
__device__ __forceinline__ void CpAsync16Hint(uint32_t smem_dst, const void* src, uint64_t policy) {
  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(smem_dst), "l"(src), "l"(policy) : "memory");
}
__device__ __forceinline__ void CpAsyncCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void CpAsyncWait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Ranges of items, walked one after the other in rounds of `step` items; a round
// belongs to one range.
struct OneRange {
  uint64_t b, e;
  __device__ __forceinline__ int count() const { return 1; }
  __device__ __forceinline__ uint64_t begin(int) const { return b; }
  __device__ __forceinline__ uint64_t end(int) const { return e; }
  __device__ __forceinline__ const unsigned char* data(int) const { return nullptr; }
};
template <typename Ranges>
struct RoundCursor {
  int q;
  uint64_t base, end;
  const unsigned char* at;
  __device__ __forceinline__ explicit RoundCursor(const Ranges& r) : q(0), base(r.begin(0)), end(r.end(0)), at(r.data(0)) { Settle(r); }
  __device__ __forceinline__ void Settle(const Ranges& r) {
    while (base >= end && ++q < r.count()) base = r.begin(q), end = r.end(q), at = r.data(q);
  }
  __device__ __forceinline__ void Next(const Ranges& r, uint64_t step) {
    base += step;
    Settle(r);
  }
  __device__ __forceinline__ bool Done(const Ranges& r) const { return q >= r.count(); }
};

// Where a part may start inside a line.
__device__ __forceinline__ void DropLine(const unsigned char* p) {
  if ((reinterpret_cast<uintptr_t>(p) & 127u) == 0) DiscardLine(p);
}
struct KeepLines {
  static constexpr bool kDrops = false;
  __device__ __forceinline__ void operator()(int, uint64_t) const {}
};
template <typename Fn>
struct DropLines {
  static constexpr bool kDrops = true;
  Fn fn;
  __device__ __forceinline__ void operator()(int v, uint64_t idx) const { fn(v, idx); }
};
template <typename Fn>
__device__ __forceinline__ DropLines<Fn> Dropping(Fn fn) {
  return DropLines<Fn>{fn};
}

// Every item of `ranges` over `nthr` threads numbered `tid`, kU items per thread
// and round, each of kRoundVecs / kU vectors: `issue(at, item, smem, stride)` starts
// the loads of one item of a range whose data lies at `at` into slots `smem`, `smem + stride`, ..., `use(item, slots,
// stride)` consumes it.  `smem`: kRoundSmemPerThread bytes for every thread of the
// block.  The loads run over the ends of ranges.  `drop(v, item)` is called for the
// vectors v of items item .. item + 7 when the warp has them: a round is 32 lines of 8
// vectors for a warp, one per lane.
template <int kU, typename Ranges, typename Issue, typename Use, typename Drop = KeepLines>
__device__ __forceinline__ void AsyncRounds(unsigned char* smem, const Ranges& ranges, unsigned tid, unsigned nthr, Issue issue, Use use, Drop drop = Drop()) {
  constexpr int kV = kRoundVecs / kU;
  static_assert(kRoundVecs == 8, "a line per lane");
  const uint64_t step = static_cast<uint64_t>(nthr) * kU;
  const uint32_t stride = blockDim.x * 16u, round_bytes = stride * kRoundVecs;
  unsigned char* const mine = smem + threadIdx.x * 16u;
  const uint32_t mine_u32 = static_cast<uint32_t>(__cvta_generic_to_shared(mine));
  RoundCursor<Ranges> in(ranges), out = in;
  uint32_t at = 0, ahead = 0;
  auto start = [&]() {
    if (!in.Done(ranges)) {
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const uint64_t idx = in.base + tid + static_cast<uint64_t>(u) * nthr;
        if (idx < in.end) issue(in.at, idx, mine_u32 + ahead + static_cast<uint32_t>(u * kV) * stride, stride);
      }
      in.Next(ranges, step);
    }
    CpAsyncCommit();
    ahead = ahead + round_bytes == kRoundDepth * round_bytes ? 0 : ahead + round_bytes;
  };
#pragma unroll
  for (int d = 0; d + 1 < kRoundDepth; ++d) start();
  while (!out.Done(ranges)) {
    start();
    CpAsyncWait<kRoundDepth - 1>();
    if constexpr (Drop::kDrops) {
      __syncwarp();  // every lane's loads of the round have landed
      const unsigned lane = threadIdx.x & 31u, chunk = lane / 4;
      const uint64_t idx = out.base + (tid - lane) + static_cast<uint64_t>(chunk / kV) * nthr + (lane & 3u) * 8;
      if (idx + 8 <= out.end) drop(static_cast<int>(chunk % kV), idx);
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint64_t idx = out.base + tid + static_cast<uint64_t>(u) * nthr;
      if (idx < out.end) use(idx, mine + at + static_cast<uint32_t>(u * kV) * stride, stride);
    }
    out.Next(ranges, step);
    at = at + round_bytes == kRoundDepth * round_bytes ? 0 : at + round_bytes;
  }
  CpAsyncWait<0>();
}

// PeerReduceUnits that way, by `nthr` threads numbered `tid`.
template <typename T, int kR, typename Store, typename Drop = KeepLines>
__device__ __forceinline__ void PeerReduce(unsigned char* smem, unsigned char* const* peer, int ws, uint64_t off, uint64_t b, uint64_t e,
                                           bool do_scale, double scale, Store store, unsigned tid, unsigned nthr, Drop drop = Drop()) {
  using A = typename Acc<T>::type;
  constexpr int kVecElems = 16 / static_cast<int>(sizeof(T));
  static_assert(kRoundVecs % kR == 0, "a round holds whole items");
  AsyncRounds<kRoundVecs / kR>(
      smem, OneRange{b, e}, tid, nthr,
      [&](const unsigned char*, uint64_t idx, uint32_t slot, uint32_t stride) {
#pragma unroll
        for (int q = 0; q < kR; ++q)
          if (q < ws) CpAsync16(slot + static_cast<uint32_t>(q) * stride, peer[q] + off + idx * 16);
      },
      [&](uint64_t idx, const unsigned char* slot, uint32_t stride) {
        A acc[kVecElems];
        VecIO<T>::Load(*reinterpret_cast<const uint4*>(slot), acc);
#pragma unroll
        for (int q = 1; q < kR; ++q)
          if (q < ws) VecIO<T>::Add(*reinterpret_cast<const uint4*>(slot + static_cast<uint32_t>(q) * stride), acc);
        if (do_scale) {
#pragma unroll
          for (int k = 0; k < kVecElems; ++k) acc[k] = ScaleAcc<A>(acc[k], scale);
        }
        store(idx, VecIO<T>::Store(acc));
      },
      drop);
}

// The kernels are compiled per world-size class kR (2, 4 or 8 ranks at most)
// with 8 / kR vectors in flight per rank: 2 ranks x 4 vectors, 4 x 2, 8 x 1.
// Loads in registers, by `nthr` threads of a CTA, numbered `tid` = 0 .. nthr - 1.
template <typename T, int kR, typename Store>
__device__ __forceinline__ void PeerReduceGroup(unsigned char* const* peer, int ws, uint64_t off, uint64_t b, uint64_t e,
                                                bool do_scale, double scale, Store store, unsigned tid, unsigned nthr) {
  PeerReduceUnits<T, kMaxRanks / kR, kR>(peer, ws, off, b, e, do_scale, scale, store, tid, nthr);
}
inline int RankClass(int world_size) { return world_size <= 2 ? 2 : (world_size <= 4 ? 4 : kMaxRanks); }

// Barrier between CTA `cta` of every rank.  Returns false when it gave up.
__device__ inline bool CrossRankBarrier(const PeerTable& peers, const WaitCtx& w, int cta, uint32_t phase, int* s_stop) {
  __syncthreads();
  const uint64_t val = (w.seq << 32) | phase;
  if (threadIdx.x < w.world_size && static_cast<int>(threadIdx.x) != w.rank) {
    // The release store orders everything this CTA wrote before the barrier
    // (observed by this thread through __syncthreads) ahead of the flag.
    StReleasePeers(&Ctl(peers, threadIdx.x)->bar[cta][w.rank], val, peers.one_gpu != 0);
    if (!WaitGE(&Ctl(peers, w.rank)->bar[cta][threadIdx.x], val, w, kWaitBarrier, threadIdx.x, static_cast<int>(phase)))
      *s_stop = 1;
  }
  __syncthreads();
  return *s_stop == 0;
}

template <typename T> struct HasMultimem { static constexpr bool value = false; };
template <> struct HasMultimem<float> { static constexpr bool value = true; };
template <> struct HasMultimem<__half> { static constexpr bool value = true; };
template <> struct HasMultimem<__nv_bfloat16> { static constexpr bool value = true; };

}  // namespace dev
}  // namespace ibcomm
