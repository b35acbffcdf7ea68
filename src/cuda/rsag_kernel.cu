// Reduce-scatter and all-gather: the two halves of the two-shot allreduce as
// collectives of their own (block r of the message belongs to rank r).  The
// reference has neither (its ring runs them back to back inside
// AllreduceRing, allreduce_cpu_impl.h:23-244); they are what tensor-, sequence-
// and fully-sharded data parallel code consumes.
//
//   reduce-scatter  in: ws blocks of m elements per rank   out: m elements
//                   rank r sums block r of every rank (switch `multimem.ld_reduce`,
//                   or peer loads added in rank order), scales, stores locally.
//   all-gather      in: m elements per rank                out: ws blocks of m
//                   rank r writes its block into block r of every rank's output
//                   (`multimem.st`, or one peer store per rank).
//
// The remote side (the input of a reduce-scatter, the output of an
// all-gather) is either a buffer every rank has mapped (symmetric memory or a
// registered buffer), used in place, or the arena's pool: then the message
// moves window by window, a window holding ws sub-blocks side by side, with
// the local copies in the same kernel.  CTA b always handles part b of every
// sub-block, on every rank and in every window, so the barriers are per CTA.
//
// Work is split in units of 16 bytes of the REMOTE side, which is what crosses
// the links: in the pool every sub-block starts on a boundary; in a mapped
// buffer block r starts wherever r * block_bytes falls, and the elements before
// its first boundary go one by one.  The last unit of a block may be short.  The
// local side of a unit (a user buffer, only element-aligned in general) is
// accessed element by element where it has to be.  Blocks of an odd length moved
// one element at a time took 311 us to scatter and 278 us to gather (8 ranks x 16
// MiB of bf16 on one B200); by units 58 and 54 us.
#include "flags.cuh"
#include "ibcomm/communicator.h"
#include "kernels.h"
#include "twoshot_common.cuh"
#include "vec_ops.cuh"

namespace ibcomm {
namespace dev {

template <typename T, bool kMultimem, int kR>
__device__ void RsAgBody(const RsAgParams& p, uint64_t seq, int& s_stop, unsigned char* smem) {
  using A = typename Acc<T>::type;
  constexpr uint64_t kE = sizeof(T);
  constexpr int kUnitElems = 16 / static_cast<int>(sizeof(T));
  constexpr int kU = 4;  // units in flight per thread of the copies
  const int cta = blockIdx.x, ncta = gridDim.x;
  const int ws = p.world_size, me = p.rank;
  WaitCtx w;
  w.peers = &p.peers;
  w.status = p.status;
  w.doorbell = p.doorbell;
  w.seq = seq;
  w.timeout_ns = p.timeout_ns;
  w.rank = me;
  w.world_size = ws;
  w.channel = cta;
  const unsigned char* send = static_cast<const unsigned char*>(p.sendbuf);
  unsigned char* recv = static_cast<unsigned char*>(p.recvbuf);
  const bool do_scale = p.scale != 1.0;
  const uint64_t step = blockDim.x;
  uint32_t phase = 0;

  // Entry: CTA `cta` of every rank has started this call, so whatever used the
  // pool or the peers' buffers before it is over.
  if (!CrossRankBarrier(p.peers, w, cta, ++phase, &s_stop)) return;

  for (uint64_t w0 = 0; w0 < p.block_elems; w0 += p.window_elems) {
    const uint64_t wn = (p.block_elems - w0 < p.window_elems) ? p.block_elems - w0 : p.window_elems;
    const bool last = w0 + wn >= p.block_elems;
    // My sub-block of the remote side, and the elements before its first boundary.
    const uint64_t mine = static_cast<uint64_t>(me) * p.sub_stride_bytes + (p.staged ? 0 : w0 * kE);
    uint64_t head = ((16 - ((reinterpret_cast<uintptr_t>(p.peer_buf[me]) + mine) & 15u)) & 15u) / kE;
    if (head > wn) head = wn;
    const uint64_t full = (wn - head) / kUnitElems;         // whole units
    const uint64_t rest = (wn - head) - full * kUnitElems;  // elements of the short one
    const uint64_t units = full + (rest != 0 ? 1 : 0);
    uint64_t b, e;
    WindowPart(p.staged ? (p.window_elems + kUnitElems - 1) / kUnitElems : units, units, 0, 1, cta, ncta, &b, &e);
    const uint64_t ev = e < full ? e : full;
    // Single elements of this CTA, by their place behind `head`: the short unit
    // (by the CTA that owns it in every window) and, by CTA 0, the head.
    auto each_element = [&](auto fn) {
      if (rest != 0 && b <= full && full < e && threadIdx.x < rest) fn(static_cast<int64_t>(full * kUnitElems + threadIdx.x));
      if (cta == 0 && threadIdx.x < head) fn(static_cast<int64_t>(threadIdx.x) - static_cast<int64_t>(head));
    };
    // Units [b, ev) from `src` to one or several places; the next round's loads
    // are on their way while this one's values are stored.
    auto copy_units = [&](const unsigned char* src, bool strong, auto store) {
      const bool src_aligned = (reinterpret_cast<uintptr_t>(src) & 15u) == 0;
      uint4 next[kU];
      auto load = [&](uint64_t i) {
#pragma unroll
        for (int u = 0; u < kU; ++u)
          if (i + u * step < ev) next[u] = strong ? Ld16Strong(src + (i + u * step) * 16) : LdUser16<T>(src + (i + u * step) * 16, src_aligned);
      };
      load(b + threadIdx.x);
      for (uint64_t i = b + threadIdx.x; i < ev; i += step * kU) {
        uint4 v[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) v[u] = next[u];
        load(i + step * kU);
#pragma unroll
        for (int u = 0; u < kU; ++u)
          if (i + u * step < ev) store(i + u * step, v[u]);
      }
    };

    if (p.mode == kRsAgReduceScatter) {
      if (p.staged) {
        // Copy my part of every sub-block into my pool window (there is no head in the pool).
        for (int s = 0; s < ws; ++s) {
          const unsigned char* src = send + (static_cast<uint64_t>(s) * p.block_elems + w0) * kE;
          unsigned char* dst = p.peer_buf[me] + static_cast<uint64_t>(s) * p.sub_stride_bytes;
          copy_units(src, false, [&](uint64_t i, uint4 v) { St16(dst + i * 16, v); });
          each_element([&](int64_t k) { reinterpret_cast<T*>(dst)[k] = reinterpret_cast<const T*>(src)[k]; });
        }
        if (!CrossRankBarrier(p.peers, w, cta, ++phase, &s_stop)) return;
      }
      const uint64_t off = mine + head * kE;
      unsigned char* out = recv + (w0 + head) * kE;
      const bool out_aligned = (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
      if constexpr (kMultimem) {
        for (uint64_t i = b + threadIdx.x; i < ev; i += step) {
          uint4 r = Multimem<T>::LdReduce(p.mc_buf + off + i * 16);
          if (do_scale) {
            A acc[kUnitElems];
            VecIO<T>::Load(r, acc);
#pragma unroll
            for (int k = 0; k < kUnitElems; ++k) acc[k] = ScaleAcc<A>(acc[k], p.scale);
            r = VecIO<T>::Store(acc);
          }
          StUser16<T>(out + i * 16, r, out_aligned);
        }
      } else {
        PeerReduce<T, kR>(smem, p.peer_buf, ws, off, b, ev, do_scale, p.scale,
                          [&](uint64_t idx, uint4 r) { StUser16<T>(out + idx * 16, r, out_aligned); }, threadIdx.x, blockDim.x);
        each_element([&](int64_t k) {
          A acc = A(0);
          for (int q = 0; q < ws; ++q) acc += ToAcc<A, T>(LdScalarStrong<T>(reinterpret_cast<const T*>(p.peer_buf[q] + off) + k));
          if (do_scale) acc = ScaleAcc<A>(acc, p.scale);
          reinterpret_cast<T*>(out)[k] = FromAcc<T, A>(acc);
        });
      }
      // The peers have read my window (my buffer): it may be overwritten.
      if (!CrossRankBarrier(p.peers, w, cta, ++phase, &s_stop)) return;
    } else {
      // All-gather: my part of the window goes into sub-block `me` everywhere.
      const unsigned char* src = send + (w0 + head) * kE;
      const uint64_t off = mine + head * kE;
      copy_units(src, false, [&](uint64_t i, uint4 v) {
        if constexpr (kMultimem) {
          Multimem<T>::St(p.mc_buf + off + i * 16, v);
        } else {
#pragma unroll
          for (int q = 0; q < kR; ++q)
            if (q < ws) St16(p.peer_buf[q] + off + i * 16, v);
        }
      });
      if constexpr (!kMultimem) {
        each_element([&](int64_t k) {
          const T v = reinterpret_cast<const T*>(src)[k];
          for (int q = 0; q < ws; ++q) reinterpret_cast<T*>(p.peer_buf[q] + off)[k] = v;
        });
      }
      // Everybody's part `cta` has arrived here.
      if (!CrossRankBarrier(p.peers, w, cta, ++phase, &s_stop)) return;
      if (p.staged) {
        for (int s = 0; s < ws; ++s) {
          const unsigned char* from = p.peer_buf[me] + static_cast<uint64_t>(s) * p.sub_stride_bytes;
          unsigned char* to = recv + (static_cast<uint64_t>(s) * p.block_elems + w0) * kE;
          const bool to_aligned = (reinterpret_cast<uintptr_t>(to) & 15u) == 0;
          copy_units(from, true, [&](uint64_t i, uint4 v) { StUser16<T>(to + i * 16, v, to_aligned); });
          each_element([&](int64_t k) { reinterpret_cast<T*>(to)[k] = LdScalarStrong<T>(reinterpret_cast<const T*>(from) + k); });
        }
        // My window is free again before anybody writes the next one into it.
        if (!last && !CrossRankBarrier(p.peers, w, cta, ++phase, &s_stop)) return;
      }
    }
  }
}

template <typename T, bool kMultimem, int kR>
__global__ void __launch_bounds__(kNvlsThreads, 1) RsAgKernel(const __grid_constant__ RankBlocks<RsAgParams> all) {
  extern __shared__ __align__(128) unsigned char smem[];
  const RsAgParams& p = all.rank[blockIdx.y];
  __shared__ int s_stop;
  __shared__ uint64_t s_seq;
  if (threadIdx.x == 0) s_stop = 0;
  const uint64_t seq = BeginCollective(p.peers, p.rank, &s_seq, gridDim.x);
  RsAgBody<T, kMultimem, kR>(p, seq, s_stop, smem);
}

}  // namespace dev

template <typename T, bool kMultimem, int kR>
static cudaError_t LaunchRsAgU(const RsAgParams* ranks, int n, int blocks, cudaStream_t stream) {
  const size_t smem = kMultimem || ranks->mode != kRsAgReduceScatter ? 0 : dev::kRoundSmemPerThread * dev::kNvlsThreads;
  if (smem != 0) {
    const cudaError_t e = AllowSharedMemory(dev::RsAgKernel<T, kMultimem, kR>, smem);
    if (e != cudaSuccess) return e;
  }
  return LaunchRanks(dev::RsAgKernel<T, kMultimem, kR>, ranks, n, blocks, dev::kNvlsThreads, smem, stream);
}

template <typename T>
static cudaError_t LaunchRsAgTyped(const RsAgParams* ranks, int n, int blocks, cudaStream_t stream) {
  if (ranks->use_multimem) {
    if constexpr (dev::HasMultimem<T>::value) {
      if ((ranks->block_elems * sizeof(T)) % 16 != 0) return cudaErrorInvalidValue;
      return LaunchRsAgU<T, true, kMaxRanks>(ranks, n, blocks, stream);
    } else {
      return cudaErrorInvalidValue;
    }
  }
  // Peer loads: compiled per world-size class (loads in flight per rank).
  switch (dev::RankClass(ranks->world_size)) {
    case 2: return LaunchRsAgU<T, false, 2>(ranks, n, blocks, stream);
    case 4: return LaunchRsAgU<T, false, 4>(ranks, n, blocks, stream);
    default: return LaunchRsAgU<T, false, kMaxRanks>(ranks, n, blocks, stream);
  }
}

cudaError_t LaunchRsAgKernel(const RsAgParams* ranks, int n, int blocks, cudaStream_t stream) {
  switch (static_cast<DType>(ranks->dtype)) {
    case DType::kFloat32: return LaunchRsAgTyped<float>(ranks, n, blocks, stream);
    case DType::kFloat16: return LaunchRsAgTyped<__half>(ranks, n, blocks, stream);
    case DType::kBFloat16: return LaunchRsAgTyped<__nv_bfloat16>(ranks, n, blocks, stream);
    case DType::kFloat64: return LaunchRsAgTyped<double>(ranks, n, blocks, stream);
    case DType::kInt32: return LaunchRsAgTyped<int>(ranks, n, blocks, stream);
    case DType::kInt64: return LaunchRsAgTyped<long long>(ranks, n, blocks, stream);
  }
  return cudaErrorInvalidValue;
}

}  // namespace ibcomm
