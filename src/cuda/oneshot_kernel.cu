// One-shot allreduce for small messages: every rank stores its whole message
// into a slot of every peer's arena, raises one flag per peer, waits for the
// peers' flags and sums the world_size copies locally in rank order (so every
// rank computes bit-identical results).  One NVLink hop instead of the
// 2*(ws-1) hops of the ring: this is the latency end of the size sweep, for
// which the reference has no dedicated path.
//
// The slots are double-buffered by the parity of the call number, so
// consecutive calls need no exit barrier: a peer can only reach call k+2 after
// it consumed this rank's data of call k+1, which this rank sent after it had
// finished reading call k.
#include "flags.cuh"
#include "ibcomm/communicator.h"
#include "kernels.h"
#include "vec_ops.cuh"

namespace ibcomm {
namespace dev {

constexpr int kOneShotThreads = 512;

// Body of the one-shot kernel for one CTA; returns early when a wait gave up.
template <typename T>
__device__ void OneShotBody(const OneShotParams& p, uint64_t seq, int& s_stop) {
  using A = typename Acc<T>::type;
  constexpr int kVecElems = 16 / static_cast<int>(sizeof(T));
  const int cta = blockIdx.x, ncta = gridDim.x;
  const int ws = p.world_size, me = p.rank;
  // Slots are double-buffered by the parity of the call number; two one-shot
  // calls with the same parity always have another collective (with its entry
  // barrier) or a one-shot call of the other parity between them.
  const unsigned parity = static_cast<unsigned>(seq & 1u);
  const T* sendbuf = static_cast<const T*>(p.sendbuf);
  T* recvbuf = static_cast<T*>(p.recvbuf);

  WaitCtx w;
  w.peers = &p.peers;
  w.status = p.status;
  w.doorbell = p.doorbell;
  w.seq = seq;
  w.timeout_ns = p.timeout_ns;
  w.rank = me;
  w.world_size = ws;
  w.channel = cta;

  // This CTA's element range, on 16-byte vector boundaries.
  uint64_t lo, hi;
  {
    const uint64_t nvec = (p.len_elements + kVecElems - 1) / kVecElems;
    const uint64_t per = (nvec + static_cast<uint64_t>(ncta) - 1) / static_cast<uint64_t>(ncta);
    lo = per * static_cast<uint64_t>(cta) * kVecElems;
    hi = lo + per * kVecElems;
    if (lo > p.len_elements) lo = p.len_elements;
    if (hi > p.len_elements) hi = p.len_elements;
  }
  auto slot = [&](int owner_rank, int src_rank) -> T* {
    return reinterpret_cast<T*>(p.peers.arena[owner_rank] + p.slot_offset +
                                (static_cast<uint64_t>(parity) * static_cast<uint64_t>(ws) + static_cast<uint64_t>(src_rank)) * p.slot_bytes);
  };
  // Slots are 16-byte aligned and so is `lo`; a user buffer may be only
  // element-aligned, then its side of a vector goes element by element.
  const unsigned char* const mine = reinterpret_cast<const unsigned char*>(sendbuf + lo);
  unsigned char* const out = reinterpret_cast<unsigned char*>(recvbuf + lo);
  const bool send_aligned = (reinterpret_cast<uintptr_t>(mine) & 15u) == 0, recv_aligned = (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  const uint64_t nfull = (hi - lo) / kVecElems;
  const uint64_t ragged = lo + nfull * kVecElems;

  // (1) push my slice to every peer: read once, stored ws - 1 times, starting
  // with a different peer on every rank.
  constexpr int kU = 4;  // vectors in flight per thread
  for (uint64_t i = threadIdx.x; i < nfull; i += static_cast<uint64_t>(blockDim.x) * kU) {
    uint4 v[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint64_t idx = i + static_cast<uint64_t>(u) * blockDim.x;
      if (idx < nfull) v[u] = LdUser16<T>(mine + idx * 16, send_aligned);
    }
    for (int k = 1; k < ws; ++k) {
      const int q = me + k < ws ? me + k : me + k - ws;
      uint4* const dst = reinterpret_cast<uint4*>(slot(q, me) + lo);
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const uint64_t idx = i + static_cast<uint64_t>(u) * blockDim.x;
        if (idx < nfull) St16(dst + idx, v[u]);
      }
    }
  }
  for (uint64_t i = ragged + threadIdx.x; i < hi; i += blockDim.x)
    for (int q = 0; q < ws; ++q)
      if (q != me) slot(q, me)[i] = sendbuf[i];
  __syncthreads();
  // (2) tell them, (3) wait for theirs.
  if (threadIdx.x < ws && static_cast<int>(threadIdx.x) != me) {
    const int q = threadIdx.x;
    StReleasePeers(&Ctl(p.peers, q)->oneshot_flag[parity][cta][me], seq, p.peers.one_gpu != 0);  // release: the pushes above come first
    if (!WaitGE(&Ctl(p.peers, me)->oneshot_flag[parity][cta][q], seq, w, kWaitOneShot, q, -1)) s_stop = 1;
  }
  __syncthreads();
  if (s_stop) return;
  // (4) sum in rank order, every rank's vector in flight.
  const bool do_scale = p.scale != 1.0;
  for (uint64_t i = threadIdx.x; i < nfull; i += blockDim.x) {
    uint4 v[kMaxRanks];
#pragma unroll
    for (int q = 0; q < kMaxRanks; ++q)
      if (q < ws) v[q] = (q == me) ? LdUser16<T>(mine + i * 16, send_aligned) : Ld16Strong(reinterpret_cast<const uint4*>(slot(me, q) + lo) + i);
    A acc[kVecElems];
    VecIO<T>::Load(v[0], acc);
#pragma unroll
    for (int q = 1; q < kMaxRanks; ++q)
      if (q < ws) VecIO<T>::Add(v[q], acc);
    if (do_scale) {
#pragma unroll
      for (int e = 0; e < kVecElems; ++e) acc[e] = ScaleAcc<A>(acc[e], p.scale);
    }
    StUser16<T>(out + i * 16, VecIO<T>::Store(acc), recv_aligned);
  }
  for (uint64_t i = ragged + threadIdx.x; i < hi; i += blockDim.x) {
    A acc = A(0);
    for (int q = 0; q < ws; ++q) acc += (q == me) ? ToAcc<A, T>(sendbuf[i]) : ToAcc<A, T>(LdScalarStrong<T>(slot(me, q) + i));
    if (do_scale) acc = ScaleAcc<A>(acc, p.scale);
    recvbuf[i] = FromAcc<T, A>(acc);
  }
}

template <typename T>
__global__ void __launch_bounds__(kOneShotThreads, 1)
OneShotKernel(const __grid_constant__ RankBlocks<OneShotParams> all) {
  const OneShotParams& p = all.rank[blockIdx.y];
  __shared__ int s_stop;
  __shared__ uint64_t s_seq;
  if (threadIdx.x == 0) s_stop = 0;
  const uint64_t seq = BeginCollective(p.peers, p.rank, &s_seq, gridDim.x);
  OneShotBody<T>(p, seq, s_stop);
}

}  // namespace dev

template <typename T>
static cudaError_t LaunchOneShotTyped(const OneShotParams* ranks, int n, int blocks, cudaStream_t stream) {
  return LaunchRanks(dev::OneShotKernel<T>, ranks, n, blocks, dev::kOneShotThreads, 0, stream);
}

cudaError_t LaunchOneShotKernel(const OneShotParams* ranks, int n, int blocks, cudaStream_t stream) {
  switch (static_cast<DType>(ranks->dtype)) {
    case DType::kFloat32: return LaunchOneShotTyped<float>(ranks, n, blocks, stream);
    case DType::kFloat64: return LaunchOneShotTyped<double>(ranks, n, blocks, stream);
    case DType::kInt32: return LaunchOneShotTyped<int>(ranks, n, blocks, stream);
    case DType::kInt64: return LaunchOneShotTyped<long long>(ranks, n, blocks, stream);
    case DType::kFloat16: return LaunchOneShotTyped<__half>(ranks, n, blocks, stream);
    case DType::kBFloat16: return LaunchOneShotTyped<__nv_bfloat16>(ranks, n, blocks, stream);
  }
  return cudaErrorInvalidValue;
}

}  // namespace ibcomm
