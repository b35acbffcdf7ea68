// Generic executor of op programs (ring and Rabenseifner allreduce).
//
// One CTA per channel.  A CTA walks the rank's program; for every op it waits
// (bounded) for the peer's data flag and for slot credit, streams its slice of
// the chunk through shared memory and, as 16-byte vectors, registers
//     staging slot / sendbuf / recvbuf  (+ sendbuf|recvbuf) (* scale) (cast)
//         -> recvbuf and/or the next peer's staging slot over NVLink,
// then publishes the data flag to the receiver and returns the credit to the
// sender.  No host round trip and no separate reduce, cast or scale kernel.
//
// The CTA is warp-specialised so that neither the synchronisation of an op nor
// the latency of its loads stops the stream of the next one:
//   waiter  (a warp)    looks at the peers' data flags and slot credits and runs
//                       ahead through the program as far as they allow;
//   loader  (a warp)    fills a ring of shared-memory stages with bulk copies
//                       (`cp.async.bulk`, this GPU's memory only) of the ops'
//                       sources, several stages and hence several ops ahead: what
//                       lies in sendbuf is fetched before the op's flag is there;
//   data warps          take stage after stage in order: read, add, scale, cast,
//                       store; no barrier among them;
//   poster  (a warp)    follows behind, fences the stores of finished ops and
//                       publishes their flags, one fence for all ops that are done.
// They hand over through counters and mbarriers in shared memory.
//
// A rank's rate is bound by the bytes its CTAs have in flight: with loads into
// registers (two groups of warps taking the ops in turn, 14 KiB each) a CTA
// moved 10-15 GB/s whether the data came from L2 or from HBM; the ring keeps
// 100 KiB (fp32) ahead of the data warps across op boundaries.  Per op, what is
// left in series (flags, plan, fence) takes about 1.2 us, and a hand-over
// between two ranks on one GPU about 3 us.  User data that is touched once goes
// through L2 as evict-first, so that the staging slots of ranks sharing a GPU
// stay there (ring 8 x 256 MiB 1.38 -> 1.23 ms, called in a loop; 1.30-1.38 with other
// work between the calls).  A slot's line has one reader;
// with `drop_lines` the data warps drop it from L2 when the stage's copy has landed,
// and the poster's fence orders that ahead of the credit that frees the slot, so
// that dead data is not written to HBM (not the ring's, whose slots stay in L2: 8 x
// 256 MiB 1.23 -> 1.25 ms).  Ranks sharing a B200, before and after:
// Rabenseifner 5 x 64 MiB 908 -> 430 us, ring 8 x 32 MiB 258 -> 192 us, ring 7 x 4
// MB 96 -> 70 us, ring 8 x 4 KiB 52 -> 46 us.
// Programs of ranks that share a GPU (kShared) have ops with one to three sources, some
// of them other ranks' buffers, and store into other ranks' recvbuf; a stage takes as many
// packs as fit with that many sources.  5 ranks x 64 MiB Rabenseifner 271 -> 158 us, 7 x 64
// MiB 458 -> 227, ring 2 x 64 MiB 71 -> 56.  The extra rank's work, the first step's sends
// and the results' slots are gone: of 5 ranks 60 block reads and writes a segment instead of 128.
// Counterpart of the reference's host event loop around _reduce_inplace_cuda
// (ibcomm/allreduce_cuda_impl.h:24-33, 103-299, 470-707).
//
// The grid is (channels, ranks): blockIdx.y selects the rank whose parameters
// to use, so that several ranks that share one GPU run as ONE cooperative
// launch (CTAs that wait on each other are co-resident).
#include <algorithm>

#include "exec_common.cuh"
#include "flags.cuh"
#include "ibcomm/communicator.h"
#include "ibcomm/tunables.h"
#include "kernels.h"
#include "tma_stage.cuh"
#include "vec_ops.cuh"
#include "warp_roles.cuh"

namespace ibcomm {
namespace dev {

constexpr int kExecServiceWarps = 3;  // waiter, loader, poster
constexpr int kExecMaxStages = 10;
// A stage holds U packs per data thread from each of two sources: 128 bytes per data thread
// for every pair of types.  Where ranks share a GPU it takes 2 U from one source (5 ranks x
// 64 MiB Rabenseifner 160 -> 157 us; the ring of ranks that send 3 % slower) and U / 2 from three.
// Half of that leaves a warp waiting for its own shared-memory reads (5 ranks x 64 MiB
// Rabenseifner 496 us against 430).
constexpr int kExecStageBytesPerThread = 128;

enum ExecTileFlags : uint32_t {
  kTileFromStaging = 1,  // source a is in the wire type
  kTileAdd = 2,          // source b is present
  kTileScale = 4,
  kTileRoundWire = 8,
  kTileLastOfOp = 16,
  kTileElements = 32,  // nothing in the stage: elements [lo, hi) of the op's cell, one by one
  kTileExit = 64,      // the program is over
  kTileReadBack = 128,  // the local store is read back by a later op
  kTileThird = 256,     // source c is present
  kTileRoundPeer = 512,  // source c, and a unless it is from staging, are rounded through the wire type
  kTilePeersReadBack = 1024,  // what goes into other ranks' recvbuf is read there by a later op
  kTilePeersShift = 16,  // from here up: the ranks whose recvbuf the value goes into, a bit each
};
// What there is of a stage and of an op only where ranks share a GPU.
template <bool kShared>
struct ExecTileMore {};
template <>
struct ExecTileMore<true> {
  const unsigned char* tail_c;
  uint64_t recv_off;  // where the first pack lies in every recvbuf, in bytes
  uint32_t stride;    // 16-byte vectors of the stage from one source to the next
};
template <bool kShared>
struct ExecPlanMore {};
template <>
struct ExecPlanMore<true> {
  const unsigned char* src_c;
  uint64_t recv_off;
  uint32_t late;  // source a is another rank's work: it is there when the op's flags are
};

// What the data warps do with one stage.
template <bool kShared>
struct ExecTile : ExecTileMore<kShared> {
  uint4* local;   // recvbuf, or null
  uint4* remote;  // the next rank's staging slot, or null
  uint32_t packs;  // the one with only `tail` elements included
  uint32_t flags;
  uint32_t op;
  uint32_t tail;  // elements of the last pack, 0 = it is whole
  uint64_t lo, hi;
  const unsigned char* tail_a;  // where the last pack lies in the user's buffers
  const unsigned char* tail_b;
  // Whole lines of the staging slot that the stage came from, to be dropped from L2.
  unsigned char* drop;
  uint32_t drop_lines;
};

// One op of this channel, worked out by a lane of the loader's warp.
template <bool kShared>
struct ExecPlan : ExecPlanMore<kShared> {
  const unsigned char* src_a;  // address of the first pack (for staging: in the wire type)
  const unsigned char* src_b;
  unsigned char* local;
  unsigned char* remote;
  uint64_t packs;      // packs, the last one with only `tail` elements unless `tail` is 0
  uint64_t lo, hi;     // elements [lo, hi) of the cell go one by one (nothing is in packs then)
  uint32_t flags;      // ExecTileFlags of every stage of the op
  uint32_t wait_local;
  uint32_t tail;
  uint32_t pad_;
};

template <bool kShared>
struct ExecShared {
  RoleSync role;  // ready: ops whose flags have arrived; done[w]: ops whose stores data warp w has issued
  ExecTile<kShared> tile[kExecMaxStages];
  ExecPlan<kShared> plan[32];
  uint64_t full[kExecMaxStages];   // the stage's copies have landed and its op may store
  uint64_t empty[kExecMaxStages];  // every data warp has read the stage
};

// Waits for a phase of one of the ring's mbarriers.  The party that completes
// it is in this CTA and itself bounded, so the limit is a safety net.
__device__ __forceinline__ bool RingWait(uint64_t* bar, uint32_t parity, RoleSync* sync, uint64_t timeout_ns) {
  if (MbarTryWait(bar, parity)) return true;
  const uint64_t t0 = GlobalTimerNs();
  for (;;) {
    if (MbarTryWait(bar, parity)) return true;
    if (GlobalTimerNs() - t0 > 3 * timeout_ns) {
      *reinterpret_cast<volatile int*>(&sync->stop) = 1;
      return false;
    }
  }
}

// The last pack of a message that ends inside it: `staged` is its place in the
// stage when source a comes from staging; the user's buffers are accessed up to
// the message's end.  A slot's pack is written whole: it lies in this channel's
// part of the slot, and nobody reads past the message's end either.
template <typename T, typename W, bool kShared>
__device__ __noinline__ void RunTailPack(const ExecTile<kShared>* t, const uint4* staged, const ExecParams& p) {
  using Tr = ExecTraits<T, W>;
  using A = typename Tr::A;
  constexpr int P = Tr::P;
  const int n = static_cast<int>(t->tail);
  A acc[P];
#pragma unroll
  for (int v = 0; v < Tr::VW; ++v)
    if (t->flags & kTileFromStaging) VecIO<W>::Load(staged[v], acc + v * VecIO<W>::kN);
  const bool round_peer = kShared && (t->flags & kTileRoundPeer) && sizeof(W) != sizeof(T);
#pragma unroll
  for (int e = 0; e < P; ++e) {
    if (!(t->flags & kTileFromStaging)) {
      acc[e] = e < n ? ToAcc<A, T>(reinterpret_cast<const T*>(t->tail_a)[e]) : A(0);
      if (round_peer) acc[e] = ThroughWire<W, A>(acc[e]);
    }
    if constexpr (kShared) {
      if ((t->flags & kTileThird) && e < n) {
        const A c = ToAcc<A, T>(reinterpret_cast<const T*>(t->tail_c)[e]);
        acc[e] += round_peer ? ThroughWire<W, A>(c) : c;
      }
    }
    if ((t->flags & kTileAdd) && e < n) acc[e] += ToAcc<A, T>(reinterpret_cast<const T*>(t->tail_b)[e]);
    if (t->flags & kTileScale) acc[e] = ScaleAcc<A>(acc[e], p.scale);
  }
  uint4 wq[Tr::VW];
#pragma unroll
  for (int v = 0; v < Tr::VW; ++v) wq[v] = VecIO<W>::Store(acc + v * VecIO<W>::kN);
  const uint32_t at = t->packs - 1;
  if (t->remote != nullptr) {
#pragma unroll
    for (int v = 0; v < Tr::VW; ++v) St16(t->remote + at * Tr::VW + v, wq[v]);
  }
  if ((t->flags & kTileRoundWire) && sizeof(W) != sizeof(T)) {
#pragma unroll
    for (int v = 0; v < Tr::VW; ++v) VecIO<W>::Load(wq[v], acc + v * VecIO<W>::kN);
  }
  auto store = [&](T* out) {
#pragma unroll
    for (int e = 0; e < P; ++e)
      if (e < n) out[e] = FromAcc<T, A>(acc[e]);
  };
  if (t->local != nullptr) store(reinterpret_cast<T*>(t->local + at * Tr::VT));
  if constexpr (kShared) {
    for (int q = 0; q < p.world_size; ++q)
      if (t->flags >> (kTilePeersShift + q) & 1u) store(reinterpret_cast<T*>(static_cast<unsigned char*>(p.peer_recv[q]) + t->recv_off + static_cast<uint64_t>(at) * Tr::VT * 16u));
  }
}

// One stage: packs of P elements, U of them per thread and turn.  `tile` is `t` in shared memory.
template <typename T, typename W, bool kShared>
__device__ __forceinline__ void RunTile(const ExecTile<kShared>& t, const ExecTile<kShared>* tile, const uint4* stage, const ExecParams& p, uint64_t* empty,
                                        uint64_t read_back_policy, uint64_t final_policy, unsigned tid, unsigned nthr, int lane) {
  using Tr = ExecTraits<T, W>;
  using A = typename Tr::A;
  constexpr int P = Tr::P, U = Tr::U, VT = Tr::VT, VW = Tr::VW;
  constexpr bool kCasts = sizeof(W) != sizeof(T);
  const bool from_staging = (t.flags & kTileFromStaging) != 0, add = (t.flags & kTileAdd) != 0, third = kShared && (t.flags & kTileThird) != 0;
  const bool round_peer = kShared && kCasts && (t.flags & kTileRoundPeer) != 0, round_wire = kCasts && (t.flags & kTileRoundWire) != 0;
  const uint32_t whole = t.packs - (t.tail != 0 ? 1u : 0u);
  uint32_t peers = 0, stride = nthr * U * VT;
  uint64_t recv_off = 0;
  if constexpr (kShared) peers = t.flags >> kTilePeersShift, stride = t.stride, recv_off = t.recv_off;
  const uint64_t local_policy = (t.flags & kTileReadBack) ? read_back_policy : final_policy;
  const uint64_t peers_policy = (t.flags & kTilePeersReadBack) ? read_back_policy : final_policy;
  for (unsigned l = tid; l < t.drop_lines; l += nthr) DiscardLine(t.drop + static_cast<size_t>(l) * 128u);
  // One turn, or two where there is one source.
  unsigned at = tid;
  for (bool more = true; more; at += U * nthr) {
    more = kShared && at - tid + U * nthr < whole;  // else a stage holds one turn
    uint4 qa[U][VT], qb[U][VT], qc[U / 2][VT];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned i = at + static_cast<unsigned>(u) * nthr;
      if (i < whole) {
        if (from_staging) {
#pragma unroll
          for (int v = 0; v < VW; ++v) qa[u][v] = stage[i * VW + v];
        } else {
#pragma unroll
          for (int v = 0; v < VT; ++v) qa[u][v] = stage[i * VT + v];
        }
        if (add) {
#pragma unroll
          for (int v = 0; v < VT; ++v) qb[u][v] = stage[stride + i * VT + v];
        }
        if (u < U / 2 && third) {
#pragma unroll
          for (int v = 0; v < VT; ++v) qc[u % (U / 2)][v] = stage[2 * stride + i * VT + v];
        }
      }
    }
    // The stage is free for the loader once every warp has read it.
    if (!more && t.tail == 0) {
      __syncwarp();
      if (lane == 0) MbarArrive(empty);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned i = at + static_cast<unsigned>(u) * nthr;
      if (i < whole) {
        A acc[P];
        if (from_staging) {
#pragma unroll
          for (int v = 0; v < VW; ++v) VecIO<W>::Load(qa[u][v], acc + v * VecIO<W>::kN);
        } else {
#pragma unroll
          for (int v = 0; v < VT; ++v) VecIO<T>::Load(qa[u][v], acc + v * VecIO<T>::kN);
          if (round_peer) {
#pragma unroll
            for (int e = 0; e < P; ++e) acc[e] = ThroughWire<W, A>(acc[e]);
          }
        }
        if (u < U / 2 && third) {
          A c[P];
#pragma unroll
          for (int v = 0; v < VT; ++v) VecIO<T>::Load(qc[u % (U / 2)][v], c + v * VecIO<T>::kN);
#pragma unroll
          for (int e = 0; e < P; ++e) acc[e] += round_peer ? ThroughWire<W, A>(c[e]) : c[e];
        }
        if (add) {
#pragma unroll
          for (int v = 0; v < VT; ++v) VecIO<T>::Add(qb[u][v], acc + v * VecIO<T>::kN);
        }
        if (t.flags & kTileScale) {
#pragma unroll
          for (int e = 0; e < P; ++e) acc[e] = ScaleAcc<A>(acc[e], p.scale);
        }
        uint4 wq[VW];
        if (t.remote != nullptr || round_wire) {
#pragma unroll
          for (int v = 0; v < VW; ++v) wq[v] = VecIO<W>::Store(acc + v * VecIO<W>::kN);
        }
        if (t.remote != nullptr) {
#pragma unroll
          for (int v = 0; v < VW; ++v) St16(t.remote + i * VW + v, wq[v]);
        }
        if (t.local != nullptr || peers != 0) {
          if (round_wire) {
#pragma unroll
            for (int v = 0; v < VW; ++v) VecIO<W>::Load(wq[v], acc + v * VecIO<W>::kN);
          }
          uint4 out[VT];
#pragma unroll
          for (int v = 0; v < VT; ++v) out[v] = VecIO<T>::Store(acc + v * VecIO<T>::kN);
          if (t.local != nullptr) {
#pragma unroll
            for (int v = 0; v < VT; ++v) St16Hint(t.local + i * VT + v, out[v], local_policy);
          }
          if (kShared && peers != 0) {
#pragma unroll
            for (int q = 0; q < kMaxRanks; ++q) {
              if (peers >> q & 1u) {
                uint4* const dst = reinterpret_cast<uint4*>(static_cast<unsigned char*>(p.peer_recv[q]) + recv_off);
#pragma unroll
                for (int v = 0; v < VT; ++v) St16Hint(dst + i * VT + v, out[v], peers_policy);
              }
            }
          }
        }
      }
    }
  }
  if (t.tail != 0) {
    if (whole % nthr == tid) RunTailPack<T, W, kShared>(tile, stage + whole * VW, p);
    __syncwarp();
    if (lane == 0) MbarArrive(empty);
  }
}

// Element-at-a-time path for chunks that do not start on a 16-byte boundary; kU
// loads of each source in flight per thread.  Bound by instructions: what the op says
// is read once, not for every element (it lies in global memory, which the stores
// below may change for all the compiler knows), and four loads keep this path and the
// tiles, which share its registers, from spilling.  With eight and the op's fields read
// anew, us: ring 8 x 4 MiB 199 -> 99, Rabenseifner 8 x 4 MiB 214 -> 113, 4 x 4 MiB of
// fp64 75 -> 33; aligned, ring 4 x 64 MiB of fp64 180 -> 157.  With eight and the fields
// read once the same here, but the aligned ring of 4 to 6 ranks that share buffers 7 % slower.
template <typename T, typename W, bool kShared>
__device__ void RunElements(const Op& op, const ExecParams& p, uint64_t lo, uint64_t hi, unsigned tid, unsigned nthr) {
  using A = typename Acc<T>::type;
  constexpr int kU = 4;
  const OpBuffers<T, W> buf(op, p);
  const T* b_src = op.src_b == kSrcSend ? buf.sendbuf : (op.src_b == kSrcRecv ? buf.recvbuf : nullptr);
  // What is another rank's: sources, and (rounded through the wire type) their values.
  const T *peer_a = nullptr, *peer_c = nullptr;
  bool round_peer = false;
  if constexpr (kShared) {
    if (op.src_a == kSrcPeer) peer_a = static_cast<const T*>(p.peer_send[op.rank_a]) + op.cell_begin;
    if (op.rank_c >= 0) peer_c = static_cast<const T*>(p.peer_send[op.rank_c]) + op.cell_begin;
    round_peer = (op.flags & kOpRoundPeer) && sizeof(W) != sizeof(T);
  }
  const uint64_t cell_begin = op.cell_begin;
  const uint8_t src_a = op.src_a, flags = op.flags, store_peers = op.store_peers;
  const T* const a_src = (src_a == kSrcSend ? buf.sendbuf : buf.recvbuf) + op.cell_begin;
  if (b_src != nullptr) b_src += op.cell_begin;
  T* const out = buf.recvbuf + op.cell_begin;
  auto of_peer = [&](T v) -> A { return round_peer ? ThroughWire<W, A>(ToAcc<A, T>(v)) : ToAcc<A, T>(v); };
#pragma unroll 1
  for (uint64_t k0 = lo + tid; k0 < hi; k0 += static_cast<uint64_t>(nthr) * kU) {
    A a[kU];
    T b[kU], c[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint64_t k = k0 + static_cast<uint64_t>(u) * nthr;
      if (k < hi) {
        if (src_a == kSrcStage) {
          a[u] = ToAcc<A, W>(LdScalarStrong<W>(buf.stage_in + k));
        } else if (kShared && peer_a != nullptr) {
          a[u] = of_peer(peer_a[k]);
        } else if (kShared && src_a == kSrcRecv) {
          a[u] = ToAcc<A, T>(LdScalarStrong<T>(out + k));  // another rank may have stored it
        } else {
          a[u] = ToAcc<A, T>(a_src[k]);
        }
        if (b_src != nullptr) b[u] = b_src[k];
        if (kShared && peer_c != nullptr) c[u] = peer_c[k];
      }
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint64_t k = k0 + static_cast<uint64_t>(u) * nthr;
      if (k < hi) {
        A v = a[u];
        if (kShared && peer_c != nullptr) v += of_peer(c[u]);
        if (b_src != nullptr) v += ToAcc<A, T>(b[u]);
        if (flags & kOpScale) v = ScaleAcc<A>(v, p.scale);
        if ((flags & kOpRoundWire) && sizeof(W) != sizeof(T)) v = ThroughWire<W, A>(v);
        if (flags & kOpStoreLocal) out[k] = FromAcc<T, A>(v);
        if (flags & kOpStoreRemote) buf.stage_out[k] = FromAcc<W, A>(v);
        if constexpr (kShared) {
          for (int q = 0; q < p.world_size; ++q)
            if (store_peers >> q & 1) static_cast<T*>(p.peer_recv[q])[cell_begin + k] = FromAcc<T, A>(v);
        }
      }
    }
  }
}

// Position in the ring of stages.
struct RingPos {
  uint32_t s = 0, parity = 0, stages;
  __device__ explicit RingPos(int n) : stages(static_cast<uint32_t>(n)) {}
  __device__ void Next() {
    if (++s == stages) s = 0, parity ^= 1u;
  }
};

// The loader: turns the program into stages, in order, ahead of the data warps.
// The lanes work out 32 ops at a time (an op is an 80-byte load and a division,
// 1.5 us one after the other); lane 0 then only issues copies.  Returns after it
// has handed out the exit stage (or could not, because the data warps gave up).
template <typename T, typename W, bool kShared>
__device__ void LoaderBody(const ExecParams& p, ExecShared<kShared>* sh, unsigned char* smem, int stages, int ch, int nch, int data_warps, int lane) {
  using Tr = ExecTraits<T, W>;
  const unsigned nthr = static_cast<unsigned>(data_warps) * 32u;
  const uint32_t stage_bytes = nthr * static_cast<uint32_t>(kExecStageBytesPerThread);
  // The user's data is read once, sendbuf and what is read back from recvbuf.
  const uint64_t user_policy = PolicyEvictFirst();
  RingPos pos(stages);
  bool first_round = true;
  uint32_t s = 0;  // stage claimed last (lane 0)
  auto next_stage = [&]() -> bool {
    s = pos.s;
    // The phase before the one the loader is about to fill: read by every data warp.
    const bool ok = first_round || RingWait(&sh->empty[s], pos.parity ^ 1u, &sh->role, p.timeout_ns);
    pos.Next();
    if (pos.s == 0) first_round = false;
    return ok;
  };
  // Hands out the exit stage; `fresh`: in a stage of its own, else in the claimed one
  // (copies into it complete before its phase does).
  auto leave = [&](bool fresh) {
    if (lane == 0 && (!fresh || next_stage())) {
      sh->tile[s].flags = kTileExit;
      MbarArrive(&sh->full[s]);
    }
  };
  unsigned ready = 0;  // ops known to have their flags; what they may read is visible to the copy engine
  for (int first = 0; first < p.num_ops; first += 32) {
    const int in_batch = p.num_ops - first < 32 ? p.num_ops - first : 32;
    bool in_bounds = true;
    if (lane < in_batch) {
      const Op op = p.ops[first + lane];
      in_bounds = OpInBounds<W, kShared>(op, p);
      if (in_bounds) {
        uint64_t lo, hi;
        ChannelSlice(op.elem_begin - op.cell_begin, op.elem_count, p.stage.slot_bytes / sizeof(W), nch, ch, &lo, &hi);
        const OpBuffers<T, W> buf(op, p);
        const uint64_t g0 = op.cell_begin + lo;
        const bool uses_send = op.src_a == kSrcSend || op.src_b == kSrcSend;
        const bool uses_recv = op.src_a == kSrcRecv || op.src_b == kSrcRecv || (op.flags & kOpStoreLocal);
        const T* const peer_a = kShared && op.src_a == kSrcPeer ? static_cast<const T*>(p.peer_send[op.rank_a]) + g0 : nullptr;
        const T* const peer_c = kShared && op.rank_c >= 0 ? static_cast<const T*>(p.peer_send[op.rank_c]) + g0 : nullptr;
        uintptr_t bits = reinterpret_cast<uintptr_t>(peer_a) | reinterpret_cast<uintptr_t>(peer_c);
        for (int q = 0; kShared && q < p.world_size; ++q)
          if (op.store_peers >> q & 1) bits |= reinterpret_cast<uintptr_t>(static_cast<T*>(p.peer_recv[q]) + g0);
        if (uses_send) bits |= reinterpret_cast<uintptr_t>(buf.sendbuf + g0);
        if (uses_recv) bits |= reinterpret_cast<uintptr_t>(buf.recvbuf + g0);
        // The place inside a staging slot follows the cell, not the user buffer: a
        // range that starts in the middle of a cell (Rabenseifner pieces, 16-bit
        // wire) can be 16-byte aligned on the user side and not in the slot.
        if (buf.stage_in != nullptr) bits |= reinterpret_cast<uintptr_t>(buf.stage_in + lo);
        if (buf.stage_out != nullptr) bits |= reinterpret_cast<uintptr_t>(buf.stage_out + lo);
        auto source = [&](uint8_t src) -> const unsigned char* {
          if (src == kSrcStage) return reinterpret_cast<const unsigned char*>(buf.stage_in + lo);
          if (src == kSrcNone) return nullptr;
          if (src == kSrcPeer) return reinterpret_cast<const unsigned char*>(peer_a);
          return reinterpret_cast<const unsigned char*>((src == kSrcSend ? buf.sendbuf : buf.recvbuf) + g0);
        };
        ExecPlan<kShared>& pl = sh->plan[lane];
        pl.src_a = source(op.src_a);
        pl.src_b = source(op.src_b);
        if constexpr (kShared) {
          pl.src_c = reinterpret_cast<const unsigned char*>(peer_c);
          pl.recv_off = g0 * sizeof(T);
          pl.late = op.src_a == kSrcStage || op.wait_peer != 0 ? 1 : 0;
        }
        pl.local = (op.flags & kOpStoreLocal) ? reinterpret_cast<unsigned char*>(buf.recvbuf + g0) : nullptr;
        pl.remote = buf.stage_out != nullptr ? reinterpret_cast<unsigned char*>(buf.stage_out + lo) : nullptr;
        const bool in_packs = lo < hi && (bits & 15u) == 0;
        pl.packs = in_packs ? (hi - lo + Tr::P - 1) / Tr::P : 0;
        pl.tail = in_packs ? static_cast<uint32_t>((hi - lo) % Tr::P) : 0;
        pl.lo = in_packs ? hi : lo;
        pl.hi = hi;
        pl.flags = (op.src_a == kSrcStage ? kTileFromStaging : 0u) | (op.src_b != kSrcNone ? kTileAdd : 0u) |
                   ((op.flags & kOpScale) ? kTileScale : 0u) | ((op.flags & kOpRoundWire) ? kTileRoundWire : 0u) |
                   ((op.flags & kOpReadBack) ? kTileReadBack : 0u) | (peer_c != nullptr ? kTileThird : 0u) |
                   ((op.flags & kOpRoundPeer) ? kTileRoundPeer : 0u) | ((op.flags & kOpPeersReadBack) ? kTilePeersReadBack : 0u) |
                   (static_cast<uint32_t>(op.store_peers) << kTilePeersShift);
        pl.wait_local = op.wait_local;
      }
    }
    // A bad op is reported by the waiter, which checks it as well; the ops before it still run.
    const unsigned bad = __ballot_sync(0xffffffffu, !in_bounds);
    const int good = bad != 0 ? __ffs(static_cast<int>(bad)) - 1 : in_batch;
    __syncwarp();
    for (int k = 0; k < good; ++k) {
      const unsigned oi = static_cast<unsigned>(first + k);
      const uint32_t wait_local = sh->plan[k].wait_local;
      // recvbuf is read only after the data warps' stores of the ops before have
      // landed: the fence orders their stores (observed through `done`) ahead of
      // what the copy engine reads.
      if (wait_local != 0) {
        bool ok = true;
        if (lane < data_warps) ok = SpinShared(&sh->role.done[lane], wait_local, &sh->role, p.timeout_ns);
        if (!__all_sync(0xffffffffu, ok)) return leave(true);
        __syncwarp();  // what the other lanes acquired is ordered before lane 0's fences
        if (lane == 0) {
          FencePeers(true);
          FenceProxyAsyncAll();
        }
      }
      int alive = 1;
      if (lane == 0) {
        const ExecPlan<kShared> pl = sh->plan[k];
        // The flags of op `oi` have arrived: one look may cover several ops, and
        // one proxy fence what all of them read from staging (written by
        // ordinary stores of the peers that the waiter's acquire made visible).
        auto get_ready = [&]() -> bool {
          if (ready > oi) return true;
          if (!SpinShared(&sh->role.ready, oi + 1u, &sh->role, p.timeout_ns)) return false;
          ready = LdAcquireShared(&sh->role.ready);
          FenceProxyAsyncAll();
          return true;
        };
        const bool a_staged = (pl.flags & kTileFromStaging) != 0;
        const bool drop = p.drop_lines != 0;
        const uint64_t a_step = static_cast<uint64_t>(a_staged ? Tr::VW : Tr::VT) * 16u;
        const unsigned char* src_c = nullptr;
        bool late = a_staged;
        uint32_t tile_packs = nthr * Tr::U;
        if constexpr (kShared) {
          src_c = pl.src_c;
          late = pl.late != 0;
          tile_packs = nthr * static_cast<uint32_t>(src_c != nullptr ? Tr::U / 2 : (pl.src_b != nullptr ? Tr::U : 2 * Tr::U));
        }
        const uint32_t source_bytes = tile_packs * Tr::VT * 16u;
        for (uint64_t j = 0; j < pl.packs; j += tile_packs) {
          if (!next_stage()) {
            alive = -1;
            break;
          }
          const uint32_t n = pl.packs - j < tile_packs ? static_cast<uint32_t>(pl.packs - j) : tile_packs;
          unsigned char* dst = smem + static_cast<size_t>(s) * stage_bytes;
          ExecTile<kShared>& t = sh->tile[s];
          t.local = pl.local != nullptr ? reinterpret_cast<uint4*>(pl.local + j * Tr::VT * 16u) : nullptr;
          t.remote = pl.remote != nullptr ? reinterpret_cast<uint4*>(pl.remote + j * Tr::VW * 16u) : nullptr;
          if constexpr (kShared) {
            t.recv_off = pl.recv_off + j * Tr::VT * 16u;
            t.stride = source_bytes / 16u;
          }
          t.packs = n;
          t.op = oi;
          const bool last = j + n >= pl.packs;
          t.flags = pl.flags | (last ? kTileLastOfOp : 0u);
          t.tail = last ? pl.tail : 0;
          t.drop_lines = 0;
          if (drop && a_staged) {
            const uintptr_t at = reinterpret_cast<uintptr_t>(pl.src_a + j * a_step), line = (at + 127u) & ~uintptr_t(127);
            const uintptr_t end = at + n * a_step;
            t.drop = reinterpret_cast<unsigned char*>(line);
            t.drop_lines = end > line ? static_cast<uint32_t>((end - line) / 128u) : 0;
          }
          const uint32_t whole = n - (t.tail != 0 ? 1u : 0u);
          if (t.tail != 0) {
            t.tail_a = pl.src_a + (j + whole) * Tr::VT * 16u;
            t.tail_b = pl.src_b + (j + whole) * Tr::VT * 16u;
            if constexpr (kShared) t.tail_c = src_c + (j + whole) * Tr::VT * 16u;
          }
          // What does not depend on a peer first, then the op's flags, then the staging slot.
          // The user's buffers end where the message ends; a slot holds whole packs.
          const uint32_t user_bytes = whole * Tr::VT * 16u, a_bytes = n * static_cast<uint32_t>(a_step);
          auto load_user = [&](uint32_t source, const unsigned char* from) {
            MbarExpectTxOnly(&sh->full[s], user_bytes);
            BulkLoadHint(dst + source * source_bytes, from + j * Tr::VT * 16u, user_bytes, &sh->full[s], user_policy);
          };
          if (pl.src_b != nullptr && whole != 0) load_user(1, pl.src_b);
          if (src_c != nullptr && whole != 0) load_user(2, src_c);
          if (!late && whole != 0) load_user(0, pl.src_a);
          if (!get_ready()) {
            alive = 0;
            break;
          }
          if (a_staged) {
            MbarExpectTxOnly(&sh->full[s], a_bytes);
            BulkLoad(dst, pl.src_a + j * a_step, a_bytes, &sh->full[s]);
          } else if (late && whole != 0) {
            load_user(0, pl.src_a);
          }
          MbarArrive(&sh->full[s]);
        }
        // A range that is not on 16-byte boundaries, or an op without elements for this channel (which still has to be reported done).
        if (alive > 0 && pl.packs == 0) {
          if (!next_stage()) {
            alive = -1;
          } else if (!get_ready()) {
            alive = 0;
          } else {
            ExecTile<kShared>& t = sh->tile[s];
            t.flags = kTileElements | kTileLastOfOp;
            t.op = oi;
            t.lo = pl.lo;
            t.hi = pl.hi;
            MbarArrive(&sh->full[s]);
          }
        }
      }
      alive = __shfl_sync(0xffffffffu, alive, 0);
      if (alive < 0) return;
      if (alive == 0) return leave(false);
    }
    if (good < in_batch) break;
    __syncwarp();  // lane 0 is done with the plans of this batch
  }
  leave(true);
}

// The waiter: a warp that looks at all of this channel's flags at once (lane q:
// data from rank q, lane 8 + q: credit from rank q, lane 16 + q: rank q's stores into
// recvbuf) and releases every op whose
// flags are there.  Lane k holds op first + k.
template <typename W, bool kShared>
__device__ void WaiterBody(const ExecParams& p, const WaitCtx& w, RoleSync* sync, uint64_t base, int ch, int lane, DeviceTraceRec* trace) {
  static_assert(kMaxRanks == 8, "one lane per flag");
  ControlPage* const me = Ctl(p.peers, p.rank);
  const uint64_t* const my_flag = lane < 8 ? &me->inflag[ch][lane] : (lane < 16 ? &me->credit[ch][lane & 7] : &me->bar[ch][lane & 7]);
  const bool watches = lane < (kShared ? 24 : 16) && (lane & 7) < p.world_size;
  const bool one_gpu = p.peers.one_gpu != 0;
  const uint64_t* const abort_word = &me->abort_seq;
  uint64_t seen = 0;
  for (int first = 0; first < p.num_ops; first += 32) {
    const int mine = first + lane;
    uint64_t need_data = 0, need_credit = 0;  // of data: a transfer into staging, or a store into recvbuf
    int from = 0, to = 0;                     // lanes that look at it
    bool bad = false;
    uint64_t elem_begin = 0, elem_count = 0;
    if (mine < p.num_ops) {
      const Op op = p.ops[mine];
      bad = !OpInBounds<W, kShared>(op, p);
      elem_begin = op.elem_begin;
      elem_count = op.elem_count;
      if (!bad && op.wait_in != 0) need_data = base | op.wait_in, from = op.peer_in;
      if (kShared && !bad && op.wait_peer != 0) need_data = (base | 1u) + op.wait_peer, from = 16 + op.peer_in;
      if (!bad && op.wait_credit != 0) need_credit = base | op.wait_credit, to = 8 + op.peer_out;
    }
    const int in_batch = p.num_ops - first < 32 ? p.num_ops - first : 32;
    int released = 0;
    uint64_t t0 = GlobalTimerNs();
    for (uint32_t spin = 0; released < in_batch; ++spin) {
      if (watches) seen = LdAcquirePeers(my_flag, one_gpu);
      const uint64_t data = __shfl_sync(0xffffffffu, seen, from), credit = __shfl_sync(0xffffffffu, seen, to);
      const bool go = !bad && (need_data == 0 || data >= need_data) && (need_credit == 0 || credit >= need_credit);
      const unsigned blocked = ~__ballot_sync(0xffffffffu, go || lane < released);
      const int upto = blocked == 0 ? 32 : __ffs(static_cast<int>(blocked)) - 1;
      const int now = upto < in_batch ? upto : in_batch;
      if (now > released) {
        if (trace != nullptr && lane >= released && lane < now && mine < p.trace_capacity) trace[mine].t_wait_done = GlobalTimerNs();
        released = now;
        __syncwarp();  // what every lane acquired is ordered before the release
        if (lane == 0) StReleaseShared(&sync->ready, static_cast<unsigned>(first + released));
        t0 = GlobalTimerNs();
        continue;
      }
      if (*reinterpret_cast<volatile int*>(&sync->stop) != 0) return;
      int give_up = 0;
      if (lane == released) {
        if (bad) {
          ReportFailure(w, kStatusBadProgram, 0, -1, mine, elem_begin, elem_count);
          BroadcastAbort(w);
          give_up = 1;
        } else if ((spin & 31u) == 31u) {
          const bool on_data = need_data != 0 && data < need_data;
          const uint32_t kind = on_data ? kWaitData : kWaitCredit;
          if (LdRelaxedSys(abort_word) == w.seq) {
            ReportFailure(w, kStatusPeerAbort, kind, (on_data ? from : to) & 7, mine, on_data ? need_data : need_credit, on_data ? data : credit);
            give_up = 1;
          } else if (GlobalTimerNs() - t0 > p.timeout_ns) {
            ReportFailure(w, kStatusWaitTimeout, kind, (on_data ? from : to) & 7, mine, on_data ? need_data : need_credit, on_data ? data : credit);
            BroadcastAbort(w);
            give_up = 1;
          }
        }
      }
      if (__any_sync(0xffffffffu, give_up)) {
        if (lane == 0) *reinterpret_cast<volatile int*>(&sync->stop) = 1;
        return;
      }
      if (spin > 4096u) __nanosleep(100);
    }
  }
}

// Body of the executor for one CTA: warps [0, data_warps) move data, then the
// waiter's, the loader's and the poster's warp.
template <typename T, typename W, bool kShared>
__device__ void ExecBody(const ExecParams& p, uint64_t seq, ExecShared<kShared>* sh, unsigned char* smem, int stages) {
  using Tr = ExecTraits<T, W>;
  const int ch = blockIdx.x, nch = gridDim.x;
  RoleSync* const sync = &sh->role;
  WaitCtx w;
  w.peers = &p.peers;
  w.status = p.status;
  w.doorbell = p.doorbell;
  w.seq = seq;
  w.timeout_ns = p.timeout_ns;
  w.rank = p.rank;
  w.world_size = p.world_size;
  w.channel = ch;
  const uint64_t base = seq << 32;
  ControlPage* const me = Ctl(p.peers, p.rank);
  volatile int* const stop = &sync->stop;

  // Entry barrier per channel: every peer's channel `ch` has started this
  // call, hence finished the previous one, so staging slots are free.
  if (threadIdx.x < p.world_size && threadIdx.x != p.rank && (p.present >> threadIdx.x & 1u)) {
    StReleasePeers(&Ctl(p.peers, threadIdx.x)->bar[ch][p.rank], base | 1u, p.peers.one_gpu != 0);
    if (!WaitGE(&me->bar[ch][threadIdx.x], base | 1u, w, kWaitBarrier, threadIdx.x, -1)) *stop = 1;
  }
  __syncthreads();
  if (*stop) return;

  DeviceTraceRec* trace = (p.trace != nullptr && p.trace_capacity > 0) ? p.trace + static_cast<size_t>(ch) * p.trace_capacity : nullptr;
  const int data_warps = static_cast<int>(blockDim.x) / 32 - kExecServiceWarps;
  const int warp = static_cast<int>(threadIdx.x) / 32, lane = static_cast<int>(threadIdx.x) % 32;
  const unsigned nthr = static_cast<unsigned>(data_warps) * 32u;
  const uint32_t stage_vecs = nthr * kExecStageBytesPerThread / 16u;

  if (warp < data_warps) {
    // A result nobody reads back should leave L2 before the staging slots and the partial
    // sums do (Rabenseifner in segments, 8 ranks x 64 MiB 457 -> 436 us, 5 ranks 298 -> 290).
    const uint64_t final_policy = PolicyEvictFirst(), partial_policy = PolicyNormal();
    for (RingPos pos(stages);; pos.Next()) {
      const uint32_t s = pos.s;
      if (!RingWait(&sh->full[s], pos.parity, sync, p.timeout_ns)) break;
      const ExecTile<kShared> t = sh->tile[s];
      if (t.flags & kTileExit) break;
      if (t.flags & kTileElements) {
        __syncwarp();
        if (lane == 0) MbarArrive(&sh->empty[s]);
        RunElements<T, W, kShared>(p.ops[t.op], p, t.lo, t.hi, threadIdx.x, nthr);
      } else {
        RunTile<T, W, kShared>(t, &sh->tile[s], reinterpret_cast<const uint4*>(smem) + static_cast<size_t>(s) * stage_vecs, p, &sh->empty[s],
                      partial_policy, final_policy, threadIdx.x, nthr, lane);
      }
      if (t.flags & kTileLastOfOp) {
        __syncwarp();
        if (lane == 0) StReleaseShared(&sync->done[warp], t.op + 1u);
      }
    }
  } else if (warp == data_warps) {
    WaiterBody<W, kShared>(p, w, sync, base, ch, lane, trace);
  } else if (warp == data_warps + 1) {
    LoaderBody<T, W, kShared>(p, sh, smem, stages, ch, nch, data_warps, lane);
  } else {
    // Poster: when every data warp has issued an op's stores, make them visible
    // to the peers and publish the op's flags.  Lane k holds op first + k.
    for (int first = 0; first < p.num_ops; first += 32) {
      const int mine = first + lane;
      uint32_t post_out = 0, post_credit = 0;
      uint32_t told[kMaxPeerPosts] = {};
      int peers = 0, told_peers = 0;
      if (mine < p.num_ops) {
        const Op op = p.ops[mine];
        post_out = op.post_out;
        post_credit = op.post_credit;
        peers = (static_cast<uint8_t>(op.peer_in) << 8) | static_cast<uint8_t>(op.peer_out);
        if constexpr (kShared) {
#pragma unroll
          for (int m = 0; m < kMaxPeerPosts; ++m) told[m] = op.post_told[m], told_peers |= static_cast<uint8_t>(op.peer_told[m]) << (8 * m);
        }
      }
      const bool tells = kShared && __any_sync(0xffffffffu, told[0] != 0);
      const int end = first + 32 < p.num_ops ? first + 32 : p.num_ops;
      int posted = first;
      while (posted < end) {
        bool ok = true;
        if (lane < data_warps) ok = SpinShared(&sync->done[lane], static_cast<unsigned>(posted) + 1u, sync, p.timeout_ns);
        if (!__all_sync(0xffffffffu, ok)) return;
        // How far the slowest data warp is by now.
        unsigned upto = lane < data_warps ? LdAcquireShared(&sync->done[lane]) : 0xffffffffu;
        upto = __reduce_min_sync(0xffffffffu, upto);
        const int until = static_cast<int>(upto) < end ? static_cast<int>(upto) : end;
        const bool fence = __any_sync(0xffffffffu, mine >= posted && mine < until && FlagsNeedFence(kShared ? post_out | told[0] : post_out, post_credit, p.drop_lines != 0));
        __syncwarp();  // what the other lanes acquired is ordered before lane 0's fence
        if (fence && lane == 0) FencePeers(p.peers.one_gpu != 0);
        for (; posted < until; ++posted) {
          const int k = posted - first;
          const uint32_t out = __shfl_sync(0xffffffffu, post_out, k), credit = __shfl_sync(0xffffffffu, post_credit, k);
          const int who = __shfl_sync(0xffffffffu, peers, k);
          if (lane == 0) {
            if (out != 0) StRelaxedSys(&Ctl(p.peers, who & 0xff)->inflag[ch][p.rank], base | out);
            if (credit != 0) StRelaxedSys(&Ctl(p.peers, who >> 8)->credit[ch][p.rank], base | credit);
            if (trace != nullptr && posted < p.trace_capacity) trace[posted].t_done = GlobalTimerNs();
          }
          if (tells) {
            const int whom = __shfl_sync(0xffffffffu, told_peers, k);
#pragma unroll
            for (int m = 0; m < kMaxPeerPosts; ++m) {
              const uint32_t n = __shfl_sync(0xffffffffu, told[m], k);
              if (lane == 0 && n != 0) StRelaxedSys(&Ctl(p.peers, whom >> (8 * m) & 0xff)->bar[ch][p.rank], (base | 1u) + n);
            }
          }
        }
      }
    }
  }
}

// kShared: programs of ranks that share a GPU and its memory (ProgramRequest::shared_gpu).
template <typename T, typename W, bool kShared>
__global__ void __launch_bounds__(kExecThreads, 1)
ExecKernel(const __grid_constant__ RankBlocks<ExecParams> all, int stages) {
  const ExecParams& p = all.rank[blockIdx.y];
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ ExecShared<kShared> s_exec;
  __shared__ uint64_t s_seq;
  {
    if (threadIdx.x == 0) {
      RoleSyncInit(&s_exec.role);
      for (int i = 0; i < kExecMaxStages; ++i) {
        MbarInit(&s_exec.full[i], 1);
        MbarInit(&s_exec.empty[i], blockDim.x / 32 - kExecServiceWarps);
      }
      MbarInitFence();
    }
  }
  if (p.world_size <= 1) return;
  const uint64_t seq = BeginCollective(p.peers, p.rank, &s_seq, gridDim.x);
  // Ranks without blocks in this launch count the call all the same.
  if (kShared && blockIdx.x == 0 && threadIdx.x < kMaxRanks && (p.counts_for >> threadIdx.x & 1u))
    atomicAdd(reinterpret_cast<unsigned long long*>(&Ctl(p.peers, static_cast<int>(threadIdx.x))->call_word), 1ull << 16);
  // num_ops <= 0: this rank sits the call out (test hook), but still counts it.
  if (p.num_ops > 0) ExecBody<T, W, kShared>(p, seq, &s_exec, smem, stages);
}

}  // namespace dev

static int ExecThreads() {
  const int v = Tunable("IBCOMM_EXEC_THREADS", 0);
  return (v >= 128 && v <= kExecThreads && v % 32 == 0) ? v : kExecThreads;
}

// Stages of the ring: what fits into an SM's shared memory, or into half of it
// for the smaller CTAs, of which two share an SM.
static int ExecStages(int threads) {
  const int stage = (threads - 32 * dev::kExecServiceWarps) * dev::kExecStageBytesPerThread;
  const int room = (threads > 256 ? 208 : 104) << 10;
  return std::min(dev::kExecMaxStages, std::max(2, room / stage));
}
static size_t ExecSmemBytes(int threads) {
  return static_cast<size_t>(ExecStages(threads)) * static_cast<size_t>((threads - 32 * dev::kExecServiceWarps) * dev::kExecStageBytesPerThread);
}

template <typename T, typename W, bool kShared>
static cudaError_t LaunchOne(const ExecParams* ranks, int n, int channels, cudaStream_t stream) {
  // Beyond one CTA per SM, two smaller CTAs share an SM: while one waits for a
  // flag, the other streams.
  const int threads = ExecKernelThreadsFor(channels * n);
  const size_t smem = ExecSmemBytes(threads);
  const auto kernel = dev::ExecKernel<T, W, kShared>;
  const cudaError_t e = AllowSharedMemory(kernel, smem);
  if (e != cudaSuccess) return e;
  return LaunchRanks(kernel, ranks, n, channels, threads, smem, stream, ExecStages(threads));
}
template <typename T, typename W>
static cudaError_t Launch(const ExecParams* ranks, int n, int channels, cudaStream_t stream) {
  // Programs that name other ranks' buffers come with them.
  return ranks->peer_recv[0] != nullptr ? LaunchOne<T, W, true>(ranks, n, channels, stream) : LaunchOne<T, W, false>(ranks, n, channels, stream);
}

cudaError_t LaunchExecKernel(const ExecParams* ranks, int n, int channels, cudaStream_t stream) {
  const DType t = static_cast<DType>(ranks->dtype), w = static_cast<DType>(ranks->wire);
  if (t == DType::kFloat32 && w == DType::kFloat32) return Launch<float, float>(ranks, n, channels, stream);
  if (t == DType::kFloat32 && w == DType::kBFloat16) return Launch<float, __nv_bfloat16>(ranks, n, channels, stream);
  if (t == DType::kFloat32 && w == DType::kFloat16) return Launch<float, __half>(ranks, n, channels, stream);
  if (t == DType::kFloat64 && w == t) return Launch<double, double>(ranks, n, channels, stream);
  if (t == DType::kInt32 && w == t) return Launch<int, int>(ranks, n, channels, stream);
  if (t == DType::kInt64 && w == t) return Launch<long long, long long>(ranks, n, channels, stream);
  if (t == DType::kFloat16 && w == t) return Launch<__half, __half>(ranks, n, channels, stream);
  if (t == DType::kBFloat16 && w == t) return Launch<__nv_bfloat16, __nv_bfloat16>(ranks, n, channels, stream);
  return cudaErrorInvalidValue;
}

int ExecKernelThreadsFor(int ctas) { return (ctas > 148 && ExecThreads() > 256) ? 256 : ExecThreads(); }

int ExecKernelMaxCoResidentBlocks(int device, int threads) {
  int per_sm = 0, sms = 0;
  if (threads <= 0) threads = kExecThreads;
  const size_t smem = ExecSmemBytes(threads);
  if (AllowSharedMemory(dev::ExecKernel<float, float, true>, smem) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dev::ExecKernel<float, float, true>, threads, smem) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
  return per_sm * sms;
}

}  // namespace ibcomm
