// What the two executors of op programs share (exec_kernel.cu, ll_kernel.cu).
#pragma once

#include <cstdint>

#include "flags.cuh"
#include "vec_ops.cuh"

namespace ibcomm {
namespace dev {

template <typename T, typename W>
struct ExecTraits {
  using A = typename Acc<T>::type;
  static constexpr int kMinBytes = sizeof(T) < sizeof(W) ? sizeof(T) : sizeof(W);
  static constexpr int P = 16 / kMinBytes;               // elements per pack
  static constexpr int VT = P / VecIO<T>::kN;            // 16-byte vectors per pack in the user type
  static constexpr int VW = P / VecIO<W>::kN;            // ... in the wire type
  static constexpr int U = VT > 1 ? 2 : 4;               // packs per thread and stage, of an op with two sources
};

// Where an op's data lies.
template <typename T, typename W>
struct OpBuffers {
  const T* sendbuf;
  T* recvbuf;
  const W* stage_in;
  W* stage_out;
  __device__ OpBuffers(const Op& op, const ExecParams& p)
      : sendbuf(static_cast<const T*>(p.sendbuf)), recvbuf(static_cast<T*>(p.recvbuf)), stage_in(nullptr), stage_out(nullptr) {
    const StageLayout& st = p.stage;
    if (op.src_a == kSrcStage)
      stage_in = reinterpret_cast<const W*>(p.peers.arena[p.rank] + st.offset +
                                            (static_cast<uint64_t>(op.region_in) * st.slots + op.slot_in) * st.slot_bytes);
    if (op.flags & kOpStoreRemote)
      stage_out = reinterpret_cast<W*>(p.peers.arena[op.peer_out] + st.offset +
                                       (static_cast<uint64_t>(op.region_out) * st.slots + op.slot_out) * st.slot_bytes);
  }
};

// Self-check of an op before any of its addresses is formed: the message
// range, the place inside the staging slot and the slot, region and peer
// indices.  A failing op is reported (status "bad program") and the call
// stops; nothing is accessed out of range and nothing traps.
template <typename W, bool kShared>
__device__ __forceinline__ bool OpInBounds(const Op& op, const ExecParams& p) {
  if (op.elem_begin > p.len_elements || op.elem_count > p.len_elements - op.elem_begin) return false;
  if (op.cell_begin > op.elem_begin || op.src_b == kSrcStage || op.src_b == kSrcPeer) return false;
  const bool reads_stage = op.src_a == kSrcStage;
  const bool writes_stage = (op.flags & kOpStoreRemote) != 0;
  if (reads_stage || writes_stage) {
    if ((op.elem_begin - op.cell_begin + op.elem_count) * sizeof(W) > p.stage.slot_bytes) return false;
  }
  if (reads_stage && (op.region_in >= p.stage.regions || op.slot_in >= p.stage.slots)) return false;
  if (writes_stage && (op.region_out >= p.stage.regions || op.slot_out >= p.stage.slots || op.peer_out < 0 ||
                       op.peer_out >= p.world_size))
    return false;
  if ((op.wait_in != 0 || op.post_credit != 0) && (op.peer_in < 0 || op.peer_in >= p.world_size)) return false;
  if ((op.wait_credit != 0 || op.post_out != 0) && (op.peer_out < 0 || op.peer_out >= p.world_size)) return false;
  // What only ranks that share a GPU have.
  if constexpr (kShared) {
    auto known = [&](int q) { return q >= 0 && q < p.world_size; };
    if (op.src_a == kSrcPeer && !known(op.rank_a)) return false;
    if (op.rank_c != -1 && !known(op.rank_c)) return false;
    if (op.wait_peer != 0 && !known(op.peer_in)) return false;
    for (int m = 0; m < kMaxPeerPosts; ++m)
      if (op.post_told[m] != 0 && !known(op.peer_told[m])) return false;
    if ((op.store_peers >> p.world_size) != 0) return false;
  } else if (op.src_a == kSrcPeer || op.rank_c != -1 || op.store_peers != 0) {
    return false;
  }
  return op.wait_local < static_cast<uint32_t>(p.num_ops);
}

}  // namespace dev
}  // namespace ibcomm
