// Executor of op programs for short messages: the same ring and Rabenseifner
// programs as exec_kernel.cu, with the transfers between ranks as lines that carry
// the call's number beside the data (ll.cuh).
//
// What bounds a short message is the chain of hand-overs from rank to rank.  In
// exec_kernel.cu one passes through six parties (data warps, poster with its fence,
// flag, waiter, loader, bulk copy): 3-4 us on one GPU.  Here a thread reads the lines of
// its packs until they are there, adds, and stores the next rank's lines: B200, us,
// ring of 8 x 64 KiB 47.3 -> 15.0, 8 x 512 KiB 49.6 -> 16.4, 5 x 1 MiB 34.8 -> 13.2;
// Rabenseifner 8 x 64 KiB 36.9 -> 16.4.  Where a transfer fills the threads (1 MiB and
// more) the looks and the doubled bytes are what L2 carries.
//
// A pack's place in its cell decides which channel and thread handle it, in every op
// and on every rank.  So what an op reads from recvbuf was stored by the thread that
// reads it, and a thread needs nothing of the others: there are no barriers, fences
// or flags in the loop.  No staging slot is used twice in a call (the host picks
// programs that fit), hence no credits.
//
// The ranks announce themselves once (ControlPage::bar), which nobody waits for: a
// wait that runs out tells from it whether the peer never came or stopped on the way.
#include "exec_common.cuh"
#include "flags.cuh"
#include "ibcomm/communicator.h"
#include "kernels.h"
#include "ll.cuh"
#include "vec_ops.cuh"

namespace ibcomm {
namespace dev {

constexpr int kLineThreads = 512;
static_assert((kLineThreads & (kLineThreads - 1)) == 0, "the thread of a pack is a mask away");

// One op of this channel.  Packs count from the start of the channel's slice of the
// cell; the pointers are those of pack 0, which the op need not include.
struct LinePlan {
  const unsigned char* user_a;  // source a in the user's buffers, or null
  const unsigned char* user_b;
  const unsigned char* lines_in;  // source a as lines, or null
  unsigned char* local;
  unsigned char* lines_out;
  uint32_t lo, hi;  // elements [lo, hi) of the slice
  uint32_t flags;   // OpFlags
  uint32_t aligned;  // packs of the user's buffers are whole 16-byte vectors
  int32_t peer_in;
  int32_t bad;  // fails its self-check
};

// Elements [e0, e1) of the pack at `p`, the others zero.
template <typename T, int VT, int P>
__device__ __forceinline__ void LdPack(const unsigned char* p, uint32_t e0, uint32_t e1, bool aligned, uint4* out) {
  if (aligned && e0 == 0 && e1 == P) {
#pragma unroll
    for (int v = 0; v < VT; ++v) out[v] = Ld16(p + v * 16);
    return;
  }
  using E = typename UIntOf<sizeof(T)>::type;
  constexpr int kN = 16 / static_cast<int>(sizeof(T));
#pragma unroll
  for (int v = 0; v < VT; ++v) {
    union { uint4 v; E e[kN]; } u;
    u.v = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int k = 0; k < kN; ++k)
      if (static_cast<uint32_t>(v * kN + k) >= e0 && static_cast<uint32_t>(v * kN + k) < e1) u.e[k] = reinterpret_cast<const E*>(p)[v * kN + k];
    out[v] = u.v;
  }
}
template <typename T, int VT, int P>
__device__ __forceinline__ void StPack(unsigned char* p, uint32_t e0, uint32_t e1, bool aligned, const uint4* q) {
  if (aligned && e0 == 0 && e1 == P) {
#pragma unroll
    for (int v = 0; v < VT; ++v) St16(p + v * 16, q[v]);
    return;
  }
  using E = typename UIntOf<sizeof(T)>::type;
  constexpr int kN = 16 / static_cast<int>(sizeof(T));
#pragma unroll
  for (int v = 0; v < VT; ++v) {
    union { uint4 v; E e[kN]; } u;
    u.v = q[v];
#pragma unroll
    for (int k = 0; k < kN; ++k)
      if (static_cast<uint32_t>(v * kN + k) >= e0 && static_cast<uint32_t>(v * kN + k) < e1) reinterpret_cast<E*>(p)[v * kN + k] = u.e[k];
  }
}

template <typename T, typename W>
__device__ void LineBody(const ExecParams& p, uint64_t half_bytes, LinePlan* plan, const uint64_t* s_seq) {
  using Tr = ExecTraits<T, W>;
  using A = typename Tr::A;
  constexpr int P = Tr::P, VT = Tr::VT;
  static_assert(Tr::VW == 1, "the wire type is never wider than the buffer type: a pack travels as one vector");
  const int ch = blockIdx.x, nch = gridDim.x;
  const unsigned tid = threadIdx.x;

  // The ops of this channel, a thread each.
  const uint64_t slot_elems = p.stage.slot_bytes / sizeof(W);
  bool bad = false;
  if (static_cast<int>(tid) < p.num_ops) {
    const Op op = p.ops[tid];
    bad = !OpInBounds<W, false>(op, p);
    plan[tid].bad = bad ? 1 : 0;
    if (!bad) {
      uint64_t lo0, unused, lo, hi;
      ChannelSlice(0, slot_elems, slot_elems, nch, ch, &lo0, &unused);
      ChannelSlice(op.elem_begin - op.cell_begin, op.elem_count, slot_elems, nch, ch, &lo, &hi);
      LinePlan pl;
      const uint64_t g0 = op.cell_begin + lo0;  // pack 0 in the user's buffers
      const unsigned char* const send = reinterpret_cast<const unsigned char*>(static_cast<const T*>(p.sendbuf) + g0);
      unsigned char* const recv = reinterpret_cast<unsigned char*>(static_cast<T*>(p.recvbuf) + g0);
      auto user = [&](uint8_t src) -> const unsigned char* { return src == kSrcSend ? send : (src == kSrcRecv ? recv : nullptr); };
      // A slot of lines is twice a slot of data: the first lines, then the second ones.
      auto lines = [&](int rank, uint64_t region, uint64_t slot) {
        return p.peers.arena[rank] + p.stage.offset + 2 * (region * p.stage.slots + slot) * p.stage.slot_bytes + lo0 * sizeof(W);
      };
      pl.user_a = user(op.src_a);
      pl.user_b = user(op.src_b);
      pl.lines_in = op.src_a == kSrcStage ? lines(p.rank, op.region_in, op.slot_in) : nullptr;
      pl.local = (op.flags & kOpStoreLocal) ? recv : nullptr;
      pl.lines_out = (op.flags & kOpStoreRemote) ? lines(op.peer_out, op.region_out, op.slot_out) : nullptr;
      pl.lo = lo < hi ? static_cast<uint32_t>(lo - lo0) : 0;
      pl.hi = lo < hi ? static_cast<uint32_t>(hi - lo0) : 0;
      pl.flags = op.flags;
      uintptr_t bits = 0;
      if (op.src_a == kSrcSend || op.src_b == kSrcSend) bits |= reinterpret_cast<uintptr_t>(send);
      if (op.src_a == kSrcRecv || op.src_b == kSrcRecv || pl.local != nullptr) bits |= reinterpret_cast<uintptr_t>(recv);
      pl.aligned = (bits & 15u) == 0 ? 1 : 0;
      pl.peer_in = op.peer_in;
      pl.bad = 0;
      plan[tid] = pl;
    }
  }
  const bool any_bad = __syncthreads_or(bad) != 0;
  const uint64_t seq = *s_seq, base = seq << 32;
  WaitCtx w;
  w.peers = &p.peers;
  w.status = p.status;
  w.doorbell = p.doorbell;
  w.seq = seq;
  w.timeout_ns = p.timeout_ns;
  w.rank = p.rank;
  w.world_size = p.world_size;
  w.channel = ch;
  if (any_bad) {
    if (tid == 0) {
      int first = 0;
      while (plan[first].bad == 0) ++first;
      const Op op = p.ops[first];
      ReportFailure(w, kStatusBadProgram, 0, -1, first, op.elem_begin, op.elem_count);
      BroadcastAbort(w);
    }
    return;
  }
  if (tid < static_cast<unsigned>(p.world_size) && static_cast<int>(tid) != p.rank)
    StRelaxedSys(&Ctl(p.peers, static_cast<int>(tid))->bar[ch][p.rank], base | 1u);

  const uint32_t number = LineNumber(seq);
  const uint64_t parity_off = (seq & 1u) * half_bytes, apart = p.stage.slot_bytes;
  for (int oi = 0; oi < p.num_ops; ++oi) {
    const LinePlan pl = plan[oi];
    const uint32_t j0 = pl.lo / P, j1 = (pl.hi + P - 1) / P;
    const bool aligned = pl.aligned != 0;
    for (uint32_t j = j0 + ((tid - j0) & (kLineThreads - 1)); j < j1; j += kLineThreads) {
      uint4 a[VT], b[VT];
      const uint32_t e0 = pl.lo > j * P ? pl.lo - j * P : 0, e1 = pl.hi < j * P + P ? pl.hi - j * P : P;
      const size_t at = static_cast<size_t>(j) * VT * 16, line = static_cast<size_t>(j) * 16 + parity_off;
      // What does not depend on a peer is on its way while the lines are looked for.
      if (pl.user_b != nullptr) LdPack<T, VT, P>(pl.user_b + at, e0, e1, aligned, b);
      if (pl.user_a != nullptr) LdPack<T, VT, P>(pl.user_a + at, e0, e1, aligned, a);
      if (pl.lines_in != nullptr) {
        LineWait wait;
        for (;;) {
          const Lines l = LdLines(pl.lines_in + line, apart);
          if (HaveArrived(l, number)) {
            a[0] = DataOf(l);
            break;
          }
          const uint32_t over = wait.Again(w);
          if (over != kStatusOk) {
            // A rank that never came says more than the one before this, which waits for it too.
            int peer = pl.peer_in;
            uint32_t kind = kWaitData;
            for (int q = p.world_size - 1; q >= 0; --q)
              if (q != p.rank && LdRelaxedSys(&Ctl(p.peers, p.rank)->bar[ch][q]) < (base | 1u)) peer = q, kind = kWaitBarrier;
            LineWaitOver(w, over, kind, peer, oi, base | 1u);
            return;
          }
        }
      }
      A acc[P];
      if (pl.lines_in != nullptr) {
        VecIO<W>::Load(a[0], acc);
      } else {
#pragma unroll
        for (int v = 0; v < VT; ++v) VecIO<T>::Load(a[v], acc + v * VecIO<T>::kN);
      }
      if (pl.user_b != nullptr) {
#pragma unroll
        for (int v = 0; v < VT; ++v) VecIO<T>::Add(b[v], acc + v * VecIO<T>::kN);
      }
      if (pl.flags & kOpScale) {
#pragma unroll
        for (int e = 0; e < P; ++e) acc[e] = ScaleAcc<A>(acc[e], p.scale);
      }
      const uint4 wire = VecIO<W>::Store(acc);
      if (pl.lines_out != nullptr) StLines(pl.lines_out + line, apart, wire, number);
      if (pl.local != nullptr) {
        if ((pl.flags & kOpRoundWire) && sizeof(W) != sizeof(T)) VecIO<W>::Load(wire, acc);
        uint4 out[VT];
#pragma unroll
        for (int v = 0; v < VT; ++v) out[v] = VecIO<T>::Store(acc + v * VecIO<T>::kN);
        StPack<T, VT, P>(pl.local + at, e0, e1, aligned, out);
      }
    }
  }
}

// Two blocks per SM: a pack at a time in 64 registers.  With four in 120, one block per SM, 8 ranks x 512 KiB take 18.5 us
// instead of 16.4 (ring) and 20.5 instead of 18.5 (Rabenseifner).
template <typename T, typename W>
__global__ void __launch_bounds__(kLineThreads, 2)
LineKernel(const __grid_constant__ RankBlocks<ExecParams> all, uint64_t half_bytes) {
  const ExecParams& p = all.rank[blockIdx.y];
  __shared__ LinePlan s_plan[kMaxLineOps];
  __shared__ uint64_t s_seq;
  // The last warp has the fewest ops to work out.
  if (threadIdx.x == kLineThreads - 1) TakeCallNumber(p.peers, p.rank, &s_seq, gridDim.x);
  __syncwarp();
  // num_ops <= 0: this rank sits the call out (test hook), but still counts it.
  if (p.num_ops > 0) LineBody<T, W>(p, half_bytes, s_plan, &s_seq);
}

}  // namespace dev

template <typename T, typename W>
static cudaError_t Launch(const ExecParams* ranks, int n, int channels, uint64_t half_bytes, cudaStream_t stream) {
  return LaunchRanks(dev::LineKernel<T, W>, ranks, n, channels, dev::kLineThreads, 0, stream, half_bytes);
}

cudaError_t LaunchLineKernel(const ExecParams* ranks, int n, int channels, uint64_t half_bytes, cudaStream_t stream) {
  for (int r = 0; r < n; ++r)
    if (ranks[r].num_ops > kMaxLineOps) return cudaErrorInvalidValue;
  const DType t = static_cast<DType>(ranks->dtype), w = static_cast<DType>(ranks->wire);
  if (t == DType::kFloat32 && w == DType::kFloat32) return Launch<float, float>(ranks, n, channels, half_bytes, stream);
  if (t == DType::kFloat32 && w == DType::kBFloat16) return Launch<float, __nv_bfloat16>(ranks, n, channels, half_bytes, stream);
  if (t == DType::kFloat32 && w == DType::kFloat16) return Launch<float, __half>(ranks, n, channels, half_bytes, stream);
  if (t == DType::kFloat64 && w == t) return Launch<double, double>(ranks, n, channels, half_bytes, stream);
  if (t == DType::kInt32 && w == t) return Launch<int, int>(ranks, n, channels, half_bytes, stream);
  if (t == DType::kInt64 && w == t) return Launch<long long, long long>(ranks, n, channels, half_bytes, stream);
  if (t == DType::kFloat16 && w == t) return Launch<__half, __half>(ranks, n, channels, half_bytes, stream);
  if (t == DType::kBFloat16 && w == t) return Launch<__nv_bfloat16, __nv_bfloat16>(ranks, n, channels, half_bytes, stream);
  return cudaErrorInvalidValue;
}

int LineKernelMaxCoResidentBlocks(int device) {
  int per_sm = 0, sms = 0;
  // The kernel with the most registers of them.
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dev::LineKernel<float, __half>, dev::kLineThreads, 0) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
  return per_sm * sms;
}

}  // namespace ibcomm
