// Host-callable launchers of the device kernels (one translation unit each).
#pragma once

#include <cuda_runtime.h>

#include "ibcomm/communicator.h"
#include "ibcomm/device_types.h"

namespace ibcomm {

// The parameter blocks of one launch, by value: block `blockIdx.y` belongs to
// the rank those CTAs work for.  A rank with a GPU of its own fills one, ranks
// that share a GPU one each.  By value, because a copy into device memory
// ahead of the launch costs the host 2 us and the stream another 2-4 us
// between two kernels, and the size costs nothing (an empty kernel: 2.3 us
// per launch with 64 bytes of parameters as with 3500).
template <typename P>
struct RankBlocks {
  P rank[kMaxRanks];
};
// grid = (blocks, ranks).  With several ranks the launch is cooperative: their
// CTAs wait on each other, so the runtime has to refuse a grid that is not
// co-resident.
template <typename P, typename... Rest>
cudaError_t LaunchRanks(void (*kernel)(RankBlocks<P>, Rest...), const P* ranks, int n, int blocks, int threads, size_t smem,
                        cudaStream_t stream, Rest... rest) {
  static_assert(sizeof(RankBlocks<P>) <= 4000, "kernel parameters");
  if (n < 1 || n > kMaxRanks) return cudaErrorInvalidValue;
  RankBlocks<P> all;
  for (int r = 0; r < n; ++r) all.rank[r] = ranks[r];
  void* args[] = {&all, &rest...};
  const dim3 grid(static_cast<unsigned>(blocks), static_cast<unsigned>(n));
  if (n > 1) return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kernel), grid, dim3(static_cast<unsigned>(threads)), args, smem, stream);
  return cudaLaunchKernel(reinterpret_cast<const void*>(kernel), grid, dim3(static_cast<unsigned>(threads)), args, smem, stream);
}
// Opts `kernel` in to `bytes` of dynamic shared memory (beyond 48 KiB it has to
// be): a property of the (function, device) pair, cheap, so set at every launch.
template <typename Kernel>
cudaError_t AllowSharedMemory(Kernel* kernel, size_t bytes) {
  return cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
}

// ---- op-program executor (ring, Rabenseifner) ----
// Here and below: `ranks` points to `n` parameter blocks, one per rank on this GPU.
cudaError_t LaunchExecKernel(const ExecParams* ranks, int n, int channels, cudaStream_t stream);
// CTA size the executor uses for a grid of `ctas` CTAs, and the largest
// grid of CTAs of `threads` threads (0 = the full-size CTA) that is co-resident
// on `device` (0 on error).  CTA b of a rank waits for CTA b of the other
// ranks, so a collective never launches more CTAs than fit at once.
int ExecKernelThreadsFor(int ctas);
int ExecKernelMaxCoResidentBlocks(int device, int threads = 0);

// The same for short messages, with transfers as lines (ll_kernel.cu).  `stage.offset` is that of an
// area used for lines only, two halves of `half_bytes` in which the program's slots take twice their
// bytes; no slot is used twice, and the program has at most kMaxLineOps ops.
constexpr int kMaxLineOps = 96;
cudaError_t LaunchLineKernel(const ExecParams* ranks, int n, int channels, uint64_t half_bytes, cudaStream_t stream);
int LineKernelMaxCoResidentBlocks(int device);

// ---- world_size == 1: out = cast(in * scale) ----
struct CopyParams {
  const void* in;
  void* out;
  uint64_t len_elements;
  int32_t dtype_in;
  int32_t dtype_out;
  double scale;
};
cudaError_t LaunchCopyKernel(const CopyParams& p, cudaStream_t stream);

// ---- two-shot allreduce: in the NVSwitch (multimem) or by direct peer loads/stores ----
struct NvlsParams {
  int32_t rank;
  int32_t world_size;
  int32_t dtype;
  int32_t use_multimem;  // 1: multimem.ld_reduce / multimem.st; 0: peer loads + peer stores
  int32_t stage_in;    // copy sendbuf into the multicast-bound staging first
  int32_t stage_out;   // results land in staging and are copied to recvbuf
  PeerTable peers;     // control pages live in the arenas
  const void* sendbuf;
  void* recvbuf;
  uint64_t len_elements;
  double scale;
  // Multicast and local addresses of the input and output windows.  When
  // staged, a window holds `window_elems` elements and the message is
  // processed in rounds; when zero-copy, the window is the whole buffer.
  unsigned char* mc_in;
  unsigned char* mc_out;
  unsigned char* local_in;
  unsigned char* local_out;
  // Unicast views of every rank's input window (direct variant; unaligned tail)
  // and output window (direct variant).
  unsigned char* peer_in[kMaxRanks];
  unsigned char* peer_out[kMaxRanks];
  uint64_t window_elems;
  // Staged input only: byte offset (from local_in / peer_in) of the 16 bytes
  // that hold the ragged end of the message, outside every window, so that
  // CTA 0, which moves the ragged end, touches no bytes that belong to another
  // CTA's part of a window.
  uint64_t tail_in_off;
  uint64_t timeout_ns;
  DeviceStatus* status;
  uint32_t* doorbell;
};
cudaError_t LaunchNvlsKernel(const NvlsParams* ranks, int n, int blocks, cudaStream_t stream);
// Largest co-resident grid of the two-shot kernels (they share CTA size and register budget).
int TwoShotKernelMaxCoResidentBlocks(int device);

// Hybrid two-shot (hybrid_kernel.cu): zero-copy symmetric buffers; CTAs
// [0, nvls_ctas) reduce 16-byte vectors [0, split_vec) in the switch, the other
// CTAs of the grid reduce the rest with peer loads and stores.
struct HybridParams {
  NvlsParams base;
  int32_t nvls_ctas;
  int32_t pad_;
  uint64_t split_vec;
};
cudaError_t LaunchHybridKernel(const HybridParams& h, int blocks, cudaStream_t stream);

// ---- pipelined staged two-shot (staged_kernel.cu) ----
// For buffers the peers cannot map, and for fp32 buffers that travel as
// bf16/fp16: the message moves through the pool in windows, and inside one
// CTA groups of warps work on several windows at the same time (copy in / two
// reducers over NVLink / copy out), with three to six buffers of each kind; or the
// roles are split over blocks.  At most 128 CTAs that reduce.
constexpr int kStagedMaxBuffers = 6;
struct StagedParams {
  int32_t rank;
  int32_t world_size;
  int32_t dtype;         // element type of the user buffers
  int32_t wire;          // element type in the pool and on the wire (== dtype, or 16-bit for fp32 buffers)
  int32_t use_multimem;  // 1: multimem.ld_reduce / multimem.st; 0: peer loads + peer stores
  int32_t use_tma;       // 1: the local copies are bulk asynchronous copies (needs wire == dtype)
  PeerTable peers;
  const void* sendbuf;   // 16-byte aligned
  void* recvbuf;         // 16-byte aligned
  uint64_t len_elements; // a whole number of 16-byte wire vectors
  double scale;
  uint64_t window_elems; // elements per window (a whole number of vectors per rank and CTA)
  // The staging memory as every rank maps it (the arena, or a larger block
  // the communicator allocated for large messages) and its multicast alias.
  unsigned char* stage[kMaxRanks];
  unsigned char* mc_stage;
  uint64_t in_off[kStagedMaxBuffers];    // byte offsets of the input windows inside the staging memory
  uint64_t out_off[kStagedMaxBuffers];   // ... and of the output windows
  int32_t buffers;       // windows of each kind in use (3 .. kStagedMaxBuffers)
  int32_t split_ctas;    // 1: the grid is 2 n blocks, [0, n) reduce and [n, 2n) copy; 0: every block does both
  uint64_t timeout_ns;
  DeviceStatus* status;
  uint32_t* doorbell;
  DeviceTraceRec* trace;   // [CTA][trace_capacity]: per window, when the reduce could start and when it was done
  int32_t trace_capacity;  // 0 = tracing off
  // W > 0: the other roles stamp too, W = number of windows, 4 W <= trace_capacity.  Records [W, 2W): the
  // loader (input buffer free, input window published), [2W, 3W): the storer (window reduced everywhere,
  // output buffer released), [3W, 4W): t_wait_done = the reducers' last store issued (before the fence).
  int32_t trace_roles;
  // Split mode: groups per role (1 .. 4) that take the windows in turn.  groups x reducing blocks <= 256
  // (a group has flag rows of its own).
  int32_t load_groups, reduce_groups, store_groups;
  int32_t copy_warps;  // unsplit, copies by the threads: warps of the loader and of the storer (0: three each)
  int32_t drop_lines;  // 1: lines of the windows leave L2 unwritten once their reader has them
  // 1: a result is stored once, in its reducer's pool, and the ranks' storers load it there (ranks on one GPU, copies by the
  // threads); 0: the reducer stores it into every rank's pool.
  int32_t pull_results;
  int32_t posters;  // split mode: a poster warp per reducer group fences and publishes behind the data warps
};
cudaError_t LaunchStagedKernel(const StagedParams* ranks, int n, int blocks, cudaStream_t stream);
// Largest grid of the staged kernel that is co-resident on `device` (0 on error).
int StagedKernelMaxCoResidentBlocks(int device);

// ---- reduce-scatter / all-gather (the halves of the two-shot allreduce) ----
enum RsAgMode : int32_t { kRsAgReduceScatter = 1, kRsAgAllGather = 2 };
struct RsAgParams {
  int32_t rank;
  int32_t world_size;
  int32_t dtype;
  int32_t use_multimem;  // 1: multimem.ld_reduce / multimem.st; 0: peer loads / peer stores
  int32_t mode;          // RsAgMode
  int32_t staged;        // the remote side is the pool (window by window), not a mapped user buffer
  PeerTable peers;
  const void* sendbuf;   // reduce-scatter: ws blocks; all-gather: one block
  void* recvbuf;         // reduce-scatter: one block; all-gather: ws blocks
  uint64_t block_elems;  // elements per block (per rank)
  double scale;          // reduce-scatter only
  // The remote side as every rank sees it (reduce-scatter: the inputs,
  // all-gather: the outputs): user buffers or pool windows, and their
  // multicast alias (null without multimem).
  unsigned char* peer_buf[kMaxRanks];
  unsigned char* mc_buf;
  // Block elements per window (the whole block when not staged) and the
  // distance in bytes between two sub-blocks of the remote side.
  uint64_t window_elems;
  uint64_t sub_stride_bytes;
  uint64_t timeout_ns;
  DeviceStatus* status;
  uint32_t* doorbell;
};
cudaError_t LaunchRsAgKernel(const RsAgParams* ranks, int n, int blocks, cudaStream_t stream);

// ---- direct collectives of ranks that share a GPU, buffers in place (local_kernel.cu) ----
enum class LocalOp : int32_t { kAllreduce, kReduceScatter, kAllGather };
struct LocalParams {
  LocalOp op;
  int32_t world_size;
  int32_t dtype;
  int32_t wire;           // == dtype, or (allreduce) a 16-bit type that fp32 values are rounded to as if they travelled
  const void* in[kMaxRanks];
  void* out[kMaxRanks];
  uint64_t len_elements;  // of the message; the halves: of a block
  double scale;
};
// Whether the buffers' 16-byte boundaries lie alike, as the kernel needs.
bool LocalKernelTakes(const LocalParams& p);
cudaError_t LaunchLocalKernel(const LocalParams& p, cudaStream_t stream);

// ---- one-shot allreduce for small messages (push to every peer, sum locally) ----
struct OneShotParams {
  int32_t rank;
  int32_t world_size;
  int32_t dtype;
  int32_t pad_;
  PeerTable peers;
  const void* sendbuf;
  void* recvbuf;
  uint64_t len_elements;
  double scale;
  uint64_t slot_offset;   // byte offset of the one-shot area in the arena
  uint64_t slot_bytes;    // bytes reserved per (parity, source rank)
  uint64_t timeout_ns;
  DeviceStatus* status;
  uint32_t* doorbell;
};
cudaError_t LaunchOneShotKernel(const OneShotParams* ranks, int n, int blocks, cudaStream_t stream);

// ---- two-sided device messaging through the peer's mailbox ----
struct P2pParams {
  int32_t rank;
  int32_t peer;
  int32_t is_send;
  int32_t world_size;
  PeerTable peers;
  const void* src;        // send: user buffer
  void* dst;              // recv: user buffer
  uint64_t bytes;
  uint64_t mailbox_offset;  // byte offset of the mailbox area in the arena
  uint64_t slot_bytes;      // bytes per mailbox slot
  uint32_t slots;           // slots per source rank
  uint32_t pad_;
  uint64_t first_piece;     // cumulative piece counter of this pair at call start
  uint64_t seq;
  uint64_t timeout_ns;
  DeviceStatus* status;
  uint32_t* doorbell;
};
// `ctas` (1..kP2pCtas) must be the same for every message of a communicator
// and on both sides: a CTA's flags count the pieces of its own part.  One SM
// sustains roughly 10 GB/s of stores to a peer, so bandwidth needs many CTAs.
cudaError_t LaunchP2pKernel(const P2pParams& p, int ctas, cudaStream_t stream);

// ---- device broadcast through NVSwitch multicast ----
// The root writes every piece ONCE (`multimem.st` into the broadcast ring of
// all ranks' mailbox areas at the same time, then the flag the same way); the
// others copy it out and return credits.  Needs the multicast alias of the
// arenas and a length that is a multiple of 16 (conditions every rank decides
// alike; a buffer that is only byte-aligned is moved byte by byte).
struct BcastParams {
  int32_t rank;
  int32_t root;
  int32_t world_size;
  int32_t pad_;
  PeerTable peers;
  void* buf;                // root: source, others: destination
  uint64_t bytes;
  uint64_t ring_offset;     // byte offset of the broadcast ring in the arena
  uint64_t slot_bytes;
  uint32_t slots;
  uint32_t pad2_;
  uint64_t first_piece;     // cumulative piece number of the communicator's broadcasts at call start
  uint64_t seq;
  uint64_t timeout_ns;
  DeviceStatus* status;
  uint32_t* doorbell;
};
cudaError_t LaunchBcastKernel(const BcastParams& p, int ctas, cudaStream_t stream);

}  // namespace ibcomm
