#include "ibcomm/emu_world.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "engine.h"
#include "ibcomm/tunables.h"

namespace ibcomm {

struct EmuWorld::Impl {
  int ws = 1;
  int device = 0;
  ArenaLayout layout;
  unsigned char* arenas = nullptr;  // ws arenas back to back
  std::vector<StatusBlock> status;
  std::vector<RankResources> ranks;
  ProgramCache cache;
  int timeout_ms = env::kDefaultTimeoutMs;
  int max_blocks = 0;
  int exec_max_blocks = 0;  // executor CTAs of the smaller size (two per SM)
  int line_max_blocks = 0;
  int last_channels = 0;
  int silent_rank = -1;
  int bad_program_rank = -1;
  // 0 in place, by one kernel for all ranks; 1 staged window by window, 2 staged through the pipelined kernel, 3 in
  // place, by the kernel ranks with a GPU each run.
  int direct_staging = 0;
  int staged_max_blocks = 0;
  uint32_t last_status = 0;
  DeviceStatus last_report{};
};

namespace {

// How the pipelined staged kernel runs when its ranks share a GPU.
struct StagedShape {
  bool split;      // copy roles in blocks of their own
  int buffers;     // windows of each kind
  int blocks;      // reducing blocks per rank (and copying blocks when split)
  uint64_t window_bytes;
  int load_groups, reduce_groups, store_groups;
};

// From which message on results are fetched from their reducers.
constexpr size_t kPullBytes = 8u << 20;

// `bytes`: of a rank's message in the wire type; `resident`: blocks of the kernel
// the GPU holds at once.  Measured on a B200 (the knobs override each choice):
//  * The windows of all ranks share one L2.  A line leaves it unwritten as soon as its
//    reader has it (StagedParams::drop_lines).  8 ranks x 32 MiB, 268 MB of results:
//    in 72 MiB 531 MB written to HBM without that and 299 MB with it, in about the
//    same time (a chain of flags per window binds); in 128 MiB, four buffers of each
//    kind, fewer chains, 460 MB and 188 us instead of 209.  4 ranks x 64 MiB 183 -> 164
//    us; without dropping, larger windows take 187 and more.
//  * No fence here waits for a link, so the copy roles need no blocks of their
//    own, and copies by the threads, with their loads rounds deep, beat the copy
//    engine's (8 x 25 MiB of fp32, bf16 wire: 156 us against 240 split; 4 x 64
//    MiB: 170 against 200 with bulk copies).
//  * A result is stored once, in its reducer's pool, and loaded there by the other ranks' storers: of 8 ranks, 2.0 times
//    the results' bytes are written instead of 2.75, and the output windows fill an eighth of their lines.  Their lines
//    have several readers and stay.  4 ranks x 64 MiB 168 -> 145 us, 8 x 32 MiB 189 -> 157, 5 x 64 MiB 225 -> 199, 8 x 12 MiB
//    79 -> 67; at 4 MiB and less within 2 %.
//  * Four warps load, four store, eight reduce: 5 ranks x 64 MiB 229 us against 239
//    with five, 2 x 12 MiB 21 against 23 (but 8 x 64 MiB 368 against 360).
//  * A block per 16 KiB: with one per 128 KiB a 0.5 MiB message on 5 ranks takes
//    27 us, with one per 16 KiB 21.
StagedShape StagedShapeOnOneGpu(uint64_t bytes, int ws, uint64_t staging_bytes, int resident, int channels) {
  StagedShape s;
  s.buffers = std::max(3, std::min(Tunable("IBCOMM_STAGED_BUFFERS", 4), kStagedMaxBuffers));
  while (s.buffers > 3 && staging_bytes / static_cast<uint64_t>(2 * s.buffers) < 4096) --s.buffers;  // a window is a page at least
  constexpr uint64_t kWindowsBytes = 128ull << 20;
  const uint64_t kinds = static_cast<uint64_t>(2 * s.buffers);
  s.window_bytes = std::min(staging_bytes / kinds, kWindowsBytes / (kinds * static_cast<uint64_t>(ws))) / 4096 * 4096;
  const int per_rank = std::max(1, resident / ws);
  s.split = Tunable("IBCOMM_STAGED_SPLIT", 0) != 0 && per_rank >= 2;
  const int most = std::min(128, s.split ? per_rank / 2 : per_rank);
  s.blocks = std::max(1, std::min(channels > 0 ? channels : static_cast<int>(std::min<uint64_t>(bytes / (16u << 10), 128)), most));
  auto groups = [](const char* knob, int dflt) { return std::max(1, std::min(Tunable(knob, dflt), 4)); };
  s.load_groups = groups("IBCOMM_STAGED_LOAD_GROUPS", 1);
  s.reduce_groups = groups("IBCOMM_STAGED_REDUCE_GROUPS", 2);
  s.store_groups = groups("IBCOMM_STAGED_STORE_GROUPS", 1);
  return s;
}

// CTAs per rank of the direct kernels for a rank's message of `bytes`: one per 16
// KiB (8 ranks on a B200: 64 KiB 8.5 us with four, 10.6 with one; 1 MiB 10.5 with
// 18, 14.7 with four), as far as the GPU holds them at once.
int ChannelsOnOneGpu(size_t bytes) {
  return static_cast<int>(std::min<size_t>(128, std::max<size_t>(1, bytes / (16u << 10))));
}

// The one-shot kernel pushes every byte to all other ranks: one per 4 KiB (8 x 64
// KiB: 6.4 us with 16, 8.2 with eight, 18 with one).
int OneShotChannelsOnOneGpu(size_t bytes) {
  return static_cast<int>(std::min<size_t>(128, std::max<size_t>(1, bytes / (4u << 10))));
}

// Half of a rank's lines area at most: a slot for every transfer of 2 MiB by three to eight ranks.
constexpr uint64_t kLinesHalfBytes = 16ull << 20;

// Whether an op program's transfers travel as lines: `bytes` of a rank's message in the wire type.  Slots with flags (as
// SharingPays says) against lines, us (IBCOMM_LINES_MAX_KIB overrides):
//                   64 KiB       512 KiB      1 MiB        2 MiB        4 MB
//   ring, 8 ranks   47.5  15.0   49.9  16.4   53.4  30.7   57.2  48.4   63.5  81
//   ring, 5 ranks   28.7  11.6   29.0  12.3   31.8  13.2   33.4  29.9   40.4  47
//   ring, 2 ranks    8.2   6.2    9.0   6.3    9.8   7.2   10.3   8.2   17.8  10
//   Rabenseifner 8  25.1  16.4   26.7  18.5   28.7  23.3   30.8  38.5
//   Rabenseifner 5  16.4  12.3   16.4  12.2   18.5  13.2   20.5  28.4
//   Rabenseifner 3   8.2   8.2    8.2   8.2    8.9  10.0   10.3  12.4
// One bound for all world sizes, although two ranks' rings are better off as lines up to 4 MB and three ranks'
// Rabenseifner is not at 1 MiB.
// `turns`: packs of a transfer that a thread handles one after the other, more than one where the caller prescribes fewer
// channels than a pack per thread takes.  Each turn waits for lines anew (ring, 8 ranks x 2 MiB in 32, 16, 8 and 4 channels
// 46, 50, 67 and 113 us as lines, 58, 56, 60 and 76 through slots), so there is a bound of all turns together, half as much
// again as that of one; from five on lines gain little or nothing (5 ranks x 256 KiB in one channel, seven turns, 44 us
// against 43).
bool LinesPay(Algo algo, uint64_t bytes, uint64_t turns) {
  const int most = Tunable("IBCOMM_LINES_MAX_KIB", algo == Algo::kRing ? 2048 : 1024);
  const uint64_t bound = static_cast<uint64_t>(std::max(0, most)) << 10;
  return turns <= 4 && bytes <= bound && bytes * turns <= bound + bound / 2;
}

// Whether an op program's ranks read each other's sendbuf and store into each other's recvbuf, or send as between
// GPUs.  `bytes` of a rank's message, `wire_bytes` of it in the wire type, `words`: of 4-byte elements that travel as they
// are; `channels` prescribed or 0.  Rabenseifner always (.28 to .97 in 2600 calls of 2 to 8 ranks).  The ring's
// transfers wait for each other, and a result that lies in recvbuf is there later than one in a slot, which does not show as
// long as the ranks are few and the parts short.  Sharing as a multiple of the time of sending, ring:
//                        4 MiB  8    12    16    24    32    64   128
//   2 ranks fp32          .67  .70   .73   .76   .79   .76   .76   .75
//   3 ranks fp32 / bf16   .83  .81   .86   .85   .88   .81   .85   .84    /  .81  .86  .86  .88  .94  .88  .88  .92
//   4 ranks fp32          .87  .87   .88   .92   .98   .99   .97   .96
//           bf16          .89  .90   .92   .96  1.05  1.04  1.04  1.03
//           fp64          .90  .88   .92   .94  1.01  1.03  1.00   .99
//           bf16 wire     .91  .89   .91   .92   .93   .99  1.03  1.01
//   6 ranks fp32          .93  .93   .95  1.00  1.05  1.00  1.01  1.03
//           bf16 / fp64   .96  .96  1.00  1.06  1.12  1.08  1.08  1.11    /  .96  .94  .98  1.03
//           bf16 wire     .96  .93   .95   .96  1.00  1.04  1.03  1.02
//   8 ranks fp32          .98  .97  1.00  1.03  1.08  1.10  1.09  1.08
//   around the bounds: 4 ranks x 20 MiB of bf16 1.01, of fp64 .98, in place .95 and .94, 24 MiB 1.06, 1.03, 1.00 and .98;
//   5 ranks x 14 MiB of bf16 .98, of fp64 .96, 15 MiB 1.02 and .99; 6 ranks x 12 MiB .99 both, 15 MiB 1.05 and 1.04
//   ragged ends 4 ranks 1.00 to 1.05, 5 ranks 1.10 to 1.15; slices off the boundary 3 ranks .86 to .97, 4 ranks 1.06 to 1.14
//   in prescribed channels, bytes a channel:  256 KiB   512 KiB    1 MiB    2 MiB
//   3 ranks fp32, 2 to 16 channels              .80       .90      1.01     1.00
//   5 ranks fp32, 2 to 16 channels              .91       .92      1.05     1.16
//   6 ranks fp32, one / two channels         1.01 .96  1.05 .96  1.07 1.07  1.21
//   and beyond a block per SM, 4 ranks in 48 channels 8 MiB .93, 16 MiB 1.10; 5 ranks in 32 channels 4 MiB .95, 8 MiB 1.05
bool SharingPays(Algo algo, int ws, size_t bytes, size_t wire_bytes, bool words, bool in_place, bool aligned, int channels) {
  if (algo == Algo::kRabenseifner) return true;
  if (!aligned || bytes % 16 != 0 || ws > 6) return false;
  if (ws == 2) return true;
  if (channels > 0) {
    size_t most = channels == 1 ? size_t(256) << 10 : static_cast<size_t>(channels) << 19;
    if (ws > 3 && channels * ws > 148) most = std::min(most, size_t(4) << 20);
    if (bytes > most) return false;
  }
  if (ws == 3) return true;
  if (ws == 4) return words || wire_bytes <= (size_t(in_place ? 24 : 20) << 20);
  return wire_bytes <= (size_t(words ? 16 : ws == 5 ? 14 : 12) << 20);
}

}  // namespace

EmuWorld::EmuWorld(int num_ranks, size_t pool_bytes, size_t work_bytes) : ws_(num_ranks), impl_(new Impl()) {
  if (num_ranks < 1 || num_ranks > kMaxRanks)
    IBCOMM_FAIL(NOT_SUPPORTED, "EmuWorld supports 1..%d ranks (got %d).\n", kMaxRanks, num_ranks);
  Impl& m = *impl_;
  m.ws = num_ranks;
  CUDACHECK(cudaGetDevice(&m.device));
  m.timeout_ms = env::ReadTimeoutMs();
  m.layout = MakeArenaLayout(pool_bytes ? pool_bytes : env::ReadPreAllocSize(), work_bytes ? work_bytes : env::ReadWorkGpuMemorySize(), num_ranks);
  // Nothing is sent to a mailbox here, so lines may have that memory.
  m.layout.lines_offset = m.layout.mailbox_offset;
  m.layout.lines_half_bytes = std::min<uint64_t>(kLinesHalfBytes, (m.layout.pool_offset - m.layout.mailbox_offset) / 2 / 4096 * 4096);
  const size_t total = static_cast<size_t>(m.layout.total_bytes) * static_cast<size_t>(num_ranks);
  CUDACHECK(cudaMalloc(&m.arenas, total));
  CUDACHECK(cudaMemset(m.arenas, 0, total));
  m.status.resize(static_cast<size_t>(num_ranks));
  m.ranks.resize(static_cast<size_t>(num_ranks));
  for (int r = 0; r < num_ranks; ++r) {
    m.status[static_cast<size_t>(r)].Create();
    RankResources& rr = m.ranks[static_cast<size_t>(r)];
    rr.rank = r;
    rr.world_size = num_ranks;
    rr.layout = m.layout;
    for (int q = 0; q < num_ranks; ++q) rr.peers.arena[q] = m.arenas + static_cast<size_t>(q) * m.layout.total_bytes;
    rr.peers.mc_arena = nullptr;
    rr.peers.one_gpu = 1;
    rr.d_status = m.status[static_cast<size_t>(r)].d_status;
    rr.h_doorbell = m.status[static_cast<size_t>(r)].h_doorbell;
    rr.d_doorbell = m.status[static_cast<size_t>(r)].d_doorbell;
  }
  m.max_blocks = TwoShotKernelMaxCoResidentBlocks(m.device);
  m.exec_max_blocks = ExecKernelMaxCoResidentBlocks(m.device, 256);
  m.line_max_blocks = LineKernelMaxCoResidentBlocks(m.device);
  m.staged_max_blocks = StagedKernelMaxCoResidentBlocks(m.device);
  CUDACHECK(cudaDeviceSynchronize());
}

EmuWorld::~EmuWorld() {
  Impl& m = *impl_;
  cudaDeviceSynchronize();
  m.cache.Clear();
  for (StatusBlock& s : m.status) s.Destroy();
  if (m.arenas != nullptr) cudaFree(m.arenas);
  (void)cudaGetLastError();
}

void EmuWorld::SetSilentRank(int r) { impl_->silent_rank = r; }
void EmuWorld::SetBadProgramRank(int r) { impl_->bad_program_rank = r; }
void EmuWorld::SetDirectStaging(int mode) { impl_->direct_staging = mode; }
void EmuWorld::SetTimeoutMs(int ms) { impl_->timeout_ms = ms > 0 ? ms : env::ReadTimeoutMs(); }
int EmuWorld::last_channels() const { return impl_->last_channels; }

uint32_t EmuWorld::LastStatus(DeviceStatus* report) const {
  if (report != nullptr) *report = impl_->last_report;
  return impl_->last_status;
}

void EmuWorld::Allreduce(Algo algo, DType dtype, const std::vector<const void*>& sendbufs, const std::vector<void*>& recvbufs,
                         size_t n, double scale, DType wire, int channels, void* stream_v, bool async) {
  Impl& m = *impl_;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  if (static_cast<int>(sendbufs.size()) != m.ws || static_cast<int>(recvbufs.size()) != m.ws)
    IBCOMM_FAIL(INVALID_ARGUMENT, "EmuWorld::Allreduce needs one buffer pair per rank.\n");
  for (int r = 0; r < m.ws; ++r)
    if (sendbufs[static_cast<size_t>(r)] == nullptr || recvbufs[static_cast<size_t>(r)] == nullptr)
      IBCOMM_FAIL(INVALID_ARGUMENT, "EmuWorld::Allreduce: null buffer.\n");
  if (dtype != DType::kFloat32) wire = dtype;
  const size_t esize = DTypeSize(dtype);
  const size_t bytes = n * esize;
  m.last_status = 0;

  if (m.ws == 1) {
    CopyParams cp{sendbufs[0], recvbufs[0], n, static_cast<int32_t>(dtype), static_cast<int32_t>(dtype), scale};
    if (!(sendbufs[0] == recvbufs[0] && scale == 1.0)) CUDACHECK(LaunchCopyKernel(cp, stream));
    m.last_channels = 0;
    if (!async) CUDACHECK(cudaStreamSynchronize(stream));
    return;
  }

  if (algo == Algo::kAuto) algo = ChooseAlgorithm(bytes, m.ws, false, false, kMaxChannels).algo;
  if (algo == Algo::kNvls)
    IBCOMM_FAIL(NOT_SUPPORTED, "Algorithm 'nvls' needs NVSwitch multicast between GPUs; it cannot be emulated on one GPU.\n");
  const uint64_t timeout_ns = static_cast<uint64_t>(m.timeout_ms) * 1000000ull;
  const int cap = std::max(1, m.max_blocks / m.ws);

  LocalParams local{};
  local.op = LocalOp::kAllreduce;
  local.world_size = m.ws;
  local.dtype = static_cast<int32_t>(dtype);
  local.wire = static_cast<int32_t>(wire);
  for (int q = 0; q < m.ws; ++q) {
    local.in[q] = sendbufs[static_cast<size_t>(q)];
    local.out[q] = recvbufs[static_cast<size_t>(q)];
  }
  local.len_elements = n;
  local.scale = scale;

  bool all_aligned = true, in_place = true;
  for (int q = 0; q < m.ws; ++q) in_place = in_place && sendbufs[static_cast<size_t>(q)] == recvbufs[static_cast<size_t>(q)];
  for (int q = 0; q < m.ws; ++q)
    all_aligned = all_aligned && ((reinterpret_cast<uintptr_t>(sendbufs[static_cast<size_t>(q)]) | reinterpret_cast<uintptr_t>(recvbufs[static_cast<size_t>(q)])) & 15u) == 0;
  const size_t wsize = DTypeSize(wire);
  const bool pipelined = algo == Algo::kDirect && (wire != dtype || m.direct_staging == 2);
  StagedShape sh{};
  if (pipelined) {
    sh = StagedShapeOnOneGpu(n * wsize, m.ws, m.layout.pool_bytes + m.layout.work_bytes, m.staged_max_blocks, channels);
    if (!all_aligned || (n * wsize) % 16 != 0 || sh.window_bytes < 4096)
      IBCOMM_FAIL(NOT_SUPPORTED, "The pipelined staged two-shot needs 16-byte aligned buffers of whole 16-byte wire vectors.\n");
  }
  const uint64_t half = m.layout.pool_bytes / 2 / 4096 * 4096;
  if (algo == Algo::kDirect && !pipelined && (!all_aligned || (m.direct_staging != 0 && m.direct_staging != 3)) && half < 8192)
    IBCOMM_FAIL(NOT_SUPPORTED, "Two-shot allreduce through the pool needs a pool of at least 16 KiB.\n");
  if (algo == Algo::kOneShot) {
    if (bytes > m.layout.oneshot_slot_bytes)
      IBCOMM_FAIL(INVALID_ARGUMENT, "One-shot allreduce handles at most %llu bytes (got %zu).\n",
                  static_cast<unsigned long long>(m.layout.oneshot_slot_bytes), bytes);
    local.wire = local.dtype;  // it has no other
  }
  // Ranks wait for each other in the staged kernel only, so that is where one that stays away is noticed.  The kernel for all
  // ranks has as many blocks as there are vectors; where the caller says how many a rank may have, those with channels run.
  const bool silent = pipelined && m.silent_rank >= 0;
  const bool one_kernel = m.direct_staging == 0 && channels <= 0 && !silent;
  if ((algo == Algo::kDirect || algo == Algo::kOneShot) && one_kernel && LocalKernelTakes(local)) {
    CUDACHECK(LaunchLocalKernel(local, stream));
    m.last_channels = 0;
  } else if (pipelined) {
    // The pipelined staged kernel (what ordinary buffers and 16-bit wires get on several GPUs).
    const int ch = sh.blocks;
    std::vector<StagedParams> ps(static_cast<size_t>(m.ws));
    for (int r = 0; r < m.ws; ++r) {
      StagedParams& p = ps[static_cast<size_t>(r)];
      memset(&p, 0, sizeof(p));
      const RankResources& rr = m.ranks[static_cast<size_t>(r)];
      p.rank = r;
      p.world_size = m.ws;
      p.dtype = static_cast<int32_t>(dtype);
      p.wire = static_cast<int32_t>(wire);
      p.use_multimem = 0;
      p.use_tma = (wire == dtype && Tunable("IBCOMM_STAGED_TMA", 0) != 0) ? 1 : 0;
      p.copy_warps = 4;
      p.drop_lines = p.use_tma == 0 ? 1 : 0;
      // Between two ranks a result is stored once either way, and what is short waits rather than streams.
      p.pull_results = p.use_tma == 0 && m.ws > 2 && n * wsize >= kPullBytes ? 1 : 0;
      p.peers = rr.peers;
      p.sendbuf = sendbufs[static_cast<size_t>(r)];
      p.recvbuf = recvbufs[static_cast<size_t>(r)];
      p.len_elements = n;
      p.scale = scale;
      p.window_elems = TwoShotWindowElems(n, sh.window_bytes / wsize, wsize, m.ws, ch);
      p.buffers = sh.buffers;
      p.split_ctas = sh.split ? 1 : 0;
      p.load_groups = sh.load_groups;
      p.reduce_groups = sh.reduce_groups;
      p.store_groups = sh.store_groups;
      p.posters = Tunable("IBCOMM_STAGED_POSTERS", 0) != 0 ? 1 : 0;
      for (int q = 0; q < m.ws; ++q) p.stage[q] = rr.peers.arena[q];
      p.mc_stage = nullptr;
      for (int j = 0; j < sh.buffers; ++j) {
        p.in_off[j] = m.layout.pool_offset + static_cast<uint64_t>(j) * sh.window_bytes;
        p.out_off[j] = m.layout.pool_offset + static_cast<uint64_t>(sh.buffers + j) * sh.window_bytes;
      }
      p.timeout_ns = timeout_ns;
      p.status = rr.d_status;
      p.doorbell = rr.d_doorbell;
      if (r == m.silent_rank) p.len_elements = 0;  // takes no part: no window, no flag
    }
    CUDACHECK(LaunchStagedKernel(ps.data(), m.ws, sh.split ? 2 * ch : ch, stream));
    m.last_channels = ch;
  } else if (algo == Algo::kDirect) {
    // The two-shot kernel with peer loads and stores, through the pool windows like
    // buffers the peers cannot map, or in place.
    int ch = channels > 0 ? channels : ChannelsOnOneGpu(bytes);
    ch = std::min(ch, cap);
    std::vector<NvlsParams> ps(static_cast<size_t>(m.ws));
    for (int r = 0; r < m.ws; ++r) {
      NvlsParams& p = ps[static_cast<size_t>(r)];
      memset(&p, 0, sizeof(p));
      const RankResources& rr = m.ranks[static_cast<size_t>(r)];
      p.rank = r;
      p.world_size = m.ws;
      p.dtype = static_cast<int32_t>(dtype);
      p.use_multimem = 0;
      p.peers = rr.peers;
      p.sendbuf = sendbufs[static_cast<size_t>(r)];
      p.recvbuf = recvbufs[static_cast<size_t>(r)];
      p.len_elements = n;
      p.scale = scale;
      p.timeout_ns = timeout_ns;
      p.status = rr.d_status;
      p.doorbell = rr.d_doorbell;
      const bool staged = (m.direct_staging != 0 && m.direct_staging != 3) || !all_aligned;
      p.stage_in = staged ? 1 : 0;
      p.stage_out = staged ? 1 : 0;
      for (int q = 0; q < m.ws; ++q) {
        if (staged) {
          p.peer_in[q] = rr.peers.arena[q] + m.layout.pool_offset;
          p.peer_out[q] = rr.peers.arena[q] + m.layout.pool_offset + half;
        } else {
          p.peer_in[q] = static_cast<unsigned char*>(const_cast<void*>(sendbufs[static_cast<size_t>(q)]));
          p.peer_out[q] = static_cast<unsigned char*>(recvbufs[static_cast<size_t>(q)]);
        }
      }
      p.local_in = p.peer_in[r];
      p.local_out = p.peer_out[r];
      p.window_elems = staged ? TwoShotWindowElems(n, (half - 4096) / esize, esize, m.ws, ch) : std::max<uint64_t>(1, n);
      p.tail_in_off = half - 4096;  // the ragged end of a staged message lives past every window
    }
    CUDACHECK(LaunchNvlsKernel(ps.data(), m.ws, ch, stream));
    m.last_channels = ch;
  } else if (algo == Algo::kOneShot) {
    std::vector<OneShotParams> ps;
    for (int r = 0; r < m.ws; ++r)
      ps.push_back(MakeOneShotParams(m.ranks[static_cast<size_t>(r)], dtype, sendbufs[static_cast<size_t>(r)],
                                     recvbufs[static_cast<size_t>(r)], n, scale, timeout_ns));
    int ch = channels > 0 ? channels : OneShotChannelsOnOneGpu(bytes);
    ch = std::min(ch, cap);
    CUDACHECK(LaunchOneShotKernel(ps.data(), m.ws, ch, stream));
    m.last_channels = ch;
  } else {
    // Validation (length, chunk size) happens while the first program is cut.
    std::vector<ExecParams> ps;
    bool fit = true, hooked_has_ops = true;
    auto programs = [&](ProgramForm form) {
      ps.clear();
      for (int r = 0; r < m.ws; ++r) {
        const CachedProgram& cp = m.cache.Get(algo, r, m.ws, n, dtype, wire, m.layout, scale != 1.0, stream, false, m.ws, form);
        fit = fit && LinesFit(cp.prog);
        if (form == ProgramForm::kShared && cp.prog.ops.empty()) {  // an extra rank: the others read its sendbuf and store into its recvbuf
          if (r == m.silent_rank || r == m.bad_program_rank) hooked_has_ops = false;
          continue;
        }
        ps.push_back(MakeExecParams(m.ranks[static_cast<size_t>(r)], cp, dtype, wire, sendbufs[static_cast<size_t>(r)],
                                    recvbufs[static_cast<size_t>(r)], n, scale, timeout_ns, nullptr, 0));
        if (r == m.silent_rank) ps.back().num_ops = 0;
        if (r == m.bad_program_rank) ps.back().len_elements = 1;
      }
    };
    // Prescribed chunks and pieces, and ranks that hand over as between GPUs, keep the slots.
    bool lines = m.direct_staging == 0 && LinesPay(algo, n * wsize, 1) && env::ReadChunkSize() <= 0 && Tunable("IBCOMM_RABEN_PIECES", 0) <= 0;
    int ch = 0;
    if (lines) {
      programs(ProgramForm::kLines);
      // A thread per pack of a transfer.
      const uint64_t blocks = (ps.back().stage.slot_bytes / 16 + 511) / 512;
      ch = channels > 0 ? channels : static_cast<int>(std::min<uint64_t>(blocks, static_cast<uint64_t>(kMaxChannels)));
      ch = std::max(1, std::min({ch, m.line_max_blocks / m.ws, kMaxChannels}));
      lines = fit && LinesPay(algo, n * wsize, (blocks + static_cast<uint64_t>(ch) - 1) / static_cast<uint64_t>(ch));
    }
    if (lines) {
      CUDACHECK(LaunchLineKernel(ps.data(), m.ws, ch, m.layout.lines_half_bytes, stream));
    } else {
      bool shared = m.direct_staging == 0 && SharingPays(algo, m.ws, bytes, n * wsize, esize == 4 && wsize == 4, in_place, all_aligned, std::min(channels, m.exec_max_blocks / m.ws));
      programs(shared ? ProgramForm::kShared : ProgramForm::kStaged);
      if (!hooked_has_ops) {
        // A rank that is to stay away, or to fail its self-check, needs ops of its own for that.
        shared = false;
        programs(ProgramForm::kStaged);
      }
      if (shared) {
        uint32_t present = 0;
        for (const ExecParams& p : ps) present |= 1u << p.rank;
        for (ExecParams& p : ps) {
          for (int q = 0; q < m.ws; ++q) {
            p.peer_send[q] = sendbufs[static_cast<size_t>(q)];
            p.peer_recv[q] = recvbufs[static_cast<size_t>(q)];
          }
          p.present = present;
        }
        ps.front().counts_for = ((1u << m.ws) - 1) & ~present;
      }
      const int rows = static_cast<int>(ps.size());
      // A channel for every 4 KiB of a transfer: the flags of ranks on one GPU are
      // cheap, and more channels shorten every step of the program.  One CTA per
      // SM at most (two smaller ones per SM are no faster).
      const uint64_t slot = ps.back().stage.slot_bytes;
      ch = channels > 0 ? channels : static_cast<int>(std::min<uint64_t>(slot / 4096, static_cast<uint64_t>(kMaxChannels)));
      // A short program may leave one rank with blocks, which the GPU holds more of than there are flags.
      ch = std::max(1, std::min({ch, (channels > 0 ? m.exec_max_blocks : m.max_blocks) / rows, kMaxChannels}));
      CUDACHECK(LaunchExecKernel(ps.data(), rows, ch, stream));
    }
    m.last_channels = ch;
  }
  if (async) return;
  CUDACHECK(cudaStreamSynchronize(stream));
  m.cache.NoteSynchronized();
  for (int r = 0; r < m.ws; ++r) {
    DeviceStatus st;
    uint32_t code = m.status[static_cast<size_t>(r)].Consume(&st, stream);
    // The report of the rank that found the problem beats "aborted by a peer".
    if (code != 0 && (m.last_status == 0 || (m.last_status == kStatusPeerAbort && code != kStatusPeerAbort))) {
      m.last_status = code;
      m.last_report = st;
    }
  }
  if (m.last_status != 0) IBCOMM_FAIL(TRANSPORT_ERROR, "%s\n", DescribeStatus(m.last_report).c_str());
}

void EmuWorld::ReduceScatterOrAllGather(bool all_gather, DType dtype, const std::vector<const void*>& sendbufs,
                                        const std::vector<void*>& recvbufs, size_t block_elems, double scale, int channels,
                                        void* stream_v, bool async) {
  Impl& m = *impl_;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  if (static_cast<int>(sendbufs.size()) != m.ws || static_cast<int>(recvbufs.size()) != m.ws)
    IBCOMM_FAIL(INVALID_ARGUMENT, "EmuWorld::ReduceScatterOrAllGather needs one buffer pair per rank.\n");
  if (block_elems == 0) IBCOMM_FAIL(NOT_SUPPORTED, "EmuWorld::ReduceScatterOrAllGather: empty block.\n");
  const size_t esize = DTypeSize(dtype);
  const size_t block_bytes = block_elems * esize;
  m.last_status = 0;
  if (m.ws == 1) {
    CopyParams cp{sendbufs[0], recvbufs[0], block_elems, static_cast<int32_t>(dtype), static_cast<int32_t>(dtype), all_gather ? 1.0 : scale};
    CUDACHECK(LaunchCopyKernel(cp, stream));
    if (!async) CUDACHECK(cudaStreamSynchronize(stream));
    return;
  }
  // In place when the remote sides agree in where their 16-byte boundaries lie.
  bool same_phase = true;
  auto remote_of = [&](int q) { return reinterpret_cast<uintptr_t>(all_gather ? recvbufs[static_cast<size_t>(q)] : sendbufs[static_cast<size_t>(q)]); };
  for (int q = 1; q < m.ws; ++q) same_phase = same_phase && ((remote_of(0) ^ remote_of(q)) & 15u) == 0;
  if (m.direct_staging == 0 && same_phase && channels <= 0) {
    LocalParams local{};
    local.op = all_gather ? LocalOp::kAllGather : LocalOp::kReduceScatter;
    local.world_size = m.ws;
    local.dtype = local.wire = static_cast<int32_t>(dtype);
    for (int q = 0; q < m.ws; ++q) {
      local.in[q] = sendbufs[static_cast<size_t>(q)];
      local.out[q] = recvbufs[static_cast<size_t>(q)];
    }
    local.len_elements = block_elems;
    local.scale = all_gather ? 1.0 : scale;
    CUDACHECK(LaunchLocalKernel(local, stream));
    m.last_channels = 0;
  } else {
    const bool staged = (m.direct_staging != 0 && m.direct_staging != 3) || !same_phase;
    const uint64_t sub = m.layout.pool_bytes / static_cast<uint64_t>(m.ws) / 4096 * 4096;
    if (staged && sub < 4096) IBCOMM_FAIL(NOT_SUPPORTED, "Reduce-scatter / all-gather through the pool need a larger pool.\n");
    const int cap = std::max(1, m.max_blocks / m.ws);
    int ch = channels > 0 ? channels : ChannelsOnOneGpu(block_bytes * static_cast<size_t>(m.ws));
    ch = std::min(ch, cap);
    std::vector<RsAgParams> ps(static_cast<size_t>(m.ws));
    for (int r = 0; r < m.ws; ++r) {
      RsAgParams& p = ps[static_cast<size_t>(r)];
      memset(&p, 0, sizeof(p));
      const RankResources& rr = m.ranks[static_cast<size_t>(r)];
      p.rank = r;
      p.world_size = m.ws;
      p.dtype = static_cast<int32_t>(dtype);
      p.mode = all_gather ? kRsAgAllGather : kRsAgReduceScatter;
      p.staged = staged ? 1 : 0;
      p.peers = rr.peers;
      p.sendbuf = sendbufs[static_cast<size_t>(r)];
      p.recvbuf = recvbufs[static_cast<size_t>(r)];
      p.block_elems = block_elems;
      p.scale = all_gather ? 1.0 : scale;
      p.timeout_ns = static_cast<uint64_t>(m.timeout_ms) * 1000000ull;
      p.status = rr.d_status;
      p.doorbell = rr.d_doorbell;
      for (int q = 0; q < m.ws; ++q) {
        if (staged) {
          p.peer_buf[q] = rr.peers.arena[q] + m.layout.pool_offset;
        } else {
          p.peer_buf[q] = all_gather ? static_cast<unsigned char*>(recvbufs[static_cast<size_t>(q)])
                                     : static_cast<unsigned char*>(const_cast<void*>(sendbufs[static_cast<size_t>(q)]));
        }
      }
      if (staged) {
        p.sub_stride_bytes = sub;
        p.window_elems = TwoShotWindowElems(block_elems, sub / esize, esize, 1, ch);
      } else {
        p.sub_stride_bytes = block_bytes;
        p.window_elems = block_elems;
      }
    }
    CUDACHECK(LaunchRsAgKernel(ps.data(), m.ws, ch, stream));
    m.last_channels = ch;
  }
  if (async) return;
  CUDACHECK(cudaStreamSynchronize(stream));
  for (int r = 0; r < m.ws; ++r) {
    DeviceStatus st;
    uint32_t code = m.status[static_cast<size_t>(r)].Consume(&st, stream);
    if (code != 0 && (m.last_status == 0 || (m.last_status == kStatusPeerAbort && code != kStatusPeerAbort))) {
      m.last_status = code;
      m.last_report = st;
    }
  }
  if (m.last_status != 0) IBCOMM_FAIL(TRANSPORT_ERROR, "%s\n", DescribeStatus(m.last_report).c_str());
}

void EmuWorld::AllreduceHostBuffers(Algo algo, DType dtype, const std::vector<const void*>& in, const std::vector<void*>& out,
                                    size_t n) {
  const size_t bytes = n * DTypeSize(dtype);
  std::vector<void*> d_in(in.size(), nullptr), d_out(out.size(), nullptr);
  std::vector<const void*> d_in_c;
  for (size_t r = 0; r < in.size(); ++r) {
    CUDACHECK(cudaMalloc(&d_in[r], std::max<size_t>(bytes, 16)));
    CUDACHECK(cudaMalloc(&d_out[r], std::max<size_t>(bytes, 16)));
    CUDACHECK(cudaMemcpy(d_in[r], in[r], bytes, cudaMemcpyHostToDevice));
    d_in_c.push_back(d_in[r]);
  }
  Allreduce(algo, dtype, d_in_c, d_out, n);
  for (size_t r = 0; r < in.size(); ++r) {
    CUDACHECK(cudaMemcpy(out[r], d_out[r], bytes, cudaMemcpyDeviceToHost));
    CUDACHECK(cudaFree(d_in[r]));
    CUDACHECK(cudaFree(d_out[r]));
  }
}

}  // namespace ibcomm
