#include "engine.h"

#include <algorithm>
#include <cstdio>
#include <cstring>

#include "ibcomm/tunables.h"

namespace ibcomm {

static uint64_t AlignUp(uint64_t v, uint64_t a) { return (v + a - 1) / a * a; }

ArenaLayout MakeArenaLayout(size_t pool_bytes, size_t work_bytes, int world_size) {
  ArenaLayout l;
  uint64_t off = 0;
  l.control_offset = off;
  off += AlignUp(sizeof(ControlPage), 65536);
  l.oneshot_offset = off;
  // A one-shot call pushes the whole message to every peer, so it needs one
  // slot per (parity, source rank): few ranks get large slots.
  const uint64_t ws = static_cast<uint64_t>(world_size < 2 ? 2 : (world_size > kMaxRanks ? kMaxRanks : world_size));
  l.oneshot_slot_bytes = kOneShotAreaBytes / (2 * ws) / 4096 * 4096;
  off += kOneShotAreaBytes;
  l.mailbox_offset = off;
  // Device Send/Recv mailboxes: per source rank a ring of slots.  A slot is
  // the unit of hand-over: before a piece's flag may be raised the sending
  // CTA waits until its stores are acknowledged over NVLink (about 6 us under
  // load, measured on B200), so a piece has to be worth several microseconds
  // of link time: 4 MiB slots, four of them (two in flight from the sender's
  // two warp groups, two being emptied by the receiver).  Knobs for experiments: IBCOMM_P2P_SLOT_KIB,
  // IBCOMM_P2P_SLOTS; all ranks must agree.
  {
    int kib = Tunable("IBCOMM_P2P_SLOT_KIB", 4096);
    if (kib < 16 || kib > (64 << 10)) kib = 4096;
    int slots = Tunable("IBCOMM_P2P_SLOTS", 4);
    if (slots < 2 || slots > kP2pMaxSlots) slots = 4;
    l.mailbox_slot_bytes = static_cast<uint64_t>(kib) << 10;
    l.mailbox_slots = static_cast<uint32_t>(slots);
  }
  // One ring per source rank, plus the ring device broadcasts are multicast into.
  l.bcast_ring_offset = off + static_cast<uint64_t>(kMaxRanks) * l.mailbox_slots * l.mailbox_slot_bytes;
  off += static_cast<uint64_t>(kMaxRanks + 1) * l.mailbox_slots * l.mailbox_slot_bytes;
  l.pool_offset = off;
  l.pool_bytes = AlignUp(pool_bytes < 4096 ? 4096 : pool_bytes, 4096);
  off += l.pool_bytes;
  l.work_offset = off;
  l.work_bytes = AlignUp(work_bytes < 4096 ? 4096 : work_bytes, 4096);
  off += l.work_bytes;
  l.total_bytes = AlignUp(off, 2u << 20);
  return l;
}

// ------------------------------------------------------------- status block
void StatusBlock::Create() {
  CUDACHECK(cudaMalloc(&d_status, sizeof(DeviceStatus)));
  CUDACHECK(cudaMemset(d_status, 0, sizeof(DeviceStatus)));
  CUDACHECK(cudaHostAlloc(reinterpret_cast<void**>(&h_doorbell), 64, cudaHostAllocMapped | cudaHostAllocPortable));
  *h_doorbell = 0;
  CUDACHECK(cudaHostGetDevicePointer(reinterpret_cast<void**>(&d_doorbell), h_doorbell, 0));
}

void StatusBlock::Destroy() {
  if (d_status != nullptr) cudaFree(d_status);
  if (h_doorbell != nullptr) cudaFreeHost(h_doorbell);
  d_status = nullptr;
  h_doorbell = nullptr;
  d_doorbell = nullptr;
  (void)cudaGetLastError();
}

uint32_t StatusBlock::Consume(DeviceStatus* out, cudaStream_t stream) {
  if (h_doorbell == nullptr) return 0;
  uint32_t bell = *reinterpret_cast<volatile uint32_t*>(h_doorbell);
  if (bell == 0) return 0;
  DeviceStatus st;
  memset(&st, 0, sizeof(st));
  CUDACHECK(cudaMemcpyAsync(&st, d_status, sizeof(st), cudaMemcpyDeviceToHost, stream));
  CUDACHECK(cudaMemsetAsync(d_status, 0, sizeof(st), stream));
  CUDACHECK(cudaStreamSynchronize(stream));
  *reinterpret_cast<volatile uint32_t*>(h_doorbell) = 0;
  if (st.code == 0) st.code = bell;
  if (out != nullptr) *out = st;
  return st.code;
}

std::string DescribeStatus(const DeviceStatus& st) {
  static const char* const codes[] = {"ok", "wait timed out", "aborted by a peer", "bad program", "message length mismatch"};
  static const char* const kinds[] = {"?", "barrier", "data flag", "slot credit", "mailbox", "one-shot flag"};
  char buf[320];
  snprintf(buf, sizeof(buf),
           "device collective failed: %s while waiting for a %s from rank %d (rank %d, channel %d, op %d, call %llu, "
           "expected %llu, saw %llu)",
           codes[st.code < 5 ? st.code : 0], kinds[st.kind < 6 ? st.kind : 0], st.peer, st.rank, st.channel, st.op_index,
           static_cast<unsigned long long>(st.seq), static_cast<unsigned long long>(st.expected & 0xffffffffull),
           static_cast<unsigned long long>(st.seen & 0xffffffffull));
  return buf;
}

// ------------------------------------------------------------ program cache
ProgramCache::~ProgramCache() { Clear(); }

void ProgramCache::Clear() {
  cache_.clear();
  for (Slab& sl : slabs_) {
    if (sl.d != nullptr) cudaFree(sl.d);
    if (sl.h != nullptr) cudaFreeHost(sl.h);
  }
  slabs_.clear();
  (void)cudaGetLastError();
}

Op* ProgramCache::Place(const std::vector<Op>& ops, cudaStream_t stream, int* slab_index) {
  const size_t n = ops.size();
  int at = -1;
  for (size_t i = 0; i < slabs_.size(); ++i)
    if (slabs_[i].cap - slabs_[i].used >= n) at = static_cast<int>(i);
  if (at < 0) {
    Slab sl;
    sl.cap = std::max<size_t>(n, (1u << 20) / sizeof(Op));
    CUDACHECK(cudaMalloc(&sl.d, sl.cap * sizeof(Op)));
    CUDACHECK(cudaHostAlloc(reinterpret_cast<void**>(&sl.h), sl.cap * sizeof(Op), cudaHostAllocPortable));
    slabs_.push_back(sl);
    at = static_cast<int>(slabs_.size()) - 1;
  }
  Slab& sl = slabs_[static_cast<size_t>(at)];
  memcpy(sl.h + sl.used, ops.data(), n * sizeof(Op));
  CUDACHECK(cudaMemcpyAsync(sl.d + sl.used, sl.h + sl.used, n * sizeof(Op), cudaMemcpyHostToDevice, stream));
  Op* d = sl.d + sl.used;
  sl.used += n;
  *slab_index = at;
  return d;
}

void ProgramCache::NoteSynchronized() {
  if (cache_.size() <= bound_) return;
  for (auto it = cache_.begin(); it != cache_.end();) {
    if (it->second->pinned) ++it;
    else it = cache_.erase(it);
  }
  // A slab without pinned programs starts over; the others keep their contents.
  for (Slab& sl : slabs_)
    if (sl.pinned == 0) sl.used = 0;
}

const CachedProgram& ProgramCache::Get(Algo algo, int rank, int world_size, size_t len_elements, DType dtype, DType wire,
                                       const ArenaLayout& layout, bool apply_scale, cudaStream_t stream, bool capturing, int ranks_on_gpu, ProgramForm form) {
  const size_t esize = DTypeSize(dtype), wsize = DTypeSize(wire);
  // Read at the point of use, like the reference: a bad value fails the call.
  const long long env_chunk = env::ReadChunkSize();
  const bool ring = algo == Algo::kRing;
  // The ring stages in the pool.  Rabenseifner lands its pieces in the work
  // region and, since one collective runs at a time, in the pool in front of
  // it as well (the two are adjacent in the arena).
  const bool lines = form == ProgramForm::kLines;
  const uint64_t stage_off = lines ? layout.lines_offset : layout.pool_offset;
  int raben_div = Tunable("IBCOMM_RABEN_PIECES", 0);
  const bool asked = raben_div >= 1 && raben_div <= 1024;
  // Ranks on one GPU run Rabenseifner in segments, unless the pieces are prescribed.
  const bool segmented = !ring && ranks_on_gpu > 1 && env_chunk <= 0 && !asked;
  // The ranks that share a GPU share its L2 too: a ring whose slots fit into it
  // together keeps its transfers there (a byte is written to staging and read back
  // 1.75 times).  Rabenseifner has the lines of its slots dropped from L2 as they are
  // read, and may then take all the staging there is, where the transfers would not
  // fit into L2 together and are of the user's type (8 x 64 MiB with a bf16 wire 346 us
  // without, 364 with).  How many times as fast that is, by the bytes of all ranks:
  //   ranks      2     3     4     5     6     7     8
  //   48 MiB   0.98  1.00  1.02  1.00  0.98  1.00  0.99
  //   64 MiB   1.02  1.15  1.00  1.05  1.01  1.00  0.99
  //   96 MiB   1.08  1.05  0.98  1.04  1.03  1.03  1.06
  //   256 MiB  1.08  1.10  0.99  1.03  1.07  1.05  1.03
  // Else, with few partners, a part of L2: four regions or more leave each two slots of
  // it, and the others wait for the extra ranks.
  const int regions = NumRegions(algo, world_size);
  const uint64_t sharers = static_cast<uint64_t>(ranks_on_gpu > 1 ? ranks_on_gpu : 1);
  const bool drop_lines = segmented && !lines && wsize == esize && sharers * len_elements * wsize >= (48ull << 20);
  uint64_t stage_bytes = ring ? RingStageBytes(layout.pool_bytes, ranks_on_gpu) : layout.pool_bytes + layout.work_bytes;
  if (lines) stage_bytes = layout.lines_half_bytes / 2;  // a line holds half its bytes
  else if (segmented && !drop_lines && regions <= 3) stage_bytes = std::min<uint64_t>(stage_bytes, kSharedGpuHalvingBytes / sharers);
  // Knobs that shape the program are part of the key: the ring's chunks per
  // rank and the number of pieces Rabenseifner cuts the message into.
  const size_t ring_cpr = lines ? 1 : ring ? RingChunksPerRank(len_elements, esize, static_cast<size_t>(world_size), ranks_on_gpu > 1) : 0;
  if (segmented) raben_div = 0;
  else if (!asked) raben_div = 8;
  Key key{static_cast<int>(algo), rank, world_size, len_elements, static_cast<int>(dtype), static_cast<int>(wire),
          env_chunk, apply_scale, stage_off, stage_bytes, ring ? static_cast<int>(ring_cpr) : raben_div, static_cast<int>(form)};
  auto it = cache_.find(key);
  if (it != cache_.end()) {
    CachedProgram& hit = *it->second;
    if (capturing && !hit.pinned) {
      hit.pinned = true;
      if (hit.slab >= 0) ++slabs_[static_cast<size_t>(hit.slab)].pinned;
    }
    return hit;
  }

  ProgramRequest req;
  req.algo = algo;
  req.rank = rank;
  req.world_size = world_size;
  if (ring) {
    // At least four slots keep the pipeline moving; two is the minimum the
    // schedule needs.
    uint64_t max_chunk_wire = stage_bytes / (static_cast<uint64_t>(regions) * 4) / 128 * 128;
    if (max_chunk_wire < 128) max_chunk_wire = 128;
    const size_t max_chunk_user = static_cast<size_t>(max_chunk_wire / wsize * esize);
    req.ranges = SplitForDevice(len_elements, esize, static_cast<size_t>(world_size), env_chunk, max_chunk_user, ring_cpr);
  } else {
    // Chunks only fix the block boundaries here; what travels are pieces:
    // IBCOMM_CHUNKSIZE when set, otherwise an eighth of the message (four
    // pieces in the largest step; knob IBCOMM_RABEN_PIECES), as far as two
    // slots per partner fit.
    req.ranges = SplitForDevice(len_elements, esize, static_cast<size_t>(world_size), env_chunk, 0);
    const size_t cap = MaxPieceElems(stage_bytes, regions, wsize);
    if (segmented) {
      // Segments: the transfers and partial sums of one stay in L2.  24 MiB, less
      // where more ranks share it, more where only two halve (2 ranks x 64 MiB 75 us
      // with 32 MiB, 80 with 24; 64 MiB per rank, the message as one and in
      // segments: 4 ranks 240 -> 182 us, 8 ranks 552 -> 435, 5 ranks 325 -> 277), and
      // one piece per block: an op costs as much as moving 100 KiB per channel does,
      // and a block of whole pieces leaves no slivers (5 ranks x 4 MiB 45 -> 38 us, 3
      // x 1 MiB 23 -> 21).  Two from 4 MiB on where only two ranks halve, since each
      // would wait for the other's only piece (2 ranks x 12 MiB 24.6 -> 22.9).
      const size_t p = static_cast<size_t>(util::FloorPow2(static_cast<uint64_t>(world_size)));
      const size_t bytes = len_elements * wsize;
      const size_t most = std::min<size_t>(std::min<size_t>(size_t(p == 2 ? 32 : 24) << 20, (size_t(128) << 20) / static_cast<size_t>(ranks_on_gpu)), cap * wsize * p);
      const size_t count = std::max<size_t>(1, util::ceilDiv(bytes, most));
      const size_t own = p == 2 && bytes / (count * p) > (size_t(4) << 20) ? 2 : 1;
      req.piece_elems = std::min<size_t>(cap, util::ceilDiv(util::ceilDiv(len_elements, count * p * own), size_t(32)) * 32);
      req.ranges = SplitSegments(len_elements, req.piece_elems, p * own, &req.segments);
    } else {
      size_t piece = env_chunk > 0 ? static_cast<size_t>(env_chunk) / esize : std::max<size_t>(util::ceilDiv(len_elements, static_cast<size_t>(raben_div)), 16384);
      if (piece > cap) {
        static bool warned = false;
        if (!warned && rank == 0) {
          warned = true;
          IBCOMM_WARN("IBCOMM_MEMORY_POOL_PRE_ALLOC + IBCOMM_WORK_GPU_MEMORY_SIZE (%llu bytes) limit Rabenseifner's transfer "
                      "pieces to %zu bytes instead of %zu; increase them for large messages.\n",
                      static_cast<unsigned long long>(stage_bytes), cap * wsize, piece * wsize);
        }
        piece = cap;
      }
      if (env_chunk <= 0 && piece >= 32) piece = util::ceilDiv(piece, size_t(32)) * 32;
      req.piece_elems = piece;
    }
  }
  req.wire_elem_bytes = wsize;
  req.stage_offset = stage_off;
  req.stage_bytes = stage_bytes;
  req.apply_scale = apply_scale;
  req.shared_gpu = form == ProgramForm::kShared;
  std::unique_ptr<CachedProgram> cp(new CachedProgram());
  cp->prog = BuildProgram(req);
  cp->drop_lines = drop_lines;
  {
    const std::string bad = ValidateProgram(cp->prog, len_elements, wsize, world_size);
    if (!bad.empty()) IBCOMM_FAIL(INVALID_ARGUMENT, "Internal error: the %s program for %zu elements on %d ranks is out of bounds (%s).\n",
                                  ring ? "ring" : "Rabenseifner", len_elements, world_size, bad.c_str());
  }
  if (!cp->prog.ops.empty()) {
    cp->d_ops = Place(cp->prog.ops, stream, &cp->slab);
    if (capturing) {
      cp->pinned = true;
      ++slabs_[static_cast<size_t>(cp->slab)].pinned;
    }
  }
  const CachedProgram& ref = *cp;
  cache_[key] = std::move(cp);
  return ref;
}

bool LinesFit(const Program& prog) {
  if (prog.ops.empty() || prog.ops.size() > static_cast<size_t>(kMaxLineOps)) return false;
  for (const uint32_t sent : prog.sent_to)
    if (sent > prog.stage.slots) return false;
  return true;
}

ExecParams MakeExecParams(const RankResources& rr, const CachedProgram& cp, DType dtype, DType wire, const void* sendbuf,
                          void* recvbuf, size_t len_elements, double scale, uint64_t timeout_ns,
                          DeviceTraceRec* trace, int trace_capacity) {
  ExecParams p;
  memset(&p, 0, sizeof(p));
  p.rank = rr.rank;
  p.world_size = rr.world_size;
  p.dtype = static_cast<int32_t>(dtype);
  p.wire = static_cast<int32_t>(wire);
  p.peers = rr.peers;
  p.sendbuf = sendbuf;
  p.recvbuf = recvbuf;
  p.len_elements = len_elements;
  p.scale = scale;
  p.ops = cp.d_ops;
  p.num_ops = static_cast<int32_t>(cp.prog.ops.size());
  p.trace_capacity = trace_capacity;
  p.stage = cp.prog.stage;
  p.drop_lines = rr.peers.one_gpu != 0 && cp.drop_lines ? 1 : 0;
  p.timeout_ns = timeout_ns;
  p.status = rr.d_status;
  p.doorbell = rr.d_doorbell;
  p.trace = trace;
  p.present = (1u << rr.world_size) - 1;
  return p;
}

OneShotParams MakeOneShotParams(const RankResources& rr, DType dtype, const void* sendbuf, void* recvbuf,
                                size_t len_elements, double scale, uint64_t timeout_ns) {
  OneShotParams p;
  memset(&p, 0, sizeof(p));
  p.rank = rr.rank;
  p.world_size = rr.world_size;
  p.dtype = static_cast<int32_t>(dtype);
  p.peers = rr.peers;
  p.sendbuf = sendbuf;
  p.recvbuf = recvbuf;
  p.len_elements = len_elements;
  p.scale = scale;
  p.slot_offset = rr.layout.oneshot_offset;
  p.slot_bytes = rr.layout.oneshot_slot_bytes;
  p.timeout_ns = timeout_ns;
  p.status = rr.d_status;
  p.doorbell = rr.d_doorbell;
  return p;
}

}  // namespace ibcomm
