// Schedule simulator tests: every rank's op program is interpreted on CPU
// threads (program_interp.h) for world sizes 1..8, message lengths around
// chunk boundaries, few and many staging slots, one and several channels, in
// place and out of place.  Results are compared with the exact integer sum;
// the per-pair transfer counts of sender and receiver must agree.
#include <cstdio>
#include <random>

#include "ibcomm/program_interp.h"
#include "mini_test.h"

using namespace ibcomm;

template <typename T>
static bool RunCase(Algo algo, int ws, size_t n, int64_t env_chunk, size_t stage_bytes, int nch, bool in_place,
                    double scale, size_t max_chunk_bytes = 0, size_t piece_elems = 0, size_t segment_pieces = 0, bool shared_gpu = false) {
  std::vector<size_t> segments;
  std::vector<Range> ranges = segment_pieces == 0 ? SplitForDevice(n, sizeof(T), static_cast<size_t>(ws), env_chunk, max_chunk_bytes)
                                                  : SplitSegments(n, piece_elems, segment_pieces, &segments);
  std::vector<std::vector<T>> in(static_cast<size_t>(ws), std::vector<T>(n)), out;
  std::mt19937 gen(static_cast<unsigned>(n * 31 + static_cast<size_t>(ws)));
  for (int r = 0; r < ws; ++r)
    for (size_t i = 0; i < n; ++i) in[static_cast<size_t>(r)][i] = static_cast<T>(static_cast<int>(gen() % 2001) - 1000);
  ProgramSimulator<T> sim(algo, ws, stage_bytes, nch, piece_elems, segments, shared_gpu);
  SimResult res = sim.Run(ranges, in, &out, scale, in_place);
  if (!res.ok) {
    fprintf(stderr, "%s ws=%d n=%zu: %s", AlgoName(algo), ws, n, res.error.c_str());
    return false;
  }
  // transfer-count audit
  const auto& progs = sim.programs();
  for (int a = 0; a < ws; ++a)
    for (int b = 0; b < ws; ++b)
      if (progs[static_cast<size_t>(a)].sent_to[b] != progs[static_cast<size_t>(b)].received_from[a]) {
        fprintf(stderr, "%s ws=%d: %d->%d sends %u, receiver expects %u\n", AlgoName(algo), ws, a, b,
                progs[static_cast<size_t>(a)].sent_to[b], progs[static_cast<size_t>(b)].received_from[a]);
        return false;
      }
  for (size_t i = 0; i < n; ++i) {
    double want = 0;
    for (int r = 0; r < ws; ++r) want += static_cast<double>(in[static_cast<size_t>(r)][i]);
    want *= scale;
    for (int r = 0; r < ws; ++r) {
      if (static_cast<double>(out[static_cast<size_t>(r)][i]) != static_cast<double>(static_cast<T>(want))) {
        fprintf(stderr, "%s ws=%d n=%zu nch=%d rank %d elem %zu: got %g want %g\n", AlgoName(algo), ws, n, nch, r, i,
                static_cast<double>(out[static_cast<size_t>(r)][i]), want);
        return false;
      }
    }
  }
  return true;
}

MINI_TEST(RingAllWorldSizes) {
  for (int ws = 2; ws <= 8; ++ws)
    for (size_t n : {size_t(ws), size_t(2 * ws), size_t(2521), size_t(4096), size_t(100003)})
      for (size_t stage : {size_t(1) << 22, size_t(1) << 16})
        CHECK_TRUE(RunCase<int>(Algo::kRing, ws, n, 0, stage, 1, false, 1.0, stage / 4));
}

MINI_TEST(RabenseifnerAllWorldSizes) {
  for (int ws = 2; ws <= 8; ++ws)
    for (size_t n : {size_t(ws), size_t(2 * ws), size_t(2521), size_t(4096), size_t(100003)})
      for (size_t stage : {size_t(1) << 22, size_t(1) << 17})
        CHECK_TRUE(RunCase<int>(Algo::kRabenseifner, ws, n, 0, stage, 1, false, 1.0, stage / 16));
}

MINI_TEST(TwoSlotsOnly) {
  // Exactly two slots per region: the tightest legal staging area.
  for (int ws = 2; ws <= 8; ++ws) {
    const size_t n = 64 * 4 * static_cast<size_t>(ws) * 3;  // chunks of 192 ints = 768 bytes
    std::vector<Range> rg = SplitForDevice(n, 4, static_cast<size_t>(ws), 0, 0);
    const size_t slot = (MaxChunkElems(rg) * 4 + 127) / 128 * 128;
    CHECK_TRUE(RunCase<int>(Algo::kRing, ws, n, 0, 2 * slot * static_cast<size_t>(NumRegions(Algo::kRing, ws)), 1, false, 1.0));
    CHECK_TRUE(RunCase<int>(Algo::kRabenseifner, ws, n, 0,
                            2 * slot * static_cast<size_t>(NumRegions(Algo::kRabenseifner, ws)), 1, false, 1.0));
  }
}

MINI_TEST(ChannelsInPlaceScale) {
  for (Algo a : {Algo::kRing, Algo::kRabenseifner})
    for (int ws : {2, 3, 4, 5, 6, 7, 8}) {
      CHECK_TRUE(RunCase<int>(a, ws, 70001, 0, size_t(1) << 20, 3, true, 1.0));
      CHECK_TRUE(RunCase<double>(a, ws, 33333, 0, size_t(1) << 20, 2, false, 0.25));
      CHECK_TRUE(RunCase<double>(a, ws, 4096, 0, size_t(1) << 20, 4, true, 0.5));
    }
}

MINI_TEST(SlotReuseWithSeveralChannels) {
  // Small staging areas (every slot is reused many times), lengths that make
  // the last chunk shorter than the others, several channels: the byte range
  // a channel owns inside a slot must not depend on the chunk in it.
  for (Algo a : {Algo::kRing, Algo::kRabenseifner})
    for (int ws : {2, 3, 4, 5, 7, 8})
      for (int nch : {2, 4, 5}) {
        const size_t stage = 400000;
        const size_t maxc = stage / (static_cast<size_t>(NumRegions(a, ws)) * 4) / 128 * 128;
        CHECK_TRUE(RunCase<int>(a, ws, 100000, 0, stage, nch, false, 1.0, maxc));
        CHECK_TRUE(RunCase<int>(a, ws, 10007, 0, 40000, nch, true, 1.0, 40000 / (static_cast<size_t>(NumRegions(a, ws)) * 4) / 128 * 128));
      }
}

MINI_TEST(RabenseifnerMergedPieces) {
  // Transfer pieces that ignore chunk boundaries: larger than a chunk, smaller
  // than a chunk, and not a divisor of anything; tight staging and several channels.
  for (int ws = 2; ws <= 8; ++ws)
    for (size_t piece : {size_t(32), size_t(1000), size_t(4096), size_t(100000)})
      for (int nch : {1, 3}) {
        CHECK_TRUE(RunCase<int>(Algo::kRabenseifner, ws, 100003, 0, size_t(1) << 22, nch, false, 1.0, 0, piece));
        const size_t regions = static_cast<size_t>(NumRegions(Algo::kRabenseifner, ws));
        CHECK_TRUE(RunCase<int>(Algo::kRabenseifner, ws, 50000, 0, 2 * regions * ((piece * 4 + 127) / 128 * 128), nch, true, 1.0, 0, piece));
      }
}

MINI_TEST(RabenseifnerSegments) {
  // One, two and many segments, the last one shorter; blocks of one piece and of
  // several; slots for a segment ahead, and two per region.
  for (int ws = 2; ws <= 8; ++ws) {
    const size_t p = ws < 4 ? 2 : ws < 8 ? 4 : 8, regions = static_cast<size_t>(NumRegions(Algo::kRabenseifner, ws));
    for (size_t piece : {size_t(256), size_t(1024)})
      for (size_t own : {size_t(1), size_t(3)})
        for (size_t n : {own * p * piece, 2 * own * p * piece - 5, 20003 + 4 * own * p * piece})
          for (size_t slots : {size_t(2), 2 * own, 4 * own + 1})
            for (int nch : {1, 3})
              CHECK_TRUE(RunCase<int>(Algo::kRabenseifner, ws, n, 0, slots * regions * piece * 4, nch, slots == 2, 1.0, 0, piece, own * p));
  }
}

MINI_TEST(RanksOnOneGpu) {
  // Programs that read the other ranks' sendbuf and store into their recvbuf: all world sizes, in place (a buffer is
  // overwritten with results while others still have to have read it), few and many slots, short and ragged lengths.
  for (int ws = 2; ws <= 8; ++ws)
    for (bool in_place : {false, true}) {
      for (size_t n : {size_t(ws), size_t(2 * ws + 1), size_t(2521), size_t(40007)})
        for (int nch : {1, 3}) {
          CHECK_TRUE(RunCase<int>(Algo::kRing, ws, n, 0, size_t(1) << 22, nch, in_place, 1.0, 0, 0, 0, true));
          CHECK_TRUE(RunCase<double>(Algo::kRing, ws, n, 0, 65536, nch, in_place, 0.5, 16384, 0, 0, true));
          CHECK_TRUE(RunCase<int>(Algo::kRabenseifner, ws, n, 0, size_t(1) << 22, nch, in_place, 1.0, 0, 1000, 0, true));
        }
      for (size_t n : {size_t(2521), size_t(40007)}) {  // prescribed chunks and pieces
        CHECK_TRUE(RunCase<int>(Algo::kRing, ws, n, 256, 65536, 2, in_place, 1.0, 16384, 0, 0, true));
        CHECK_TRUE(RunCase<double>(Algo::kRabenseifner, ws, n, 512, 65536, 2, in_place, 0.5, 0, 64, 0, true));
      }
      const size_t p = ws < 4 ? 2 : ws < 8 ? 4 : 8, regions = static_cast<size_t>(NumRegions(Algo::kRabenseifner, ws));
      for (size_t own : {size_t(1), size_t(3)})
        for (size_t n : {own * p * 256, 2 * own * p * 256 - 5, 20003 + 4 * own * p * 256})
          for (size_t slots : {size_t(2), 4 * own + 1})
            CHECK_TRUE(RunCase<double>(Algo::kRabenseifner, ws, n, 0, slots * regions * 256 * 8, 2, in_place, 0.25, 0, 256, own * p, true));
    }
}

// A partial sum as what it costs in precision: every addition rounds a sum of so many
// terms, and the error of a rounding grows with the sum.
struct Rounded {
  int terms = 1, cost = 0;
  Rounded() = default;
  explicit Rounded(int) {}
  Rounded operator*(double) const { return *this; }
};
static Rounded operator+(const Rounded& a, const Rounded& b) {
  Rounded s;
  s.terms = a.terms + b.terms;
  s.cost = a.cost + b.cost + s.terms;
  return s;
}

MINI_TEST(RabenseifnerRoundsLikeAFold) {
  // With extra ranks every element's sum is as good as where each extra rank is added to a
  // partner of its own first: 2 terms there, all terms once per step of the halving.
  for (int ws = 2; ws <= 8; ++ws) {
    const int p = ws < 4 ? 2 : ws < 8 ? 4 : 8, exp = util::GetExpOfTwo(static_cast<uint64_t>(p));
    const size_t n = 3001, piece = 128;
    for (size_t slots : {size_t(2), size_t(64)})  // contributions of extra ranks before all else, and where they are needed
      for (int form = 0; form < 3; ++form) {
        const bool in_segments = form != 0, shared_gpu = form == 2;
        std::vector<size_t> segments;
        const std::vector<Range> ranges = in_segments ? SplitSegments(n, piece, 4 * static_cast<size_t>(p), &segments)
                                                      : SplitForDevice(n, sizeof(Rounded), static_cast<size_t>(ws), 0, 0);
        const size_t stage = slots * static_cast<size_t>(NumRegions(Algo::kRabenseifner, ws)) * piece * sizeof(Rounded);
        ProgramSimulator<Rounded> sim(Algo::kRabenseifner, ws, stage, 1, piece, segments, shared_gpu);
        std::vector<std::vector<Rounded>> out;
        CHECK_TRUE(sim.Run(ranges, std::vector<std::vector<Rounded>>(static_cast<size_t>(ws), std::vector<Rounded>(n)), &out, 1.0, false).ok);
        int worst = 0, terms = 0;
        for (const auto& o : out)
          for (const Rounded& e : o) worst = std::max(worst, e.cost), terms = std::max(terms, std::abs(e.terms - ws));
        CHECK_EQ(terms, 0);
        CHECK_EQ(worst, 2 * (ws - p) + exp * ws);
      }
  }
}

MINI_TEST(FlagsBehindWritesNeedAFence) {
  // Where the lines of a slot are dropped as they are read, freeing the slot comes after a
  // write too: every op that writes what its flags hand over has a fence before them.
  for (int ws : {2, 5, 7, 8}) {
    const size_t p = ws < 4 ? 2 : ws < 8 ? 4 : 8, piece = 1024;
    std::vector<size_t> segments;
    ProgramRequest q;
    q.algo = Algo::kRabenseifner;
    q.world_size = ws;
    q.ranges = SplitSegments(6 * p * piece - 5, piece, 2 * p, &segments);
    q.segments = segments;
    q.piece_elems = piece;
    q.stage_bytes = 2 * static_cast<size_t>(NumRegions(q.algo, ws)) * piece * 4;
    size_t frees_only = 0, reuses = 0;
    for (int r = 0; r < ws; ++r) {
      q.rank = r;
      for (const Op& op : BuildProgram(q).ops) {
        for (bool drop : {false, true}) {
          const bool hands_over = op.post_out != 0 && (op.flags & kOpStoreRemote) != 0;
          const bool frees = op.post_credit != 0 && op.src_a == kSrcStage && drop;
          CHECK_EQ(FlagsNeedFence(op.post_out, op.post_credit, drop), hands_over || frees);
        }
        frees_only += op.post_out == 0 && op.post_credit != 0 ? 1 : 0;
        reuses += op.wait_credit != 0 ? 1 : 0;
      }
    }
    CHECK_TRUE(frees_only != 0 && reuses != 0);
  }
}

MINI_TEST(RingStaging) {
  // A rank with a GPU of its own stages in its whole pool, however large; ranks on one GPU share.
  for (uint64_t mib : {1, 64, 65, 1024}) CHECK_EQ(RingStageBytes(mib << 20, 1), mib << 20);
  CHECK_EQ(RingStageBytes(uint64_t(64) << 20, 8), uint64_t(8) << 20);
  CHECK_EQ(RingStageBytes(uint64_t(64) << 20, 2), uint64_t(32) << 20);
  CHECK_EQ(RingStageBytes(uint64_t(1) << 20, 8), uint64_t(1) << 20);
}

MINI_TEST(LongestPieceLeavesTwoSlots) {
  // Staging sizes that do not divide evenly among the regions, every element size on the
  // wire: the longest piece still fits twice into each region.
  for (int ws = 2; ws <= 8; ++ws)
    for (size_t stage : {size_t(4096) * 2, size_t(4096) * 3, size_t(128) << 20, (size_t(96) << 20) / 7, (size_t(100) << 20) + 4096, size_t(65536) * 11})
      for (size_t wire : {size_t(2), size_t(4), size_t(8)}) {
        ProgramRequest q;
        q.algo = Algo::kRabenseifner;
        q.world_size = ws;
        q.wire_elem_bytes = wire;
        q.stage_bytes = stage;
        const int regions = NumRegions(q.algo, ws);
        q.piece_elems = MaxPieceElems(stage, regions, wire);
        CHECK_TRUE(PlanStage(q).slots >= 2);
        CHECK_TRUE((q.piece_elems + 64) * wire * 2 * static_cast<size_t>(regions) + 128 > stage);  // and is not much shorter than it might be
      }
}

MINI_TEST(EnvChunkSizes) {
  for (int64_t chunk : {4, 8, 16, 32, 64, 128})
    CHECK_TRUE(RunCase<int>(Algo::kRing, 4, 256, chunk, size_t(1) << 16, 1, false, 1.0));
  CHECK_TRUE(RunCase<int>(Algo::kRabenseifner, 4, 256, 32, size_t(1) << 16, 1, false, 1.0));
}

MINI_TEST(RingOwnershipAfterReduceScatter) {
  // The op that stores locally with the scale flag marks the block a rank owns
  // after the reduce-scatter: it must be the block of rank r+1.
  const int ws = 4;
  std::vector<Range> rg = SplitForDevice(1600, 4, ws, 0, 0);
  auto blocks = GetRankToChunk(rg.size(), ws);
  for (int r = 0; r < ws; ++r) {
    ProgramRequest q;
    q.algo = Algo::kRing; q.rank = r; q.world_size = ws; q.ranges = rg; q.stage_bytes = 1 << 20; q.apply_scale = true;
    Program p = BuildProgram(q);
    std::vector<uint64_t> owned;
    for (const Op& op : p.ops)
      if (op.flags & kOpScale) owned.push_back(op.elem_begin);
    std::vector<uint64_t> want;
    for (auto it = blocks[(r + 1) % ws].rbegin(); it != blocks[(r + 1) % ws].rend(); ++it) want.push_back(rg[*it].first);
    CHECK_TRUE(owned == want);
    // first op: own block's highest chunk, straight from the send buffer
    CHECK_EQ(p.ops[0].src_a, uint8_t(kSrcSend));
    CHECK_EQ(p.ops[0].elem_begin, uint64_t(rg[blocks[r].back()].first));
  }
}

MINI_TEST(RandomConfigurations) {
  // Seeded fuzz over world size, length, channels, staging size, in-place and scale: the directed cases
  // above came from bugs that only some combinations showed.
  std::mt19937 gen(20240607u);
  auto pick = [&](size_t lo, size_t hi) { return lo + static_cast<size_t>(gen() % (hi - lo + 1)); };
  for (int it = 0; it < 250; ++it) {
    const Algo a = (gen() & 1u) ? Algo::kRing : Algo::kRabenseifner;
    const int ws = static_cast<int>(pick(2, 8));
    const size_t n = (gen() % 4 == 0) ? pick(static_cast<size_t>(ws), 64) : pick(static_cast<size_t>(ws), 150000);
    const int nch = static_cast<int>(pick(1, 6));
    const size_t stage = pick(40000, size_t(1) << 20);
    const size_t maxc = std::max<size_t>(128, stage / (static_cast<size_t>(NumRegions(a, ws)) * 4) / 128 * 128);
    const bool in_place = (gen() & 1u) != 0;
    bool ok;
    if (gen() % 3 == 0) ok = RunCase<double>(a, ws, n, 0, stage, nch, in_place, 0.5, maxc);
    else ok = RunCase<int>(a, ws, n, 0, stage, nch, in_place, 1.0, maxc);
    if (!ok) fprintf(stderr, "failing configuration: %s ws=%d n=%zu nch=%d stage=%zu in_place=%d\n", AlgoName(a), ws, n, nch, stage, in_place ? 1 : 0);
    CHECK_TRUE(ok);
  }
}

MINI_TEST(ValidateProgramFindsOutOfBoundsOps) {
  // Every program the builders cut passes; an op pushed out of the message,
  // out of its slot or out of the staging area is named.
  for (Algo algo : {Algo::kRing, Algo::kRabenseifner})
    for (int ws : {2, 3, 5, 8}) {
      const size_t n = 100003;
      std::vector<Range> rg = SplitForDevice(n, 4, ws, 0, 0);
      for (int r = 0; r < ws; ++r) {
        ProgramRequest q;
        q.algo = algo; q.rank = r; q.world_size = ws; q.ranges = rg; q.stage_bytes = 1 << 20;
        Program p = BuildProgram(q);
        CHECK_TRUE(ValidateProgram(p, n, 4, ws).empty());
        CHECK_TRUE(!ValidateProgram(p, n / 2, 4, ws).empty());  // the same ops against a shorter message
        Program bad = p;
        for (Op& op : bad.ops)
          if (op.flags & kOpStoreRemote) { op.slot_out = bad.stage.slots; break; }
        CHECK_TRUE(ValidateProgram(bad, n, 4, ws).find("output slot") != std::string::npos);
        q.shared_gpu = true;
        Program shared = BuildProgram(q);
        CHECK_TRUE(ValidateProgram(shared, n, 4, ws).empty());
        for (Op& op : shared.ops)
          if (op.store_peers != 0) { op.store_peers = static_cast<uint8_t>(1u << ws); break; }
        CHECK_TRUE(shared.ops.empty() || ws == 8 || ValidateProgram(shared, n, 4, ws).find("a rank that is none") != std::string::npos);
        bad = p;
        bad.stage.slot_bytes = 64;
        CHECK_TRUE(ValidateProgram(bad, n, 4, ws).find("does not fit") != std::string::npos);
      }
    }
}

int main(int argc, char** argv) { return mini::RunAll(argc > 1 ? argv[1] : nullptr); }
