#include "ibcomm/schedule.h"

#include <algorithm>
#include <cstdio>
#include <functional>
#include <unordered_map>

#include "ibcomm/tunables.h"

namespace ibcomm {

namespace {

inline int Mod(int x, int m) { return ((x % m) + m) % m; }

// Per-rank program under construction with the per-peer transfer counters
// that make both ends of a pair agree on slot numbers and flag values.
struct Builder {
  const ProgramRequest& req;
  Program prog;
  uint32_t slots;
  std::vector<int> my_in_peers;
  uint32_t told[kMaxRanks] = {0}, heard[kMaxRanks] = {0};  // stores into another rank's recvbuf, and into this one's

  explicit Builder(const ProgramRequest& r) : req(r) {
    prog.stage = PlanStage(r);
    slots = prog.stage.slots;
    my_in_peers = InPeers(r.algo, r.rank, r.world_size);
    prog.in_peers = my_in_peers;
  }

  int RegionOf(int receiver, int sender) const {
    std::vector<int> peers = (receiver == req.rank) ? my_in_peers : InPeers(req.algo, receiver, req.world_size);
    for (size_t i = 0; i < peers.size(); ++i)
      if (peers[i] == sender) return static_cast<int>(i);
    IBCOMM_FAIL(INVALID_ARGUMENT, "schedule: rank %d is not an in-peer of rank %d.\n", sender, receiver);
  }

  Op Base(const Range& g) const {
    Op op{};
    op.peer_in = -1;
    op.peer_out = -1;
    op.rank_a = op.rank_c = -1;
    for (int8_t& p : op.peer_told) p = -1;
    op.elem_begin = g.first;
    op.elem_count = g.second - g.first;
    op.cell_begin = g.first;
    if (req.algo == Algo::kRabenseifner && req.piece_elems != 0) op.cell_begin = g.first / req.piece_elems * req.piece_elems;
    return op;
  }
  Range ChunkRange(int chunk) const { return req.ranges[static_cast<size_t>(chunk)]; }

  // Cuts the contiguous chunk list `chunks` into transfer pieces: one piece per
  // chunk, or, when the request names a piece length, pieces of that length
  // over the whole contiguous element range (fewer, larger ops).
  std::vector<Range> Pieces(const std::vector<int>& chunks) const {
    std::vector<Range> out;
    if (chunks.empty()) return out;
    if (req.piece_elems == 0 || req.algo != Algo::kRabenseifner) {
      for (int c : chunks) out.push_back(ChunkRange(c));
      return out;
    }
    // Pieces are the cells of a fixed grid over the message (multiples of the
    // piece length), clipped to the run: an element lies in the same cell in
    // every step.
    const size_t b = ChunkRange(chunks.front()).first, e = ChunkRange(chunks.back()).second;
    size_t x = b;
    while (x < e) {
      const size_t cell_end = (x / req.piece_elems + 1) * req.piece_elems;
      out.emplace_back(x, std::min(e, cell_end));
      x = std::min(e, cell_end);
    }
    return out;
  }

  void AttachOut(Op* op, int to) {
    uint32_t k = prog.sent_to[to]++;
    op->flags |= kOpStoreRemote;
    op->peer_out = static_cast<int8_t>(to);
    op->region_out = static_cast<uint8_t>(RegionOf(to, req.rank));
    op->slot_out = k % slots;
    op->wait_credit = k >= slots ? k - slots + 1 : 0;
    op->post_out = k + 1;
  }

  void AttachIn(Op* op, int from) {
    uint32_t k = prog.received_from[from]++;
    op->src_a = kSrcStage;
    op->peer_in = static_cast<int8_t>(from);
    op->region_in = static_cast<uint8_t>(RegionOf(req.rank, from));
    op->slot_in = k % slots;
    op->wait_in = k + 1;
    op->post_credit = k + 1;
  }

  // ---- ranks on one GPU (ProgramRequest::shared_gpu) ----
  // Source a (or c) is rank `who`'s sendbuf.
  void PullA(Op* op, int who) {
    op->src_a = kSrcPeer;
    op->rank_a = static_cast<int8_t>(who);
    op->flags |= kOpRoundPeer;
  }
  void PullC(Op* op, int who) {
    op->rank_c = static_cast<int8_t>(who);
    op->flags |= kOpRoundPeer;
  }
  // The value goes into `to`'s recvbuf; `read_on`: and is read there by an op of that rank.
  void StoreTo(Op* op, int to, bool read_on) {
    op->store_peers = static_cast<uint8_t>(op->store_peers | (1u << to));
    if (!read_on) return;
    op->flags |= kOpPeersReadBack;
    int m = 0;
    while (m < kMaxPeerPosts && op->post_told[m] != 0) ++m;
    if (m == kMaxPeerPosts) IBCOMM_FAIL(INVALID_ARGUMENT, "schedule: an op tells too many ranks.\n");
    op->peer_told[m] = static_cast<int8_t>(to);
    op->post_told[m] = ++told[to];
  }
  // Source a is what `from` stored into recvbuf.
  void TakeArrived(Op* op, int from) {
    op->src_a = kSrcRecv;
    op->peer_in = static_cast<int8_t>(from);
    op->wait_peer = ++heard[from];
  }
  void Finish(Op* op) {
    op->flags |= kOpStoreLocal | kOpRoundWire;
    if (req.apply_scale) op->flags |= kOpScale;
  }

  // Plain send of a chunk taken from `src` (sendbuf or recvbuf).
  void Send(const Range& g, OpSrc src, int to) {
    Op op = Base(g);
    op.src_a = src;
    AttachOut(&op, to);
    prog.ops.push_back(op);
  }

  // Receive a chunk; optionally add `add` to it, store locally and/or forward.
  void Recv(const Range& g, int from, OpSrc add, bool store_local, bool scale, int forward_to) {
    Op op = Base(g);
    op.src_b = add;
    if (store_local) op.flags |= kOpStoreLocal;
    if (scale) op.flags |= kOpRoundWire;
    if (scale && req.apply_scale) op.flags |= kOpScale;
    AttachIn(&op, from);
    if (forward_to >= 0) AttachOut(&op, forward_to);
    prog.ops.push_back(op);
  }

  // A piece, and the rank of the halving that ends up with it (-1: a run of several
  // ranks' blocks).
  struct Piece {
    Range range;
    int owner;
  };
  // What a step receives, in order.  The first `forward` pieces go on to
  // `forward_to` in the same op, and are stored here as well when `keep`; the
  // others always are.
  struct Arrivals {
    std::vector<Piece> pieces;
    OpSrc add = kSrcNone;
    bool final_sum = false;
    size_t forward = 0;
    int forward_to = -1;
    bool keep = true;
  };
  // Contributions of extra ranks that this rank adds in a step (see Joiner).
  struct Joins {
    std::function<int(const Piece&)> from;  // the extra rank, or -1
    bool done;                              // they are in recvbuf already
    int From(const Piece& g) const { return from ? from(g) : -1; }
  };
  // One exchange step with a single partner: `sends` leave, of which the first
  // `sent` already did (forwarded as they arrived), and `in` arrives.  Sends run at
  // most `slots` ahead of the receives so that neither side can block on credits
  // the other side has not had a chance to return.
  void Exchange(int peer, const std::vector<Piece>& sends, size_t sent, OpSrc send_src, const Arrivals& in, const Joins& joins = Joins()) {
    size_t si = sent, ri = 0;
    auto send = [&]() {
      const Piece& g = sends[si++];
      const int from = joins.From(g);
      if (from >= 0 && !joins.done) Recv(g.range, from, send_src, false, false, peer);
      else Send(g.range, from >= 0 ? kSrcRecv : send_src, peer);
    };
    while (si < sends.size() && si < slots) send();
    for (const Piece& g : in.pieces)
      if (joins.From(g) >= 0 && !joins.done) Recv(g.range, joins.From(g), in.add, true, false, -1);
    while (ri < in.pieces.size()) {
      const Piece& g = in.pieces[ri];
      const bool fwd = ri < in.forward;
      const int from = joins.From(g);
      Recv(g.range, peer, from >= 0 ? kSrcRecv : in.add, in.keep || !fwd, in.final_sum, fwd ? in.forward_to : -1);
      ++ri;
      if (si < sends.size()) send();
    }
    while (si < sends.size()) send();
  }
};

std::vector<int> ChunksOfBlocks(const std::vector<std::vector<int>>& blocks, int b, int e) {
  std::vector<int> out;
  for (int i = b; i < e; ++i) out.insert(out.end(), blocks[static_cast<size_t>(i)].begin(), blocks[static_cast<size_t>(i)].end());
  return out;
}

// The ring of ranks that share a GPU.  The steps, the order of the additions and the owners are those of BuildRing.
// The first step's partner is read where it is, and a result travels from recvbuf to recvbuf: 34 reads and writes
// per eight elements and rank instead of 44 (8 ranks).
template <typename ChunkAt>
void BuildRingOnOneGpu(Builder* bld, size_t positions, size_t group, ChunkAt at) {
  const ProgramRequest& q = bld->req;
  const int ws = q.world_size, r = q.rank;
  const int from = Mod(r - 1, ws), to = Mod(r + 1, ws);
  for (size_t i0 = 0; i0 < positions; i0 += group) {
    const size_t i1 = std::min(positions, i0 + group);
    for (int k = 0; k <= ws - 2; ++k) {  // reduce-scatter
      for (size_t i = i0; i < i1; ++i) {
        const int c = at(Mod(r - 1 - k, ws), i);
        if (c < 0) continue;
        Op op = bld->Base(bld->ChunkRange(c));
        op.src_b = kSrcSend;
        if (k == 0) bld->PullA(&op, from);
        else bld->AttachIn(&op, from);
        if (k < ws - 2) {
          bld->AttachOut(&op, to);
        } else {
          bld->Finish(&op);
          bld->StoreTo(&op, to, ws > 2);
        }
        bld->prog.ops.push_back(op);
      }
    }
    for (int k = 0; k <= ws - 3; ++k) {  // all-gather
      for (size_t i = i0; i < i1; ++i) {
        const int c = at(Mod(r - k, ws), i);
        if (c < 0) continue;
        Op op = bld->Base(bld->ChunkRange(c));
        bld->TakeArrived(&op, from);
        bld->StoreTo(&op, to, k < ws - 3);
        bld->prog.ops.push_back(op);
      }
    }
  }
}

void BuildRing(Builder* bld) {
  const ProgramRequest& q = bld->req;
  const int ws = q.world_size, r = q.rank;
  const int from = Mod(r - 1, ws), to = Mod(r + 1, ws);
  const std::vector<std::vector<int>> blocks = GetRankToChunk(q.ranges.size(), static_cast<size_t>(ws));
  size_t positions = 0;
  for (const auto& b : blocks) positions = std::max(positions, b.size());
  // i-th chunk of a block, ids descending inside the block.
  auto at = [&](int blk, size_t i) -> int {
    const std::vector<int>& b = blocks[static_cast<size_t>(blk)];
    return i < b.size() ? b[b.size() - 1 - i] : -1;
  };
  // Chunks at the same position of their blocks form a chain: every op of a
  // chain waits for the op the upstream rank ran one step earlier.  Chains
  // are independent of each other, so a group of them is walked step by step
  // (all chains' step k before any chain's step k + 1): while one chain's
  // flag travels, the CTA moves the others' data.  A group of g chains keeps
  // up to g transfers ahead of the downstream rank's receives, so it needs
  // g + 1 staging slots (with g slots every rank would wait for a credit that
  // its neighbour can only return after the same wait).  With s slots an op
  // needs its neighbour's op s - g before it: with g + 1 the ranks go op by op,
  // each waiting for the other's hand-over (4 us on one GPU), so half the
  // slots are left to run ahead into.
  const size_t group = std::max<size_t>(1, std::min<size_t>(positions, bld->slots / 2));
  if (q.shared_gpu) return BuildRingOnOneGpu(bld, positions, group, at);
  for (size_t i0 = 0; i0 < positions; i0 += group) {
    const size_t i1 = std::min(positions, i0 + group);
    for (size_t i = i0; i < i1; ++i) {
      const int c = at(r, i);
      if (c >= 0) bld->Send(bld->ChunkRange(c), kSrcSend, to);
    }
    for (int k = 0; k <= ws - 2; ++k) {  // reduce-scatter
      const bool final_step = (k == ws - 2);
      for (size_t i = i0; i < i1; ++i) {
        const int c = at(Mod(r - 1 - k, ws), i);
        if (c < 0) continue;
        bld->Recv(bld->ChunkRange(c), from, kSrcSend, /*store_local=*/final_step, /*scale=*/final_step, to);
      }
    }
    for (int k = 0; k <= ws - 2; ++k) {  // all-gather
      for (size_t i = i0; i < i1; ++i) {
        const int c = at(Mod(r - k, ws), i);
        if (c < 0) continue;
        bld->Recv(bld->ChunkRange(c), from, kSrcNone, true, false, k != ws - 2 ? to : -1);
      }
    }
  }
}

// The halving of `p` ranks (a power of two) over their `blocks`, and the order in
// which pieces travel so that a piece can be handed on in the op that receives it.
struct Halving {
  using Piece = Builder::Piece;
  const Builder& bld;
  const std::vector<std::vector<int>>& blocks;
  int p, exp;

  // Blocks rank `v` still works on after `steps` steps.
  std::pair<int, int> Run(int v, int steps) const {
    int b = 0, e = p;
    for (int s = 0; s < steps; ++s) {
      const int mid = e - (e - b) / 2;
      if (v < (v ^ (1 << s))) b = mid;
      else e = mid;
    }
    return {b, e};
  }
  std::vector<Piece> Pieces(int v, int steps) const {
    const std::pair<int, int> run = Run(v, steps);
    std::vector<Piece> out;
    for (const Range& g : bld.Pieces(ChunksOfBlocks(blocks, run.first, run.second))) out.push_back({g, run.second - run.first == 1 ? v : -1});
    return out;
  }
  std::vector<Piece> Own(int v) const { return Pieces(v, exp); }
  size_t LongestOwn() const {
    size_t most = 0;
    for (int v = 0; v < p; ++v) most = std::max(most, Own(v).size());
    return most;
  }

  // What rank `v` receives in step `s`, in order: first what it gives away in
  // step s + 1, as its partner there wants it, then what it keeps.
  std::vector<Piece> Kept(int v, int s) const {
    if (s + 1 == exp) return Own(v);
    std::vector<Piece> out = Kept(v ^ (1 << (s + 1)), s + 1);
    const std::vector<Piece> rest = Pieces(v, s + 2);
    out.insert(out.end(), rest.begin(), rest.end());
    return out;
  }
  // What rank `v` stores into its partner's recvbuf in step `t` of the doubling, in order (ranks on one GPU): its own
  // block, then what came in the steps before.
  std::vector<Piece> Delivered(int v, int t) const {
    std::vector<Piece> out = Own(v);
    for (int u = 0; u < t; ++u) {
      const std::vector<Piece> came = Delivered(DoublingPartner(v, u), u);
      out.insert(out.end(), came.begin(), came.end());
    }
    return out;
  }
  int DoublingPartner(int v, int t) const { return v ^ (1 << (exp - 1 - t)); }
  // What rank `v` has collected when step `t` of the doubling begins, in the order
  // it passes it on: what came in last first, since that is handed on on arrival.
  std::vector<Piece> Collected(int v, int t) const {
    if (t == 0) return Own(v);
    std::vector<Piece> out = Collected(DoublingPartner(v, t - 1), t - 1);
    const std::vector<Piece> before = Collected(v, t - 1);
    out.insert(out.end(), before.begin(), before.end());
    return out;
  }
};

// The rank of the halving that adds extra rank `x`'s contribution to the block of
// `owner`.  No sum may get longer before its last additions than where an extra rank is
// folded into a partner first: with all of them added by the owner after the halving, one
// by one, 7 ranks' sums of bf16 were 13 % further from the exact ones, 5 ranks' 5 %.
//   * One extra rank: the owner adds it to the sum of two that the first step leaves.
//     (Before that step: 5 ranks x 16 MiB 79 us against 76.5, 3 x 16 MiB 53.4 against 52.)
//   * Two or three: before the halving, to what a rank has of its own, a different rank for
//     every extra one.  Every rank does so for one block of each, so all have the same to
//     do.  Against the owner after the halving: 6 ranks x 64 MiB 365 -> 353 us, 7 ranks
//     475 -> 457; 7 x 64 MiB with a bf16 wire 408 -> 412.
int Joiner(int owner, int x) { return owner ^ x; }

// A segment of the message: chunks [first, second).
using Segment = std::pair<size_t, size_t>;

// The chunks of every rank of the halving in a segment.
std::vector<std::vector<int>> SegmentBlocks(const Segment& segment, int p) {
  std::vector<std::vector<int>> blocks = GetRankToChunk(segment.second - segment.first, static_cast<size_t>(p));
  for (std::vector<int>& b : blocks)
    for (int& c : b) c += static_cast<int>(segment.first);
  return blocks;
}

// Halving and doubling of one segment.
void BuildHalvingDoubling(Builder* bld, const Segment& segment) {
  const int ws = bld->req.world_size, r = bld->req.rank;
  const int p = static_cast<int>(util::FloorPow2(static_cast<uint64_t>(ws)));
  const int extra = ws - p;
  const int exp = util::GetExpOfTwo(static_cast<uint64_t>(p));
  auto real_rank = [extra](int v) { return v < extra ? 2 * v + 1 : v + extra; };
  const std::vector<std::vector<int>> blocks = SegmentBlocks(segment, p);
  const Halving half{*bld, blocks, p, exp};
  const std::vector<Builder::Piece> none;
  using Piece = Builder::Piece;
  using Arrivals = Builder::Arrivals;

  const int vrank = r < 2 * extra ? r / 2 : r - extra;
  const size_t slots = bld->slots;
  // Where there are extra ranks, at most four ranks halve, and every piece is of one
  // block.  Their contributions are added before step `join_step` (see Joiner), in the op
  // that sends a piece or ahead of those that add to what is kept.  That relies on an extra
  // rank getting rid of all it sends; where its blocks do not fit into the slots, it waits
  // for ranks that have got further, and they for it.  There the contributions come before
  // all else.
  Builder::Joins joins{};
  int join_step = extra > 1 ? 0 : 1;
  if (extra != 0) {
    joins.from = [&](const Piece& g) -> int {
      for (int x = 0; x < extra; ++x)
        if (Joiner(g.owner, x) == vrank) return 2 * x;
      return -1;
    };
    joins.done = join_step < exp && half.LongestOwn() > slots;
    if (joins.done) join_step = 0;
    for (int x = 0; x < extra && joins.done; ++x)
      for (const Piece& g : half.Own(Joiner(vrank, x))) bld->Recv(g.range, 2 * x, kSrcSend, true, false, -1);
  }
  const bool join_last = extra != 0 && join_step == exp;

  // Halving.  A partial sum that goes to the next step's partner is forwarded in
  // the op that computes it and not stored, up to the partner's slots: those are
  // all free until that step, so no forward waits for a credit that the partner
  // could only return after waiting for one of ours.
  size_t sent = 0;        // of what this step sends, forwarded during the one before
  size_t first_sent = 0;  // of my own block, to the first partner of the doubling
  const std::vector<Piece> own = half.Own(vrank);
  for (int s = 0; s < exp; ++s) {
    const int vpeer = vrank ^ (1 << s);
    const std::vector<Piece> sends = half.Kept(vpeer, s);
    Arrivals in;
    in.pieces = half.Kept(vrank, s);
    in.add = s == 0 ? kSrcSend : kSrcRecv;
    size_t next_sent = 0;
    if (s + 1 < exp) {
      in.forward = next_sent = std::min(half.Kept(vrank ^ (1 << (s + 1)), s + 1).size(), slots);
      in.forward_to = real_rank(vrank ^ (1 << (s + 1)));
      in.keep = false;
    } else if (!join_last) {
      // My block is final.  Its way back leads to the same partner: behind what
      // goes there in this step, into the slots that leaves free.
      in.final_sum = true;
      in.forward = first_sent = sends.size() < slots ? std::min(own.size(), slots - sends.size()) : 0;
      in.forward_to = real_rank(vpeer);
    }
    bld->Exchange(real_rank(vpeer), sends, sent, s == 0 ? kSrcSend : kSrcRecv, in, s == join_step ? joins : Builder::Joins());
    sent = next_sent;
  }
  if (join_last) {
    Arrivals in;
    in.pieces = own;
    in.add = kSrcRecv;
    in.final_sum = true;
    in.forward = first_sent = std::min(own.size(), slots);
    in.forward_to = real_rank(half.DoublingPartner(vrank, 0));
    bld->Exchange(0, none, 0, kSrcNone, in);
  }
  for (int x = 0; x < extra; ++x) bld->Exchange(2 * x, own, 0, kSrcRecv, Arrivals());
  // Doubling, with the same forwards: what arrives in a step goes on in the next.
  sent = first_sent;
  for (int t = 0; t < exp; ++t) {
    const int vpeer = half.DoublingPartner(vrank, t);
    Arrivals in;
    in.pieces = half.Collected(vpeer, t);
    if (t + 1 < exp) {
      in.forward = std::min(in.pieces.size(), slots);
      in.forward_to = real_rank(half.DoublingPartner(vrank, t + 1));
    }
    bld->Exchange(real_rank(vpeer), half.Collected(vrank, t), sent, kSrcRecv, in);
    sent = in.forward;
  }
}

// Halving and doubling of one segment by ranks that share a GPU.  The first step's partner and the extra ranks'
// contributions are read where they are, final blocks go straight to every rank that the doubling takes them to from
// here, and extra ranks have nothing to do.  An extra rank's contribution is added to a sum of two (its partner's, in
// the op (a + c) + b), so that every sum is as long at its last additions as where extra ranks are folded first:
//   one: in the last step, by the owner;  two: in the first step, by the two ranks that keep the block, one each;
//   three: in the first step, two of them by the owner (one to each term), one by the other rank.
void BuildHalvingDoublingOnOneGpu(Builder* bld, const Segment& segment) {
  using Piece = Builder::Piece;
  const int ws = bld->req.world_size, r = bld->req.rank;
  const int p = static_cast<int>(util::FloorPow2(static_cast<uint64_t>(ws)));
  const int extra = ws - p;
  const int exp = util::GetExpOfTwo(static_cast<uint64_t>(p));
  auto real_rank = [extra](int v) { return v < extra ? 2 * v + 1 : v + extra; };
  const std::vector<std::vector<int>> blocks = SegmentBlocks(segment, p);
  const Halving half{*bld, blocks, p, exp};
  const int vrank = r < 2 * extra ? r / 2 : r - extra;
  const size_t slots = bld->slots;

  // The extra rank whose contribution this rank adds to a piece in step `s`, or -1.
  auto joins = [&](const Piece& g, int s) -> int {
    if (extra == 0 || g.owner < 0) return -1;
    if (extra == 1) return s == exp - 1 ? 0 : -1;
    if (s != 0) return -1;
    return g.owner == vrank ? 2 * (extra - 2) : 2 * (extra == 2 ? 1 : 2);
  };
  size_t sent = 0;  // of what this step sends, forwarded during the one before
  for (int s = 0; s < exp; ++s) {
    const int peer = real_rank(vrank ^ (1 << s));
    const std::vector<Piece> sends = s == 0 ? std::vector<Piece>() : half.Kept(vrank ^ (1 << s), s);
    const std::vector<Piece> arrivals = half.Kept(vrank, s);
    const bool last = s + 1 == exp;
    const int next = last ? -1 : real_rank(vrank ^ (1 << (s + 1)));
    const size_t forward = last ? 0 : std::min(half.Kept(vrank ^ (1 << (s + 1)), s + 1).size(), slots);
    size_t si = sent;
    while (si < sends.size() && si < slots) bld->Send(sends[si++].range, kSrcRecv, peer);
    for (size_t ri = 0; ri < arrivals.size(); ++ri) {
      const Piece& g = arrivals[ri];
      OpSrc mine = s == 0 ? kSrcSend : kSrcRecv;
      if (extra == 3 && s == 0 && g.owner == vrank) {
        Op first = bld->Base(g.range);
        bld->PullA(&first, 0);
        first.src_b = kSrcSend;
        first.flags |= kOpStoreLocal;
        bld->prog.ops.push_back(first);
        mine = kSrcRecv;
      }
      Op op = bld->Base(g.range);
      op.src_b = mine;
      if (s == 0) bld->PullA(&op, peer);
      else bld->AttachIn(&op, peer);
      if (const int x = joins(g, s); x >= 0) bld->PullC(&op, x);
      if (last) {
        bld->Finish(&op);
        for (int t = 0; t < exp; ++t) bld->StoreTo(&op, real_rank(half.DoublingPartner(vrank, t)), t + 1 < exp);
        for (int x = 0; x < extra; ++x) bld->StoreTo(&op, 2 * x, false);
      } else if (ri < forward) {
        bld->AttachOut(&op, next);
      } else {
        op.flags |= kOpStoreLocal;
      }
      bld->prog.ops.push_back(op);
      if (si < sends.size()) bld->Send(sends[si++].range, kSrcRecv, peer);
    }
    while (si < sends.size()) bld->Send(sends[si++].range, kSrcRecv, peer);
    sent = forward;
  }
  // What comes in one step of the doubling goes to the partners of all later ones at once.
  for (int t = 0; t + 1 < exp; ++t) {
    const int vpeer = half.DoublingPartner(vrank, t);
    for (const Piece& g : half.Delivered(vpeer, t)) {
      Op op = bld->Base(g.range);
      bld->TakeArrived(&op, real_rank(vpeer));
      for (int u = t + 1; u < exp; ++u) bld->StoreTo(&op, real_rank(half.DoublingPartner(vrank, u)), u + 1 < exp);
      bld->prog.ops.push_back(op);
    }
  }
}

// An extra rank hands every block of its message to the rank that adds it (Joiner) and
// gets the results back from the owners.  Piece by piece over the blocks, so that all of
// them have something to work on.  It sends a segment ahead of the one it receives if the
// others' slots hold one: its sends then wait only for what those take in before they
// return anything of the segment being received (5 ranks x 64 MiB 301 -> 298 us, 6 ranks
// 395 -> 386).
void BuildExtraRank(Builder* bld, const std::vector<Segment>& segments) {
  const int ws = bld->req.world_size, x = bld->req.rank / 2;
  const int p = static_cast<int>(util::FloorPow2(static_cast<uint64_t>(ws)));
  const int extra = ws - p;
  auto real_rank = [extra](int v) { return v < extra ? 2 * v + 1 : v + extra; };
  std::vector<std::vector<Builder::Piece>> moves(segments.size());
  std::vector<bool> ahead(segments.size());
  for (size_t k = 0; k < segments.size(); ++k) {
    const std::vector<std::vector<int>> blocks = SegmentBlocks(segments[k], p);
    const Halving half{*bld, blocks, p, util::GetExpOfTwo(static_cast<uint64_t>(p))};
    std::vector<std::vector<Builder::Piece>> pieces;
    for (int v = 0; v < p; ++v) pieces.push_back(half.Own(v));
    const size_t most = half.LongestOwn();
    ahead[k] = most <= bld->slots;
    for (size_t i = 0; i < most; ++i)
      for (const std::vector<Builder::Piece>& b : pieces)
        if (i < b.size()) moves[k].push_back(b[i]);
  }
  auto send = [&](size_t k) {
    for (const Builder::Piece& m : moves[k]) bld->Send(m.range, kSrcSend, real_rank(Joiner(m.owner, x)));
  };
  send(0);
  for (size_t k = 0; k < segments.size(); ++k) {
    const bool next = k + 1 < segments.size();
    if (next && ahead[k + 1]) send(k + 1);
    for (const Builder::Piece& m : moves[k]) bld->Recv(m.range, real_rank(m.owner), kSrcNone, true, false, -1);
    if (next && !ahead[k + 1]) send(k + 1);
  }
}

// Segment after segment.  No op of a segment waits for one of a later segment, so
// what holds for one segment (all slots free when it begins) holds for each.
void BuildRabenseifner(Builder* bld) {
  const ProgramRequest& q = bld->req;
  std::vector<Segment> segments;
  for (size_t k = 0; k < q.segments.size(); ++k)
    segments.emplace_back(q.segments[k], k + 1 < q.segments.size() ? q.segments[k + 1] : q.ranges.size());
  if (segments.empty()) segments.emplace_back(0, q.ranges.size());
  const int extra = q.world_size - static_cast<int>(util::FloorPow2(static_cast<uint64_t>(q.world_size)));
  const bool is_extra = q.rank < 2 * extra && (q.rank & 1) == 0;
  if (q.shared_gpu) {
    for (size_t k = 0; k < segments.size() && !is_extra; ++k) BuildHalvingDoublingOnOneGpu(bld, segments[k]);
    return;
  }
  if (is_extra) return BuildExtraRank(bld, segments);
  for (const Segment& g : segments) BuildHalvingDoubling(bld, g);
}

}  // namespace

std::vector<int> InPeers(Algo algo, int rank, int world_size) {
  std::vector<int> peers;
  if (world_size <= 1) return peers;
  if (algo == Algo::kRing) {
    peers.push_back(Mod(rank - 1, world_size));
    return peers;
  }
  // Rabenseifner: the halving partners by step, then the extra ranks; an extra
  // rank hears from every rank of the halving.
  const int p = static_cast<int>(util::FloorPow2(static_cast<uint64_t>(world_size)));
  const int extra = world_size - p;
  const int exp = util::GetExpOfTwo(static_cast<uint64_t>(p));
  auto real_rank = [extra](int v) { return v < extra ? 2 * v + 1 : v + extra; };
  if (rank < 2 * extra && (rank & 1) == 0) {
    for (int v = 0; v < p; ++v) peers.push_back(real_rank(v));
    return peers;
  }
  const int vrank = rank < 2 * extra ? rank / 2 : rank - extra;
  for (int s = 0; s < exp; ++s) peers.push_back(real_rank(vrank ^ (1 << s)));
  for (int x = 0; x < extra; ++x) peers.push_back(2 * x);
  return peers;
}

int NumRegions(Algo algo, int world_size) {
  int m = 1;
  for (int r = 0; r < world_size; ++r) m = std::max(m, static_cast<int>(InPeers(algo, r, world_size).size()));
  return m;
}

size_t MaxChunkElems(const std::vector<Range>& ranges) {
  size_t m = 0;
  for (const Range& g : ranges) m = std::max(m, g.second - g.first);
  return m;
}

StageLayout PlanStage(const ProgramRequest& req) {
  StageLayout st{};
  st.offset = req.stage_offset;
  st.regions = static_cast<uint32_t>(NumRegions(req.algo, req.world_size));
  const bool pieces = req.algo == Algo::kRabenseifner && req.piece_elems != 0;
  uint64_t bytes = (pieces ? req.piece_elems : MaxChunkElems(req.ranges)) * req.wire_elem_bytes;
  st.slot_bytes = (bytes + 127) & ~uint64_t(127);
  if (st.slot_bytes == 0) st.slot_bytes = 128;
  uint64_t per_region = req.stage_bytes / st.regions;
  uint64_t slots = per_region / st.slot_bytes;
  st.slots = slots > 64 ? 64u : static_cast<uint32_t>(slots);
  if (st.slots < 2) st.slots = 0;
  return st;
}

Program BuildProgram(const ProgramRequest& req) {
  if (req.world_size < 1 || req.world_size > kMaxRanks)
    IBCOMM_FAIL(NOT_SUPPORTED, "Device collectives support 1..%d ranks (got %d).\n", kMaxRanks, req.world_size);
  Builder bld(req);
  if (req.world_size == 1) return bld.prog;
  if (bld.slots == 0)
    IBCOMM_FAIL(INVALID_ARGUMENT,
                "The staging area (%llu bytes) cannot hold two slots of %llu bytes for each of %u "
                "regions.\n",
                static_cast<unsigned long long>(req.stage_bytes),
                static_cast<unsigned long long>(bld.prog.stage.slot_bytes), bld.prog.stage.regions);
  switch (req.algo) {
    case Algo::kRing: BuildRing(&bld); break;
    case Algo::kRabenseifner: BuildRabenseifner(&bld); break;
    default:
      IBCOMM_FAIL(INVALID_ARGUMENT, "No op program exists for algorithm '%s'.\n", AlgoName(req.algo));
  }
  // A cell is stored and read as a whole or in parts, never across cells.
  std::unordered_map<uint64_t, uint32_t> stored;  // cell -> 1 + the last op that stored into it
  for (size_t i = 0; i < bld.prog.ops.size(); ++i) {
    Op& op = bld.prog.ops[i];
    if (op.src_a == kSrcRecv || op.src_b == kSrcRecv) {
      const auto it = stored.find(op.cell_begin);
      if (it != stored.end()) {
        op.wait_local = it->second;
        bld.prog.ops[it->second - 1].flags |= kOpReadBack;
      }
    }
    if (op.flags & kOpStoreLocal) stored[op.cell_begin] = static_cast<uint32_t>(i + 1);
  }
  return bld.prog;
}

std::vector<Range> SplitForDevice(size_t len_elements, size_t elem_bytes, size_t world_size,
                                  int64_t env_chunk_bytes, size_t max_chunk_bytes, size_t chunks_per_rank) {
  std::vector<Range> base = SplitBuffer(len_elements, elem_bytes, world_size, env_chunk_bytes);
  const size_t vec_elems = 128 / elem_bytes;
  if (env_chunk_bytes <= 0) {
    if (chunks_per_rank < 1) chunks_per_rank = 1;
    size_t per = util::ceilDiv(len_elements, chunks_per_rank * world_size);
    const bool round = per >= 4 * vec_elems && per % vec_elems != 0;
    if (round) per = util::ceilDiv(per, vec_elems) * vec_elems;
    if (round || chunks_per_rank != 4) {
      base.clear();
      for (size_t b = 0; b < len_elements; b += per) base.emplace_back(b, std::min(len_elements, b + per));
    }
  }
  size_t largest = MaxChunkElems(base) * elem_bytes;
  if (max_chunk_bytes == 0 || largest <= max_chunk_bytes) return base;
  // Cut every chunk into `f` pieces on 128-byte boundaries.
  const size_t f = util::ceilDiv(largest, max_chunk_bytes);
  size_t piece = util::ceilDiv(MaxChunkElems(base), f);
  piece = util::ceilDiv(piece, vec_elems) * vec_elems;
  std::vector<Range> out;
  out.reserve(base.size() * f);
  for (const Range& g : base) {
    size_t b = g.first;
    for (size_t k = 0; k < f; ++k) {
      size_t e = (k + 1 == f) ? g.second : std::min(g.second, b + piece);
      out.emplace_back(b, e);  // possibly empty; keeps f pieces per chunk
      b = e;
    }
  }
  return out;
}

std::vector<Range> SplitSegments(size_t len_elements, size_t piece_elems, size_t segment_pieces, std::vector<size_t>* segments) {
  std::vector<Range> out;
  for (size_t b = 0; b < len_elements; b += piece_elems) out.emplace_back(b, std::min(len_elements, b + piece_elems));
  for (size_t c = 0; c < out.size(); c += segment_pieces) segments->push_back(c);
  return out;
}

size_t MaxPieceElems(uint64_t stage_bytes, int regions, size_t wire_elem_bytes) {
  const size_t step = std::max<size_t>(32, 128 / wire_elem_bytes);
  const size_t most = static_cast<size_t>(stage_bytes / (static_cast<uint64_t>(regions) * 2) / wire_elem_bytes) / step * step;
  return std::max(most, step);
}

uint64_t RingStageBytes(uint64_t pool_bytes, int ranks_on_gpu) {
  return ranks_on_gpu > 1 ? std::min(pool_bytes, kSharedGpuStageBytes / static_cast<uint64_t>(ranks_on_gpu)) : pool_bytes;
}

size_t RingChunksPerRank(size_t len_elements, size_t elem_bytes, size_t world_size, bool one_gpu) {
  const int positions = Tunable("IBCOMM_RING_POSITIONS", one_gpu ? 2 : 4);
  size_t cpr = positions >= 1 && positions <= 64 ? static_cast<size_t>(positions) : 4;
  const int min_env = Tunable("IBCOMM_RING_MIN_CHUNK", one_gpu ? 65536 : 16384);
  const size_t min_chunk = min_env > 0 ? static_cast<size_t>(min_env) : 1;
  const size_t bytes = len_elements * elem_bytes;
  while (cpr > 1 && bytes / (cpr * world_size) < min_chunk) --cpr;
  return cpr;
}

uint64_t TwoShotWindowElems(uint64_t n, uint64_t cap_elems, size_t esize, int world_size, int channels) {
  if (cap_elems == 0) cap_elems = 1;
  if (n <= 1) return 1;
  const uint64_t windows = (n + cap_elems - 1) / cap_elems;
  const uint64_t per = (n + windows - 1) / windows;
  const uint64_t granule = static_cast<uint64_t>(16 / esize) * static_cast<uint64_t>(world_size) * static_cast<uint64_t>(channels > 0 ? channels : 1);
  const uint64_t rounded = (per + granule - 1) / granule * granule;
  // The pool holds a whole number of vectors, so the cap keeps windows aligned.
  return rounded < cap_elems ? rounded : cap_elems;
}

std::string ValidateProgram(const Program& prog, uint64_t len_elements, size_t wire_elem_bytes, int world_size) {
  for (size_t i = 0; i < prog.ops.size(); ++i) {
    const Op& op = prog.ops[i];
    const char* why = nullptr;
    const bool reads_stage = op.src_a == kSrcStage;
    const bool writes_stage = (op.flags & kOpStoreRemote) != 0;
    auto is_rank = [world_size](int r) { return r >= 0 && r < world_size; };
    bool told_ok = true;
    for (int m = 0; m < kMaxPeerPosts; ++m) told_ok = told_ok && (op.post_told[m] == 0 || is_rank(op.peer_told[m]));
    told_ok = told_ok && (op.wait_peer == 0 || is_rank(op.peer_in));
    if (op.elem_begin > len_elements || op.elem_count > len_elements - op.elem_begin) {
      why = "range outside the message";
    } else if (op.cell_begin > op.elem_begin) {
      why = "cell starts after the range";
    } else if ((reads_stage || writes_stage) &&
               (op.elem_begin - op.cell_begin + op.elem_count) * wire_elem_bytes > prog.stage.slot_bytes) {
      why = "range does not fit its staging slot";
    } else if (reads_stage && (op.region_in >= prog.stage.regions || op.slot_in >= prog.stage.slots)) {
      why = "input slot outside the staging area";
    } else if (writes_stage && (op.region_out >= prog.stage.regions || op.slot_out >= prog.stage.slots)) {
      why = "output slot outside the staging area";
    } else if ((writes_stage || op.wait_credit != 0 || op.post_out != 0) && (op.peer_out < 0 || op.peer_out >= world_size)) {
      why = "peer_out is not a rank";
    } else if ((op.wait_in != 0 || op.post_credit != 0) && (op.peer_in < 0 || op.peer_in >= world_size)) {
      why = "peer_in is not a rank";
    } else if ((op.src_a == kSrcPeer && !is_rank(op.rank_a)) || (op.rank_c != -1 && !is_rank(op.rank_c)) || (op.store_peers >> world_size) != 0 || !told_ok) {
      why = "names a rank that is none";
    } else if (op.src_b == kSrcStage || op.src_b == kSrcPeer) {
      why = "second source is not this rank's";
    } else if (op.wait_local > i) {
      why = "waits for an op that comes later";
    }
    if (why != nullptr) return "op " + std::to_string(i) + ": " + why + ": " + DescribeOp(op);
  }
  return std::string();
}

std::string DescribeOp(const Op& op) {
  static const char* const src[] = {"-", "send", "recv", "stage", "peer", "?", "?", "?"};
  char buf[256];
  snprintf(buf, sizeof(buf),
           "[%llu+%llu] a=%s b=%s%s%s%s in=%d(r%u s%u w%u c%u) out=%d(r%u s%u w%u p%u)",
           static_cast<unsigned long long>(op.elem_begin), static_cast<unsigned long long>(op.elem_count),
           src[op.src_a & 7], src[op.src_b & 7], (op.flags & kOpScale) ? " scale" : "",
           (op.flags & kOpStoreLocal) ? " local" : "", (op.flags & kOpStoreRemote) ? " remote" : "", op.peer_in,
           op.region_in, op.slot_in, op.wait_in, op.post_credit, op.peer_out, op.region_out, op.slot_out,
           op.wait_credit, op.post_out);
  return buf;
}

}  // namespace ibcomm
