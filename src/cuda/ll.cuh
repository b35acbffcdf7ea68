// Hand-over of small amounts of data between ranks without flags of its own: a
// line of 16 bytes carries eight of data, and beside each four of them the
// number of the call.  Whoever reads a line again and again until both numbers
// are there has the data with the same access; a hand-over costs a store and a
// load, no fence, no flag and no second trip for the data.  Twice the bytes, so it
// is for messages that wait rather than stream.  (The idea is that of the low-latency
// protocols of collective libraries; layout, numbering and code are this library's.)
//
// A half line is one 64-bit access, so its data and its number cannot be seen
// apart; nothing depends on the order of the halves.  The memory is used for
// lines only (what is left of earlier calls has other numbers), and a line is
// written once per call.  It is double-buffered by the parity of the call: a rank
// that stores into call k + 2's lines has finished call k + 1, so every rank has
// started that call, and thus finished call k, whose lines these were.
#pragma once

#include "flags.cuh"
#include "vec_ops.cuh"

namespace ibcomm {
namespace dev {

// The number lines of call `seq` carry: never 0, which memory holds at first.
__device__ __forceinline__ uint32_t LineNumber(uint64_t seq) {
  const uint32_t n = static_cast<uint32_t>(seq);
  return n != 0 ? n : 0xffffffffu;
}

// 16 bytes of data as two lines `apart` bytes from each other, and back once both are there.  The first lines of
// a warp's data lie side by side, and so do the second ones: whole sectors.
__device__ __forceinline__ void StLines(unsigned char* p, uint64_t apart, uint4 v, uint32_t number) {
  const uint64_t hi = static_cast<uint64_t>(number) << 32;
  asm volatile("st.relaxed.sys.global.v2.u64 [%0], {%1,%2};" ::"l"(p), "l"(hi | v.x), "l"(hi | v.y) : "memory");
  asm volatile("st.relaxed.sys.global.v2.u64 [%0], {%1,%2};" ::"l"(p + apart), "l"(hi | v.z), "l"(hi | v.w) : "memory");
}
struct Lines {
  uint64_t w[4];
};
__device__ __forceinline__ Lines LdLines(const unsigned char* p, uint64_t apart) {
  Lines l;
  asm volatile("ld.relaxed.sys.global.v2.u64 {%0,%1}, [%2];" : "=l"(l.w[0]), "=l"(l.w[1]) : "l"(p) : "memory");
  asm volatile("ld.relaxed.sys.global.v2.u64 {%0,%1}, [%2];" : "=l"(l.w[2]), "=l"(l.w[3]) : "l"(p + apart) : "memory");
  return l;
}
__device__ __forceinline__ bool HaveArrived(const Lines& l, uint32_t number) {
  return static_cast<uint32_t>(l.w[0] >> 32) == number && static_cast<uint32_t>(l.w[1] >> 32) == number &&
         static_cast<uint32_t>(l.w[2] >> 32) == number && static_cast<uint32_t>(l.w[3] >> 32) == number;
}
__device__ __forceinline__ uint4 DataOf(const Lines& l) {
  return make_uint4(static_cast<uint32_t>(l.w[0]), static_cast<uint32_t>(l.w[1]), static_cast<uint32_t>(l.w[2]), static_cast<uint32_t>(l.w[3]));
}

// One thread's patience while it reads lines again: every 64 rounds it looks at the
// abort word and at the clock.
struct LineWait {
  uint64_t t0 = 0;
  uint32_t spin = 0;
  // kStatusOk: go on reading; else why the call is over for this thread.
  __device__ __forceinline__ uint32_t Again(const WaitCtx& w) {
    if ((++spin & 63u) != 0) return kStatusOk;
    if (LdRelaxedSys(&Ctl(*w.peers, w.rank)->abort_seq) == w.seq) return kStatusPeerAbort;
    const uint64_t now = GlobalTimerNs();
    if (t0 == 0) t0 = now;
    return now - t0 > w.timeout_ns ? kStatusWaitTimeout : kStatusOk;
  }
};
// Reports that, and stops everybody else where this thread is the first to know.
__device__ inline void LineWaitOver(const WaitCtx& w, uint32_t status, uint32_t kind, int peer, int op_index, uint64_t expected) {
  ReportFailure(w, status, kind, peer, op_index, expected, 0);
  if (status == kStatusWaitTimeout) BroadcastAbort(w);
}

}  // namespace dev
}  // namespace ibcomm
