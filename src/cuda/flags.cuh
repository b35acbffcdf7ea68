// Device-side synchronisation primitives: system-scope acquire/release
// accesses to the peer-visible control words, the bounded wait every spin in
// this library goes through, and failure reporting.  A wait that runs out
// never traps or hangs: it records what it was waiting for, tells the other
// CTAs and the peers to stop, and makes the kernel return normally.
#pragma once

#include <cstdint>

#include "ibcomm/device_types.h"

namespace ibcomm {
namespace dev {

__device__ __forceinline__ uint64_t LdAcquireSys(const uint64_t* p) {
  uint64_t v;
  asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint64_t LdRelaxedSys(const uint64_t* p) {
  uint64_t v;
  asm volatile("ld.relaxed.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void StReleaseSys(uint64_t* p, uint64_t v) {
  asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void StRelaxedSys(uint64_t* p, uint64_t v) {
  asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void FenceSys() { asm volatile("fence.acq_rel.sys;" ::: "memory"); }
// The same with the scope the ranks of a collective need (PeerTable::one_gpu).
__device__ __forceinline__ uint64_t LdAcquirePeers(const uint64_t* p, bool one_gpu) {
  if (!one_gpu) return LdAcquireSys(p);
  uint64_t v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void StReleasePeers(uint64_t* p, uint64_t v, bool one_gpu) {
  if (!one_gpu) StReleaseSys(p, v);
  else asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void FencePeers(bool one_gpu) {
  if (!one_gpu) FenceSys();
  else asm volatile("fence.acq_rel.gpu;" ::: "memory");
}
__device__ __forceinline__ uint64_t GlobalTimerNs() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ ControlPage* Ctl(const PeerTable& peers, int rank) {
  return reinterpret_cast<ControlPage*>(peers.arena[rank]);
}

// What a waiter needs to know to give up cleanly.
struct WaitCtx {
  const PeerTable* peers;
  DeviceStatus* status;  // device memory
  uint32_t* doorbell;    // host-mapped word, set non-zero on failure
  uint64_t seq;
  uint64_t timeout_ns;
  int rank;
  int world_size;
  int channel;
};

__device__ inline void ReportFailure(const WaitCtx& w, uint32_t code, uint32_t kind, int peer, int op_index,
                                     uint64_t expected, uint64_t seen) {
  if (w.status != nullptr && atomicCAS(&w.status->code, 0u, code) == 0u) {
    w.status->kind = kind;
    w.status->rank = w.rank;
    w.status->peer = peer;
    w.status->channel = w.channel;
    w.status->op_index = op_index;
    w.status->expected = expected;
    w.status->seen = seen;
    w.status->seq = w.seq;
    __threadfence_system();
  }
  if (w.doorbell != nullptr) *reinterpret_cast<volatile uint32_t*>(w.doorbell) = code;
}

// Sequence number of the running collective: one more than the number this
// rank has begun before.  Every CTA of the rank takes it exactly once: by one
// thread, `scratch` may be read behind the CTA's next barrier; `ctas` = CTAs of this rank, `scratch` is a __shared__ word.
//
// ControlPage::call_word holds (calls begun << 16) | CTAs of the running call
// that have taken their number.  The last CTA to take it advances the count:
// nothing else reads the word before this rank's next kernel, so it need not
// wait for the call's end, and one atomic does for the load at the start and
// the counter, fence and barrier at the end that it replaced (1.5-2 us of an 8 us
// call on one GPU).
__device__ __forceinline__ void TakeCallNumber(const PeerTable& peers, int rank, uint64_t* scratch, unsigned ctas) {
  unsigned long long* const word = reinterpret_cast<unsigned long long*>(&Ctl(peers, rank)->call_word);
  const unsigned long long old = atomicAdd(word, 1ull);
  if (static_cast<unsigned>(old & 0xffffu) + 1u == ctas) atomicAdd(word, (1ull << 16) - ctas);
  *scratch = static_cast<uint64_t>(old >> 16) + 1;
}
// The same with all threads of the CTA, barrier included.
__device__ inline uint64_t BeginCollective(const PeerTable& peers, int rank, uint64_t* scratch, unsigned ctas) {
  if (threadIdx.x == 0) TakeCallNumber(peers, rank, scratch, ctas);
  __syncthreads();
  return *scratch;
}

// Makes every CTA of every rank of this call stop waiting.
__device__ inline void BroadcastAbort(const WaitCtx& w) {
  for (int r = 0; r < w.world_size; ++r) StRelaxedSys(&Ctl(*w.peers, r)->abort_seq, w.seq);
  __threadfence_system();
}

// Spins until *flag >= target.  Returns false after the limit, or when this
// call was aborted elsewhere; the failure has then been reported.
__device__ inline bool WaitGE(const uint64_t* flag, uint64_t target, const WaitCtx& w, uint32_t kind, int peer,
                              int op_index) {
  const bool one_gpu = w.peers->one_gpu != 0;
  uint64_t v = LdAcquirePeers(flag, one_gpu);
  if (v >= target) return true;
  const uint64_t t0 = GlobalTimerNs();
  const uint64_t* abort_word = &Ctl(*w.peers, w.rank)->abort_seq;
  for (uint32_t spin = 1;; ++spin) {
    v = LdAcquirePeers(flag, one_gpu);
    if (v >= target) return true;
    if ((spin & 31u) == 0u) {
      if (LdRelaxedSys(abort_word) == w.seq) {
        ReportFailure(w, kStatusPeerAbort, kind, peer, op_index, target, v);
        return false;
      }
      if (GlobalTimerNs() - t0 > w.timeout_ns) {
        ReportFailure(w, kStatusWaitTimeout, kind, peer, op_index, target, v);
        BroadcastAbort(w);
        return false;
      }
      if (spin > 4096u) __nanosleep(100);
    }
  }
}

}  // namespace dev
}  // namespace ibcomm
