/* Allreduce entry point that performs no allocation of any kind.
 *
 * This function has no counterpart in the reference; it exists for programs
 * that must not allocate device memory while they run: code whose whole memory
 * budget is handed to another allocator at start-up (a framework's caching
 * allocator, a fixed arena of a real-time service), where a stray cudaMalloc
 * can fail or fragment the budget, and code on latency-critical paths, where
 * cudaMalloc / cudaFree stall the whole device.  Such callers cannot create an
 * EmuWorld or a Communicator, both of which allocate an arena.
 *
 * What it does: the allreduce (sum, times `scale`) of `num_ranks` float buffers
 * that live on the CURRENT device, i.e. the single-GPU, several-ranks form of
 * the library's small-message allreduce.  One kernel reads every rank's buffer,
 * adds in rank order (every rank gets the same bits) and writes every rank's
 * result; sendbufs[r] == recvbufs[r] is allowed.
 *
 *     limit  IBCOMM_NO_ALLOC_MAX_RANKS ranks (8), IBCOMM_NO_ALLOC_MAX_BYTES
 *            bytes per buffer (32 KiB = 8192 floats)
 *     cost   none: the kernel needs no memory beside the caller's buffers
 *
 * Larger requests are refused with code 1 and a message; nothing is launched.
 * The function calls no cudaMalloc, cudaFree or other allocating routine
 * (torch's included); the caller passes the inputs and the outputs.
 *
 * First call on a device: with CUDA's lazy module loading (the default) the
 * driver may load the kernel only at that moment, which is work on the
 * driver's side that can take time or fail: make one warm-up call per device
 * at start-up (or run with CUDA_MODULE_LOADING=EAGER); the no-allocation
 * guarantee holds from the second call on.
 *
 * Stream capture: none of the calls may be made while `stream` is being
 * captured, since every call ends by synchronising the stream.
 *
 * Threads: calls share nothing; several threads and streams may be in a call
 * at the same time, on one GPU or on several.
 *
 * The call enqueues its work on `stream` (0 = the null stream), waits for it
 * and returns 0, or 1 (bad argument / beyond the limits) or 3 (a CUDA call
 * failed).  `errbuf` (may be NULL) receives a description of a failure.
 */
#pragma once

#include <stddef.h>

#define IBCOMM_NO_ALLOC_MAX_RANKS 8
#define IBCOMM_NO_ALLOC_MAX_BYTES (32 * 1024)

#ifdef __cplusplus
extern "C" {
#endif

int ibcomm_emu_oneshot_allreduce_f32_noalloc(const float* const* sendbufs, float* const* recvbufs, int num_ranks,
                                             size_t len_elements, float scale, void* stream, char* errbuf,
                                             size_t errbuf_len);

#ifdef __cplusplus
}
#endif
