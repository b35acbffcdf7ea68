"""The kernels at the lengths and alignments where their splits can go wrong, each against a plain PyTorch
computation of the same operation."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch

import allreduce_proto_b200 as ar

pytestmark = pytest.mark.gpu


def values(n, dtype, seed, offset=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    if dtype in (torch.int32, torch.int64):
        t = torch.randint(-1000, 1000, (n + offset,), device="cuda", dtype=dtype, generator=g)
    else:
        t = (torch.rand(n + offset, device="cuda", generator=g) * 2 - 1).to(dtype)
    return t[offset:]


@pytest.mark.parametrize("offsets", [(0, 0), (1, 1), (3, 3), (1, 0), (4, 4)])
@pytest.mark.parametrize("types", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32),
                                   (torch.float16, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.float64, torch.float64),
                                   (torch.int64, torch.int64)])
def test_copy_scale_quanta_heads_and_tails(types, offsets):
    # One quantum per thread, 256 threads per block: lengths around a quantum, a block and several blocks; slices that
    # share an offset (peeled up to the boundary) and slices that do not (element by element).
    for n in (1, 3, 7, 8, 15, 16, 17, 33, 2047, 2048, 2049, 4096 + 5, 100003):
        x = values(n, types[0], n, offsets[0])
        guard = torch.full((n + offsets[1] + 8,), 7, device="cuda", dtype=types[1])
        y = guard[offsets[1]:offsets[1] + n]
        scale = 1.0 if types[0] == torch.int64 else 0.5
        ar.ops.copy_scale(x, y, scale=scale)
        assert torch.equal(y, (x.double() * scale).to(types[1])), n
        assert torch.all(guard[:offsets[1]] == 7) and torch.all(guard[offsets[1] + n:] == 7), n


@pytest.mark.parametrize("staged", [0, 1, 3])
@pytest.mark.parametrize("offset", [0, 1, 3])
@pytest.mark.parametrize("ws", [2, 3, 8])
def test_reduce_scatter_and_all_gather_ragged_blocks(ws, offset, staged):
    # Blocks that start off the 16-byte boundary of the remote side (every rank's head differs), shorter than a unit,
    # a unit and a bit, and long enough for parts on cache lines; buffers that miss the boundary alike.
    world = ar.EmuWorld(ws, 1 << 20, 1 << 20)
    world.set_direct_staging(staged)
    for dtype in (torch.float32, torch.bfloat16, torch.float64):
        for m in (1, 2, 5, 9, 1023, 70001):
            full = [values(m * ws, dtype, 10 * m + r, offset) for r in range(ws)]
            want = torch.stack([t.double() for t in full]).sum(0) * 0.5
            guard = [torch.full((m + offset + 8,), 7, device="cuda", dtype=dtype) for _ in range(ws)]
            shards = [g[offset:offset + m] for g in guard]
            world.reduce_scatter(full, shards, scale=0.5)
            tol = 1e-5 if dtype == torch.float32 else (2e-2 if dtype == torch.bfloat16 else 1e-12)
            for r in range(ws):
                torch.testing.assert_close(shards[r].double(), want[r * m:(r + 1) * m], rtol=tol, atol=tol)
                assert torch.all(guard[r][:offset] == 7) and torch.all(guard[r][offset + m:] == 7)
            guard = [torch.full((m * ws + offset + 8,), 7, device="cuda", dtype=dtype) for _ in range(ws)]
            gathered = [g[offset:offset + m * ws] for g in guard]
            world.all_gather(shards, gathered)
            whole = torch.cat(shards)
            for r in range(ws):
                assert torch.equal(gathered[r], whole)
                assert torch.all(guard[r][:offset] == 7) and torch.all(guard[r][offset + m * ws:] == 7)
    world.close()


@pytest.mark.parametrize("mode", [0, 3])
@pytest.mark.parametrize("algo", ["oneshot", "direct", "ring", "rabenseifner"])
@pytest.mark.parametrize("ws", [2, 3, 5, 8])
def test_allreduce_ragged_ends(ws, algo, mode):
    # Lengths around a vector, a round of loads per thread, a stage of the executor and a part on cache lines, all with
    # a ragged end; slices off the boundary; 16-bit wires where there are op programs.
    world = ar.EmuWorld(ws)
    world.set_direct_staging(mode)
    wires = [None, torch.bfloat16] if algo in ("ring", "rabenseifner") else [None]
    for dtype in (torch.float32, torch.bfloat16, torch.float64):
        for offset in (0, 1):
            for n in (ws + 1, 129, 2047, 8 * 512 * ws + 5, 100003):
                for wire in wires if dtype == torch.float32 else [None]:
                    ins = [values(n, dtype, n + r, offset) for r in range(ws)]
                    guard = [torch.full((n + offset + 8,), 7, device="cuda", dtype=dtype) for _ in range(ws)]
                    outs = [g[offset:offset + n] for g in guard]
                    world.allreduce(ins, outs, algo=algo, scale=1.0 / ws, wire=wire)
                    want = torch.stack([t.double() for t in ins]).sum(0) / ws
                    tol = 2e-2 if dtype == torch.bfloat16 or wire is not None else (1e-5 if dtype == torch.float32 else 1e-12)
                    for g, o in zip(guard, outs):
                        torch.testing.assert_close(o.double(), want, rtol=tol, atol=tol)
                        assert torch.equal(o, outs[0])
                        assert torch.all(g[:offset] == 7) and torch.all(g[offset + n:] == 7)
    world.close()


@pytest.mark.parametrize("mode", [0, 3])
@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("ws", [2, 3, 4, 5, 6, 7, 8])
def test_rabenseifner_segments(ws, in_place, mode):
    # A small staging area makes segments of a few pieces: one, an exact number of them, a last one that is shorter
    # or lacks blocks, and many; partial sums read back from recvbuf.
    p = 1 << (ws.bit_length() - 1)
    regions = max(p.bit_length() - 1 + ws - p, p if ws != p else 0)
    area = 2 * regions * 65536
    world = ar.EmuWorld(ws, area // 2, area // 2)
    world.set_direct_staging(mode)
    for wire, size in ((None, 4), (torch.bfloat16, 2)):
        piece = 65536 // size
        for n in (p, piece * p, piece * p + 1, 2 * piece * p - 5, 5 * piece * p + piece + 3):
            if n < 4 * ws:
                n = 4 * ws
            ins = [values(n, torch.float32, n + r, 0) for r in range(ws)]
            want = torch.stack([t.double() for t in ins]).sum(0) / ws
            outs = ins if in_place else [torch.full_like(t, 7) for t in ins]
            world.allreduce(ins, outs, algo="rabenseifner", scale=1.0 / ws, wire=wire)
            tol = 2e-2 if wire is not None else 1e-5
            for o in outs:
                torch.testing.assert_close(o.double(), want, rtol=tol, atol=tol)
                assert torch.equal(o, outs[0])
    world.close()


@pytest.mark.parametrize("wire", [None, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("ws", [2, 3, 5, 8])
def test_staged_windows_reused(ws, wire):
    # Windows that are reused many times while their lines are dropped as they are read: parts that end inside a
    # 128-byte line, parts of whole lines, a short last window; a second call on the same windows.
    world = ar.EmuWorld(ws, 64 << 10, 64 << 10)
    world.set_direct_staging(2)
    for n in (8 * ws, 8 * 1237, 8 * 16384 * ws, 1000000 + 8):
        for call in range(2):
            ins = [values(n, torch.float32, n + r + call, 0) for r in range(ws)]
            before = [t.clone() for t in ins]
            outs = [torch.full_like(t, 7) for t in ins]
            world.allreduce(ins, outs, algo="direct", scale=1.0 / ws, wire=wire)
            want = torch.stack([t.double() for t in ins]).sum(0) / ws
            tol = 2e-2 if wire is not None else 1e-5
            for o, i, b in zip(outs, ins, before):
                torch.testing.assert_close(o.double(), want, rtol=tol, atol=tol)
                assert torch.equal(i, b)
    world.close()


@pytest.mark.parametrize("mode", [0, 3])
@pytest.mark.parametrize("ws", [2, 5, 8])
def test_rabenseifner_drops_lines(ws, mode):
    # Long enough for slots whose lines are dropped as they are read; a ragged end, in place as well, two calls.
    world = ar.EmuWorld(ws)
    world.set_direct_staging(mode)
    n = (52 << 20) // 4 // ws + 7
    for in_place in (False, True):
        for call in range(2):
            ins = [values(n, torch.float32, r + call, 0) for r in range(ws)]
            want = torch.stack([t.double() for t in ins]).sum(0) / ws
            outs = ins if in_place else [torch.full_like(t, 7) for t in ins]
            world.allreduce(ins, outs, algo="rabenseifner", scale=1.0 / ws)
            for o in outs:
                torch.testing.assert_close(o.double(), want, rtol=1e-5, atol=1e-5)
    world.close()


@pytest.mark.parametrize("mode", [0, 3])
@pytest.mark.parametrize("ws", [2, 5, 7, 8])
def test_rabenseifner_drops_lines_of_reused_slots(ws, mode):
    # Two slots per partner for many transfers (two ranks that share buffers have none): a slot is written again, by a peer, right after its lines were
    # dropped.  Small whole numbers are summed, exactly, so a transfer that a late drop destroyed cannot come out right by chance.
    area = 4 << 20
    p = 1 << (ws.bit_length() - 1)
    regions = max(p.bit_length() - 1 + ws - p, p if ws != p else 0)
    n = (64 << 20) // 4 // ws + 7
    largest_piece = area // (2 * regions) // 4
    assert n // largest_piece // 2 > 2 * 2  # half the message goes to the first partner
    world = ar.EmuWorld(ws, area // 2, area // 2)
    world.set_direct_staging(mode)
    for in_place in (False, True):
        for call in range(3):
            ins = [values(n, torch.float32, r + call, 0) if call == 0 else torch.full((n,), float(1 + r + call), device="cuda") for r in range(ws)]
            want = torch.stack([t.double() for t in ins]).sum(0)
            outs = ins if in_place else [torch.full_like(t, 7) for t in ins]
            world.allreduce(ins, outs, algo="rabenseifner")
            for o in outs:
                if call == 0:
                    torch.testing.assert_close(o.double(), want, rtol=1e-5, atol=1e-5)
                else:
                    assert torch.equal(o.double(), want)
    world.close()


@pytest.mark.parametrize("mode", [0, 3])
@pytest.mark.parametrize("ws", [3, 5, 6, 7])
def test_rabenseifner_blocks_longer_than_the_slots(ws, mode):
    # The message as one, in small pieces of which the slots hold a few: what the extra ranks send (mode 3) comes before
    # all else then.  In place as well.
    lib = ar._native.lib()
    lib.ibcomm_set_tunable(b"IBCOMM_RABEN_PIECES", 64)
    try:
        world = ar.EmuWorld(ws, 1 << 20, 1 << 20)
        world.set_direct_staging(mode)
        for dtype in (torch.float32, torch.bfloat16):
            n = 64 * 16384 + 5
            for in_place in (False, True):
                ins = [values(n, dtype, n + r) for r in range(ws)]
                want = torch.stack([t.double() for t in ins]).sum(0) / ws
                outs = ins if in_place else [torch.full_like(t, 7) for t in ins]
                world.allreduce(ins, outs, algo="rabenseifner", scale=1.0 / ws)
                tol = 2e-2 if dtype == torch.bfloat16 else 1e-5
                for o in outs:
                    torch.testing.assert_close(o.double(), want, rtol=tol, atol=tol)
                    assert torch.equal(o, outs[0])
        world.close()
    finally:
        lib.ibcomm_set_tunable(b"IBCOMM_RABEN_PIECES", -1)


def test_ranks_as_rows_of_one_tensor():
    # The rows are tensors made while the call reads them.
    world = ar.EmuWorld(4)
    x = values(4 * 4096, torch.float32, 1).view(4, 4096)
    want = x.double().sum(0)
    y = torch.zeros_like(x)
    world.allreduce(x, y, algo="oneshot")
    shards, whole = torch.zeros(4, 1024, device="cuda"), torch.zeros_like(x)
    world.reduce_scatter(x, shards)
    world.all_gather(shards, whole)
    for r in range(4):
        torch.testing.assert_close(y[r].double(), want, rtol=1e-5, atol=1e-5)
        torch.testing.assert_close(whole[r].double(), want, rtol=1e-5, atol=1e-5)
    world.close()


def test_longer_and_pinned_outputs():
    # A prefix of a longer output is written, and memory of the host that the GPU can reach.
    x = values(1000, torch.float32, 1)
    y = torch.full((1008,), 7.0, device="cuda")
    ar.ops.copy_scale(x, y, scale=0.5)
    assert torch.equal(y[:1000], x * 0.5) and torch.all(y[1000:] == 7)
    h = torch.zeros(1000, pin_memory=True)
    ar.ops.copy_scale(x, h, scale=0.5)
    torch.cuda.synchronize()
    assert torch.equal(h, (x * 0.5).cpu())
    world = ar.EmuWorld(2)
    ins, outs = [x, y], [torch.full((1003,), 7.0, device="cuda") for _ in range(2)]
    world.allreduce(ins, outs, algo="oneshot")
    for o in outs:
        assert torch.equal(o[:1000], x + y[:1000]) and torch.all(o[1000:] == 7)
    world.close()


@pytest.mark.parametrize("mode", [2, 0])
@pytest.mark.parametrize("pages", [6, 7, 8])
def test_staged_in_the_smallest_staging(pages, mode):
    # Three windows of each kind is the least the staged kernel works with: six pages of staging.
    world = ar.EmuWorld(2, (pages - 1) * 4096, 4096)
    world.set_direct_staging(mode)
    ins = [values(8 * 3001, torch.float32, r) for r in range(2)]
    outs = [torch.full_like(t, 7) for t in ins]
    world.allreduce(ins, outs, algo="direct", wire=torch.bfloat16)
    want = ins[0].double() + ins[1].double()
    for o in outs:
        torch.testing.assert_close(o.double(), want, rtol=2e-2, atol=2e-2)
    world.close()


@pytest.mark.parametrize("wire", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("ws", [2, 3, 5, 8])
def test_direct_wire_in_place_and_through_the_pool(ws, wire):
    # fp32 buffers with a 16-bit wire: used in place, and through the pool with the roles in every block and in blocks
    # of their own.  The same values are rounded at the same places: the same bits.  What the pool refuses stays refused.
    world = ar.EmuWorld(ws, 1 << 20, 1 << 20)
    for n in (8, 8 * ws, 8 * 1237, 8 * 512 * ws + 8, 300000, 1 << 20):
        ins = [values(n, torch.float32, n + r) for r in range(ws)]
        want = torch.stack([t.double() for t in ins]).sum(0) / ws
        results = []
        for mode, split in ((0, 0), (2, 0), (2, 1), (1, 0)):
            world.set_direct_staging(mode)
            ar.utils.set_tunable("IBCOMM_STAGED_SPLIT", split)
            try:
                outs = [torch.full_like(t, 7) for t in ins]
                world.allreduce(ins, outs, algo="direct", scale=1.0 / ws, wire=wire)
                bufs = [t.clone() for t in ins]
                world.allreduce(bufs, None, algo="direct", scale=1.0 / ws, wire=wire)
            finally:
                ar.utils.set_tunable("IBCOMM_STAGED_SPLIT", -1)
            results += outs + bufs
        for o in results:
            assert torch.equal(o, results[0])
        torch.testing.assert_close(results[0].double(), want, rtol=2e-2, atol=2e-2)
    for mode in (0, 2):
        world.set_direct_staging(mode)
        for n, offset in ((4097, 0), (4096, 1)):
            bufs = [values(n, torch.float32, r, offset) for r in range(ws)]
            with pytest.raises(ar.IbcommError) as e:
                world.allreduce(bufs, None, algo="direct", wire=wire)
            assert e.value.code == ar.NOT_SUPPORTED
    world.close()


@pytest.mark.parametrize("ws", [2, 3, 4, 5, 8])
def test_direct_in_place_kernels_agree(ws):
    # One kernel for all ranks, and each rank's own with barriers (in place, and through the pool): the same sums in rank
    # order, so the same bits.  Lengths around a block of threads and a vector, slices that miss the boundary alike or not.
    world = ar.EmuWorld(ws, 1 << 20, 1 << 20)
    for dtype in (torch.float32, torch.float64, torch.bfloat16, torch.float16, torch.int32, torch.int64):
        k = 16 // torch.empty(0, dtype=dtype).element_size()
        scale = 1.0 if dtype in (torch.int32, torch.int64) else 1.0 / ws
        for n in (ws, 1, k, 128 * k - 1, 128 * k + 1, 70001):
            for off_in, off_out in ((0, 0), (1, 1), (1, 0), (k - 1, k - 1)):
                ins = [values(n, dtype, n + r, off_in) for r in range(ws)]
                results = []
                for mode in (0, 3, 1):
                    world.set_direct_staging(mode)
                    guard = [torch.full((n + off_out + 8,), 7, device="cuda", dtype=dtype) for _ in range(ws)]
                    outs = [g[off_out:off_out + n] for g in guard]
                    world.allreduce(ins, outs, algo="direct", scale=scale)
                    for g in guard:
                        assert torch.all(g[:off_out] == 7) and torch.all(g[off_out + n:] == 7)
                    results += outs
                for o in results:
                    assert torch.equal(o, results[0])
                full = [values(n * ws, dtype, n + r, off_in) for r in range(ws)]
                halves = []
                for mode in (0, 3, 1):
                    world.set_direct_staging(mode)
                    guard = [torch.full((n + off_out + 8,), 7, device="cuda", dtype=dtype) for _ in range(ws)]
                    shards = [g[off_out:off_out + n] for g in guard]
                    world.reduce_scatter(full, shards, scale=scale)
                    whole = [torch.full((n * ws + off_in + 8,), 7, device="cuda", dtype=dtype) for _ in range(ws)]
                    outs = [g[off_in:off_in + n * ws] for g in whole]
                    world.all_gather(shards, outs)
                    for g in guard:
                        assert torch.all(g[:off_out] == 7) and torch.all(g[off_out + n:] == 7)
                    for g in whole:
                        assert torch.all(g[:off_in] == 7) and torch.all(g[off_in + n * ws:] == 7)
                    halves.append(outs)
                for outs in halves:
                    for o in outs:
                        assert torch.equal(o, halves[0][0])
    want = torch.stack([t.double() for t in ins]).sum(0)
    assert torch.equal(results[0].double(), want)  # int64: exact
    world.close()


@pytest.mark.parametrize("slots", [0, 3])
@pytest.mark.parametrize("algo", ["ring", "rabenseifner"])
@pytest.mark.parametrize("ws", [2, 3, 4, 5, 6, 7, 8])
def test_short_messages_as_lines_and_through_slots(ws, algo, slots):
    # Transfers as lines, and through the slots with flags: fewer elements than a pack per rank, packs that two ops share,
    # a pack per thread and several, more than one channel; slices off the boundary; 16-bit wires; in place.
    world = ar.EmuWorld(ws)
    world.set_direct_staging(slots)
    for dtype in (torch.float32, torch.float64, torch.bfloat16, torch.float16, torch.int32, torch.int64):
        whole = dtype in (torch.int32, torch.int64)
        scale = 1.0 if whole else 1.0 / ws
        for n in (ws, 2 * ws + 1, 129, 2521, 70001):
            for off_in, off_out in ((0, 0), (1, 1), (1, 0)):
                for wire in (None, torch.bfloat16, torch.float16) if dtype == torch.float32 else (None,):
                    ins = [values(n, dtype, n + r, off_in) for r in range(ws)]
                    want = torch.stack([t.double() for t in ins]).sum(0) * scale
                    guard = [torch.full((n + off_out + 8,), 7, device="cuda", dtype=dtype) for _ in range(ws)]
                    outs = [g[off_out:off_out + n] for g in guard]
                    world.allreduce(ins, outs, algo=algo, scale=scale, wire=wire)
                    tol = 0.0 if whole else (2e-2 if dtype in (torch.bfloat16, torch.float16) or wire is not None else (1e-5 if dtype == torch.float32 else 1e-12))
                    for g, o in zip(guard, outs):
                        torch.testing.assert_close(o.double(), want, rtol=tol, atol=tol)
                        assert torch.equal(o, outs[0])
                        assert torch.all(g[:off_out] == 7) and torch.all(g[off_out + n:] == 7)
                    world.allreduce(ins, None, algo=algo, scale=scale, wire=wire)
                    for i in ins:
                        torch.testing.assert_close(i.double(), want, rtol=tol, atol=tol)
    world.close()


@pytest.mark.parametrize("ws", [2, 5, 8])
def test_lines_of_many_calls(ws):
    # Calls of different lengths and algorithms back to back, other kernels between them: what earlier calls left in the
    # lines is not taken for a transfer.  Whole numbers, so that every call's result is exact.
    world = ar.EmuWorld(ws)
    sizes = [ws, 300000, 1000, 4096, 70001, 131072, 64, 262144]
    for turn in range(6):
        calls = []
        for k, n in enumerate(sizes):
            ins = [torch.full((n,), float(turn + k + r), device="cuda") + torch.arange(n, device="cuda") % 13 for r in range(ws)]
            want = torch.stack([t.double() for t in ins]).sum(0)
            outs = [torch.full_like(t, 7) for t in ins]
            world.allreduce(ins, outs, algo=("ring", "rabenseifner", "oneshot")[(turn + k) % 3 if n <= 262144 else 0], sync=False)
            calls.append((outs, want))
        torch.cuda.synchronize()
        for outs, want in calls:
            for o in outs:
                assert torch.equal(o.double(), want)
    world.close()


@pytest.mark.parametrize("algo", ["ring", "rabenseifner"])
def test_lines_wait_runs_out(algo):
    # A rank that takes no part in a short call: the others' waits for its lines end, the status says that it never came,
    # and the world stays usable.
    world = ar.EmuWorld(4)
    world.set_timeout_ms(200)
    ins = [values(4096, torch.float32, r) for r in range(4)]
    outs = [torch.zeros_like(t) for t in ins]
    world.set_silent_rank(1)
    with pytest.raises(ar.IbcommError) as e:
        world.allreduce(ins, outs, algo=algo)
    assert e.value.code == ar.TRANSPORT_ERROR
    assert world.last_status()["code"] in (1, 2)
    world.set_silent_rank(-1)
    world.set_timeout_ms(5000)
    world.allreduce(ins, outs, algo=algo)
    want = torch.stack([t.double() for t in ins]).sum(0)
    for o in outs:
        torch.testing.assert_close(o.double(), want, rtol=1e-5, atol=1e-5)
    world.close()


@pytest.fixture
def slots_only():
    # Messages of every length through the executor with slots and flags.
    ar.utils.set_tunable("IBCOMM_LINES_MAX_KIB", 0)
    yield
    ar.utils.set_tunable("IBCOMM_LINES_MAX_KIB", -1)


@pytest.mark.parametrize("mode", [0, 3])
@pytest.mark.parametrize("algo", ["ring", "rabenseifner"])
@pytest.mark.parametrize("ws", [2, 3, 4, 5, 6, 7, 8])
def test_op_programs_of_ranks_that_share_memory(slots_only, ws, algo, mode):
    # Programs that read the other ranks' sendbuf and store into their recvbuf, and those that send as between GPUs:
    # ragged ends, slices off the boundary, stages of one, two and three sources, few slots that are used many times, in
    # place (a buffer is overwritten while others still have to have read it), 16-bit wires.
    for pool in (0, 1 << 20):
        world = ar.EmuWorld(ws, pool, pool)
        world.set_direct_staging(mode)
        for dtype in (torch.float32, torch.float64, torch.bfloat16, torch.int64) if pool == 0 else (torch.float32, torch.bfloat16):
            whole = dtype == torch.int64
            scale = 1.0 if whole else 1.0 / ws
            for n, offset in ((4 * ws, 0), (2521, 0), (2521, 1), (8 * 512 * ws + 5, 0), (8 * 512 * ws, 0), (1 << 20, 0), (1000003, 0)):
                for wire in (None, torch.bfloat16) if dtype == torch.float32 else (None,):
                    ins = [values(n, dtype, n + r, offset) for r in range(ws)]
                    want = torch.stack([t.double() for t in ins]).sum(0) * scale
                    guard = [torch.full((n + offset + 8,), 7, device="cuda", dtype=dtype) for _ in range(ws)]
                    outs = [g[offset:offset + n] for g in guard]
                    tol = 0.0 if whole else (2e-2 if dtype == torch.bfloat16 or wire is not None else (1e-5 if dtype == torch.float32 else 1e-12))
                    for call in range(2):
                        world.allreduce(ins, outs, algo=algo, scale=scale, wire=wire)
                    world.allreduce(ins, None, algo=algo, scale=scale, wire=wire)
                    for g, o, i in zip(guard, outs, ins):
                        torch.testing.assert_close(o.double(), want, rtol=tol, atol=tol)
                        assert torch.equal(o, outs[0]) and torch.equal(i, o)
                        assert torch.all(g[:offset] == 7) and torch.all(g[offset + n:] == 7)
        world.close()


@pytest.mark.parametrize("mode", [0, 3])
@pytest.mark.parametrize("algo,ws", [("ring", 4), ("rabenseifner", 4), ("rabenseifner", 5)])
def test_executor_gives_up_cleanly(slots_only, algo, ws, mode):
    # A rank that takes no part, and one whose ops fail their self-check, with and without ranks that have no blocks in the
    # launch; the calls are counted for those too, so the world stays usable by every kernel.
    world = ar.EmuWorld(ws, 1 << 20, 1 << 20)
    world.set_direct_staging(mode)
    ins = [values(8192, torch.float32, r) for r in range(ws)]
    outs = [torch.zeros_like(t) for t in ins]
    want = torch.stack([t.double() for t in ins]).sum(0)
    for hook, codes in ((world.set_silent_rank, (1, 2)), (world.set_bad_program_rank, (3,))):
        world.set_timeout_ms(200)
        hook(1)
        with pytest.raises(ar.IbcommError) as e:
            world.allreduce(ins, outs, algo=algo)
        assert e.value.code == ar.TRANSPORT_ERROR
        assert world.last_status()["code"] in codes
        hook(-1)
        world.set_timeout_ms(5000)
        for other in (algo, "oneshot", "ring", algo):
            world.allreduce(ins, outs, algo=other)
            for o in outs:
                torch.testing.assert_close(o.double(), want, rtol=1e-5, atol=1e-5)
    world.close()


@pytest.mark.parametrize("dtype,wire", [(torch.float32, None), (torch.bfloat16, None), (torch.float32, torch.bfloat16)])
@pytest.mark.parametrize("ws", [2, 3, 4, 7, 8])
def test_staged_results_fetched_from_their_reducer(ws, dtype, wire):
    # Results that the storers fetch from their reducers' windows (more than two ranks, 8 MiB or more, copies by the threads)
    # and that are stored into every rank's window: windows that are reused many times, a short last one, parts that end
    # inside a line, several channels, copy roles in blocks of their own, calls back to back.
    world = ar.EmuWorld(ws, 128 << 10, 128 << 10)
    world.set_direct_staging(2)
    k = 8 if wire is not None or dtype == torch.bfloat16 else 4
    from_8_mib = (8 << 20) * k // 16
    for n in (k * ws, k * 1237, from_8_mib - k, from_8_mib, from_8_mib + k * 5003):
        ins = [values(n, dtype, n + r) for r in range(ws)]
        results = []
        for tma, split, channels in ((0, 0, 0), (0, 0, 3), (0, 1, 0), (1, 0, 0)):
            ar.utils.set_tunable("IBCOMM_STAGED_TMA", tma)
            ar.utils.set_tunable("IBCOMM_STAGED_SPLIT", split)
            try:
                outs = [torch.full_like(t, 7) for t in ins]
                for call in range(2):
                    world.allreduce(ins, outs, algo="direct", scale=1.0 / ws, wire=wire, channels=channels, sync=False)
                torch.cuda.synchronize()
                results += outs
            finally:
                ar.utils.set_tunable("IBCOMM_STAGED_TMA", -1)
                ar.utils.set_tunable("IBCOMM_STAGED_SPLIT", -1)
        want = torch.stack([t.double() for t in ins]).sum(0) / ws
        tol = 1e-5 if dtype == torch.float32 and wire is None else 2e-2
        torch.testing.assert_close(results[0].double(), want, rtol=tol, atol=tol)
        for o in results:
            assert torch.equal(o, results[0])
    world.close()


@pytest.mark.parametrize("mode", [0, 3])
@pytest.mark.parametrize("ws", [2, 3, 5, 8])
def test_one_shot_pushed_and_in_place(ws, mode):
    # The push into every rank's slot, several calls in a row on slots that alternate, and one kernel for all ranks: every
    # element type, a wire type that one-shot does not have, ragged ends, slices that miss the boundary alike or not.
    world = ar.EmuWorld(ws)
    world.set_direct_staging(mode)
    for dtype in (torch.float32, torch.float64, torch.bfloat16, torch.float16, torch.int32, torch.int64):
        whole = dtype in (torch.int32, torch.int64)
        scale = 1.0 if whole else 0.5
        for n in (1, 7, 2048, 2049, 70001):
            for off_in, off_out in ((0, 0), (1, 1), (1, 0)):
                ins = [values(n, dtype, n + r, off_in) for r in range(ws)]
                acc = ins[0].float() if dtype in (torch.bfloat16, torch.float16) else ins[0].clone()
                for t in ins[1:]:
                    acc += t
                want = acc.to(dtype) if whole else (acc * scale).to(dtype)
                guard = [torch.full((n + off_out + 8,), 7, device="cuda", dtype=dtype) for _ in range(ws)]
                outs = [g[off_out:off_out + n] for g in guard]
                for call in range(3):
                    world.allreduce(ins, outs, algo="oneshot", scale=scale, wire=torch.bfloat16 if dtype == torch.float32 else None, sync=False)
                world.allreduce(ins, None, algo="oneshot", scale=scale)
                for g, o, i in zip(guard, outs, ins):
                    assert torch.equal(o, want) and torch.equal(i, want)
                    assert torch.all(g[:off_out] == 7) and torch.all(g[off_out + n:] == 7)
    world.close()


@pytest.mark.parametrize("hook,codes", [("silent", (1, 2)), ("bad_program", (3,))])
@pytest.mark.parametrize("ws,rank", [(3, 0), (5, 0), (6, 2), (7, 4)])
def test_hooks_reach_extra_ranks(ws, rank, hook, codes):
    # Ranks that have no blocks where ranks share buffers: one that is to stay away, or to fail its self-check, still does.
    # Longer than what goes as lines.
    world = ar.EmuWorld(ws)
    world.set_timeout_ms(200)
    ins = [values(2000000, torch.float32, r) for r in range(ws)]
    outs = [torch.zeros_like(t) for t in ins]
    set_hook = world.set_silent_rank if hook == "silent" else world.set_bad_program_rank
    set_hook(rank)
    with pytest.raises(ar.IbcommError) as e:
        world.allreduce(ins, outs, algo="rabenseifner")
    assert e.value.code == ar.TRANSPORT_ERROR
    assert world.last_status()["code"] in codes
    set_hook(-1)
    world.set_timeout_ms(5000)
    for algo in ("rabenseifner", "ring"):
        world.allreduce(ins, outs, algo=algo)
        want = torch.stack([t.double() for t in ins]).sum(0)
        for o in outs:
            torch.testing.assert_close(o.double(), want, rtol=1e-5, atol=1e-5)
    world.close()


def test_silent_rank_of_direct_with_16_bit_wire():
    # The others wait for it in the staged kernel, although the buffers could be used in place.
    world = ar.EmuWorld(4)
    world.set_timeout_ms(200)
    ins = [values(1 << 16, torch.float32, r) for r in range(4)]
    outs = [torch.zeros_like(t) for t in ins]
    world.set_silent_rank(1)
    with pytest.raises(ar.IbcommError) as e:
        world.allreduce(ins, outs, algo="direct", wire=torch.bfloat16)
    assert e.value.code == ar.TRANSPORT_ERROR
    assert world.last_status()["code"] in (1, 2)
    world.set_silent_rank(-1)
    world.set_timeout_ms(5000)
    world.allreduce(ins, outs, algo="direct", wire=torch.bfloat16)
    want = torch.stack([t.double() for t in ins]).sum(0)
    for o in outs:
        torch.testing.assert_close(o.double(), want, rtol=2e-2, atol=2e-2)
    world.close()


def test_one_rank_with_blocks_in_prescribed_channels(slots_only):
    # One piece, one rank that sums it: as many blocks as there are flags of a rank (256) at most.
    world = ar.EmuWorld(2)
    for n in (2, 31):
        ins = [values(n, torch.float32, n + r) for r in range(2)]
        outs = [torch.full_like(t, 7) for t in ins]
        world.allreduce(ins, outs, algo="rabenseifner", channels=1000)
        assert 1 <= world.last_channels <= 256
        for o in outs:
            torch.testing.assert_close(o, ins[0] + ins[1], rtol=1e-6, atol=1e-6)
    world.close()


@pytest.mark.parametrize("mode", [0, 3])
@pytest.mark.parametrize("algo", ["ring", "rabenseifner"])
@pytest.mark.parametrize("ws", [2, 3, 5, 8])
def test_op_programs_in_prescribed_channels(ws, algo, mode):
    # Few channels for what goes as lines otherwise (packs that a thread handles one after the other, up to four and more),
    # for programs that share buffers and for those that send; more channels than there are packs, or than the GPU holds.
    world = ar.EmuWorld(ws)
    world.set_direct_staging(mode)
    for n in (ws, 2521, 16384, 65536 + 5, 262144, 600001):
        for dtype in (torch.float32, torch.bfloat16):
            ins = [values(n, dtype, n + r) for r in range(ws)]
            want = torch.stack([t.double() for t in ins]).sum(0) / ws
            tol = 1e-5 if dtype == torch.float32 else 2e-2
            for channels in (1, 2, 3, 8, 31, 1000):
                outs = [torch.full_like(t, 7) for t in ins]
                for call in range(2):
                    world.allreduce(ins, outs, algo=algo, scale=1.0 / ws, channels=channels)
                assert 1 <= world.last_channels <= channels
                for o in outs:
                    torch.testing.assert_close(o.double(), want, rtol=tol, atol=tol)
                    assert torch.equal(o, outs[0])
    world.close()


@pytest.mark.parametrize("ws", [2, 3, 8])
def test_prescribed_channels_of_buffers_in_place(ws):
    # Direct (with and without a 16-bit wire), one-shot and the halves keep to the blocks that the caller allows; the bits are
    # those of the kernel that runs for all ranks otherwise.
    world = ar.EmuWorld(ws)
    for n in (8 * ws, 8 * 1237, 65536):
        ins = [values(n, torch.float32, n + r) for r in range(ws)]
        for algo, wire in (("direct", None), ("direct", torch.bfloat16), ("oneshot", None)):
            want = [torch.full_like(t, 7) for t in ins]
            world.allreduce(ins, want, algo=algo, scale=1.0 / ws, wire=wire)
            for channels in (1, 3, 8):
                outs = [torch.full_like(t, 7) for t in ins]
                world.allreduce(ins, outs, algo=algo, scale=1.0 / ws, wire=wire, channels=channels)
                assert world.last_channels == channels
                for o, t in zip(outs, want):
                    assert torch.equal(o, t)
        block = n // ws
        full = [t[:block * ws] for t in ins]
        shards = [torch.full((block,), 7.0, device="cuda") for _ in range(ws)]
        world.reduce_scatter(full, shards, scale=0.5)
        for channels in (1, 3, 8):
            again = [torch.full_like(t, 7) for t in shards]
            world.reduce_scatter(full, again, scale=0.5, channels=channels)
            assert world.last_channels == channels
            whole = [torch.full_like(t, 7) for t in full]
            world.all_gather(shards, whole, channels=channels)
            assert world.last_channels == channels
            for r in range(ws):
                assert torch.equal(again[r], shards[r]) and torch.equal(whole[r], torch.cat(shards))
    world.close()


REPORTED_ONCE = """
import torch
import allreduce_proto_b200 as ar

world = ar.EmuWorld(2)
ins = [torch.arange(1000.0, device="cuda") + r for r in range(2)]
outs = [torch.full_like(t, 7) for t in ins]
shards = [torch.full((500,), 7.0, device="cuda") for _ in range(2)]
calls = [lambda: world.allreduce(ins, outs, algo="direct"), lambda: world.allreduce(ins, outs, algo="oneshot"),
         lambda: world.reduce_scatter(ins, shards), lambda: ar.ops.copy_scale(ins[0], outs[0], scale=1.0)]
for call in calls:
    call()
torch.cuda.synchronize()
stream = torch.cuda.Stream()
for call in calls:
    try:
        with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=stream):
            world.allreduce(ins, outs, algo="direct", stream=stream)
    except Exception:
        call()
    else:
        raise SystemExit("captured")
torch.cuda.synchronize()
assert torch.equal(torch.cat(shards), ins[0] + ins[1])
assert torch.equal(outs[0], ins[0]) and torch.equal(outs[1], ins[0] + ins[1])
"""


def test_an_error_is_reported_once():
    # A synchronous call cannot be captured and raises; what is launched after that does not report it again.  In a process
    # of its own: the capture that failed leaves torch's random generator unusable.
    run = subprocess.run([sys.executable, "-c", REPORTED_ONCE], cwd=Path(__file__).resolve().parent.parent, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
