"""The one-GPU interpreter where it can go wrong: several CTAs and slices per threadblock, chunks and buffers at every
alignment, reduces longer than one batch - bit for bit against the CPU interpreter."""
import pytest
import torch

from msccl.interp import input_chunks_of, run_algorithm
from msccl.language import MSCCLProgram, ThreadblockPolicy
from msccl.language.collectives import AllGather, AllReduce, AllToAll, ReduceScatter
from msccl.programs.allgather import allgather_direct, reduce_scatter_direct
from msccl.programs.allreduce import allreduce_one_shot, allreduce_ring, allreduce_two_shot
from msccl.programs.alltoall import alltoall_direct
from msccl.topologies import fully_connected
from msccl.xml import load_xml

pytestmark = pytest.mark.gpu

BODIES = {
    'ring': (lambda n: AllReduce(n, n, True), lambda n: allreduce_ring(n, min(n, 2)), True),
    'two_shot': (lambda n: AllReduce(n, n, True), allreduce_two_shot, True),
    'one_shot': (lambda n: AllReduce(n, 1, True), allreduce_one_shot, True),
    'allgather': (lambda n: AllGather(n, 1, False), allgather_direct, False),
    'reduce_scatter': (lambda n: ReduceScatter(n, 1, False), reduce_scatter_direct, False),
    'alltoall': (lambda n: AllToAll(n, 1, False), alltoall_direct, False),
}


def _algo(name, ranks, protocol):
    coll, body, manual = BODIES[name]
    policy = dict(threadblock_policy=ThreadblockPolicy.manual) if manual else {}
    prog = MSCCLProgram(name, fully_connected(ranks), coll(ranks), 1, protocol=protocol, **policy)
    with prog:
        body(ranks)
    return load_xml(prog.generate_xml())


def _check(algo, chunk, dtype, misalign=0, fifo_bytes=8 << 20, direct='auto', tile=None, monkeypatch=None, streams=1):
    from msccl.runtime import Communicator, Executor
    import msccl.runtime.plan as P
    if tile:
        monkeypatch.setattr(P, 'ONE_GPU_TILE_BYTES', tile)
    comm = Communicator.emulated(algo.ngpus, fifo_bytes=fifo_bytes)
    try:
        ex = Executor(comm)
        plan = ex.compile(algo)
        gen = torch.Generator().manual_seed(chunk)
        host = [torch.randn(input_chunks_of(algo, r) * chunk, generator=gen).to(dtype) for r in range(algo.ngpus)]
        want = run_algorithm(algo, host, chunk, dtype=dtype)

        def place(t, guard):
            holder = torch.full((t.numel() + misalign + 16,), 7.0, dtype=dtype, device='cuda')
            holder[misalign:misalign + t.numel()].copy_(t)
            guard.append((holder, t.numel()))
            return holder[misalign:misalign + t.numel()]

        for _ in range(2):                             # a second launch: counters and flags go on
            guard = []
            ins = {r: place(host[r], guard) for r in range(algo.ngpus)}
            outs = {} if algo.inplace else {r: place(torch.zeros(algo.gpus[r].o_chunks * chunk, dtype=dtype), guard) for r in range(algo.ngpus)}
            got = ex.run(plan, ins, outs, direct=direct)
            ex.check()
            for r in range(algo.ngpus):
                n = min(got[r].numel(), want[r].numel())
                assert torch.equal(got[r].cpu()[:n].view(torch.uint8), want[r][:n].view(torch.uint8)), f'rank {r} differs'
            for holder, n in guard:                    # nothing beside the buffers was written
                assert torch.all(holder[:misalign] == 7) and torch.all(holder[misalign + n:] == 7)
        geometry = next(iter(plan.geometry.values()))
        assert geometry[1] >= streams
        plan.close()
    finally:
        comm.close()


@pytest.mark.parametrize('name', ['ring', 'two_shot', 'alltoall', 'reduce_scatter'])
@pytest.mark.parametrize('chunk', [65536, 65536 + 8, 70000])
def test_several_slices_per_cta(name, chunk, monkeypatch):
    # tiles of 2 KB: two CTAs' worth of slices with several tiles each, the last one short
    _check(_algo(name, 4, 'Simple'), chunk, torch.bfloat16, tile=2048, monkeypatch=monkeypatch, streams=1 if name == 'alltoall' else 4)


@pytest.mark.parametrize('name', ['ring', 'two_shot', 'allgather', 'reduce_scatter', 'alltoall'])
@pytest.mark.parametrize('dtype,chunk,misalign', [(torch.float16, 1, 0), (torch.float16, 7, 1), (torch.bfloat16, 9, 5), (torch.float32, 3, 1),
                                                  (torch.float16, 3071, 0), (torch.bfloat16, 12345, 7), (torch.float32, 4097, 3),
                                                  (torch.float16, 50001, 2)])
@pytest.mark.parametrize('direct', [True, False])
def test_every_alignment(name, dtype, chunk, misalign, direct):
    _check(_algo(name, 3, 'Simple'), chunk, dtype, misalign, direct=direct)


@pytest.mark.parametrize('protocol', ['Simple', 'LL', 'LL128'])
@pytest.mark.parametrize('name,ranks', [('one_shot', 2), ('one_shot', 9), ('one_shot', 12), ('two_shot', 8)])
def test_folded_reduces(name, ranks, protocol):
    # 9 and 12 ranks: eight and eleven adds, a whole batch and more than one
    _check(_algo(name, ranks, protocol), 2056, torch.bfloat16)


def test_small_fifos_and_flag_protocols():
    for protocol in ('LL', 'LL128'):
        _check(_algo('ring', 4, protocol), 40008, torch.float16, fifo_bytes=1 << 20)


def test_bounds_failure_is_reported_as_such_by_every_slice(monkeypatch):
    """Four slices per CTA: the slice that finds its step outside the declared buffer says so before any other warp of the CTA can
    report that it gave up.  The tensor is larger than declared, so nothing outside owned memory is named."""
    from msccl.runtime import Communicator, Executor, ExecutorError
    import msccl.runtime.plan as P
    monkeypatch.setattr(P, 'ONE_GPU_TILE_BYTES', 2048)
    chunk, algo = 65536, _algo('ring', 4, 'Simple')
    comm = Communicator.emulated(4, fifo_bytes=8 << 20)
    try:
        ex = Executor(comm)
        plan = ex.compile(algo)
        for _ in range(3):
            comm.timeout_ns = int(0.5e9)                       # the other ranks wait this long for the rank that stopped
            ins = {r: torch.full((4 * chunk,), float(r + 1), device='cuda') for r in range(4)}
            ex.run(plan, ins, declared_elems={r: ((3 if r == 2 else 4) * chunk, 0, 0) for r in range(4)})
            with pytest.raises(ExecutorError):
                ex.check()
            status = comm.native.read_status(comm.sync_ptr(2))
            assert status[0] == 6 and status[1] == 2           # STATUS_BOUNDS, reported by rank 2
            comm.reset_after_failure()
            comm.timeout_ns = int(20e9)
            ins = {r: torch.full((4 * chunk,), float(r + 1), device='cuda') for r in range(4)}
            out = ex.run(plan, ins)
            ex.check()
            assert all(torch.all(out[r] == 10) for r in range(4))
        assert next(iter(plan.geometry.values()))[1] == 4
        plan.close()
    finally:
        comm.close()


@pytest.mark.parametrize('protocol', ['Simple', 'LL', 'LL128'])
def test_a_receive_that_nothing_feeds_is_reported_as_such(protocol, monkeypatch):
    """Under Simple the control warp waits for the tile, under LL and LL128 the data warps poll its packets: either way the
    (short) wait ends in the same status, and the device stays usable."""
    from msccl.runtime import Communicator, Executor, ExecutorError
    import msccl.runtime.executor as executor
    lonely = load_xml(f'<algo name="lonely" proto="{protocol}" nchannels="1" nchunksperloop="1" ngpus="2" coll="custom" inplace="0">'
                      '<gpu id="0" i_chunks="1" o_chunks="1" s_chunks="0"><tb id="0" send="-1" recv="1" chan="0">'
                      '<step s="0" type="r" srcbuf="i" srcoff="0" dstbuf="o" dstoff="0" cnt="1" depid="-1" deps="-1" hasdep="0"/>'
                      '</tb></gpu><gpu id="1" i_chunks="1" o_chunks="1" s_chunks="0"></gpu></algo>')
    comm = Communicator.emulated(2, fifo_bytes=1 << 20)
    try:
        comm.timeout_ns = int(0.2e9)
        ex = Executor(comm)
        checked = executor.compile_plan
        with monkeypatch.context() as patch:
            patch.setattr(executor, 'compile_plan', lambda algo, ranks, slot: checked(algo, ranks, slot, check=False))
            plan = ex.compile(lonely)
        ex.run(plan, {r: torch.ones(1024, device='cuda') for r in range(2)})
        with pytest.raises(ExecutorError) as err:
            ex.check()
        assert err.value.code == 2 and err.value.rank == 0 and err.value.aux0 == 1      # STATUS_TIMEOUT_DATA, waiting for rank 1
        comm.reset_after_failure()
        comm.timeout_ns = int(20e9)
        ins = {r: torch.full((2 * 1024,), float(r + 1), device='cuda') for r in range(2)}
        ex.run(ex.compile(_algo('ring', 2, protocol)), ins)
        ex.check()
        assert all(torch.all(ins[r] == 3) for r in range(2))
    finally:
        comm.close()


@pytest.mark.parametrize('protocol', ['LL', 'LL128', 'Simple'])
def test_a_rank_without_threadblocks_keeps_up_with_the_others(protocol):
    """Flags of LL and LL128 packets name the launch: a rank with nothing to do in one launch counts it all the same."""
    from msccl.runtime import Communicator, Executor
    step = '<step s="0" type="{}" srcbuf="i" srcoff="0" dstbuf="i" dstoff="0" cnt="1" depid="-1" deps="-1" hasdep="0"/>'
    gpu = '<gpu id="{}" i_chunks="1" o_chunks="0" s_chunks="0">{}</gpu>'
    head = '<algo name="pair" proto="LL" nchannels="1" nchunksperloop="1" ngpus="3" coll="custom" inplace="1">'
    pair = load_xml(head + gpu.format(0, '<tb id="0" send="1" recv="-1" chan="0">' + step.format('s') + '</tb>') +
                    gpu.format(1, '<tb id="0" send="-1" recv="0" chan="0">' + step.format('rrc') + '</tb>') + gpu.format(2, '') + '</algo>')
    comm = Communicator.emulated(3, fifo_bytes=1 << 20)
    try:
        comm.timeout_ns = int(2e9)
        ex = Executor(comm)
        plans = ex.compile(pair), ex.compile(_algo('ring', 3, protocol))
        for _ in range(3):
            ins = {r: torch.full((3 * 1024,), float(r + 1), device='cuda') for r in range(3)}
            ex.run(plans[0], ins)
            ex.check()
            assert [float(ins[r][5]) for r in range(3)] == [1, 3, 3]
            ex.run(plans[1], ins)
            ex.check()
            assert all(torch.all(ins[r] == 7) for r in range(3))
    finally:
        comm.close()
