"""The interpreter kernel of one-process-per-GPU jobs (csrc/exec_kernel.cu) on a single GPU.

``Executor.run`` on an emulated communicator takes the one-GPU interpreter, so these tests launch the other kernel
themselves: the compiled program as it stands (no folded chains, no copies apart), the threadblocks of all ranks in one cooperative
launch, every rank's buffers in an uploaded rank table.  Results are compared bit for bit with the CPU interpreter, with both ways
in which the warps of a CTA learn that a step may start (``MSCCL_EXEC_WAIT``)."""
import functools

import pytest
import torch

from msccl.interp import input_chunks_of, run_algorithm
from msccl.language import Buffer, ThreadblockPolicy, chunk
from msccl.language.collectives import AllGather, AllReduce
from msccl.programs.allgather import allgather_direct
from msccl.programs.allreduce import allreduce_allpairs, allreduce_ring
from msccl.xml import load_xml
from test_gpu_executor import _cases, _program
from test_plan_compile import refilled_source

pytestmark = pytest.mark.gpu
DTYPES = {torch.float32: 0, torch.bfloat16: 1, torch.float16: 2}
WAITS = {'poll': 0, 'barrier': 1}


@functools.lru_cache(maxsize=None)
def _algo(name):
    """The programs of test_gpu_executor, each built once (the synthesised ones run the solver)."""
    return _cases()[name]()


class Launcher:
    """A program on ``exec_kernel``: plan arrays and scratch on the device, one launch per call."""

    def __init__(self, comm, algo, check=True):
        from msccl.runtime.executor import MAX_SLOT_BYTES
        from msccl.runtime.plan import K_FIFO_SLOTS, compile_plan, fifo_index_tables, occupy_idle_ranks
        self.comm, self.algo = comm, occupy_idle_ranks(algo)
        algo = self.algo
        conns = max(max(len(t) for t in fifo_index_tables(algo).values()), 1)
        self.slot = min(MAX_SLOT_BYTES, comm.fifo_bytes // (conns * K_FIFO_SLOTS)) // 1024 * 1024
        self.host = compile_plan(algo, comm.local_ranks, self.slot, check=check)
        self.tbs, self.steps = comm.native.upload(self.host.tb_bytes), comm.native.upload(self.host.step_bytes)
        self.keep = []

    def __call__(self, inputs, outputs=None, direct=True, wait='barrier', trace=False, declared=None):
        from msccl.runtime.plan import access_width, tile_geometry
        nat, comm, algo = self.comm.native, self.comm, self.algo
        gathered = algo.inplace and algo.coll == 'allgather'
        first = inputs[0]
        chunk = first.numel() // (algo.gpus[0].o_chunks if gathered else algo.gpus[0].i_chunks)
        buffers, sizes, results = {}, {}, {}
        for r in range(algo.ngpus):
            used = self.host.extents[r]
            i, o = inputs[r], (outputs or {}).get(r)
            if gathered:
                i, o = None, inputs[r]
            elif o is None and used['o'] > 0:
                o = torch.empty(algo.gpus[r].o_chunks * chunk, dtype=first.dtype, device='cuda')
            s = torch.empty(used['s'] * chunk, dtype=first.dtype, device='cuda') if used['s'] else None
            results[r] = inputs[r] if o is None else o
            self.keep += [i, o, s]
            buffers[r] = tuple(0 if t is None else t.data_ptr() for t in (i, o, s))
            sizes[r] = declared[r] if declared else tuple(0 if t is None else t.numel() for t in (i, o, s))
        width = access_width(chunk, first.element_size(), [p for b in buffers.values() for p in b])
        proto = 1 if self.host.proto == 2 and width != 16 else self.host.proto
        tile, iterations = tile_geometry(self.host, chunk, first.element_size(), self.slot, width, proto)
        grid, dtype = self.host.total_tbs(), DTYPES[first.dtype]
        assert grid <= nat.max_coresident_ctas(dtype, proto, width)
        table = nat.upload(comm.rankctx_bytes(buffers, sizes))
        steps = max(len(tb.steps) for g in algo.gpus for tb in g.tbs)
        record = torch.zeros(grid, steps, 6, dtype=torch.int64, device='cuda') if trace else None
        nat.launch(self.tbs, self.steps, table, [chunk, tile, self.slot, iterations, comm.world, 0, grid, dtype, proto, width],
                   comm.timeout_ns, torch.cuda.current_stream().cuda_stream, True, direct_mask=7 if direct else 0,
                   trace=record.data_ptr() if trace else 0, trace_steps=steps if trace else 0, wait_mode=WAITS[wait])
        torch.cuda.synchronize()
        nat.device_free(table)
        return (results, record) if trace else results

    def close(self):
        for p in (self.tbs, self.steps):
            self.comm.native.device_free(p)


@pytest.fixture
def emulated():
    from msccl.runtime import Communicator
    made = []

    def make(ranks, fifo_bytes):
        made.append(Communicator.emulated(ranks, fifo_bytes=fifo_bytes))
        return made[-1]
    yield make
    for comm in made:
        comm.close()


def _compare(emulated, algo, chunk, dtype, fifo_bytes=8 << 20, direct=True, misalign=0, wait='barrier'):
    comm = emulated(algo.ngpus, fifo_bytes)
    run = Launcher(comm, algo)
    gen = torch.Generator().manual_seed(42)
    host = [torch.randn(input_chunks_of(algo, r) * chunk, generator=gen).to(dtype) for r in range(algo.ngpus)]
    want = run_algorithm(algo, host, chunk, dtype=dtype)

    def place(t):
        holder = torch.zeros(t.numel() + misalign, dtype=dtype, device='cuda')
        holder[misalign:].copy_(t)
        return holder[misalign:]

    for _ in range(2):                                         # a second launch: counters and flags go on
        ins, outs = {}, {}
        for r in range(algo.ngpus):
            if algo.inplace and algo.coll == 'allgather':
                full = torch.zeros(algo.gpus[r].o_chunks * chunk, dtype=dtype)
                full[r * host[r].numel():(r + 1) * host[r].numel()] = host[r]
                ins[r] = place(full)
            else:
                ins[r] = place(host[r])
                if algo.gpus[r].o_chunks > 0 and not algo.inplace:
                    outs[r] = place(torch.zeros(algo.gpus[r].o_chunks * chunk, dtype=dtype))
        got = run(ins, outs, direct=direct, wait=wait)
        comm.check()
        for r in range(algo.ngpus):
            n = min(got[r].numel(), want[r].numel())
            assert torch.equal(got[r].cpu()[:n].view(torch.uint8), want[r][:n].view(torch.uint8)), f'rank {r} differs'
    run.close()


@pytest.mark.parametrize('wait', list(WAITS))
@pytest.mark.parametrize('name', list(_cases()))
def test_programs_bit_exact(emulated, name, wait):
    _compare(emulated, _algo(name), 256, torch.float32, wait=wait)


@pytest.mark.parametrize('name', ['ring8_simple', 'ring8_ll_x2', 'two_shot8_x2', 'allpairs4_ll_nop', 'alltoall8'])
@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float16])
def test_low_precision_bit_exact(emulated, name, dtype):
    _compare(emulated, _algo(name), 1024, dtype)


@pytest.mark.parametrize('wait', list(WAITS))
@pytest.mark.parametrize('name', ['ring8_simple', 'ring8_ll_x2', 'two_shot8_x2', 'synth_allgather_nvswitch'])
def test_many_iterations_through_small_fifos(emulated, name, wait):
    _compare(emulated, _algo(name), 40000, torch.float32, 1 << 20, wait=wait)


@pytest.mark.parametrize('name', ['ring8_simple', 'two_shot8_x2', 'alltoall8', 'allgather8_ring', 'reduce_scatter4',
                                  'synth_allgather_nvswitch'])
def test_fifo_only_path(emulated, name):
    _compare(emulated, _algo(name), 4096, torch.float32, direct=False)


@pytest.mark.parametrize('wait', list(WAITS))
@pytest.mark.parametrize('dtype,chunk', [(torch.float32, 256), (torch.bfloat16, 40000), (torch.float16, 1000)])
@pytest.mark.parametrize('name', ['ring4_ll128', 'ring8', 'allgather8', 'allpairs4'])
def test_ll128_lines(emulated, name, dtype, chunk, wait):
    manual = dict(threadblock_policy=ThreadblockPolicy.manual, protocol='LL128')
    algo = {'ring4_ll128': lambda: _algo('ring4_ll128'),
            'ring8': lambda: _program('ring', AllReduce(8, 8, True), lambda: allreduce_ring(8, 4), 2, **manual),
            'allgather8': lambda: _program('ag', AllGather(8, 1, False), lambda: allgather_direct(8), 1, protocol='LL128'),
            'allpairs4': lambda: _program('allpairs', AllReduce(4, 16, True), lambda: allreduce_allpairs(4), 1, **manual)}[name]()
    _compare(emulated, algo, chunk, dtype, 1 << 20, wait=wait)


@pytest.mark.parametrize('name', ['ring8_simple', 'ring8_ll_x2', 'ring4_ll128', 'two_shot8_x2', 'alltoall8',
                                  'synth_allgather_nvswitch', 'allpairs4_ll_nop'])
@pytest.mark.parametrize('dtype,chunk,misalign', [(torch.float16, 500, 0), (torch.bfloat16, 1001, 0), (torch.float32, 333, 0),
                                                  (torch.float32, 256, 1), (torch.bfloat16, 4099, 3)])
def test_chunks_that_are_not_multiples_of_16_bytes(emulated, name, dtype, chunk, misalign):
    _compare(emulated, _algo(name), chunk, dtype, 2 << 20, misalign=misalign)


@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
@pytest.mark.parametrize('nop', [False, True])
def test_batched_reduces(emulated, dtype, nop):
    algo = _program('allpairs', AllReduce(8, 64, True), lambda: allreduce_allpairs(8), 1,
                    threadblock_policy=ThreadblockPolicy.manual, dependence_nop=nop)
    _compare(emulated, algo, 2048, dtype)


def test_step_outside_the_declared_buffer(emulated):
    """As in test_gpu_executor: the declared size is smaller than the tensor, so nothing outside owned memory is named."""
    from msccl.runtime import ExecutorError
    comm = emulated(4, 1 << 20)
    comm.timeout_ns = int(1e9)                                 # the other ranks wait this long for the rank that stopped
    run = Launcher(comm, _program('ag', AllGather(4, 1, False), lambda: allgather_direct(4)))
    ins = {r: torch.full((256,), float(r + 1), device='cuda') for r in range(4)}
    outs = {r: torch.zeros(4 * 256, device='cuda') for r in range(4)}
    run(ins, outs, declared={r: (256, 4 * 256 if r != 2 else 3 * 256, 0) for r in range(4)})
    with pytest.raises(ExecutorError):
        comm.check()
    status = comm.native.read_status(comm.sync_ptr(2))
    assert status[0] == 6 and status[1] == 2                   # STATUS_BOUNDS, reported by rank 2
    assert torch.all(outs[2][3 * 256:] == 0)
    comm.reset_after_failure()
    comm.timeout_ns = int(20e9)
    out = run(ins, outs)
    comm.check()
    assert torch.equal(out[2].view(4, 256)[:, 0].cpu(), torch.tensor([1.0, 2.0, 3.0, 4.0]))
    run.close()


@pytest.mark.parametrize('wait', list(WAITS))
def test_step_trace(emulated, wait):
    algo = _algo('ring8_simple')
    comm = emulated(8, 4 << 20)
    run = Launcher(comm, algo)
    out, record = run({r: torch.ones(8 * 65536, device='cuda') for r in range(8)}, wait=wait, trace=True)
    comm.check()
    record = record.cpu()
    cta = 0
    for g in algo.gpus:
        for tb in g.tbs:
            start, end, waited, moved, signalled, _ = record[cta, :len(tb.steps)].unbind(1)
            assert torch.all(start > 0) and torch.all(end >= start) and int((end - start).max()) < 5e9
            assert torch.all(waited >= 0) and torch.all(moved >= 0) and torch.all(signalled >= 0)
            assert torch.all(record[cta, len(tb.steps):] == 0)
            cta += 1
    assert torch.all(out[0] == 8.0)
    run.close()


@pytest.mark.parametrize('wait', list(WAITS))
def test_wait_runs_out_and_context_survives(emulated, wait):
    """A receive that nothing feeds gives up after the (short) limit and reports where it waited; the device stays usable."""
    from msccl.runtime import ExecutorError
    lonely = load_xml(
        '<algo name="lonely" proto="Simple" nchannels="1" nchunksperloop="1" ngpus="2" coll="custom" inplace="0">'
        '<gpu id="0" i_chunks="1" o_chunks="1" s_chunks="0"><tb id="0" send="-1" recv="1" chan="0">'
        '<step s="0" type="r" srcbuf="i" srcoff="0" dstbuf="o" dstoff="0" cnt="1" depid="-1" deps="-1" hasdep="0"/>'
        '</tb></gpu><gpu id="1" i_chunks="1" o_chunks="1" s_chunks="0"></gpu></algo>')
    comm = emulated(2, 1 << 20)
    comm.timeout_ns = int(0.2e9)
    ins = {r: torch.ones(64, device='cuda') for r in range(2)}
    run = Launcher(comm, lonely, check=False)
    run(ins, wait=wait)
    run.close()
    with pytest.raises(ExecutorError) as err:
        comm.check()
    assert err.value.code == 2 and err.value.rank == 0 and err.value.aux0 == 1
    comm.reset_after_failure()
    comm.timeout_ns = int(20e9)
    good = Launcher(comm, _program('ag', AllGather(2, 1, False), lambda: allgather_direct(2)))
    out = good({0: torch.full((64,), 1.0, device='cuda'), 1: torch.full((64,), 2.0, device='cuda')}, wait=wait)
    comm.check()
    assert torch.all(out[0] == out[1]) and torch.all(out[0][:64] == 1) and torch.all(out[0][64:] == 2)
    good.close()


def test_both_interpreters_share_a_communicator(emulated):
    """Launches of the two kernels and with and without direct stores alternate: they share the launch epoch and the FIFO area."""
    from msccl.runtime import Executor
    comm = emulated(8, 4 << 20)
    ex = Executor(comm)
    algos = [_algo(name) for name in ('ring8_simple', 'ring8_ll_x2', 'two_shot8_x2')]
    plans = [(ex.compile(a), Launcher(comm, a)) for a in algos]
    for round_ in range(12):
        plan, run = plans[round_ % 3]
        ins = {r: torch.full((8 * 2048,), float(r + round_), device='cuda') for r in range(8)}
        if round_ // 3 % 2:
            ex.run(plan, ins, direct=round_ % 2 == 0)
        else:
            run(ins, direct=round_ % 2 == 0)
        ex.check()
        assert all(torch.all(ins[r] == float(28 + 8 * round_)) for r in range(8))
    for plan, run in plans:
        plan.close()
        run.close()


@pytest.mark.parametrize('protocol', ['Simple', 'LL', 'LL128'])
def test_adds_whose_source_is_refilled_between_them(emulated, protocol):
    """Two adds into one slot, the second of which waits for what comes after the first: not one multi-input add, in either kernel."""
    from msccl.runtime import Executor
    algo = _program('refilled', AllReduce(2, 1, True), lambda: refilled_source(5), threadblock_policy=ThreadblockPolicy.manual,
                    protocol=protocol)
    comm = emulated(2, 1 << 20)
    comm.timeout_ns = int(2e9)
    ex, run = Executor(comm), Launcher(comm, algo)
    plan = ex.compile(algo)
    for launch in (lambda ins: ex.run(plan, ins), run):
        ins = {r: torch.full((5000,), float(r + 1), device='cuda') for r in range(2)}
        launch(ins)
        ex.check()
        assert torch.all(ins[0] == 1) and torch.all(ins[1] == 7)
    plan.close()
    run.close()


@pytest.mark.parametrize('protocol', ['LL', 'LL128'])
def test_a_rank_without_threadblocks_keeps_up(emulated, protocol):
    """A program that leaves rank 2 idle, then one whose packet flags name the launch: every rank must have counted both."""
    def pair():
        chunk(1, Buffer.input, 0).reduce(chunk(0, Buffer.input, 0))
    comm = emulated(3, 1 << 20)
    comm.timeout_ns = int(2e9)
    idle = _program('pair', AllReduce(3, 1, True), pair, protocol=protocol)
    assert not idle.gpus[2].tbs
    first = Launcher(comm, idle)
    ring = Launcher(comm, _program('ring', AllReduce(3, 3, True), lambda: allreduce_ring(3, 1), 1,
                                   threadblock_policy=ThreadblockPolicy.manual, protocol=protocol))
    for _ in range(3):
        ins = {r: torch.full((3 * 512,), float(r + 1), device='cuda') for r in range(3)}
        first(ins)
        comm.check()
        assert [float(ins[r][5]) for r in range(3)] == [1, 3, 3]
        ring(ins)
        comm.check()
        assert all(torch.all(ins[r] == 7) for r in range(3))
    first.close()
    ring.close()
