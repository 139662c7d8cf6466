"""Host side of the one-GPU interpreter: folded reduce chains against the unfolded program, and its launch geometry."""
import time
from dataclasses import replace

import pytest
import torch

from msccl.interp import RaceError, input_chunks_of, run_algorithm
from msccl.language import MSCCLProgram, ThreadblockPolicy
from msccl.language.collectives import AllGather, AllReduce, AllToAll, ReduceScatter
from msccl.programs.allgather import allgather_direct, allgather_ring, reduce_scatter_direct
from msccl.programs.allreduce import allreduce_allpairs, allreduce_one_shot, allreduce_ring, allreduce_two_shot
from msccl.programs.alltoall import alltoall_direct
from msccl.runtime import plan as P
from msccl.topologies import fully_connected
from msccl.xml import load_xml
from msccl.xml.validator import validate

PROGRAMS = {'one_shot': (allreduce_one_shot, 1), 'two_shot': (allreduce_two_shot, None), 'ring': (lambda n: allreduce_ring(n, 2), None),
            'allpairs': (allreduce_allpairs, 'square')}


def _program(name, ranks, instances=1, **kw):
    body, chunks = PROGRAMS[name]
    chunks = ranks * ranks if chunks == 'square' else chunks or ranks
    prog = MSCCLProgram(name, fully_connected(ranks), AllReduce(ranks, chunks, True), instances,
                        threadblock_policy=ThreadblockPolicy.manual, **kw)
    with prog:
        body(ranks)
    return load_xml(prog.generate_xml())


@pytest.mark.parametrize('name,ranks,instances', [('one_shot', 2, 1), ('one_shot', 3, 2), ('one_shot', 8, 1), ('two_shot', 4, 1),
                                                  ('two_shot', 8, 2), ('one_shot', 12, 1), ('ring', 4, 2), ('allpairs', 4, 1)])
def test_folded_chains_round_like_the_program(name, ranks, instances):
    # 12 ranks: eleven adds, more than one multi-input add takes
    algo = _program(name, ranks, instances)
    before = [[(st.type, st.depid, st.deps) for tb in g.tbs for st in tb.steps] for g in algo.gpus]
    folded = P.fold_reduce_chains(algo)
    assert [[(st.type, st.depid, st.deps) for tb in g.tbs for st in tb.steps] for g in algo.gpus] == before
    assert validate(folded) == []
    reduces = lambda a: sum(1 / st.parts for g in a.gpus for tb in g.tbs for st in tb.steps if st.type == 're')   # noqa: E731
    assert abs(reduces(folded) - reduces(algo)) < 1e-6
    if name in ('one_shot', 'two_shot') and ranks > 2:
        waits = lambda a: sum(st.type == 're' and a.gpus[0].tbs[st.depid].steps[st.deps].type == 're'    # noqa: E731
                              for tb in a.gpus[0].tbs for st in tb.steps if st.depid >= 0)
        assert waits(folded) <= (ranks - 1) // P.K_MAX_BATCH < waits(algo)
    gen = torch.Generator().manual_seed(3)
    host = [torch.randn(input_chunks_of(algo, r) * 24, generator=gen).bfloat16() for r in range(ranks)]
    want = run_algorithm(algo, host, 24, dtype=torch.bfloat16)
    got = run_algorithm(folded, host, 24, dtype=torch.bfloat16)
    assert all(torch.equal(w.view(torch.int16), g.view(torch.int16)) for w, g in zip(want, got))


def _rounds(ranks, rounds):
    """The one-shot all-reduce ``rounds`` times: the sends of a round wait for the sum of the one before."""
    algo = _copy(_program('one_shot', ranks))
    for gpu in algo.gpus:
        once = [tb.steps for tb in gpu.tbs]
        waited = {(st.depid, st.deps) for steps in once for st in steps}
        end_tb, end = next((t, i) for t, steps in enumerate(once) for i, st in enumerate(steps)
                           if st.type == 're' and (t, i) not in waited)
        once[end_tb][end].hasdep = True
        for t, tb in enumerate(gpu.tbs):
            tb.steps = []
            for k in range(rounds):
                for st in once[t]:
                    st = replace(st, s=len(tb.steps), deps=st.deps + k * len(once[st.depid]) if st.depid >= 0 else -1)
                    if k and st.type == 's' and t != end_tb:
                        st.depid, st.deps = end_tb, (k - 1) * len(once[end_tb]) + end
                    tb.steps.append(st)
    return algo


def test_long_programs_fold_in_time():
    # 2600 steps per GPU, 100 chains: a search that starts again behind every chain takes minutes, one pass a second
    algo = _rounds(8, 100)
    assert validate(algo) == []
    start = time.perf_counter()
    folded = P.fold_reduce_chains(algo)
    assert time.perf_counter() - start < 20
    assert validate(folded) == [] and sum(st.parts == 7 for tb in folded.gpus[0].tbs for st in tb.steps) == 7 * 7 * 100


def test_programs_that_would_get_too_long_stay_as_they_are(monkeypatch):
    algo = _rounds(4, 10)
    assert P.fold_reduce_chains(algo) is not algo
    monkeypatch.setattr(P, 'K_MAX_STEPS_PER_TB', max(len(tb.steps) for tb in algo.gpus[0].tbs))
    assert P.fold_reduce_chains(algo) is algo
    P.compile_plan(P.fold_reduce_chains(algo), range(4), 64 << 10)


def test_dependencies_on_missing_steps_are_left_to_the_validator():
    algo = _copy(_program('one_shot', 3))
    next(st for tb in algo.gpus[0].tbs for st in tb.steps if st.type == 're' and st.depid >= 0).deps = 99
    algo.gpus[1].tbs[0].steps[-1].depid = 7
    with pytest.raises(P.PlanError):
        P.compile_plan(P.split_copies(P.fold_reduce_chains(algo), 64), range(3), 64 << 10)


@pytest.mark.parametrize('coll,body,moves', [
    (lambda n: AllToAll(n, 1, False), alltoall_direct, True), (lambda n: AllGather(n, 1, False), allgather_direct, True),
    (lambda n: AllGather(n, 1, False), lambda n: allgather_ring(n, 2), None), (lambda n: ReduceScatter(n, 1, False), reduce_scatter_direct, None)])
@pytest.mark.parametrize('ranks,instances', [(2, 1), (4, 1), (8, 2)])
def test_copies_that_move_to_threadblocks_of_their_own(coll, body, moves, ranks, instances):
    prog = MSCCLProgram('p', fully_connected(ranks), coll(ranks), instances)
    with prog:
        body(ranks)
    algo = load_xml(prog.generate_xml())
    split = P.split_copies(algo, 256)
    assert validate(split) == [] and split.num_steps() == algo.num_steps()
    assert P.split_copies(algo, algo.num_threadblocks()) is algo
    if moves and ranks > 2:
        assert split.num_threadblocks() == algo.num_threadblocks() + ranks * instances
        assert max(sum(st.type in ('s', 'cpy') for st in tb.steps) for g in split.gpus for tb in g.tbs) == 1
    gen = torch.Generator().manual_seed(4)
    host = [torch.randn(input_chunks_of(algo, r) * 8, generator=gen) for r in range(ranks)]
    want, got = run_algorithm(algo, host, 8), run_algorithm(split, host, 8)
    assert all(torch.equal(w, g) for w, g in zip(want, got))


def _copy(algo):
    return replace(algo, gpus=[replace(g, tbs=[replace(tb, steps=[replace(st) for st in tb.steps]) for tb in g.tbs]) for g in algo.gpus])


def _race_check(algo, chunk=24):
    host = [torch.ones(input_chunks_of(algo, r) * chunk) for r in range(algo.ngpus)]
    run_algorithm(algo, host, chunk, race_check=True)


@pytest.mark.parametrize('name,ranks,instances', [('one_shot', 3, 2), ('one_shot', 8, 1), ('two_shot', 4, 1), ('two_shot', 8, 2),
                                                  ('one_shot', 9, 1), ('one_shot', 12, 1), ('ring', 4, 2), ('allpairs', 4, 1)])
def test_rewritten_programs_are_free_of_races(name, ranks, instances):
    folded = P.fold_reduce_chains(_program(name, ranks, instances))
    _race_check(folded)
    _race_check(P.split_copies(folded, 1 << 20))


@pytest.mark.parametrize('name,ranks', [('two_shot', 4), ('two_shot', 8), ('one_shot', 3), ('one_shot', 12)])
def test_a_wait_that_is_dropped_from_a_folded_program_is_a_race(name, ranks):
    """Every wait for one part of an add (and for what fills its sources) is needed, whichever part it is.  With 12 ranks a chain of
    eight adds follows one of three: a part of the second waits for all three and overlaps with one or two of them."""
    folded = P.fold_reduce_chains(_program(name, ranks))
    dropped = races = parts_after_the_first = 0
    for t, tb in enumerate(folded.gpus[0].tbs):
        for i, st in enumerate(tb.steps):
            if st.depid < 0:
                continue
            awaited = folded.gpus[0].tbs[st.depid].steps[st.deps]
            less = _copy(folded)
            less.gpus[0].tbs[t].steps[i].depid = less.gpus[0].tbs[t].steps[i].deps = -1
            dropped += 1
            try:
                _race_check(less)
            except RaceError:
                races += 1
                parts_after_the_first += awaited.type == 're' and awaited.part > 0
    # 8 x 3 pairs of parts, of which 8 + 3 - gcd(8, 3) overlap
    assert races == dropped - ((8 * 3 - 10) if ranks == 12 else 0) > 0
    assert parts_after_the_first > 0 or (name, ranks) == ('one_shot', 3)


@pytest.mark.parametrize('chunk,esize', [(1, 2), (7, 4), (8, 2), (333333, 2), (4096, 4), (1 << 22, 2), (5 * (1 << 20) + 8, 4)])
@pytest.mark.parametrize('proto', [0, 1, 2])
@pytest.mark.parametrize('max_ctas', [32, 148, 592])
def test_one_gpu_geometry_covers_the_chunk(chunk, esize, proto, max_ctas):
    plan = P.compile_plan(_program('two_shot', 4, 2, protocol='LL'), range(4), 256 << 10)
    width = P.access_width(chunk, esize)
    proto = 1 if proto == 2 and width != 16 else proto
    ctas, streams, slice_elems, tile, slot = P.one_gpu_geometry(plan, chunk, esize, 256 << 10, width, proto, max_ctas)
    slices = ctas * streams
    assert ctas * plan.total_tbs() <= max_ctas and (streams == 1 or proto == 0)
    assert (ctas - 1) * streams * slice_elems < chunk <= slices * slice_elems
    assert slice_elems * esize % width == 0 and 0 < tile <= slice_elems and tile * esize % width == 0
    assert slot % 128 == 0 and slot * slices <= 256 << 10
    accesses = tile * esize // width
    fifo = {0: accesses * width, 1: accesses * (32 if width == 16 else 8), 2: -(-2 * accesses // 15) * 128}[proto]
    assert fifo * plan.max_cnt <= slot


def _wide(count):
    """Two ranks, one message of ``count`` chunks, stored by the receiver (``rrc``: never straight into its slot)."""
    tb = '<tb id="0" send="{}" recv="{}" chan="0"><step s="0" type="{}" srcbuf="i" srcoff="0" dstbuf="i" dstoff="0" cnt="{}" ' \
         'depid="-1" deps="-1" hasdep="0"/></tb>'
    gpu = '<gpu id="{}" i_chunks="{}" o_chunks="0" s_chunks="0">{}</gpu>'
    return load_xml('<algo name="wide" proto="Simple" nchannels="1" nchunksperloop="1" ngpus="2" coll="custom" inplace="1">' +
                    gpu.format(0, count, tb.format(1, -1, 's', count)) + gpu.format(1, count, tb.format(-1, 0, 'rrc', count)) + '</algo>')


@pytest.mark.parametrize('count,chunk,slot_bytes,max_ctas', [(1, 1 << 33, 4 << 20, 592), (1025, 1 << 28, 4 << 20, 2), (1025, 1 << 33, 256 << 20, 592),
                                                             (2000, 9 * (1 << 20) * 196, 256 << 20, 16), (4097, 1 << 28, 256 << 20, 16)])
def test_tiles_of_wide_steps_keep_within_the_iteration_limit(count, chunk, slot_bytes, max_ctas):
    """128 KB over more than a thousand chunks leaves tiles of less than a line: they grow until the iterations fit."""
    plan = P.compile_plan(_wide(count), range(2), slot_bytes)
    assert P.tile_geometry(plan, chunk, 2, slot_bytes)[1] < P.K_MAX_ITERATIONS
    _, _, slice_elems, tile, slot = P.one_gpu_geometry(plan, chunk, 2, slot_bytes, 16, 0, max_ctas)
    assert -(-slice_elems // tile) < P.K_MAX_ITERATIONS and tile % 8 == 0 and tile * 2 * count <= slot


@pytest.mark.parametrize('coll,body', [(AllToAll, alltoall_direct), (AllGather, allgather_direct)])
@pytest.mark.parametrize('chunk,esize,direct', [(1, 4, True), (333333, 2, True), (1 << 21, 2, True), (1 << 21, 2, False), (1 << 24, 4, True)])
def test_geometry_of_single_hop_programs(coll, body, chunk, esize, direct):
    prog = MSCCLProgram('p', fully_connected(8), coll(8, 1, False), 1)
    with prog:
        body(8)
    slot_bytes = 4 << 20
    plan = P.compile_plan(P.split_copies(load_xml(prog.generate_xml()), 296), range(8), slot_bytes)
    assert plan.single_hop
    width = P.access_width(chunk, esize)
    ctas, streams, slice_elems, tile, slot = P.one_gpu_geometry(plan, chunk, esize, slot_bytes, width, 0, 592, direct)
    slices = ctas * streams
    assert ctas * plan.total_tbs() <= 592 and (ctas - 1) * streams * slice_elems < chunk <= slices * slice_elems
    assert slot * slices <= slot_bytes and 0 < tile <= slice_elems and tile * esize % width == 0 and tile * esize * plan.max_cnt <= slot
    if direct:
        assert streams == 1 and tile == min(slice_elems, slot // (plan.max_cnt * width) * (width // esize))


def test_empty_buffers_are_refused():
    plan = P.compile_plan(_program('two_shot', 4), range(4), 64 << 10)
    with pytest.raises(P.PlanError):
        P.one_gpu_geometry(plan, 0, 2, 64 << 10, 2, 0, 592)


def test_every_rank_has_a_threadblock():
    algo = _wide(1)
    idle = replace(algo, ngpus=3, gpus=algo.gpus + [replace(algo.gpus[0], id=2, tbs=[])])
    assert P.occupy_idle_ranks(algo) is algo
    filled = P.occupy_idle_ranks(idle)
    assert validate(filled) == [] and not idle.gpus[2].tbs and [len(g.tbs) for g in filled.gpus] == [1, 1, 1]
    assert P.compile_plan(filled, range(3), 64 << 10).num_tbs == {0: 1, 1: 1, 2: 1}
