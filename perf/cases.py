"""The work this framework is used for on one GPU, as timed cases.

Two halves of the framework, each through its public entry points:

* ``program`` - a collective stated as an MSCCLang (or solver-synthesised) program, compiled to MSCCL-IR and executed
  by ``Executor.run`` with every rank of the program on this GPU (``Communicator.emulated``).  Messages of 1 KB to
  256 MB per rank, 2 to 8 ranks, sums in fp32 / bf16 / fp16, the three protocols in the size ranges in which the
  B200 plan table registers them, chunk sizes that are and are not multiples of 16 bytes.
* ``gemm`` / ``gemm_mxfp8`` / ``mlp`` / ``moe`` - the tensor-core operators and the layers built from them:
  the Llama-3-8B MLP (hidden 4096, FFN 14336 or one rank's shard of it) in bf16 and block-scaled fp8, from a decode
  batch to 8192 tokens, and the mixture-of-experts layer with 8 experts per GPU and top-2 routing.

``draw`` picks further cases from the same ranges.
"""
import functools
import math
import os
import weakref

import torch
import torch.distributed as dist

from msccl import collectives as synthesis_collectives
from msccl.language import MSCCLProgram, ThreadblockPolicy
from msccl.language.collectives import AllGather, AllReduce, AllToAll, ReduceScatter
from msccl.ncclize import ncclize
from msccl.ops.gemm import gemm_bf16, gemm_mxfp8, interleave_gate_up, quantize_mxfp8_packed
from msccl.parallel import ExpertParallelMoE, TensorParallelMLP
from msccl.programs.allgather import allgather_direct, reduce_scatter_direct
from msccl.programs.allreduce import allreduce_one_shot, allreduce_ring, allreduce_two_shot
from msccl.programs.alltoall import alltoall_direct
from msccl.runtime import Communicator, Executor
from msccl.strategies import solve_least_steps
from msccl.topologies import fully_connected
from msccl.xml import load_xml

DTYPES = {'f32': torch.float32, 'bf16': torch.bfloat16, 'f16': torch.float16}
KB, MB = 1 << 10, 1 << 20
HIDDEN, FFN = 4096, 14336
MAX_PROGRAM_BYTES = 8 * 256 * MB * 2          # what the largest listed program reads and writes
# The co-residency limit: threadblocks of a program wait on one another and one SM runs one of them.
MAX_THREADBLOCKS = 128

# name -> (collective, chunks per rank of the program's input as a function of the ranks, in place)
PROGRAMS = {
    'one_shot': ('allreduce', lambda n: 1), 'two_shot': ('allreduce', lambda n: n), 'ring': ('allreduce', lambda n: n),
    'allgather': ('allgather', lambda n: 1), 'reduce_scatter': ('reduce_scatter', lambda n: n),
    'alltoall': ('alltoall', lambda n: n), 'synthesised': ('allgather', lambda n: 1),
}


def listed():
    program = dict(kind='program', ranks=8, instances=1)
    return [
        # a scalar or a norm summed over the ranks: the smallest message, all latency (the plan registered below 64 KB)
        dict(program, name='allreduce_1k', program='one_shot', protocol='LL', dtype='bf16', elems=512),
        # a small gradient bucket: the two-shot program in its LL128 range (256 KB - 1 MB)
        dict(program, name='allreduce_1m', program='two_shot', protocol='LL128', dtype='bf16', elems=MB // 2, instances=2),
        # the benchmark's one-GPU workload: ring all-reduce of 256 MB per rank, 4 channels x 4 instances
        dict(program, name='allreduce_256m', program='ring', protocol='Simple', dtype='bf16', elems=128 * MB, instances=4),
        # the solver's all-gather for the NVSwitch topology, fp16 buffers, in the middle of its 64 KB - 256 MB range
        dict(program, name='allgather_synth_8m', program='synthesised', protocol='Simple', dtype='f16', elems=4 * MB),
        # a shard whose element count is odd: no 16-byte access fits its chunks
        dict(program, name='allgather_odd', program='allgather', protocol='Simple', dtype='f16', elems=333333),
        # token exchange of an expert-parallel layer: 4096 tokens of 4096 bf16 values per rank
        dict(program, name='alltoall_32m', program='alltoall', protocol='Simple', dtype='bf16', elems=16 * MB),
        # one projection of a ragged prefill batch with the SwiGLU epilogue
        dict(name='gemm_ragged', kind='gemm', m=1000, n=7168, k=HIDDEN, swiglu=True),
        # the same kind of projection on block-scaled fp8, activations quantised on the way
        dict(name='gemm_mxfp8', kind='gemm_mxfp8', m=4096, n=HIDDEN, k=FFN),
        # the Llama-3-8B MLP of the benchmark: 8192 tokens, bf16 and block-scaled fp8
        dict(name='mlp_bf16', kind='mlp', tokens=8192, ffn=FFN, precision='bf16'),
        dict(name='mlp_mxfp8', kind='mlp', tokens=8192, ffn=FFN, precision='mxfp8'),
        # a decode batch on one of eight tensor-parallel shards
        dict(name='mlp_decode', kind='mlp', tokens=256, ffn=FFN // 8, precision='bf16'),
        # the MoE layer of the benchmark: 4096 tokens, 8 experts, top-2
        dict(name='moe', kind='moe', tokens=4096, ffn=FFN, experts=8, topk=2),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _draw_program(rng):
    ranks = rng.choice((2, 4, 8, 8))
    dtype = rng.choice(('f32', 'bf16', 'f16'))
    esize = 4 if dtype == 'f32' else 2
    name = rng.choice(('allreduce', 'allreduce', 'allgather', 'reduce_scatter', 'alltoall', 'synthesised'))
    odd = rng.random() < 0.25
    nbytes = _log(rng, KB, 4 * MB if odd else 256 * MB)
    if name in ('allgather', 'synthesised'):           # every rank writes the blocks of all ranks
        nbytes = min(nbytes, MAX_PROGRAM_BYTES // (ranks * (ranks + 1)))
    if name == 'allreduce':
        if nbytes < 64 * KB:
            name, protocol = 'one_shot', 'LL'
        elif nbytes < MB:
            name, protocol = 'two_shot', 'LL128'
        else:
            name, protocol = rng.choice(('ring', 'two_shot')), 'Simple'
    elif name == 'synthesised':
        protocol = 'Simple'
    else:
        protocol = 'LL' if nbytes < 512 * KB else ('LL128' if nbytes < 2 * MB else 'Simple')
    per_rank = {'ring': min(ranks, 4), 'one_shot': ranks, 'two_shot': ranks}.get(name, 2 * ranks)
    most = max(1, MAX_THREADBLOCKS // (per_rank * ranks))
    instances = 1 if name == 'synthesised' or nbytes < 64 * KB else min(most, rng.choice((1, 2, 4, 8)))
    pieces = PROGRAMS[name][1](ranks) * instances
    chunk = max(1, nbytes // (esize * pieces))
    chunk = chunk | 1 if odd else max(16 // esize, chunk * esize // 16 * 16 // esize)
    return dict(kind='program', ranks=ranks, instances=instances, program=name, protocol=protocol, dtype=dtype,
                elems=chunk * pieces)


def draw(rng):
    kind = rng.choice(('program', 'program', 'program', 'gemm', 'gemm_mxfp8', 'mlp', 'mlp', 'moe'))
    if kind == 'program':
        return _draw_program(rng)
    if kind == 'gemm':
        return dict(kind=kind, m=_log(rng, 16, 8192), n=rng.choice((3584, 4096, 7168, 14336)),
                    k=rng.choice((1792, 3584, HIDDEN, FFN // 2)), swiglu=rng.random() < 0.5)
    if kind == 'gemm_mxfp8':
        return dict(kind=kind, m=_log(rng, 16, 8192), n=rng.choice((3584, 4096, 7168)),
                    k=rng.choice((1792, HIDDEN, FFN // 2, FFN)))
    if kind == 'mlp':
        return dict(kind=kind, tokens=128 * _log(rng, 1, 63), ffn=FFN // rng.choice((1, 2, 4, 8)),
                    precision=rng.choice(('bf16', 'mxfp8')))
    return dict(kind=kind, tokens=_log(rng, 128, 4095), ffn=FFN // rng.choice((1, 2)), experts=8, topk=2)


# ------------------------------------------------------------------------------------------- handles a program keeps
@functools.lru_cache(maxsize=None)
def _executor(ranks):
    """One communicator and executor per number of ranks, kept for the life of the process."""
    return Executor(Communicator.emulated(ranks, fifo_bytes=128 * MB))


@functools.lru_cache(maxsize=None)
def _plan(ranks, program, protocol, instances):
    if program == 'synthesised':
        text = ncclize(solve_least_steps(fully_connected(ranks), synthesis_collectives.allgather(ranks)), instances=instances)
        return _executor(ranks).compile(load_xml(text))
    coll, body, manual = {
        'one_shot': (AllReduce(ranks, 1, True), lambda: allreduce_one_shot(ranks), True),
        'two_shot': (AllReduce(ranks, ranks, True), lambda: allreduce_two_shot(ranks), True),
        'ring': (AllReduce(ranks, ranks, True), lambda: allreduce_ring(ranks, min(ranks, 4)), True),
        'allgather': (AllGather(ranks, 1, False), lambda: allgather_direct(ranks), False),
        'reduce_scatter': (ReduceScatter(ranks, 1, False), lambda: reduce_scatter_direct(ranks), False),
        'alltoall': (AllToAll(ranks, 1, False), lambda: alltoall_direct(ranks), False),
    }[program]
    policy = dict(threadblock_policy=ThreadblockPolicy.manual) if manual else {}
    prog = MSCCLProgram(program, fully_connected(ranks), coll, instances, protocol=protocol, **policy)
    with prog:
        body()
    return _executor(ranks).compile(load_xml(prog.generate_xml()))


def _one_rank_communicator(arena_bytes):
    """The communicator of a job with one process: what the layers take on a single GPU."""
    if not dist.is_initialized():
        os.environ.setdefault('GLOO_SOCKET_IFNAME', 'lo')
        dist.init_process_group('gloo', store=dist.HashStore(), rank=0, world_size=1)
    return Communicator.from_process_group(fifo_bytes=16 * MB, arena_bytes=arena_bytes)


class _State(dict):
    """What ``prepare`` hands to ``run``; closes the communicator it owns when it is dropped."""

    def own(self, comm):
        weakref.finalize(self, comm.close)
        return comm


def _generator(seed):
    return torch.Generator(device='cuda').manual_seed(seed)


def _normal(gen, *shape, std=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, device='cuda', generator=gen) * std).to(dtype)


# ----------------------------------------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    gen = _generator(seed)
    state = _State(kind=case['kind'])
    if case['kind'] == 'program':
        ranks, elems, dtype = case['ranks'], case['elems'], DTYPES[case['dtype']]
        collective = PROGRAMS[case['program']][0]
        state['executor'] = _executor(ranks)
        state['plan'] = _plan(ranks, case['program'], case['protocol'], case['instances'])
        # gradients and activations: N(0, 0.05); the synthesised all-gather moves uniform values
        make = (lambda: torch.rand(elems, device='cuda', generator=gen).to(dtype)) if case['program'] == 'synthesised' \
            else (lambda: _normal(gen, elems, std=0.05, dtype=dtype))
        state['inputs'] = {r: make() for r in range(ranks)}
        # in place the sums of one pass are the inputs of the next, as in any in-place all-reduce that is repeated
        size = {'allreduce': 0, 'allgather': elems * ranks, 'reduce_scatter': elems // ranks, 'alltoall': elems}[collective]
        state['outputs'] = {r: torch.empty(size, dtype=dtype, device='cuda') for r in range(ranks)} if size else None
    elif case['kind'] == 'gemm':
        state['a'] = _normal(gen, case['m'], case['k'])
        if case['swiglu']:
            gate, up = (_normal(gen, case['n'] // 2, case['k'], std=0.02) for _ in range(2))
            state['b'] = interleave_gate_up(gate, up)
        else:
            state['b'] = _normal(gen, case['n'], case['k'], std=0.02)
        state['epilogue'] = 'swiglu' if case['swiglu'] else 'none'
    elif case['kind'] == 'gemm_mxfp8':
        state['a'] = _normal(gen, case['m'], case['k'])
        state['b'], state['sfb'] = quantize_mxfp8_packed(_normal(gen, case['n'], case['k'], std=0.02))
    elif case['kind'] == 'mlp':
        tokens, ffn = case['tokens'], case['ffn']
        comm = state.own(_one_rank_communicator(tokens * HIDDEN * 8 + 4 * MB))
        gate, up = (_normal(gen, ffn, HIDDEN, std=0.02) for _ in range(2))
        state['layer'] = TensorParallelMLP(comm, tokens, HIDDEN, ffn, w_gate=gate, w_up=up,
                                           w_down=_normal(gen, HIDDEN, ffn, std=0.02), precision=case['precision'])
        state['x'] = _normal(gen, tokens, HIDDEN)
    else:
        tokens, experts = case['tokens'], case['experts']
        rows = 2 * tokens * case['topk'] + 256 * experts
        comm = state.own(_one_rank_communicator((rows + tokens * case['topk']) * HIDDEN * 4 + 16 * MB))
        state['layer'] = ExpertParallelMoE(comm, tokens, HIDDEN, case['ffn'], experts, case['topk'], seed=seed)
        state['x'] = _normal(gen, tokens, HIDDEN)
        state['logits'] = torch.randn(tokens, experts, device='cuda', generator=gen)
    return state


def run(state):
    kind = state['kind']
    if kind == 'program':
        return state['executor'].run(state['plan'], state['inputs'], state['outputs'])
    if kind == 'gemm':
        return gemm_bf16(state['a'], state['b'], epilogue=state['epilogue'])
    if kind == 'gemm_mxfp8':
        q, scales = quantize_mxfp8_packed(state['a'])
        return gemm_mxfp8(q, scales, state['b'], state['sfb'])
    if kind == 'mlp':
        return state['layer'](state['x'])
    return state['layer'](state['x'], gate_logits=state['logits'])


# ---------------------------------------------------------------------------------------------------- work and tolerance
def work(case):
    """Bytes: every input and weight read once, every result written once.  FLOPs of the contractions."""
    if case['kind'] == 'program':
        n, nbytes = case['ranks'], case['elems'] * DTYPES[case['dtype']].itemsize
        written = {'allreduce': nbytes, 'allgather': nbytes * n, 'reduce_scatter': nbytes / n, 'alltoall': nbytes}
        sums = {'allreduce': (n - 1) * case['elems'], 'reduce_scatter': (n - 1) * case['elems']}
        collective = PROGRAMS[case['program']][0]
        return {'bytes': n * (nbytes + written[collective]), 'flops': sums.get(collective, 0)}
    if case['kind'] in ('gemm', 'gemm_mxfp8'):
        m, n, k = case['m'], case['n'], case['k']
        if case['kind'] == 'gemm':
            return {'bytes': 2 * (m * k + n * k + m * (n // 2 if case['swiglu'] else n)), 'flops': 2 * m * n * k}
        return {'bytes': 2 * m * k + n * k * 33 // 32 + 2 * m * n, 'flops': 2 * m * n * k}
    tokens, ffn = case['tokens'], case['ffn']
    if case['kind'] == 'mlp':
        weight_bytes = 3 * HIDDEN * ffn * (2 if case['precision'] == 'bf16' else 33 / 32)
        return {'bytes': weight_bytes + 2 * 2 * tokens * HIDDEN, 'flops': 6 * tokens * HIDDEN * ffn}
    weight_bytes = case['experts'] * 3 * HIDDEN * ffn * 2
    return {'bytes': weight_bytes + 2 * 2 * tokens * HIDDEN + 4 * tokens * case['experts'],
            'flops': 6 * tokens * case['topk'] * HIDDEN * ffn}


def tolerance(case):
    """Programs: the order of every sum and its rounding are part of the program, so results are bit exact.

    The others are compared with the same path in 64 bits (operands and intermediates rounded where the path rounds
    them): the one bf16 rounding of the result is 1.66e-3 of the norm, and 2.4e-3 with the expert outputs rounded before
    they are combined; the largest single difference is 0.004 (GEMMs), 0.015 (fp8 MLP, a value of the intermediate on
    the other side of an e4m3 step) and 0.012 (experts).  Four times that is stated."""
    if case['kind'] == 'program':
        return 'exact'
    if case['kind'] == 'moe':
        return {'rel': 1e-2, 'max': 0.05}
    return {'rel': 6.6e-3, 'max': 0.06 if case['kind'] == 'mlp' else 0.016}
