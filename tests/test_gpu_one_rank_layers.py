"""The layers on one GPU (a communicator of one process): the MLP that runs on the plain GEMM kernels there."""
import os

import pytest
import torch
import torch.distributed as dist

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def one_rank():
    from msccl.runtime import Communicator
    os.environ.setdefault('GLOO_SOCKET_IFNAME', 'lo')
    dist.init_process_group('gloo', store=dist.HashStore(), rank=0, world_size=1)
    made = []

    def make(arena_bytes):
        made.append(Communicator.from_process_group(fifo_bytes=1 << 20, arena_bytes=arena_bytes))
        return made[-1]
    yield make
    for comm in made:
        comm.close()
    dist.destroy_process_group()


def _normal(gen, *shape, std=1.0):
    return (torch.randn(*shape, device='cuda', generator=gen) * std).bfloat16()


def _weights(gen, hidden, ffn):
    return [_normal(gen, ffn, hidden, std=0.02), _normal(gen, ffn, hidden, std=0.02), _normal(gen, hidden, ffn, std=0.02)]


def _swiglu(gate, up):
    return gate / (1 + torch.exp(-gate)) * up


def _mx(t):
    from msccl.ops.gemm import dequantize_mxfp8, quantize_mxfp8
    return dequantize_mxfp8(*quantize_mxfp8(t.float())).double()


@pytest.mark.parametrize('precision', ['bf16', 'mxfp8'])
@pytest.mark.parametrize('tokens', [128, 384, 1024])
def test_mlp_on_one_rank(one_rank, tokens, precision):
    """Against 64 bits with operands and intermediates rounded where the layer rounds them.

    bf16: the result's own rounding is at most 2^-9 of its norm; an intermediate on the other side of a rounding is off by
    2^-8 of itself, and even 5 % of them would add 2^-8 sqrt(0.05) < 2^-10: together below 2^-8.  Block-scaled fp8: an
    intermediate on the other side of an e4m3 step is off by up to 2^-3; one in a thousand of them adds 4e-3: below 6.6e-3."""
    from msccl.ops import check_gemm_errors
    from msccl.parallel import TensorParallelMLP
    hidden, ffn = 1024, 1280                           # long enough sums that few tokens split them (bf16)
    gen = torch.Generator(device='cuda').manual_seed(tokens)
    w_gate, w_up, w_down = _weights(gen, hidden, ffn)
    layer = TensorParallelMLP(one_rank(tokens * hidden * 8 + (4 << 20)), tokens, hidden, ffn, w_gate=w_gate, w_up=w_up, w_down=w_down,
                              precision=precision)
    assert layer.plain and (layer.h is None) == (precision == 'mxfp8')
    holder = torch.full((tokens + 2, hidden), 7.0, dtype=torch.bfloat16, device='cuda')
    raw = torch.zeros(tokens * hidden * 2, dtype=torch.uint8, device='cuda')
    for call in range(3):
        x = _normal(gen, tokens, hidden)
        if precision == 'bf16':
            h = _swiglu(x.double() @ w_gate.double().t(), x.double() @ w_up.double().t()).bfloat16().double()
            want = h @ w_down.double().t()
        else:
            h = _swiglu(_mx(x) @ _mx(w_gate).t(), _mx(x) @ _mx(w_up).t()).bfloat16()
            want = _mx(h) @ _mx(w_down).t()
        # the result in a tensor of its own, in the middle of another one, and in plain bytes of that size
        got = layer(x) if call == 0 else layer(x, out=holder[1:-1] if call == 1 else raw)
        check_gemm_errors()
        if call == 2:
            assert got is raw
            got = raw.view(torch.bfloat16).view(tokens, hidden)
        error = float((got.double() - want).norm() / want.norm())
        assert error < (2.0 ** -8 if precision == 'bf16' else 6.6e-3), error
        assert torch.equal(layer(x), got)
    assert torch.all(holder[0] == 7) and torch.all(holder[-1] == 7)


@pytest.mark.parametrize('precision', ['bf16', 'mxfp8'])
@pytest.mark.parametrize('switch', ['MSCCL_FUSED_PAIR', 'MSCCL_GEMM_PAIR'])
def test_switches_take_the_layer_back_to_the_fused_kernels(one_rank, switch, precision, monkeypatch):
    from msccl.parallel import TensorParallelMLP
    tokens, hidden, ffn = 256, 1024, 1280
    gen = torch.Generator(device='cuda').manual_seed(1)
    w_gate, w_up, w_down = _weights(gen, hidden, ffn)
    x = _normal(gen, tokens, hidden)
    build = lambda: TensorParallelMLP(one_rank(8 << 20), tokens, hidden, ffn, w_gate=w_gate, w_up=w_up, w_down=w_down,    # noqa: E731
                                      precision=precision)
    plain = build()(x)
    monkeypatch.setenv(switch, '0')
    layer = build()
    assert not layer.plain and layer.fused.pair == (switch == 'MSCCL_GEMM_PAIR')
    got = layer(x)
    if precision == 'mxfp8':
        assert torch.equal(got, plain)
    else:                                              # the plain kernels split K here: bits may differ by a rounding
        assert float((got.double() - plain.double()).norm() / plain.double().norm()) < 2.0 ** -8
