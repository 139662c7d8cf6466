"""The layers on one GPU (a communicator of one process): the MLP that runs on the plain GEMM kernels there, the GEMM epilogue
that quantises its SwiGLU result, and the MoE dispatch in which every CTA moves rows."""
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


@pytest.mark.parametrize('tokens', [128, 256, 384, 1024])
def test_quantised_swiglu_gives_the_bytes_of_the_separate_kernels(one_rank, tokens):
    """The fused all-gather GEMM on one rank stores the bf16 SwiGLU, which the quantisation kernel then reads."""
    from msccl.ops import check_gemm_errors
    from msccl.ops.fused_tp import FusedTensorParallel
    from msccl.ops.gemm import gemm_mxfp8_swiglu, interleave_gate_up, pack_mx_scales, quantize_mxfp8, quantize_mxfp8_packed
    hidden, ffn = 1024, 1280
    gen = torch.Generator(device='cuda').manual_seed(tokens)
    w_gate, w_up, _ = _weights(gen, hidden, ffn)
    x = _normal(gen, tokens, hidden) * torch.exp2(torch.randint(-8, 9, (tokens, 1), device='cuda', generator=gen).float()).bfloat16()
    fused = FusedTensorParallel(one_rank(tokens * hidden * 8 + (4 << 20)), tokens, hidden)
    packed = {}
    for tile in (256, fused.mx_gate_up_tile):
        q, s = quantize_mxfp8(interleave_gate_up(w_gate, w_up, tile=tile).float())
        packed[tile] = q, pack_mx_scales(s, row_multiple=128)
    xq, sx = quantize_mxfp8_packed(x)
    want_q, want_sf = quantize_mxfp8_packed(fused.all_gather_gemm_mxfp8(xq, sx, *packed[fused.mx_gate_up_tile], epilogue='swiglu'))
    q = torch.empty(tokens, ffn, dtype=torch.float8_e4m3fn, device='cuda')
    sf = torch.empty(tokens // 128 * (ffn // 128) * 512, dtype=torch.uint8, device='cuda')
    gemm_mxfp8_swiglu(xq, sx, *packed[256], q, sf)
    check_gemm_errors()
    assert torch.equal(q.view(torch.uint8), want_q.view(torch.uint8)) and torch.equal(sf, want_sf)


@pytest.mark.parametrize('m', [1, 130, 257])
def test_quantised_swiglu_writes_its_rows_only(m):
    from msccl.ops import check_gemm_errors
    from msccl.ops.gemm import gemm_mxfp8_swiglu, quantize_mxfp8_packed
    n, k, padded = 1024, 512, -(-m // 256) * 256
    gen = torch.Generator(device='cuda').manual_seed(m)
    a, b = _normal(gen, padded, k), _normal(gen, n, k, std=0.05)
    bq, sb = quantize_mxfp8_packed(b)
    full_q = torch.empty(padded, n // 2, dtype=torch.float8_e4m3fn, device='cuda')
    full_sf = torch.empty(padded // 128 * (n // 256) * 512, dtype=torch.uint8, device='cuda')
    gemm_mxfp8_swiglu(*quantize_mxfp8_packed(a), bq, sb, full_q, full_sf)
    q = torch.full((m + 2, n // 2), 85, dtype=torch.uint8, device='cuda')
    blocks = -(-m // 128) * (n // 256)
    sf = torch.full(((blocks + 2) * 512,), 255, dtype=torch.uint8, device='cuda')
    gemm_mxfp8_swiglu(*quantize_mxfp8_packed(a[:m]), bq, sb, q[1:-1].view(torch.float8_e4m3fn), sf[512:-512])
    check_gemm_errors()
    assert torch.equal(q[1:-1], full_q[:m].view(torch.uint8)) and torch.all(q[0] == 85) and torch.all(q[-1] == 85)
    assert torch.all(sf[:512] == 255) and torch.all(sf[-512:] == 255)
    # byte (r % 32) * 16 + (r // 32) * 4 + j of a block is row r's
    byte = torch.arange(512, device='cuda')
    row = byte // 16 + byte % 16 // 4 * 32
    got, want = sf[512:-512].view(-1, n // 256, 512), full_sf.view(-1, n // 256, 512)
    for block in range(got.shape[0]):
        mine = row + 128 * block < m
        assert torch.equal(got[block][:, mine], want[block][:, mine]) and torch.all(got[block][:, ~mine] == 255)


def _moe_reference(x, logits, topk, layer, hidden, ffn):
    from msccl.ops.moe import route_top_k
    experts, weights = route_top_k(logits, topk)
    want = torch.zeros(x.shape[0], hidden, dtype=torch.float64, device='cuda')
    gate_up = layer.w_gate_up.view(-1, ffn // 128, 2, 128, hidden).double()
    down = layer.w_down.view(-1, hidden, ffn).double()
    for e in range(down.shape[0]):
        gate, up = (gate_up[e, :, i].reshape(ffn, hidden) for i in (0, 1))
        h = _swiglu(x.double() @ gate.t(), x.double() @ up.t()).bfloat16().double()
        share = torch.where(experts == e, weights.double(), 0).sum(1, keepdim=True)
        want += share * (h @ down[e].t())
    return want


@pytest.mark.parametrize('tokens,topk', [(1, 1), (5, 2), (6, 1), (130, 2), (1776, 2), (1777, 2), (4100, 1)])
def test_moe_dispatch_by_every_cta(one_rank, tokens, topk):
    """Fewer copies than one batch, a short last batch, both sides of the line between one and two copies per warp (4 x 6 x 148
    copies), several calls: the counters start again.  The products of an expert are rounded to bf16 before the sum over the
    experts and the sum once more, 2^-8 together, and the intermediate rounding adds less than 2^-10 (see the MLP test)."""
    from msccl.ops import check_gemm_errors
    from msccl.parallel import ExpertParallelMoE
    hidden, ffn, experts = 256, 256, 8
    comm = one_rank((2 * tokens * topk + 2048 + tokens * topk) * hidden * 4 + (4 << 20))
    layer = ExpertParallelMoE(comm, tokens, hidden, ffn, experts, topk, seed=3)
    gen = torch.Generator(device='cuda').manual_seed(tokens)
    for _ in range(4):
        x, logits = _normal(gen, tokens, hidden), torch.randn(tokens, experts, device='cuda', generator=gen)
        got = layer(x, gate_logits=logits)
        check_gemm_errors()
        want = _moe_reference(x, logits, topk, layer, hidden, ffn)
        assert float((got.double() - want).norm() / want.norm()) < 2.0 ** -8 + 2.0 ** -10
        assert torch.equal(layer(x, gate_logits=logits), got)


def test_moe_beside_another_stream(one_rank):
    """CTAs that another stream's kernels keep off the GPU have no share of the rows that the others wait for."""
    from msccl.ops import check_gemm_errors
    from msccl.parallel import ExpertParallelMoE
    tokens, hidden, ffn = 1024, 512, 512
    layer = ExpertParallelMoE(one_rank((3 * tokens * 2 + 2048) * hidden * 4 + (4 << 20)), tokens, hidden, ffn, 8, 2, seed=4)
    gen = torch.Generator(device='cuda').manual_seed(9)
    x, logits = _normal(gen, tokens, hidden), torch.randn(tokens, 8, device='cuda', generator=gen)
    want = layer(x, gate_logits=logits)
    a = _normal(gen, 4096, 4096)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        products = [a @ a for _ in range(40)]
    got = [layer(x, gate_logits=logits) for _ in range(10)]
    torch.cuda.synchronize()
    check_gemm_errors()
    assert all(torch.equal(t, want) for t in got) and all(torch.equal(t, products[0]) for t in products)
