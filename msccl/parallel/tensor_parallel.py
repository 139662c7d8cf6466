"""Tensor + sequence parallel SwiGLU MLP: activations sharded by tokens, weights by the FFN dimension.

``forward`` = all-gather -> (gate|up) GEMM -> SwiGLU  (one fused kernel)  then
            down GEMM -> reduce-scatter               (one fused kernel).

``precision='mxfp8'`` runs both kernels on block-scaled fp8 operands (OCP MX: e4m3 values, one power-of-two scale per
32 K elements): the weights are quantised once, the activations per call (the token shard before the all-gather, the
SwiGLU output before the down projection); accumulation is fp32 and the result bf16 either way.

With one rank there is nothing to gather or to scatter: the layer runs on the plain GEMM kernels, whose tiles have the whole
GPU (the fused kernels set 8 and 12 SMs aside for the exchange) and walk the rows of a group first, so that activations stay
in L2 while the weights stream.
"""
import os

import torch

from msccl.ops.fused_tp import FusedTensorParallel
from msccl.ops.gemm import (gemm_bf16, gemm_mxfp8, gemm_mxfp8_swiglu, interleave_gate_up, pack_mx_scales, quantize_mxfp8,
                            quantize_mxfp8_packed)


class TensorParallelMLP:
    def __init__(self, comm, tokens_per_rank, hidden, ffn, w_gate=None, w_up=None, w_down=None, std=0.02, seed=0,
                 precision='bf16'):
        """``ffn`` is the full FFN width; this rank holds ``ffn / world`` of it.  Weights default to N(0, std)."""
        assert precision in ('bf16', 'mxfp8')
        self.precision = precision
        self.comm = comm
        self.shard = ffn // comm.world
        assert self.shard * comm.world == ffn and self.shard % 128 == 0
        dev = f'cuda:{comm.device}'
        gen = torch.Generator(device=dev).manual_seed(seed + comm.rank)
        mk = lambda *s: (torch.randn(*s, device=dev, generator=gen) * std).bfloat16()   # noqa: E731
        w_gate = mk(self.shard, hidden) if w_gate is None else w_gate
        w_up = mk(self.shard, hidden) if w_up is None else w_up
        self.w_gate_up = interleave_gate_up(w_gate, w_up)
        self.w_down = mk(hidden, self.shard) if w_down is None else w_down.contiguous()
        self.fused = FusedTensorParallel(comm, tokens_per_rank, hidden)
        # MSCCL_FUSED_PAIR=0 asks for the fused single-CTA kernels whatever the number of ranks; MSCCL_GEMM_PAIR=0 takes the plain
        # GEMMs off the CTA pairs that make them the faster choice (the quantising epilogue exists on pairs only)
        self.plain = (comm.world == 1 and os.environ.get('MSCCL_FUSED_PAIR', '1') != '0'
                      and os.environ.get('MSCCL_GEMM_PAIR', '1') == '1')
        # SwiGLU of the last call; with the quantising epilogue it exists as h_q and h_sf only
        self.h = None
        if not (self.plain and precision == 'mxfp8'):
            self.h = torch.empty(comm.world * tokens_per_rank, self.shard, dtype=torch.bfloat16, device=dev)
        if precision == 'mxfp8':
            if self.plain:
                self.h_q = torch.empty(tokens_per_rank, self.shard, dtype=torch.float8_e4m3fn, device=dev)
                self.h_sf = torch.empty(tokens_per_rank // 128 * (self.shard // 128) * 512, dtype=torch.uint8, device=dev)
            gu = interleave_gate_up(w_gate, w_up, tile=256 if self.plain else self.fused.mx_gate_up_tile)   # 256 on CTA pairs
            self.wq_gate_up, s = quantize_mxfp8(gu.float())
            self.sf_gate_up = pack_mx_scales(s, row_multiple=128)
            self.wq_down, s = quantize_mxfp8(self.w_down.float())
            self.sf_down = pack_mx_scales(s, row_multiple=128)

    def forward(self, x_local, out=None):
        """x_local: [tokens_per_rank, hidden] -> this rank's [tokens_per_rank, hidden] of the MLP output."""
        if self.plain:
            assert x_local.shape == (self.fused.rows, self.fused.hidden) and x_local.is_contiguous() and x_local.dtype == torch.bfloat16
            rows, hidden = x_local.shape
            if out is None:
                out = torch.empty(rows, hidden, dtype=torch.bfloat16, device=x_local.device)
            assert out.is_contiguous()
            y = out.view(-1).view(torch.bfloat16)[:rows * hidden].view(rows, hidden)      # any contiguous memory of that size will do
            self.fused.launches += 3 if self.precision == 'mxfp8' else 2
            if self.precision == 'mxfp8':
                xq, sx = quantize_mxfp8_packed(x_local)
                hq, sh = gemm_mxfp8_swiglu(xq, sx, self.wq_gate_up, self.sf_gate_up, self.h_q, self.h_sf)
                gemm_mxfp8(hq, sh, self.wq_down, self.sf_down, out=y)
            else:
                gemm_bf16(gemm_bf16(x_local, self.w_gate_up, out=self.h, epilogue='swiglu'), self.w_down, out=y)
            return out
        if self.precision == 'mxfp8':
            xq, sx = quantize_mxfp8_packed(x_local)                  # one kernel each: values + packed scales
            self.fused.all_gather_gemm_mxfp8(xq, sx, self.wq_gate_up, self.sf_gate_up, epilogue='swiglu', out=self.h)
            hq, sh = quantize_mxfp8_packed(self.h)
            return self.fused.gemm_reduce_scatter_mxfp8(hq, sh, self.wq_down, self.sf_down, out=out)
        self.fused.all_gather_gemm(x_local, self.w_gate_up, epilogue='swiglu', out=self.h)
        return self.fused.gemm_reduce_scatter(self.h, self.w_down, out=out)

    __call__ = forward
