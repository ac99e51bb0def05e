"""Tensor-parallel MLP block (Megatron-style column-parallel up projection, row-parallel down
projection, activations sharded over tokens between blocks) built on the fused kernels:

    x_shard [T / n, H]  --all-gather -> GEMM-->  h [T, F / n]  --act-->  --GEMM -> reduce-scatter-->  y_shard [T / n, H]

The forward pass is two kernel launches: ``AllGatherGemm``, whose epilogue also stores the activation, and
``GemmReduceScatter``.  The backward pass runs the transposed products through the same tcgen05 GEMM (operands as they
are stored, the derivative of the activation in the epilogue) and the library's own collectives.  This is the "fuse the collectives with your own kernels" use case the reference names as its
purpose (README.md:5) but does not implement; the shapes of the benchmark are the Llama-3-8B MLP ones
(tokens 8192, hidden 4096, ffn 14336, TP = 8).
"""
from __future__ import annotations

from typing import Optional

import torch

from ..ops.gemm import AllGatherGemm, GemmReduceScatter, gemm_dsilu, gemm_t


def _operand(t: torch.Tensor) -> torch.Tensor:
    """``t`` as TMA takes it: contiguous, on a 16-byte boundary.  A saved tensor is what a saved-tensor hook made of it."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


class _MLPFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x_shard, w_up, w_down, mlp):
        h, a = mlp.ag_gemm.call_silu(x_shard, w_up)          # [T, F/n], and silu of it
        y = mlp.gemm_rs(a, w_down)                           # [T/n, H]
        ctx.mlp, ctx.epoch = mlp, mlp.ag_gemm.epoch
        ctx.save_for_backward(x_shard, w_up, w_down, h, a)
        return y

    @staticmethod
    def backward(ctx, dy_shard):
        mlp = ctx.mlp
        comm = mlp.comm
        x_shard, w_up, w_down, h, a = map(_operand, ctx.saved_tensors)
        n, T = comm.world_size, mlp.tokens
        dy_shard = dy_shard.contiguous()
        # all-gather dy and x over tokens (plain collectives of this library); x is still in the plan's buffer, but for this
        # rank's own rows, unless another forward pass went through the plan since (the same answer on every rank)
        dy = mlp._gather(dy_shard)                           # [T, H]
        if n == 1:
            x = x_shard
        elif mlp.ag_gemm.epoch == ctx.epoch:
            x = mlp.ag_gemm.gathered.clone()
            x[comm.rank * (T // n):(comm.rank + 1) * (T // n)].copy_(x_shard)
        else:
            x = x_shard.new_empty((n, *x_shard.shape))
            comm.allgather(x, inp=x_shard)
            x = x.view(T, -1)
        dh = gemm_dsilu(dy, w_down, h)                       # [T, F/n] = (dy @ w_down) * silu'(h)   (w_down: [H, F/n])
        dw_down = gemm_t(dy, a, ta=True, tb=True)            # [H, F/n] = dy^T @ a
        dw_up = gemm_t(dh, x, ta=True, tb=True)              # [F/n, H] = dh^T @ x
        dx_shard = mlp.gemm_rs_bwd.call_transposed(dh, w_up)      # reduce_scatter(dh @ w_up)    (w_up: [F/n, H])
        return dx_shard, dw_up, dw_down, None


class TensorParallelMLP(torch.nn.Module):
    """``tokens`` is the global token count of a step (fixed: the fused plans own buffers of that size)."""

    def __init__(self, comm, tokens: int, hidden: int, ffn: int, ncomm: Optional[int] = None, seed: int = 0):
        super().__init__()
        n = comm.world_size
        if ffn % n or tokens % n:
            raise ValueError("ffn and tokens must be divisible by the world size")
        self.comm, self.tokens, self.hidden, self.ffn_local = comm, tokens, hidden, ffn // n
        dev = torch.device("cuda", comm.device)
        g = torch.Generator(device=dev).manual_seed(seed + 1000 * comm.rank)
        self.w_up = torch.nn.Parameter((torch.randn(self.ffn_local, hidden, generator=g, device=dev) * 0.02).to(torch.bfloat16))
        self.w_down = torch.nn.Parameter((torch.randn(hidden, self.ffn_local, generator=g, device=dev) * 0.02).to(torch.bfloat16))
        self.ag_gemm = AllGatherGemm(comm, tokens, self.ffn_local, hidden, ncomm=ncomm)
        self.gemm_rs = GemmReduceScatter(comm, tokens, hidden, self.ffn_local)
        self.gemm_rs_bwd = GemmReduceScatter(comm, tokens, hidden, self.ffn_local)
        self._gbuf: Optional[torch.Tensor] = None

    def _gather(self, shard: torch.Tensor) -> torch.Tensor:
        n = self.comm.world_size
        if n == 1:
            return shard
        if self._gbuf is None:
            self._gbuf = self.comm.symm_empty((n, shard.shape[0], shard.shape[1]), torch.bfloat16)
        self.comm.allgather(self._gbuf, inp=shard)
        return self._gbuf.view(-1, shard.shape[1])

    def forward(self, x_shard: torch.Tensor) -> torch.Tensor:
        return _MLPFunction.apply(x_shard, self.w_up, self.w_down, self)


def smoke_mlp() -> None:
    """One tiny forward + backward of the block on ``cuda:0`` (world size 1), checked against PyTorch."""
    import mintccl_b200
    from mintccl_b200 import Config
    cfg = Config.from_env(max_channels=2, num_blocks=2, buff_size=1 << 20, heap_bytes=256 << 20, scratch_bytes=1 << 20,
                          wait_timeout_ms=4000)
    from mintccl_b200.parallel.rendezvous import SingleControl
    comm = mintccl_b200.Communicator(control=SingleControl(), device=0, config=cfg)
    T, H, F = 256, 256, 512
    mlp = TensorParallelMLP(comm, T, H, F)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16).requires_grad_(True)
    dy = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    y = mlp(x)
    y.backward(dy)
    torch.cuda.synchronize()
    comm.check()
    xr, up, down = (t.detach().float().requires_grad_(True) for t in (x, mlp.w_up, mlp.w_down))
    ref = torch.nn.functional.silu(xr @ up.t()) @ down.t()
    torch.testing.assert_close(y.detach().float(), ref.detach(), rtol=5e-2, atol=5e-2)
    for got, want in zip((x.grad, mlp.w_up.grad, mlp.w_down.grad), torch.autograd.grad(ref, [xr, up, down], dy.float())):
        assert float((got.float() - want).norm() / want.norm()) < 1e-2      # a few roundings to bf16
    comm.close()
