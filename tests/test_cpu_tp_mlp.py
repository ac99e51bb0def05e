"""The autograd wiring of the tensor-parallel MLP on two ranks, without a GPU: two threads as ranks, the fused plans and
the GEMMs as torch expressions on fp32, gradients against autograd through the whole block."""
import threading

import pytest
import torch

from mintccl_b200.models import tp_mlp

N, T, H, F = 2, 8, 6, 10      # ranks, tokens, hidden, ffn


class Bus:
    """What the ranks exchange: each puts its tensor in, all see all of them."""

    def __init__(self):
        self.slots, self.bar = [None] * N, threading.Barrier(N, timeout=20)

    def swap(self, rank, t):
        self.slots[rank] = t
        self.bar.wait()
        out = [s.clone() for s in self.slots]
        self.bar.wait()
        return out


class Comm:
    world_size = N

    def __init__(self, bus, rank):
        self.bus, self.rank = bus, rank

    def symm_empty(self, shape, dtype):
        return torch.empty(shape)

    def allgather(self, out, inp):
        out.copy_(torch.stack(self.bus.swap(self.rank, inp.detach())))


class FakeGather:
    """``AllGatherGemm``: the peers' rows go to one buffer per plan, this rank's own are read in place."""

    def __init__(self, comm):
        self.comm, self.epoch, self.gathered = comm, 0, torch.full((T, H), float("nan"))

    def call_silu(self, x, w):
        self.epoch += 1
        xs, me, per = self.comm.bus.swap(self.comm.rank, x.detach()), self.comm.rank, T // N
        for r in range(N):
            if r != me:
                self.gathered[r * per:(r + 1) * per] = xs[r]
        h = torch.cat(xs) @ w.detach().t()
        return h, torch.nn.functional.silu(h)


class FakeScatter:
    def __init__(self, comm):
        self.comm = comm

    def __call__(self, a, w):
        return self.scatter(a.detach() @ w.detach().t())

    def call_transposed(self, a, w):
        return self.scatter(a.detach() @ w.detach())

    def scatter(self, full):
        per = T // N
        return sum(self.comm.bus.swap(self.comm.rank, full))[self.comm.rank * per:(self.comm.rank + 1) * per]


def mlp_of(comm, w_up, w_down):
    m = tp_mlp.TensorParallelMLP.__new__(tp_mlp.TensorParallelMLP)
    torch.nn.Module.__init__(m)
    m.comm, m.tokens, m._gbuf = comm, T, None
    m.w_up, m.w_down = torch.nn.Parameter(w_up.clone()), torch.nn.Parameter(w_down.clone())
    m.ag_gemm, m.gemm_rs, m.gemm_rs_bwd = FakeGather(comm), FakeScatter(comm), FakeScatter(comm)
    return m


def dsilu(d, w, h):
    s = torch.sigmoid(h)
    return (d @ w) * (s * (1 + h * (1 - s)))


@pytest.mark.parametrize("between", [0, 1, 2], ids=["backward_at_once", "two_in_flight", "evaluation_between"])
def test_gradients_of_two_ranks(between, monkeypatch):
    """0: forward, backward.  1: two forward passes, then their backward passes.  2: a forward pass without gradients
    between forward and backward.  The buffer of the gather belongs to the last forward pass."""
    monkeypatch.setattr(tp_mlp, "gemm_t", lambda a, b, ta=False, tb=False: (a.t() if ta else a) @ (b if tb else b.t()))
    monkeypatch.setattr(tp_mlp, "gemm_dsilu", dsilu)
    g = torch.Generator().manual_seed(between)
    ups, downs = torch.randn(N, F, H, generator=g), torch.randn(N, H, F, generator=g)
    xs, dys = torch.randn(2, T, H, generator=g), torch.randn(2, T, H, generator=g)
    used = [0] if between != 1 else [0, 1]
    got, errors, bus, per = {}, [], Bus(), T // N

    def rank(r):
        try:
            m, rows = mlp_of(Comm(bus, r), ups[r], downs[r]), slice(r * per, (r + 1) * per)
            shards = [xs[i][rows].clone().requires_grad_(True) for i in used]
            outs = [m(s) for s in shards]
            if between == 2:
                with torch.no_grad():
                    m(xs[1][rows])
            got[r] = [(y.detach(), *torch.autograd.grad(y, [s, m.w_up, m.w_down], dys[i][rows]))
                      for i, s, y in zip(used, shards, outs)]
        except Exception as e:      # the other rank waits: end its barrier too
            errors.append(e)
            bus.bar.abort()

    threads = [threading.Thread(target=rank, args=(r,)) for r in range(N)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(60)
    assert not errors, errors
    for k, i in enumerate(used):
        x = xs[i].clone().requires_grad_(True)
        u, d = ups.clone().requires_grad_(True), downs.clone().requires_grad_(True)
        y = sum(torch.nn.functional.silu(x @ u[r].t()) @ d[r].t() for r in range(N))
        dx, du, dd = torch.autograd.grad(y, [x, u, d], dys[i])
        for r in range(N):
            rows = slice(r * per, (r + 1) * per)
            for a, b in zip(got[r][k], (y.detach()[rows], dx[rows], du[r], dd[r])):
                torch.testing.assert_close(a, b, rtol=1e-4, atol=1e-4)     # fp32 sums of at most 20 terms
