"""tcgen05 GEMM and the fused GEMM + collective kernels against fp32 PyTorch references."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def ref_mm(a, w):
    return a.float() @ w.float().t()


def close(got, ref32, k):
    # bf16 output of an fp32-accumulated product: one rounding of the result (2^-8 relative)
    torch.testing.assert_close(got.float(), ref32, rtol=1.6e-2, atol=2e-2 * (k ** 0.5) * 0.05 + 1e-2)


@pytest.fixture(params=[1, 0], ids=["cta_pair", "single_cta"])
def gemm_kernel(request):
    """Plain GEMMs run on CTA pairs (tcgen05 cta_group::2, 256 rows and 64 to 256 columns a tile), or on the
    single-CTA kernel (128 x 256 tiles) with MINTCCL_GEMM_PAIR=0 and where 128 leftover rows make that faster; every shape
    is tested with both settings."""
    from mintccl_b200 import _native as N
    N.lib().mt_gemm_set_pair(request.param)
    yield request.param
    assert N.lib().mt_gemm_pair_error() == 0, "a bounded wait of the CTA-pair GEMM expired"
    N.lib().mt_gemm_set_pair(-1)


@pytest.mark.parametrize("shape", [(128, 256, 64), (256, 256, 64), (256, 512, 128), (384, 256, 1024), (1024, 1792, 4096),
                                   (2048, 4096, 1792), (4096, 2048, 512)])
def test_gemm_matches_fp32_reference(shape, gemm_kernel):
    from mintccl_b200.ops.gemm import gemm
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    out = gemm(a, w)
    torch.cuda.synchronize()
    close(out, ref_mm(a, w), K)
    # a second call on the same stream (fresh barriers, TMEM re-allocated) and fewer CTAs than tiles
    out2 = gemm(a, w, nctas=3)
    torch.cuda.synchronize()
    assert torch.equal(out, out2)


@pytest.mark.parametrize("bn", ["224", "256"])
@pytest.mark.parametrize("shape", [(256, 1792, 128), (2048, 1792, 512), (8192, 1792, 1024)])
def test_gemm_tile_width(shape, bn, monkeypatch):
    """The CTA-pair GEMM with 224-column tiles (chosen by itself when that saves a wave, forced here) against
    the fp32 reference and, bit for bit, against the 256-column tiles."""
    from mintccl_b200 import _native as N
    from mintccl_b200.ops.gemm import gemm
    M, Nn, K = shape
    g = torch.Generator(device="cuda").manual_seed(7 * M + K)
    a = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(Nn, K, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    N.lib().mt_gemm_set_pair(1)
    try:
        monkeypatch.setenv("MINTCCL_GEMM_BN", bn)
        out = gemm(a, w)
        monkeypatch.setenv("MINTCCL_GEMM_BN", "256")
        ref256 = gemm(a, w)
        torch.cuda.synchronize()
        assert N.lib().mt_gemm_pair_error() == 0
    finally:
        N.lib().mt_gemm_set_pair(-1)
    close(out, ref_mm(a, w), K)
    assert torch.equal(out, ref256)


_worlds = {}


def world(n):
    from mintccl_b200 import Config, emulated
    if n not in _worlds:
        cfg = Config.from_env(max_channels=4, num_blocks=4, buff_size=1 << 20, heap_bytes=768 << 20, scratch_bytes=1 << 20,
                              wait_timeout_ms=4000)
        _worlds[n] = emulated(n, 0, cfg)
    return _worlds[n]


@pytest.mark.parametrize("mode", ["push", "fan"])
@pytest.mark.parametrize("n", [1, 2, 4])
@pytest.mark.parametrize("N", [512, 1792])       # 1792: the fused kernel picks 224-column tiles
def test_ag_gemm_emulated(n, mode, N):
    from mintccl_b200.ops.gemm import AllGatherGemm
    w_ = world(n)
    M, K = 128 * n * 2, 256
    plan = AllGatherGemm(w_, M, N, K, ncomm=4, mode=mode)
    for it in range(3):  # counters keep growing across calls
        g = torch.Generator(device="cuda").manual_seed(it)
        shards = [torch.randn(M // n, K, generator=g, device="cuda").to(torch.bfloat16) for _ in range(n)]
        ws = [(torch.randn(N, K, generator=g, device="cuda") * 0.05).to(torch.bfloat16) for _ in range(n)]
        outs = plan(shards, ws)
        w_.check()
        full = torch.cat(shards, 0)
        for r in range(n):
            close(outs[r], ref_mm(full, ws[r]), K)


@pytest.mark.parametrize("n", [1, 2, 4])
def test_gemm_rs_emulated(n):
    from mintccl_b200.ops.gemm import GemmReduceScatter
    w_ = world(n)
    M, N, K = 128 * n * 2, 512, 192
    plan = GemmReduceScatter(w_, M, N, K)
    for it in range(3):
        g = torch.Generator(device="cuda").manual_seed(10 + it)
        As = [torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16) for _ in range(n)]
        ws = [(torch.randn(N, K, generator=g, device="cuda") * 0.05).to(torch.bfloat16) for _ in range(n)]
        outs = plan(As, ws)
        w_.check()
        # partial products are rounded to bf16 before the fp32 sum over ranks
        ref = sum(ref_mm(a, w).to(torch.bfloat16).float() for a, w in zip(As, ws))
        rows = M // n
        for r in range(n):
            torch.testing.assert_close(outs[r].float(), ref[r * rows:(r + 1) * rows], rtol=2e-2, atol=3e-2)


def test_tp_mlp_forward_backward_single_rank():
    from mintccl_b200.models.tp_mlp import smoke_mlp
    smoke_mlp()


@pytest.mark.parametrize("shape", [(128, 256, 128), (256, 256, 128), (256, 512, 512), (1024, 1792, 4096), (2048, 1024, 1024)])
def test_mxfp8_gemm_matches_dequantised_reference(shape, gemm_kernel):
    """Block-scaled fp8 GEMM against the fp32 product of the dequantised operands (the quantisation error is in
    both; what is compared is the tensor-core arithmetic and the scale plumbing)."""
    from mintccl_b200.ops import mxfp8 as mx
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, generator=g, device="cuda") * torch.logspace(-2, 2, M, device="cuda")[:, None]
    w = torch.randn(N, K, generator=g, device="cuda") * 0.02
    ad, asc = mx.quantize_rows_mxfp8(a)
    wd, wsc = mx.quantize_rows_mxfp8(w)
    out = mx.gemm_mxfp8(ad, asc, wd, wsc)
    torch.cuda.synchronize()
    a_dq = mx.dequantize_mxfp8(ad.reshape(-1), asc.reshape(-1)).view(M, K)
    w_dq = mx.dequantize_mxfp8(wd.reshape(-1), wsc.reshape(-1)).view(N, K)
    ref = a_dq @ w_dq.t()
    err = (out.float() - ref).abs()
    tol = 1.6e-2 * ref.abs() + 2e-3 * (a_dq.abs().amax(dim=1, keepdim=True) * (K ** 0.5) * 0.02)
    assert bool((err <= tol).all()), f"max err {err.max().item()} worst ratio {(err / tol).max().item()}"


@pytest.mark.parametrize("n", [1, 2, 4])
def test_fused_kernels_mxfp8_emulated(n):
    from mintccl_b200.ops import mxfp8 as mx
    from mintccl_b200.ops.gemm import AllGatherGemm, GemmReduceScatter
    w_ = world(n)
    M, N, K = 128 * n * 2, 512, 256
    g = torch.Generator(device="cuda").manual_seed(5)
    ag = AllGatherGemm(w_, M, N, K, ncomm=4, fp8=True)
    rs = GemmReduceScatter(w_, M, N, K)
    for it in range(2):
        shards = [torch.randn(M // n, K, generator=g, device="cuda") * (r + 1) for r in range(n)]
        ws = [torch.randn(N, K, generator=g, device="cuda") * 0.05 for _ in range(n)]
        qa = [mx.quantize_rows_mxfp8(t) for t in shards]
        qw = [mx.quantize_rows_mxfp8(t) for t in ws]
        outs = ag.call_mxfp8([q[0] for q in qa], [q[1] for q in qa], [q[0] for q in qw], [q[1] for q in qw])
        w_.check()
        a_dq = torch.cat([mx.dequantize_mxfp8(d.reshape(-1), s.reshape(-1)).view(M // n, K) for d, s in qa], 0)
        for r in range(n):
            w_dq = mx.dequantize_mxfp8(qw[r][0].reshape(-1), qw[r][1].reshape(-1)).view(N, K)
            torch.testing.assert_close(outs[r].float(), a_dq @ w_dq.t(), rtol=2e-2, atol=5e-2)
        As = [torch.randn(M, K, generator=g, device="cuda") for _ in range(n)]
        qA = [mx.quantize_rows_mxfp8(t) for t in As]
        ys = rs.call_mxfp8([q[0] for q in qA], [q[1] for q in qA], [q[0] for q in qw], [q[1] for q in qw])
        w_.check()
        ref = 0
        for r in range(n):
            A_dq = mx.dequantize_mxfp8(qA[r][0].reshape(-1), qA[r][1].reshape(-1)).view(M, K)
            w_dq = mx.dequantize_mxfp8(qw[r][0].reshape(-1), qw[r][1].reshape(-1)).view(N, K)
            ref = ref + (A_dq @ w_dq.t()).to(torch.bfloat16).float()
        rows = M // n
        for r in range(n):
            torch.testing.assert_close(ys[r].float(), ref[r * rows:(r + 1) * rows], rtol=2e-2, atol=6e-2)


@pytest.mark.parametrize("ta,tb", [(False, True), (True, True)])
@pytest.mark.parametrize("shape", [(128, 256, 64), (384, 256, 128), (256, 1792, 192), (1920, 512, 448), (8192, 1792, 256)])
def test_gemm_with_operands_stored_transposed(shape, ta, tb):
    """Same product, same accumulation order as on K-major copies: the same bits on the same tiles (N = 1792 takes
    224-column tiles where that saves a wave); M % 256 == 128 leaves the last CTA pair half empty."""
    from mintccl_b200.ops.gemm import gemm, gemm_t
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    out = gemm_t(a.t().contiguous() if ta else a, w.t().contiguous() if tb else w, ta=ta, tb=tb)
    torch.cuda.synchronize()
    close(out, ref_mm(a, w), K)
    if M % 256 == 0:
        assert torch.equal(out, gemm(a, w))


@pytest.mark.parametrize("n,rows", [(1, 128), (2, 256), (2, 128), (4, 256)])   # 128 rows a rank: single-CTA kernels
def test_gemm_rs_with_a_transposed_weight(n, rows):
    from mintccl_b200.ops.gemm import GemmReduceScatter
    w_ = world(n)
    M, N, K = rows * n, 512, 192
    plan = GemmReduceScatter(w_, M, N, K)
    for it in range(2):
        g = torch.Generator(device="cuda").manual_seed(20 + it)
        As = [torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16) for _ in range(n)]
        ws = [(torch.randn(N, K, generator=g, device="cuda") * 0.05).to(torch.bfloat16) for _ in range(n)]
        want = [t.clone() for t in plan(As, ws)]
        got = plan.call_transposed(As, [w.t().contiguous() for w in ws])
        w_.check()
        for x, y in zip(got, want):
            assert torch.equal(x, y)


@pytest.mark.parametrize("n,T,F,K", [(1, 128, 256, 64), (1, 384, 1792, 128), (1, 8192, 1792, 256), (2, 512, 512, 128), (2, 256, 512, 128),
                                     (4, 1024, 1792, 192)])
def test_silu_in_the_epilogue(n, T, F, K):
    """h is the same with and without the activation (same tiles, same order), and the activation is torch's silu of h."""
    from mintccl_b200.ops.gemm import AllGatherGemm
    w_ = world(n)
    plan = AllGatherGemm(w_, T, F, K, ncomm=4)
    g = torch.Generator(device="cuda").manual_seed(T + F)
    xs = [torch.randn(T // n, K, generator=g, device="cuda").to(torch.bfloat16) for _ in range(n)]
    ws = [torch.randn(F, K, generator=g, device="cuda").to(torch.bfloat16) for _ in range(n)]
    xs[0][0, :] = 100.0            # products far outside the range of the exponential
    plain = [h.clone() for h in plan(xs, ws)]
    hs, acts = plan.call_silu(xs, ws)
    w_.check()
    for h, a, p in zip(hs, acts, plain):
        assert torch.equal(h, p)
        assert torch.equal(a, torch.nn.functional.silu(h))


def all_bf16(rows, cols):
    """Every bit pattern of the type, once."""
    return torch.arange(rows * cols, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.bfloat16).view(rows, cols)


def same(a, b):
    return torch.equal(a.isnan(), b.isnan()) and torch.equal(a.nan_to_num(nan=0.0), b.nan_to_num(nan=0.0))


def test_silu_of_every_finite_bf16():
    """One-hot rows of x hand the weights through: h takes every finite value, those below -87 included, whose activation is
    tiny but normal."""
    from mintccl_b200.ops.gemm import AllGatherGemm
    T, F = 128, 512
    w_ = world(1)
    v = all_bf16(T, F)
    v = torch.where(v.isfinite(), v, torch.zeros_like(v))
    hs, acts = AllGatherGemm(w_, T, F, T).call_silu([torch.eye(T, device="cuda").to(torch.bfloat16)], [v.t().contiguous()])
    w_.check()
    assert torch.equal(hs[0], v)
    assert torch.equal(acts[0], torch.nn.functional.silu(v))
    assert bool((acts[0][(v < -87.4) & (v > -88.6)] != 0).all())
    hs, acts = AllGatherGemm(w_, T, F, T).call_silu([torch.eye(T, device="cuda").to(torch.bfloat16) * 3e38], [v.t().contiguous()])
    assert bool(hs[0].isposinf().any()) and bool(hs[0].isneginf().any())
    assert same(acts[0], torch.nn.functional.silu(hs[0]))


@pytest.mark.parametrize("shape", [(128, 256, 64), (128, 512, 64), (384, 1792, 128), (8192, 1792, 256), (2048, 512, 448)])
def test_silu_derivative_in_the_epilogue(shape):
    """The bits of the separate fp32 operations on the rounded product; (128, 512) has every bf16 value of h."""
    from mintccl_b200.ops.gemm import gemm_dsilu, gemm_t
    T, F, K = shape
    g = torch.Generator(device="cuda").manual_seed(T + K)
    d = torch.randn(T, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(K, F, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    h = (torch.randn(T, F, generator=g, device="cuda") * 3).to(torch.bfloat16)
    h[0, :8] = torch.tensor([-1e4, -90.0, -88.0, 0.0, 88.0, 90.0, 1e4, -20.0], device="cuda").to(torch.bfloat16)
    if (T, F) == (128, 512):
        h = all_bf16(T, F)
    got = gemm_dsilu(d, w, h)
    da = gemm_t(d, w, tb=True).float()
    sig = torch.sigmoid(h.float())
    assert same(got, (da * (sig * (1 + h.float() * (1 - sig)))).to(torch.bfloat16))


@pytest.mark.parametrize("form", ["plain", "tb", "ta_tb", "dsilu", "mxfp8"])
@pytest.mark.parametrize("bn", ["128", "64"])
@pytest.mark.parametrize("shape", [(128, 256, 128), (256, 512, 1152), (640, 1792, 512), (2432, 768, 256)])
def test_narrow_tiles_give_the_bits_of_wide_ones(shape, bn, form, monkeypatch):
    """The tiles of problems with too few 256-column ones (forced here; 64 columns exist for K-major bf16 only and fall
    back): every output is summed over K in the same order, so the bits are those of 256-column tiles."""
    from mintccl_b200.ops import gemm as G
    from mintccl_b200.ops import mxfp8 as mx
    M, Nn, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + Nn + K)
    a = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(Nn, K, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    h = torch.randn(M, Nn, generator=g, device="cuda").to(torch.bfloat16)
    at, wt = a.t().contiguous(), w.t().contiguous()
    qa, qw = mx.quantize_rows_mxfp8(a), mx.quantize_rows_mxfp8(w)
    call = {"plain": lambda: G.gemm(a, w), "tb": lambda: G.gemm_t(a, wt, tb=True), "ta_tb": lambda: G.gemm_t(at, wt, True, True),
            "dsilu": lambda: G.gemm_dsilu(a, wt, h), "mxfp8": lambda: mx.gemm_mxfp8(*qa, *qw)}[form]
    monkeypatch.setenv("MINTCCL_GEMM_BN", bn)
    out = call()
    monkeypatch.setenv("MINTCCL_GEMM_BN", "256")
    wide = call()
    monkeypatch.delenv("MINTCCL_GEMM_BN")
    chosen = call()
    torch.cuda.synchronize()
    if form == "plain":
        close(out, ref_mm(a, w), K)
    assert torch.equal(out, wide) and torch.equal(chosen, wide)


@pytest.mark.parametrize("shape", [(1152, 4096, 128), (1152, 4096, 1024), (128, 14336, 512), (2176, 1792, 256), (4224, 4096, 512)])
def test_128_leftover_rows_give_the_bits_of_pairs(shape, monkeypatch):
    """Shapes on both sides of the rule that sends a problem with 128 leftover rows to single CTAs (all but the last)."""
    from mintccl_b200.ops import gemm as G
    from mintccl_b200.ops import mxfp8 as mx
    M, Nn, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + Nn + K)
    a = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(Nn, K, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    qa, qw = mx.quantize_rows_mxfp8(a), mx.quantize_rows_mxfp8(w)
    for call in (lambda **k: G.gemm(a, w, **k), lambda **k: mx.gemm_mxfp8(*qa, *qw, **k)):
        chosen, few = call(), call(nctas=1)
        monkeypatch.setenv("MINTCCL_GEMM_BN", "256")
        pairs = call()
        monkeypatch.delenv("MINTCCL_GEMM_BN")
        assert torch.equal(chosen, pairs) and torch.equal(few, pairs)
    close(G.gemm(a, w), ref_mm(a, w), K)


def test_one_rank_plans_refuse_what_the_fused_kernels_do():
    """One CTA is no pair, and the reducers of the C interface have to leave one: refused although nothing is gathered or
    reduced at one rank.  128 rows run on single CTAs, where one is enough."""
    from mintccl_b200 import _native as N
    from mintccl_b200.ops.gemm import AllGatherGemm, GemmReduceScatter
    w_ = world(1)
    for rows, refused in ((256, True), (128, False)):
        a = torch.zeros(rows, 128, device="cuda", dtype=torch.bfloat16)
        b = torch.zeros(256, 128, device="cuda", dtype=torch.bfloat16)
        for plan in (AllGatherGemm(w_, rows, 256, 128), GemmReduceScatter(w_, rows, 256, 128)):
            if refused:
                with pytest.raises(RuntimeError, match="CTAs|nred"):
                    plan([a], [b], nctas=1)
            else:
                assert bool((plan([a], [b], nctas=1)[0] == 0).all())
    out = torch.empty(256, 256, device="cuda", dtype=torch.bfloat16)
    a = torch.zeros(256, 128, device="cuda", dtype=torch.bfloat16)
    ptrs = [N.ptr_array([t.data_ptr()]) for t in (a, b, out)]
    lib, args = w_.lib, (0, 0, 1, 256, 256, 128)
    for nred, nctas in ((-1, 0), (148, 0), (3, 4)):
        assert lib.mt_gemm_rs(w_._handle, w_._stream(), *ptrs, *args, nred, nctas) == -1
        assert "nred" in N.last_error()
    assert lib.mt_ag_gemm(w_._handle, w_._stream(), *ptrs, *args, 256, 0, 0, 4, 0, 1) == -1


@pytest.mark.parametrize("rows", [128, 512])
def test_one_rank_plans_leave_the_heap_alone(rows, gemm_kernel):
    """What they do not gather or stage is not allocated either, and they still give the product."""
    from mintccl_b200.ops.gemm import AllGatherGemm, GemmReduceScatter
    w_ = world(1)
    used = sum(w_._allocs.values())
    ag, rs = AllGatherGemm(w_, rows, 512, 1024), GemmReduceScatter(w_, rows, 512, 1024)
    assert sum(w_._allocs.values()) - used <= 4 * 256
    g = torch.Generator(device="cuda").manual_seed(rows)
    a = torch.randn(rows, 1024, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(512, 1024, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    for plan in (ag, rs):
        close(plan([a], [w])[0], ref_mm(a, w), 1024)
    w_.check()
    for t in (ag.gathered, ag.flags, rs.stage, rs.flags):
        w_.symm_free(t)
    assert sum(w_._allocs.values()) == used


def one_rank_mlp(T, H, F):
    import mintccl_b200
    from mintccl_b200 import Config
    from mintccl_b200.models.tp_mlp import TensorParallelMLP
    from mintccl_b200.parallel.rendezvous import SingleControl
    cfg = Config.from_env(max_channels=2, num_blocks=2, buff_size=1 << 20, heap_bytes=64 << 20, scratch_bytes=1 << 20,
                          wait_timeout_ms=4000)
    comm = mintccl_b200.Communicator(control=SingleControl(), device=0, config=cfg)
    return comm, TensorParallelMLP(comm, T, H, F)


def mlp_step(mlp, x, dy):
    x = x.detach().requires_grad_(True)
    y = mlp(x)
    return (y.detach(), *torch.autograd.grad(y, [x, mlp.w_up, mlp.w_down], dy))


@pytest.mark.parametrize("form", ["strided", "misaligned"])
def test_mlp_backward_takes_saved_tensors_in_any_layout(form):
    """A saved-tensor hook may hand a tensor back in another layout or off the 16-byte grid."""
    T, H, F = 384, 256, 512
    comm, mlp = one_rank_mlp(T, H, F)
    g = torch.Generator(device="cuda").manual_seed(2)
    x, dy = (torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    want = mlp_step(mlp, x, dy)

    def unpack(t):
        if form == "strided":
            return t.t().contiguous().t()
        return torch.cat([t.new_zeros(1), t.reshape(-1)])[1:].view(t.shape)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
        got = mlp_step(mlp, x, dy)
    comm.check()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    comm.close()


@pytest.mark.parametrize("T,H,F", [(384, 256, 512), (1024, 512, 1792)])
def test_mlp_gradients_against_autograd(T, H, F, gemm_kernel):
    """Forward and gradients of the block against fp32 autograd on the same bf16 inputs; 384 tokens leave 128 rows over.
    Up to four values on a path are rounded to bf16 (h, its activation, the two gradients behind them, the result), each
    2^-9 at most of its size: 2-norms within 8e-3 of the result's."""
    comm, mlp = one_rank_mlp(T, H, F)
    g = torch.Generator(device="cuda").manual_seed(T)
    x, dy = (torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    with torch.no_grad():
        mlp.w_up.copy_(torch.randn(F, H, generator=g, device="cuda") * H ** -0.5)
        mlp.w_down.copy_(torch.randn(H, F, generator=g, device="cuda") * F ** -0.5)
    got = mlp_step(mlp, x, dy)
    comm.check()
    xr, up, down = (t.detach().float().requires_grad_(True) for t in (x, mlp.w_up, mlp.w_down))
    y = torch.nn.functional.silu(xr @ up.t()) @ down.t()
    for a, b in zip(got, (y.detach(), *torch.autograd.grad(y, [xr, up, down], dy.float()))):
        assert float((a.float() - b).norm() / b.norm()) < 8e-3
    comm.close()
