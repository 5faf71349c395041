"""CUDA kernels of siirl_b200.ops.dense against plain PyTorch fp32 statements of the same op."""
import pytest
import torch

from siirl_b200 import ops
from siirl_b200.ops import dense, lib, reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rel_err(a, b):
    return ((a.float() - b.float()).norm() / (b.float().norm() + 1e-12)).item()


@pytest.mark.parametrize("tile_n", [128, 256])
@pytest.mark.parametrize("shape", [(128, 256, 64), (256, 512, 256), (300, 520, 200), (1024, 4608, 3584)])
def test_gemm_nt(shape, tile_n):
    M, N, K = shape
    torch.manual_seed(0)
    a = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    b = torch.randn(N, K, device=DEV, dtype=torch.bfloat16)
    bias = torch.randn(N, device=DEV, dtype=torch.bfloat16)
    out = ops.gemm(a, b, bias=bias, tile_n=tile_n)
    lib.check_status()
    want = a.float() @ b.float().t() + bias.float()
    assert _rel_err(out, want) < 1e-2
    out32 = ops.gemm(a, b, epi=dense.EPI_F32, tile_n=tile_n)
    lib.check_status()
    assert _rel_err(out32, a.float() @ b.float().t()) < 1e-3


@pytest.mark.parametrize("shape", [(128, 128, 64), (256, 320, 192), (520, 384, 264), (2048, 3584, 4608)])
def test_gemm_dgrad_layout(shape):
    """B stored [K, N] (weight [out,in] used for dx = dy @ W)."""
    M, N, K = shape
    torch.manual_seed(1)
    a = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    b = torch.randn(K, N, device=DEV, dtype=torch.bfloat16)
    out = ops.gemm(a, b, b_mn=True)
    lib.check_status()
    assert _rel_err(out, a.float() @ b.float()) < 1e-2


@pytest.mark.parametrize("shape", [(128, 128, 64), (320, 256, 192), (384, 520, 1000), (3584, 4608, 2048)])
def test_gemm_wgrad_layout(shape):
    """A stored [K, M], B stored [K, N]; fp32 accumulate epilogue (dW += dy^T x)."""
    M, N, K = shape
    torch.manual_seed(2)
    a = torch.randn(K, M, device=DEV, dtype=torch.bfloat16)
    b = torch.randn(K, N, device=DEV, dtype=torch.bfloat16)
    acc = torch.randn(M, N, device=DEV, dtype=torch.float32)
    want = acc + a.float().t() @ b.float()
    ops.gemm(a, b, out=acc, a_mn=True, b_mn=True, epi=dense.EPI_F32_ACC)
    lib.check_status()
    assert _rel_err(acc, want) < 1e-3


def test_linear_autograd_matches_torch():
    torch.manual_seed(3)
    x = torch.randn(4, 96, 256, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    w = torch.randn(384, 256, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    b = torch.randn(384, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    y = ops.linear(x, w, b)
    g = torch.randn_like(y)
    y.backward(g)
    xr, wr, br = (t.detach().float().requires_grad_() for t in (x, w, b))
    yr = torch.nn.functional.linear(xr, wr, br)
    yr.backward(g.float())
    assert _rel_err(y, yr) < 1e-2
    assert _rel_err(x.grad, xr.grad) < 1e-2
    assert _rel_err(w.grad, wr.grad) < 1e-2
    assert _rel_err(b.grad, br.grad) < 1e-2


@pytest.mark.parametrize("H", [128, 3584, 8192])
@pytest.mark.parametrize("with_res", [False, True])
def test_rmsnorm_fwd_bwd(H, with_res):
    torch.manual_seed(4)
    T = 77
    x = torch.randn(T, H, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    r = torch.randn(T, H, device=DEV, dtype=torch.bfloat16, requires_grad=True) if with_res else None
    w = (1 + 0.1 * torch.randn(H, device=DEV)).to(torch.bfloat16).requires_grad_()
    y, h = ops.rmsnorm(x, w, 1e-6, residual=r)
    gy, gh = torch.randn_like(y), torch.randn_like(y)
    (y.float() * gy.float()).sum().add((h.float() * gh.float()).sum()).backward()
    xr = x.detach().float().requires_grad_()
    rr = r.detach().float().requires_grad_() if with_res else None
    wr = w.detach().float().requires_grad_()
    hr = xr + rr if with_res else xr
    if with_res:
        hr = hr + (hr.to(torch.bfloat16).float() - hr).detach()  # kernel rounds h to bf16
    yr = hr * torch.rsqrt(hr.pow(2).mean(-1, keepdim=True) + 1e-6) * wr
    ((yr * gy.float()).sum() + (hr * gh.float()).sum()).backward()
    assert _rel_err(y, yr) < 1e-2
    assert _rel_err(x.grad, xr.grad) < 2e-2
    assert _rel_err(w.grad, wr.grad) < 2e-2
    if with_res:
        assert _rel_err(r.grad, rr.grad) < 2e-2


def test_rope_matches_reference_and_inverse():
    torch.manual_seed(5)
    T, hq, hk, D = 50, 4, 2, 128
    qkv = torch.randn(T, (hq + 2 * hk) * D, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    pos = torch.randint(0, 500, (T,), device=DEV)
    cos, sin = ops.rope_tables(D, 512, 1e6, device=DEV)
    out = ops.rope(qkv, hq + hk, D, pos, cos, sin)
    want = ref.rope(qkv.detach()[:, : (hq + hk) * D].reshape(T, hq + hk, D), pos, cos, sin).reshape(T, -1)
    assert _rel_err(out[:, : (hq + hk) * D], want) < 1e-2
    assert torch.equal(out[:, (hq + hk) * D:], qkv[:, (hq + hk) * D:])
    g = torch.randn_like(out)
    out.backward(g)
    want_g = ref.rope(g[:, : (hq + hk) * D].reshape(T, hq + hk, D), pos, cos, sin, inverse=True).reshape(T, -1)
    assert _rel_err(qkv.grad[:, : (hq + hk) * D], want_g) < 1e-2


def test_mrope_sections():
    torch.manual_seed(6)
    T, nh, D = 33, 3, 128
    x = torch.randn(T, nh * D, device=DEV, dtype=torch.bfloat16)
    pos = torch.randint(0, 100, (3, T), device=DEV)
    cos, sin = ops.rope_tables(D, 128, 1e6, device=DEV)
    sec = (16, 24, 24)
    out = ops.rope(x, nh, D, pos, cos, sin, mrope_section=sec)
    want = ref.rope(x.reshape(T, nh, D), pos, cos, sin, mrope_section=sec).reshape(T, -1)
    assert _rel_err(out, want) < 1e-2


def test_swiglu_fwd_bwd():
    torch.manual_seed(7)
    gu = torch.randn(65, 2 * 352, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    out = ops.swiglu(gu)
    g = torch.randn_like(out)
    out.backward(g)
    gr = gu.detach().float().requires_grad_()
    a, b = gr.chunk(2, -1)
    outr = torch.nn.functional.silu(a) * b
    outr.backward(g.float())
    assert _rel_err(out, outr) < 1e-2
    assert _rel_err(gu.grad, gr.grad) < 1e-2


def test_embedding_fwd_bwd():
    torch.manual_seed(8)
    V, H = 1000, 256
    table = torch.randn(V, H, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    ids = torch.randint(0, V, (7, 19), device=DEV)
    out = ops.embedding(ids, table)
    assert torch.equal(out, table.detach()[ids])
    g = torch.randn_like(out)
    out.backward(g)
    want = torch.zeros(V, H, device=DEV).index_add_(0, ids.reshape(-1), g.reshape(-1, H).float())
    assert _rel_err(table.grad, want) < 1e-2


@pytest.mark.parametrize("shape", [(64, 3584, 3584), (7, 3584, 18944), (128, 4608, 3584), (33, 256, 1024),
                                   (200, 4608, 3584), (256, 3584, 18944), (256, 37888, 3584), (300, 1000, 1024),
                                   (512, 3584, 1792), (129, 136, 64)])
def test_skinny_split_k_linear(shape):
    M, N, K = shape
    torch.manual_seed(9)
    x = (0.5 * torch.randn(M, K, device=DEV)).to(torch.bfloat16)
    w = (0.05 * torch.randn(N, K, device=DEV)).to(torch.bfloat16)
    b = torch.randn(N, device=DEV).to(torch.bfloat16)
    with torch.no_grad():
        y = ops.linear(x, w, b)
    lib.check_status()
    want = x.float() @ w.float().t() + b.float()
    assert _rel_err(y, want) < 1e-2
    # no row or column of the (possibly transposed-store) tile went astray: element-wise bound, bf16 output rounding
    assert (y.float() - want).abs().max().item() < 0.05 * want.abs().max().item() + 0.05
    assert dense._skinny_splits(64, 3584, 18944) > 1
    if M > 128:     # the operand-swapped form and the plain form agree
        dense.SWAP_OPERANDS_ABOVE_128_ROWS = False
        try:
            with torch.no_grad():
                y2 = ops.linear(x, w, b)
        finally:
            dense.SWAP_OPERANDS_ABOVE_128_ROWS = True
        assert _rel_err(y, y2) < 1e-2


def test_optimizer_state_offload_round_trip():
    """Adam moments parked in pinned host memory between steps give the same updates as resident ones."""
    import torch

    from siirl_b200.parallel.flat_params import FlatParamStore

    def make():
        torch.manual_seed(0)
        m = torch.nn.Linear(256, 512, bias=True).cuda().bfloat16()
        return m, FlatParamStore(m)

    (ma, sa), (mb, sb) = make(), make()
    g = torch.Generator(device="cuda").manual_seed(1)
    for step in range(3):
        grad = torch.randn(sa.total, device="cuda", generator=g)
        for s in (sa, sb):
            s.flat_grad.copy_(grad)
        # no clipping: the clip factor comes from an atomically accumulated norm whose last bits vary run to run
        sa.step(1e-2, max_grad_norm=0.0)
        sb.step(1e-2, max_grad_norm=0.0)
        sb.offload_state()
        assert sb.exp_avg is None and sb._host_state["exp_avg"].is_pinned()
    sb.reload_state()
    assert torch.equal(sa.flat_param, sb.flat_param) and torch.equal(sa.exp_avg, sb.exp_avg)
    assert torch.equal(sa.exp_avg_sq, sb.exp_avg_sq)


@pytest.mark.parametrize("rows", [1, 8, 100, 129, 256, 300])
@pytest.mark.parametrize("hidden,inter,hq,hkv,d", [(896, 2432, 14, 2, 64), (1024, 1536, 4, 4, 128)])
def test_partial_sums_and_their_consumers(rows, hidden, inter, hq, hkv, d):
    """Projections of few rows whose partial sums go to the norm, the gated activation, and rope with the cache append."""
    from siirl_b200.ops import kv_cache as kvc
    torch.manual_seed(0)
    mk = lambda *s: (torch.randn(*s, device=DEV) / s[-1] ** 0.5).to(torch.bfloat16)  # noqa: E731
    x = torch.randn(rows, hidden, device=DEV).to(torch.bfloat16)
    h, w = torch.randn_like(x), (1 + 0.1 * torch.randn(hidden, device=DEV)).to(torch.bfloat16)
    wo, wg, wq, bias = mk(hidden, hidden), mk(2 * inter, hidden), mk((hq + 2 * hkv) * d, hidden), mk((hq + 2 * hkv) * d)
    so, sg, sq = (ops.linear_slabs(x, t) for t in (wo, wg, wq))
    assert so is not None and sq is not None and sg is not None
    y, hs = ops.rmsnorm_slabs(so, w, 1e-6, h)
    want = x.double() @ wo.double().T + h.double()
    # results rounded to bf16 once (2^-9 relative), the norm's input as well
    assert ((hs.double() - want).norm() / want.norm()).item() < 3e-3
    want = want * torch.rsqrt(want.square().mean(-1, keepdim=True) + 1e-6) * w.double()
    assert ((y.double() - want).norm() / want.norm()).item() < 5e-3
    g, u = (x.double() @ wg.double().T).chunk(2, -1)
    want = torch.nn.functional.silu(g) * u
    assert ((ops.swiglu_slabs(sg).double() - want).norm() / want.norm()).item() < 3e-3
    cos, sin = ops.rope_tables(d, 64, 10000.0, device=DEV)
    pos = (torch.arange(rows, device=DEV) % 64).to(torch.int32)
    seq = torch.arange(rows, device=DEV, dtype=torch.int32)
    seq[rows // 2] = -1
    table = torch.arange(rows, device=DEV, dtype=torch.int32)[:, None].contiguous()
    cache = [torch.zeros(rows, 2, hkv, 64, d, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    a = kvc.rope_kv_append(sq, pos, cos, sin, None, seq, pos, table, cache[0], hq, hkv, d, bias)
    b = kvc.rope_kv_append(ops.linear(x, wq, bias), pos, cos, sin, None, seq, pos, table, cache[1], hq, hkv, d)
    # the sums enter unrounded here, rounded to bf16 there
    assert ((a.double() - b.double()).norm() / b.double().norm()).item() < 4e-3
    assert ((cache[0].double() - cache[1].double()).norm() / (cache[1].double().norm() + 1e-9)).item() < 4e-3
    for p, q in zip(*cache):
        assert torch.equal(p.abs().sum(-1) != 0, q.abs().sum(-1) != 0)


@pytest.mark.parametrize("T,heads,rot,d,mrope", [(1, 18, 16, 64, None), (300, 36, 32, 128, None), (77, 6, 6, 16, None),
                                                 (130, 8, 5, 128, [16, 24, 24]), (9, 5, 3, 24, None)])
def test_rope_rows(T, heads, rot, d, mrope):
    """Rotated and copied heads, three position rows, and a width that takes the copy and the scalar kernel."""
    torch.manual_seed(0)
    x = torch.randn(T, heads * d, device=DEV).to(torch.bfloat16).requires_grad_()
    cos, sin = ops.rope_tables(d, 512, 10000.0, device=DEV)
    pos = torch.randint(0, 512, (3, T) if mrope else (T,), device=DEV)
    y = ops.rope(x, rot, d, pos, cos, sin, mrope)
    g = torch.randn_like(y)
    y.backward(g)
    for src, got, inverse in ((x.detach(), y.detach(), False), (g, x.grad, True)):
        want = ref.rope(src[:, :rot * d].double().reshape(T, rot, d), pos, cos.double(), sin.double(), mrope,
                        inverse).reshape(T, rot * d)
        # one rounding to bf16: 2^-9 of the larger operand
        assert (got[:, :rot * d].double() - want).abs().max() <= 2 ** -8 * want.abs().max()
        assert torch.equal(got[:, rot * d:], src[:, rot * d:])


@pytest.mark.parametrize("T,I", [(1, 8), (2, 1024), (3, 1032), (301, 4864), (5000, 264)])
def test_swiglu_rows(T, I):
    torch.manual_seed(0)
    gu = (2 * torch.randn(T, 2 * I, device=DEV)).to(torch.bfloat16).requires_grad_()
    y = ops.swiglu(gu)
    d = torch.randn_like(y)
    y.backward(d)
    x = gu.detach().double().requires_grad_()
    a, b = x.chunk(2, -1)
    want = torch.nn.functional.silu(a) * b
    want.backward(d.double())
    # one rounding to bf16 each (2^-9 relative)
    assert ((y.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-6).all()
    assert ((gu.grad.double() - x.grad).abs() <= 2 ** -8 * x.grad.abs() + 1e-5).all()


@pytest.mark.parametrize("M,N,K,splits", [(1152, 896, 9600, 3), (136, 128, 4104, 8), (896, 896, 1000, 1), (9728, 896, 4096, 1)])
def test_weight_gradient_splits(M, N, K, splits):
    """Contractions of few tiles are split over the tokens; the sums are added to what the gradient holds."""
    got = dense._grad_splits(M, N, K)
    assert (got > 1) == (splits > 1), got
    torch.manual_seed(0)
    dy, x = (torch.randn(K, n, device=DEV).to(torch.bfloat16) for n in (M, N))
    out = torch.randn(M, N, device=DEV)
    want = out.double() + dy.double().T @ x.double()
    dense._accumulate_weight_grad(dy, x, out)
    lib.check_status()
    assert ((out.double() - want).norm() / want.norm()).item() < 1e-5      # 32-bit sums


@pytest.mark.parametrize("T,N", [(1, 8), (31, 136), (33, 1152), (9000, 4608), (5, 20)])
def test_column_sums(T, N):
    torch.manual_seed(0)
    x = torch.randn(T, N, device=DEV).to(torch.bfloat16)
    out = torch.randn(N, device=DEV)
    want = out.double() + x.double().sum(0)
    torch.testing.assert_close(dense._column_sums(x, out).double(), want, rtol=1e-5, atol=1e-4 * T ** 0.5)
    torch.testing.assert_close(dense._column_sums(x).double(), x.double().sum(0), rtol=1e-5, atol=1e-4 * T ** 0.5)


@pytest.mark.parametrize("T,H", [(1, 8), (700, 896), (595, 1024), (300, 1032), (40, 3584), (2500, 64)])
def test_rmsnorm_backward_widths(T, H):
    """Both block widths, more rows than blocks and fewer."""
    torch.manual_seed(0)
    x, r = (torch.randn(T, H, device=DEV).to(torch.bfloat16).requires_grad_() for _ in range(2))
    w = (1 + 0.1 * torch.randn(H, device=DEV)).to(torch.bfloat16).requires_grad_()
    y, h = ops.rmsnorm(x, w, 1e-6, residual=r)
    gy, gh = torch.randn_like(y), torch.randn_like(h)
    torch.autograd.backward([y, h], [gy, gh])
    hd, wd = h.detach().double().requires_grad_(), w.detach().double().requires_grad_()
    yd = hd * torch.rsqrt(hd.square().mean(-1, keepdim=True) + 1e-6) * wd
    torch.autograd.backward([yd], [gy.double()])
    want = hd.grad + gh.double()
    # one rounding to bf16 (2^-9 relative); the weight's gradient is rounded after a 32-bit sum
    assert ((x.grad.double() - want).norm() / want.norm()).item() < 3e-3 and torch.equal(x.grad, r.grad)
    assert ((w.grad.double() - wd.grad).norm() / wd.grad.norm()).item() < 4e-3


@pytest.mark.parametrize("with_residual", [True, False])
@pytest.mark.parametrize("T,H", [(1, 8), (3, 2048), (2500, 2056), (1300, 3584), (5, 4104), (1200, 8192)])
def test_rmsnorm_forward_widths(T, H, with_residual):
    """Every number of vectors per thread, at its edges, with fewer rows than blocks and more."""
    torch.manual_seed(0)
    x, r = (torch.randn(T, H, device=DEV).to(torch.bfloat16) for _ in range(2))
    w = (1 + 0.1 * torch.randn(H, device=DEV)).to(torch.bfloat16)
    y, h = ops.rmsnorm(x, w, 1e-6, residual=r if with_residual else None)
    if with_residual:
        assert torch.equal(h, (x.float() + r.float()).to(torch.bfloat16))
    want = h.double() * torch.rsqrt(h.double().square().mean(-1, keepdim=True) + 1e-6) * w.double()
    # one rounding to bf16 (2^-9 relative) of a value that 32 bits give to 1e-6
    assert ((y.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-6).all()


@pytest.mark.parametrize("T,I", [(9000, 8), (15000, 1048), (7, 768), (2000, 264), (40, 520)])
def test_swiglu_narrow_rows(T, I):
    """Rows that share a block, rows divided evenly over blocks, and single rows or pairs per thread."""
    test_swiglu_rows(T, I)


def test_refused_launch_leaves_no_error_behind():
    """A launch that the runtime refuses (a grid of 70000 in y) is reported by its own call and by none after it."""
    import ctypes
    logits = torch.zeros(1, 128, device=DEV)
    tok, lp, ws = torch.zeros(1, dtype=torch.int64, device=DEV), torch.zeros(1, device=DEV), torch.zeros(4, device=DEV)
    rc = lib.get_lib().sb_sample(lib.ptr(logits), lib.ptr(logits), ctypes.c_longlong(128), ctypes.c_float(1.0),
                                 ctypes.c_ulonglong(0), ctypes.c_ulonglong(0), None, lib.ptr(tok), lib.ptr(lp), 1, 128,
                                 lib.ptr(ws), 70000, lib.stream())
    assert rc != 0
    assert float((lp + 1).sum()) == 1.0


def test_launch_counter_follows_the_sizes():
    """Calls whose number of kernels depends on the sizes."""
    from siirl_b200.ops import kv_cache as kvc, rl
    from siirl_b200.ops.attention import SeqInfo, attention_packed, bwd_head_splits
    from siirl_b200.ops.sampling import sample

    def launches(fn):
        before = lib.launch_count()
        fn()
        return lib.launch_count() - before
    for rows, want in ((8, 2), (2048, 2), (2049, 4)):
        x, gid = torch.ones(rows, 3, device=DEV), torch.zeros(rows, dtype=torch.int32, device=DEV)
        assert launches(lambda: rl.grpo_group_advantage(x, x, gid, 1)) == want
    for seqlens, hq, want in (([256], 2, 4), ([64] * 300, 2, 3), ([256], 1, 3)):
        assert (bwd_head_splits(seqlens, hq, 1, True) > 1) == (want == 4)
        x = torch.randn(sum(seqlens), (hq + 2) * 64, device=DEV).to(torch.bfloat16).requires_grad_()
        out = attention_packed(x, SeqInfo(seqlens, device=DEV), hq, 1, 64)
        assert launches(lambda: out.backward(torch.ones_like(out))) == want
    q, table = torch.zeros(2, 6 * 64, device=DEV, dtype=torch.bfloat16), torch.arange(34, dtype=torch.int32, device=DEV).reshape(2, 17)
    cache, n = torch.zeros(34, 2, 1, 64, 64, device=DEV, dtype=torch.bfloat16), torch.ones(2, dtype=torch.int32, device=DEV)
    for blocks, want in ((16, 1), (17, 2)):
        t = table[:, :blocks].contiguous()
        assert launches(lambda: kvc.decode_attention(q, cache, n, t, 4, 1, 64)) == want
    for V, want in ((4000, 1), (40000, 2)):
        assert launches(lambda: sample(torch.zeros(2, V, device=DEV))) == want
    cos, sin = ops.rope_tables(24, 8, 10000.0, device=DEV)
    x = torch.zeros(4, 5 * 24, device=DEV, dtype=torch.bfloat16)
    assert launches(lambda: ops.rope(x, 3, 24, torch.arange(4, device=DEV), cos, sin, None)) == 1


def test_column_sums_of_other_layouts():
    """Rows apart and sums kept in another type go through the plain form."""
    torch.manual_seed(0)
    x = torch.randn(300, 64, device=DEV).to(torch.bfloat16)
    want = x.double().sum(0)
    for src, out, tol in ((x, torch.zeros(64, device=DEV, dtype=torch.bfloat16), 2 ** -8),
                          (x, torch.zeros(64, device=DEV, dtype=torch.float64), 1e-5),
                          (torch.cat([x, x], 1)[:, :64], torch.zeros(64, device=DEV), 1e-5),
                          (torch.cat([x, x], 1)[:, :64], None, 1e-5),
                          (x, torch.zeros(64, 2, device=DEV)[:, 0], 1e-5)):
        got = dense._column_sums(src, out)
        assert out is None or got.data_ptr() == out.data_ptr() and got.dtype == out.dtype
        # one rounding to the output's type of a 32-bit sum of 300 numbers
        assert ((got.double() - want).abs() <= tol * (want.abs() + 20)).all()


@pytest.mark.parametrize("clip", [0.0, 0.5])
@pytest.mark.parametrize("n,shift", [(1, 0), (3, 0), (4, 0), (5, 0), (1027, 0), (1030, 1), (64 * 148 * 1024 + 261, 0),
                                     (64 * 148 * 1024 * 2 + 12, 0), (300001, 3)])
def test_adamw_kernel(n, shift, clip):
    """Every element is updated once and none beyond the last: vectors and the rest, pieces of one and of several sweeps,
    blocks without work, and buffers that do not start on 16 bytes."""
    import ctypes
    torch.manual_seed(0)
    guard = 8
    mk = lambda dtype=torch.float32: torch.randn(shift + n + guard, device=DEV).to(dtype)  # noqa: E731
    w, m, v, g, p = mk(), mk(), mk().abs(), mk(), mk(torch.bfloat16)
    sumsq, norm = (torch.zeros(1, device=DEV) for _ in range(2))
    f, at = ctypes.c_float, lambda t: ctypes.c_void_p(t.data_ptr() + shift * t.element_size())
    before = [t.clone() for t in (w, m, v, p)]
    inside = slice(shift, shift + n)
    sumsq += g[inside].double().square().sum().float()
    lr, b1, b2, eps, wd, step, scale = 1e-2, 0.9, 0.99, 1e-8, 0.1, 3, 0.25
    lib.check(lib.get_lib().sb_adamw_step(at(w), at(m), at(v), at(g), at(p), lib.ptr(sumsq), lib.ptr(norm), ctypes.c_longlong(n),
                                          f(lr), f(b1), f(b2), f(eps), f(wd), step, f(clip), f(scale), lib.stream()), "adamw")
    total = sumsq.double().sqrt() * scale
    assert abs(float(norm) / float(total) - 1) < 1e-5
    g64 = g[inside].double() * scale * (min(1.0, clip / (float(total) + 1e-6)) if clip else 1.0)
    m64 = b1 * before[1][inside].double() + (1 - b1) * g64
    v64 = b2 * before[2][inside].double() + (1 - b2) * g64 * g64
    w64 = before[0][inside].double() * (1 - lr * wd) - lr * (m64 / (1 - b1 ** step)) / ((v64 / (1 - b2 ** step)).sqrt() + eps)
    # a handful of 32-bit operations each; one rounding to bf16 of the weight
    for got, want, tol in ((m, m64, 1e-6), (v, v64, 1e-6), (w, w64, 1e-5), (p, w64, 2 ** -8)):
        assert ((got[inside].double() - want).abs() <= tol * want.abs() + 1e-6).all()
    for got, old in zip((w, m, v, p), before):
        assert torch.equal(got[:shift], old[:shift]) and torch.equal(got[shift + n:], old[shift + n:])
