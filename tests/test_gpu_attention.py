"""tcgen05 varlen attention forward/backward against an eager fp32 statement."""
import math

import pytest
import torch

from siirl_b200.ops import lib, reference as ref
from siirl_b200.ops.attention import SeqInfo, attention_packed, bwd_head_splits, bwd_ordered, fwd_tile_rows

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rel(a, b):
    return ((a.float() - b.float()).norm() / (b.float().norm() + 1e-12)).item()


def _ref(qkv, seqlens, hq, hkv, d, causal):
    T = qkv.shape[0]
    x = qkv.detach().float().requires_grad_()
    q, k, v = x.split([hq * d, hkv * d, hkv * d], dim=-1)
    out = ref.attention_varlen(q.reshape(T, hq, d), k.reshape(T, hkv, d), v.reshape(T, hkv, d),
                               torch.tensor([0] + list(torch.tensor(seqlens).cumsum(0))), causal=causal,
                               scale=1.0 / math.sqrt(d))
    return x, out.reshape(T, hq * d)


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("cfg", [
    (128, 4, 2, [128]),
    (128, 4, 2, [64, 200, 37, 300]),
    (64, 4, 4, [100, 129, 256]),
    (128, 7, 1, [513, 90]),
    (32, 4, 2, [40, 77]),
    (128, 4, 2, [1024, 384]),
    (64, 2, 2, [257]),
])
def test_attention_fwd_bwd(cfg, causal):
    d, hq, hkv, seqlens = cfg
    torch.manual_seed(0)
    T = sum(seqlens)
    qkv = (0.5 * torch.randn(T, (hq + 2 * hkv) * d, device=DEV)).to(torch.bfloat16).requires_grad_()
    info = SeqInfo(seqlens, device=DEV)
    out = attention_packed(qkv, info, hq, hkv, d, causal=causal)
    lib.check_status()
    xr, outr = _ref(qkv, seqlens, hq, hkv, d, causal)
    assert _rel(out, outr) < 2e-2
    g = torch.randn_like(out)
    out.backward(g)
    lib.check_status()
    outr.backward(g.float())
    hq_w, hk_w = hq * d, hkv * d
    assert _rel(qkv.grad[:, :hq_w], xr.grad[:, :hq_w]) < 3e-2
    assert _rel(qkv.grad[:, hq_w:hq_w + hk_w], xr.grad[:, hq_w:hq_w + hk_w]) < 3e-2
    assert _rel(qkv.grad[:, hq_w + hk_w:], xr.grad[:, hq_w + hk_w:]) < 3e-2
    # element-wise bounds as well: a Frobenius norm hides a wrong row or column (bf16 rounding of O(1) values is
    # ~4e-3; gradients are sums of a few hundred such terms)
    assert (out.float() - outr).abs().max().item() < 3e-2
    gmax = xr.grad.abs().max().item()
    assert (qkv.grad.float() - xr.grad).abs().max().item() < 4e-2 * max(gmax, 1.0)
    # per-row check: no single token's gradient is off
    row_err = (qkv.grad.float() - xr.grad).norm(dim=1) / (xr.grad.norm(dim=1) + 1e-3)
    assert row_err.max().item() < 0.1, row_err.argmax().item()


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("d,hq,hkv,scale,gain", [(128, 4, 2, None, 0.5), (64, 7, 1, None, 0.5), (128, 2, 2, -0.11, 0.5),
                                                 (64, 2, 1, 0.0, 0.5), (128, 2, 1, None, 4.0), (64, 2, 2, None, 4.0)])
def test_attention_fwd_tiles(d, hq, hkv, scale, gain, causal):
    """Sequences around the tile sizes (128 keys, 256 rows), more key tiles than the ring has stages, scales of either
    sign, and scores so far apart that the running maximum moves and the output so far is scaled."""
    seqlens = [1, 127, 128, 129, 255, 256, 257, 385, 1500, 2]
    torch.manual_seed(1)
    T = sum(seqlens)
    scale = scale if scale is not None else 1.0 / math.sqrt(d)
    qkv = (gain * torch.randn(T, (hq + 2 * hkv) * d, device=DEV)).to(torch.bfloat16)
    out = attention_packed(qkv, SeqInfo(seqlens, device=DEV), hq, hkv, d, causal=causal, scale=scale)
    lib.check_status()
    q, k, v = qkv.float().split([hq * d, hkv * d, hkv * d], dim=-1)
    want = ref.attention_varlen(q.reshape(T, hq, d), k.reshape(T, hkv, d), v.reshape(T, hkv, d),
                                torch.tensor([0] + list(torch.tensor(seqlens).cumsum(0))), causal=causal,
                                scale=scale).reshape(T, hq * d)
    # weights and outputs are rounded to bf16 (2^-9 each, relative): 1e-2 of a row leaves a factor of two and a half
    row_err = (out.float() - want).norm(dim=1) / want.norm(dim=1)
    assert row_err.max().item() < 1e-2, row_err.argmax().item()


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("d,hq,hkv,seqlens,scale", [(128, 4, 2, [1, 127, 128, 64, 65, 63, 129, 2], None),
                                                    (64, 7, 1, [1, 127, 128, 64, 65, 63, 129, 2], -0.2),
                                                    (128, 4, 1, [129, 385, 256, 257, 512] * 12, None), (64, 2, 2, [20] * 40 + [1500], 0.0)])
def test_attention_fwd_short_sequences(d, hq, hkv, seqlens, scale, causal):
    """The form with one query tile of 128 rows: sequences around its tiles and more key tiles than the ring has stages."""
    torch.manual_seed(1)
    T = sum(seqlens)
    assert fwd_tile_rows(len(seqlens), T, hq, d) == 128
    scale = scale if scale is not None else 1.0 / math.sqrt(d)
    qkv = (0.7 * torch.randn(T, (hq + 2 * hkv) * d, device=DEV)).to(torch.bfloat16)
    out = attention_packed(qkv, SeqInfo(seqlens, device=DEV), hq, hkv, d, causal=causal, scale=scale)
    lib.check_status()
    q, k, v = qkv.float().split([hq * d, hkv * d, hkv * d], dim=-1)
    want = ref.attention_varlen(q.reshape(T, hq, d), k.reshape(T, hkv, d), v.reshape(T, hkv, d),
                                torch.tensor([0] + list(torch.tensor(seqlens).cumsum(0))), causal=causal,
                                scale=scale).reshape(T, hq * d)
    # weights and outputs are rounded to bf16 (2^-9 each, relative): 1e-2 of a row leaves a factor of two and a half
    row_err = (out.float() - want).norm(dim=1) / want.norm(dim=1)
    assert row_err.max().item() < 1e-2, row_err.argmax().item()


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("d,hq,hkv,repeat,splits", [(128, 3, 1, 1, 3), (64, 4, 2, 1, 2), (128, 2, 1, 80, 1), (64, 6, 2, 80, 1)])
def test_attention_bwd_tiles(d, hq, hkv, repeat, splits, causal):
    """Sequences around the 128-row tiles with the heads of a group in one block and divided over several."""
    seqlens = [1, 127, 128, 129, 257] * repeat + [385]
    assert bwd_head_splits(seqlens, hq, hkv, causal) == splits
    torch.manual_seed(2)
    T, tail = sum(seqlens), sum(seqlens[-6:])
    scale = 1.0 / math.sqrt(d)
    qkv = (0.7 * torch.randn(T, (hq + 2 * hkv) * d, device=DEV)).to(torch.bfloat16).requires_grad_()
    out = attention_packed(qkv, SeqInfo(seqlens, device=DEV), hq, hkv, d, causal=causal)
    g = torch.randn_like(out)
    out.backward(g)
    lib.check_status()
    x = qkv.detach()[-tail:].float().requires_grad_()       # the last sequences stand for all
    q, k, v = x.split([hq * d, hkv * d, hkv * d], dim=-1)
    want = ref.attention_varlen(q.reshape(tail, hq, d), k.reshape(tail, hkv, d), v.reshape(tail, hkv, d),
                                torch.tensor([0] + list(torch.tensor(seqlens[-6:]).cumsum(0))), causal=causal,
                                scale=scale).reshape(tail, hq * d)
    want.backward(g[-tail:].float())
    got = qkv.grad[-tail:].float()
    for a, b in ((0, hq * d), (hq * d, (hq + hkv) * d), ((hq + hkv) * d, None)):
        # P, dS and the results are rounded to bf16 (2^-9 each): 2.5e-3 measured over these sizes, four times that allowed
        assert _rel(got[:, a:b], x.grad[:, a:b]) < 1e-2
    assert torch.isfinite(qkv.grad.float()).all()


@pytest.mark.parametrize("d,hq,hkv,seqlens,causal", [
    (64, 14, 2, [904, 1232, 33, 568], True), (128, 6, 2, [1500, 130], True), (64, 4, 4, [600] * 80, True),
    (128, 7, 1, [4000], True), (64, 14, 2, [4097, 129], True), (128, 28, 4, [300, 500, 1550], False)])
def test_attention_bwd_repeats_itself(d, hq, hkv, seqlens, causal):
    """Equal inputs give equal gradients, bit by bit, however the blocks are scheduled: with the heads of a group in one
    block and divided, fewer blocks than SMs and several waves, alone and beside other work.  Causal sequences of up to
    64 d rows do so by themselves, the last two cases when torch asks for it."""
    torch.manual_seed(3)
    T = sum(seqlens)
    assert bwd_ordered(max(seqlens), d, causal) == (causal and max(seqlens) <= 4096)
    info = SeqInfo(seqlens, device=DEV)
    qkv = torch.randn(T, (hq + 2 * hkv) * d, device=DEV).to(torch.bfloat16).requires_grad_()
    out = attention_packed(qkv, info, hq, hkv, d, causal=causal)
    g = torch.randn_like(out)
    side, busy = torch.cuda.Stream(), torch.randn(1 << 22, device=DEV)
    torch.use_deterministic_algorithms(not bwd_ordered(max(seqlens), d, causal))
    try:
        want, = torch.autograd.grad(out, qkv, g, retain_graph=True)
        for i in range(6):
            if i % 2:
                side.wait_stream(torch.cuda.current_stream())
                with torch.cuda.stream(side):
                    for _ in range(20):
                        busy.mul_(1.0)
            got, = torch.autograd.grad(out, qkv, g, retain_graph=True)
            assert torch.equal(got, want), i
    finally:
        torch.use_deterministic_algorithms(False)
    torch.cuda.synchronize()
    lib.check_status()
    # the same sums in the other order: fp32 rounding moves a few results to the next bf16 number
    torch.testing.assert_close(want, _other_order(qkv, info, out, g, hq, hkv, d, causal), rtol=2 ** -6, atol=1e-3)


def _other_order(qkv, info, out, g, hq, hkv, d, causal):
    """The gradient with one block per kv head and unordered sums of dQ."""
    from siirl_b200.ops import attention as att
    keep = att.bwd_ordered, att.bwd_head_splits
    att.bwd_ordered, att.bwd_head_splits = lambda *a: False, lambda *a: 1
    try:
        return torch.autograd.grad(out, qkv, g)[0]
    finally:
        att.bwd_ordered, att.bwd_head_splits = keep
