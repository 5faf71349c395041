"""RL post-processing kernels against the PyTorch statements of the same formulas."""
import types

import pytest
import torch

from siirl_b200.dag_worker import core_algos as A
from siirl_b200.ops import rl

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _mask(B, R):
    lens = torch.randint(1, R + 1, (B,))
    m = (torch.arange(R)[None, :] < lens[:, None]).float()
    m[0, 3:7] = 0  # a hole inside a response (multi-turn style)
    return m


def test_gae_scan_matches_loop():
    torch.manual_seed(0)
    B, R = 37, 301
    r, v, m = torch.randn(B, R), torch.randn(B, R), _mask(B, R)
    adv_ref, ret_ref = rl.gae_scan_reference(r, v, m, 0.99, 0.95)
    adv, ret = rl.gae_scan(r.to(DEV), v.to(DEV), m.to(DEV), 0.99, 0.95)
    torch.testing.assert_close(adv.cpu(), adv_ref, rtol=1e-4, atol=1e-4)
    torch.testing.assert_close(ret.cpu(), ret_ref, rtol=1e-4, atol=1e-4)


def test_grpo_group_adv_matches_formula():
    torch.manual_seed(1)
    B, R, G = 48, 64, 13
    rewards = torch.zeros(B, R)
    m = _mask(B, R)
    rewards[torch.arange(B), (m.sum(-1) - 1).long().clamp(min=0)] = torch.rand(B)
    gid = torch.randint(0, G, (B,))
    gid[0] = G - 1
    gid[1:][gid[1:] == G - 1] = 0  # make one singleton group
    want, _ = A.compute_grpo_outcome_advantage(rewards, m, gid)
    got = rl.grpo_group_advantage(rewards.to(DEV), m.to(DEV), gid.to(DEV), G)
    torch.testing.assert_close(got.cpu(), want, rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("B,R,G", [(1, 1, 1), (2048, 5, 300), (2049, 5, 300), (9, 2100, 2)])
def test_grpo_group_adv_sizes(B, R, G):
    """Both forms of the group statistics (rows up to and above the scan's limit) and more columns than one sweep."""
    g = torch.Generator().manual_seed(3)
    rewards, m = torch.randn(B, R, generator=g), (torch.rand(B, R, generator=g) < 0.7).float()
    gid = torch.randint(0, G, (B,), generator=g)
    s = rewards.double().sum(-1)
    want = torch.zeros(B, dtype=torch.float64)
    for k in range(G):
        at = gid == k
        one = int(at.sum()) == 1
        want[at] = (s[at] - (0.0 if one else s[at].mean())) / ((1.0 if one else s[at].std()) + 1e-6)
    got = rl.grpo_group_advantage(rewards.to(DEV), m.to(DEV), gid.to(DEV), G)
    # groups of two close scores divide small differences of 32-bit sums
    torch.testing.assert_close(got.cpu().double(), want[:, None] * m, rtol=1e-3, atol=1e-4)


@pytest.mark.parametrize("B,R", [(1, 1), (3, 257), (1200, 33), (2, 5000)])
def test_ppo_loss_sizes(B, R):
    """One token, rows and columns beyond one sweep of the grid; every token against 64 bits."""
    torch.manual_seed(4)
    m = (torch.rand(B, R, device=DEV) < 0.8).float()
    m[:, 0] = 1
    old, adv = -torch.rand(B, R, device=DEV) * 3, torch.randn(B, R, device=DEV)
    logp = (old + 0.3 * torch.randn(B, R, device=DEV)).requires_grad_()
    loss, met = rl.ppo_token_loss(logp, old, adv, m, mode="gspo")
    loss.backward()
    lp = logp.detach().double().requires_grad_()
    mean = (((lp - old) * m).sum(-1) / m.sum(-1)).detach()
    ratio = torch.exp(mean[:, None] + lp - lp.detach())
    pg = torch.maximum(-adv * ratio, -adv * ratio.clamp(0.8, 1.2))
    want = ((pg * m).sum(-1) / m.sum(-1)).mean()
    want.backward()
    torch.testing.assert_close(loss.double(), want, rtol=1e-4, atol=1e-5)
    # ratios at the clip's edge apart, gradients agree to 32-bit rounding
    near = ((ratio.detach() - 0.8).abs() < 1e-5) | ((ratio.detach() - 1.2).abs() < 1e-5)
    assert ((logp.grad.double() - lp.grad).abs() * ~near).max() <= 1e-4 * lp.grad.abs().max() + 1e-9
    torch.testing.assert_close(met["pg_loss"].double(), want.detach(), rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("mode", ["vanilla", "gspo", "cpgd"])
@pytest.mark.parametrize("agg", ["token-mean", "seq-mean-token-sum", "seq-mean-token-mean", "seq-mean-token-sum-norm"])
def test_fused_ppo_loss_matches_torch(mode, agg):
    torch.manual_seed(2)
    B, R = 16, 50
    m = _mask(B, R).to(DEV)
    old = (-torch.rand(B, R) * 3).to(DEV)
    logp = (old + 0.3 * torch.randn(B, R, device=DEV)).requires_grad_()
    ref_lp = old + 0.2 * torch.randn(B, R, device=DEV)
    adv = torch.randn(B, R, device=DEV)
    ent = torch.rand(B, R, device=DEV).requires_grad_()
    cfg = types.SimpleNamespace(clip_ratio=0.2, clip_ratio_low=0.2, clip_ratio_high=0.28, clip_ratio_c=3.0)
    loss, met = rl.ppo_token_loss(logp, old, adv, m, entropy=ent, ref_logp=ref_lp, mode=mode, loss_agg_mode=agg,
                                  clip_lo=0.2, clip_hi=0.28, clip_c=3.0, kl_kind="low_var_kl", kl_coef=0.01,
                                  entropy_coef=0.001)
    loss.backward()
    lp2 = logp.detach().clone().requires_grad_()
    ent2 = ent.detach().clone().requires_grad_()
    fn = A.get_policy_loss_fn(mode)
    pg, clipfrac, ppo_kl, clip_lower = fn(old, lp2, adv, m, agg, cfg)
    agg_eff = "seq-mean-token-mean" if mode == "gspo" else agg
    kl = A.agg_loss(A.kl_penalty(lp2, ref_lp, "low_var_kl"), m, agg_eff)
    el = A.agg_loss(ent2, m, agg_eff)
    total = pg + 0.01 * kl - 0.001 * el
    total.backward()
    torch.testing.assert_close(loss.detach(), total.detach(), rtol=1e-4, atol=1e-5)
    torch.testing.assert_close(met["pg_loss"], pg.detach(), rtol=1e-4, atol=1e-5)
    torch.testing.assert_close(met["pg_clipfrac"], clipfrac.detach(), rtol=1e-4, atol=1e-5)
    torch.testing.assert_close(met["ppo_kl"], ppo_kl.detach(), rtol=1e-4, atol=1e-5)
    torch.testing.assert_close(logp.grad, lp2.grad, rtol=1e-3, atol=1e-6)
    torch.testing.assert_close(ent.grad, ent2.grad, rtol=1e-4, atol=1e-7)


@pytest.mark.parametrize("B,R,G", [(2048, 3000, 300), (700, 2100, 90), (1185, 257, 1185)])
def test_grpo_group_adv_many_rows(B, R, G):
    """One block per row, each with many columns, and two."""
    test_grpo_group_adv_sizes(B, R, G)
