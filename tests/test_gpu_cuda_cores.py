"""Tile edges of the CUDA-core kernels (64-row tiles, 4 or 8 rows per thread)."""
import pytest
import torch

from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Sq,Sk", [(1, 1), (63, 65), (64, 64), (65, 129), (200, 130)])
@pytest.mark.parametrize("D,causal,off", [(32, True, 0), (64, True, -70), (128, False, 0), (128, True, 60)])
def test_fp32_tiles_match_the_oracle(Sq, Sk, D, causal, off):
    """fp32 sums of at most 200 terms of unit size: 1e-5 is a hundred roundings."""
    import sp_aurora_b200 as spa
    from sp_aurora_b200 import local_attn as la
    B, Hq, Hkv = 2, 4, 2
    g = torch.Generator().manual_seed(5)
    q, do = (torch.randn(B, Sq, Hq, D, generator=g) for _ in range(2))
    kv = torch.randn(B, Sk, 2, Hkv, D, generator=g)
    qc, doc, kvc = q.cuda(), do.cuda(), kv.cuda()
    kc, vc = kvc[:, :, 0], kvc[:, :, 1]
    scale = D ** -0.5
    out, lse = torch.empty_like(qc), torch.empty(B, Hq, Sq, device="cuda")
    la.attn_fwd_step(qc, kc, vc, scale, causal, lse, out=out, causal_off=off)
    dq, dkv = torch.empty_like(qc), torch.empty_like(kvc)
    la.attn_bwd_step(qc, kc, vc, doc, lse, la.bwd_delta(out, doc), scale, causal, None, dkv[:, :, 0], dkv[:, :, 1],
                     causal_off=off, dq=dq, dq_overwrite=True)
    spa.check_status()
    # plain reference in 64 bits, rows without a visible key give zeros
    qd, kd, vd, dd = (t.double().transpose(1, 2) for t in (q, kv[:, :, 0], kv[:, :, 1], do))
    kd, vd = (t.repeat_interleave(Hq // Hkv, 1) for t in (kd, vd))
    qd, kd, vd = (t.requires_grad_(True) for t in (qd, kd, vd))
    s = scale * qd @ kd.transpose(2, 3)
    seen = torch.ones(Sq, Sk, dtype=torch.bool)
    if causal:
        seen = torch.arange(Sk)[None] <= torch.arange(Sq)[:, None] + off
    any_key = seen.any(1)[:, None]
    p = torch.softmax(s.masked_fill(~seen & any_key, -torch.inf), -1) * any_key
    o = p @ vd
    gq, gk, gv = torch.autograd.grad(o, (qd, kd, vd), dd)
    gk, gv = (t.view(B, Hkv, Hq // Hkv, Sk, D).sum(2) for t in (gk, gv))
    for got, want in ((out, o), (dq, gq), (dkv[:, :, 0], gk), (dkv[:, :, 1], gv)):
        assert (got.cpu().double().transpose(1, 2) - want).abs().max() <= 1e-5 * max(1.0, want.abs().max().item())


def _forward(q, k, v, causal, off=0, scale=None, **kw):
    from sp_aurora_b200 import local_attn as la
    out = torch.empty_like(q)
    lse = kw.pop("lse", None)
    if lse is None:
        lse = torch.empty(q.shape[0], q.shape[2], q.shape[1], device="cuda")
    la.attn_fwd_step(q, k, v, scale or q.shape[-1] ** -0.5, causal, lse, out=out, causal_off=off, **kw)
    return out, lse


@pytest.mark.parametrize("D,dtype", [(32, torch.bfloat16), (64, torch.float32), (128, torch.float32)])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_rows_without_a_visible_key_ignore_the_values(D, dtype, bad):
    """Query i sees the keys up to i - 10: rows 0-9 give zeros, or keep what they held, whatever is
    in V. A NaN in q stays visible in its own row."""
    q, k, v = (torch.randn(1, 64, 2, D, device="cuda").to(dtype) for _ in range(3))
    v[:, 20] = bad
    q[:, 60] = float("nan")
    out, lse = _forward(q, k, v, True, -10)
    assert (out[:, :10] == 0).all() and torch.isneginf(lse[:, :, :10]).all()
    assert out[:, 60].isnan().all() and torch.isfinite(lse[:, :, 10:60]).all()
    acc, old = torch.randn(1, 64, 2, D, device="cuda"), torch.randn(1, 2, 64, device="cuda")
    acc2, lse2 = acc.clone(), old.clone()
    _forward(q, k, v, True, -10, lse=lse2, out_acc=acc2, merge_prev=True)
    assert torch.equal(acc2[:, :10], acc[:, :10]) and torch.equal(lse2[..., :10], old[..., :10])


@pytest.mark.parametrize("D,dtype", [(32, torch.float16), (64, torch.float32)])
def test_keys_and_queries_outside_a_block_s_range_stay_outside(D, dtype):
    """Infinities in keys that no query of a block sees, and in queries that see no key of a block,
    leave the block's results as they are (the masked weight is 0, but 0 * Inf is not)."""
    from sp_aurora_b200 import local_attn as la
    inf = float("inf")

    def grads(q, k, v, do, off):
        out, lse = _forward(q, k, v, True, off)
        dq, dk, dv = (torch.empty_like(t) for t in (q, k, v))
        la.attn_bwd_step(q, k, v, do, lse, la.bwd_delta(out, do), D ** -0.5, True, None, dk, dv, causal_off=off,
                         dq=dq, dq_overwrite=True)
        return out, lse, dq, dk, dv
    # 20 queries see the keys 0-19; key 40 is in the same tile
    q, do = (torch.randn(1, 20, 2, D, device="cuda").to(dtype) for _ in range(2))
    k, v = (torch.randn(1, 64, 2, D, device="cuda").to(dtype) for _ in range(2))
    want = grads(q, k, v, do, 0)
    k[:, 40], v[:, 40] = inf, inf
    got = grads(q, k, v, do, 0)
    for a, b in zip(got[:3], want[:3]):
        assert torch.equal(a, b)
    for a, b in zip(got[3:], want[3:]):
        assert torch.equal(a[:, :40], b[:, :40]) and torch.equal(a[:, 41:], b[:, 41:])
    # query i sees the keys up to i - 40: the keys from 64 on are seen from query 104 on
    q, k, v, do = (torch.randn(1, 128, 2, D, device="cuda").to(dtype) for _ in range(4))
    want = grads(q, k, v, do, -40)
    do[:, 70], q[:, 80] = inf, inf
    got = grads(q, k, v, do, -40)
    for a, b in zip(got[3:], want[3:]):
        assert torch.equal(a[:, 64:], b[:, 64:])


def test_scores_at_head_dim_32_are_summed_in_four_chains():
    """One key, scale 1: lse is the bare score q . k. Its error against 64 bits is that of four
    chains of 8 multiply-adds joined by three additions (two chains of 16: 20 % more). 65536
    scores put the ratio of the two root mean squares within 1 %."""
    g = torch.Generator().manual_seed(21)
    q, k = torch.randn(256, 64, 4, 32, generator=g), torch.randn(256, 1, 4, 32, generator=g)
    _, lse = _forward(q.cuda(), k.cuda(), k.cuda(), False, scale=1.0)
    exact = (q.double() * k.double()).sum(-1).transpose(1, 2)
    chains = [torch.zeros(exact.shape) for _ in range(4)]
    prod = (q.double() * k.double()).transpose(1, 2)      # exact: 48 bits
    for e in range(32):
        c = 2 * (e // 16) + e % 2
        chains[c] = (chains[c].double() + prod[..., e]).float()
    four = (chains[0] + chains[1]) + (chains[2] + chains[3])
    rms = lambda x: (x.double() - exact).square().mean().sqrt().item()
    assert rms(lse.cpu()) <= 1.03 * rms(four)
