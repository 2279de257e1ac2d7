"""CTAs that loop over several query blocks: bitwise the results of calls on parts of the batch that
are too small for that (a block goes through the same tiles in the same order either way)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Sq,Sk,H,Hk,D,causal,off,part", [
    (4, 1000, 1000, 32, 8, 128, True, 0, 1),       # ragged, every walk length
    (4, 1024, 2900, 32, 32, 64, False, 0, 1),      # equal walks, odd and even numbers of tiles
    (5, 900, 700, 32, 4, 128, True, -300, 1),      # query tiles without a visible key
    (4, 1100, 1300, 32, 16, 64, True, 150, 1),
    (300, 130, 130, 64, 64, 64, True, 0, 2),       # more items than one CTA per SM may take
])
def test_loop_equals_single_items(B, Sq, Sk, H, Hk, D, causal, off, part):
    import sp_aurora_b200 as spa
    from sp_aurora_b200 import local_attn as la
    g = torch.Generator(device="cuda").manual_seed(9)
    q, do = (torch.randn(B, Sq, H, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    kv = torch.randn(B, Sk, 2, Hk, D, device="cuda", generator=g).bfloat16()

    def call(q, kv, do):
        k, v = kv[:, :, 0], kv[:, :, 1]
        out, dq, dkv = torch.empty_like(q), torch.empty_like(q), torch.empty_like(kv)
        lse = torch.empty(q.shape[0], H, Sq, device="cuda")
        la.attn_fwd_step(q, k, v, D ** -0.5, causal, lse, out=out, causal_off=off)
        la.attn_bwd_step(q, k, v, do, lse, la.bwd_delta(out, do), D ** -0.5, causal, None, dkv[:, :, 0],
                         dkv[:, :, 1], causal_off=off, dq=dq, dq_overwrite=True)
        return out, lse, dq, dkv
    whole = call(q, kv, do)
    for b in range(0, B, part):
        sl = slice(b, b + part)
        for x, y in zip(whole, call(q[sl], kv[sl], do[sl])):
            assert torch.equal(x[sl], y), b
    spa.check_status()


def test_loop_over_packed_sequences():
    """As above for a packed batch: all heads at once against one kv group at a time."""
    import sp_aurora_b200 as spa
    from sp_aurora_b200 import local_attn as la
    lengths = [700, 1, 129, 1500, 256, 300]
    seqs, T = [], 0
    for n in lengths:
        seqs.append((T, n, T, n, 0))
        T += n
    H, Hk, D = 64, 16, 128
    q, do = (torch.randn(T, H, D, device="cuda").half() for _ in range(2))
    k, v = (torch.randn(T, Hk, D, device="cuda").half() for _ in range(2))
    out, lse = la.packed_forward(q, k, v, seqs, D ** -0.5, True)
    dq, dk, dv = la.packed_backward(do, q, k, v, out, lse, seqs, D ** -0.5, True)
    for h in range(Hk):
        hq, hk = slice(4 * h, 4 * h + 4), slice(h, h + 1)
        o, l = la.packed_forward(q[:, hq], k[:, hk], v[:, hk], seqs, D ** -0.5, True)
        g = la.packed_backward(do[:, hq], q[:, hq], k[:, hk], v[:, hk], o, l, seqs, D ** -0.5, True)
        for x, y in zip((out[:, hq], lse[hq], dq[:, hq], dk[:, hk], dv[:, hk]), (o, l, *g)):
            assert torch.equal(x, y), h
    spa.check_status()


@pytest.mark.parametrize("D", [64, 128])
def test_gradients_added_to_16_bit_tensors_beside_the_dq_pass(D):
    """Both passes in one call, 13 key tiles (the dK/dV pass starts beside the dQ pass), dK/dV added
    to element-type tensors: the fp32 gradient plus the old row, rounded once."""
    import sp_aurora_b200 as spa
    from sp_aurora_b200 import local_attn as la
    B, S, H, Hk = 1, 1600, 4, 2
    q, do = (torch.randn(B, S, H, D, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(B, S, Hk, D, device="cuda").bfloat16() for _ in range(2))
    out, lse = spa.flash_attn_forward(q, k, v, None, True)
    delta = la.bwd_delta(out, do)
    dk32, dv32 = (torch.empty(B, S, Hk, D, device="cuda") for _ in range(2))
    dq = torch.empty_like(q)
    la.attn_bwd_step(q, k, v, do, lse, delta, D ** -0.5, True, None, dk32, dv32, dq=dq, dq_overwrite=True,
                     deterministic=True)
    old = torch.randn(B, S, 2, Hk, D, device="cuda").bfloat16()
    dkv = torch.empty_like(old)
    for _ in range(3):                      # the tensors are written again just before each call
        dkv.copy_(old)
        la.attn_bwd_step(q, k, v, do, lse, delta, D ** -0.5, True, None, dkv[:, :, 0], dkv[:, :, 1],
                         dkv_accumulate=True, dq=dq, dq_overwrite=True)
        assert torch.equal(dkv[:, :, 0], (dk32 + old[:, :, 0].float()).bfloat16())
        assert torch.equal(dkv[:, :, 1], (dv32 + old[:, :, 1].float()).bfloat16())
    spa.check_status()


@pytest.mark.parametrize("off", [0, -300])       # -300: query tiles without a visible key
@pytest.mark.parametrize("overwrite", [False, True])
@pytest.mark.parametrize("with_dq", [False, True])
def test_loop_over_a_running_sum(off, overwrite, with_dq):
    """A ring step's form of the dQ pass (fp32 sum in and out): bitwise the calls on one batch
    entry, which have too few query tiles to loop."""
    import sp_aurora_b200 as spa
    from sp_aurora_b200 import _lib, local_attn as la
    B, Sq, Sk, H, Hk, D = 5, 900, 700, 32, 4, 128
    g = torch.Generator(device="cuda").manual_seed(13)
    q, do = (torch.randn(B, Sq, H, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    k, v = (torch.randn(B, Sk, Hk, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    acc0 = torch.randn(B, Sq, H, D, device="cuda", generator=g)
    out, lse = torch.empty_like(q), torch.empty(B, H, Sq, device="cuda")
    la.attn_fwd_step(q, k, v, D ** -0.5, True, lse, out=out, causal_off=off)
    delta = la.bwd_delta(out, do)

    def call(sl):
        acc = acc0[sl].clone()
        dq = torch.zeros_like(q[sl]) if with_dq else None
        la.attn_bwd_step(q[sl], k[sl], v[sl], do[sl], lse[sl], delta[sl], D ** -0.5, True, acc, None, None,
                         causal_off=off, dq=dq, dq_overwrite=overwrite, passes=_lib.SPA_BWD_DQ_ONLY)
        return acc, dq
    acc, dq = call(slice(0, B))
    for b in range(B):
        a, d = call(slice(b, b + 1))
        assert torch.equal(acc[b:b + 1], a), b
        assert d is None or torch.equal(dq[b:b + 1], d), b
    spa.check_status()
    if off and not overwrite:
        assert torch.equal(acc[:, :300], acc0[:, :300])      # rows that see nothing keep their sum
