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
