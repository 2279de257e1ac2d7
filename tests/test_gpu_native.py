"""The one-rank C++ autograd node against the Python autograd functions it stands in for."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _randn(*shape, dtype=torch.bfloat16):
    return torch.randn(*shape, device="cuda", dtype=dtype)


def _is_node(t):
    """t came out of the C++ node and not of a Python autograd function."""
    return "CppNode" in t.grad_fn.name()


def _grads(fn, leaves, dout, node):
    leaves = [t.detach().clone().requires_grad_(True) for t in leaves]
    out, lse, _ = fn(*leaves)
    assert _is_node(out) == node, out.grad_fn.name()
    return [out.detach(), lse.detach(), *torch.autograd.grad(out, leaves, dout)]


@pytest.fixture
def general(monkeypatch):
    """Calls inside `with general():` go the Python way."""
    import contextlib
    from sp_aurora_b200 import local_attn

    @contextlib.contextmanager
    def ctx():
        local_attn.KERNEL_TIMERS = {}
        try:
            yield
        finally:
            local_attn.KERNEL_TIMERS = None
    return ctx


@pytest.mark.parametrize("kind", ["no", "kv", "qkv", "ulysses", "zigzag", "varlen", "llama3"])
@pytest.mark.parametrize("dtype,D", [(torch.bfloat16, 128), (torch.float16, 64), (torch.float32, 32)])
def test_same_results_as_the_python_functions(general, kind, dtype, D):
    """Bitwise: the same kernels on the same operands."""
    import sp_aurora_b200 as spa
    torch.manual_seed(3)
    B, S, H, Hk = 2, 300, 4, 2
    kw = dict(causal=True, return_attn_probs=True)
    if kind in ("varlen", "llama3"):
        q, do = _randn(S, H, D, dtype=dtype), _randn(S, H, D, dtype=dtype)
        leaves = [q, _randn(S, Hk, D, dtype=dtype), _randn(S, Hk, D, dtype=dtype)]
        cu = torch.tensor([0, 100, 100, 163, S], dtype=torch.int32)
        if kind == "varlen":
            fn = lambda *x: spa.ring_flash_attn_varlen_func(*x, cu, **kw)
        else:
            cq, ck, mq, mk, ks = spa.llama3_flash_attn_prepare_cu_seqlens(cu, True, 0, 1)
            fn = lambda *x: spa.llama3_flash_attn_varlen_func(*x, cq, ck, mq, mk, heads_k_stride=1,
                                                              local_k_slice=ks, **kw)
    else:
        do = _randn(B, S, H, D, dtype=dtype)
        leaves = {"kv": [_randn(B, S, H, D, dtype=dtype), _randn(B, S, 2, Hk, D, dtype=dtype)],
                  "qkv": [_randn(B, S, 3, H, D, dtype=dtype)]}.get(
                      kind, [_randn(B, S, n, D, dtype=dtype) for n in (H, Hk, Hk)])
        fn = {"no": spa.ring_flash_attn_func, "kv": spa.ring_flash_attn_kvpacked_func,
              "qkv": spa.ring_flash_attn_qkvpacked_func, "ulysses": spa.ulysses_flash_attn_func,
              "zigzag": spa.zigzag_ring_flash_attn_func}[kind]
        fn = (lambda f: lambda *x: f(*x, **kw))(fn)
    a = _grads(fn, leaves, do, node=True)
    with general():
        b = _grads(fn, leaves, do, node=False)
    spa.check_status()
    for x, y in zip(a, b):
        assert x.shape == y.shape and torch.equal(x, y)


def test_node_behaves_like_an_autograd_function():
    """Saved-tensor hooks see the saved tensors, a grad with a stride of 0 works, a second
    backward needs retain_graph, an in-place change of an input is noticed."""
    import sp_aurora_b200 as spa
    q, k, v = (_randn(1, 130, 2, 64).requires_grad_(True) for _ in range(3))
    assert _is_node(spa.select_flash_attn_impl()(q, k, v))
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or t.cpu(), lambda t: t.cuda()):
        out = spa.ring_flash_attn_func(q, k, v, causal=True)
    assert len(packed) == 5
    g1 = torch.autograd.grad(out.sum(), (q, k, v))
    out = spa.ring_flash_attn_func(q, k, v, causal=True)
    g2 = torch.autograd.grad(out, (q, k, v), torch.ones_like(out), retain_graph=True)
    assert all(torch.equal(a, b) for a, b in zip(g1, g2))
    torch.autograd.grad(out, (q,), torch.ones_like(out))
    with pytest.raises(RuntimeError, match="second time|freed"):
        torch.autograd.grad(out, (q,), torch.ones_like(out))
    k2 = k.detach().clone()
    out = spa.ring_flash_attn_func(q, k2, v)
    k2.add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace"):
        out.sum().backward()
    _, lse = spa.select_flash_attn_impl()(q, k, v, return_attn_probs=True)
    assert not lse.requires_grad


def test_what_the_node_leaves_to_the_general_way():
    """Errors keep their types and words; transforms and tangents are not swallowed."""
    import sp_aurora_b200 as spa
    q = _randn(1, 64, 2, 64)
    with pytest.raises(ValueError, match="head_dim"):
        spa.ring_flash_attn_func(_randn(1, 64, 2, 48), _randn(1, 64, 2, 48), _randn(1, 64, 2, 48))
    with pytest.raises(ValueError, match="contiguous in its last"):
        spa.ring_flash_attn_func(q.transpose(1, 3).contiguous().transpose(1, 3), q, q)
    with pytest.raises(spa.SpaError, match="scale"):
        spa.ring_flash_attn_func(q, q, q, softmax_scale=-1.0)
    with pytest.raises(NotImplementedError):
        spa.ring_flash_attn_func(q, q, q, dropout_p=0.5)
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda x: spa.ring_flash_attn_func(x, x, x))(q[None])
    import torch.autograd.forward_ad as fwad
    with fwad.dual_level():
        d = fwad.make_dual(q, torch.ones_like(q))
        with pytest.raises((RuntimeError, NotImplementedError)):
            spa.ring_flash_attn_func(d, q, q)
    bad = _randn(1, 64 * 2 * 64 + 1)[:, 1:].view(1, 64, 2, 64)     # 2-byte aligned
    with pytest.raises(spa.SpaError, match="16 bytes"):
        spa.ring_flash_attn_func(bad, q, q)
    x = q.clone().requires_grad_(True)
    out = spa.ring_flash_attn_func(x, q, q)
    g = _randn(1, 64 * 2 * 64 + 1)[:, 1:].view(1, 64, 2, 64)
    with pytest.raises(spa.SpaError, match="16 bytes"):
        torch.autograd.grad(out, x, g)


@pytest.mark.parametrize("S", [500, 2000])     # 2000: the dK/dV pass starts beside the dQ pass, keys split
def test_forward_and_backward_are_captured_in_a_graph(S):
    import sp_aurora_b200 as spa
    q, k, v, do = (_randn(1, S, 4, 128) for _ in range(4))
    leaves = [t.requires_grad_(True) for t in (q, k, v)]

    def step():
        out = spa.ring_flash_attn_func(*leaves, causal=True)
        return [out.detach(), *torch.autograd.grad(out, leaves, do)]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step()
    with torch.no_grad():
        for t in (q, k, v, do):
            t.copy_(torch.randn_like(t))
    graph.replay()
    want = step()
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("mode", ["ring", "ulysses"])
@pytest.mark.parametrize("rope_base", [None, 10000.0])
def test_block_node_equals_the_sliced_form(general, monkeypatch, mode, rope_base):
    """Rotation, attention and the joined gradient of one projection output. Bitwise: adding the
    zeros of the other slices changes nothing, the rotation is undone from the same 16-bit rows."""
    import sp_aurora_b200 as spa
    torch.manual_seed(4)
    blk = spa.SequenceParallelAttentionBlock(512, 4, 2, mode=mode, device="cuda", rope_base=rope_base)
    x, dy = _randn(2, 129, 512), _randn(2, 129, 512)

    def step():
        t = x.clone().requires_grad_(True)
        y = blk(t, causal=True)
        return [y.detach(), *torch.autograd.grad(y, (t, *blk.parameters()), dy)]
    from sp_aurora_b200 import native
    taken, call = [], native.attention_heads_packed
    monkeypatch.setattr(native, "attention_heads_packed", lambda *x: taken.append(call(*x)) or taken[-1])
    a = step()
    with general():
        b = step()
    assert taken[0] is not None and taken[1] is None     # the node, then the sliced form
    spa.check_status()
    for p, q in zip(a, b):
        assert torch.equal(p, q)


def test_other_modes():
    """inference_mode, create_graph, a dispatch mode and a non-default stream."""
    import sp_aurora_b200 as spa
    from torch.utils._python_dispatch import TorchDispatchMode
    q, kv = _randn(1, 130, 4, 64), _randn(1, 130, 2, 2, 64)
    want = spa.ring_flash_attn_kvpacked_func(q, kv, causal=True)
    with torch.inference_mode():
        assert torch.equal(spa.ring_flash_attn_kvpacked_func(q, kv, causal=True), want)

    class Seen(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))
    with Seen():
        assert torch.equal(spa.ring_flash_attn_kvpacked_func(q, kv, causal=True), want)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        x = q.clone().requires_grad_(True)
        out = spa.ring_flash_attn_kvpacked_func(x, kv, causal=True)
        g, = torch.autograd.grad(out, x, torch.ones_like(out), create_graph=True)
    torch.cuda.current_stream().wait_stream(side)
    y = q.clone().requires_grad_(True)
    h, = torch.autograd.grad(spa.ring_flash_attn_kvpacked_func(y, kv, causal=True), y, torch.ones_like(want))
    assert torch.equal(out, want) and torch.equal(g, h)


@pytest.mark.parametrize("rope_base", [None, 10000.0])
def test_hybrid_block_calls_its_submodule(rope_base):
    """A forward hook on the block's attention module fires, and a module put in its place is used."""
    import sp_aurora_b200 as spa
    blk = spa.SequenceParallelAttentionBlock(512, 4, 2, mode="hybrid", device="cuda", rope_base=rope_base)
    x, seen = _randn(1, 129, 512), []
    handle = blk.hybrid.register_forward_hook(lambda mod, args, out: seen.append(out.shape))
    y = blk(x)
    assert seen == [(1, 129, 4, 128)]
    handle.remove()
    ring = spa.SequenceParallelAttentionBlock(512, 4, 2, mode="ring", device="cuda", rope_base=rope_base)
    ring.load_state_dict(blk.state_dict())
    assert torch.equal(ring(x), y)

    class Zeros(torch.nn.Module):
        def forward(self, q, k, v, causal):
            return torch.zeros_like(q)
    blk.hybrid = Zeros()
    assert (blk(x) == 0).all()
