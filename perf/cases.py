"""The calls whose speed this package answers for: attention on one GPU through its public
entry points, at the sizes its users have.

A case is a dict of plain values. `entry` names the public function:

  ring     ring_flash_attn_func / _kvpacked_func / _qkvpacked_func (`pack`: "no", "kv", "qkv")
  ulysses  ulysses_flash_attn_func
  hybrid   LongContextAttentionQKVPacked
  varlen   ring_flash_attn_varlen_func on packed sequences (`lengths`)
  packed   llama3_flash_attn_varlen_func on a packed stream (`lengths`)
  local    the function select_flash_attn_impl hands out, queries and keys of different length
  block    SequenceParallelAttentionBlock (projection, rotary embedding, attention, projection)

With `train` the pass is a forward and a backward and gives the output and every gradient;
without it the pass is an inference forward that gives the output and, where the entry point
returns it, the log-sum-exp.
"""
import math
import random

import torch

import sp_aurora_b200 as spa

_DTYPE = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def listed():
    return [
        # One short prompt through the ring entry point: launches and host time are all there is.
        dict(name="infer_short", entry="ring", pack="no", B=1, S=512, Hq=4, Hkv=2, D=128, dtype="bf16",
             causal=True, train=False),
        # A small model's training step, head_dim 64.
        dict(name="train_small", entry="ring", pack="no", B=2, S=1024, Hq=8, Hkv=8, D=64, dtype="fp16",
             causal=True, train=True),
        # The fp32 parity configuration (B=2, S=1024, H=32, D=64): what a port is validated with.
        dict(name="fp32_anchor", entry="ring", pack="no", B=2, S=1024, Hq=32, Hkv=32, D=64, dtype="fp32",
             causal=True, train=True),
        # Short sequences packed back to back, the shapes of the varlen tests.
        dict(name="varlen_short", entry="varlen", lengths="64,128,256,512", Hq=8, Hkv=8, D=64, dtype="fp16",
             causal=True, train=True),
        # Documents of mixed length packed into one stream, as the transformers adapter trains on
        # them (one kv head gathered at a time, its default).
        dict(name="packed_docs", entry="packed", lengths="1210,3877,96,2048,517,4501,1366,2769", stride=1,
             Hq=32, Hkv=8, D=128, dtype="bf16", causal=True, train=True),
        # A batch of ordinary length that no tile size divides, grouped-query heads.
        dict(name="train_ragged", entry="ring", pack="kv", B=2, S=3001, Hq=32, Hkv=8, D=128, dtype="bf16",
             causal=True, train=True),
        # A short block of queries over a long context (cross attention, a chunk of a long prompt).
        dict(name="short_query", entry="local", B=2, Sq=128, Sk=16384, Hq=32, Hkv=8, D=128, dtype="bf16",
             causal=False, train=False),
        # A transformer layer's attention block with rotary embedding.
        dict(name="block_rope", entry="block", B=1, S=8192, d_model=4096, Hq=32, Hkv=8, D=128, dtype="bf16",
             causal=True, train=True),
        # The long-context training configuration with as many kv heads as query heads.
        dict(name="train_32k", entry="ring", pack="no", B=1, S=32768, Hq=32, Hkv=32, D=128, dtype="bf16",
             causal=True, train=True),
        # Inference prefill of the hybrid configuration with the log-sum-exp returned.
        dict(name="prefill_64k", entry="hybrid", B=1, S=65536, Hq=16, Hkv=16, D=128, dtype="bf16",
             causal=True, train=False),
        # One GPU's heads of the Ulysses configuration: full sequence, 4 of 32 heads, no mask.
        dict(name="ulysses_64k", entry="ulysses", B=2, S=65536, Hq=4, Hkv=4, D=128, dtype="bf16",
             causal=False, train=True),
        # The headline configuration: grouped-query, kv-packed, 128k tokens.
        dict(name="train_128k", entry="ring", pack="kv", B=1, S=131072, Hq=32, Hkv=8, D=128, dtype="bf16",
             causal=True, train=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _most(case, name, lo, flops):
    """Halve case[name] until the pass needs no more than `flops`."""
    while case[name] > lo and work(case)["flops"] > flops:
        case[name] = max(lo, case[name] // 2)
    return case


def draw(rng: random.Random):
    entry = rng.choice(["ring", "ring", "ring", "ring", "fp32", "varlen", "packed", "local", "block", "hybrid",
                        "ulysses"])
    D = rng.choice([64, 128, 128])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    heads = rng.choice([(4, 2), (8, 8), (16, 16), (32, 8), (32, 32)])
    if entry == "fp32":
        Hq, Hkv = rng.choice([(4, 2), (8, 8), (32, 32)])
        return _most(dict(entry="ring", pack="no", B=rng.choice([1, 2]), S=_log(rng, 64, 3000), Hq=Hq, Hkv=Hkv,
                          D=rng.choice([32, 64, 128]), dtype="fp32", causal=rng.random() < 0.7,
                          train=rng.random() < 0.7), "S", 64, 2e11)
    if entry in ("varlen", "packed"):
        n = rng.randint(2, 12)
        top = rng.choice([512, 2048, 6000])
        lengths = [_log(rng, 48, top) for _ in range(n)]
        Hq, Hkv = heads
        case = dict(entry=entry, lengths=",".join(str(x) for x in lengths), Hq=Hq, Hkv=Hkv, D=D, dtype=dtype,
                    causal=True, train=rng.random() < 0.8)
        if entry == "packed":
            case["stride"] = rng.choice([1, Hkv])
        return case
    if entry == "local":
        Hq, Hkv = heads
        return dict(entry="local", B=rng.choice([1, 2, 4]), Sq=_log(rng, 1, 2048), Sk=_log(rng, 500, 32768), Hq=Hq,
                    Hkv=Hkv, D=D, dtype=dtype, causal=False, train=False)
    if entry == "block":
        d_model, Hq, Hkv = rng.choice([(512, 4, 2), (2048, 16, 4), (4096, 32, 8)])
        return dict(entry="block", B=rng.choice([1, 2]), S=_log(rng, 300, 8192), d_model=d_model, Hq=Hq, Hkv=Hkv,
                    D=128, dtype="bf16", causal=True, train=True)
    if entry == "hybrid":
        H = rng.choice([4, 8, 16])
        return dict(entry="hybrid", B=1, S=_log(rng, 1024, 65536), Hq=H, Hkv=H, D=D, dtype=dtype, causal=True,
                    train=False)
    if entry == "ulysses":
        H = rng.choice([4, 8])
        return _most(dict(entry="ulysses", B=rng.choice([1, 2]), S=_log(rng, 256, 65536), Hq=H, Hkv=H, D=D,
                          dtype=dtype, causal=rng.random() < 0.5, train=rng.random() < 0.8), "S", 256, 6e13)
    Hq, Hkv = heads
    pack = rng.choice(["no", "kv", "qkv"] if Hq == Hkv else ["no", "kv"])
    return _most(dict(entry="ring", pack=pack, B=rng.choice([1, 1, 2]), S=_log(rng, 100, 131072), Hq=Hq, Hkv=Hkv,
                      D=D, dtype=dtype, causal=rng.random() < 0.75, train=rng.random() < 0.75), "S", 100, 1.5e14)


def _lengths(case):
    return [int(x) for x in case["lengths"].split(",")]


def _randn(shape, case, gen, sigma=1.0):
    return torch.randn(shape, dtype=_DTYPE[case["dtype"]], device="cuda", generator=gen).mul_(sigma)


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    Hq, Hkv, D, entry, train = case["Hq"], case["Hkv"], case["D"], case["entry"], case["train"]
    st = {"case": case}
    if entry in ("varlen", "packed"):
        lengths = _lengths(case)
        T = sum(lengths)
        cu = torch.tensor([0] + lengths, dtype=torch.int32).cumsum(0, dtype=torch.int32)
        inputs = [_randn((T, Hq, D), case, gen), _randn((T, Hkv, D), case, gen), _randn((T, Hkv, D), case, gen)]
        if entry == "varlen":
            st["cu"] = cu
        else:
            st["tables"] = spa.llama3_flash_attn_prepare_cu_seqlens(cu, case["causal"], 0, 1)
        out_shape = (T, Hq, D)
    elif entry == "local":
        B = case["B"]
        inputs = [_randn((B, case["Sq"], Hq, D), case, gen), _randn((B, case["Sk"], Hkv, D), case, gen),
                  _randn((B, case["Sk"], Hkv, D), case, gen)]
        st["fn"] = spa.select_flash_attn_impl()
        out_shape = (B, case["Sq"], Hq, D)
    elif entry == "block":
        B, S, d = case["B"], case["S"], case["d_model"]
        block = spa.SequenceParallelAttentionBlock(d, Hq, Hkv, mode="ring", dtype=_DTYPE[case["dtype"]],
                                                   device="cuda", rope_base=10000.0)
        with torch.no_grad():
            for p in block.parameters():
                p.copy_(_randn(p.shape, case, gen, d ** -0.5))
        st["block"] = block
        inputs = [_randn((B, S, d), case, gen)]
        out_shape = (B, S, d)
    else:
        B, S = case["B"], case["S"]
        sigma = 0.5 if case.get("pack") == "kv" else 1.0
        if entry == "hybrid" or case.get("pack") == "qkv":
            inputs = [_randn((B, S, 3, Hq, D), case, gen, sigma)]
        elif case.get("pack") == "kv":
            inputs = [_randn((B, S, Hq, D), case, gen, sigma), _randn((B, S, 2, Hkv, D), case, gen, sigma)]
        else:
            inputs = [_randn((B, S, Hq, D), case, gen, sigma), _randn((B, S, Hkv, D), case, gen, sigma),
                      _randn((B, S, Hkv, D), case, gen, sigma)]
        if entry == "hybrid":
            st["module"] = spa.LongContextAttentionQKVPacked()
        out_shape = (B, S, Hq, D)
    if train:
        st["inputs"] = [t.requires_grad_(True) for t in inputs]
        st["dout"] = _randn(out_shape, case, gen)
    else:
        st["inputs"] = inputs
    return st


def _forward(st):
    case, x = st["case"], st["inputs"]
    entry, causal = case["entry"], case["causal"]
    if entry == "varlen":
        return spa.ring_flash_attn_varlen_func(*x, st["cu"], causal=causal)
    if entry == "packed":
        cu_q, cu_k, max_q, max_k, k_slice = st["tables"]
        return spa.llama3_flash_attn_varlen_func(*x, cu_q, cu_k, max_q, max_k, heads_k_stride=case["stride"],
                                                 local_k_slice=k_slice, causal=causal)
    if entry == "local":
        return st["fn"](*x, causal=causal, return_attn_probs=True)
    if entry == "block":
        return st["block"](x[0], causal=causal)
    if entry == "hybrid":
        return st["module"](x[0], causal=causal, return_attn_probs=True)
    if entry == "ulysses":
        return spa.ulysses_flash_attn_func(*x, causal=causal)
    fn = {"no": spa.ring_flash_attn_func, "kv": spa.ring_flash_attn_kvpacked_func,
          "qkv": spa.ring_flash_attn_qkvpacked_func}[case["pack"]]
    return fn(*x, causal=causal)


def run(st):
    if not st["case"]["train"]:
        with torch.no_grad():
            res = _forward(st)
        return [t for t in res if t is not None] if isinstance(res, tuple) else [res]
    out = _forward(st)
    leaves = list(st["inputs"])
    if "block" in st:
        leaves += list(st["block"].parameters())
    return [out.detach(), *torch.autograd.grad(out, leaves, st["dout"])]


def _pairs(Sq, Sk, causal):
    """Query-key pairs that the mask lets through (query i sees keys 0..i under `causal`)."""
    if not causal:
        return Sq * Sk
    n = min(Sq, Sk)
    return n * (n + 1) // 2 + (Sq - n) * Sk


def work(case):
    Hq, Hkv, D, train = case["Hq"], case["Hkv"], case["D"], case["train"]
    elt = 4 if case["dtype"] == "fp32" else 2
    if "lengths" in case:
        rows_q = rows_k = sum(_lengths(case))
        pairs = sum(_pairs(n, n, case["causal"]) for n in _lengths(case))
    elif case["entry"] == "local":
        rows_q, rows_k = case["B"] * case["Sq"], case["B"] * case["Sk"]
        pairs = case["B"] * _pairs(case["Sq"], case["Sk"], case["causal"])
    else:
        rows_q = rows_k = case["B"] * case["S"]
        pairs = case["B"] * _pairs(case["S"], case["S"], case["causal"])
    flops = 4.0 * Hq * D * pairs * (3.5 if train else 1.0)
    if case["entry"] == "block":
        d = case["d_model"]
        weights = d * (Hq + 2 * Hkv) * D + d * d
        # x in, out out; with training dout in, dx and the weight gradients out
        nbytes = elt * (2.0 * rows_q * d + weights) * (2 if train else 1)
        return {"bytes": nbytes, "flops": flops + 2.0 * rows_q * weights * (3 if train else 1)}
    q_b, kv_b = rows_q * Hq * D * elt, 2 * rows_k * Hkv * D * elt
    # q, k, v in, out out; with training dout in, dq, dk, dv out
    nbytes = 2.0 * q_b + kv_b + (2.0 * q_b + kv_b if train else 0)
    return {"bytes": nbytes, "flops": flops}


# Four times the relative error of the path against the same attention in 64 bits (S = 64..4096,
# head_dim 64 and 128, out, dq, dk and dv: bf16 2.5e-3, fp16 3.5e-4, fp32 1.9e-6); the block adds
# the roundings of its projections and of the rotated q and k.
def tolerance(case):
    if case["entry"] == "block":
        return {"rel": 1.5e-2}
    return {"rel": {"bf16": 1e-2, "fp16": 1.4e-3, "fp32": 1e-5}[case["dtype"]]}
