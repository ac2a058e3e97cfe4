"""The work that users of deltanet_b200 have it do, as measurable cases.

A case names one of five kinds of pass through the public operators:

  decode   one token for each of B running sequences (``*_decode_step``), the inner loop of text generation
  prefill  the forward pass over prompts, ``is_inference=True`` with the final state handed to decoding
  train    forward and backward of one recurrence, all gradients
  layer    a whole Gated DeltaNet mixer between its projections: short convolution, gates, recurrence and
           gated RMSNorm, forward and backward (or forward only)

Head counts, head widths and value distributions are those of this repository's benchmark and tests; lengths
and batch sizes run from one token and one sequence to the largest that the benchmark uses.
"""
import math
import os
import random
import sys

import torch

_PKG = os.path.join(os.getcwd(), "deltanet-tpu_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import deltanet_b200 as dn  # noqa: E402

BF16, F32 = torch.bfloat16, torch.float32

# What a case may say, and what it means where it does not.
DEFAULTS = dict(
    kind="train", op="gdn2", B=1, L=1, Hk=16, Hv=32, K=128, V=128, dtype="bf16", gates="fp32", chunk=128,
    docs="none",            # none | half | segment_ids | cu_seqlens
    mean_doc=1024, init=False, recompute=False, fused=False, streaming=False, state="bf16", in_place=False,
    reset=False, backward=True)

HEADS = ((16, 32), (12, 24), (32, 32), (16, 16), (4, 8), (2, 4), (8, 8))


def _full(case):
    c = dict(DEFAULTS)
    c.update(case)
    return c


def listed():
    return [
        # One interactive user: a single sequence, scalar gates, bf16 state; nothing but latency.
        dict(name="decode_one", kind="decode", op="gdn", B=1, Hk=16, Hv=32, state="bf16"),
        # A lightly loaded server: an odd number of slots, the default fp32 state, some slots just refilled.
        dict(name="decode_slots_fp32", kind="decode", op="kda", B=37, Hk=32, Hv=32, state="fp32", reset=True),
        # A full server: 256 sequences, channel-wise gates, bf16 state updated in place.
        dict(name="decode_serving", kind="decode", op="gdn2", B=256, Hk=16, Hv=32, state="bf16", in_place=True),
        # A short chat turn: a prompt below one tile, latency again.
        dict(name="prompt_short", kind="prefill", op="gdn", B=1, L=75, Hk=16, Hv=32),
        # A long prompt that continues a stored state, streamed in blocks; ragged length.
        dict(name="prefill_streaming", kind="prefill", op="gdn2", B=1, L=20011, Hk=16, Hv=32, init=True, streaming=True),
        # Packed documents through Gated DeltaNet, the batch prefill of the benchmark.
        dict(name="prefill_packed", kind="prefill", op="gdn", B=4, L=8192, Hk=16, Hv=32, docs="segment_ids"),
        # The single-precision configuration at small size: debugging, numerics work, small research models.
        dict(name="train_fp32_small", kind="train", op="gdn2", B=1, L=256, Hk=2, Hv=4, K=64, V=64, dtype="fp32",
             chunk=64, docs="half"),
        # The headline training shape of the benchmark.
        dict(name="train_headline", kind="train", op="gdn2", B=1, L=2048, Hk=12, Hv=24, docs="half"),
        # Mixed-precision training with gate pre-activations in bf16, packed documents, odd length.
        dict(name="train_fused_packed", kind="train", op="gdn2", B=1, L=6001, Hk=12, Hv=24, gates="bf16", fused=True,
             docs="cu_seqlens"),
        # DeltaNet with narrow heads.
        dict(name="train_delta_rule_64", kind="train", op="delta_rule", B=4, L=2048, Hk=16, Hv=16, K=64, V=64),
        # A Gated DeltaNet mixer in training, packed documents, odd length.
        dict(name="layer_train", kind="layer", B=2, L=4001, Hk=16, Hv=32, docs="segment_ids"),
        # Long-context training: one packed sequence, channel-wise decay, states recomputed in the backward.
        dict(name="train_long", kind="train", op="kda", B=1, L=131072, Hk=32, Hv=32, chunk=64, recompute=True,
             docs="segment_ids", mean_doc=17408),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(("decode", "decode", "prefill", "prefill", "train", "train", "train", "layer"))
    Hk, Hv = rng.choice(HEADS)
    c = dict(kind=kind, Hk=Hk, Hv=Hv)
    if kind == "decode":
        c.update(op=rng.choice(("gdn2", "gdn", "kda", "gla", "delta_rule")), B=_log_int(rng, 1, 256),
                 state=rng.choice(("bf16", "bf16", "fp32")), reset=rng.random() < 0.25)
        c["in_place"] = c["op"] == "gdn2" and rng.random() < 0.5
        return c
    B = rng.choice((1, 1, 2, 4))
    docs = rng.choice(("none", "half", "segment_ids", "cu_seqlens"))
    c.update(B=B, docs=docs, mean_doc=_log_int(rng, 128, 8192))
    if kind == "prefill":
        c.update(op=rng.choice(("gdn", "gdn", "gdn2", "kda", "gla", "delta_rule")), L=_log_int(rng, 4, 32768 // B),
                 init=rng.random() < 0.4, streaming=rng.random() < 0.2 and docs == "none")
        if c["streaming"]:
            c["op"] = "gdn2"
        return c
    if kind == "layer":
        c.update(L=_log_int(rng, 32, 16384 // B), backward=rng.random() < 0.7)
        return c
    c["op"] = rng.choice(("gdn2", "gdn2", "gdn", "kda", "gla", "delta_rule"))
    form = rng.choice(("bf16", "bf16", "bf16", "fused", "narrow", "fp32"))
    c["recompute"] = rng.random() < 0.3
    c["chunk"] = rng.choice((64, 128, 128))
    if form == "fp32":
        Hk, Hv = rng.choice(((2, 4), (4, 4), (4, 8)))
        c.update(dtype="fp32", Hk=Hk, Hv=Hv, L=_log_int(rng, 32, 2048 // B), K=rng.choice((64, 128)))
        c["V"] = c["K"]
        return c
    c.update(L=_log_int(rng, 32, 16384 // B), init=rng.random() < 0.15)
    if form == "fused":
        c.update(op="gdn2", fused=True, gates=rng.choice(("bf16", "fp32")))
    if form == "narrow":
        c.update(K=64, V=64, L=_log_int(rng, 32, 8192 // B))
    return c


# ------------------------------------------------------------------------------------------------- inputs
def _documents(c, seed, dev):
    """(segment_ids, cu_seqlens) of a case; documents of geometric length, at least 32 tokens."""
    B, L = c["B"], c["L"]
    if c["docs"] == "none":
        return None, None
    if c["docs"] == "half":
        return (torch.arange(L, device=dev) >= L // 2).to(torch.int32)[None].expand(B, L).contiguous(), None
    rnd = random.Random(seed)
    cuts = []
    for _ in range(B if c["docs"] == "segment_ids" else 1):
        at, row = 0, []
        while True:
            at += max(32, int(rnd.expovariate(1.0 / c["mean_doc"])))
            if at >= L:
                break
            row.append(at)
        cuts.append(row)
    if c["docs"] == "cu_seqlens":
        return None, torch.tensor([0] + cuts[0] + [L], dtype=torch.int32, device=dev)
    pos = torch.arange(L, device=dev)
    rows = [torch.searchsorted(torch.tensor(r, device=dev, dtype=pos.dtype), pos, right=True) for r in cuts]
    return torch.stack(rows).to(torch.int32), None


def _gates(c, rn, rows):
    """The gate tensors of one operator, activated unless `fused`; `rows`: the leading dimensions."""
    Hk, Hv, K, V = c["Hk"], c["Hv"], c["K"], c["V"]
    dt = BF16 if c["gates"] == "bf16" else F32
    if c["op"] == "gdn2":
        b, w, g = rn(*rows, Hk, K) * 0.39, rn(*rows, Hv, V) * 0.39, rn(*rows, Hk, K) * 0.39 - 1.0
        if not c["fused"]:
            b, w, g = torch.sigmoid(b), torch.sigmoid(w), -torch.exp(g)
        return dict(g=g.to(dt), b=b.to(dt), w=w.to(dt))
    if c["op"] == "gdn":
        A = 1.0 + 15.0 * torch.sigmoid(rn(Hv))
        return dict(g=(-A * torch.nn.functional.softplus(rn(*rows, Hv) + 0.5 * rn(Hv))).to(dt),
                    beta=torch.sigmoid(rn(*rows, Hv)).to(dt))
    if c["op"] == "kda":
        return dict(g=(-torch.exp(0.39 * rn(*rows, Hk, K) - 1.0)).to(dt), beta=torch.sigmoid(rn(*rows, Hk)).to(dt))
    if c["op"] == "gla":
        return dict(g=(-torch.exp(0.39 * rn(*rows, Hk, K) - 1.0)).to(dt))
    return dict(beta=torch.sigmoid(rn(*rows, Hk)).to(dt))


def prepare(case, seed):
    c = _full(case)
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(int(seed))

    def rn(*shape):
        return torch.randn(*shape, generator=gen, device=dev)

    B, L, Hk, Hv, K, V = (c[n] for n in ("B", "L", "Hk", "Hv", "K", "V"))
    dt = F32 if c["dtype"] == "fp32" else BF16
    s = dict(case=c)
    if c["kind"] == "decode":
        s.update(q=rn(B, Hk, K).to(dt), k=rn(B, Hk, K).to(dt), v=rn(B, Hv, V).to(dt), gates=_gates(c, rn, (B,)))
        s["state"] = (rn(B, Hv, K, V) * 0.1).to(BF16 if c["state"] == "bf16" else F32)
        s["reset"] = (torch.rand(B, generator=gen, device=dev) < 0.1) if c["reset"] else None
        return s
    seg, cu = _documents(c, int(seed), dev)
    s["kw"] = kw = dict(qk_l2norm=True, chunk_size=c["chunk"], precision=c["dtype"])
    if seg is not None:
        kw["segment_ids"] = seg
    if cu is not None:
        kw["cu_seqlens"] = cu
    if c["kind"] == "layer":
        D = 2 * Hk * K + Hv * V
        s["heads"] = (Hk, Hv, K, V)
        s["kw"] = dict(qk_l2norm=True)
        s["docs"] = seg
        if seg is None and cu is not None:            # the convolution takes ids: the same ids for both
            s["docs"] = torch.searchsorted(cu[1:].contiguous(), torch.arange(L, device=dev, dtype=torch.int32), right=True
                                           ).to(torch.int32)[None].expand(B, L).contiguous()
        leaves = dict(x=rn(B, L, D).to(dt), conv=(rn(D, 1, 4) * 0.3).to(dt), a=rn(B, L, Hv).to(dt), b=rn(B, L, Hv).to(dt),
                      A_log=torch.log(1.0 + 15.0 * torch.rand(Hv, generator=gen, device=dev)), dt_bias=0.5 * rn(Hv),
                      z=rn(B, L, Hv, V).to(dt), norm=1.0 + 0.1 * rn(V))
    else:
        leaves = dict(q=rn(B, L, Hk, K).to(dt), k=rn(B, L, Hk, K).to(dt), v=rn(B, L, Hv, V).to(dt))
        leaves.update(_gates(c, rn, (B, L)))
        if c["init"]:
            leaves["initial_state"] = rn(B, Hv, K, V) * 0.1
    train = c["kind"] == "train" or (c["kind"] == "layer" and c["backward"])
    if train:
        leaves = {n: t.requires_grad_() for n, t in leaves.items()}
        s["d_out"] = rn(B, L, Hv, V).to(dt)
    if c["kind"] == "prefill":
        kw.update(is_inference=True, output_final_state=True)
        if c["streaming"]:
            kw.update(streaming_prefill=True)
    if c["kind"] == "train" and c["recompute"]:
        kw["recompute_states"] = True
    if c["fused"]:
        kw["fuse_prologue"] = True
    s["leaves"], s["train"] = leaves, train
    return s


# ------------------------------------------------------------------------------------------------- one pass
_CHUNK = dict(gdn2=dn.chunk_gdn2, gdn=dn.chunk_gdn, kda=dn.chunk_kda, gla=dn.chunk_gla, delta_rule=dn.chunk_delta_rule)
_STEP = dict(gdn2=dn.gdn2_decode_step, gdn=dn.gdn_decode_step, kda=dn.kda_decode_step, gla=dn.gla_decode_step,
             delta_rule=dn.delta_rule_decode_step)


def run(s):
    c = s["case"]
    if c["kind"] == "decode":
        kw = dict(out_state=s["state"]) if c["in_place"] else {}
        if c["state"] == "bf16":
            kw["state_dtype"] = "bfloat16"
        return _STEP[c["op"]](s["q"], s["k"], s["v"], *s["gates"].values(), s["state"], qk_l2norm=True, reset=s["reset"], **kw)
    t = s["leaves"]
    if c["kind"] == "layer":
        Hk, Hv, K, V = s["heads"]
        q, k, v = dn.gdn_qkv_producer(t["x"], t["conv"], num_k_heads=Hk, num_v_heads=Hv, head_k_dim=K, head_v_dim=V,
                                      segment_ids=s["docs"])
        g, beta = dn.gdn_gates(t["a"], t["b"], t["A_log"], t["dt_bias"])
        o = dn.chunk_gdn(q, k, v, g, beta, segment_ids=s["docs"], is_inference=not s["train"], **s["kw"])
        out = dn.gated_rmsnorm(o, t["z"], t["norm"])
    else:
        out = _CHUNK[c["op"]](**t, **s["kw"])
    if not s["train"]:
        return out
    return (out,) + torch.autograd.grad(out, list(t.values()), s["d_out"])


# ------------------------------------------------------------------------------------------------- accounting
def _numel(c):
    """Elements of (q and k, v, all gates together) of the un-broadcast user tensors."""
    rows = c["B"] * (1 if c["kind"] == "decode" else c["L"])
    Hk, Hv, K, V = c["Hk"], c["Hv"], c["K"], c["V"]
    gates = dict(gdn2=2 * Hk * K + Hv * V, gdn=2 * Hv, kda=Hk * K + Hk, gla=Hk * K, delta_rule=Hk)[c["op"]]
    return rows * 2 * Hk * K, rows * Hv * V, rows * gates


def work(case):
    """Every user tensor read once (twice where a backward pass follows a forward pass over the same tensor: the
    saved inputs), every result written once; flops of the token recurrence: decay, read, rank-one update and
    query of the state, and twice that for its adjoint."""
    c = _full(case)
    B, Hv, K, V = c["B"], c["Hv"], c["K"], c["V"]
    es = 4 if c["dtype"] == "fp32" else 2
    gs = 2 if c["gates"] == "bf16" else 4
    if c["kind"] == "decode":
        qk, v, g = _numel(c)
        ss = 2 if c["state"] == "bf16" else 4
        return {"bytes": 2 * B * Hv * K * V * ss + (qk + 2 * v) * es + g * gs, "flops": 7 * B * Hv * K * V}
    L = c["L"]
    flops = 7 * B * L * Hv * K * V
    if c["kind"] == "layer":
        x = B * L * (2 * c["Hk"] * K + Hv * V) * es
        v, ab = B * L * Hv * V * es, 2 * B * L * Hv * es
        fwd = x + ab + v + v
        return {"bytes": fwd + (2 * (x + ab + v) + v if c["backward"] else 0), "flops": flops * (3 if c["backward"] else 1)}
    qk, v, g = _numel(c)
    ins = (qk + v) * es + g * gs
    state = B * Hv * K * V * 4
    if c["kind"] == "prefill":
        return {"bytes": ins + v * es + state * (2 if c["init"] else 1), "flops": flops}
    return {"bytes": 3 * ins + 2 * v * es + (3 * state if c["init"] else 0), "flops": 3 * flops}


def tolerance(case):
    c = _full(case)
    if c["kind"] == "decode":
        return {"rel": 5e-3}                 # fp32 arithmetic; the results are rounded to bf16 once
    if c["dtype"] == "fp32":
        return {"rel": 2e-5}                 # fp32 sums, carried along the sequence
    if c["kind"] == "prefill" or not c["backward"]:
        return {"rel": 1e-2}                 # bf16 operands
    return {"rel": 2e-2}                     # bf16 operands in a chain of products; gate gradients are differences of them
