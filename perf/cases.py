"""The work a user of this package has it do, as cases to be timed and compared.

A case names a family and its sizes:

  op         `nsa_attention`: pooling, compression attention, block scoring + top-n, selection,
             window, gate blend; forward alone (prefill) or forward + every gradient (training)
  fused      `nsa_fused_forward`: the three branches with mean pooling and given block lists, the
             call an unmodified reference model makes through the drop-in
  selection  `selection_attn_triton` alone, forward + backward, on given block lists
  layer      `NSAAttentionB200` under bf16 autocast: the projections, the op and `out_proj`

Inputs are made on the GPU from the seed: q, k, v and the upstream gradient ~ N(0, 1), gate logits
~ N(0, 1), compressor parameters as the model initialises them with 0.02-std noise on the two that
start at zero, block lists as the benchmark ("recent": the newest complete blocks) or as unrelated
queries have them ("scattered": distinct visible blocks drawn at random).
"""
import importlib
import math

import torch

nsa = importlib.import_module("openbox-llm_b200")
NSAAttentionB200 = importlib.import_module("openbox-llm_b200.module").NSAAttentionB200

KV = ("kc", "vc", "ks", "vs", "kw", "vw")
COMP = ("k_intra", "k_logits", "k_proj", "v_intra", "v_logits", "v_proj")


def _case(name, family, grad, B, T, Hq, Hkv, D, block=64, sel=16, window=512, dtype="bf16", **more):
    return dict(name=name, family=family, grad=grad, B=B, T=T, Hq=Hq, Hkv=Hkv, D=D, block=block, sel=sel,
                window=window, dtype=dtype, **more)


def listed():
    return [
        # inference with the layer's default sizes (block 16, 4 blocks, window 32): the smallest call
        _case("layer_default_fwd", "layer", False, 1, 256, 8, 2, 64, block=16, sel=4, window=32),
        # a short prompt through the op: launches and host work
        _case("op_t512_fwd", "op", False, 1, 512, 16, 4, 64, pooling="learned"),
        # one training step of the op on a short sequence, 64-token blocks
        _case("op_t1k_train", "op", True, 1, 1024, 16, 4, 64, pooling="learned"),
        # the reference's operator sweep, forward, on its own kind of lists
        _case("fused_t4k_fwd", "fused", False, 1, 4096, 16, 4, 64, lists="recent"),
        # the reference's selection benchmark, forward + backward
        _case("selection_t8k_train", "selection", True, 1, 8192, 16, 4, 64, lists="recent"),
        # 16-token blocks at the head sizes of the 1.5B model, batch 2 x 1024 tokens, training
        _case("op_block16_train", "op", True, 2, 1024, 16, 4, 128, block=16, sel=8, pooling="learned"),
        # single precision, as the reference's own checks run the three branches
        _case("fused_f32_train", "fused", True, 1, 2048, 8, 2, 64, dtype="f32", lists="scattered"),
        # the published geometry: summaries of 32 tokens every 16, block 0 and two local blocks forced
        _case("op_strided_train", "op", True, 1, 2048, 8, 2, 64, pooling="learned", cmp_len=32, cmp_stride=16,
              n_init=1, n_local=2),
        # a length that is a multiple of nothing, three query heads per kv head, batch 3
        _case("op_ragged_train", "op", True, 3, 3001, 12, 4, 64, pooling="learned"),
        # one layer of the 12-layer model, micro-batch 8 x 4096 tokens, training
        _case("layer_t4k_train", "layer", True, 8, 4096, 12, 4, 64),
        # long-context prefill: 64 query heads, 65536 tokens
        _case("op_t64k_fwd", "op", False, 1, 65536, 64, 4, 128, pooling="learned"),
        # the training shape of the headline benchmark: batch 8 x 32768 tokens
        _case("op_t32k_train", "op", True, 8, 32768, 16, 2, 128, pooling="learned"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges.  Batch x tokens x heads stays within the largest listed case."""
    family = rng.choice(("op", "op", "op", "op16", "fused", "selection", "layer", "f32"))
    c = dict(family=family, grad=rng.random() < 0.6, block=64, sel=16, window=rng.choice((512, 512, 256, 200)), dtype="bf16")
    c["Hq"], c["Hkv"] = rng.choice(((8, 2), (12, 4), (16, 4), (16, 2), (16, 1), (64, 4)))
    c["D"] = rng.choice((64, 128))
    most = 32768
    if family == "op16":
        # small blocks: the layer's default and the block-16 models
        c.update(family="op", block=rng.choice((16, 32)), sel=rng.choice((4, 8)), window=rng.choice((32, 64, 512)))
        c["Hq"], c["Hkv"] = rng.choice(((8, 2), (12, 4), (16, 4)))
        most = 2048
    elif family == "f32":
        c.update(family="fused", dtype="f32", D=64, window=rng.choice((133, 512)))
        c["Hq"], c["Hkv"] = rng.choice(((8, 2), (12, 4)))
        most = 2048
    elif family == "layer":
        c["Hq"], c["Hkv"] = rng.choice(((8, 2), (12, 4), (16, 4)))
        most = 8192
    c["T"] = _log_int(rng, 128, most)
    if rng.random() < 0.5:
        c["T"] = (c["T"] + 63) // 64 * 64
    tokens = min(4 * most, 8 * 32768 * 16 * 128 // (4 * c["Hq"] * c["D"]))
    c["B"] = rng.randint(1, max(1, min(8, tokens // c["T"])))
    if c["family"] == "op":
        c["pooling"] = rng.choice(("learned", "learned", "mean"))
        if c["block"] == 64 and c["Hq"] != 64 and rng.random() < 0.25:
            c.update(pooling="learned", cmp_len=32, cmp_stride=16, n_init=1, n_local=2)
            c["Hq"], c["Hkv"] = rng.choice(((8, 2), (16, 4), (16, 1)))
    if c["family"] in ("fused", "selection"):
        c["lists"] = rng.choice(("recent", "scattered"))
        if c["T"] > 8192:                 # making scattered lists takes T x T / 64 random numbers
            c["lists"] = "recent"
    return c


def _lists(c, g, device):
    """Block lists [B, Hkv, T, sel] int32 of complete blocks, -1 where a query has fewer."""
    B, Hkv, T, bs, S = c["B"], c["Hkv"], c["T"], c["block"], c["sel"]
    n_blk = T // bs
    done = (torch.arange(T, device=device) + 1) // bs               # complete blocks at query t
    if c["lists"] == "recent":
        idx = done[:, None] - 1 - torch.arange(S, device=device)[None, :]
        idx = torch.where(idx >= 0, idx, torch.full_like(idx, -1)).to(torch.int32)
        return idx[None, None].expand(B, Hkv, T, S).contiguous()
    idx = torch.full((B, Hkv, T, S), -1, device=device, dtype=torch.int32)
    k = min(S, n_blk)
    if k:
        hidden = torch.arange(n_blk, device=device)[None, :] >= done[:, None]
        for b in range(B):
            r = torch.rand(Hkv, T, n_blk, generator=g, device=device).masked_fill_(hidden, -1.0)
            v, j = r.topk(k, dim=-1)
            idx[b, :, :, :k] = torch.where(v >= 0, j, torch.full_like(j, -1)).to(torch.int32)
    return idx


def prepare(case, seed):
    c = dict(case)
    dev = torch.device("cuda")
    dtype = torch.bfloat16 if c["dtype"] == "bf16" else torch.float32
    g = torch.Generator(device=dev).manual_seed(seed)
    B, T, Hq, Hkv, D, grad = c["B"], c["T"], c["Hq"], c["Hkv"], c["D"], c["grad"]

    def normal(*shape, dt=dtype):
        return torch.randn(*shape, generator=g, device=dev).to(dt)

    s = {"case": c}
    if c["family"] == "layer":
        layer = NSAAttentionB200(Hq * D, Hq, Hkv, block_size=c["block"], n_selected_blocks=c["sel"],
                                 window=c["window"]).to(dev)
        for name, p in layer.named_parameters():
            if name != "gate.bias":
                p.data.normal_(0.0, 0.02, generator=g)
            else:
                p.data.zero_()
            p.requires_grad_(grad)
        s["layer"] = layer
        s["x"] = normal(B, T, Hq * D, dt=torch.float32).requires_grad_(grad)     # as LayerNorm leaves it
        if grad:
            s["leaves"] = [s["x"]] + list(layer.parameters())
            s["do"] = normal(B, T, Hq * D)
        return s
    s["q"] = normal(B, Hq, T, D)
    names = ("ks", "vs") if c["family"] == "selection" else KV
    for n in names:
        s[n] = normal(B, Hkv, T, D)
    leaves = ["q", *names]
    if c["family"] != "selection":
        s["gate"] = normal(B, Hq, T, 3)
        leaves.append("gate")
    if c["family"] != "op":
        s["idx"] = _lists(c, g, dev)
    elif c["pooling"] == "learned":
        n = c.get("cmp_len", c["block"])
        for p in ("k", "v"):
            s[p + "_intra"] = 0.02 * normal(n, D, dt=torch.float32)
            s[p + "_logits"] = 0.02 * normal(n, dt=torch.float32)
            s[p + "_proj"] = (torch.rand(D, D, generator=g, device=dev) * 2 - 1) * D ** -0.5
        leaves += COMP
    if grad:
        for n in leaves:
            s[n].requires_grad_(True)
        s["leaves"] = [s[n] for n in leaves]
        s["do"] = normal(B, Hq, T, D)
    return s


def _forward(s):
    c = s["case"]
    if c["family"] == "layer":
        with torch.autocast("cuda", dtype=torch.bfloat16):
            return s["layer"](s["x"])
    if c["family"] == "selection":
        return nsa.selection_attn_triton(s["q"], s["ks"], s["vs"], s["idx"], c["block"])
    kv = [s[n] for n in KV]
    if c["family"] == "fused":
        return nsa.nsa_fused_forward(s["q"], *kv, s["gate"], s["idx"], c["block"], c["window"])
    comp = {n: s[n] for n in COMP} if c["pooling"] == "learned" else None
    return nsa.nsa_attention(s["q"], *kv, s["gate"], c["block"], c["sel"], c["window"], compressor=comp,
                             n_init_blocks=c.get("n_init", 0), n_local_blocks=c.get("n_local", 0),
                             cmp_len=c.get("cmp_len"), cmp_stride=c.get("cmp_stride"))


def run(state):
    """One forward (prefill), or one forward and every gradient (training)."""
    if not state["case"]["grad"]:
        with torch.no_grad():
            return _forward(state)
    out = _forward(state)
    return [out.detach(), *torch.autograd.grad(out, state["leaves"], state["do"])]


def work(case):
    """Each input read once and each output written once; 4 D operations per attended (query head,
    key) pair forward, 2.5 times that backward, and the layer's projections."""
    c = case
    B, T, Hq, Hkv, D, bs, S, W = (c[k] for k in ("B", "T", "Hq", "Hkv", "D", "block", "sel", "window"))
    size = 2 if c["dtype"] == "bf16" else 4
    cl = c.get("cmp_len", bs)
    cs = c.get("cmp_stride", cl)
    keys = 0
    for t in range(T):
        done = (t + 1) // bs
        if c.get("n_local"):              # the block that holds t is forced into the list
            keys += min(S - 1, t // bs) * bs + t % bs + 1
        else:
            keys += min(S, done) * bs
        if c["family"] != "selection":
            keys += min(W, t + 1) + ((t + 1 - cl) // cs + 1 if t + 1 >= cl else 0)
    flops = 4 * D * keys * B * Hq * (3.5 if c["grad"] else 1.0)
    q = B * Hq * T * D * size
    kv = B * Hkv * T * D * size
    if c["family"] == "layer":
        dm = Hq * D
        weights = dm * (2 * Hq * D + 6 * Hkv * D + 3 * Hq)
        flops += 2 * B * T * weights * (3 if c["grad"] else 1)
        x = B * T * dm * 4
        moved = x + x // 2 + 4 * weights                                  # x, y, parameters
        return {"bytes": moved + (x + x // 2 + 4 * weights if c["grad"] else 0), "flops": flops}
    n_kv = 2 if c["family"] == "selection" else 6
    gate = 0 if c["family"] == "selection" else B * Hq * T * 3 * size
    lists = B * Hkv * T * S * 4 if c["family"] != "op" else 0
    moved = 2 * q + n_kv * kv + gate + lists                              # inputs and the output
    if c["grad"]:
        moved += 2 * q + n_kv * kv + gate                                 # dO and the gradients
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    if case["dtype"] == "f32":
        return {"rel": 1e-5, "max": 1e-3}       # fp32 products and sums, in any order
    # bf16 results of fp32 accumulation.  A single entry may be off by more: two blocks whose scores
    # tie to the last fp32 bits may swap, which changes one of a row's few listed blocks.
    return {"rel": 1e-2, "max": 0.9}
