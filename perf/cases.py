"""Performance cases of the routed quantized SwiGLU expert FFN, measured through the package's public entry points.

A case names the entry point (`kind`), the weight format and shape of a layer, the router, the number of token rows and
the number of layers one pass walks through.  Every layer has its own experts, router and hidden states: in a model the
attention of the next layer lies between two calls, so a pass never feeds one layer's output to the next.

  device   moe_layer_forward_device on torch's current stream: rows already on the GPU, what a serving loop calls
  host     moe_layer_forward: rows and routing in ordinary host memory, synchronous
  step     LinearGate.route + moe_step_weighted_into, one token: the calls the reference's engine makes per layer
  miss     the same layers with too few HBM slots: each routed expert is looked up in the logical tier and
           demand-admitted from host memory before the layer runs
  expert   expert_forward_noalloc: one expert on flat blocks, no handle
"""
import functools
import math

import numpy as np
import torch

import mer_b200

FORMATS = {"q4_0": (mer_b200.DTYPE_Q4_0, 18, 0.002, 0.01), "q8_0": (mer_b200.DTYPE_Q8_0, 34, 0.0005, 0.002)}
MAX_PAIR_FLOPS = 3.3e12   # of a drawn case: the largest listed one does 3.25e12
MAX_STATE_BYTES = 6.5e9   # expert bytes of a drawn case: the largest listed one holds 6.4e9

_BASE = dict(kind="device", format="q8_0", d_model=2048, d_ff=768, experts=128, top_k=8, tokens=1, layers=1, zipf=0.0,
             sigmoid=False, n_group=1, topk_group=1, scaling=1.0, shared=False, block=False, pinned=False)


def _case(**kw):
    unknown = set(kw) - set(_BASE) - {"name"}
    assert not unknown, unknown
    return {**_BASE, **kw}


_LARGE_FEW = dict(format="q4_0", d_model=4096, d_ff=14336, experts=8, top_k=2)
_SMALL_MANY = dict(format="q8_0", d_model=2048, d_ff=768, experts=128, top_k=8)
_WIDE_GROUPED = dict(format="q4_0", d_model=7168, d_ff=2048, experts=256, top_k=8, sigmoid=True, n_group=8, topk_group=4,
                     scaling=2.5, shared=True)


def listed():
    return [
        # One user's token through a stretch of the Qwen3-30B-A3B-shaped stack: eight 5 MB experts per layer, the smallest
        # device call there is; launches and latency count.  Eight layers, so that the weights come from HBM.
        _case(name="decode-q8-128x8-b1", layers=8, **_SMALL_MANY),
        # The same stack under a serving batch: nearly all experts hit, about four tokens each.
        _case(name="decode-q8-128x8-b64", layers=4, tokens=64, **_SMALL_MANY),
        # One token through Mixtral-8x7B-shaped layers, the workload the reference's `run` executes.
        _case(name="decode-q4-8x2-b1", layers=3, **_LARGE_FEW),
        # A small batch on the same stack with the skewed routing of the decode sweep: all experts hit, a few tokens each.
        _case(name="decode-q4-8x2-b16", layers=2, tokens=16, zipf=1.1, **_LARGE_FEW),
        # The top of that sweep: 64 tokens per expert on average, between decode and prefill.
        _case(name="batch-q4-8x2-b256", layers=1, tokens=256, zipf=1.1, **_LARGE_FEW),
        # A prompt's prefill through the 128-expert layers with the benchmark's load imbalance.
        _case(name="prefill-q8-128x8-b2048", layers=2, tokens=2048, zipf=1.0, **_SMALL_MANY),
        # Decode on a DeepSeek-V3-shaped block as a model calls it: RMSNorm in front, sigmoid routing in groups, the gated
        # shared expert, the residual add behind.
        _case(name="decode-q4-256x8-block-b16", tokens=16, block=True, **_WIDE_GROUPED),
        # The largest call: a 4096-token prefill of that layer, 128 tokens per expert and all of them on the shared one.
        _case(name="prefill-q4-256x8-b4096", tokens=4096, **_WIDE_GROUPED),
        # A layer whose d_ff is no multiple of 256 (many published models have such sizes) under a ragged batch.
        _case(name="ragged-q8-2048x1408-b37", d_model=2048, d_ff=1408, experts=64, top_k=6, tokens=37, layers=2),
        # The engine's own calls, token by token on host memory: the smallest calls, bound by their latency.
        _case(name="step-q8-128x8", kind="step", layers=4, **_SMALL_MANY),
        # Expert streaming: more experts than HBM slots, payloads in ordinary (not pinned) host memory.
        _case(name="miss-q4-8x2-b1", kind="miss", layers=3, **_LARGE_FEW),
        # A host that owns every byte of the device runs one expert at a time on flat blocks, a few rows each.
        _case(name="expert-q4-4096x14336-b4", kind="expert", tokens=4, layers=2, **_LARGE_FEW),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choices(["device", "host", "step", "miss", "expert"], [8, 1, 1, 1, 1])[0]
    while True:
        fmt = rng.choice(["q4_0", "q8_0"])
        # mostly whole 256-value tiles, sometimes only whole 32-value blocks
        step = rng.choices([256, 32], [4, 1])[0]
        d_model, d_ff = (max(step, _log_int(rng, 512, 8192) // step * step) for _ in range(2))
        if step == 256 and rng.random() < 0.2:
            d_ff = rng.choice([10240, 12288, 14336])
        experts = rng.choice([8, 8, 16, 32, 60, 64, 96, 128, 160, 256])
        top_k = min(experts // 2, rng.choice([1, 2, 2, 4, 6, 8, 8]))
        sigmoid = experts % 8 == 0 and experts >= 64 and rng.random() < 0.3
        c = _case(kind=kind, format=fmt, d_model=d_model, d_ff=d_ff, experts=experts, top_k=top_k, layers=rng.randint(1, 4),
                  zipf=rng.choice([0.0, 0.0, round(rng.uniform(0.5, 1.2), 2)]), sigmoid=sigmoid)
        if sigmoid:
            c.update(n_group=8, topk_group=rng.choice([4, 8]), scaling=2.5, shared=rng.random() < 0.5)
        aligned = d_model % 256 == 0 and d_ff % 256 == 0
        if kind == "device":
            c.update(tokens=_log_int(rng, 1, 4096 if aligned else 256), block=rng.random() < 0.25)
        elif kind == "host":
            c.update(tokens=_log_int(rng, 1, 256))
        elif kind == "miss":
            c.update(tokens=_log_int(rng, 1, 4), layers=3, pinned=rng.random() < 0.5)
        elif kind == "expert":
            c.update(tokens=rng.randint(1, 8), sigmoid=False, n_group=1, topk_group=1, scaling=1.0, shared=False)
        stack = (experts + c["shared"]) * c["layers"] if kind != "expert" else c["layers"]
        moved = c["layers"] * c["tokens"] * top_k * _expert_bytes(c) if kind == "miss" else 0
        slow = 1 if aligned and kind != "expert" else 20
        if (stack * _expert_bytes(c) <= MAX_STATE_BYTES and moved <= 6e8
                and c["layers"] * c["tokens"] * _slots(c) * 6.0 * d_model * d_ff * slow <= MAX_PAIR_FLOPS):
            return c


def _slots(c):
    return 1 if c["kind"] == "expert" else c["top_k"] + int(c["shared"])


def _expert_bytes(c):
    return 3 * (c["d_model"] * c["d_ff"] // 32) * FORMATS[c["format"]][1]


@functools.lru_cache(maxsize=256)
def _routed_experts_hit(experts, top_k, tokens, zipf, spread):
    """Distinct routed experts one layer pass reads: the mean over a few simulated draws of its routing."""
    rng, hits = np.random.default_rng(0), []
    for _ in range(4):
        logits = rng.standard_normal((tokens, experts)) * spread - zipf * np.log(np.arange(experts) + 1.0)
        hits.append(np.unique(np.argpartition(-logits, top_k - 1, axis=1)[:, :top_k]).size)
    return float(np.mean(hits))


def work(case):
    c = case
    D, T, L = c["d_model"], c["tokens"], c["layers"]
    rows = T * D * 4 * 2  # the input rows read, the output rows written
    if c["kind"] == "expert":
        return {"bytes": L * (_expert_bytes(c) + rows), "flops": L * T * 6.0 * D * c["d_ff"]}
    hit = _routed_experts_hit(c["experts"], c["top_k"], T, c["zipf"], 0.02 * math.sqrt(D)) + int(c["shared"])
    layer = hit * _expert_bytes(c) + c["experts"] * D * 4 + rows
    return {"bytes": L * layer, "flops": L * (T * _slots(c) * 6.0 * D * c["d_ff"] + 2.0 * T * c["experts"] * D)}


def tolerance(case):
    # fp32 rows, outputs and sums over weights that are exact in fp32; products of 22 significant bits at least, sums of up
    # to 14336 terms in another order.  The path's stated bar is 1e-3 of the rows' root mean square for the largest error.
    return {"rel": 1e-4, "max": 1e-3}


# ------------------------------------------------------------------------------------------------ inputs


def _generator(seed, *tags):
    key = 0
    for v in (seed, *tags):
        key = (key * 1000003 + int(v) + 1) % (1 << 62)
    return torch.Generator(device="cuda").manual_seed(key)


def _blobs(c, n, gen):
    """n experts' gate||up||down block streams on the GPU: uniform quants, uniform f16 scales (the benchmark's ranges)."""
    _, bb, lo, hi = FORMATS[c["format"]]
    blocks = 3 * (c["d_model"] * c["d_ff"] // 32)
    out = torch.empty((n, blocks, bb), dtype=torch.uint8, device="cuda")
    for i in range(n):
        if c["format"] == "q4_0":
            out[i, :, 2:] = torch.randint(0, 256, (blocks, 16), dtype=torch.uint8, device="cuda", generator=gen)
        else:
            out[i, :, 2:] = torch.randint(-127, 128, (blocks, 32), dtype=torch.int8, device="cuda", generator=gen).view(torch.uint8)
        scale = torch.rand((blocks, 1), device="cuda", generator=gen) * (hi - lo) + lo
        out[i, :, :2] = scale.to(torch.float16).view(torch.uint8)
    return out.reshape(n, blocks * bb)


def _choose(c, x, w, bias, rms):
    """The experts each row selects, and whether the choice is clear of the resolution of fp32 sums (a tie has two right
    answers)."""
    x = x.double()
    if rms is not None:
        x = x * torch.rsqrt(x.square().mean(1, keepdim=True) + 1e-6) * rms.double()
    s = x @ w.double().T + bias.double()
    k, E, G = c["top_k"], c["experts"], c["n_group"]
    least = 1e-4
    ok = torch.ones(x.shape[0], dtype=torch.bool, device=x.device)
    if c["sigmoid"]:
        s, least = torch.sigmoid(s), 1e-5
        if c["topk_group"] < G:
            per = s.reshape(-1, G, E // G)
            g = per.topk(2, dim=2).values.sum(2)
            top = g.topk(c["topk_group"] + 1, dim=1)
            ok &= top.values[:, -2] - top.values[:, -1] > least
            keep = torch.zeros_like(g, dtype=torch.bool).scatter_(1, top.indices[:, :-1], True)
            s = per.masked_fill(~keep[:, :, None], -1.0).reshape(-1, E)
    top = s.topk(k + 1, dim=1)
    return top.indices[:, :k], ok & (top.values[:, k - 1] - top.values[:, k] > least)


class _State:
    pass


def prepare(case, seed):
    c, s = case, _State()
    dtype, _, _, _ = FORMATS[c["format"]]
    D, F, E, L, T = c["d_model"], c["d_ff"], c["experts"], c["layers"], c["tokens"]
    s.case, s.dtype = c, dtype
    x_gen = _generator(seed, 1)
    s.x = [torch.randn((T, D), device="cuda", generator=x_gen) for _ in range(L)]
    s.out = [torch.empty((T, D), device="cuda") for _ in range(L)]
    if c["kind"] == "expert":
        s.blobs = _blobs(c, L, _generator(seed, 2))
        return s

    # ---- routers, and rows whose routing is unambiguous
    shared = int(c["shared"])
    n_ids, eb = L * (E + shared), _expert_bytes(c)
    stride = (256 + eb + 4095) // 4096 * 4096
    gates, norms, need = [], [], []
    for l in range(L):
        gen = _generator(seed, 3, l)
        w = torch.randn((E, D), device="cuda", generator=gen) * 0.02
        rank = torch.randperm(E, device="cuda", generator=gen)
        bias = -c["zipf"] * torch.log(rank + 1.0)
        rms = 1.0 + 0.1 * torch.randn(D, device="cuda", generator=gen) if c["block"] else None
        for _ in range(20):
            ids, clear = _choose(c, s.x[l], w, bias, rms)
            bad = ~clear
            n = int(bad.sum())
            if n == 0:
                break
            s.x[l][bad] = torch.randn((n, D), device="cuda", generator=gen)
        gate = mer_b200.LinearGate.with_routing(w.cpu().numpy(), E, D, c["top_k"], int(c["sigmoid"]), True, None, c["n_group"],
                                                c["topk_group"], c["scaling"])
        if c["zipf"]:
            gate.logit_bias = bias.cpu().numpy()
        gates.append(gate)
        sg = 0.02 * torch.randn(D, device="cuda", generator=gen) if c["block"] and shared else None
        norms.append((rms, sg))
        need.append([l * E + i for i in torch.unique(ids).tolist()] + [L * E + l] * shared)

    # ---- the backend: all experts resident, or (miss) slots for about half of what a pass over the layers routes to
    n_slots = n_ids if c["kind"] != "miss" else max(max(map(len, need)), sum(map(len, need)) // 2)
    s.backend = b = mer_b200.Backend(dtype, D, F, stride * n_slots, n_ids, max_tokens=max(T, 64), max_top_k=_slots(c))
    for l, gate in enumerate(gates):
        gate.bind(b, l, L * E + l if shared else mer_b200.EXPERT_NONE)
        rms, sg = norms[l]
        if c["block"]:
            b.install_layer(l, rms.cpu().numpy(), 1e-6, None if sg is None else sg.cpu().numpy(), residual=True)
    s.gates = gates
    if c["kind"] == "miss":
        # the payloads of the experts that the rows route to, in host memory, and the trace of the ids, as a replay has it
        s.cache = mer_b200.GpuExpertCache(2 * n_slots * eb, 0.5, 1 << 30)
        s.need, s.payload = need, {}
        gen = _generator(seed, 4)
        for gid in sum(need, []):
            blob = _blobs(c, 1, gen)[0].cpu()
            s.payload[gid] = (blob.pin_memory() if c["pinned"] else blob).numpy()
    else:
        gen, at_once = _generator(seed, 4), 32
        for g0 in range(0, n_ids, at_once):
            n = min(at_once, n_ids - g0)
            blobs = _blobs(c, n, gen)
            torch.cuda.synchronize()
            for i in range(n):
                b.admit_device(g0 + i, 1, blobs[i].data_ptr(), eb, wait=False)
            b.synchronize()
    if c["kind"] in ("host", "step"):
        s.x = [x.cpu().numpy() for x in s.x]
    return s


def run(state):
    s, c = state, state.case
    b, T, kind = getattr(s, "backend", None), c["tokens"], c["kind"]
    if kind == "host":
        return [b.moe_layer_forward(l, x) for l, x in enumerate(s.x)]
    if kind == "step":
        outs = []
        for l, x in enumerate(s.x):
            choice = s.gates[l].route(x[0])
            outs.append(b.moe_step_weighted_into(l, x[0], choice.experts + np.uint32(l * c["experts"]), choice.weights))
        return outs
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "expert":
        for blob, x, out in zip(s.blobs, s.x, s.out):
            mer_b200.expert_forward_noalloc(s.dtype, c["d_model"], c["d_ff"], blob.data_ptr(), x.data_ptr(), T, out.data_ptr(), 0.0, stream)
        return s.out
    for l in range(c["layers"]):
        if kind == "miss":
            for gid in s.need[l]:
                if s.cache.get(gid)[0] == mer_b200.GpuLookup.Miss:
                    b.demand_admit(s.cache, gid, s.payload[gid])
        b.moe_layer_forward_device(l, s.x[l].data_ptr(), T, s.out[l].data_ptr(), stream)
    return s.out
