"""The work that a user of this library has it do, as cases that can be timed and compared.

Three families, all through the public entry points:

  sparse   one sparse denoising step of one attention layer of a video-diffusion transformer, every CFG branch of it,
           through `EchoSparseAttention.__call__`: the call that runs 40 of 50 steps of a video in all but the first layer
  dense    the calls of the same processor that attend to everything: a layer that always runs dense, a dense step that
           follows another one, and sequences too short for the sparse path
  vsa      the VSA2 operator of `vsa`: routed attention, forward (inference) or forward and backward (training), the
           split-KV scheduling of skewed selections, and the fine branch with 64 / RM / 1 representative tiers

A state holds what a program keeps between calls: the processor with the plan and the LSE of the steps before, the
activations, the block layout. Inputs are made on the GPU from the seed alone.
"""
import math

import torch

from self_trainable_or_free_attn_b200 import EchoSparseAttention
from self_trainable_or_free_attn_b200 import vsa

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
LAYER = 7                      # any layer that is not one of `dense_layers`
MOST_FLOPS = 31e12             # no drawn case computes more than the largest listed one


# ------------------------------------------------------------------------------------------------------------ the cases
def _sparse(name, grid, heads, branches, density, text=0, flagged=0.005):
    return dict(name=name, kind="sparse", t=grid[0], h=grid[1], w=grid[2], heads=heads, branches=branches,
                density=density, text=text, flagged=flagged)


def _dense(name, mode, grid, heads, branches=1):
    return dict(name=name, kind="dense", mode=mode, t=grid[0], h=grid[1], w=grid[2], heads=heads, branches=branches)


def _vsa(name, mode, grid, heads, topk, batch=1, dim=128, dtype="bf16", gate="token", R=16, backward=True, skew="routed",
         split=False):
    return dict(name=name, kind="vsa", mode=mode, t=grid[0], h=grid[1], w=grid[2], batch=batch, heads=heads, dim=dim,
                dtype=dtype, gate=gate, R=R, topk=topk, backward=backward, skew=skew, split=split)


def listed():
    return [
        # the headline: one layer of Wan2.1-14B at 720p, both CFG branches, 10 % of the blocks kept, and half a percent of
        # the query tiles whose logits moved so far since the last step that they are recomputed
        _sparse("sparse_wan14b_720p", (21, 45, 80), 40, 2, 0.10),
        # the small model of the family at 480p: 32,760 tokens (not a multiple of 64), 15 % kept
        _sparse("sparse_wan1.3b_480p", (21, 30, 52), 12, 2, 0.15),
        # joint video and text attention: one forward per step, 256 text tokens behind the video as a sink every tile
        # computes exactly, the longest sequence of the presets
        _sparse("sparse_hunyuan_720p", (33, 45, 80), 24, 1, 0.12, text=256),
        # the shortest sequences that run sparse (65 blocks, ragged): host path, launches and latencies
        _sparse("sparse_4152_tokens", (1, 8, 519), 2, 1, 0.10),
        # a dense step that follows another dense step (steps 1 .. 8 of 50): every block at the previous step's LSE
        _dense("dense_step_wan1.3b", "step", (21, 30, 52), 12, 2),
        # a layer that always runs dense (the first layer in the presets, every step), and the first step of a video
        _dense("dense_layer_wan1.3b", "layer", (21, 30, 52), 12, 1),
        # one latent frame at 480p: shorter than the sparse path takes, so every step and layer runs like this
        _dense("dense_1560_tokens", "layer", (1, 30, 52), 12, 1),
        # training: one layer of 32,768 tokens, the router and the exact top-k on every call, forward and backward
        _vsa("vsa2_train_32k", "routed", (16, 32, 64), 12, 32),
        # inference on a ragged latent grid (edge tiles of 8 to 64 tokens), no gradients
        _vsa("vsa2_infer_wan1.3b", "routed", (21, 30, 52), 12, 64, gate="elem", backward=False),
        # a small ragged training step in fp16 with head dim 64 and two samples: launches and host work count
        _vsa("vsa2_small_fp16", "routed", (5, 18, 22), 4, 8, batch=2, dim=64, dtype="fp16", gate="none", R=8),
        # a frozen, skewed selection (10 % of the query blocks hold four times as many pairs) with the split-KV planner
        _vsa("vsa2_split_skewed", "frozen", (16, 32, 64), 12, 32, skew="tenth_x4", split=True),
        # the fine branch that keeps dropped blocks as 4 group means or 1 block mean: routing, forward and backward
        _vsa("vsa2_tiers_32k", "tiers", (16, 32, 64), 12, 32, gate="none"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, tokens):
    t = rng.randint(1, 33)
    h = max(2, int(round(math.sqrt(tokens / t) * rng.uniform(0.5, 1.0))))
    return t, h, max(2, round(tokens / (t * h)))


def draw(rng):
    while True:
        kind = rng.choice(["sparse", "sparse", "dense", "vsa", "vsa", "vsa"])
        if kind == "sparse":
            grid = _grid(rng, _log_int(rng, 4200, 120000))
            c = _sparse("", grid, _log_int(rng, 1, 40), rng.randint(1, 2), round(rng.uniform(0.05, 0.2), 3),
                        text=rng.choice([0, 0, rng.randint(1, 400)]), flagged=rng.choice([0.0, 0.005]))
            if _tokens(c) < 4096 + 64 or _tokens(c) > 125000:
                continue
        elif kind == "dense":
            c = _dense("", rng.choice(["step", "layer"]), _grid(rng, _log_int(rng, 256, 34000)), _log_int(rng, 1, 40),
                       rng.randint(1, 2))
        else:
            mode = rng.choice(["routed", "routed", "frozen", "tiers"])
            grid = _grid(rng, _log_int(rng, 2000, 66000))
            nb = _blocks(grid)
            c = _vsa("", mode, grid, _log_int(rng, 1, 24), min(_log_int(rng, 4, 96), max(1, nb // 4)), batch=rng.randint(1, 2),
                     dim=rng.choice([64, 128, 128]), dtype=rng.choice(["bf16", "bf16", "fp16"]),
                     gate=rng.choice(["token", "elem", "none"]) if mode != "tiers" else "none",
                     R=rng.choice([8, 16, 16, 32]), backward=rng.random() < 0.7,
                     skew=rng.choice(["even", "tenth_x4"]) if mode == "frozen" else "routed", split=rng.random() < 0.4 and mode != "tiers")
            if nb > 1600:
                continue
        del c["name"]
        if work(c)["flops"] <= MOST_FLOPS:
            return c


# ------------------------------------------------------------------------------------------------------------ sizes
def _tokens(c):
    return c["t"] * c["h"] * c["w"] + c.get("text", 0)


def _blocks(grid):
    t, h, w = grid
    return -(-t // 4) * -(-h // 4) * -(-w // 4)


def work(case):
    c = case
    if c["kind"] in ("sparse", "dense"):
        L, n = _tokens(c), c["heads"] * c["branches"]
        nb = -(-L // 64)
        if c["kind"] == "dense" or nb < 64:
            cols = L
        else:
            # columns of a query row: tokens of the exact blocks, one mean per skipped block, four representatives for the
            # most probable third of those
            top = max(1, round(c["density"] * nb))
            refined = round((nb - top) / 3)
            cols = top * 64 + c["text"] + (nb - top - refined) + 4 * refined
        return dict(bytes=float(4 * L * n * 256 + 2 * L * n * 4), flops=4.0 * 128 * L * cols * n)
    nb, D, bh = _blocks((c["t"], c["h"], c["w"])), c["dim"], c["batch"] * c["heads"]
    tok = c["t"] * c["h"] * c["w"] * bh * D * 2.0
    pairs = float(nb * min(c["topk"], nb))
    cols = pairs * 64
    if c["mode"] == "tiers":
        mid = 0.2 * nb * nb
        cols += mid * 4 + (nb * nb - pairs - mid)
    flops = 4.0 * 64 * D * cols * bh
    if c["mode"] != "tiers":
        flops += 4.0 * nb * nb * D * bh                              # the coarse branch
    gate = {"none": 0.0, "token": tok / D, "elem": tok}[c["gate"]]
    nbytes = 4 * tok + gate                                          # q, k, v, gate in, o out
    if c["backward"]:
        flops *= 3.5
        nbytes += 4 * tok + gate                                     # dO in, dq, dk, dv, dgate out
    if c["mode"] in ("routed", "tiers"):
        flops += 2.0 * (nb * (64 // c["R"])) ** 2 * D * bh           # the router's logits
    return dict(bytes=nbytes, flops=flops)


# ------------------------------------------------------------------------------------------------------------ inputs
def _video_qkv(c, gen, branches):
    """q, k, v of every branch, [1, L, H, 128] bf16: unit noise plus a smooth component per head through a random
    projection each, so that attention is biased to near-by tokens; text tokens are noise."""
    grid, H = (c["t"], c["h"], c["w"]), c["heads"]
    n, L = grid[0] * grid[1] * grid[2], _tokens(c)
    ax = torch.meshgrid(*[torch.arange(s, device=DEV, dtype=torch.float32) / s for s in grid], indexing="ij")
    pos = torch.stack(ax, -1).reshape(n, 3)
    out = [[torch.empty(1, L, H, 128, device=DEV, dtype=torch.bfloat16) for _ in range(3)] for _ in range(branches)]
    for head in range(H):
        smooth = torch.zeros(n, 128, device=DEV)
        for _ in range(4):
            f = torch.randint(0, 4, (3, 128), device=DEV, generator=gen).float()
            phase = torch.rand(128, device=DEV, generator=gen)
            smooth += torch.cos(2 * math.pi * (pos @ f + phase))
        w = torch.randn(128, 384, device=DEV, generator=gen) / math.sqrt(128.0)
        for b in range(branches):
            base = torch.randn(n, 128, device=DEV, generator=gen).add_(smooth, alpha=1.5)
            x = base @ w
            for i in range(3):
                out[b][i][0, :n, head] = x[:, 128 * i: 128 * i + 128]
                if L > n:
                    out[b][i][0, n:, head] = torch.randn(L - n, 128, device=DEV, generator=gen)
    return out


def _moved(x, gen, by=0.02):
    """The same activations one denoising step away."""
    return x + by * torch.randn(x.shape, device=DEV, generator=gen, dtype=x.dtype)


def _with_jumps(q, share, gen):
    """q with a share of its 128-row tiles scaled three times: tiles whose logits moved far since the last step."""
    L, H = q.shape[1], q.shape[2]
    nq = -(-L // 128)
    jump = (torch.rand(nq, H, device=DEV, generator=gen) < share).repeat_interleave(128, 0)[:L]
    return torch.where(jump[None, :, :, None], q * 3.0, q)


def _prepare_video(c, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    qkv = _video_qkv(c, gen, c["branches"])
    sink = None
    if c["kind"] == "sparse":
        attn = EchoSparseAttention(density=c["density"], dense_steps=2, dense_layers=())
        sink = c["t"] * c["h"] * c["w"] // 64 if c["text"] else None
    else:
        attn = EchoSparseAttention(dense_steps=1 << 20, dense_layers=(LAYER,) if c["mode"] == "layer" else ())
    calls, first = [], 0
    if c["kind"] == "sparse" or c["mode"] == "step":
        # the steps before: the processor's plan and LSE come from activations one step away
        first = 2 if c["kind"] == "sparse" else 1
        for step in range(first):
            for b, (q, k, v) in enumerate(qkv):
                attn(_moved(q, gen), _moved(k, gen), v, step, b, LAYER, sink=sink)
    for q, k, v in qkv:
        if c["kind"] == "sparse":
            calls.append(([_with_jumps(q, c["flagged"], gen), _with_jumps(_moved(q, gen), c["flagged"], gen)], k, v))
        else:
            calls.append(([q, _moved(q, gen)], k, v))
    return dict(kind=c["kind"], attn=attn, calls=calls, step=first, sink=sink, tokens=_tokens(c))


def _frozen_selection(c, gen):
    """A random-but-local selection: Gaussian of the distance between tiles times U(0, 1), nb * topk pairs per head, the
    list lengths even or with a tenth of the query blocks four times as long."""
    dims = [-(-c[a] // 4) for a in ("t", "h", "w")]
    nb, bh = dims[0] * dims[1] * dims[2], c["batch"] * c["heads"]
    ax = torch.meshgrid(*[torch.arange(s, device=DEV, dtype=torch.float32) for s in dims], indexing="ij")
    pos = torch.stack(ax, -1).reshape(nb, 3)
    score = torch.exp(-torch.cdist(pos, pos).square() / 18.0) * torch.rand(bh, nb, nb, device=DEV, generator=gen)
    total = nb * c["topk"]
    length = torch.full((bh, nb), c["topk"], device=DEV, dtype=torch.long)
    if c["skew"] == "tenth_x4" and nb >= 20:
        n_long = round(0.1 * nb)
        long_len = min(4 * c["topk"], nb)
        rest, extra = divmod(total - n_long * long_len, nb - n_long)
        row = torch.full((nb,), rest, device=DEV, dtype=torch.long)
        row[:n_long] = long_len
        row[n_long: n_long + extra] += 1
        order = torch.rand(bh, nb, device=DEV, generator=gen).argsort(1)
        length = row[order]
    rank = score.sort(dim=2, descending=True, stable=True).indices.argsort(2)
    return vsa.mask_to_selection((rank < length[:, :, None]).view(c["batch"], c["heads"], nb, nb))


def _prepare_vsa(c, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    grid, B, H, D, dt = (c["t"], c["h"], c["w"]), c["batch"], c["heads"], c["dim"], DTYPES[c["dtype"]]
    lay = vsa.build_layout(grid, R=c["R"], device=DEV)
    n = grid[0] * grid[1] * grid[2]
    ax = torch.meshgrid(*[torch.arange(s, device=DEV, dtype=torch.float32) / s for s in grid], indexing="ij")
    pos = torch.stack(ax, -1).reshape(n, 3)
    leaves = []
    for _ in range(3):
        f = torch.randn(4, 3, device=DEV, generator=gen) * 2.0
        phase = torch.rand(4, D, device=DEV, generator=gen)
        smooth = torch.cos(2 * math.pi * ((pos @ f.t())[:, :, None] + phase)).sum(1) * 0.75
        x = torch.randn(B, H, n, D, device=DEV, generator=gen).add_(smooth)
        leaves.append(vsa.to_blocked(x.to(dt), lay).contiguous())
    gate = None
    if c["gate"] != "none":
        shape = (B, H, n) if c["gate"] == "token" else (B, H, n, D)
        gate = vsa.to_blocked((torch.randn(shape, device=DEV, generator=gen) * 1.5).to(dt), lay).contiguous()
    s = dict(kind="vsa", mode=c["mode"], cnt=lay.blk_cnt, R=c["R"], topk=c["topk"], backward=c["backward"],
             split="auto" if c["split"] else None, sel=None)
    if c["backward"]:
        s["dout"] = vsa.to_blocked(torch.randn(B, H, n, D, device=DEV, generator=gen).to(dt), lay).contiguous()
        for x in leaves + ([gate] if gate is not None else []):
            x.requires_grad_(True)
    if c["mode"] == "frozen":
        s["sel"] = _frozen_selection(c, gen)
    if c["mode"] == "tiers":
        nb = lay.num_blocks
        s["tiers"] = vsa.RepTiers(frac_full=c["topk"] / nb, frac_mid=min(0.2, 1.0 - c["topk"] / nb), mid_reps=4)
    return dict(s, q=leaves[0], k=leaves[1], v=leaves[2], gate=gate)


def prepare(case, seed):
    return _prepare_vsa(case, seed) if case["kind"] == "vsa" else _prepare_video(case, seed)


# ------------------------------------------------------------------------------------------------------------ one pass
def _run_video(s):
    """One denoising step of one layer: every branch's output, and the log2 LSE that the step leaves for the next one."""
    attn, step = s["attn"], s["step"]
    s["step"] += 1
    out = [attn(q[step & 1], k, v, step, b, LAYER, sink=s["sink"]) for b, (q, k, v) in enumerate(s["calls"])]
    # rows past the sequence's end hold a constant and belong to no token
    return dict(out=out, lse=[attn._states[(b, LAYER)].offset[: s["tokens"]] for b in range(len(out))
                              if (b, LAYER) in attn._states])


def _forward_vsa(s):
    if s["mode"] == "tiers":
        sel = vsa.route_tiers(s["q"], s["k"], s["cnt"], s["tiers"], R=s["R"])
        return vsa.rep_fine_attention(s["q"], s["k"], s["v"], s["cnt"], sel, mid_reps=s["tiers"].mid_reps)[0]
    return vsa.vsa2_attention(s["q"], s["k"], s["v"], s["gate"], s["cnt"], R=s["R"], topk=s["topk"], selection=s["sel"],
                              split_kv=s["split"])


def _run_vsa(s):
    if not s["backward"]:
        with torch.no_grad():
            return dict(o=_forward_vsa(s))
    leaves = [x for x in (s["q"], s["k"], s["v"], s["gate"]) if x is not None]
    o = _forward_vsa(s)
    return dict(o=o, grads=torch.autograd.grad(o, leaves, s["dout"]))


def run(state):
    return _run_vsa(state) if state["kind"] == "vsa" else _run_video(state)


# ------------------------------------------------------------------------------------------------------------ tolerance
def tolerance(case):
    # P (and dS in the backward) enter their products as bf16 / fp16 and outputs are stored in that type. Measured: every
    # path against itself with the blocks in another order, or with another LSE offset (other roundings of every P), differs
    # by 1.1e-3 to 2.6e-3 (bf16), 2.5e-4 (fp16), in single values by up to 0.12 of the root mean square (gradients). A block
    # whose score ties at the cut may be chosen or not: on 4152 to 119,056 tokens that moved single rows by up to 0.6.
    if case.get("dtype") == "fp16":
        return {"rel": 2e-3, "max": 0.3}
    return {"rel": 1e-2, "max": 0.5}


# ------------------------------------------------------------------------------------------------------------ 64 bits
MOST_EXACT_FLOPS = 1.2e14      # beyond this the 64-bit computation takes too long


def _exact_dense(c, seed):
    """Softmax attention of the first pass's inputs over every token, and its log2 LSE where the step leaves one."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    qkv = _video_qkv(c, gen, c["branches"])
    if c["mode"] == "step":
        for q, k, _ in qkv:                                          # the step before
            _moved(q, gen), _moved(k, gen)
    out, lse = [], []
    for q, k, v in qkv:
        moved = _moved(q, gen)
        q = moved if c["mode"] == "step" else q
        o = torch.empty(q.shape, device=DEV, dtype=torch.float64)
        l2 = torch.empty(q.shape[1:3], device=DEV, dtype=torch.float64)
        for h in range(q.shape[2]):
            kh, vh = k[0, :, h].double(), v[0, :, h].double()
            for r in range(0, q.shape[1], 4096):
                s = q[0, r: r + 4096, h].double() @ kh.t() / math.sqrt(128.0)
                l = torch.logsumexp(s, 1)
                l2[r: r + 4096, h] = l / math.log(2.0)
                o[0, r: r + 4096, h] = s.sub_(l[:, None]).exp_() @ vh
        out.append(o)
        lse.append(l2)
    keeps = c["mode"] == "step" and -(-_tokens(c) // 64) >= 64
    return dict(out=out, lse=lse if keeps else [])


def _exact_frozen(c, seed):
    """Fine attention over the selected blocks plus tanh(gate) (1 without a gate) times the attention of the block means,
    and the gradients; one (sample, head) and a slab of query blocks at a time."""
    s = _prepare_vsa(c, seed)
    q, k, v, gate, cnt, sel = s["q"], s["k"], s["v"], s["gate"], s["cnt"].long(), s["sel"]
    B, H, L, D = q.shape
    nb = L // 64
    ok = (torch.arange(64, device=DEV)[None] < cnt[:, None]).reshape(L).double()
    leaves = [x for x in (q, k, v, gate) if x is not None]
    o = torch.zeros(B, H, L, D, device=DEV, dtype=torch.float64)
    grads = [torch.zeros(x.shape, device=DEV, dtype=torch.float64) for x in leaves]
    for bh in range(B * H):
        b, h = divmod(bh, H)
        x = [t[b, h].detach().double().requires_grad_(c["backward"]) for t in leaves]
        mean = [(t * ok[:, None]).reshape(nb, 64, D).sum(1) / cnt[:, None] for t in x[:3]]
        coarse = torch.softmax(mean[0] @ mean[1].t() / math.sqrt(D), 1) @ mean[2]
        cut = coarse.detach().requires_grad_(c["backward"])
        ptr = sel.q2k_ptr[b, h].long()
        mask = torch.zeros(nb, nb, device=DEV, dtype=torch.bool)
        mask[torch.repeat_interleave(torch.arange(nb, device=DEV), ptr[1:] - ptr[:-1]),
             sel.q2k_idx[int(ptr[0]): int(ptr[-1])].long()] = True
        for i in range(0, nb, 32):
            r = slice(64 * i, min(64 * (i + 32), L))
            keep = mask[i: i + 32].repeat_interleave(64, 0).repeat_interleave(64, 1) & (ok > 0)[None]
            some = keep.any(1)
            a = (x[0][r] @ x[1].t() / math.sqrt(D)).masked_fill(~keep, -math.inf)
            fine = torch.softmax(a.masked_fill(~some[:, None], 0.0), 1).masked_fill(~some[:, None], 0.0) @ x[2]
            if gate is None:
                w = 1.0
            else:
                w = torch.tanh(x[3][r])
                w = w[:, None] if w.dim() == 1 else w
            y = (fine + w * cut[i: i + 32].repeat_interleave(64, 0)) * ok[r, None]
            o[b, h, r] = y.detach()
            if c["backward"]:
                y.backward(s["dout"][b, h, r].double())
        if c["backward"]:
            coarse.backward(cut.grad)
            for g, t in zip(grads, x):
                g[b, h] = t.grad
    return dict(o=o, grads=grads) if c["backward"] else dict(o=o)


def exact(case, seed):
    """What `run` returns on a fresh state, in 64 bits. A step or a routing whose block choice hangs on rounded scores has no
    such value."""
    c = case
    if c["kind"] == "dense" and 4.0 * 128 * _tokens(c) ** 2 * c["heads"] * c["branches"] < MOST_EXACT_FLOPS:
        return _exact_dense(c, seed)
    if c["kind"] == "vsa" and c["mode"] == "frozen":
        L = 64 * _blocks((c["t"], c["h"], c["w"]))
        if 14.0 * c["dim"] * L ** 2 * c["batch"] * c["heads"] < MOST_EXACT_FLOPS:
            return _exact_frozen(c, seed)
    return None
