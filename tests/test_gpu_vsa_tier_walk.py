"""The walk of a query block over its three tiers at its edges: tier-B lists that are empty, fill units exactly or straddle the
1024-block windows of the bitmaps, every group size, ragged blocks, both head dims. Outputs and dQ of a few query blocks and the
table gradients' sum over tokens against fp64 torch on the GPU. Tolerance: bf16 means, P and dS, 1e-2 of the 2-norm; gradients of
keys 2e-2 (two roundings more)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("RM", [2, 4, 8, 16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("nb", [33, 1100])
def test_tier_walk(RM, D, nb):
    from self_trainable_or_free_attn_b200.vsa import tiers as T
    g = torch.Generator(device="cuda").manual_seed(nb + RM)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    cnt = torch.randint(1, 65, (nb,), device="cuda", generator=g, dtype=torch.int32)
    cnt[::2] = 64
    ok = torch.arange(64, device="cuda")[None] < cnt[:, None]
    L, R, per = nb * 64, 64 // RM, 64 // RM
    q, k, v, do = [(rnd(nb, 64, D) * ok[..., None]).reshape(1, 1, L, D).to(torch.bfloat16) for _ in range(4)]
    # rows with 0, 1, per - 1, per, per + 1 and many tier-B blocks, and a row without tier C
    want_b = [0, 1, per - 1, per, per + 1, nb // 2, nb - 3]
    order = torch.rand(nb, nb, device="cuda", generator=g).argsort(1).argsort(1)
    nb_b = torch.tensor([want_b[i % len(want_b)] for i in range(nb)], device="cuda").clamp(max=nb - 3)
    a = order < 3
    a[0] = False
    b = (order >= 3) & (order < 3 + nb_b[:, None])
    sel = T.selection_from_masks(a[None, None], (a | b)[None, None])
    x = [t.clone().requires_grad_(True) for t in (q, k, v)]
    o, lse = T.rep_fine_attention(*x, cnt, sel, mid_reps=RM)
    only = torch.zeros(nb, 64, 1, device="cuda")
    rows = list(range(min(nb, 15))) + [nb - 1]
    only[rows] = 1
    dout = (do.view(nb, 64, D) * only).reshape(1, 1, L, D).to(torch.bfloat16)
    grads = torch.autograd.grad(o, x, dout)

    kd, vd = (t.double().view(nb, 64, D).detach().requires_grad_(True) for t in (k, v))
    rounded = lambda t: t + (t.to(torch.bfloat16).double() - t).detach()
    mean = lambda t, n: rounded(t.sum(-2) / n.clamp(min=1)[..., None])
    okd = ok.double()
    gc = okd.view(nb, RM, R).sum(-1)
    km, vm = (mean((t * okd[..., None]).view(nb, RM, R, D), gc) for t in (kd, vd))
    kt, vt = (mean(t * okd[..., None], okd.sum(1)) for t in (kd, vd))
    ref_o, ref_q = {}, {}
    for i in rows:
        qi = q[0, 0, 64 * i: 64 * i + 64].double().requires_grad_(True)
        c = ~(a[i] | b[i])
        keys = torch.cat([kd[a[i]][ok[a[i]]], km[b[i]][gc[b[i]] > 0], kt[c]])
        vals = torch.cat([vd[a[i]][ok[a[i]]], vm[b[i]][gc[b[i]] > 0], vt[c]])
        bias = torch.cat([torch.zeros(int(ok[a[i]].sum()), device="cuda", dtype=torch.float64),
                          gc[b[i]][gc[b[i]] > 0].log(), cnt[c].double().log()])
        s = qi @ keys.t() / math.sqrt(D) + bias
        oi = torch.softmax(s, 1) @ vals * ok[i, :, None]
        oi.backward(do.view(nb, 64, D)[i].double(), retain_graph=True)
        ref_o[i], ref_q[i] = oi.detach(), qi.grad
        n = int(cnt[i])
        assert (lse[0, 0, 64 * i: 64 * i + n] - torch.logsumexp(s, 1)[:n]).abs().max() <= 1e-3

    def near(got, exp, tol, what):
        got = got.detach().double()
        assert torch.isfinite(got).all(), what
        assert (got - exp).norm() <= tol * exp.norm(), (what, float((got - exp).norm() / exp.norm()))
    pick = lambda t: torch.stack([t.view(nb, 64, D)[i] for i in rows])
    near(pick(o), torch.stack([ref_o[i] for i in rows]), 1e-2, "o")
    near(pick(grads[0]), torch.stack([ref_q[i] * ok[i, :, None] for i in rows]), 1e-2, "dq")
    near(grads[1].view(nb, 64, D), kd.grad * okd[..., None], 2e-2, "dk")
    near(grads[2].view(nb, 64, D), vd.grad * okd[..., None], 2e-2, "dv")


@pytest.mark.parametrize("RM", [2, 4, 16])
@pytest.mark.parametrize("nb", [1, 33, 64, 97, 130])
def test_tables_that_few_query_blocks_use(RM, nb):
    """The table gradients walk only the query blocks that use a row of the tile: none, one, two, an odd number, at the edges of the
    bitmap's words. Tiers B and C alone, against the CPU restatement in fp64 (tolerances of the module)."""
    from test_gpu_vsa_tiers import oracle_subset
    from self_trainable_or_free_attn_b200.vsa import tiers as T
    g = torch.Generator().manual_seed(nb + RM)
    D = 64
    cnt = torch.randint(1, 65, (nb,), generator=g, dtype=torch.int32)
    ok = (torch.arange(64)[None] < cnt[:, None]).reshape(1, 1, -1, 1)
    q, k, v, do = [(torch.randn(1, 1, nb * 64, D, generator=g) * ok).to(torch.bfloat16) for _ in range(4)]
    b, c = torch.zeros(2, nb, nb, dtype=torch.bool)
    edges = [i for i in (0, 31, 32, 63, 64, nb // 2, nb - 1) if i < nb]
    for j in range(0, nb, 3):                                      # two of three column blocks are in neither tier
        users = [edges[i] for i in torch.randperm(len(edges), generator=g)[: (j // 3) % 4].tolist()]
        (b if (j // 3) % 2 else c)[users, j] = True
    b[0, 0] = True
    a = ~(b | c)
    x = [t.cuda().requires_grad_(True) for t in (q, k, v)]
    o, _ = T.rep_fine_attention(*x, cnt.cuda(), T.selection_from_masks(a[None, None].cuda(), (a | b)[None, None].cuda()), mid_reps=RM,
                                phases=T.PHASE_B | T.PHASE_C)
    grads = torch.autograd.grad(o, x, do.cuda())
    ref = [t.double().requires_grad_(True) for t in (q, k, v)]
    o_ref, _ = oracle_subset(ref, cnt, a[None, None] & False, b[None, None], c[None, None], mid_reps=RM)
    ref_grads = torch.autograd.grad(o_ref, ref, do.double())
    for name, got, exp, tol in zip(("o", "dq", "dk", "dv"), (o, *grads), (o_ref, *ref_grads), (1e-2, 2e-2, 2e-2, 2e-2)):
        got, exp = got.detach().double().cpu(), exp.detach()
        # nb = 1: one group or a few columns only, dq and dk are small differences
        assert (got - exp).norm() <= tol * exp.norm() + (0.3 if nb == 1 else 0.0), (name, float((got - exp).norm() / exp.norm()))
        if nb > 1:
            assert torch.equal((got == 0).all(-1), (exp == 0).all(-1)), name


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("phases", [2, 4])
def test_bias_of_every_token_count(D, phases):
    """With q = 0 and one block of n tokens per list the LSE is ln(n): the bias in fp32, its product with the scale, log2 e undone,
    four roundings (2^-24 each) at most, and three more in the four columns' row sum. dV of that block's tokens is then dO's sum over
    the query block over n: P is 1 (or the groups' shares) in both passes."""
    from self_trainable_or_free_attn_b200.vsa import tiers as T
    nb = 64
    cnt = torch.arange(1, 65, dtype=torch.int32).cuda()
    q = torch.zeros(1, 1, nb * 64, D, device="cuda", dtype=torch.bfloat16)
    k, v, do = (torch.randn_like(q) for _ in range(3))
    eye = torch.eye(nb, dtype=torch.bool)[None, None].cuda()
    sel = T.selection_from_masks(eye & False, eye if phases == 2 else ~eye)
    x = [t.requires_grad_(True) for t in (q, k, v)]
    o, lse = T.rep_fine_attention(*x, cnt, sel, mid_reps=4, phases=phases)
    want = cnt.double().log()
    err = ((lse.view(nb, 64)[:, 0].double() - want).abs() / want.clamp(min=1)).max()
    assert err <= (4 if phases == 4 else 7) * 2.0 ** -24, float(err * 2 ** 24)
    dv = torch.autograd.grad(o, x, do)[2].view(nb, 64, D).double()
    ok = (torch.arange(64, device="cuda")[None] < cnt[:, None]).double()[..., None]
    exp = (do.view(nb, 64, D).double() * ok).sum(1, keepdim=True) / cnt[:, None, None] * ok
    assert (dv - exp).norm() <= 4e-3 * exp.norm()
