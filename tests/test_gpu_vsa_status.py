"""A VSA2 kernel that starts while the device status word is set (a wait of an earlier kernel gave up) leaves NaN in everything it
owns, vsa.check_status raises and clears the word, and the same calls then give the same bits as before. The wait that runs out is
the library's self test: a barrier nobody arrives on, for 2 ms."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,dtype", [(64, torch.float16), (128, torch.bfloat16)])
def test_outputs_are_nan_until_the_word_is_read(D, dtype):
    from self_trainable_or_free_attn_b200 import _native as N, vsa as V
    from self_trainable_or_free_attn_b200.vsa import tiers as T
    nb = 9
    g = torch.Generator().manual_seed(0)
    q, k, v, do = [torch.randn(1, 2, nb * 64, D, generator=g).to(dtype).cuda() for _ in range(4)]
    cnt = torch.full((nb,), 64, dtype=torch.int32).cuda()
    mask = torch.rand(1, 2, nb, nb, generator=g) < 0.6
    mask[0, 0, 1] = False
    sel = V.mask_to_selection(mask.cuda())
    tsel = T.selection_from_masks(mask.cuda(), (torch.rand(1, 2, nb, nb, generator=g) < 0.5).cuda())
    calls = [lambda *x: V.fine_block_sparse_attention(*x, cnt, sel)[0],
             lambda *x: V.fine_block_sparse_attention(*x, cnt, sel, split_kv=V.SplitKV(chunk=2))[0],
             lambda *x: V.vsa2_attention(*x, None, cnt, selection=sel),
             lambda *x: V.rep_fine_attention(*x, cnt, tsel, mid_reps=4)[0]]

    def run():
        outs = []
        for f in calls:
            x = [t.clone().requires_grad_(True) for t in (q, k, v)]
            o = f(*x)
            outs.append([o.detach(), *torch.autograd.grad(o, x, do)])
        return outs

    V.check_status()
    good = run()
    assert all(torch.isfinite(t).all() for outs in good for t in outs)
    N.check(N.load().es_selftest_wait_timeout(2000, N.stream_ptr()), "selftest")
    for i, outs in enumerate(run()):
        for j, t in enumerate(outs):
            assert torch.isnan(t).all(), (i, j)
    with pytest.raises(N.NativeError, match="status 777"):
        V.check_status()
    V.check_status()
    for a, b in zip(good, run()):
        assert all(torch.equal(x, y) for x, y in zip(a, b))
    V.check_status()
