"""Calls on a stream of their own and in a captured graph: the same bits as on the default stream, for new inputs as well."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _dense(L, H):
    """Cut tiles: scratch of the call, and a second kernel that may begin before the first has ended."""
    from self_trainable_or_free_attn_b200 import _native as N, backends
    K = backends.kernels(backends.resolve("auto", DEV))
    assert N.load().es_dense_scratch_bytes(L, H) > 0
    draw = lambda seed: torch.randn(3, L, H, 128, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed)).to(torch.bfloat16)

    def call(x):
        out, lse = torch.empty_like(x[0]), torch.empty(-(-L // 128) * 128, H, device=DEV)
        K.dense_attention(x[0], x[1], x[2], out, lse)
        return out, lse
    return draw, call


def _vsa2(nb, H):
    from self_trainable_or_free_attn_b200 import vsa
    cnt = torch.full((nb,), 64, device=DEV, dtype=torch.int32)
    cnt[1] = 17
    draw = lambda seed: torch.randn(3, 1, H, nb * 64, 128, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed)).to(torch.bfloat16)
    return draw, lambda x: (vsa.vsa2_attention(x[0], x[1], x[2], None, cnt, R=16, topk=3),)


@pytest.mark.parametrize("make", [lambda: _dense(1560, 12), lambda: _dense(4096, 1), lambda: _vsa2(24, 3)], ids=["dense1560", "dense4096", "vsa2"])
def test_side_stream_and_graph(make):
    from self_trainable_or_free_attn_b200 import _native as N
    draw, call = make()
    first, second = draw(0), draw(1)
    want = [call(x) for x in (first, second)]
    torch.cuda.synchronize()
    # the inputs arrive late on the side stream: behind copies that take far longer than the launch of the calls
    side, x = torch.cuda.Stream(), torch.zeros_like(first)
    big = torch.empty(1 << 28, device=DEV, dtype=torch.uint8)
    torch.cuda.synchronize()
    got = []
    with torch.cuda.stream(side):
        for src in (first, second):
            for _ in range(8):
                big.copy_(big.flip(0))
            x.copy_(src)
            got.append([t.clone() for t in call(x)])
    side.synchronize()
    for a, b in zip(got, want):
        assert all(torch.equal(s, t) for s, t in zip(a, b))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call(x)
    for src, w in ((first, want[0]), (second, want[1]), (first, want[0])):
        x.copy_(src)
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(s, t) for s, t in zip(out, w))
    assert N.device_status() == 0
