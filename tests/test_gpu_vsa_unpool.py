"""Gradients of the representatives spread over their tokens: vector accesses where all tensors are aligned, single ones elsewhere."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("mid_reps", [2, 4, 16])
def test_unaligned_tensors_give_the_same_bits(D, dtype, mid_reps):
    """Every source absent in turn, every tensor in turn (and all) 4 bytes past an aligned place: the same sums in the same order, so the
    same bits. The aligned one against float64: four float32 terms and one rounding to the element type, u = 2^-8 (bf16) or 2^-11 of
    the value, 2^-22 of the largest for the sums."""
    from self_trainable_or_free_attn_b200 import _native as N
    lib = N.load()
    BH, nb = 3, 5
    g = torch.Generator(device=DEV).manual_seed(D + mid_reps)
    cnt = torch.tensor([64, 1, 33, 64, 17], device=DEV, dtype=torch.int32)
    R, ms, ts = 64 // mid_reps, -(-nb * mid_reps // 64) * 64, 64
    shapes = {"tok": (BH, nb * 64, D), "mid": (BH, ms, D), "tail": (BH, ts, D), "add": (BH, nb + 2, D)}

    def place(x, off):                                    # a copy of x that starts `off` elements into aligned memory
        buf = torch.empty(x.numel() + 8, device=DEV, dtype=x.dtype)
        buf[off:off + x.numel()] = x.reshape(-1)
        return buf[off:off + x.numel()]

    src = {n: torch.randn(s, device=DEV, generator=g) for n, s in shapes.items()}

    def run(present, off):
        t = {n: place(src[n], off.get(n, 0)) if n in present else None for n in src}
        out = place(torch.full((BH, nb * 64, D), 7.0, device=DEV, dtype=dtype), off.get("out", 0))
        N.check(lib.es_vsa_tier_unpool(N.ptr(t["tok"]), N.ptr(t["mid"]), N.ptr(t["tail"]), N.ptr(t["add"]), nb + 2, out.data_ptr(),
                                       cnt.data_ptr(), BH, nb * 64, D, mid_reps, ms, ts, 0 if dtype == torch.bfloat16 else 1,
                                       N.stream_ptr()), "unpool")
        return out.reshape(BH, nb * 64, D)

    r = torch.arange(64, device=DEV)
    valid = (r[None] < cnt[:, None]).reshape(-1)
    per = (cnt[:, None] - (r[None] // R) * R).clamp(0, R).reshape(-1).clamp(min=1).double()      # tokens of the row's group
    group = (torch.arange(nb, device=DEV)[:, None] * mid_reps + r[None] // R).reshape(-1)
    block = torch.arange(nb, device=DEV).repeat_interleave(64)
    for absent in (None, "tok", "mid", "tail", "add"):
        present = set(src) - {absent}
        got = run(present, {})
        want = torch.zeros(BH, nb * 64, D, device=DEV, dtype=torch.float64)
        for n in present:
            x = src[n].double()
            want += x if n == "tok" else x[:, group] / per[None, :, None] if n == "mid" else x[:, block] / cnt[block].double()[None, :, None]
        want *= valid[None, :, None]
        u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
        assert ((got.double() - want).abs() <= u * want.abs() + 2.0 ** -22 * float(want.abs().max())).all()
        step = {"out": 2, **{n: 1 for n in src}}
        for off in [{n: step[n]} for n in (*present, "out")] + [step]:
            assert torch.equal(run(present, off), got), (absent, off)
