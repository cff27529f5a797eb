"""The C-ABI library loads and exports every symbol that the headers under include/ declare. No GPU needed: nothing is
launched."""
import ctypes
import os
import re

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    inc = os.path.join(ROOT, "include")
    text = "".join(open(os.path.join(inc, f)).read() for f in sorted(os.listdir(inc)) if f.endswith(".h"))
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(es_[a-z0-9_]+)\s*\(", text)))


def test_library_builds_and_exports_the_header():
    from self_trainable_or_free_attn_b200 import build
    lib = ctypes.CDLL(build.build())
    names = declared_symbols()
    assert len(names) >= 17
    for name in names:
        assert hasattr(lib, name), f"{name} is declared in the header but not exported"


def test_binding_covers_the_header():
    from self_trainable_or_free_attn_b200 import _native
    assert sorted(_native.SIGNATURES) == declared_symbols()
    lib = _native.load()
    assert lib.es_abi_version() == 1
    assert lib.es_reps_gram_splits(75600) == 32 and lib.es_reps_gram_splits(0) == 0


def test_argument_checks_come_before_any_launch():
    """Rejected calls return a negative code and a message; none of these reaches a kernel."""
    from self_trainable_or_free_attn_b200 import _native
    lib = _native.load()
    before = _native.launch_count()
    assert lib.es_block_means(None, None, None, None, 128, 1, None) < 0
    assert "null" in _native.last_error()
    assert lib.es_select_blocks(None, None, None, None, None, None, None, None, None, 4, None, 0, 1, 0, 128, 1, 1 << 30,
                                None) < 0
    assert lib.es_pack_plan(ctypes.c_void_p(16), ctypes.c_void_p(16), 1, 1, 1, 64, None) < 0     # 32 bits < 64 blocks
    assert "bits" in _native.last_error()
    assert _native.launch_count() == before


# entry point -> arguments by value, with P for a pointer; one (argument index, bytes) per pointer that a kernel accesses in pieces
# larger than its elements.
P = "P"
ALIGNED = {
    "es_block_means": ([P, P, P, P, 128, 1, None], [(0, 16), (1, 16)]),
    "es_estimate_skipped": ([P] * 8 + [128, 1, None], [(0, 4), (1, 16)]),
    "es_sparse_attention": ([P, P, P, P, P, P, 4, P, P, P, 2, P, P, P, P, 32, P, P, P, None, 128, 1, 60.0, None], [(14, 16), (18, 16)]),
    "es_reps_metric": ([P, P, P, P, P, 128, 1, None], [(0, 16), (1, 16), (3, 16)]),
    "es_reps_metric_static": ([P, P, P, P, 128, 1, None], [(0, 16), (2, 16)]),
    "es_reps_kmeans": ([P] * 9 + [128, 1, 6, None], [(0, 16), (1, 16), (2, 16), (3, 4), (4, 4), (5, 4), (7, 4), (8, 4)]),
    "es_vsa_pool": ([P] * 10 + [1, 128, 64, 16, 64, 64, 0, None], [(i, 4) for i in range(9)]),
    "es_vsa_router_lse": ([P] * 4 + [1, 2, 64, 16, 64, 0, None], [(0, 16), (1, 16)]),
    "es_vsa_router_scores": ([P] * 5 + [1, 2, 64, 16, 64, 0, 1, 1, 0, None], [(0, 16), (1, 16)]),
    "es_vsa_block_scores": ([P] * 3 + [1, 2, 64, 64, 0, 1, 0, None], [(0, 4), (1, 4)]),
    "es_vsa_fuse_fwd": ([P] * 5 + [1, 128, 64, 64, 2, 0, 0, None], [(i, 4) for i in range(4)]),
    "es_vsa_fuse_bwd": ([P] * 10 + [1, 128, 64, 64, 2, 0, 0, None], [(i, 4) for i in (0, 1, 2, 3, 4, 6, 8)]),
    "es_vsa_finalize": ([P] * 4 + [1, 128, 64, 64, 0, None], [(2, 4)]),
    "es_vsa_split_merge_fwd": ([P] * 4 + [1, P, P, P, 128, 64, 1, 0, None], [(0, 16), (2, 16), (6, 8)]),
    "es_vsa_split_merge_sum": ([P] * 3 + [1, P, 64, P, P, P, 128, 64, 0, None], [(0, 16), (1, 16), (4, 16), (7, 8), (8, 16)]),
    "es_vsa_attn_fwd": ([P] * 8 + [1, 128, 64, 0, None], [(3, 4)]),
    "es_vsa_attn_fwd_tasks": ([P] * 9 + [2, P, P, 1, 128, 64, 0, None], [(3, 4), (7, 16), (10, 8)]),
    "es_vsa_attn_bwd_kv": ([P] * 12 + [64, P, P, P, 1, 128, 64, 0, None], [(6, 4), (7, 4), (8, 8), (9, 8)]),
    "es_vsa_attn_bwd_q": ([P] * 9 + [64, P, P, P, 1, 128, 64, 0, None], [(6, 4), (7, 8)]),
    "es_vsa_coarse_fwd": ([P] * 5 + [1, 64, 2, 64, 0, None], [(3, 4)]),
    "es_vsa_coarse_bwd": ([P] * 9 + [1, 64, 2, 64, 0, None], [(7, 8), (8, 8)]),
    "es_vsa_tier_attn_fwd": ([P] * 14 + [1, 128, 64, 4, 64, 64, 7, 0, None], [(7, 4)]),
    "es_vsa_tier_attn_bwd_q": ([P] * 12 + [64] + [P] * 5 + [1, 128, 64, 4, 64, 64, 7, 0, None], [(10, 4)]),
    "es_vsa_tier_rep_bwd": ([P] * 15 + [1, 128, 64, 4, 64, 64, 7, 0, None], [(i, 8) for i in (8, 9, 10, 11)]),
    "es_vsa_tier_unpool": ([P] * 4 + [64, P, P, 1, 128, 64, 4, 64, 64, 0, None], [(5, 4)]),
}


@pytest.mark.skipif(torch.cuda.is_available(), reason="the pointers are made up: without a GPU no call can reach a kernel with them")
@pytest.mark.parametrize("name", sorted(ALIGNED))
def test_pointers_that_vector_accesses_could_not_take_are_refused(name):
    """A pointer between the multiples its kernel needs (a contiguous view that starts at an odd element) would fault the GPU. At
    the multiple itself the call gets past the checks, as far as a machine without a GPU lets it: nothing more is refused."""
    from self_trainable_or_free_attn_b200 import _native
    args, needs = ALIGNED[name]
    fn = getattr(_native.load(), name)
    where = [0x10000 * (i + 1) if a == P else a for i, a in enumerate(args)]
    rc = fn(*where)
    assert rc < -1, (rc, _native.last_error())                       # only the missing GPU
    for i, bytes_ in needs:
        assert args[i] == P
        for off in {2 if bytes_ == 4 else 4, bytes_ // 2}:
            assert fn(*where[:i], where[i] + off, *where[i + 1:]) == -1, (i, off)
            assert "aligned" in _native.last_error()
        assert fn(*where[:i], where[i] + bytes_, *where[i + 1:]) == rc, (i, _native.last_error())


def test_missing_library_fails_loudly(monkeypatch):
    from self_trainable_or_free_attn_b200 import _native
    monkeypatch.setattr(_native, "_lib", None)
    monkeypatch.setattr(_native, "LIB_PATH", "/nonexistent/libechosparse_sm100.so")
    with pytest.raises(_native.NativeError, match="no CPU or Triton fallback"):
        _native.load()
