"""Tolerance-mode attention with less workspace than tenzo_cuda_attention_workspace_bytes gives, or none: nothing is written behind it."""
import pytest
import torch
from gpu_helpers import host
from helpers import rel_err
from test_gpu_attention_fast import random_cache
from test_gpu_attention_fast_tiles import TOL

pytestmark = pytest.mark.gpu


def setup(B, nq, nkv, T):
    ms = (T + 15) // 16 * 16
    g = torch.Generator(device="cuda").manual_seed(T)
    q = torch.randn(B, nq * 128, generator=g, device="cuda")
    pos = torch.tensor([T - 1 - 37 * (b % 3) for b in range(B)], dtype=torch.int32, device="cuda")
    return (q, None, None, *random_cache(B, nkv, ms, 21), pos), dict(layer=0, n_q=nq, n_kv=nkv, max_seq=ms, max_len=T, append=False)


@pytest.mark.parametrize("nq,nkv", [(4, 1), (8, 1)])
@pytest.mark.parametrize("room", [0, 64])
def test_position_outside_with_one_split(cuda_lib, nq, nkv, room):
    """One split keeps no partial results: a refused sequence has none either, in front of the workspace's end or behind it."""
    from tenzo_b200 import kernels
    args, kw = setup(3, nq, nkv, 112)
    good = kernels.attention_int8(*args, **kw, mode=1)
    buf = torch.full((1 << 20,), 0x5a, dtype=torch.uint8, device="cuda")
    for bad in (-1, 112):
        args[-1][1] = bad
        out = kernels.attention_int8(*args, **kw, mode=1, out=torch.full_like(good, 7.0), workspace=buf[:room])
        torch.cuda.synchronize()
        assert cuda_lib.tenzo_cuda_attention_take_timeouts() == 2 and cuda_lib.tenzo_cuda_attention_take_timeouts() == 0
        assert torch.equal(out[0], good[0]) and torch.equal(out[2], good[2]) and bool((out[1] == 7.0).all())
        assert bool((buf == 0x5a).all())
