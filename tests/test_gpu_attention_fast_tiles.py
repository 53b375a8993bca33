"""Tolerance-mode attention with up to four query heads a kv head: lengths around the ends of a 16-key tile, of a warp's 32-key block
and of the 128 keys of a round, heads that fill the columns and heads that do not, against the exact-order kernel. The bound is
the error of rounding the weights to fp16 (2^-11 each, averaged over the keys; at most that for one key), twice over."""
import pytest
import torch
from gpu_helpers import host
from helpers import rel_err
from test_gpu_attention_fast import random_cache

pytestmark = pytest.mark.gpu
TOL = 2.0 ** -10


@pytest.mark.parametrize("nq,nkv", [(8, 2), (4, 2), (3, 3)])
@pytest.mark.parametrize("split", [0, 128])
def test_tile_edges(cuda_lib, nq, nkv, split):
    from tenzo_b200 import kernels
    lens = [1, 2, 7, 8, 9, 15, 16, 17, 24, 31, 32, 33, 47, 48, 49, 127, 128, 129, 144, 160, 255, 256, 257, 300]
    B, ms = len(lens), 320
    ck, cv, sk, sv = random_cache(B, nkv, ms, 11)
    g = torch.Generator(device="cuda").manual_seed(12)
    q = torch.randn(B, nq * 128, generator=g, device="cuda") * torch.tensor([0.1, 1.0, 6.0], device="cuda")[torch.arange(B, device="cuda") % 3, None]
    pos = torch.tensor(lens, dtype=torch.int32, device="cuda") - 1
    for b in range(B):                                       # keys behind the last are not to be used, whatever they hold
        sk[b, :, :, lens[b]:] = float("nan")
        sv[b, :, :, lens[b]:] = float("inf")
    args = dict(layer=0, n_q=nq, n_kv=nkv, max_seq=ms, max_len=ms, append=False)
    want = kernels.attention_int8(q, None, None, ck, cv, sk, sv, pos, **args)
    got = kernels.attention_int8(q, None, None, ck, cv, sk, sv, pos, mode=1, split_keys=split, **args)
    torch.cuda.synchronize()
    assert cuda_lib.tenzo_cuda_attention_take_timeouts() == 0
    assert torch.isfinite(got).all()
    for b in range(B):
        assert rel_err(host(got[b]), host(want[b])) < TOL, f"length {lens[b]}"
