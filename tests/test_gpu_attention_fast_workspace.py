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


@pytest.mark.parametrize("B,nq,nkv,T", [(2, 8, 2, 1000), (3, 16, 2, 2100), (56, 16, 16, 1500)])
def test_fewer_splits_where_the_workspace_is_short(cuda_lib, B, nq, nkv, T):
    """Every workspace gives a result, also one just short of another split; splits asked for by the caller still need their room."""
    from tenzo_b200 import kernels
    args, kw = setup(B, nq, nkv, T)
    want = kernels.attention_int8(*args, **kw)
    split = B * nq * 130 * 4                                # partial results of one split
    buf = torch.empty(kernels.attention_workspace_bytes(B, nq, nkv, T) + 16, dtype=torch.uint8, device="cuda")
    for room in (0, 64, split, 2 * split - 1, 2 * split, 3 * split, 4 * split - 4, 8 * split):
        n = min(room, buf.numel() - 16)
        buf.fill_(0x5a)
        got = kernels.attention_int8(*args, **kw, mode=1, workspace=buf[:n])
        torch.cuda.synchronize()
        assert bool((buf[n:] == 0x5a).all())
        assert max(rel_err(host(got[b]), host(want[b])) for b in range(B)) < TOL, f"room {room}"
    kernels.attention_int8(*args, **kw, mode=1, workspace=buf[8:])                                   # off its alignment: not used
    with pytest.raises(RuntimeError, match="rc=-1"):
        kernels.attention_int8(*args, **kw, mode=1, workspace=buf[:split], split_keys=(T + 1) // 2)
    torch.cuda.synchronize()
    assert cuda_lib.tenzo_cuda_attention_take_timeouts() == 0


def test_launches_are_counted(cuda_lib):
    """A step whose attention is one split launches no merge: a kernel fewer a layer than one with several."""
    from helpers import synth
    from tenzo_b200.engine import Engine
    cfg = dict(hidden_size=512, num_q_heads=4, num_kv_heads=2, head_dim=128, num_layers=3, ffn_dim=1536, vocab_size=4096, max_seq_len=512)
    m = synth.SyntheticModel(cfg, seed=5)
    with Engine(m.config_struct(), batch=2, attention_mode=1).load_synthetic(m) as e:
        e.kv_fill_random(400, seed=1)
        n = []
        for length in (100, 400, 100, 400):
            for s in range(2):
                e.set_seq_len(s, length)
            before = e.kernel_launches()
            e.decode_greedy([1, 2], 1)
            n.append(e.kernel_launches() - before)
    assert n[:2] == n[2:] and n[1] - n[0] == cfg["num_layers"]
