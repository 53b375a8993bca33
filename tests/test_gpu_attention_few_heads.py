"""Value sums of a few heads (a head and 64 dims a CTA, 256-key chunks in a ring of three), bit for bit against the oracle: lengths around
the ends of the first chunks, fewer chunks than the ring holds and more, contiguous cache and block pools, every head grouping."""
import numpy as np
import pytest
import torch
from gpu_helpers import dev, host
from helpers import ora
from test_gpu_norm_attn_lm import rope_tables
from test_gpu_paged_kv import oracle_paged

pytestmark = pytest.mark.gpu
P = ora.ptr


@pytest.mark.parametrize("nq,nkv", [(8, 2), (4, 4), (40, 10)])
@pytest.mark.parametrize("lens", [[1, 255, 256, 257], [263, 264, 511, 512], [513, 767, 769, 1030], [1281, 1536, 1537, 40]])
def test_few_heads(cuda_lib, nq, nkv, lens):
    from tenzo_b200 import kernels
    O = ora.load_oracle()
    B, ms = len(lens), 1552
    rng = np.random.default_rng([97, nq, lens[0]])
    per_seq = ms // 16
    table = rng.permutation(B * per_seq).astype(np.int32).reshape(B, per_seq)
    ck, cv = (rng.integers(-127, 128, (B, 1, nkv, ms, 128)).astype(np.int8) for _ in range(2))
    sk, sv = ((0.01 + 0.02 * rng.random((B, 1, nkv, ms))).astype(np.float32) for _ in range(2))
    pk, pv = (rng.integers(-127, 128, (B * per_seq, 1, nkv, 16, 128)).astype(np.int8) for _ in range(2))
    psk, psv = ((0.01 + 0.02 * rng.random((B * per_seq, 1, nkv, 16))).astype(np.float32) for _ in range(2))
    q, k, v = (rng.standard_normal((B, h * 128)).astype(np.float32) for h in (nq, nkv, nkv))
    cs, sn = rope_tables(ms, 10000.0)
    pos = np.array(lens, np.int32) - 1
    ws = torch.empty(cuda_lib.tenzo_cuda_attention_exact_workspace_bytes(B, nq, nkv, ms), dtype=torch.uint8, device="cuda")
    args = dict(layer=0, n_q=nq, n_kv=nkv, max_seq=ms, max_len=ms, rope_cos=dev(cs), rope_sin=dev(sn), tiles=3, workspace=ws)
    out = kernels.attention_int8(dev(q), dev(k), dev(v), dev(ck), dev(cv), dev(sk), dev(sv), dev(pos), **args)
    paged = kernels.attention_int8(dev(q), dev(k), dev(v), dev(pk), dev(pv), dev(psk), dev(psv), dev(pos), block_table=dev(table), n_layers=1, **args)
    torch.cuda.synchronize()
    assert cuda_lib.tenzo_cuda_attention_take_timeouts() == 0
    opk, opv, osk, osv = pk.reshape(-1).copy(), pv.reshape(-1).copy(), psk.reshape(-1).copy(), psv.reshape(-1).copy()
    for b in range(B):
        c = [t[b].reshape(-1).copy() for t in (ck, cv, sk, sv)]
        qq, kk, vv, o = q[b].copy(), k[b].copy(), v[b].copy(), np.zeros(nq * 128, np.float32)
        O.ora_attention_int8(0, int(pos[b]), nq, nkv, 128, ms, 10000.0, P(qq, ora.c_f32p), P(kk, ora.c_f32p), P(vv, ora.c_f32p),
                             P(o, ora.c_f32p), P(c[0], ora.c_i8p), P(c[1], ora.c_i8p), P(c[2], ora.c_f32p), P(c[3], ora.c_f32p))
        assert np.array_equal(host(out)[b], o), f"sequence {b} (length {lens[b]})"
        o = oracle_paged(O, 0, int(pos[b]), nq, nkv, 1, q[b], k[b], v[b], opk, opv, osk, osv, table[b])
        assert np.array_equal(host(paged)[b], o), f"block pools, sequence {b} (length {lens[b]})"


@pytest.mark.parametrize("paged,B,nq,last", [(False, 1, 20, 768), (False, 2, 20, 768), (False, 4, 20, 1024), (True, 1, 20, 512), (True, 4, 20, 640)])
@pytest.mark.parametrize("over", [0, 1])
def test_line_between_the_forms(cuda_lib, paged, B, nq, last, over):
    """Either side of the line between one kernel and three: the three use the workspace, and the bits are the other form's."""
    from tenzo_b200 import kernels
    nkv, T = 5, last + over
    ms = (T + 15) // 16 * 16
    g = torch.Generator(device="cuda").manual_seed(T)
    shape = (B * ms // 16, 1, nkv, 16, 128) if paged else (B, 1, nkv, ms, 128)
    ck, cv = (torch.randint(-127, 128, shape, generator=g, device="cuda", dtype=torch.int8) for _ in range(2))
    sk, sv = (0.01 + 0.02 * torch.rand(shape[:-1], generator=g, device="cuda") for _ in range(2))
    q = torch.randn(B, nq * 128, generator=g, device="cuda")
    pos = torch.full((B,), T - 1, dtype=torch.int32, device="cuda")
    ws = torch.full((cuda_lib.tenzo_cuda_attention_exact_workspace_bytes(B, nq, nkv, T),), 0x5a, dtype=torch.uint8, device="cuda")
    args = dict(layer=0, n_q=nq, n_kv=nkv, max_seq=ms, max_len=T, append=False, workspace=ws)
    if paged:
        args.update(block_table=torch.randperm(B * ms // 16, generator=g, device="cuda").int().view(B, -1), n_layers=1)
    got = kernels.attention_int8(q, None, None, ck, cv, sk, sv, pos, **args)
    assert bool((ws != 0x5a).any()) == bool(over)
    other = kernels.attention_int8(q, None, None, ck, cv, sk, sv, pos, tiles=2 if over else 3, **args)
    torch.cuda.synchronize()
    assert cuda_lib.tenzo_cuda_attention_take_timeouts() == 0
    assert torch.equal(got, other)
