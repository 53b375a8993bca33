"""Exact-order attention of up to 256 keys (what the automatic choice takes there), bit for bit against the oracle: lengths around
the 64 and 128 keys at which threads share a key, every head grouping, appended and cached last rows, contiguous caches of one and
several sequences and block pools, and positions that are refused."""
import numpy as np
import pytest
import torch
from gpu_helpers import dev, host
from helpers import ora
from test_gpu_norm_attn_lm import rope_tables
from test_gpu_paged_kv import oracle_paged

pytestmark = pytest.mark.gpu
P = ora.ptr
EDGES = [1, 2, 7, 8, 9, 63, 64, 65, 100, 127, 128, 129, 191, 193, 255, 256]


def draw(rng, B, nq, nkv):
    q = rng.standard_normal((B, nq * 128)).astype(np.float32) * np.float32([1.0, 5.0, 0.01])[np.arange(B) % 3][:, None]
    return q, rng.standard_normal((B, nkv * 128)).astype(np.float32), rng.standard_normal((B, nkv * 128)).astype(np.float32)


@pytest.mark.parametrize("B,nq,nkv,max_len,pdl", [
    (1, 20, 5, 256, True), (3, 20, 5, 64, True), (16, 20, 5, 256, False), (48, 20, 5, 200, True), (16, 16, 2, 256, True),
    (40, 8, 4, 129, False), (16, 4, 4, 256, True)])
def test_contiguous_cache(cuda_lib, B, nq, nkv, max_len, pdl):
    from tenzo_b200 import kernels
    O = ora.load_oracle()
    lens = [min(EDGES[(5 * i + 8) % len(EDGES)], max_len) for i in range(B)]
    rng = np.random.default_rng([95, B, nq, max_len])
    ms = 272
    ck, cv = (rng.integers(-127, 128, (B, 1, nkv, ms, 128)).astype(np.int8) for _ in range(2))
    sk, sv = ((0.01 + 0.02 * rng.random((B, 1, nkv, ms))).astype(np.float32) for _ in range(2))
    q, k, v = draw(rng, B, nq, nkv)
    cs, sn = rope_tables(ms, 10000.0)
    pos = np.array(lens, np.int32) - 1
    dck, dcv, dsk, dsv = dev(ck), dev(cv), dev(sk), dev(sv)
    args = dict(layer=0, n_q=nq, n_kv=nkv, max_seq=ms, max_len=max_len, rope_cos=dev(cs), rope_sin=dev(sn), use_pdl=pdl)
    out = kernels.attention_int8(dev(q), dev(k), dev(v), dck, dcv, dsk, dsv, dev(pos), **args)
    again = kernels.attention_int8(dev(q), None, None, dck, dcv, dsk, dsv, dev(pos), append=False, **args)     # the same rows, now cached
    torch.cuda.synchronize()
    assert cuda_lib.tenzo_cuda_attention_take_timeouts() == 0
    for b in range(B):
        ock, ocv, osk, osv = ck[b].reshape(-1).copy(), cv[b].reshape(-1).copy(), sk[b].reshape(-1).copy(), sv[b].reshape(-1).copy()
        qq, kk, vv, o = q[b].copy(), k[b].copy(), v[b].copy(), np.zeros(nq * 128, np.float32)
        O.ora_attention_int8(0, int(pos[b]), nq, nkv, 128, ms, 10000.0, P(qq, ora.c_f32p), P(kk, ora.c_f32p), P(vv, ora.c_f32p),
                             P(o, ora.c_f32p), P(ock, ora.c_i8p), P(ocv, ora.c_i8p), P(osk, ora.c_f32p), P(osv, ora.c_f32p))
        assert np.array_equal(host(out)[b], o) and np.array_equal(host(again)[b], o), f"sequence {b} (length {lens[b]})"
        for got, want in ((dck, ock), (dcv, ocv), (dsk, osk), (dsv, osv)):
            assert np.array_equal(host(got)[b].reshape(-1), want)


@pytest.mark.parametrize("B,nq,nkv", [(1, 8, 2), (16, 8, 1), (40, 16, 4), (16, 4, 4)])
def test_block_pools(cuda_lib, B, nq, nkv):
    from tenzo_b200 import kernels
    O = ora.load_oracle()
    L, layer, per_seq = 2, 1, 16
    lens = [EDGES[(3 * i + 12) % len(EDGES)] for i in range(B)]
    rng = np.random.default_rng([96, B, nq])
    table = rng.permutation(B * per_seq).astype(np.int32).reshape(B, per_seq)
    pk, pv = (rng.integers(-127, 128, (B * per_seq, L, nkv, 16, 128)).astype(np.int8) for _ in range(2))
    psk, psv = ((0.01 + 0.02 * rng.random((B * per_seq, L, nkv, 16))).astype(np.float32) for _ in range(2))
    q, k, v = draw(rng, B, nq, nkv)
    cs, sn = rope_tables(256, 10000.0)
    pos = np.array(lens, np.int32) - 1
    dpk, dpv, dsk, dsv = dev(pk), dev(pv), dev(psk), dev(psv)
    out = kernels.attention_int8(dev(q), dev(k), dev(v), dpk, dpv, dsk, dsv, dev(pos), layer=layer, n_q=nq, n_kv=nkv, max_seq=256, max_len=256,
                                 rope_cos=dev(cs), rope_sin=dev(sn), block_table=dev(table), n_layers=L)
    torch.cuda.synchronize()
    assert cuda_lib.tenzo_cuda_attention_take_timeouts() == 0
    opk, opv, osk, osv = pk.reshape(-1).copy(), pv.reshape(-1).copy(), psk.reshape(-1).copy(), psv.reshape(-1).copy()
    for b in range(B):
        o = oracle_paged(O, layer, int(pos[b]), nq, nkv, L, q[b], k[b], v[b], opk, opv, osk, osv, table[b])
        assert np.array_equal(host(out)[b], o), f"sequence {b} (length {lens[b]})"
    for got, want in ((dpk, opk), (dpv, opv), (dsk, osk), (dsv, osv)):
        assert np.array_equal(host(got).reshape(-1), want)


def test_position_outside_is_refused(cuda_lib):
    from tenzo_b200 import kernels
    ck, cv = (torch.zeros(2, 1, 1, 64, 128, dtype=torch.int8, device="cuda") for _ in range(2))
    sk, sv = (torch.ones(2, 1, 1, 64, device="cuda") for _ in range(2))
    q = torch.ones(2, 4 * 128, device="cuda")
    pos = torch.tensor([3, 40], dtype=torch.int32, device="cuda")
    kernels.attention_int8(q, None, None, ck, cv, sk, sv, pos, layer=0, n_q=4, n_kv=1, max_seq=64, max_len=32, append=False)
    torch.cuda.synchronize()
    assert cuda_lib.tenzo_cuda_attention_take_timeouts() == 2 and cuda_lib.tenzo_cuda_attention_take_timeouts() == 0
