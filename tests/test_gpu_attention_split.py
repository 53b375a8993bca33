"""Exact-order attention as three kernels over the whole machine (tiles = 3), bit for bit against the oracle: lengths around
the 64-key tile, the 512-key span, the 64-key value chunk and the softmax chunks, every head grouping, batches that take the
fine and the coarse cut of the value sums and both together, several passes through a small scratch buffer, block pools."""
import numpy as np
import pytest
import torch
from gpu_helpers import dev, host
from helpers import ora
from test_gpu_norm_attn_lm import rope_tables
from test_gpu_paged_kv import oracle_paged

pytestmark = pytest.mark.gpu
P = ora.ptr
EDGES = [1, 2, 63, 64, 65, 127, 128, 129, 191, 193, 511, 512, 513, 700]


def vectors(rng, B, nq, nkv):
    q = rng.standard_normal((B, nq * 128)).astype(np.float32)
    q[::2] *= 4.0                                    # peaked rows: sums dominated by a few keys, weights under the 1e-7 cut
    q[::5] *= 0.01                                   # flat rows: long runs inside one binade, many ties
    return q, rng.standard_normal((B, nkv * 128)).astype(np.float32), rng.standard_normal((B, nkv * 128)).astype(np.float32)


@pytest.mark.parametrize("B,lens_cycle,ms,nq,nkv,passes", [
    (14, EDGES, 704, 20, 5, 1), (14, EDGES, 704, 4, 4, 3), (14, EDGES, 703, 4, 2, 1), (5, EDGES, 704, 16, 2, 2),
    (62, [300, 65, 513, 128, 1], 520, 20, 5, 1),     # 310 items: a whole round of coarse items and fourteen fine ones
    (40, [257, 64, 300], 304, 16, 8, 4),             # 320 items in passes of 80, all coarse
    (2, [8192, 4099], 8192, 20, 5, 1)])
def test_split_attention_against_oracle(cuda_lib, B, lens_cycle, ms, nq, nkv, passes):
    from tenzo_b200 import kernels
    O = ora.load_oracle()
    lens = [lens_cycle[i % len(lens_cycle)] for i in range(B)]
    rng = np.random.default_rng([71, B, nq])
    ck = rng.integers(-127, 128, (B, 1, nkv, ms, 128)).astype(np.int8)
    cv = rng.integers(-127, 128, (B, 1, nkv, ms, 128)).astype(np.int8)
    sk = (0.01 + 0.02 * rng.random((B, 1, nkv, ms))).astype(np.float32)
    sv = (0.01 + 0.02 * rng.random((B, 1, nkv, ms))).astype(np.float32)
    q, k, v = vectors(rng, B, nq, nkv)
    cs, sn = rope_tables(ms, 10000.0)
    pos = np.array([n - 1 for n in lens], np.int32)
    need = cuda_lib.tenzo_cuda_attention_exact_workspace_bytes((B + passes - 1) // passes, nq, nkv, ms)
    dck, dcv, dsk, dsv = dev(ck), dev(cv), dev(sk), dev(sv)
    out = kernels.attention_int8(dev(q), dev(k), dev(v), dck, dcv, dsk, dsv, dev(pos), layer=0, n_q=nq, n_kv=nkv, max_seq=ms, max_len=ms,
                                 rope_cos=dev(cs), rope_sin=dev(sn), tiles=3, workspace=torch.empty(need, dtype=torch.uint8, device="cuda"))
    torch.cuda.synchronize()
    assert cuda_lib.tenzo_cuda_attention_take_timeouts() == 0
    got, gck, gcv, gsk, gsv = host(out), host(dck), host(dcv), host(dsk), host(dsv)
    for b in range(B):
        ock, ocv, osk, osv = ck[b].reshape(-1).copy(), cv[b].reshape(-1).copy(), sk[b].reshape(-1).copy(), sv[b].reshape(-1).copy()
        qq, kk, vv, o = q[b].copy(), k[b].copy(), v[b].copy(), np.zeros(nq * 128, np.float32)
        O.ora_attention_int8(0, int(pos[b]), nq, nkv, 128, ms, 10000.0, P(qq, ora.c_f32p), P(kk, ora.c_f32p), P(vv, ora.c_f32p),
                             P(o, ora.c_f32p), P(ock, ora.c_i8p), P(ocv, ora.c_i8p), P(osk, ora.c_f32p), P(osv, ora.c_f32p))
        assert np.array_equal(got[b], o), f"sequence {b} (length {lens[b]})"
        assert np.array_equal(gck[b].reshape(-1), ock) and np.array_equal(gcv[b].reshape(-1), ocv)
        assert np.array_equal(gsk[b].reshape(-1), osk) and np.array_equal(gsv[b].reshape(-1), osv)


@pytest.mark.parametrize("B,nq,nkv,passes", [(14, 8, 2, 1), (14, 8, 1, 2), (14, 4, 4, 1), (75, 16, 4, 1)])
def test_split_attention_block_pools_against_oracle(cuda_lib, B, nq, nkv, passes):
    from tenzo_b200 import kernels
    O = ora.load_oracle()
    L, layer, per_seq = 2, 1, 44
    lens = [EDGES[i % len(EDGES)] for i in range(B)]
    rng = np.random.default_rng([72, B, nq])
    table = rng.permutation(B * per_seq).astype(np.int32).reshape(B, per_seq)
    pk = rng.integers(-127, 128, (B * per_seq, L, nkv, 16, 128)).astype(np.int8)
    pv = rng.integers(-127, 128, (B * per_seq, L, nkv, 16, 128)).astype(np.int8)
    psk = (0.01 + 0.02 * rng.random((B * per_seq, L, nkv, 16))).astype(np.float32)
    psv = (0.01 + 0.02 * rng.random((B * per_seq, L, nkv, 16))).astype(np.float32)
    q, k, v = vectors(rng, B, nq, nkv)
    cs, sn = rope_tables(per_seq * 16, 10000.0)
    pos = np.array([n - 1 for n in lens], np.int32)
    need = cuda_lib.tenzo_cuda_attention_exact_workspace_bytes((B + passes - 1) // passes, nq, nkv, per_seq * 16)
    dpk, dpv, dsk, dsv = dev(pk), dev(pv), dev(psk), dev(psv)
    out = kernels.attention_int8(dev(q), dev(k), dev(v), dpk, dpv, dsk, dsv, dev(pos), layer=layer, n_q=nq, n_kv=nkv, max_seq=per_seq * 16,
                                 max_len=per_seq * 16, rope_cos=dev(cs), rope_sin=dev(sn), block_table=dev(table), n_layers=L, tiles=3,
                                 workspace=torch.empty(need, dtype=torch.uint8, device="cuda"))
    torch.cuda.synchronize()
    assert cuda_lib.tenzo_cuda_attention_take_timeouts() == 0
    opk, opv, osk, osv = pk.reshape(-1).copy(), pv.reshape(-1).copy(), psk.reshape(-1).copy(), psv.reshape(-1).copy()
    for b in range(B):
        o = oracle_paged(O, layer, int(pos[b]), nq, nkv, L, q[b], k[b], v[b], opk, opv, osk, osv, table[b])
        assert np.array_equal(host(out)[b], o), f"sequence {b} (length {lens[b]})"
    assert np.array_equal(host(dpk).reshape(-1), opk) and np.array_equal(host(dpv).reshape(-1), opv)
    assert np.array_equal(host(dsk).reshape(-1), osk) and np.array_equal(host(dsv).reshape(-1), osv)
