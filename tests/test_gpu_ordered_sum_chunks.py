"""Sums of exponentials in key order, chunk by chunk: lengths around the ends of the first chunk (960, 1984 or 4032 keys, by the
heads of a CTA) and of the next, for rows whose sum keeps one exponent for long, changes it often, or is one key's."""
import numpy as np
import pytest
import torch
from gpu_helpers import dev, host
from helpers import ora
from test_gpu_norm_attn_lm import rope_tables

pytestmark = pytest.mark.gpu
P = ora.ptr


@pytest.mark.parametrize("nq,nkv,batch,lens", [
    (8, 2, 75, [959, 960, 961, 1023, 1024, 1025, 1855, 1856, 1857, 64, 65]),       # four heads a CTA
    (8, 2, 225, [961, 1857, 64, 960]),                                              # the same, with half the evaluating threads
    (4, 2, 75, [1983, 1984, 1985, 3903, 3904, 3905, 65]),                           # two heads
    (8, 2, 4, [4031, 4032, 4033, 8001])])                                           # one head
def test_sum_across_chunk_ends(cuda_lib, nq, nkv, batch, lens):
    from tenzo_b200 import kernels
    O = ora.load_oracle()
    rng = np.random.default_rng([93, nq, batch])
    ms = (max(lens) + 15) // 16 * 16
    n = [lens[i % len(lens)] for i in range(batch)]
    ck, cv = (torch.randint(-127, 128, (batch, 1, nkv, ms, 128), dtype=torch.int8, device="cuda") for _ in range(2))
    sk, sv = (0.01 + 0.02 * torch.rand(batch, 1, nkv, ms, device="cuda") for _ in range(2))
    q = rng.standard_normal((batch, nq * 128)).astype(np.float32) * np.float32([0.001, 1.0, 8.0])[np.arange(batch) % 3][:, None]
    k, v = (rng.standard_normal((batch, nkv * 128)).astype(np.float32) for _ in range(2))
    cs, sn = rope_tables(ms, 10000.0)
    pos = np.array(n, np.int32) - 1
    check = sorted(set(range(min(batch, 2 * len(lens)))) | {batch - 1})
    before = {b: [host(t[b]).reshape(-1).copy() for t in (ck, cv, sk, sv)] for b in check}
    ws = torch.empty(cuda_lib.tenzo_cuda_attention_exact_workspace_bytes(batch, nq, nkv, ms), dtype=torch.uint8, device="cuda")
    out = kernels.attention_int8(dev(q), dev(k), dev(v), ck, cv, sk, sv, dev(pos), layer=0, n_q=nq, n_kv=nkv, max_seq=ms, max_len=ms,
                                 rope_cos=dev(cs), rope_sin=dev(sn), tiles=3, workspace=ws)
    torch.cuda.synchronize()
    assert cuda_lib.tenzo_cuda_attention_take_timeouts() == 0
    for b in check:
        ock, ocv, osk, osv = before[b]
        qq, kk, vv, want = q[b].copy(), k[b].copy(), v[b].copy(), np.zeros(nq * 128, np.float32)
        O.ora_attention_int8(0, int(pos[b]), nq, nkv, 128, ms, 10000.0, P(qq, ora.c_f32p), P(kk, ora.c_f32p), P(vv, ora.c_f32p),
                             P(want, ora.c_f32p), P(ock, ora.c_i8p), P(ocv, ora.c_i8p), P(osk, ora.c_f32p), P(osv, ora.c_f32p))
        assert np.array_equal(host(out)[b], want), f"sequence {b} (length {n[b]})"
