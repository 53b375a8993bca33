"""Attention of many query rows over one cache (a prompt's rows), 64 query vectors of a kv head together: bit for bit against the oracle fed
token by token, and against the three kernels that take an item a time: every head grouping, rows in any order, lengths around the
tiles' and chunks' edges, several passes, refused positions, infinite scales."""
import ctypes

import numpy as np
import pytest
import torch
from gpu_helpers import dev, host
from helpers import ora
from test_gpu_norm_attn_lm import rope_tables

pytestmark = pytest.mark.gpu
P = ora.ptr


def attend(lib, q, ck, cv, sk, sv, pos, nq, nkv, ms, max_len, cs, sn, ws, tiles=0):
    from tenzo_b200 import abi
    a, out = abi.AttentionArgs(), torch.full((q.shape[0], nq * 128), 7.0, device="cuda")
    a.q, a.out, a.q_stride = q.data_ptr(), out.data_ptr(), q.stride(0)
    a.cache_k, a.cache_v, a.scale_k, a.scale_v = (t.data_ptr() for t in (ck, cv, sk, sv))
    a.pos, a.rope_cos, a.rope_sin = pos.data_ptr(), cs.data_ptr(), sn.data_ptr()
    a.layer, a.n_q, a.n_kv, a.head_dim, a.max_seq, a.batch, a.max_len, a.tiles = 1, nq, nkv, 128, ms, q.shape[0], max_len, tiles
    a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
    assert lib.tenzo_cuda_attention_int8(ctypes.byref(a), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    return out


def took_rows(ws, ck, nkv, max_len):
    """The form writes the first chain's elements of the first key tile as floats at the start of the scratch."""
    n = min(128, max_len)
    return torch.equal(ws[:512].view(torch.float32)[:n], ck[1, 0, :n, 0].float())


@pytest.mark.parametrize("n,before,nq,nkv", [(300, 0, 20, 5), (257, 0, 32, 4), (300, 97, 16, 8), (290, 5, 16, 16)])
def test_rows_against_oracle(cuda_lib, n, before, nq, nkv):
    O = ora.load_oracle()
    T, ms = before + n, before + n + 3
    rng = np.random.default_rng([131, n, nq])
    ck, cv = (np.zeros((2, nkv, ms, 128), np.int8) for _ in range(2))
    sk, sv = (np.ones((2, nkv, ms), np.float32) for _ in range(2))
    q, k, v = (rng.standard_normal((T, h * 128)).astype(np.float32) for h in (nq, nkv, nkv))
    q[::3] *= 4.0
    q[::7] *= 0.01
    want = np.zeros((T, nq * 128), np.float32)
    for t in range(T):                                # token by token, as the reference feeds a prompt
        O.ora_attention_int8(1, t, nq, nkv, 128, ms, 10000.0, P(q[t].copy(), ora.c_f32p), P(k[t].copy(), ora.c_f32p), P(v[t].copy(), ora.c_f32p), P(want[t], ora.c_f32p),
                             P(ck, ora.c_i8p), P(cv, ora.c_i8p), P(sk, ora.c_f32p), P(sv, ora.c_f32p))
    order = rng.permutation(n) + before
    cs, sn = rope_tables(ms, 10000.0)
    ws = torch.full((cuda_lib.tenzo_cuda_attention_rows_workspace_bytes(n, nq, nkv, T),), 0x5a, dtype=torch.uint8, device="cuda")
    dck = dev(ck)
    out = attend(cuda_lib, dev(q[order]), dck, dev(cv), dev(sk), dev(sv), dev(order.astype(np.int32)), nq, nkv, ms, T, dev(cs), dev(sn), ws)
    assert cuda_lib.tenzo_cuda_attention_take_timeouts() == 0
    assert took_rows(ws, dck, nkv, T)
    assert np.array_equal(host(out), want[order])


@pytest.mark.parametrize("n,max_len,nq,nkv,passes", [(300, 700, 20, 5, 1), (300, 1290, 32, 8, 1), (1000, 640, 32, 8, 2), (340, 300, 32, 4, 1), (400, 517, 16, 16, 1)])
def test_rows_equal_three_kernels(cuda_lib, n, max_len, nq, nkv, passes):
    g = torch.Generator(device="cuda").manual_seed(n + max_len)
    ms = max_len + 1
    ck, cv = (torch.randint(-128, 128, (2, nkv, ms, 128), generator=g, device="cuda", dtype=torch.int8) for _ in range(2))
    sk, sv = (0.001 + 0.02 * torch.rand(2, nkv, ms, generator=g, device="cuda") for _ in range(2))
    q = torch.randn(n, nq * 128 + 64, generator=g, device="cuda")[:, :nq * 128]             # strided rows
    pos = torch.randint(0, max_len, (n,), generator=g, device="cuda", dtype=torch.int32)
    edges = torch.tensor([e for e in (0, 1, 30, 31, 32, 63, 64, 126, 127, 128, 129, 255, 256, 511, 512, max_len - 2, max_len - 1) if e < max_len], dtype=torch.int32)
    pos[5:5 + len(edges)] = edges.cuda()
    cs, sn = (torch.from_numpy(t).cuda() for t in rope_tables(ms, 10000.0))
    rows = 64 // (nq // nkv) * -(-n // (64 // (nq // nkv) * passes))                         # whole tiles
    ws = torch.full((cuda_lib.tenzo_cuda_attention_rows_workspace_bytes(rows, nq, nkv, max_len),), 0x5a, dtype=torch.uint8, device="cuda")
    call = lambda tiles: attend(cuda_lib, q, ck, cv, sk, sv, pos, nq, nkv, ms, max_len, cs, sn, ws, tiles)
    got = call(0)
    assert took_rows(ws, ck, nkv, max_len)
    assert cuda_lib.tenzo_cuda_attention_take_timeouts() == 0
    assert torch.equal(got, call(3))
    # refused positions: nothing is written for them, the others come out as before
    pos[3], pos[n - 1] = -1, max_len
    bad = call(0)
    assert cuda_lib.tenzo_cuda_attention_take_timeouts() == 2
    assert bool((bad[[3, n - 1]] == 7.0).all())
    keep = [i for i in range(n) if i not in (3, n - 1)]
    assert torch.equal(bad[keep], got[keep])
    # an infinite scale: infinite scores, and NaN where the reference has them
    sk[1, 0, 17] = float("inf")
    a, b = call(0), call(3)
    assert torch.isnan(b).any() and torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(a.nan_to_num(), b.nan_to_num())
    cuda_lib.tenzo_cuda_attention_take_timeouts()


@pytest.mark.parametrize("blown,nq,nkv", [(1, 20, 5), (37, 16, 16)])
def test_rows_whose_scores_all_lie_below_the_maximums_start(cuda_lib, blown, nq, nkv):
    """The first keys of kv head 0 score -1e34 with their own queries, those of kv head 1 -inf: the reference's maximum stays at its start, -1e30, every
    exponential is 0, and the row is 0 / 0. Slots behind such a row's last key are no keys, whatever rows lie beside it."""
    O = ora.load_oracle()
    n, ms = 300, 303
    rng = np.random.default_rng([132, blown, nq])
    ck, cv = (np.zeros((2, nkv, ms, 128), np.int8) for _ in range(2))
    sk, sv = (np.ones((2, nkv, ms), np.float32) for _ in range(2))
    q, k, v = (rng.standard_normal((n, h * 128)).astype(np.float32) for h in (nq, nkv, nkv))
    k[:blown, :128], k[:blown, 128:256] = 1e30, 3e38
    q[:blown, :2 * (nq // nkv) * 128] = -1000.0
    want = np.zeros((n, nq * 128), np.float32)
    for t in range(n):
        O.ora_attention_int8(1, t, nq, nkv, 128, ms, 10000.0, P(q[t].copy(), ora.c_f32p), P(k[t].copy(), ora.c_f32p), P(v[t].copy(), ora.c_f32p), P(want[t], ora.c_f32p),
                             P(ck, ora.c_i8p), P(cv, ora.c_i8p), P(sk, ora.c_f32p), P(sv, ora.c_f32p))
    assert np.isnan(want[0, :2 * (nq // nkv) * 128]).all() and np.isfinite(want[0, 2 * (nq // nkv) * 128:]).all()
    order = rng.permutation(n)
    cs, sn = (dev(t) for t in rope_tables(ms, 10000.0))
    ws = torch.full((cuda_lib.tenzo_cuda_attention_rows_workspace_bytes(n, nq, nkv, n),), 0x5a, dtype=torch.uint8, device="cuda")
    args = [dev(a) for a in (q[order], ck, cv, sk, sv, order.astype(np.int32))]
    call = lambda tiles: host(attend(cuda_lib, *args, nq, nkv, ms, n, cs, sn, ws, tiles))
    got = call(0)
    assert took_rows(ws, args[1], nkv, n)
    assert cuda_lib.tenzo_cuda_attention_take_timeouts() == 0
    assert np.array_equal(got, want[order], equal_nan=True)
    assert np.array_equal(call(3), want[order], equal_nan=True)


@pytest.mark.parametrize("n,max_len,nq,nkv,scratch_rows", [(700, 640, 20, 5, 352), (1000, 300, 32, 8, 176), (520, 517, 16, 16, 320)])
def test_rows_in_several_passes_of_one_value_cta_an_sm(cuda_lib, n, max_len, nq, nkv, scratch_rows):
    """Scratch for 160 to 220 CTAs of the value sums: two passes and more, the last one smaller, give what the three kernels do."""
    g = torch.Generator(device="cuda").manual_seed(n)
    ck, cv = (torch.randint(-128, 128, (2, nkv, max_len, 128), generator=g, device="cuda", dtype=torch.int8) for _ in range(2))
    sk, sv = (0.001 + 0.02 * torch.rand(2, nkv, max_len, generator=g, device="cuda") for _ in range(2))
    q = torch.randn(n, nq * 128, generator=g, device="cuda")
    pos = torch.randint(0, max_len, (n,), generator=g, device="cuda", dtype=torch.int32)
    cs, sn = (torch.from_numpy(t).cuda() for t in rope_tables(max_len, 10000.0))
    ws = torch.full((cuda_lib.tenzo_cuda_attention_rows_workspace_bytes(scratch_rows, nq, nkv, max_len),), 0x5a, dtype=torch.uint8, device="cuda")
    call = lambda tiles: attend(cuda_lib, q, ck, cv, sk, sv, pos, nq, nkv, max_len, max_len, cs, sn, ws, tiles)
    got = call(0)
    assert took_rows(ws, ck, nkv, max_len)
    assert torch.equal(got, call(3))
    assert cuda_lib.tenzo_cuda_attention_take_timeouts() == 0


def rows_engine(max_seq):
    from tenzo_b200 import synth
    from tenzo_b200.engine import Engine
    m = synth.SyntheticModel(dict(synth.TINY, hidden_size=2560, num_q_heads=20, num_kv_heads=5, ffn_dim=768, num_layers=2, vocab_size=2048, max_seq_len=max_seq), seed=43)
    return lambda: Engine(m.config_struct(max_seq_len=max_seq)).load_synthetic(m)


def test_engine_without_memory_for_the_rows_scratch_takes_the_smaller_one(cuda_lib):
    """A prompt whose rows' scratch (243 MB here) does not fit on the device any more runs in the scratch of any batch (64 MB): same cache, same tokens."""
    from tenzo_b200 import synth
    new, prompt, left = rows_engine(8192), synth.prompt_tokens(13, 301, 2048), 160 << 20
    assert cuda_lib.tenzo_cuda_attention_rows_workspace_bytes(300, 20, 5, 8192) > left + (64 << 20)

    def run(e):
        e.prefill_chunk(prompt[:-1])
        return [e.kv_export(0, l, 300) for l in range(2)], e.decode_greedy([int(prompt[-1])], 8)

    with new() as e:
        kv, tokens = run(e)
    with new() as e:
        hog = []
        try:
            while (free := torch.cuda.mem_get_info()[0]) > left + (8 << 20):
                hog.append(torch.empty(min(free - left, 8 << 30), dtype=torch.uint8, device="cuda"))
            kv_few, tokens_few = run(e)
        finally:
            del hog
            torch.cuda.empty_cache()
    assert np.array_equal(tokens, tokens_few) and all(np.array_equal(a, b) for x, y in zip(kv, kv_few) for a, b in zip(x, y))


@pytest.mark.parametrize("chunks", [[700], [300, 400], [20, 680]])
def test_engine_chunks_take_the_rows_form(cuda_lib, chunks):
    """A prompt through the engine as it runs by default (overlapped launches, every layer on one scratch, a cache longer than the prompt, 20/5 heads):
    the cache and the tokens that follow are those of the prompt fed token by token."""
    from tenzo_b200 import synth
    new, prompt = rows_engine(1100), synth.prompt_tokens(14, 701, 2048)
    with new() as e:
        for t in prompt[:-1]:
            e.prefill_token(int(t))
        kv = [e.kv_export(0, l, 700) for l in range(2)]
        tokens = e.decode_greedy([int(prompt[-1])], 8)
    with new() as e:
        done = 0
        for c in chunks:
            before = e.kernel_launches()
            e.prefill_chunk(prompt[done:done + c])
            done += c
            if c >= 300:
                assert e.kernel_launches() - before == 1 + 2 * (1 + 4 * 2 + 4)          # the embedding; a layer's append, products and four attention kernels
        for l in range(2):
            assert all(np.array_equal(got, want) for got, want in zip(e.kv_export(0, l, 700), kv[l])), f"layer {l}"
        assert np.array_equal(e.decode_greedy([int(prompt[-1])], 8), tokens)
