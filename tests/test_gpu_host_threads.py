"""Per-kernel calls from host threads: from a thread that has made no CUDA call yet, and of different sizes from two threads side
by side (a call's dynamic shared memory lies under a limit that is an attribute of the kernel, not of the launch)."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch
from gpu_helpers import dev
from helpers import abi, synth

pytestmark = pytest.mark.gpu


class Call:
    """A C entry point with its arguments in hand (all but the stream, the last one) and the tensors that they point into."""

    def __init__(self, fn, args, out, *keep):
        self.fn, self.args, self.out, self.keep = fn, args, out, keep

    def __call__(self, stream, times=1):
        fn, args = self.fn, (*self.args, stream.cuda_stream)
        return next((rc for rc in (fn(*args) for _ in range(times)) if rc), 0)


def product(lib, batch, K, N=128):
    rng = np.random.default_rng([91, batch, K])
    w, x, out = dev(synth.random_tl1_packed(rng, N, K)), dev(rng.standard_normal((batch, K)).astype(np.float32)), torch.zeros(batch, N, device="cuda")
    ws = torch.empty(lib.tenzo_cuda_tl1_gemv_workspace_bytes(batch, K) + 16, dtype=torch.uint8, device="cuda")
    g = abi.Tl1GemvArgs(x=x.data_ptr(), do_norm=1, eps=1e-5, w=w.data_ptr(), n_blocks=N // 64, K=K, seg_end=(C.c_int * 3)(*[N // 64] * 3),
                        seg_scale=(C.c_float * 3)(0.02, 0.02, 0.02), out=out.data_ptr(), batch=batch, x_stride=K, out_stride=N, workspace=ws.data_ptr())
    return Call(lib.tenzo_cuda_tl1_gemv, (C.byref(g),), out, g, w, x, ws)


def attention(lib, context, tiles, mode=0, nq=4, nkv=1):
    g = torch.Generator(device="cuda").manual_seed(92)
    rows = (context + 15) // 16 * 16
    ck, cv = (torch.randint(-127, 128, (1, nkv, rows, 128), generator=g, device="cuda", dtype=torch.int8) for _ in range(2))
    sk, sv = (0.01 + 0.02 * torch.rand(1, nkv, rows, generator=g, device="cuda") for _ in range(2))
    q, out = torch.randn(1, nq * 128, generator=g, device="cuda"), torch.zeros(1, nq * 128, device="cuda")
    pos = torch.full((1,), context - 1, dtype=torch.int32, device="cuda")
    need = lib.tenzo_cuda_attention_workspace_bytes if mode else lib.tenzo_cuda_attention_exact_workspace_bytes
    ws = torch.empty(need(1, nq, nkv, context), dtype=torch.uint8, device="cuda")
    a = abi.AttentionArgs(q=q.data_ptr(), out=out.data_ptr(), cache_k=ck.data_ptr(), cache_v=cv.data_ptr(), scale_k=sk.data_ptr(), scale_v=sv.data_ptr(),
                          seq_stride_kv=nkv * rows * 128, seq_stride_sc=nkv * rows, pos=pos.data_ptr(), n_q=nq, n_kv=nkv, head_dim=128, max_seq=rows, batch=1,
                          max_len=context, tiles=tiles, mode=mode, workspace=ws.data_ptr(), workspace_bytes=ws.numel())
    return Call(lib.tenzo_cuda_attention_int8, (C.byref(a),), out, a, ck, cv, sk, sv, q, pos, ws)


def lm_head(lib, batch, hidden, static):
    g = torch.Generator(device="cuda").manual_seed(93)
    w, s = torch.randint(-127, 128, (1024, hidden), generator=g, device="cuda", dtype=torch.int8), torch.full((1024,), 0.01, device="cuda")
    x, out = torch.randn(batch, hidden, generator=g, device="cuda"), torch.zeros(batch, 1024, device="cuda")
    scratch = torch.empty(lib.tenzo_cuda_lm_head_scratch_bytes(batch), dtype=torch.uint8, device="cuda")
    args = (x.data_ptr(), None, 1, 1e-5, w.data_ptr(), s.data_ptr(), 1024, hidden, batch, hidden, out.data_ptr(), None, None)
    if static:
        return Call(lib.tenzo_cuda_lm_head_i8_static, (*args, 0), out, w, s, x)
    return Call(lib.tenzo_cuda_lm_head_i8, (*args, scratch.data_ptr(), 0), out, w, s, x, scratch)


# Both calls of a pair launch the same instantiation of a kernel, with different amounts of shared memory.
PAIRS = {
    "product": lambda lib: (product(lib, 1, 3840), product(lib, 1, 4096)),
    "product, long rows": lambda lib: (product(lib, 1, 5120), product(lib, 1, 8192)),
    "product, rows above 8192": lambda lib: (product(lib, 1, 8224), product(lib, 1, 16384)),
    "product, three sequences": lambda lib: (product(lib, 3, 2560), product(lib, 3, 16384)),
    "product, tensor cores": lambda lib: (product(lib, 16, 2560), product(lib, 256, 2560)),
    "attention in one kernel": lambda lib: (attention(lib, 200, 2), attention(lib, 1000, 2)),
    "attention in one kernel, tiles": lambda lib: (attention(lib, 200, 1), attention(lib, 4000, 1)),
    "attention in three kernels": lambda lib: (attention(lib, 700, 3), attention(lib, 4096, 3)),
    "attention, tolerance mode": lambda lib: (attention(lib, 700, 0, 1), attention(lib, 4096, 0, 1)),
    "lm head, one sequence": lambda lib: (lm_head(lib, 1, 10240, True), lm_head(lib, 1, 16384, True)),
    "lm head, eight sequences": lambda lib: (lm_head(lib, 8, 1536, True), lm_head(lib, 8, 4096, True)),
    "lm head, tensor cores": lambda lib: (lm_head(lib, 2, 256, False), lm_head(lib, 64, 256, False)),
}


def in_threads(calls, times):
    """Return codes of the calls, each made by a thread of its own on a stream of its own."""
    torch.cuda.synchronize()
    rcs, streams, start = [None] * len(calls), [torch.cuda.Stream() for _ in calls], threading.Barrier(len(calls))

    def work(i):
        start.wait()
        rcs[i] = calls[i](streams[i], times)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    return rcs


@pytest.mark.parametrize("name", PAIRS)
def test_first_cuda_call_of_a_thread(cuda_lib, name):
    for call in PAIRS[name](cuda_lib):
        assert call(torch.cuda.current_stream()) == 0
        torch.cuda.synchronize()
        want = call.out.clone()
        call.out.zero_()
        assert in_threads([call], 1) == [0]
        assert torch.equal(call.out, want)


@pytest.mark.parametrize("name", PAIRS)
def test_two_threads_with_different_sizes(cuda_lib, name):
    calls = PAIRS[name](cuda_lib)
    assert [c(torch.cuda.current_stream()) for c in calls] == [0, 0]
    torch.cuda.synchronize()
    want = [c.out.clone() for c in calls]
    assert in_threads(calls, 4000) == [0, 0]
    for c, w in zip(calls, want):
        assert torch.equal(c.out, w)


def test_calls_go_to_the_current_stream(cuda_lib):
    from tenzo_b200 import kernels
    side = torch.cuda.Stream()
    assert kernels._stream() == torch.cuda.current_stream().cuda_stream
    with torch.cuda.stream(side):
        assert kernels._stream() == side.cuda_stream
    assert kernels._stream() == torch.cuda.current_stream().cuda_stream
