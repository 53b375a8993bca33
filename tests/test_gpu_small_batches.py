"""Where the tensor-core paths begin (two sequences for the LM head, nine for TL1 products), and the cluster form of the
sampler's candidate selection, against the one-sequence kernels and numpy."""
import numpy as np
import pytest
import torch
from gpu_helpers import dev, host
from helpers import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,H,B", [(5000, 256, 2), (1028, 128, 7), (4096, 2560, 15)])
def test_lm_head_of_a_few_sequences_matches_one_at_a_time(cuda_lib, V, H, B):
    from tenzo_b200 import kernels
    rng = np.random.default_rng([81, V, B])
    w = rng.integers(-127, 128, (V, H), dtype=np.int8)
    w[V - 3] = w[5]                                  # equal rows: the first maximum wins
    dw, ds = dev(w), dev(np.full(V, 0.01, np.float32))
    x, fn = dev(rng.standard_normal((B, H)).astype(np.float32)), dev((1 + 0.1 * rng.standard_normal(H)).astype(np.float32))
    lg, acc, arg = (host(t) for t in kernels.lm_head_i8(x, dw, ds, norm_w=fn, want_acc=True))
    for b in range(B):
        l1, a1, g1 = (host(t) for t in kernels.lm_head_i8(x[b:b + 1].contiguous(), dw, ds, norm_w=fn, want_acc=True))
        assert np.array_equal(lg[b], l1[0]) and np.array_equal(acc[b], a1[0]) and arg[b] == g1[0] == np.argmax(l1[0])
    assert cuda_lib.tenzo_cuda_lm_head_take_timeouts() == 0


@pytest.mark.parametrize("B", [8, 9, 15])
@pytest.mark.parametrize("N,K", [(192, 256), (640, 2560), (128, 6912)])
def test_tl1_product_of_a_few_sequences_matches_one_at_a_time(cuda_lib, N, K, B):
    from tenzo_b200 import kernels
    rng = np.random.default_rng([82, N, B])
    w, x = dev(synth.random_tl1_packed(rng, N, K)), dev(rng.standard_normal((B, K)).astype(np.float32))
    res, nw = dev(rng.standard_normal((B, N)).astype(np.float32)), dev((1 + 0.1 * rng.standard_normal(K)).astype(np.float32))
    run = lambda a, r: host(kernels.tl1_gemv(a, w, N // 64, K, [0.02], epilogue=kernels.EPI_RESIDUAL, resid=r, norm_w=nw, do_norm=True)["out"])
    many = run(x, res)
    for b in range(B):
        assert np.array_equal(many[b], run(x[b:b + 1].contiguous(), res[b:b + 1].contiguous())[0])
    assert cuda_lib.tenzo_cuda_tl1_gemv_take_timeouts() == 0


@pytest.mark.parametrize("V,k,shape", [(128256, 40, "normal"), (128256, 1, "normal"), (128256, 64, "clustered"), (128256, 256, "normal"),
                                       (128256, 257, "normal"), (1001, 40, "normal"), (37, 37, "normal"), (128256, 40, "ties"), (128256, 3, "many ties")])
def test_candidate_selection(cuda_lib, V, k, shape):
    rng = np.random.default_rng([83, V, k])
    l = rng.standard_normal(V).astype(np.float32)
    if shape == "clustered":
        l[5000:5300] += 10.0                         # the largest ones side by side
    if shape == "ties":
        l = np.round(l * 50) / np.float32(50)        # runs of equal values at the threshold
    if shape == "many ties":
        l[:] = 0.0                                   # more than the list holds
        l[::3] = -0.0
    d = dev(l)
    cap = cuda_lib.tenzo_cuda_topk_max_candidates()
    cnt, vals, idxs = (torch.zeros(n, dtype=t, device="cuda") for n, t in ((1, torch.int32), (cap, torch.float32), (cap, torch.int32)))
    assert cuda_lib.tenzo_cuda_topk_candidates(d.data_ptr(), V, k, cnt.data_ptr(), vals.data_ptr(), idxs.data_ptr(), None) == 0
    torch.cuda.synchronize()
    want = np.nonzero(l >= np.sort(l)[-k])[0]
    assert int(host(cnt)[0]) == want.size
    if want.size <= cap:
        assert np.array_equal(host(idxs)[:want.size], want) and np.array_equal(host(vals)[:want.size], l[want])
