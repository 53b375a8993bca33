"""The one-sequence TL1 product against the batched one, where the tensor-core paths begin (two sequences for the LM head, nine
for TL1 products) against the one-sequence kernels, and the cluster form of the sampler's candidate selection against numpy."""
import numpy as np
import pytest
import torch
from gpu_helpers import dev, host
from helpers import ora, synth

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


@pytest.mark.parametrize("what", ["normal", "halves", "zeros", "tiny", "plain"])
@pytest.mark.parametrize("N,K", [(128, 32), (64, 64), (12800, 128), (192, 2592), (128, 4128), (128, 6912), (128, 8192),
                                 (4736, 64), (4800, 64), (9472, 2560), (9600, 4096), (4800, 4128), (9600, 6912), (4800, 8192)])     # half and whole row blocks a CTA
def test_tl1_product_of_one_sequence_matches_the_batched_kernel(cuda_lib, N, K, what):
    from tenzo_b200 import kernels
    rng = np.random.default_rng([84, N, K])
    x, nw = rng.standard_normal((1, K)).astype(np.float32), (1 + 0.1 * rng.standard_normal(K)).astype(np.float32)
    if what == "halves":                             # quotients on the rounding boundary: the presumed integers do not stand
        x[0] = ((rng.integers(-31, 31, K) + 0.5) / 31).astype(np.float32)
        x[0, K // 3], nw[:] = 1.0, 1.0
    x *= {"zeros": 0.0, "tiny": 1e-20}.get(what, 1.0)
    w, n_blocks, norm = dev(synth.random_tl1_packed(rng, N, K)), N // 64, what != "plain"
    two = lambda a: dev(np.concatenate([a, a[:, ::-1]]))
    epilogues = [kernels.EPI_STORE, kernels.EPI_RESIDUAL] + ([kernels.EPI_RELU2_GLU] if n_blocks % 2 == 0 else [])
    assert cuda_lib.tenzo_cuda_tl1_gemv_take_repeats() >= 0
    for epi in epilogues:
        glu, res = epi == kernels.EPI_RELU2_GLU, rng.standard_normal((1, N)).astype(np.float32)
        args = (w, n_blocks, K, [0.02, 0.03] if glu else [0.02], [n_blocks // 2, n_blocks] if glu else None)
        kw = dict(epilogue=epi, norm_w=dev(nw) if norm else None, do_norm=norm)
        resid = epi == kernels.EPI_RESIDUAL
        one = kernels.tl1_gemv(dev(x), *args, resid=dev(res) if resid else None, **kw)["out"]
        many = kernels.tl1_gemv(two(x), *args, resid=two(res) if resid else None, **kw)["out"]
        assert np.array_equal(host(one)[0], host(many)[0])
    repeats = cuda_lib.tenzo_cuda_tl1_gemv_take_repeats()
    assert repeats in {"normal": range(len(epilogues) + 1), "plain": [0], "zeros": [0]}.get(what, [len(epilogues)])     # halves, tiny: each time
    assert cuda_lib.tenzo_cuda_tl1_gemv_take_timeouts() == 0


@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("what", ["nan", "inf", "all nan", "nan weight", "inf weight", "overflow"])
@pytest.mark.parametrize("N,K", [(128, 64), (12800, 128), (192, 2592), (128, 6912)])
def test_tl1_product_of_one_sequence_with_non_finite_activations(cuda_lib, N, K, what, norm):
    """An element that is no number becomes the integer 0 (the CPU engine's conversion), so it must not reach the sum of the
    activations either: integers, scale, accumulators and outputs equal those of the batched kernel, and the oracle's where the
    vector goes into the quantiser as it is."""
    from tenzo_b200 import kernels
    rng = np.random.default_rng([85, N, K])
    x, nw = rng.standard_normal((1, K)).astype(np.float32), (1 + 0.1 * rng.standard_normal(K)).astype(np.float32)
    at = [0, K // 3, K - 1]
    if what in ("nan", "inf"):
        x[0, at] = [np.nan, np.nan, -np.nan] if what == "nan" else [np.inf, 1.0, -np.inf]
    elif what == "all nan":
        x[0] = np.nan
    elif what == "overflow":                         # x * w overflows before it is divided by the root mean square
        x[0, at], nw[at] = np.float32(1e18), np.float32(1e30)
    else:
        nw[at] = np.nan if what == "nan weight" else np.inf
    w = dev(synth.random_tl1_packed(rng, N, K))
    for epi in (kernels.EPI_STORE, kernels.EPI_RELU2_GLU):
        args = (w, N // 64, K, [0.02, 0.03], [N // 128, N // 64])
        kw = dict(epilogue=epi, norm_w=dev(nw) if norm else None, do_norm=norm, want_acc=True, want_act=True)
        if epi == kernels.EPI_RELU2_GLU and N // 64 % 2:
            continue
        one, two = (kernels.tl1_gemv(dev(v), *args, **kw) for v in (x, np.concatenate([x, x[:, ::-1]])))
        for k in ("a", "inv", "acc", "out"):
            assert np.array_equal(host(one[k])[0], host(two[k])[0], equal_nan=True), f"{k} differs from the batched kernel's"
        if not norm:
            a = np.zeros(K, np.int8)
            inv = ora.load_oracle().ora_act_quant31(ora.ptr(x[0], ora.c_f32p), K, ora.ptr(a, ora.c_i8p))
            assert np.array_equal(host(one["a"])[0], a) and host(one["inv"])[0] == np.float32(inv)
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
