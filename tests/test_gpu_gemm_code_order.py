"""Tensor-core TL1 product: the order of K in which codes and activations meet (codes left in place, even activations times
four, sums shifted back). Accumulators, plain activations and outputs bit for bit against the CPU, with the quantiser's
register path and its element-by-element path (rows above 14336, rows not on a 16-byte boundary), the smallest K, all four K
splits and weights and activations at their extremes, where the scaled sums are largest."""
import numpy as np
import pytest
import torch
from gpu_helpers import cpu_bitlinear, cpu_rms_norm, dev, host
from helpers import ora, synth

pytestmark = pytest.mark.gpu
P = ora.ptr


@pytest.mark.parametrize("N,K,batch,aligned,extreme", [
    (128, 128, 9, True, False), (64, 256, 16, False, False), (192, 640, 17, True, True), (128, 2560, 70, True, False),
    (128, 6912, 9, False, True), (2560, 1024, 33, True, False), (128, 14464, 12, True, True)])
def test_order_of_codes_and_activations(cuda_lib, N, K, batch, aligned, extreme):
    from tenzo_b200 import kernels
    rng = np.random.default_rng([91, N, K, batch])
    w = synth.random_tl1_packed(rng, N, K)
    x = rng.standard_normal((batch, K)).astype(np.float32)
    if extreme:                                              # every code 2, every activation +31: the largest sum there is
        w = np.full_like(w, 0xAA)
        x[:] = 1.0
        x[1::2] = -1.0
        x[2, ::3] = 0.5
    flat = torch.zeros(batch * K + 1, device="cuda")
    dx = flat[:-1] if aligned else flat[1:]                  # one float off a 16-byte boundary
    dx = dx.view(batch, K)
    dx.copy_(dev(x))
    r = kernels.tl1_gemv(dx, dev(w), N // 64, K, [0.016], want_acc=True, want_act=True)
    torch.cuda.synchronize()
    acc, act, out = host(r["acc"]), host(r["a"]), host(r["out"])
    for b in range(batch):
        want_out, want_acc, inv = cpu_bitlinear(x[b], w, N, K, 0.016)
        a = np.zeros(K, np.int8)
        ora.load_oracle().ora_act_quant31(P(x[b], ora.c_f32p), K, P(a, ora.c_i8p))
        assert np.array_equal(act[b], a)
        assert np.array_equal(acc[b], want_acc), f"sequence {b}"
        assert np.array_equal(out[b], want_out), f"sequence {b}"


@pytest.mark.parametrize("K,batch", [(6912, 297), (4224, 300), (14336, 149)])
def test_many_rows_quantiser(cuda_lib, K, batch):
    """More rows than the quantiser that holds the norm's weights has places for: the one that loads them late, same bits."""
    from tenzo_b200 import kernels
    rng = np.random.default_rng([92, K, batch])
    N = 64
    w, nw = synth.random_tl1_packed(rng, N, K), (1.0 + 0.1 * rng.standard_normal(K)).astype(np.float32)
    x = rng.standard_normal((batch, K)).astype(np.float32)
    r = kernels.tl1_gemv(dev(x), dev(w), N // 64, K, [0.016], norm_w=dev(nw), do_norm=True, want_acc=True, want_act=True)
    few = kernels.tl1_gemv(dev(x[:12]), dev(w), N // 64, K, [0.016], norm_w=dev(nw), do_norm=True, want_acc=True, want_act=True)
    torch.cuda.synchronize()
    assert all(np.array_equal(host(r[k])[:12], host(few[k])) for k in ("a", "inv", "acc", "out"))
    for b in (0, 1, batch // 2, batch - 1):
        want_out, want_acc, _ = cpu_bitlinear(cpu_rms_norm(x[b], nw), w, N, K, 0.016)
        assert np.array_equal(host(r["acc"])[b], want_acc) and np.array_equal(host(r["out"])[b], want_out), f"sequence {b}"


@pytest.mark.parametrize("N,K,B", [(2560, 2560, 65), (2560, 2560, 97), (3840, 2560, 129), (3840, 2560, 257), (640, 5120, 161), (2560, 1280, 337),
                                   (640, 2560, 513), (13824, 384, 385), (1344, 2560, 305), (3840, 1280, 1537)])
def test_tiles_of_sequences_match_one_tile(cuda_lib, N, K, B):
    """Sequences over several CTAs a row tile, the last tile of them ragged: every epilogue gives what a call for up to 64 of the sequences does."""
    from tenzo_b200 import kernels
    rng = np.random.default_rng([97, N, K, B])
    w, x = dev(synth.random_tl1_packed(rng, N, K)), dev(rng.standard_normal((B, K)).astype(np.float32))
    res, nw = dev(rng.standard_normal((B, N)).astype(np.float32)), dev((1 + 0.1 * rng.standard_normal(K)).astype(np.float32))
    for epi in (kernels.EPI_STORE, kernels.EPI_RESIDUAL) + ((kernels.EPI_RELU2_GLU,) if N // 64 % 2 == 0 else ()):
        glu = epi == kernels.EPI_RELU2_GLU

        def run(a, r):
            return kernels.tl1_gemv(a, w, N // 64, K, [0.02, 0.03] if glu else [0.02], [N // 128, N // 64] if glu else None, epilogue=epi,
                                    resid=r if epi == kernels.EPI_RESIDUAL else None, norm_w=nw, do_norm=True)["out"]

        many = run(x, res)
        few = torch.cat([run(x[i:i + 64].contiguous(), res[i:i + 64].contiguous()) for i in range(0, B, 64)])
        assert torch.equal(many, few), f"epilogue {epi}: {int((many != few).any(1).sum())} sequences differ"
    assert cuda_lib.tenzo_cuda_tl1_gemv_take_timeouts() == 0


@pytest.mark.parametrize("N,K,B,sequences,ksplit", [(4096, 14336, 128, 128, 4), (4096, 14336, 144, 144, 4), (4096, 14336, 240, 240, 4), (4096, 14336, 256, 256, 4),
                                                    (4096, 14336, 320, 160, 2), (4096, 14336, 497, 256, 2), (768, 16384, 206, 112, 8), (768, 16384, 320, 160, 8),
                                                    (512, 14336, 390, 144, 8)])
def test_clusters_with_four_activation_tiles(cuda_lib, N, K, B, sequences, ksplit):
    """K split over a cluster whose CTAs hold more than 96 sequences each (four activation tiles, the partial tiles in the rings): every epilogue gives
    what calls for up to 64 of the sequences do, and those of eight on the other path. The shapes are the chosen ones, for 148 SMs."""
    from tenzo_b200 import kernels
    rng = np.random.default_rng([98, N, K, B])
    w, x = dev(synth.random_tl1_packed(rng, N, K)), dev(rng.standard_normal((B, K)).astype(np.float32))
    res, nw = dev(rng.standard_normal((B, N)).astype(np.float32)), dev((1 + 0.1 * rng.standard_normal(K)).astype(np.float32))
    for epi in (kernels.EPI_STORE, kernels.EPI_RESIDUAL, kernels.EPI_RELU2_GLU):
        glu = epi == kernels.EPI_RELU2_GLU
        assert cuda_lib.tenzo_cuda_tl1_gemm_sequences(N // 64, K, B, epi) == sequences > 96
        assert cuda_lib.tenzo_cuda_tl1_gemm_ksplit(N // 64, K, B, epi) == ksplit > 1

        def run(i, n):
            return kernels.tl1_gemv(x[i:i + n].contiguous(), w, N // 64, K, [0.02, 0.03] if glu else [0.02], [N // 128, N // 64] if glu else None, epilogue=epi,
                                    resid=res[i:i + n].contiguous() if epi == kernels.EPI_RESIDUAL else None, norm_w=nw, do_norm=True)["out"]

        many = run(0, B)
        few = torch.cat([run(i, 64) for i in range(0, B, 64)])
        assert torch.equal(many, few), f"epilogue {epi}: {int((many != few).any(1).sum())} sequences differ"
        for i in (0, sequences - 8, B - 8):
            assert torch.equal(many[i:i + 8], run(i, 8)), f"epilogue {epi}, sequences from {i}"
    assert cuda_lib.tenzo_cuda_tl1_gemv_take_timeouts() == 0


@pytest.mark.parametrize("N,K,B,plain", [(13824, 2560, 385, 208), (13824, 384, 416, 208), (4096, 4096, 897, 240), (2560, 2560, 1345, 208)])
def test_tiles_of_sequences_by_the_rounds_of_their_stores(cuda_lib, N, K, B, plain):
    """Tiles whose stores would take two rounds more than those of 16 sequences more give way to them where a unit does more than store; all give what a
    call for up to 64 of the sequences does."""
    from tenzo_b200 import kernels
    rng = np.random.default_rng([99, N, K, B])
    w, x = dev(synth.random_tl1_packed(rng, N, K)), dev(rng.standard_normal((B, K)).astype(np.float32))
    res = dev(rng.standard_normal((B, N)).astype(np.float32))
    for epi in (kernels.EPI_STORE, kernels.EPI_RESIDUAL, kernels.EPI_RELU2_GLU):
        glu = epi == kernels.EPI_RELU2_GLU
        assert cuda_lib.tenzo_cuda_tl1_gemm_sequences(N // 64, K, B, epi) == (plain if epi == kernels.EPI_STORE else plain + 16)

        def run(i, n):
            return kernels.tl1_gemv(x[i:i + n].contiguous(), w, N // 64, K, [0.02, 0.03] if glu else [0.02], [N // 128, N // 64] if glu else None, epilogue=epi,
                                    resid=res[i:i + n].contiguous() if epi == kernels.EPI_RESIDUAL else None)["out"]

        assert torch.equal(run(0, B), torch.cat([run(i, 64) for i in range(0, B, 64)])), f"epilogue {epi}"
    assert cuda_lib.tenzo_cuda_tl1_gemv_take_timeouts() == 0
