"""BCQ quantiser (the step before the matmul path): oracle pinned on vectors made by the reference's own code;
the device quantiser against the oracle and the same vectors."""
import os

import numpy as np
import pytest

from oracle import bcq_quantizer as bq

GOLD = np.load(os.path.join(os.path.dirname(__file__), "golden", "bcq_quantizer_reference.npz"))
CASES = sorted({k.rsplit("_", 1)[0] for k in GOLD.files})


def _cfg(name):
    N, K, g, q, rounds, _ = (int(v) for v in GOLD[name + "_cfg"])
    return N, K, g, q, rounds


def _compare(alpha, B, alpha_ref, B_ref, w):
    """alpha to fp32 summation-order rounding; codes equal except for weights on a decision boundary, and the
    reconstruction error no worse."""
    assert np.allclose(alpha, alpha_ref, rtol=2e-5, atol=1e-9), np.abs(alpha - alpha_ref).max()
    mismatch = (B != B_ref).any(-1).mean()
    assert mismatch <= 2e-3, mismatch
    N = w.shape[0]
    rec = np.einsum("ngkq,ngq->ngk", B.astype(np.float32), alpha).reshape(N, -1)
    rec_ref = np.einsum("ngkq,ngq->ngk", B_ref.astype(np.float32), alpha_ref).reshape(N, -1)
    e, e_ref = ((rec - w) ** 2).mean(), ((rec_ref - w) ** 2).mean()
    assert e <= e_ref * (1 + 1e-4) + 1e-12, (e, e_ref)


@pytest.mark.parametrize("name", CASES)
def test_oracle_matches_reference_vectors(name):
    N, K, g, q, rounds = _cfg(name)
    w = GOLD[name + "_w"]
    w_hat, B, alpha = bq.quantize(w, q, rounds, g)
    _compare(alpha, B.astype(np.int8), GOLD[name + "_alpha"], GOLD[name + "_B"], w)
    assert np.abs(w_hat - GOLD[name + "_ret"]).max() <= 1e-6


def test_refinement_does_not_increase_the_error():
    rng = np.random.default_rng(0)
    w = rng.normal(0, 0.02, (16, 512)).astype(np.float32)
    errs = [((bq.quantize(w, 3, r, 128)[0] - w) ** 2).mean() for r in (0, 1, 5)]
    assert errs[1] <= errs[0] and errs[2] <= errs[1] * 1.001, errs


@pytest.mark.gpu
@pytest.mark.parametrize("name", CASES)
def test_device_quantiser_matches_reference_vectors(name):
    import lutgemm_b200 as L
    N, K, g, q, rounds = _cfg(name)
    w = GOLD[name + "_w"]
    w_hat, B, alpha = L.bcq_quantize(w, q, rounds, g)
    _compare(alpha, B, GOLD[name + "_alpha"], GOLD[name + "_B"], w)


@pytest.mark.gpu
@pytest.mark.parametrize("N,K,g,q,rounds", [(64, 1024, 128, 3, 15), (48, 768, 32, 4, 6), (8, 2048, 1024, 2, 3),
                                             (33, 640, 64, 8, 2), (16, 4096, 256, 5, 4),
                                             # groups wider than 1024: the CTA-per-group kernel (-1 = one group per row)
                                             (6, 4096, -1, 3, 5), (5, 6144, 2048, 4, 3), (3, 12288, -1, 2, 2), (4, 2080, -1, 1, 0)])
def test_device_quantiser_matches_oracle(N, K, g, q, rounds):
    import lutgemm_b200 as L
    rng = np.random.default_rng(N + K + q)
    w = (rng.standard_t(5, (N, K)) * 0.02).astype(np.float32)
    _, B_ref, alpha_ref = bq.quantize(w, q, rounds, g)
    _, B, alpha = L.bcq_quantize(w, q, rounds, g)
    _compare(alpha, B, alpha_ref, B_ref.astype(np.int8), w)


@pytest.mark.gpu
@pytest.mark.parametrize("N,K,g,q,rounds", [
    # groups up to 512 wide and up to four planes share a warp: every lane count, full and ragged lanes, a group count that
    # is no multiple of a warp's, widths that are no multiple of 4, no refinement at all, weights that are exactly 0
    (5, 192, 64, 3, 4), (7, 96, 32, 2, 3), (3, 512, 512, 4, 5), (9, 400, 400, 3, 3), (11, 200, 50, 3, 3), (13, 129, 43, 4, 2),
    (6, 384, 192, 2, 15), (33, 256, 128, 1, 3), (4, 260, 65, 4, 0), (1, 128, 128, 3, 1)])
def test_device_quantiser_several_groups_per_warp(N, K, g, q, rounds):
    import torch
    import lutgemm_b200 as L
    rng = np.random.default_rng(N * K + q)
    w = (rng.normal(0, 0.02, (N, K))).astype(np.float32)
    w[:, ::17] = 0.0
    _, B_ref, alpha_ref = bq.quantize(w, q, rounds, g)
    _, B, alpha = L.bcq_quantize(w, q, rounds, g)
    _compare(alpha, B, alpha_ref, B_ref.astype(np.int8), w)
    if g % 32 == 0:
        # the container layout holds the same codes (+1 = set bit) and the same scales
        bW, alpha_k = L.bcq_quantize_device(torch.from_numpy(w).cuda(), q, rounds=rounds, group_size=g)
        bits = (B.reshape(N, K // 32, 32, q) > 0).astype(np.uint64) << np.arange(32, dtype=np.uint64)[:, None]
        assert np.array_equal(bW.cpu().numpy().view(np.uint32), bits.sum(2).transpose(1, 2, 0).astype(np.uint32))
        assert np.array_equal(alpha_k.cpu().numpy(), alpha.transpose(1, 2, 0).astype(np.float16))


@pytest.mark.gpu
@pytest.mark.parametrize("N,K,g,q,rounds,zeros", [
    # layers large enough for a group to go to a lane: whole and ragged words, quads and columns, one round, residuals that are
    # 0, a group count that is no multiple of a warp's
    (5, 192, 64, 3, 4, False), (7, 96, 32, 2, 3, True), (3, 512, 512, 4, 5, False), (9, 400, 400, 3, 3, True), (13, 129, 43, 4, 2, False),
    (6, 384, 192, 2, 15, False), (16, 1024, 128, 3, 15, False), (4, 256, 256, 3, 1, True), (11, 200, 50, 3, 3, False)])
def test_device_quantiser_group_per_lane(N, K, g, q, rounds, zeros):
    import torch
    import lutgemm_b200 as L
    rng = np.random.default_rng(N * K + q)
    w = (rng.normal(0, 0.02, (N, K))).astype(np.float32)
    if zeros:
        w[:, ::17] = 0.0
    times = (4 << 20) * (4 if g > 256 else 2 if g > 128 else 1) // w.size + 1
    _, B_ref, alpha_ref = bq.quantize(w, q, rounds, g)
    _, B, alpha = L.bcq_quantize(np.tile(w, (times, 1)), q, rounds, g)
    B, alpha = B.reshape((times, N) + B.shape[1:]), alpha.reshape((times, N) + alpha.shape[1:])
    assert (B == B[0]).all() and (alpha == alpha[0]).all()           # the same rows again, in other lanes and warps
    _, B_small, alpha_small = L.bcq_quantize(w, q, rounds, g)        # the tiled kernel: the same bits
    assert (B_small.reshape(B[0].shape) == B[0]).all() and (alpha_small.reshape(alpha[0].shape) == alpha[0]).all()
    _compare(alpha[0], B[0], alpha_ref, B_ref.astype(np.int8), w)
    if g % 32 == 0:
        bW, alpha_k = L.bcq_quantize_device(torch.from_numpy(np.tile(w, (times, 1))).cuda(), q, rounds=rounds, group_size=g)
        bits = ((B[0].reshape(N, K // 32, 32, q) > 0).astype(np.uint64) << np.arange(32, dtype=np.uint64)[:, None]).sum(2).astype(np.uint32)
        assert (bW.cpu().numpy().view(np.uint32).transpose(2, 0, 1).reshape(times, N, K // 32, q) == bits).all()
        assert (alpha_k.cpu().numpy().transpose(2, 0, 1).reshape(times, N, K // g, q) == alpha[0].astype(np.float16)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("g,q,rounds", [(64, 2, 4), (128, 3, 3), (96, 4, 3)])
def test_device_quantiser_group_per_lane_of_the_smallest_weights(g, q, rounds):
    """Weights of a few times the smallest float, where the float below a weight is no rounding of a sum: large layers, a group to
    a lane, and small ones, several to a warp, get the same bits."""
    import lutgemm_b200 as L
    rng = np.random.default_rng(g + q)
    w = (rng.integers(-40, 41, (33, 4 * g)) * 2.0 ** -149).astype(np.float32)
    times = (4 << 20) // w.size + 1
    _, B, alpha = L.bcq_quantize(np.tile(w, (times, 1)), q, rounds, g)
    _, B_small, alpha_small = L.bcq_quantize(w, q, rounds, g)
    B, alpha = B.reshape((times,) + B_small.shape), alpha.reshape((times,) + alpha_small.shape)
    assert (alpha_small > 0).any()
    assert (alpha == alpha_small).all() and (B == B_small).all()


@pytest.mark.gpu
@pytest.mark.parametrize("g,q,rounds", [(64, 2, 4), (128, 3, 3), (96, 4, 3)])
def test_device_quantiser_group_per_lane_weights_not_finite(g, q, rounds):
    """A group with an infinite or NaN weight has no scales (NaN), and its neighbours keep their bits."""
    import lutgemm_b200 as L
    rng = np.random.default_rng(g + q)
    w = rng.normal(0, 0.02, ((4 << 20) // (4 * g) + 1, 4 * g)).astype(np.float32)
    _, B, alpha = L.bcq_quantize(w, q, rounds, g)
    bad = np.zeros(alpha.shape[:2], dtype=bool)
    for i, value in enumerate((np.inf, -np.inf, np.nan)):
        w[5 + 40 * i, g + 3] = value
        bad[5 + 40 * i, 1] = True
    _, B_bad, alpha_bad = L.bcq_quantize(w, q, rounds, g)
    assert np.isnan(alpha_bad[bad]).all()
    assert (alpha_bad[~bad] == alpha[~bad]).all() and (B_bad[~bad] == B[~bad]).all()


@pytest.mark.gpu
def test_device_quantiser_feeds_the_matmul():
    """Quantise on the device straight into the container layout, multiply, compare with x W_hat^T from the oracle."""
    import torch
    import lutgemm_b200 as L
    from lutgemm_b200 import synth
    from parity_utils import MAE, MAX_REL, error_metrics
    N, K, g, q = 512, 1024, 128, 3
    rng = np.random.default_rng(3)
    w = rng.normal(0, 0.02, (N, K)).astype(np.float32)
    bW, alpha = L.bcq_quantize_device(torch.from_numpy(w).cuda(), q, rounds=5, group_size=g)
    nq = L.nQWeight_fp16.from_device(bW, alpha, None, K, N, q, False, K // g, copy=False)
    x = synth.activations(1, K, seed=1)
    y = torch.empty((1, N), dtype=torch.float16, device="cuda")
    L.matmul(y, torch.from_numpy(x.view(np.int16)).cuda().view(torch.float16), nq, 1)
    _, B_ref, alpha_ref = bq.quantize(w, q, 5, g)
    a16 = alpha_ref.astype(np.float16).astype(np.float32)
    w_hat16 = np.einsum("ngkq,ngq->ngk", B_ref, a16).reshape(N, K)
    ref = x.astype(np.float32) @ w_hat16.T
    rel, mae = error_metrics(y.float().cpu().numpy(), ref)
    assert rel <= 2 * MAX_REL and mae <= 2 * MAE, (rel, mae)       # a few boundary codes may differ from the oracle's
