"""The surrogate's prediction kernels at the edges of their tiles: the fused
forward pass against an FP64 restatement with the same BF16 rounding points,
its reciprocal against the IEEE division, and the screen's narrow gene tile."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _forward(p, d, x):
    from oracle.mlp_ref import bf16, silu, unpack
    W = unpack(p, d)
    w = {k: bf16(v) if k.startswith("w") else v for k, v in W.items()}
    a = np.zeros((x.shape[0], 16))
    a[:, :x.shape[1]] = x
    a = bf16(a)
    for i in "123":
        a = bf16(silu(a @ w["w" + i] + w["b" + i]))
    return a @ w["w4"] + w["b4"]


@pytest.mark.parametrize("rows,members,K", [(1, 1, 1), (127, 3, 53), (128, 4, 53), (129, 2, 64), (257, 2, 65),
                                            (70000, 4, 53), (300, 2, 128), (130, 1, 129)])
def test_predictions_match_fp64_forward(built, rows, members, K):
    from abc_inference_transcription_gb300.surrogate import Surrogate
    from oracle.mlp_ref import dims
    rng = np.random.default_rng(rows)
    with Surrogate(14, K, ensemble=members, seed=3) as sg:
        sg.set_norm(np.zeros(14), np.ones(14), np.zeros(K), np.ones(K))
        p = sg.params()
        p += rng.normal(0.0, 0.02, p.shape).astype(np.float32)  # biases too
        sg.set_params(p)
        x = rng.normal(size=(rows, 14))
        x[0] *= 40.0  # saturated units
        mean, var, dis = sg.predict(x)
    pick = np.unique(np.concatenate([np.arange(min(rows, 300)), rng.integers(0, rows, 200), [rows - 1]]))
    d = dims(14, K)
    y = np.stack([_forward(p[e], d, x[pick].astype(np.float32).astype(np.float64)) for e in range(members)])
    mu, lv = y[..., :K], np.clip(y[..., K:2 * K], -9.0, 9.0)
    ale, epi = np.exp(lv).mean(0), mu.var(0)
    # activations that round the other way (about 1 in 2,000, by 2^-8) move a sum of 256 terms by ~1e-4 of its size
    tol = 5e-3
    scale = np.sqrt(np.mean(mu ** 2, axis=(0, 2)))[:, None] + 1.0
    assert (np.abs(mean[pick] - mu.mean(0)) <= tol * scale).all()
    assert (np.abs(var[pick] - (ale + epi)) <= 4 * tol * scale ** 2 * (ale + epi + 1.0)).all()
    want = np.sqrt(epi / np.maximum(ale, 1e-12)).max(1)
    assert (np.abs(dis[pick] - want) <= 8 * tol * scale[:, 0] ** 2 * (want + 1.0)).all()


def test_reciprocal_and_sigmoid_equal_division(built, tmp_path):
    so = tmp_path / "librecip.so"
    subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", os.path.join(ROOT, "tests", "gpu_helpers", "recip.cu"), "-o", str(so)], check=True)
    bad = (C.c_ulonglong * 2)(1, 1)
    assert C.CDLL(str(so)).recip_check(bad) == 0
    assert list(bad) == [0, 0]


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("genes,rows", [(1, 127), (16, 129), (17, 300), (32, 128), (33, 1000), (130, 257)])
def test_screen_gene_tiles_agree(built, mode, genes, rows):
    """The bounds of a gene set equal those of its genes screened 20 at a time."""
    torch = pytest.importorskip("torch")
    from abc_inference_transcription_gb300.surrogate import Surrogate
    rng = np.random.default_rng(genes)
    K = 53
    data = rng.normal(size=(genes, K))
    se = 0.1 + rng.random((genes, K))
    thr = np.full(genes, 0.5)
    with Surrogate(14, K, ensemble=2, seed=5) as sg:
        sg.set_norm(np.zeros(14), np.ones(14), np.zeros(K), np.ones(K))
        x = torch.as_tensor(rng.normal(size=(rows, 14)), device="cuda")
        keep = torch.empty(rows, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()

        def bounds(g0, g1):
            low = np.zeros((rows, g1 - g0))
            n = sg.screen_device(x.data_ptr(), 14, rows, data[g0:g1], se[g0:g1], thr[g0:g1], 0.0, 1e9,
                                 keep.data_ptr(), err_out=low, z=0.5, mode=mode)
            return low, keep.cpu().numpy().astype(bool), n

        low, kept, n = bounds(0, genes)
        parts = [bounds(g, min(g + 20, genes)) for g in range(0, genes, 20)]
        assert np.array_equal(low, np.concatenate([p[0] for p in parts], axis=1))
        assert np.array_equal(kept, np.logical_or.reduce([p[1] for p in parts])) and n == kept.sum()
        assert np.array_equal(kept, (low.astype(np.float32) <= np.float32(0.5)).any(axis=1))


@pytest.mark.parametrize("rows,K", [(1, 53), (31, 8), (33, 53), (255, 53), (256, 8), (257, 53), (1100, 53)])
def test_gradients_at_batch_edges(built, rows, K):
    """Batches around the 32 rows of a gradient tile, the 256 rows of a column
    sum's stage and the loss's block partials, outputs with (53) and without (8)
    padding, against the FP64 network that rounds to BF16 where the GPU does.
    Gradients within 2e-2 of their norm, as for the batch of 96."""
    from abc_inference_transcription_gb300 import surrogate as S
    from oracle import mlp_ref

    rng = np.random.default_rng(rows)
    theta, stats = rng.uniform(-3, 3, (rows, 5)), rng.normal(2.0, 1.5, (rows, K))
    if rows > 1:
        stats[0, 2] = np.nan
    with S.Surrogate(5, K, ensemble=2, seed=11) as sg:
        p = sg.params()
        p = p + rng.normal(0, 0.02, p.shape).astype(np.float32)
        sg.set_params(p)
        norm = np.zeros(5), np.full(5, 1.7), np.full(K, 2.0), np.full(K, 1.5)
        sg.set_norm(*norm)
        loss, grads = sg.gradients(theta, stats)
        d = mlp_ref.dims(5, K)
        for e in range(2):
            rl, rg = mlp_ref.loss_and_grads(p[e], d, theta, stats, *norm)
            assert abs(loss[e] - rl) <= 2e-4 * abs(rl) + 1e-6
            for name in ("w1", "b1", "w2", "b2", "w3", "b3", "w4", "b4"):
                a, b = d[name]
                got, want = grads[e, a:b].astype(np.float64), rg[a:b]
                assert np.linalg.norm(got - want) < 2e-2 * max(np.linalg.norm(want), 1e-12), (e, name)


@pytest.mark.parametrize("rows,K", [(130, 140), (257, 120), (20000, 53)])
def test_gradients_of_wide_outputs_and_many_tiles(built, rows, K):
    """Outputs too wide for the fused training passes (280 columns: layer by layer), of
    two output tiles (240), and batches of more row tiles than the GPU has SMs, against the FP64
    network; bounds as above."""
    from abc_inference_transcription_gb300 import surrogate as S
    from oracle import mlp_ref

    rng = np.random.default_rng(rows)
    theta, stats = rng.uniform(-3, 3, (rows, 5)), rng.normal(2.0, 1.5, (rows, K))
    with S.Surrogate(5, K, ensemble=2, seed=12) as sg:
        p = sg.params()
        p = p + rng.normal(0, 0.02, p.shape).astype(np.float32)
        sg.set_params(p)
        norm = np.zeros(5), np.full(5, 1.7), np.full(K, 2.0), np.full(K, 1.5)
        sg.set_norm(*norm)
        loss, grads = sg.gradients(theta, stats)
        d = mlp_ref.dims(5, K)
        for e in range(2):
            rl, rg = mlp_ref.loss_and_grads(p[e], d, theta, stats, *norm)
            assert abs(loss[e] - rl) <= 2e-4 * abs(rl) + 1e-6
            for name in ("w1", "b1", "w2", "b2", "w3", "b3", "w4", "b4"):
                a, b = d[name]
                got, want = grads[e, a:b].astype(np.float64), rg[a:b]
                assert np.linalg.norm(got - want) < 2e-2 * max(np.linalg.norm(want), 1e-12), (e, name)
