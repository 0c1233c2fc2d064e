"""The learned predictor's tensor-core kernels against the network oracle, and its training loop.

Forward and backward run as BF16 products on the tcgen05 tensor cores with FP32 accumulation; the
oracle (oracle/mlp.py) rounds to BF16 at the same points and sums in float64, so the two agree to
FP32 summation order plus the occasional BF16 rounding flip that it causes (tolerances below)."""
import numpy as np
import pytest

from oracle import mlp as om

pytestmark = pytest.mark.gpu


def _net(seed=3):
    from dac_vtsa_b200.predictor import NewtonPredictor
    net = NewtonPredictor(sample_capacity=0, seed=seed)
    P = om.init_params(seed=seed + 2, scale_out=1.0)
    nrm = np.zeros(32)
    nrm[:20] = [0.02, 0.5, 40, 1, 5, 1e7, 2e-3, 5e-2, 4, 0.1, 0.5, 1e6, 10, 1, 1, 1, 1, 1, 1, 8]
    net.set_params(P, nrm)
    return net, P


def _inputs(rows, seed):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((rows, om.NIN)).astype(np.float32)
    X[:, 97:] = 0.0
    T = rng.standard_normal((rows, 8)).astype(np.float32)
    return X, T


@pytest.mark.parametrize("rows", [128, 300, 1000])
def test_forward_matches_oracle(rows):
    net, P = _net()
    X, _ = _inputs(rows, rows)
    out = net.forward(X)
    ref, _ = om.forward(P, X)
    assert out.shape == (rows, om.NOUT)
    err = np.abs(out - ref).max() / np.abs(ref).max()
    assert err < 2e-2, err


def test_parameters_round_trip():
    net, P = _net()
    P2, nrm = net.params()
    assert np.array_equal(P2, P)
    assert nrm[12] == 10.0


@pytest.mark.parametrize("rows", [700, 4096])
def test_gradient_matches_oracle(rows):
    """Every parameter block of the backward kernels' gradient against the oracle's (BF16-rounded
    back-propagation), and the loss."""
    net, P = _net()
    X, T = _inputs(rows, 7 + rows)
    g, L = net.gradient(X, T)
    go, Lo = om.gradient(P, X, T)
    assert L == pytest.approx(Lo, rel=2e-3)
    o = 0
    for name, shape in om.SIZES:
        n = int(np.prod(shape))
        a, b = g[o:o + n].astype(np.float64), go[o:o + n]
        o += n
        if name == "b4":
            b = b.copy()
        rel = np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)
        assert rel < 2e-2, (name, rel)


def test_training_reduces_the_loss_on_recorded_stage_solutions():
    """Samples recorded from the plain solver's own stage solutions (4x4x16 adsorption, every cell of
    every converged stage), then Adam on the GPU: the batch loss falls well below its starting value
    (the untrained network predicts no correction)."""
    import json
    import torch
    from cases import golden, build
    from dac_vtsa_b200.model import TVSAModel
    from dac_vtsa_b200.predictor import NewtonPredictor
    from dac_vtsa_b200.solver import TRBDF2
    d = golden("trajectory_c0.npz")
    over = json.loads(str(d["over"]))
    meta = json.loads(str(d["s0_meta"]))
    m, cfg = build(TVSAModel, over, meta["step"], d["s0_P0"], meta["T_jacket_prev"], duration=meta["duration"])
    net = NewtonPredictor(sample_capacity=1 << 16, seed=1)
    integ = TRBDF2(m, cfg, h_max=cfg.solver.h_max_fraction * meta["duration"])
    net.attach(integ, "adsorption", predict=False, record_stride=1)
    res = integ.integrate(d["s0_y0"], meta["duration"], [meta["duration"]])
    assert res.t == pytest.approx(meta["duration"])
    assert net.samples >= 4096, net.samples
    hist = net.train(300, lr=2e-3, seed=5)
    torch.cuda.synchronize()
    assert np.all(np.isfinite(hist))
    first, last = float(np.mean(hist[:10])), float(np.mean(hist[-20:]))
    assert last < 0.5 * first, (first, last)


@pytest.mark.parametrize("M,N,K", [(128, 16, 16), (128, 112, 64), (256, 128, 400), (128, 48, 448), (384, 128, 1040)])
def test_product_kernel_over_ring_and_remainders(M, N, K):
    """The product kernel with fewer, as many and more 64-column chunks than it stages, and with a last chunk
    of part of the columns: exact BF16 inputs, FP32 accumulation (error at most K steps of 2^-24 on the sum
    of the magnitudes)."""
    import ctypes as C
    from dac_vtsa_b200 import _lib
    rng = np.random.default_rng(M + N + K)
    A, B = (rng.integers(-64, 65, s).astype(np.float32) / 64 for s in ((M, K), (N, K)))      # 7 bits: exact in BF16
    A *= 2.0 ** rng.integers(-6, 7, (M, 1)).astype(np.float32)
    D = np.full((M, N), np.nan, dtype=np.float32)
    ptr = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert _lib.load().dv_mlp_gemm_host(M, N, K, ptr(A), ptr(B), ptr(D)) == 0
    ref = A.astype(np.float64) @ B.astype(np.float64).T
    bound = K * 2.0 ** -24 * (np.abs(A).astype(np.float64) @ np.abs(B).astype(np.float64).T)
    assert (np.abs(D - ref) <= bound + 2.0 ** -24 * np.abs(ref)).all()


def _drawn(seed, step, count):
    """Sample indices of a training batch: the library's hash of seed, step and row."""
    with np.errstate(over="ignore"):
        x = (np.uint64(seed) * np.uint64(0x9E3779B97F4A7C15) + np.uint64(step) * np.uint64(1000003)
             + np.arange(4096, dtype=np.uint64))
        x ^= x >> np.uint64(30)
        x *= np.uint64(0xBF58476D1CE4E5B9)
        x ^= x >> np.uint64(27)
        x *= np.uint64(0x94D049BB133111EB)
        x ^= x >> np.uint64(31)
    return (x % np.uint64(count)).astype(np.int64)


def test_training_step_on_a_drawn_batch_matches_oracle():
    """The batch a training step draws (hash, scaled and clipped targets, its transposed copy) against the
    oracle on the same rows: the loss of 70 steps at learning rate 0 (more than are read back together), and
    every block of the gradient, recovered from Adam's first step p - lr g / (|g| + 1e-8).  Outputs and targets
    of about 1e-5 keep |g| where that step is far from saturated: |g| from 1e-13 (a change of 1e-5, FP32
    parameters resolve 1e-8 of it) to 1e-5 (1 - |step| = 1e-3, resolved to 1e-4).  Tolerances of the tests above."""
    import json
    from cases import build, golden
    from dac_vtsa_b200.model import TVSAModel
    from dac_vtsa_b200.predictor import NewtonPredictor
    from dac_vtsa_b200.solver import TRBDF2
    d = golden("trajectory_c0.npz")
    meta = json.loads(str(d["s0_meta"]))
    m, cfg = build(TVSAModel, json.loads(str(d["over"])), meta["step"], d["s0_P0"], meta["T_jacket_prev"],
                   duration=meta["duration"])
    net = NewtonPredictor(sample_capacity=1 << 14, seed=1)
    integ = TRBDF2(m, cfg, h_max=cfg.solver.h_max_fraction * meta["duration"])
    net.attach(integ, "adsorption", predict=False, record_stride=1)
    integ.integrate(d["s0_y0"], meta["duration"], [meta["duration"]])
    X, T = net.get_samples()
    P = om.init_params(seed=9, scale_out=1e-5)
    P[-om.NOUT:] *= 1e-4
    nrm = net.params()[1]
    nrm[13:19] = 1e5 * np.maximum(np.sqrt(np.mean(T[:, :6].astype(np.float64) ** 2, axis=0)), 1e-6)
    nrm[19] = 2e-5
    tgt = np.clip(T[:, :6].astype(np.float64) / nrm[13:19], -nrm[19], nrm[19]).astype(np.float32)
    assert (np.abs(tgt) == np.float32(nrm[19])).any()
    seed = 123456789
    net.set_params(P, nrm)
    hist = net.train(70, lr=0.0, seed=seed, keep_scales=True)
    out, _ = om.forward(P, X)
    err = ((out[:, :6] - tgt) ** 2).mean(axis=1)
    ref = np.array([err[_drawn(seed, k, len(X))].mean() for k in range(70)])
    assert np.ptp(ref) > 10 * 2e-3 * ref.mean()                  # the batches differ by more than the tolerance
    assert np.abs(hist / ref - 1.0).max() < 2e-3
    net.set_params(P, nrm)                                       # the optimiser starts again, with batch 0
    net.train(1, lr=1.0, seed=seed, keep_scales=True)
    step = P.astype(np.float64) - net.params()[0].astype(np.float64)
    g = 1e-8 * step / (1.0 - np.abs(step))
    rows = _drawn(seed, 0, len(X))
    go, _ = om.gradient(P, X[rows], np.pad(tgt[rows], ((0, 0), (0, 2))))
    o = 0
    for name, shape in om.SIZES:
        n = int(np.prod(shape))
        a, b = g[o:o + n], go[o:o + n]
        o += n
        rel = np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)
        assert rel < 2e-2, (name, rel)
