"""The bias gradients of the surrogate's fused backward (default shape) against
the same sums in 64 bits.  The network is chosen so that every summand is known
exactly: a zero lift and zero biases leave every activation 0 (GELU's
derivative 0.5), identity layers without spectral weights pass the gradient on,
and each channel feeds one projection channel, so a summand is a product of two
BF16 values, or dq = 0.5 (W2^T dout) with one FP32 rounding.

Tolerance 2^-23 of a sum (all summands have one sign): half of it is the
rounding of the result to FP32, the other half is for the additions within a
line, whose roundings average out over the lines."""
import numpy as np
import pytest

from oracle import fno_oracle as fo

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("batch", [1, 3, 9])
def test_bias_gradients_are_fp32_sums(lib, batch):
    from atmosphericturbulencesimul_gb300 import fno as F
    cfg = fo.Cfg(nin=8, width=64, modes=32, layers=2, proj=128, nout=2, grid=256)
    lay = fo.layout(cfg)
    p = np.zeros(lay["_total"][1], np.float32)
    rng = np.random.default_rng(batch)
    at = lambda name: slice(lay[name][0], lay[name][0] + lay[name][1])
    bf16 = lambda a: torch.as_tensor(a, dtype=torch.float32).bfloat16()
    W1 = np.zeros((128, 64), np.float32)
    W1[2 * np.arange(64), np.arange(64)] = bf16(rng.uniform(0.5, 2.0, 64)).float().numpy()
    W2 = bf16(rng.uniform(0.5, 2.0, (2, 128))).float().numpy()
    p[at("proj1_W")], p[at("proj2_W")] = W1.ravel(), W2.ravel()
    for l in range(2):
        p[at(f"W{l}")] = np.eye(64, dtype=np.float32).ravel()
    m = F.Surrogate(F.FnoConfig(**cfg.__dict__), seed=1)
    m.set_params(p)
    g = torch.Generator().manual_seed(batch)
    x = torch.randn(batch, 8, 256, 256, generator=g).cuda()
    t = (torch.rand(batch, 2, 256, 256, generator=g) + 1.0).cuda()
    out = torch.empty_like(t)
    m.zero_grads()
    m.loss_grad(x, t, out=out)
    grads = m.get_grads().astype(np.float64)
    m.close()
    assert not out.any()
    dout = (2.0 / np.float32(t.numel())).astype(np.float32).item() * -t
    assert dout.dtype == torch.float32
    d = dout.bfloat16().double()
    w1, w2 = torch.tensor(W1).cuda().double(), torch.tensor(W2).cuda().double()
    want = {"proj2_b": dout.double().sum((0, 2, 3)), "proj1_b": 0.0, "b1": 0.0, "b0": 0.0, "lift_b": 0.0}
    for s in range(batch):
        dq = (w2.T @ d[s].flatten(1)).float() * 0.5
        want["proj1_b"] = want["proj1_b"] + dq.double().sum(1)
        dh = w1.T @ dq.bfloat16().double()                 # one product each: exact
        want["b1"] = want["b1"] + dh.sum(1)
        du = dh.float().bfloat16().double() * 0.5
        want["b0"] = want["b0"] + du.sum(1)
        want["lift_b"] = want["lift_b"] + du.sum(1)
    for name, w in want.items():
        w = w.cpu().numpy()
        err = np.abs(grads[at(name)] - w) / np.abs(w)
        assert err.max() <= 2.0 ** -23, (name, err.max())
    assert lib.atmwfs_fno_umma_status(0) == 0
