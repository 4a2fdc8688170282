"""The learned warm start's GPU kernels: the BF16 tensor-core GEMM and the MLP's forward / backward pass, checked
against the FP64 numpy restatement in oracle/mlp_oracle.py (which rounds to bfloat16 where the GPU stores
bfloat16, so the comparison measures the FP32 accumulation, not the input rounding)."""
import ctypes as C

import numpy as np
import pytest

import mlp_oracle
import pdhg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("M,N,K,slices", [(256, 384, 512, 1), (37, 203, 91, 1), (64, 512, 4096, 8), (128, 1000, 256, 3)])
def test_gemm_bf16(engine_lib, ta, tb, M, N, K, slices):
    import torch
    rng = np.random.default_rng(M + N + K)
    A = mlp_oracle.bf16(rng.standard_normal((K, M) if ta else (M, K)))
    B = mlp_oracle.bf16(rng.standard_normal((N, K) if tb else (K, N)))
    dev = torch.device("cuda")
    dA = torch.tensor(A, dtype=torch.bfloat16, device=dev)
    dB = torch.tensor(B, dtype=torch.bfloat16, device=dev)
    dC = torch.zeros((M, N), dtype=torch.float32, device=dev)
    ws = torch.zeros(slices * M * N, dtype=torch.float32, device=dev)
    code = pdhg.lib().taral_gemm_bf16(M, N, K, ta, tb, C.c_void_p(dA.data_ptr()), C.c_void_p(dB.data_ptr()),
                                      C.c_void_p(dC.data_ptr()), slices, C.c_void_p(ws.data_ptr()), None)
    assert code == pdhg.OK
    torch.cuda.synchronize()
    ref = (A.T if ta else A) @ (B.T if tb else B)
    got = dC.cpu().numpy().astype(np.float64)
    assert np.max(np.abs(got - ref)) <= 1e-5 * np.sqrt(K) * np.max(np.abs(ref)) + 1e-6


def test_mlp_gradients_match_oracle(engine_lib):
    net = pdhg.Mlp(24, 64, 3, 136, max_batch=32)
    net.init(seed=3)
    p = net.get_params().astype(np.float64)
    rng = np.random.default_rng(1)
    x = rng.standard_normal((20, 24))
    t = rng.standard_normal((20, 136)) * 0.5
    y_gpu = net.forward(x)
    y_ref, _, _ = mlp_oracle.forward(p, net.shapes(), x)
    assert np.max(np.abs(y_gpu - y_ref)) <= 2e-3 * (1 + np.max(np.abs(y_ref)))
    loss, g = net.gradients(x, t)
    loss_ref, g_ref = mlp_oracle.loss_and_grads(p, net.shapes(), x, t)
    assert abs(loss - loss_ref) <= 1e-3 * loss_ref
    k = 0
    for (fi, fo), _ in net.shapes():  # per tensor: relative error of the gradient in the 2-norm
        for size in (fi * fo, fo):
            a, b = g[k:k + size], g_ref[k:k + size]
            assert np.linalg.norm(a - b) <= 2e-2 * np.linalg.norm(b) + 1e-9, (k, size)
            k += size


def test_mlp_training_reduces_loss(engine_lib):
    rng = np.random.default_rng(0)
    x = rng.uniform(-1, 1, (512, 16))
    Wt = rng.standard_normal((16, 200)) * 0.5
    t = np.tanh(x @ Wt)  # a smooth target the network can fit
    net = pdhg.Mlp(16, 128, 3, 200, max_batch=64)
    net.init(seed=0)
    l0, _ = net.gradients(x[:64], t[:64])
    net.set_dataset(x, t)
    last = net.train(epochs=40, batch=64, lr=2e-3, seed=1)
    assert last < 0.1 * l0, (l0, last)


@pytest.mark.parametrize("dims,batch", [
    ((256, 64, 2, 901), 16),   # tcgen05 throughout, ragged output width
    ((24, 40, 1, 33), 130),    # more rows than one tile, widths below a tile
    ((20, 24, 1, 50), 8),      # input width not a multiple of 8: the first layer on mma.sync
    ((16, 12, 2, 70), 9),      # hidden width not a multiple of 8: products on both paths in one network
    ((16, 16, 1, 40), 300),    # rows in more than one chunk of the column sums
])
def test_mlp_training_step_is_adam_on_the_gradients(engine_lib, dims, batch):
    """Every step of train() on one batch moves each parameter by Adam's step on what gradients() reports for it. The
    weights' gradients come from the same products, so the difference is rounding: a few ulp of the step, and the bias
    corrections 1 - b^t formed in FP32 (an ulp of 0.999^t is 6e-5 of 1 - 0.999^t, 3e-5 of the step), plus an ulp of the
    parameter."""
    net = pdhg.Mlp(*dims, max_batch=batch)
    net.init(3)
    rng = np.random.default_rng(4)
    x = rng.standard_normal((batch, dims[0])).astype(np.float32)
    t = rng.standard_normal((batch, dims[3])).astype(np.float32)
    net.set_dataset(x, t)
    lr, b1, b2 = 1e-3, np.float64(np.float32(0.9)), np.float64(np.float32(0.999))
    w = net.get_params().astype(np.float64)
    m, v = np.zeros_like(w), np.zeros_like(w)
    for step in range(1, 4):
        before, grads = net.gradients(x, t)
        loss = net.train(epochs=1, batch=batch, lr=lr, seed=step)
        assert abs(loss - before) <= 1e-5 * abs(before)  # rows in another order
        g = grads.astype(np.float64)
        m, v = b1 * m + (1 - b1) * g, b2 * v + (1 - b2) * g * g
        c1, c2 = (np.float64(np.float32(1) - np.float32(b) ** np.float32(step)) for b in (b1, b2))
        expected = w - lr * (m / c1) / (np.sqrt(v / c2) + 1e-8)
        w = net.get_params().astype(np.float64)
        # the shuffled rows change the summation order of the gradients: 1e-5 of a gradient's size moves a step by
        # at most lr * 1e-5 * max|g| / (|g| + eps)
        slack = lr * np.minimum(2.0, 1e-5 * np.max(np.abs(g)) / (np.abs(g) + 1e-8))
        assert np.all(np.abs(w - expected) <= lr * 1e-4 + slack + 1.3e-7 * np.abs(expected)), step


@pytest.mark.parametrize("entries", [(1 << 20) - 1, 1 << 20, (1 << 20) + 1, 20 * (1 << 17) - 3, 33 * (1 << 17) + 5])
def test_mlp_large_transfers(engine_lib, entries, monkeypatch):
    """Transfers below, at and above the size from which several threads share them, with ragged last chunks and fewer or
    more chunks than threads: the same bytes as the runtime's own copies give, also into pinned memory."""
    import torch
    rng = np.random.default_rng(entries)
    p = rng.standard_normal(2 * entries).astype(np.float32)  # one layer of 1 x entries: weights and biases
    x = rng.standard_normal((1, 1)).astype(np.float32)
    t = rng.standard_normal((1, entries)).astype(np.float32)
    got = {}
    for threads in ("0", "16", None):
        if threads is None:
            monkeypatch.delenv("TARAL_STAGING")
        else:
            monkeypatch.setenv("TARAL_STAGING", threads)
        net = pdhg.Mlp(1, 8, 0, entries, max_batch=1)
        net.set_params(p)
        assert np.array_equal(net.get_params(), p)
        pinned = torch.zeros(2 * entries, dtype=torch.float32, pin_memory=True)
        net._err(pdhg.lib().taral_mlp_get_params(net.h, C.cast(pinned.data_ptr(), C.POINTER(C.c_float))))
        assert np.array_equal(pinned.numpy(), p)
        loss, g = net.gradients(x, t)
        got[threads] = (net.forward(x), np.float64(loss), g)
        net.close()
    for threads in ("16", None):
        for a, b in zip(got["0"], got[threads]):
            assert np.array_equal(a, b)
