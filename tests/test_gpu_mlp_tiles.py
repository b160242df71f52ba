"""The network's gradient at the edges of its tiles (64 samples, one CTA an SM)
against float64 autograd of the same roundings' network, and training that
does not depend on timing: two runs give the same bits."""

import ctypes
import importlib

import numpy as np
import pytest
import torch

import helpers as H

L = importlib.import_module("d3-force-wasm_b200.learned")
pytestmark = pytest.mark.gpu
FP = ctypes.POINTER(ctypes.c_float)


def _samples(n, seed):
    rng = np.random.default_rng(seed)
    return (rng.standard_normal((n, L.N_IN)).astype(np.float32),
            rng.standard_normal((n, L.N_OUT)).astype(np.float32))


def _bf(t):
    """Rounded to bf16 going forward, straight through going back."""
    return t + (t.detach().to(torch.bfloat16).to(t.dtype) - t.detach())


def _reference(x, y, params):
    p = torch.tensor(params, dtype=torch.float64, requires_grad=True)
    o, w = 0, []
    for i, k in ((L.N_IN, L.N_HID), (L.N_HID, L.N_HID), (L.N_HID, L.N_OUT)):
        w.append((_bf(p[o:o + i * k]).reshape(k, i), p[o + i * k:o + i * k + k]))
        o += i * k + k
    h = _bf(torch.tensor(x, dtype=torch.float64))
    for k, (a, b) in enumerate(w):
        h = h @ a.T + b
        if k < 2:
            h = _bf(torch.nn.functional.gelu(h))
    loss = ((h - torch.tensor(y, dtype=torch.float64)) ** 2).sum(1).mean()
    loss.backward()
    return p.grad.numpy(), float(loss.detach())


@pytest.mark.parametrize("n", [1, 63, 64, 65, 1000, 64 * 148, 64 * 148 + 1, 20011])
def test_gpu_mlp_gradient_tiles(gcore, n):
    x, y = _samples(n, n)
    params = L.init_params(3)
    tx, ty = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    grad, loss = np.zeros(L.N_PARAMS, np.float32), ctypes.c_float(0)
    lib = L._bind(gcore.lib)
    rc = lib.d3_mlp_grad(ctypes.c_void_p(tx.data_ptr()), ctypes.c_void_p(ty.data_ptr()), n,
                         params.ctypes.data_as(FP), grad.ctypes.data_as(FP), ctypes.byref(loss))
    assert rc == 0
    ref, ref_loss = _reference(x, y, params)
    # an activation on a bf16 rounding boundary may round the other way in
    # FP32 (2^-8 of its value): at most a few in 64 n, 0.4 % of the whole
    assert np.linalg.norm(grad - ref) <= 4e-3 * np.linalg.norm(ref)
    assert abs(loss.value - ref_loss) <= 4e-3 * ref_loss


@pytest.mark.parametrize("n,batch", [(500, 500), (3000, 1000)])
def test_gpu_mlp_training_repeats(gcore, n, batch):
    x, y = _samples(n, 7)
    a, la = L.train(gcore, x, y, steps=30, batch=batch)
    b, lb = L.train(gcore, x, y, steps=30, batch=batch)
    assert np.array_equal(a, b) and np.array_equal(la, lb)
    assert la[-5:].mean() < la[:5].mean()
