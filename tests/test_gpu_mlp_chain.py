"""The gradient of a large batch: a tile's sum is formed by itself before it is
added to the CTA's, so its error does not grow with the batch as that of one
long chain does. All samples are the same one, so every term of a gradient sum
is equal and the sum's exact value is the one sample's; equal terms lose bits
the same way at every step, the chain's worst case."""

import ctypes
import importlib

import numpy as np
import pytest

import helpers as H  # noqa: F401 (the package on sys.path)

torch = pytest.importorskip("torch")
L = importlib.import_module("d3-force-wasm_b200.learned")
FP = ctypes.POINTER(ctypes.c_float)
pytestmark = pytest.mark.gpu


def _grad(lib, x, y, n, params):
    tx = torch.from_numpy(x).cuda().expand(n, -1).contiguous()
    ty = torch.from_numpy(y).cuda().expand(n, -1).contiguous()
    torch.cuda.synchronize()
    grad, loss = np.zeros(L.N_PARAMS, np.float32), ctypes.c_float(0)
    rc = lib.d3_mlp_grad(ctypes.c_void_p(tx.data_ptr()), ctypes.c_void_p(ty.data_ptr()), n,
                         params.ctypes.data_as(FP), grad.ctypes.data_as(FP), ctypes.byref(loss))
    assert rc == 0
    return grad.astype(np.float64), float(loss.value)


@pytest.mark.parametrize("tiles", [1, 2, 64])
def test_gpu_mlp_gradient_of_a_large_batch(gcore, tiles):
    lib = L._bind(gcore.lib)
    ctas = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(7)
    x = rng.standard_normal((1, L.N_IN)).astype(np.float32)
    y = rng.standard_normal((1, L.N_OUT)).astype(np.float32)
    params = L.init_params(3)
    one, loss1 = _grad(lib, x, y, 1, params)
    many, loss = _grad(lib, x, y, 64 * tiles * ctas, params)
    # roundings a term passes, each at most 2^-24: 64 samples of a tile, the
    # tiles, the CTAs in eight groups and their sum; the terms themselves differ
    # by four (1 / n, and the products that carry it)
    bound = (64 + tiles + (ctas + 7) // 8 + 8 + 4) * 2.0 ** -24
    assert np.abs(many - one).max() > 0 or tiles == 1
    assert (np.abs(many - one) <= bound * np.abs(one)).all()
    assert abs(loss - loss1) <= bound * loss1
