"""GPU test of the training kernel in builds of other feature step counts (more inputs than one group of 64 columns):
its gradients against 64-bit autograd, at the bars of the default build's test."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest
import torch

from megamol_gb300 import build as nbuild

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
H = 64


@pytest.mark.parametrize("steps", [8, 16])
def test_gradients_of_wider_inputs(tmp_path, steps):
    so = str(tmp_path / "train.so")
    subprocess.run([nbuild.nvcc(), *nbuild.ARCH, *nbuild.NVCC_FLAGS, f"-DP2V_MLP_FSTEPS_BUILD={steps}", "-shared",
                    os.path.join(HERE, "mlp_train_step.cu"), os.path.join(nbuild.CSRC, "mlp.cu"), "-o", so], check=True)
    lib = C.CDLL(so)
    k = lib.inputs()
    assert k == 8 * steps + 6
    rng = np.random.default_rng(steps)
    shapes = [(H, k), (H,), (H, H), (H,), (H,), (1,)]
    w = [rng.normal(0.0, 0.2, s).astype(np.float32) for s in shapes]
    n = 304 * 16 + 37  # a second group of samples for some CTAs, the last one ragged
    x = rng.uniform(0, 1, (n, k)).astype(np.float32)
    t = rng.uniform(0, 1, n).astype(np.float32)
    flat = np.concatenate([a.ravel() for a in w])
    grad = np.empty(flat.size + 1, np.float32)
    f32 = lambda a: a.ctypes.data_as(C.POINTER(C.c_float))
    assert lib.train_step(f32(flat), f32(x), f32(t), n, f32(grad)) == 0
    p = [torch.tensor(a, dtype=torch.float64, requires_grad=True) for a in w]
    h = torch.nn.functional.silu(torch.tensor(x, dtype=torch.float64) @ p[0].T + p[1])
    h = torch.nn.functional.silu(h @ p[2].T + p[3])
    loss = ((torch.sigmoid(h @ p[4] + p[5]) - torch.tensor(t, dtype=torch.float64)) ** 2).mean()
    loss.backward()
    ref = np.concatenate([a.grad.numpy().ravel() for a in p])
    assert abs(grad[-1] / n - loss.item()) <= 1e-5 * max(1.0, loss.item())
    rel = np.abs(grad[:-1] - ref).max() / np.abs(ref).max()
    assert rel <= 1e-4, rel
