"""Camera and background floats are read in place where the tensor's memory
holds its values, and converted otherwise."""
import ctypes

import numpy as np
import pytest
import torch

from polysplat_gb300 import ops


def _floats(p, n):
    return list(ctypes.cast(p, ctypes.POINTER(ctypes.c_float))[:n])


def _forms():
    t = torch.arange(1.0, 10.0)
    z = torch.complex(torch.zeros(9), t).conj()
    return {"plain": t, "view": torch.arange(0.0, 12.0)[1:10], "matrix": t.reshape(3, 3), "transposed": t.reshape(3, 3).t(),
            "strided": torch.arange(0.0, 18.0)[::2], "double": t.double(), "half": t.half(), "gradient": t.clone().requires_grad_(),
            "negated": torch._neg_view(t), "imaginary": torch.imag(z), "numpy": t.numpy(), "list": t.tolist()}


@pytest.mark.parametrize("form", sorted(_forms()))
def test_host_floats_are_the_tensors_values(form):
    t = _forms()[form]
    want = np.asarray(t.detach().float().resolve_neg().reshape(-1) if isinstance(t, torch.Tensor) else t, np.float32)
    assert _floats(ops._host_floats(t, 9, "t"), 9) == want.tolist()
    with pytest.raises(ValueError):
        ops._host_floats(t, 10, "t")
