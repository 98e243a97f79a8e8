"""Products whose kernels read the caller's operands themselves, over operands that are not one dense matrix."""
import os

import numpy as np
import pytest

from vkml_b200 import DeviceTensor, NodeDesc, Op

pytestmark = pytest.mark.gpu


def context(value):
    import vkml_b200
    os.environ["VKML_B200_GEMM_INLINE"] = value
    b = vkml_b200.Backend(0)
    del os.environ["VKML_B200_GEMM_INLINE"]
    return b


# the largest pitch that TF32 terms are split at inside the kernel, and the first that planes serve; rows 32 and 64 of the right operand's tile are used
@pytest.mark.parametrize("pitch", [(1 << 24) - 4, 1 << 24])
def test_rows_far_apart(pitch):
    import torch
    b = context("8")  # (TF32 terms inside the kernel wherever they fit)
    m, k, n = 300, 1024, 72
    rng = np.random.default_rng(pitch)
    x, w = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal((n, k), dtype=np.float32)
    dx, wide = DeviceTensor.from_host(b, x.reshape(1, 1, m, k)), DeviceTensor.empty(b, (n, pitch))
    b.synchronize()
    face = type("Face", (), {"__cuda_array_interface__": {"shape": (n, pitch), "typestr": "<f4", "data": (wide.desc.data, False), "strides": None, "version": 3}})()
    torch.as_tensor(face, device="cuda")[:, :k] = torch.from_numpy(w).cuda()
    torch.cuda.synchronize()
    dw = DeviceTensor(b, wide.storage, (1, 1, k, n), (0, 0, 4, 4 * pitch), wide.dtype, 0)
    out = DeviceTensor.empty(b, (1, 1, m, n))
    b.compute([NodeDesc(int(Op.MATMUL), out.desc, [dx.desc, dw.desc])])
    want, terms = x.astype(np.float64) @ w.T.astype(np.float64), np.abs(x).astype(np.float64) @ np.abs(w.T).astype(np.float64)
    assert np.all(np.abs(out.numpy().reshape(m, n) - want) <= (k / 8 / 4 * 2.0 ** -23 + 2.0 ** -20) * terms)
    b.close()
