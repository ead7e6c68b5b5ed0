"""The batched solver's correction is rounded to FP32 once: it is unscaled in FP64.

After one refinement step from x = 0 the unknowns are the correction itself, the product of two FP32
numbers: 48 significant bits, so that hardly one of them is an FP32 number (a product rounded to
FP32 is one everywhere).
"""
import numpy as np
import pytest

import ffgpu
from ffgpu import batch, mesh

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib_built():
    from ffgpu.build import build
    build()
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    ffgpu.context(0)
    yield


@pytest.mark.parametrize("n", [12, 100])
def test_correction_keeps_the_bits_of_its_product(n):
    m = mesh.square(n, n + 1)
    B = batch.Batch([m])
    B.assemble([np.exp(np.random.Generator(np.random.PCG64(n)).standard_normal(m.nt))])
    x = np.zeros(B.ndof)
    with pytest.raises(ffgpu.FFGPUError):   # one step does not reach this tolerance
        B.solve(eps=1e-14, max_outer=1, out=x)
    free = B.onbc == 0   # (the others start from b/tgv)
    assert np.count_nonzero(x[free]) == (n - 1) * n
    assert np.mean(x[free] == x[free].astype(np.float32)) < 0.1
