"""ops.device_min at the edges of its grid: one block, several, and blocks that
stride (more than 296 blocks of 1024 values)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 4096, 4097, 303_103, 303_104, 303_105, 3_000_001])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_min_is_exact_wherever_it_lies(cuda, n, dtype):
    from hipims_b200 import ops

    x = torch.rand(n, dtype=dtype, device=cuda) + 1.0
    for at in {0, n // 2, n - 1}:
        y = x.clone()
        y[at] = -3.0
        for _ in range(2):  # the workspace's counter is left at zero
            assert float(ops.device_min(y)) == -3.0
    assert torch.equal(ops.device_min(x), x.min().reshape(1))
