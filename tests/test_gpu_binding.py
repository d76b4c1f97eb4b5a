"""Calls through the compiled binding whose arguments lie at the edge of what it takes."""
import numpy as np
import pytest
import torch

from helpers import normal

pytestmark = pytest.mark.gpu


def cpu(t):
    return t.detach().cpu().numpy()


@pytest.mark.parametrize("shape", [(2, 8), (4, 4), (6, 40), (34, 1544)])
def test_materialize_rows_of_partial_groups(pkg, oracle, dev, shape):
    """With logical scales the 16-groups run over the flat tensor; a row need not hold whole ones."""
    z = torch.from_numpy(normal(81, shape, 0.02).astype(np.float32))
    x = z + torch.from_numpy(normal(82, shape, 0.003).astype(np.float32))
    t, amax = pkg.OptimizerModule().materialize_schedule_free(z.to(dev), x.to(dev), 0.9, packed=False)
    y = oracle.schedule_free_value(z.numpy(), x.numpy(), 0.9).reshape(1, -1)
    want = oracle.tensor_amax(y)[1]
    ob, os_, og = oracle.four_six(y, want, False)
    assert cpu(amax).tobytes() == want.tobytes() and (t.rows, t.cols) == shape
    assert np.array_equal(cpu(t.bytes), ob) and np.array_equal(cpu(t.scales), os_) and np.array_equal(cpu(t.global_scales), og)
