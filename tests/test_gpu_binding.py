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


def test_backward_outputs_decide_their_dtype(pkg, dev):
    """`grad_dtype` is the type of the gradients the call allocates; with both given it is not looked at."""
    t, i, o = 64, 64, 128
    q, bwd, sc = pkg.Nvfp4QuantModule(), pkg.LinearBackwardModule(), pkg.LinearBackwardScratch(64, 64, 128, dev)
    xq = q.quantize_four_six(torch.randn(t, i, device=dev), rowwise=True, packed=True)
    wq = q.quantize_four_six(torch.randn(o, i, device=dev), rowwise=False, packed=True)
    args = dict(e=torch.randn(t, o, device=dev), weight=wq, input=xq, scratch=sc, sign_seed=1, scale_seed=2)
    want = bwd.backward_ms_eden(**args)
    dx, dw = torch.empty(t, i, device=dev), torch.empty(o, i, device=dev)
    got = bwd.backward_ms_eden(**args, grad_dtype=torch.float16, dinput=dx, dweight=dw)
    assert got[0] is dx and got[1] is dw and torch.equal(dx, want[0]) and torch.equal(dw, want[1])
    for given in (dict(), dict(dinput=dx), dict(dweight=dw)):
        with pytest.raises(TypeError):
            bwd.backward_ms_eden(**args, grad_dtype=torch.float16, **given)
