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


def valid_calls(pkg, dev, side):
    """A valid argument list for every entry of the binding."""
    t, i, o = 64, 64, 128
    q = pkg.Nvfp4QuantModule()
    f32 = lambda *shape: torch.randn(shape, device=dev)  # noqa: E731
    x, e, bias = f32(t, i), f32(t, o), f32(o)
    xp, xl = q.quantize_four_six(x, rowwise=True, packed=True, decoded_amax=True), q.quantize_four_six(x, rowwise=True, packed=False)
    w = f32(o, i)
    wp, wl = q.quantize_four_six(w, packed=True), q.quantize_four_six(w, packed=False)
    bq = q.quantize_four_six(f32(1, o), packed=False)
    triple = lambda v: (v.bytes, v.scales, v.global_scales)  # noqa: E731
    sc = pkg.LinearBackwardScratch(t, i, o, dev)
    row_amax = q.row_amax(x)
    return {
        "quantize_new": [x, row_amax, True, True, False],
        "quantize_into": [x, row_amax, True, True, None, *triple(xp)],
        "four_six_rowwise_f32": [x, row_amax],
        "row_amax": [x, torch.empty(t, device=dev)],
        "decode": [*triple(xl), t, i, True, False],
        "materialize": [w, f32(o, i), 0.5, False],
        "gemm": [*triple(xp), *triple(wp), f32(t, o), f32(t, o), bias, None, None, None, t, o, i, o, pkg.GS_ROWWISE_A, 1.0,
                 pkg.EPI_RELU2, torch.empty(t, device=dev)],
        "projection_forward": [x, True, True, *triple(wp), o, i, bias, pkg.EPI_BIAS, pkg.DTYPE_F32, None],
        "projection": [2, xl.bytes, xl.scales, False, xl.global_scales, wl.bytes, wl.scales, False, wl.global_scales, *triple(bq),
                       f32(t, o), f32(t, o), torch.empty(t, device=dev), t, i, o],
        "linear_backward": [False, e, wp.bytes, wp.scales, True, wp.global_scales, xp.bytes, xp.scales, True, xp.global_scales,
                            sc.e_h, sc.e_t_h, sc.weight_t_h, sc.input_t_h, f32(t, i), f32(o, i), f32(o), True, pkg.DTYPE_F32, t, i,
                            o, 1, 2, 0, 0, torch.ones(1, device=dev), xp.decoded_amax, *side.numbers(), 0, False],
    }


ENTRIES = ["quantize_new", "quantize_into", "four_six_rowwise_f32", "row_amax", "decode", "materialize", "gemm",
           "projection_forward", "projection", "linear_backward"]


@pytest.mark.parametrize("name", ENTRIES)
def test_wrong_arguments_raise(pkg, dev, name):
    """Every tensor argument of every entry, replaced by one on the CPU, one that is not contiguous and no tensor at all;
    every number replaced by a text; too few arguments; unknown element types.  Each is a Python exception raised before
    anything is launched, and a whole call still goes through afterwards."""
    side = pkg.SideStream(dev)
    calls = valid_calls(pkg, dev, side)
    assert set(calls) == set(ENTRIES) == {n for n in dir(pkg._native()) if not n.startswith("_") and n != "set_error_type"}
    fn, args = getattr(pkg._native(), name), calls[name]
    fn(*args)
    torch.cuda.synchronize()
    launched = pkg.launch_count()

    def refuses(error, position, value):
        with pytest.raises(error):
            fn(*args[:position], value, *args[position + 1:])

    for p, a in enumerate(args):
        if isinstance(a, torch.Tensor):
            refuses(AssertionError, p, a.cpu())
            refuses(AssertionError, p, torch.empty((4, 2), dtype=a.dtype, device=dev)[:, 0])
            refuses(TypeError, p, 7)
        elif isinstance(a, dict):
            for key, value in a.items():
                refuses(AssertionError, p, {**a, key: value.cpu()})
                refuses(KeyError, p, {k: v for k, v in a.items() if k != key})
        elif isinstance(a, (int, float)) and not isinstance(a, bool):
            refuses(TypeError, p, "text")
        elif isinstance(a, bool):
            refuses(ValueError, p, np.zeros(2))
    with pytest.raises(TypeError):
        fn(*args[:-1])
    if name == "projection_forward":  # with an output given its own type counts: the type code stands unread
        refuses(AssertionError, 11, torch.empty(64, 128))
    typed = {"quantize_new": 0, "quantize_into": 0, "row_amax": 0, "projection_forward": 0, "gemm": 6, "linear_backward": 1}
    if name in typed:
        refuses(TypeError, typed[name], args[typed[name]].half())
    assert pkg.launch_count() == launched
    fn(*args)
    torch.cuda.synchronize()
    assert pkg.read_device_status() == 0
