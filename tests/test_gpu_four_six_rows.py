"""The rowwise four-six kernel whose warps take whole rows (or parts of rows with given maxima): every form of it, odd and pad rows,
both sides of the row counts that it starts at, against the oracle bit for bit."""
import numpy as np
import pytest
import torch

from helpers import bf16_normal

pytestmark = pytest.mark.gpu


def cpu(t):
    return t.detach().cpu().numpy()


def check(oracle, t, x, amax):
    rows, cols = x.shape
    ob, os_, og = oracle.four_six(x, amax, True)
    assert np.array_equal(cpu(t.bytes), ob) and np.array_equal(cpu(t.global_scales), og)
    assert np.array_equal(cpu(t.scales), oracle.scale_pack(os_, rows, cols) if t.packed else os_)
    if t.decoded_amax is not None:
        assert cpu(t.decoded_amax)[0] == oracle.nvfp4_amax(ob, os_, og, rows, cols, True)[1]


def values(rows, cols, dtype, seed):
    x = bf16_normal(seed, (rows, cols)).float().numpy()
    x *= np.exp2(np.arange(rows) % 23 - 11).astype(np.float32)[:, None]
    x[1], x[-1, 16:48] = 0, -0.0
    x[2, ::7] *= 40
    if dtype == torch.float32:
        return x * np.float32(1.0 / 3)
    return torch.from_numpy(x).to(torch.bfloat16).float().numpy()


# widths of the six forms; rows: below and at the first count that is taken (592 warps; what four_six_rowwise_kernel does no longer
# in one turn of its CTAs, 2220 rows of 768 and 888 of 2048), odd, one more than whole 128-row blocks, warps of several units
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("cols,rows", [(256, 1183), (256, 1185), (512, 592), (768, 1024), (768, 1185), (768, 4737), (1024, 593),
                                       (1536, 641), (2048, 2369), (768, 2220), (768, 2221), (2048, 888), (2048, 889), (2048, 1777),
                                       (256, 14209)])
@pytest.mark.parametrize("packed", [False, True])
def test_own_rows(pkg, oracle, dev, dtype, cols, rows, packed):
    x = values(rows, cols, dtype, cols + rows)
    t = pkg.Nvfp4QuantModule().quantize_four_six(torch.from_numpy(x).to(dev).to(dtype), rowwise=True, packed=packed, decoded_amax=True)
    check(oracle, t, x, oracle.row_amax(x))


# two, three and four groups a lane, one unit a row and several; one turn of the warps, two, more; nearly full, and not enough
@pytest.mark.parametrize("cols,rows", [(2048, 1793), (3072, 887), (3072, 1281), (4096, 900), (4224, 1700), (6144, 889), (1024, 2300),
                                       (1024, 9601), (1536, 2001), (3072, 1100), (4096, 2300), (4096, 3585), (5120, 1300), (7680, 1500)])
@pytest.mark.parametrize("relu2,packed", [(True, True), (True, False), (False, True)])
def test_given_rows(pkg, oracle, dev, cols, rows, relu2, packed):
    q = pkg.Nvfp4QuantModule()
    x = values(rows, cols, torch.bfloat16, cols + rows)
    xd = torch.from_numpy(x).to(dev).to(torch.bfloat16)
    if relu2:
        x = np.square(np.maximum(x, 0)).astype(np.float32)
    amax = oracle.row_amax(x)
    amax[5] *= 0.5  # a caller's maximum need not be the row's
    given = torch.from_numpy(amax).to(dev)
    if relu2:
        t = q.quantize_relu2_four_six_rowwise(xd, given, packed=packed, decoded_amax=True)
    else:
        t = q.quantize_four_six(xd, given, rowwise=True, packed=packed)
    check(oracle, t, x, amax)


def test_own_rows_relu2_and_unusual_values(pkg, oracle, dev):
    """NaN (dropped by both maxima), infinities, the largest and the smallest values, with and without the square on load."""
    q = pkg.Nvfp4QuantModule()
    x = values(1500, 1024, torch.bfloat16, 5)
    x[3, 5], x[4], x[6, 100], x[7, 3] = np.nan, np.nan, np.inf, -np.inf
    x[8] *= np.float32(2.0 ** 100)
    x[9] *= np.float32(2.0 ** -120)
    x = torch.from_numpy(x).to(torch.bfloat16)
    for relu2 in (False, True):
        t = q.quantize_relu2_four_six_rowwise(x.to(dev), packed=False) if relu2 else q.quantize_four_six(x.to(dev), rowwise=True, packed=False)
        with np.errstate(over="ignore", invalid="ignore"):
            y = np.square(np.fmax(x.float().numpy(), 0)) if relu2 else x.float().numpy()
        ob, os_, og = oracle.four_six(y, oracle.row_amax(y), True)
        assert np.array_equal(cpu(t.bytes), ob) and np.array_equal(cpu(t.scales), os_)
        assert np.array_equal(cpu(t.global_scales), og, equal_nan=True)
