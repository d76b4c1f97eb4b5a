"""Which GEMMs of three to four tiles a CTA keep their B panel (those whose banded schedule keeps every CTA busy), which tile two
outputs take, and that they compute what another tile computes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# (rows, columns, K): tile width, resident, CTAs per column block on 148 SMs, of a bf16 output
@pytest.mark.parametrize("m,n,k,width,resident,cpn", [
    (8192, 2304, 768, 256, 1, 16),    # 64 row blocks on 16 CTAs
    (8100, 2304, 704, 256, 1, 16),    # ragged rows, K of three k-tiles less an atom
    (4096, 2304, 768, 128, 1, 8),
    (7424, 2304, 768, 192, 1, 12),    # 58 row blocks, 3.6 turns of 16: four tiles of 192 columns a CTA, not three of 256
    (16384, 768, 768, 128, 1, 24),    # no panel of 256 columns here: it would take three CTAs of 128 row blocks, 49 a column block
])
def test_three_tiles_a_cta(pkg, dev, m, n, k, width, resident, cpn):
    if torch.cuda.get_device_properties(dev).multi_processor_count != 148:
        pytest.skip("the expectations are for a 148-SM part")
    q, gemm = pkg.Nvfp4QuantModule(), pkg.Nvfp4GemmModule()
    g = torch.Generator(device=dev)
    g.manual_seed(m + n)
    x = q.quantize_four_six(torch.randn(m, k, generator=g, device=dev).to(torch.bfloat16), rowwise=True, packed=True)
    w = q.quantize_four_six((torch.randn(n, k, generator=g, device=dev) * 0.02).to(torch.bfloat16), rowwise=False, packed=True)
    bias = torch.randn(n, generator=g, device=dev)
    plan = gemm.plan(x, w, bias=bias, epilogue=pkg.EPI_BIAS, out=torch.empty(m, n, device=dev, dtype=torch.bfloat16))
    assert (plan.block_m, plan.block_n, plan.b_resident, plan.resident_cpn) == (128, width, resident, cpn)
    for dtype in (torch.bfloat16, torch.float32):
        kw = dict(bias=bias, epilogue=pkg.EPI_BIAS, out=torch.empty(m, n, device=dev, dtype=dtype))
        planned = gemm.plan(x, w, **kw).block_n
        y = gemm.gemm(x, w, **kw)
        pkg.set_gemm_tile_override(128 if planned != 128 else 192)
        try:
            want = gemm.gemm(x, w, bias=bias, epilogue=pkg.EPI_BIAS, out_dtype=torch.float32)
        finally:
            pkg.set_gemm_tile_override(0)
        # sums over K of 704 to 768 in f32, each of order sqrt(K) 0.02 beside a bias of order 1: a bf16 rounding, or some f32 ones
        limit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -18
        assert float((y.float() - want).norm() / want.norm()) < limit
    assert pkg.read_device_status() == 0


@pytest.mark.parametrize("m,n,k,dtype,width", [
    (1000, 4096, 1024, torch.float32, 128), (1000, 4096, 1024, torch.bfloat16, 128), (2048, 4096, 1024, torch.float32, 128),
    (4096, 3072, 768, torch.bfloat16, 128),
    (4096, 8192, 2048, torch.float32, 192),   # a main loop that hides the turns of 192 columns
    (4096, 12288, 3072, torch.float32, 192), (1024, 12288, 8192, torch.bfloat16, 256),   # not the tall tile
    (8192, 3072, 768, torch.bfloat16, 256),   # resident, two staging buffers a group
])
def test_two_outputs(pkg, dev, m, n, k, dtype, width):
    if torch.cuda.get_device_properties(dev).multi_processor_count != 148:
        pytest.skip("the expectations are for a 148-SM part")
    q, gemm = pkg.Nvfp4QuantModule(), pkg.Nvfp4GemmModule()
    g = torch.Generator(device=dev)
    g.manual_seed(m + n)
    x = q.quantize_four_six(torch.randn(m, k, generator=g, device=dev).to(torch.bfloat16), rowwise=True, packed=True)
    w = q.quantize_four_six((torch.randn(n, k, generator=g, device=dev) * 0.02).to(torch.bfloat16), rowwise=False, packed=True)
    bias = torch.randn(n, generator=g, device=dev) * 0.02
    out, pre = torch.empty(m, n, device=dev, dtype=dtype), torch.empty(m, n, device=dev, dtype=dtype)
    kw = dict(bias=bias, epilogue=pkg.EPI_RELU2)
    plan = gemm.plan(x, w, out=out, aux=pre, **kw)
    assert (plan.block_m, plan.block_n) == (128, width)
    gemm.gemm(x, w, out=out, aux=pre, **kw)
    pkg.set_gemm_tile_override(192, 256)
    try:
        want_pre = torch.empty(m, n, device=dev)
        want = gemm.gemm(x, w, out=torch.empty(m, n, device=dev), aux=want_pre, **kw)
    finally:
        pkg.set_gemm_tile_override(0)
    # f32 sums over K up to 8192 in another order, or one bf16 rounding (doubled by the square)
    limit = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -17
    assert float((pre.float() - want_pre).norm() / want_pre.norm()) < limit
    assert float((out.float() - want).norm() / want.norm()) < limit
    assert pkg.read_device_status() == 0
