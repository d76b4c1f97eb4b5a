"""The `_cleared` entries beside their plain forms: the call leaves what the word or the row amaxes hold in place and takes the
maximum with it, for every row length and route; everything else it writes is the plain form's, bit for bit."""
import pytest
import torch

from helpers import bf16_normal

pytestmark = pytest.mark.gpu
bf16, f32 = torch.bfloat16, torch.float32


def quantize(pkg, entry, x, given, held, packed):
    """One call of `entry`: its outputs, and the decoded amax, whose word holds `held` before."""
    rows, cols = x.shape
    by = torch.zeros(rows * cols // 2, dtype=torch.uint8, device=x.device)
    sc = torch.zeros(pkg.scale_packed_len(rows, cols) if packed else rows * cols // 16, dtype=torch.uint8, device=x.device)
    gs, amax = torch.zeros(rows, device=x.device), torch.zeros(rows, device=x.device)
    relu2 = (pkg._ptr(given),) if "relu2" in entry else ()
    pkg._call(entry, pkg._stream(), pkg._ptr(x), pkg._dtype_code(x), rows, cols, *relu2, pkg._ptr(by), pkg._ptr(sc),
              pkg.SCALES_PACKED if packed else pkg.SCALES_LOGICAL, pkg._ptr(gs), pkg._ptr(amax), pkg._ptr(held))
    return [by, sc, gs, amax]


# 4096 values are the longest row of the one-pass quantizers; relu2 takes longer ones with their row amax given
@pytest.mark.parametrize("entry,cols,given", [
    ("nvfp4_quantize_four_six_rowwise_fused", 64, False), ("nvfp4_quantize_four_six_rowwise_fused", 4096, False),
    ("nvfp4_quantize_four_six_rowwise_fused", 4112, False), ("nvfp4_quantize_four_six_rowwise_fused", 8192, False),
    ("nvfp4_quantize_relu2_four_six_rowwise", 64, False), ("nvfp4_quantize_relu2_four_six_rowwise", 4096, False),
    ("nvfp4_quantize_relu2_four_six_rowwise", 64, True), ("nvfp4_quantize_relu2_four_six_rowwise", 8192, True)])
@pytest.mark.parametrize("dtype", [bf16, f32])
def test_cleared_quantizers_keep_a_larger_amax(pkg, dev, entry, cols, given, dtype):
    x = bf16_normal(cols, (131, cols)).to(dev).to(dtype)
    packed = cols % 64 == 0
    row_amax = (x.float().clamp(min=0) ** 2).amax(dim=1).contiguous() if given else None
    word = torch.full((1,), 12345.0, device=dev)
    want = quantize(pkg, entry, x, row_amax, word, packed)
    own = word.clone()  # the plain form clears the word
    assert 0 < own.item() < 12345.0
    for factor in (0.0, 0.5, 2.0):
        held = own * factor
        word.copy_(held)
        got = quantize(pkg, entry + "_cleared", x, row_amax, word, packed)
        assert torch.equal(word, torch.maximum(held, own)), factor
        for g, w in zip(got, want):
            assert torch.equal(g, w)


@pytest.mark.parametrize("cols", [768, 4160])
def test_cleared_quantizers_gather_one_amax_over_calls(pkg, dev, cols):
    """The largest tensor first: a call that cleared the word would leave the last one's."""
    parts = [bf16_normal(i, (64, cols), std).to(dev) for i, std in enumerate((3.0, 1.0, 0.1))]
    word, single = torch.zeros(1, device=dev), []
    for x in parts:
        quantize(pkg, "nvfp4_quantize_four_six_rowwise_fused_cleared", x, None, word, True)
        own = torch.zeros(1, device=dev)
        quantize(pkg, "nvfp4_quantize_four_six_rowwise_fused", x, None, own, True)
        single.append(own.item())
    assert word.item() == max(single) == single[0]


def test_cleared_gemm_keeps_larger_row_amaxes(pkg, dev):
    m, n, k = 131, 264, 192
    q, gemm = pkg.Nvfp4QuantModule(), pkg.Nvfp4GemmModule()
    a = q.quantize_four_six(bf16_normal(1, (m, k)).to(dev), rowwise=True, packed=True)
    b = q.quantize_four_six(bf16_normal(2, (n, k)).to(dev), rowwise=False, packed=True)
    out, own = torch.empty(m, n, dtype=bf16, device=dev), torch.full((m,), 12345.0, device=dev)
    gemm.gemm(a, b, out=out, relu2_row_amax=own)  # clears the amaxes
    assert own.max().item() < 12345.0
    factor = torch.tensor([0.0, 0.5, 2.0], device=dev).repeat(m)[:m]
    held = own * factor
    got, again = held.clone(), torch.empty_like(out)
    args, keep = gemm._args(a, b, again, None, None, pkg.GS_ROWWISE_A, pkg.EPI_NONE, 1.0, n, n, got)
    pkg._call("nvfp4_gemm_cleared", pkg._stream(), args)
    assert torch.equal(got, torch.maximum(held, own)) and torch.equal(again, out)
