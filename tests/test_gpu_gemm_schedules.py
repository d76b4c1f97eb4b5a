"""GEMM forms that depend on what a CTA does next: accumulators that share columns with the next tile's, a last tile staged in
the operands' memory, resident panels with their scale factors in tensor memory, contiguous and banded walks, CTA pairs; and the
partial maxima the backward's scale is derived from.  Against the oracle on sampled row blocks, with the sizes where each form
begins and ends; plans are asserted, so that a test keeps to the form it names."""
import numpy as np
import pytest
import torch

from helpers import rel_fro
from test_gpu_gemm_paths import GEMM_TOL, assert_plan, check_rows, cpu, no_timeouts, rand_nvfp4, row_blocks, run_case, tile, to_dev  # noqa: F401

pytestmark = pytest.mark.gpu
bf16, f32 = torch.bfloat16, torch.float32


@pytest.mark.parametrize("m,n,k,epi", [(19072, 1024, 768, 1), (19000, 1000, 768, 2), (19072, 2304, 1024, 1), (19072, 768, 832, 0)])
@pytest.mark.parametrize("dtype", [bf16, f32])
def test_resident_forms(pkg, oracle, dev, m, n, k, epi, dtype):
    """Resident panels of three and four k-tiles (the last one short), many tiles per CTA, ragged rows and columns: 1000
    columns end in the first half of a 256-column tile, so that the half taken first may be empty."""
    run_case(pkg, oracle, dev, m, n, k, out_dtype=dtype, epi=epi, want_plan=dict(b_resident=1, tma_store=1))


@pytest.mark.parametrize("width", [128, 192, 256])
@pytest.mark.parametrize("k", [64, 256, 320, 512])
@pytest.mark.parametrize("dtype", [bf16, f32])
def test_resident_forms_of_one_and_two_k_tiles(pkg, oracle, dev, tile, width, k, dtype):
    """Shorter panels leave room for more A stages, over which a CTA's last tile is staged; the second k-tile whole and of one atom.
    Many tiles per CTA, ragged rows and columns; banded (19000 rows), and contiguous with the panel replaced (1000)."""
    tile(width)
    for m, n, epi in ((19000, 1000, 1), (1000, 20400, 0)):
        run_case(pkg, oracle, dev, m, n, k, out_dtype=dtype, epi=epi, blocks=row_blocks(m)[-2:],
                 want_plan=dict(block_n=width, b_resident=1, resident_cpn=(lambda c: c > 0) if m == 19000 else (lambda c: c <= 1)))


@pytest.mark.parametrize("m,n,k,cpn,dtype", [(840, 32000, 768, 0, f32), (2176, 32000, 768, 1, bf16), (2000, 32000, 768, 1, bf16),
                                             (1920, 32000, 704, 0, bf16)])
def test_vocabulary_walks(pkg, oracle, dev, m, n, k, cpn, dtype):
    """125 column blocks for 148 CTAs: banded from 16 row blocks, contiguous below (840 rows of f32 are an output beyond L2,
    stored evict-first); the contiguous walk replaces its panel."""
    run_case(pkg, oracle, dev, m, n, k, out_dtype=dtype, epi=0, want_plan=dict(block_n=256, b_resident=1, resident_cpn=cpn),
             blocks=row_blocks(m)[::2])


@pytest.mark.parametrize("n,dtype,cpn,tma", [(5696, bf16, 4, 1), (5695, bf16, 0, 0), (5695, f32, 4, 0)])
def test_bf16_direct_stores_walk_on_every_sm(pkg, oracle, dev, tile, n, dtype, cpn, tma):
    """30 column blocks: four CTAs for each leave 28 SMs idle, which TMA stores are worth, and direct ones of f32; those of bf16
    are not."""
    tile(192)
    run_case(pkg, oracle, dev, 8192, n, 448, out_dtype=dtype, epi=1,
             want_plan=dict(block_n=192, b_resident=1, resident_cpn=cpn, tma_store=tma))


@pytest.mark.parametrize("m,n,k,epi,dtype", [(128, 256, 8192, 0, bf16), (300, 520, 8256, 1, bf16), (384, 512, 8128, 2, bf16),
                                             (10000, 768, 8192, 0, bf16), (1000, 512, 8256, 2, f32), (4096, 1024, 8192, 0, f32)])
def test_pairs(pkg, oracle, dev, tile, m, n, k, epi, dtype):
    """CTA pairs from 32 k-tiles: one tile and several a pair, a second CTA without rows, with some, ragged columns and K."""
    tile(256)
    run_case(pkg, oracle, dev, m, n, k, out_dtype=dtype, epi=epi, blocks=row_blocks(m)[-2:],
             want_plan=dict(block_m=128, block_n=256, pair=1, k_splits=1, grid=lambda g: g % 2 == 0))


@pytest.mark.parametrize("m,n,k,splits", [(1024, 1024, 32768, 4), (3072, 1024, 32768, 3), (768, 2048, 24576, 3)])
@pytest.mark.parametrize("epi", [0, 1])
def test_split_k_over_pairs(pkg, oracle, dev, m, n, k, splits, epi):
    """dW of d_model 1024 and a like shape: even splits and uneven ones (43 + 43 + 42 k-tiles), whose partial tiles both CTAs of a
    pair add into the output; a bias joins with the first split."""
    run_case(pkg, oracle, dev, m, n, k, out_dtype=f32, epi=epi, blocks=row_blocks(m)[:2],
             want_plan=dict(block_m=128, block_n=256, pair=1, k_splits=splits, tma_store=1))


@pytest.mark.parametrize("m,n,k,epi,deterministic", [(1000, 1020, 32768, 0, False), (1000, 1020, 32832, 1, False),
                                                     (900, 776, 32832, 1, False), (300, 520, 24832, 1, True), (100, 260, 16640, 0, True)])
def test_split_k_over_pairs_with_tails(pkg, oracle, dev, tile, m, n, k, epi, deterministic):
    """Ragged rows, columns and K; a second CTA with few rows and with none; capped at two splits."""
    tile(256)
    pkg.set_deterministic_reductions(deterministic)
    try:
        run_case(pkg, oracle, dev, m, n, k, out_dtype=f32, epi=epi, blocks=row_blocks(m)[-2:],
                 want_plan=dict(block_n=256, pair=1, k_splits=(lambda s: s == 2) if deterministic else (lambda s: s > 1)))
    finally:
        pkg.set_deterministic_reductions(False)


def test_pairs_begin_at_32_k_tiles(pkg, oracle, dev, tile):
    tile(256)
    run_case(pkg, oracle, dev, 300, 512, 7936, out_dtype=bf16, epi=0, want_plan=dict(block_n=256, pair=0))


@pytest.mark.parametrize("m", [256, 700])
def test_pairs_on_the_residual_stream(pkg, oracle, dev, tile, m):
    tile(256)
    n, k = 512, 8192
    rng = np.random.default_rng(m)
    a, b = rand_nvfp4(rng, m, k, True), rand_nvfp4(rng, n, k, False)
    A, B = to_dev(pkg, dev, a, m, k, True), to_dev(pkg, dev, b, n, k, False)
    bias, res = rng.normal(0, 40.0, n).astype(np.float32), rng.normal(0, 40.0, (m, n)).astype(np.float32)
    out = torch.from_numpy(res).to(dev)
    kw = dict(bias=torch.from_numpy(bias).to(dev), epilogue=pkg.EPI_RESIDUAL, out=out)
    gemm = pkg.Nvfp4GemmModule()
    assert_plan(gemm.plan(A, B, **kw), block_n=256, pair=1, tma_store=1)
    gemm.gemm(A, B, **kw)
    no_timeouts(pkg)
    assert rel_fro(cpu(out), oracle.gemm(a, b, m, k, n, 2, bias=bias, epi=3, residual=res)) <= GEMM_TOL


def test_pair_wait_runs_out(pkg, dev, tile):
    """The first CTA never loads its first stage: both CTAs of the pair end, with a status, and the next GEMM is right."""
    tile(256)
    rng = np.random.default_rng(3)
    a, b = rand_nvfp4(rng, 512, 8192, True), rand_nvfp4(rng, 256, 8192, False)
    A, B = to_dev(pkg, dev, a, 512, 8192, True), to_dev(pkg, dev, b, 256, 8192, False)
    gemm = pkg.Nvfp4GemmModule()
    want = gemm.gemm(A, B, out_dtype=bf16)
    no_timeouts(pkg)
    pkg.set_gemm_wait_timeout_ns(200_000_000)
    pkg.set_gemm_debug_flags(1)
    try:
        gemm.gemm(A, B, out_dtype=bf16)
        torch.cuda.synchronize()
        assert pkg.read_device_status() != 0
    finally:
        pkg.set_gemm_debug_flags(0)
        pkg.set_gemm_wait_timeout_ns(0)
    got = gemm.gemm(A, B, out_dtype=bf16)
    no_timeouts(pkg)
    assert torch.equal(got, want)


@pytest.mark.parametrize("m,n,k,epi,dtype", [(300, 520, 8256, 1, bf16), (300, 520, 8256, 2, bf16), (512, 512, 8192, 2, f32),
                                             (900, 776, 32832, 1, f32)])
def test_refused_output_maps_plan_again(pkg, oracle, dev, tile, m, n, k, epi, dtype):
    """Without its TMA stores a GEMM that would run on pairs, split or not, is planned for direct stores, one CTA a tile."""
    tile(256)
    pkg.set_gemm_debug_flags(2)
    try:
        run_case(pkg, oracle, dev, m, n, k, out_dtype=dtype, epi=epi, blocks=row_blocks(m)[-2:], want_plan=dict(pair=1))
    finally:
        pkg.set_gemm_debug_flags(0)


@pytest.mark.parametrize("chunks", [1, 2, 257, 1184, 1185])
def test_backward_scale_from_partial_maxima(pkg, dev, chunks):
    """A caller's chunk maxima, the largest in the last place, up to what the pair kernel reduces itself (1184) and one more:
    the same bytes as the pass over dY, and the scale is published."""
    t, i, o = 1024, 128, 1280
    gen = torch.Generator(device=dev).manual_seed(chunks)
    e = (torch.randn(t, o, device=dev, generator=gen) * 1e-3).to(bf16)
    q = pkg.Nvfp4QuantModule()
    w = q.quantize_four_six(torch.randn(o, i, device=dev, generator=gen).to(bf16), rowwise=False, packed=True)
    x = q.quantize_four_six(torch.randn(t, i, device=dev, generator=gen).to(bf16), rowwise=True, packed=True, decoded_amax=True)
    results = []
    for given in (0, chunks):
        s = pkg.LinearBackwardScratch(t, i, o, dev)
        if given:
            amax = e.abs().max().float()
            s.e_h["chunk_amax"][:given] = amax * torch.rand(given, device=dev, generator=gen)
            s.e_h["chunk_amax"][given - 1] = amax
        pkg.LinearBackwardModule().backward_ms_eden(e=e, weight=w, input=x, scratch=s, sign_seed=5, scale_seed=6, want_dbias=True,
                                                    precomputed_e_amax_chunks=given)
        results.append([s.e_h[k] for k in ("bytes", "scales_packed", "global_scales", "global_scale")] +
                       [s.e_t_h[k] for k in ("bytes", "scales_packed", "global_scales")])
    for own, theirs in zip(*results):
        assert torch.equal(own, theirs)


@pytest.mark.parametrize("maxima", [[float("nan")], [-2.0], [-0.0], [float("inf")], [3e-3], [float("nan"), 2e-3], [-2.0, float("nan")]])
def test_backward_scale_from_unusual_partial_maxima(pkg, dev, maxima):
    """A NaN among a caller's maxima drops out and a negative one counts as zero, however many there are: the scale that
    nvfp4_quartet_backward_ms_eden_global_scale_from_chunks derives from them."""
    t, i, o = 128, 64, 64
    q = pkg.Nvfp4QuantModule()
    e = (torch.randn(t, o, device=dev) * 1e-3).to(bf16)
    w = q.quantize_four_six(torch.randn(o, i, device=dev).to(bf16), rowwise=False, packed=True)
    x = q.quantize_four_six(torch.randn(t, i, device=dev).to(bf16), rowwise=True, packed=True, decoded_amax=True)
    s = pkg.LinearBackwardScratch(t, i, o, dev)
    given = torch.tensor(maxima, device=dev)
    s.e_h["chunk_amax"][:len(maxima)] = given
    want = q.quartet_backward_ms_eden_global_scale_from_chunks(given, len(maxima))
    pkg.LinearBackwardModule().backward_ms_eden(e=e, weight=w, input=x, scratch=s, sign_seed=5, scale_seed=6, want_dbias=False,
                                                precomputed_e_amax_chunks=len(maxima))
    assert torch.equal(s.e_h["global_scale"].reshape(-1)[:1], want.reshape(-1)[:1])


@pytest.mark.parametrize("m,n,k,dtype,epi,want", [
    (3072, 768, 8192, f32, 0, (128, 128, 1)), (2304, 768, 8192, f32, 0, (128, 192, 2)), (768, 768, 65536, f32, 0, (256, 192, 12)),
    (4096, 4096, 2048, bf16, 1, (128, 256, 1)), (4096, 8192, 2048, f32, 2, (128, 192, 1)), (2048, 2304, 768, bf16, 1, (128, 128, 1)),
    (32000, 768, 8192, f32, 0, (128, 256, 1)), (16, 768, 768, bf16, 1, (128, 128, 1)), (200, 768, 4352, f32, 0, (128, 128, 2)),
    (1024, 2979, 1536, bf16, 1, (128, 128, 1)), (13568, 571, 2432, bf16, 0, (128, 192, 1)), (31360, 3039, 5312, f32, 0, (256, 192, 1)),
    (768, 1685, 12736, f32, 1, (128, 128, 1))])
def test_the_estimate_takes_the_measured_tile(pkg, dev, m, n, k, dtype, epi, want):
    """The fastest tile, or one within a few per cent of it, where a wave more or less, the f32 or the second output, or the time
    of direct stores (odd columns) decides."""
    stub, one = torch.zeros(16, dtype=torch.uint8, device=dev), torch.ones(1, device=dev)
    A = pkg.Nvfp4Tensor(stub, stub, one, m, k, packed=True, rowwise=True)
    B = pkg.Nvfp4Tensor(stub, stub, one, n, k, packed=True, rowwise=False)
    out = torch.empty(16, dtype=dtype, device=dev)
    plan = pkg.Nvfp4GemmModule().plan(A, B, out=out, epilogue=epi, bias=one if epi else None, aux=out if epi == 2 else None)
    assert (plan.block_m, plan.block_n, plan.k_splits) == want
