"""Tiled quantizer kernels of the linear backward at the sizes where tiling can go wrong: one row, a row either side of
a 128-row tile, column counts inside and beyond a 64-column tile and a 128-row scale block, and the values that leave
the straight-line path.  Bit-exact against the oracle, and against the generic one-thread-per-chunk kernel on a tensor
large enough for a single wrong rounding in a few million block scales to show."""
import numpy as np
import pytest
import torch

from helpers import bf16_normal

pytestmark = pytest.mark.gpu
SIGN, SCALE = 0x12345678, 0x9ABCDEF0


def cpu(t):
    return t.detach().cpu().numpy()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens,in_dim,out_dim", [(1, 64, 64), (127, 64, 72), (128, 192, 136), (129, 128, 200),
                                                   (257, 320, 64), (130, 64, 1000)])
def test_backward_operands_ragged_tiles(pkg, oracle, dev, tokens, in_dim, out_dim, dtype):
    q, bwd = pkg.Nvfp4QuantModule(), pkg.LinearBackwardModule()
    x, w = bf16_normal(701, (tokens, in_dim)), bf16_normal(702, (out_dim, in_dim), 0.02)
    dy = bf16_normal(703, (tokens, out_dim), 1e-3)
    dy[tokens // 2] = 0.0                     # zero groups, negative zeros, sub-normal block scales, one outlier
    dy[:, out_dim // 3] = -0.0
    dy[: max(1, tokens // 4)] *= 2.0 ** -20
    dy[-1, -1] = 3.0e4
    x[tokens // 3] = 0.0
    w[:, in_dim // 2] = 0.0
    w[out_dim // 2] *= 2.0 ** -14
    xq = q.quantize_four_six(x.to(dev), rowwise=True, packed=True, decoded_amax=True)
    wq = q.quantize_four_six(w.to(dev), rowwise=False, packed=True)
    sc = pkg.LinearBackwardScratch(tokens, in_dim, out_dim, dev)
    e = dy.to(dev) if dtype == torch.bfloat16 else dy.float().to(dev)
    _, _, db = bwd.backward_ms_eden(e=e, weight=wq, input=xq, scratch=sc, sign_seed=SIGN, scale_seed=SCALE)
    torch.cuda.synchronize()
    assert pkg.read_device_status() == 0
    xf, wf, ef = x.float().numpy(), w.float().numpy(), dy.float().numpy()
    oxq, owq = oracle.four_six(xf, oracle.row_amax(xf), True), oracle.four_six(wf, oracle.tensor_amax(wf)[1], False)
    ok, tk = oracle.padded_k(out_dim), oracle.padded_k(tokens)
    gs_e = oracle.ms_eden_global_scale(float(np.abs(ef).max()))
    gs_w = oracle.ms_eden_global_scale(float(oracle.nvfp4_amax(*owq, out_dim, in_dim, False)[1][0]))
    gs_x = oracle.ms_eden_global_scale(float(oracle.nvfp4_amax(*oxq, tokens, in_dim, True)[1][0]))
    want = {
        "e_h": (oracle.ms_eden(0, ef, tokens, ok, gs_e, SIGN, SCALE, want_chunk_amax=False), tokens, ok),
        "e_t_h": (oracle.ms_eden(1, ef, out_dim, tk, gs_e, SIGN, SCALE ^ 0x85EBCA6B, want_chunk_amax=False), out_dim, tk),
        "weight_t_h": (oracle.ms_eden(2, (*owq, out_dim, in_dim), in_dim, ok, gs_w, SIGN, SCALE ^ 0x9E3779B9,
                                      want_chunk_amax=False), in_dim, ok),
        "input_t_h": (oracle.ms_eden(3, (*oxq, tokens, in_dim), in_dim, tk, gs_x, SIGN, SCALE ^ 0xC2B2AE35,
                                     want_chunk_amax=False), in_dim, tk),
    }
    for name, (ref, rows, k) in want.items():
        op = getattr(sc, name)
        assert np.array_equal(cpu(op["bytes"]), ref[0]), name
        assert np.array_equal(cpu(op["scales_packed"]), oracle.scale_pack(ref[1], rows, k)), name
        assert np.array_equal(cpu(op["global_scales"]), ref[2]), name
    assert np.array_equal(cpu(db), oracle.bias_grad_tiled(ef))


def test_pair_rows_equal_generic_kernel_large(pkg, dev):
    """16.4 million block scales of dY rows: the pair kernel against the generic kernel, every byte."""
    q, bwd = pkg.Nvfp4QuantModule(), pkg.LinearBackwardModule()
    tokens, in_dim, out_dim = 8192, 64, 32000
    g = torch.Generator(device=dev).manual_seed(11)
    e = (torch.randn((tokens, out_dim), generator=g, device=dev) * 1e-3).to(torch.bfloat16)
    x = torch.randn((tokens, in_dim), generator=g, device=dev).to(torch.bfloat16)
    w = (torch.randn((out_dim, in_dim), generator=g, device=dev) * 0.02).to(torch.bfloat16)
    xq = q.quantize_four_six(x, rowwise=True, packed=True, decoded_amax=True)
    wq = q.quantize_four_six(w, rowwise=False, packed=True)
    sc = pkg.LinearBackwardScratch(tokens, in_dim, out_dim, dev)
    bwd.backward_ms_eden(e=e, weight=wq, input=xq, scratch=sc, sign_seed=SIGN, scale_seed=SCALE)
    ref, _ = q.ms_eden_quantize(src_kind=pkg.SRC_F32_ROWS, x=e, rows=tokens, cols=out_dim, dst_row_len=out_dim,
                                global_scale=sc.e_h["global_scale"], sign_seed=SIGN, scale_seed=SCALE, packed=True)
    assert torch.equal(sc.e_h["bytes"], ref.bytes)
    assert torch.equal(sc.e_h["scales_packed"], ref.scales)


# factors on the global scale the tensor's amax gives, and scale overrides: signs, block scales that all saturate or all
# round to zero, quotients that overflow
SCALES = [(-1.0, None), (1.0, -0.988125), (-1.0, -0.988125), (1e-30, None), (1e30, None), (1.0, 1e-20), (1.0, 0.03), (1.0, 30.0),
          (1.0, 1e20)]


@pytest.mark.parametrize("factor,override", SCALES)
@pytest.mark.parametrize("rows,cols", [(128, 64), (130, 96)])
@pytest.mark.parametrize("rowwise", [False, True])
def test_nvfp4_transpose_any_scale(pkg, oracle, dev, rows, cols, rowwise, factor, override):
    """A caller's global scale and scale override may have any sign and size: bytes of the oracle."""
    q = pkg.Nvfp4QuantModule()
    x = bf16_normal(711, (rows, cols)).float().numpy()
    x[3], x[:, 5] = 0.0, -0.0
    src = oracle.four_six(x, oracle.row_amax(x) if rowwise else oracle.tensor_amax(x)[1], rowwise)
    gs = float(np.float32(factor * oracle.ms_eden_global_scale(float(oracle.nvfp4_amax(*src, rows, cols, rowwise)[1][0]))))
    so = pkg.QUARTET_MS_EDEN_SCALE_OVERRIDE if override is None else override
    k = oracle.padded_k(rows)
    want = oracle.ms_eden(3 if rowwise else 2, (*src, rows, cols), cols, k, gs, SIGN, SCALE, so=so, want_chunk_amax=False)
    t = pkg.Nvfp4Tensor(*(torch.from_numpy(a).to(dev) for a in src), rows, cols, packed=False, rowwise=rowwise)
    got, _ = q.ms_eden_quantize(src_kind=pkg.SRC_ROWWISE_NVFP4_TRANSPOSED if rowwise else pkg.SRC_NVFP4_TRANSPOSED, src=t,
                                rows=rows, cols=cols, dst_row_len=k, global_scale=gs, sign_seed=SIGN, scale_seed=SCALE,
                                scale_override=so)
    assert np.array_equal(cpu(got.bytes), want[0])
    assert np.array_equal(cpu(got.scales), want[1])
    assert np.array_equal(cpu(got.global_scales), want[2])


@pytest.mark.parametrize("factor", [-1.0, 1e-30, 1e30])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens,out_dim", [(128, 128), (129, 72)])
def test_pair_any_scale(pkg, oracle, dev, tokens, out_dim, dtype, factor):
    """The same for dY in both orientations, whose scale a caller may give."""
    q, bwd, in_dim = pkg.Nvfp4QuantModule(), pkg.LinearBackwardModule(), 64
    dy = bf16_normal(712, (tokens, out_dim), 1e-3)
    dy[7], dy[:, 9] = 0.0, -0.0
    ef = dy.float().numpy()
    gs = np.float32(factor * oracle.ms_eden_global_scale(float(np.abs(ef).max())))
    xq = q.quantize_four_six(bf16_normal(713, (tokens, in_dim)).to(dev), rowwise=True, packed=True, decoded_amax=True)
    wq = q.quantize_four_six(bf16_normal(714, (out_dim, in_dim), 0.02).to(dev), rowwise=False, packed=True)
    sc = pkg.LinearBackwardScratch(tokens, in_dim, out_dim, dev)
    bwd.backward_ms_eden(e=dy.to(dev).to(dtype), weight=wq, input=xq, scratch=sc, sign_seed=SIGN, scale_seed=SCALE,
                         e_global_scale=torch.tensor([gs], device=dev))
    ok, tk = oracle.padded_k(out_dim), oracle.padded_k(tokens)
    for name, kind, rows, k, seed in (("e_h", 0, tokens, ok, SCALE), ("e_t_h", 1, out_dim, tk, SCALE ^ 0x85EBCA6B)):
        ref = oracle.ms_eden(kind, ef, rows, k, float(gs), SIGN, seed, want_chunk_amax=False)
        op = getattr(sc, name)
        assert np.array_equal(cpu(op["bytes"]), ref[0]), name
        assert np.array_equal(cpu(op["scales_packed"]), oracle.scale_pack(ref[1], rows, k)), name
        assert np.array_equal(cpu(op["global_scales"]), ref[2]), name
    torch.cuda.synchronize()
    assert pkg.read_device_status() == 0


def cross_entropy_gradient(dev, tokens, classes, spread):
    """(softmax - one-hot) / tokens: most block scales of it lie below the smallest normal E4M3 value."""
    g = torch.Generator(device=dev).manual_seed(19)
    p = torch.softmax(torch.randn((tokens, classes), generator=g, device=dev) * spread, 1)
    target = torch.randint(0, classes, (tokens, 1), generator=g, device=dev)
    return p.scatter_add_(1, target, torch.full((tokens, 1), -1.0, device=dev)) / tokens


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens,out_dim", [(1024, 8192), (1000, 8200)])
@pytest.mark.parametrize("kind", ["gradient", "zeros", "not finite"])
def test_pair_general_scales_many_tiles(pkg, dev, tokens, out_dim, dtype, kind):
    """Several tiles a CTA, the general scale code and the generic redo between a tile's loads and its column sums: the bytes of
    the generic kernel in both orientations, and the column sums of the tiles."""
    q, bwd, in_dim = pkg.Nvfp4QuantModule(), pkg.LinearBackwardModule(), 64
    e = cross_entropy_gradient(dev, tokens, out_dim, 1.0 if kind == "gradient" else 0.0)
    if kind == "zeros":
        e = e * torch.exp2(-torch.randint(0, 30, (tokens // 8, 1), device=dev).float()).repeat_interleave(8, 0)
        e[::5], e[:, ::17], e[64:128], e[:, 128:200] = 0, -0.0, 0, 0
    if kind == "not finite":
        e[3, 40], e[700, 8000], e[990:, 5] = float("nan"), float("-nan"), float("nan")
    e = e.to(dtype)
    xq = q.quantize_four_six(bf16_normal(741, (tokens, in_dim)).to(dev), rowwise=True, packed=True, decoded_amax=True)
    wq = q.quantize_four_six(bf16_normal(742, (out_dim, in_dim), 0.02).to(dev), rowwise=False, packed=True)
    sc = pkg.LinearBackwardScratch(tokens, in_dim, out_dim, dev)
    _, _, db = bwd.backward_ms_eden(e=e, weight=wq, input=xq, scratch=sc, sign_seed=SIGN, scale_seed=SCALE)
    for name, kind_, k, seed in (("e_h", pkg.SRC_F32_ROWS, -(-out_dim // 64) * 64, SCALE),
                                 ("e_t_h", pkg.SRC_F32_TRANSPOSED, -(-tokens // 64) * 64, SCALE ^ 0x85EBCA6B)):
        ref, _ = q.ms_eden_quantize(src_kind=kind_, x=e, rows=tokens, cols=out_dim, dst_row_len=k,
                                    global_scale=sc.e_h["global_scale"], sign_seed=SIGN, scale_seed=seed, packed=True)
        op = getattr(sc, name)
        assert torch.equal(op["bytes"], ref.bytes), name
        assert torch.equal(op["scales_packed"], ref.scales), name
    # every partial sum is bounded by the sum of the magnitudes: one rounding of 2^-24 per addition
    ef = e.double()
    assert bool(((db.double() - ef.sum(0)).abs() <= tokens * 2.0 ** -24 * ef.abs().sum(0))[~ef.sum(0).isnan()].all())
    assert torch.equal(db.isnan(), ef.sum(0).isnan())
    torch.cuda.synchronize()
    assert pkg.read_device_status() == 0


def test_general_scales_cost_no_second_pass(pkg, dev):
    """The gradient of a cross-entropy, two thirds of whose chunks hold a block scale below the normal E4M3 range, against
    normal values: only the scale bytes are computed again (at in_dim 768 1.11 times the time; 3.0 times when every thread
    quantized such chunks again, 2.0 when the CTA shared them)."""
    q, bwd = pkg.Nvfp4QuantModule(), pkg.LinearBackwardModule()
    tokens, in_dim, out_dim = 8192, 64, 32000
    x, w = bf16_normal(751, (tokens, in_dim)).to(dev), bf16_normal(752, (out_dim, in_dim), 0.02).to(dev)
    xq = q.quantize_four_six(x, rowwise=True, packed=True, decoded_amax=True)
    wq = q.quantize_four_six(w, rowwise=False, packed=True)
    sc = pkg.LinearBackwardScratch(tokens, in_dim, out_dim, dev)

    def fastest(e):
        times = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            bwd.backward_ms_eden(e=e, weight=wq, input=xq, scratch=sc, sign_seed=SIGN, scale_seed=SCALE, want_dbias=False)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    gradient = cross_entropy_gradient(dev, tokens, out_dim, 0.02).to(torch.bfloat16)
    normal = (torch.randn((tokens, out_dim), device=dev) * 1e-3).to(torch.bfloat16)
    assert fastest(gradient) < 1.6 * fastest(normal)


@pytest.mark.parametrize("tokens,in_dim,out_dim,offset", [(4352, 64, 64, 0), (8192, 768, 200, 0), (4500, 128, 72, 0), (4352, 64, 64, 1),
                                                          (256, 64, 64, 0)])
def test_backward_clears_dweight_before_it_adds(pkg, dev, tokens, in_dim, out_dim, offset):
    """A dW GEMM that splits K adds into dW, which the pair kernel clears on the way (a launch of its own does where dW is
    not 16-byte aligned): whatever dW held before is gone, and nothing beside it is touched."""
    q, gemm, bwd = pkg.Nvfp4QuantModule(), pkg.Nvfp4GemmModule(), pkg.LinearBackwardModule()
    e = bf16_normal(731, (tokens, out_dim), 1e-3).to(dev)
    xq = q.quantize_four_six(bf16_normal(732, (tokens, in_dim)).to(dev), rowwise=True, packed=True, decoded_amax=True)
    wq = q.quantize_four_six(bf16_normal(733, (out_dim, in_dim), 0.02).to(dev), rowwise=False, packed=True)
    sc = pkg.LinearBackwardScratch(tokens, in_dim, out_dim, dev)
    memory = torch.full((out_dim * in_dim + 8,), float("nan"), device=dev)
    dw = memory[offset: offset + out_dim * in_dim].view(out_dim, in_dim)
    bwd.backward_ms_eden(e=e, weight=wq, input=xq, scratch=sc, sign_seed=SIGN, scale_seed=SCALE, dweight=dw)
    k = -(-tokens // 64) * 64
    a = pkg.Nvfp4Tensor(sc.e_t_h["bytes"], sc.e_t_h["scales_packed"], sc.e_t_h["global_scales"], out_dim, k, packed=True, rowwise=True)
    b = pkg.Nvfp4Tensor(sc.input_t_h["bytes"], sc.input_t_h["scales_packed"], sc.input_t_h["global_scale"], in_dim, k, packed=True,
                        rowwise=False)
    want = torch.empty((out_dim, in_dim), device=dev)
    assert (gemm.plan(a, b, out=want).k_splits > 1) == (tokens > 4096)
    gemm.gemm(a, b, out=want)
    # the same partial sums in another order: 32 additions at most
    assert float((dw - want).norm() / want.norm()) <= 32 * 2.0 ** -24
    assert bool(memory[:offset].isnan().all()) and bool(memory[offset + out_dim * in_dim:].isnan().all())
    torch.cuda.synchronize()
    assert pkg.read_device_status() == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens,out_dim", [(128, 64 * 295), (128, 64 * 296), (250, 64 * 148), (300, 64 * 100)])
def test_pair_beside_a_side_stream(pkg, dev, tokens, out_dim, dtype):
    """One CTA less than the chip holds, as many, more tiles than CTAs: beside the transposers of a side stream, where the pair
    kernel starts early or not, the operands and gradients of a call that has one stream, call after call."""
    q, bwd, in_dim = pkg.Nvfp4QuantModule(), pkg.LinearBackwardModule(), 64
    xq = q.quantize_four_six(bf16_normal(781, (tokens, in_dim)).to(dev), rowwise=True, packed=True, decoded_amax=True)
    wq = q.quantize_four_six(bf16_normal(782, (out_dim, in_dim), 0.02).to(dev), rowwise=False, packed=True)
    es = [bf16_normal(783 + i, (tokens, out_dim), 1e-3).to(dev).to(dtype) for i in range(2)]
    sc, side = pkg.LinearBackwardScratch(tokens, in_dim, out_dim, dev), pkg.SideStream(dev)

    def call(e, stream):
        # bf16 gradients: GEMMs into f32 of this K split it and add their partial sums in the order they arrive
        grads = bwd.backward_ms_eden(e=e, weight=wq, input=xq, scratch=sc, sign_seed=SIGN, scale_seed=SCALE, side=stream,
                                     grad_dtype=torch.bfloat16)
        return [t.clone() for t in (*grads, sc.e_h["bytes"], sc.e_h["scales_packed"], sc.e_t_h["bytes"], sc.e_t_h["scales_packed"])]

    want = []
    for e in es:
        torch.cuda.synchronize()
        want.append(call(e, None))
        torch.cuda.synchronize()
    got = [call(es[i & 1], side) for i in range(8)]
    torch.cuda.synchronize()
    for i, tensors in enumerate(got):
        assert all(torch.equal(a, b) for a, b in zip(tensors, want[i & 1])), i
    assert pkg.read_device_status() == 0


@pytest.mark.parametrize("with_side", [False, True])
@pytest.mark.parametrize("inside", [None, "e", "input", "e_h", "weight_t_h"])
def test_backward_dweight_inside_what_the_steps_before_it_read(pkg, dev, inside, with_side):
    """dW may lie in memory that is free by the time its GEMM runs: dY, the saved X, the operands of dX.  Then it is not cleared
    ahead of that.  Calls follow one another with changing inputs and nothing synchronised in between; dX and dbias are the
    bits of calls that ran alone, dW the same partial sums in another order."""
    q, bwd, tokens, in_dim, out_dim = pkg.Nvfp4QuantModule(), pkg.LinearBackwardModule(), 4352, 64, 64
    wq = q.quantize_four_six(bf16_normal(761, (out_dim, in_dim), 0.02).to(dev), rowwise=False, packed=True)
    side = pkg.SideStream(dev) if with_side else None
    source = [(bf16_normal(762 + i, (tokens, out_dim), 1e-3).to(dev), bf16_normal(772 + i, (tokens, in_dim)).to(dev)) for i in range(3)]

    def call(i, place):
        e, x = source[i]
        e, xq = e.clone(), q.quantize_four_six(x, rowwise=True, packed=True, decoded_amax=True)
        memory = {None: None, "e": e, "input": xq.bytes, "e_h": sc.e_h["bytes"], "weight_t_h": sc.weight_t_h["bytes"]}[place]
        dw = torch.full((out_dim, in_dim), float("nan"), device=dev) if memory is None else \
            memory.view(-1).view(torch.float32)[: out_dim * in_dim].view(out_dim, in_dim)
        dx, dw, db = bwd.backward_ms_eden(e=e, weight=wq, input=xq, scratch=sc, sign_seed=SIGN + i, scale_seed=SCALE, dweight=dw,
                                          side=side)
        return dx, dw.clone(), db

    sc = pkg.LinearBackwardScratch(tokens, in_dim, out_dim, dev)
    # room for dW inside the operands' buffers (they are larger than the call needs; the extents it passes stay the same)
    sc.weight_t_h["bytes"] = torch.empty(out_dim * in_dim * 4, dtype=torch.uint8, device=dev)
    want = []
    for i in range(3):
        torch.cuda.synchronize()
        want.append(call(i, None))
        torch.cuda.synchronize()
    for repeat in range(4):
        got = [call(i, inside) for i in range(3)]
        torch.cuda.synchronize()
        for (dx, dw, db), (dx0, dw0, db0) in zip(got, want):
            assert torch.equal(dx, dx0) and torch.equal(db, db0)
            assert float((dw - dw0).norm() / dw0.norm()) <= 32 * 2.0 ** -24
    assert pkg.read_device_status() == 0
