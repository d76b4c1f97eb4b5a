"""dX and dW GEMM of a backward call beside one another: the same bits as one after the other, what follows on the stream sees both,
small and large grids, split K, with and without a side stream, captured, timed; one after the other where dW lies in dX's operands."""
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

pytestmark = pytest.mark.gpu


class Call:
    def __init__(self, pkg, dev, tokens, i, o, dtype, grad, side):
        q = pkg.Nvfp4QuantModule()
        g = torch.Generator(device=dev)
        g.manual_seed(tokens + i + o)
        self.bwd, self.grad, self.side = pkg.LinearBackwardModule(), grad, pkg.SideStream(dev) if side else None
        self.es = [(torch.randn(tokens, o, generator=g, device=dev) * 1e-3).to(dtype) for _ in range(3)]
        self.w = q.quantize_four_six((torch.randn(o, i, generator=g, device=dev) * 0.02).to(torch.bfloat16), rowwise=False, packed=True)
        self.x = q.quantize_four_six(torch.randn(tokens, i, generator=g, device=dev).to(torch.bfloat16), rowwise=True, packed=True,
                                     decoded_amax=True)
        self.scratch = pkg.LinearBackwardScratch(tokens, i, o, dev)
        self.dx = torch.empty(tokens, i, device=dev, dtype=grad)
        self.dw = torch.empty(o, i, device=dev)

    def run(self, k):
        self.bwd.backward_ms_eden(e=self.es[k], weight=self.w, input=self.x, scratch=self.scratch, sign_seed=7 + k, scale_seed=9,
                                  grad_dtype=self.grad, dinput=self.dx, dweight=self.dw, side=self.side)

    def alone(self, k):
        """The same operands through the entry whose GEMMs run one after the other."""
        self.run(k)
        torch.cuda.synchronize()
        dx, dw = torch.empty_like(self.dx), torch.empty_like(self.dw)
        self.bwd.backward_device_scale(self.scratch, dx, dw)
        torch.cuda.synchronize()
        return dx, dw


# grids: a few tiles each; dX below and dW at the SMs' number; split K with the output cleared along the way; pairs; ragged; dX split
# and clearing its own output; many waves
@pytest.mark.parametrize("tokens,i,o,dtype,grad", [
    (128, 256, 256, torch.bfloat16, torch.bfloat16), (1000, 768, 3072, torch.float32, torch.float32),
    (4096, 768, 768, torch.bfloat16, torch.bfloat16), (8192, 768, 2304, torch.bfloat16, torch.bfloat16),
    (1024, 1024, 8192, torch.bfloat16, torch.bfloat16), (515, 320, 264, torch.bfloat16, torch.float32),
    (512, 768, 8192, torch.bfloat16, torch.float32),
    (16384, 1024, 4096, torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("side", [False, True])
def test_side_by_side_is_one_after_the_other(pkg, dev, tokens, i, o, dtype, grad, side):
    pkg.set_deterministic_reductions(True)  # at most two splits: sums without an order
    try:
        c = Call(pkg, dev, tokens, i, o, dtype, grad, side)
        want = [c.alone(k) for k in range(3)]
        seen = []
        for n in range(9):
            c.run(n % 3)
            seen.append((c.dx.clone(), c.dw.clone()))  # the stream's next kernels, while the next call follows at once
        graph = torch.cuda.CUDAGraph()
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream), torch.cuda.graph(graph, stream=stream):
            captured = []
            for n in range(3):
                c.run(n)
                captured.append((c.dx.clone(), c.dw.clone()))
        for _ in range(2):
            graph.replay()
        torch.cuda.synchronize()
        for n, (dx, dw) in enumerate(seen + captured):
            assert torch.equal(dx, want[n % 3][0]) and torch.equal(dw, want[n % 3][1])
        assert pkg.read_device_status() == 0
    finally:
        pkg.set_deterministic_reductions(False)


@pytest.mark.parametrize("tokens,dx_splits", [(1000, False), (512, True)])
def test_dw_starts_before_dx_has_ended(pkg, dev, tokens, dx_splits):
    """Also behind a dX whose output is cleared in front of it: its wait for what runs before it covers the clearing."""
    i, o = 768, 8192 if dx_splits else 3072
    c = Call(pkg, dev, tokens, i, o, torch.bfloat16, torch.float32, True)
    c.run(0)
    torch.cuda.synchronize()
    e_h, weight_t_h = c.scratch.as_tensor("e_h"), c.scratch.as_tensor("weight_t_h")
    assert (pkg.Nvfp4GemmModule().plan(e_h, weight_t_h, out=c.dx).k_splits > 1) == dx_splits
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream), torch.cuda.graph(graph, stream=stream):
        c.run(0)
    graph.replay()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as prof:
        graph.replay()
        torch.cuda.synchronize()
    spans = sorted((e.time_range.start, e.time_range.end) for e in prof.events() if "nvfp4_gemm_tcgen05_kernel" in e.name)
    if not spans:
        pytest.skip("no kernel activity records on this machine")
    (dx_start, dx_end), (dw_start, _) = spans
    assert dw_start < dx_start + 0.75 * (dx_end - dx_start), spans
    assert pkg.read_device_status() == 0


@pytest.mark.parametrize("side", [False, True])
@pytest.mark.parametrize("inside,field", [("e_h", "bytes"), ("weight_t_h", "bytes"), ("e_h", "scales_packed"), ("weight_t_h", "scales_packed")])
def test_dweight_inside_the_operands_of_dx(pkg, dev, inside, field, side):
    """dW may lie where dX's operands do, which its GEMM alone needs no longer: it then waits for all of dX.  Neither is split, so that
    nothing is cleared between the two, and dX has more tiles than there are SMs."""
    tokens, i, o = 3840, 2304, 768
    c = Call(pkg, dev, tokens, i, o, torch.bfloat16, torch.bfloat16, side)
    gemm = pkg.Nvfp4GemmModule()
    dx_plan = gemm.plan(c.scratch.as_tensor("e_h"), c.scratch.as_tensor("weight_t_h"), out=c.dx)
    tiles = -(-tokens // dx_plan.block_m) * -(-i // dx_plan.block_n)
    assert dx_plan.k_splits == 1 and tiles > 2 * torch.cuda.get_device_properties(dev).multi_processor_count
    assert gemm.plan(c.scratch.as_tensor("e_t_h"), c.scratch.as_tensor("input_t_h"), out=c.dw).k_splits == 1
    want = []
    for k in range(3):
        c.run(k)
        torch.cuda.synchronize()
        want.append((c.dx.clone(), c.dw.clone()))
    # the operand's plane in front of a buffer as large as dW (the call's extents stay what they are)
    memory = torch.empty(o * i * 4, dtype=torch.uint8, device=dev)
    getattr(c.scratch, inside)[field] = memory
    c.dw = memory.view(torch.float32).view(o, i)
    got = []
    for k in range(6):
        c.run(k % 3)
        got.append((c.dx.clone(), c.dw.clone()))
    torch.cuda.synchronize()
    for k, (dx, dw) in enumerate(got):
        assert torch.equal(dx, want[k % 3][0]) and torch.equal(dw, want[k % 3][1])
    assert pkg.read_device_status() == 0


@pytest.mark.parametrize("tokens,o", [(1000, 3072), (512, 8192)])
def test_timed_one_after_the_other(pkg, dev, tokens, o):
    """The events around each GEMM stand between the two."""
    pkg.set_deterministic_reductions(True)
    try:
        c = Call(pkg, dev, tokens, 768, o, torch.bfloat16, torch.float32, True)
        want = c.alone(0)
        pkg.gemm_timing_begin(8)
        try:
            c.run(0)
        finally:
            timed = pkg.gemm_timing_end()
        torch.cuda.synchronize()
        assert timed[0] == 2
        assert torch.equal(c.dx, want[0]) and torch.equal(c.dw, want[1])
        assert pkg.read_device_status() == 0
    finally:
        pkg.set_deterministic_reductions(False)
