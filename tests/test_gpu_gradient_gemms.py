"""dX and dW GEMM of a backward call beside one another: the same bits as one after the other, what follows on the stream sees both,
small and large grids, split K, with and without a side stream, captured."""
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
