"""Kernels that start while the one before them drains: chains in which a small grid follows a large one and the other way
round, every call rewrites the buffers of the call before it, the inputs change from call to call and nothing is synchronised
in between -- on the default stream, on another one, and in a captured graph whose backward call forks onto a side stream and
joins it.  Every result is the one of a call that ran alone."""
import pytest
import torch

from helpers import bf16_normal

pytestmark = pytest.mark.gpu
SIGN, SCALE = 0x12345678, 0x9ABCDEF0


class Chain:
    """Tensor amax -> four-six -> decode of X, logical scales packed for a GEMM, and a linear backward (dY amax, both quantizers
    of dY, column sums, both transposers, GEMMs that do not split K), everything into buffers of its own."""

    def __init__(self, pkg, dev, tokens, in_dim, out_dim):
        self.q, self.gemm, self.bwd, self.decode = (pkg.Nvfp4QuantModule(), pkg.Nvfp4GemmModule(), pkg.LinearBackwardModule(),
                                                    pkg.Nvfp4DecodeModule())
        self.x = torch.empty((tokens, in_dim), dtype=torch.bfloat16, device=dev)
        self.e = torch.empty((tokens, out_dim), dtype=torch.bfloat16, device=dev)
        self.inputs = [(bf16_normal(801 + i, (tokens, in_dim), 1.0 + i).to(dev), bf16_normal(811 + i, (tokens, out_dim), 1e-3 * (1 + i)).to(dev))
                       for i in range(3)]
        w = bf16_normal(821, (out_dim, in_dim), 0.02).to(dev)
        self.wq = self.q.quantize_four_six(w, rowwise=False, packed=True)
        self.tensor = self.q.quantize_four_six(self.inputs[0][0], rowwise=False, packed=False)
        self.rows = self.q.quantize_four_six(self.inputs[0][0], rowwise=True, packed=True, decoded_amax=True)
        self.scratch, self.side = pkg.LinearBackwardScratch(tokens, in_dim, out_dim, dev), pkg.SideStream(dev)
        bf16 = dict(dtype=torch.bfloat16, device=dev)
        self.y, self.dx, self.dw = (torch.empty(s, **bf16) for s in ((tokens, out_dim), (tokens, in_dim), (out_dim, in_dim)))
        self.db = torch.empty(out_dim, device=dev)

    def call(self, i):
        """Outputs as copies, taken on the stream as well."""
        x, e = self.inputs[i]
        self.x.copy_(x)
        self.e.copy_(e)
        self.q.quantize_four_six(self.x, rowwise=False, packed=False, out=self.tensor)
        out = [self.decode.decode(self.tensor)]
        self.q.quantize_four_six(self.x, rowwise=True, packed=True, out=self.rows, decoded_amax=True)
        self.gemm.gemm(self.rows, self.wq, out=self.y)
        self.bwd.backward_ms_eden(e=self.e, weight=self.wq, input=self.rows, scratch=self.scratch, sign_seed=SIGN, scale_seed=SCALE,
                                  dinput=self.dx, dweight=self.dw, dbias=self.db, side=self.side)
        return out + [t.clone() for t in (self.tensor.bytes, self.rows.bytes, self.rows.scales, self.y, self.dx, self.dw, self.db,
                                          self.scratch.input_t_h["bytes"], self.scratch.e_t_h["scales_packed"])]


@pytest.mark.parametrize("tokens,in_dim,out_dim", [(128, 64, 64), (1000, 768, 72), (4096, 64, 2304), (2048, 768, 3072)])
def test_chains_read_what_the_kernels_before_them_wrote(pkg, dev, tokens, in_dim, out_dim):
    chain = Chain(pkg, dev, tokens, in_dim, out_dim)
    want = []
    for i in range(3):
        torch.cuda.synchronize()
        want.append(chain.call(i))
        torch.cuda.synchronize()
    assert not torch.equal(want[0][4], want[1][4])

    def check(results):
        torch.cuda.synchronize()
        for i, tensors in results:
            for k, (a, b) in enumerate(zip(tensors, want[i])):
                assert torch.equal(a, b), (i, k)

    check([(i % 3, chain.call(i % 3)) for i in range(9)])
    other = torch.cuda.Stream()
    other.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(other):
        results = [(i % 3, chain.call(i % 3)) for i in range(9)]
    check(results)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = [(i, chain.call(i)) for i in range(3)]
    for _ in range(3):
        graph.replay()
    check(captured)
    assert pkg.read_device_status() == 0
