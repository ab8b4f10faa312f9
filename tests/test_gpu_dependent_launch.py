"""Kernels that come in early (programmatic dependent launch) between a memset, another stream, a collective kernel and torch's
own kernels: a chain gives the bits it gives with a synchronisation after every call, eager and captured."""
import pytest
import torch

from tinyinfinitrain_b200._lib import C

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16


class _Chain:
    """Small operands, so that every kernel is shorter than the launch of the next one and their ends overlap.  The weight
    gradients are split in two, whose order of addition to zeros does not matter."""

    def __init__(self, tokens, width):
        g = torch.Generator(device=DEV).manual_seed(31)
        rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
        self.x = rnd(tokens, width).to(BF)
        self.w = [(rnd(width, width) * width ** -0.5).to(BF) for _ in range(3)]
        self.qkv = (rnd(3 * width, width) * width ** -0.5).to(BF)
        self.gamma, self.beta = rnd(width).to(BF), rnd(width).to(BF)
        self.f32 = rnd(width, 40)
        self.acc = torch.empty(width, width, device=DEV)
        self.pad = torch.zeros(8 * 16, dtype=torch.int32, device=DEV)
        self.epoch = torch.zeros(1, dtype=torch.int32, device=DEV)
        self.side = torch.cuda.Stream()

    def run(self, settle):
        cur, width = torch.cuda.current_stream(), self.x.shape[1]

        def done(*results):
            settle()
            return results if len(results) > 1 else results[0]

        h = done(C.gemm(self.x, self.w[0])[0])
        y, mean, rstd = done(*C.layernorm_fwd(h, self.gamma, self.beta, 1e-5))
        self.side.wait_stream(cur)
        with torch.cuda.stream(self.side):                       # another stream reads what an early kernel wrote
            z = done(C.gemm(y, self.w[1])[0])
            zs = done(C.colsum(z))
        dw = done(C.gemm(y, h, True, True, out_fp32=True, splits=2)[0])      # memset, then reduce-adds
        cur.wait_stream(self.side)
        done(C.comm_barrier([self.pad.data_ptr()], 0, 0, self.epoch, 1.0) or z)
        u = done(C.gemm(z, self.w[2], epilogue=1, bias=self.beta)[0])
        qkv = done(C.gemm(u, self.qkv)[0]).view(1, -1, 3, width // 64, 64)
        q, k, v = (qkv[:, :, i] for i in range(3))
        o, lse = done(*C.attn_fwd(q, k, v, 0.125))
        dq, dk, dv = done(*C.attn_bwd(o, q, k, v, o, lse, 0.125))
        self.acc.zero_()                                         # torch's kernel between two of the library
        settle()
        done(C.gemm(o.view(-1, width), u, True, True, out=self.acc, accumulate=True)[0])
        s = done(C.sgemm(self.acc, self.f32))
        t = done(C.sgemm(s, self.f32, False, True, out=self.acc, accumulate=True))   # reads and writes what came before
        return [r.clone() for r in (h, y, mean, rstd, z, zs, dw, u, o, lse, dk, dv, s, t, dq)]


@pytest.mark.parametrize("tokens,width", [(128, 128), (100, 768), (640, 256)])
def test_chain_of_early_kernels(tokens, width):
    chain = _Chain(tokens, width)
    # dQ of more than two key blocks is a sum in any order
    exact = slice(None) if tokens <= 256 else slice(0, -1)
    inputs = [chain.x] + [torch.randn_like(chain.x.float()).to(BF) for _ in range(5)]
    want = []
    for x in inputs:
        chain.x = x
        want.append(chain.run(torch.cuda.synchronize)[exact])
    for _ in range(4):
        got = []
        for x in inputs:                                         # back to back: the next chain follows the last one's tail
            chain.x = x
            got.append(chain.run(lambda: None)[exact])
        torch.cuda.synchronize()
        for a, b in zip(want, got):
            assert all(torch.equal(p, q) for p, q in zip(a, b))
    x = chain.x = inputs[0].clone()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        chain.run(lambda: None)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = chain.run(lambda: None)[exact]
    for i in (0, 3, 1, 5, 2):
        x.copy_(inputs[i])
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(p, q) for p, q in zip(want[i], out)), i
    assert C.status_read(True) == 0
    del graph
