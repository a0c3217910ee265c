"""Kernels launched as programmatic dependents start before the kernel in front of them has ended: calls that read what the call before
them wrote, over every pair of paths, enqueued without waiting and captured into a graph, against the same calls one at a time."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF, F32 = torch.bfloat16, torch.float32


def rand(shape, dtype, seed):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(dtype)


class Chain:
    """Each step reads the result of the step before it (in another shape) as its K or V."""

    def __init__(self, pkg, cuda):
        self.pkg = pkg
        self.inputs = [rand((1, 4, 64, 128), BF, 0).to(cuda), rand((1, 4, 64, 64), F32, 1).to(cuda)]
        self.bf = {(h, l, d): rand((1, h, l, d), BF, 10 + i).to(cuda)
                   for i, (h, l, d) in enumerate([(2, 128, 128), (1, 200, 512), (8, 4, 128), (4, 64, 128), (2, 100, 80)])}
        self.long = rand((1, 8, 1000, 128), BF, 20).to(cuda)
        self.f = rand((1, 4, 100, 64), F32, 21).to(cuda)
        self.results = {}

    def out(self, name, like):
        if name not in self.results:
            self.results[name] = torch.empty_like(like)
        return self.results[name]

    def run(self, flags):
        """Every step's result; the paths taken."""
        p, b, paths = self.pkg, self.bf, []

        def step(name, q, k, v, **kw):
            o = p.forward(q, k, v, out=self.out(name, q), flags=flags, **kw)
            paths.append(p.last_path())
            if not flags:
                torch.cuda.synchronize()
            return o
        x, y = self.inputs
        o = step("stream", x, x, x, pe=p.PE_ROPE_INTERLEAVED)                                             # [4, 64, 128]
        o = step("fused", b[2, 128, 128], o.view(1, 2, 128, 128), b[2, 128, 128])                         # [2, 128, 128]
        o = step("wide", b[1, 200, 512], o.view(1, 1, 64, 512), o.view(1, 1, 64, 512))                    # [1, 200, 512]
        k = self.long
        k.view(-1)[:o.numel()].copy_(o.view(-1))
        o = step("decode", b[8, 4, 128], k, k, pe=p.PE_NONE)                                              # [8, 4, 128]
        o = step("odd", b[2, 100, 80], o.reshape(-1)[:3200].view(1, 2, 20, 80), o.reshape(-1)[:3200].view(1, 2, 20, 80))
        o = step("stream_again", b[4, 64, 128], o.reshape(-1)[:15360].view(1, 4, 30, 128), o.reshape(-1)[:15360].view(1, 4, 30, 128))
        r = p.rope_k(o, pos0=3, stream=torch.cuda.current_stream().cuda_stream)
        o = step("stream_of_rotated", b[4, 64, 128], r, o, pe=p.PE_ROPE_Q_ONLY)
        z = step("short", y, y, y)                                                                        # fp32 [4, 64, 64]
        z = step("short_encoded", y, z, z, pe=p.PE_SINUSOIDAL)
        z = step("long", self.f, z, z)
        z = step("short_again", y, z[:, :, :64].contiguous(), y)
        return paths

    def refill(self, seed):
        for i, t in enumerate(self.inputs):
            t.copy_(rand(t.shape, t.dtype, seed + i), non_blocking=False)

    def check(self, want):
        for name, w in want.items():
            # the order in which slices add their scores is not fixed; a stale read differs by the size of the values
            torch.testing.assert_close(self.results[name], w, rtol=2.0 ** -6 if w.dtype == BF else 1e-4, atol=2e-2 if w.dtype == BF else 1e-4)


def test_each_call_sees_what_the_one_before_it_wrote(pkg, cuda):
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        chain, wants = Chain(pkg, cuda), []
        for seed in (100, 200, 300):
            chain.refill(seed)
            paths = chain.run(0)
            wants.append({n: t.clone() for n, t in chain.results.items()})
        assert paths == ["splitd_stream", "tc_fused", "tc_wide", "tc_decode", "tc_f32", "splitd_stream", "splitd_stream", "splitd_tc",
                         "splitd_stream", "tc_f32", "splitd_tc"]
        assert all((wants[0][n].float() - wants[1][n].float()).abs().max() > 0.05 for n in ("stream", "short", "short_encoded", "long"))
        for seed, want in zip((100, 200, 300), wants):
            chain.refill(seed)
            chain.run(pkg.FLAG_ASYNC)
            s.synchronize()
            chain.check(want)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            chain.run(pkg.FLAG_ASYNC)
        for seed, want in zip((300, 100, 200), (wants[2], wants[0], wants[1])):
            chain.refill(seed)
            for t in chain.results.values():
                t.fill_(float("nan"))
            g.replay()
            s.synchronize()
            chain.check(want)
        del g
    torch.cuda.synchronize()
    pkg.lib().b200attn_release_workspace()   # the ring of splitd_tc counts calls on the host: a captured one only once
