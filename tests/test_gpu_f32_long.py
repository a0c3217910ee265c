"""fp32 on the tensor cores beyond 64 queries or keys (csrc/tc_f32.cuh) against the oracle, at the sizes where the tiles,
the 64-column groups, the key steps and the split over a cluster have their edges."""
import numpy as np
import pytest
import torch

import oracle_lib as ol
from gpu_util import to_dev

pytestmark = pytest.mark.gpu
# uniform inputs: outputs are below 1; the library errs by 1e-7 to 2e-7 of them, the fp32 oracle (sums of up to 1000 terms) by ~1e-6
MAX_ABS = 5e-6

SHAPES = [(1, 1, 1, 65, 1), (1, 2, 65, 1, 4), (1, 3, 128, 128, 64), (2, 1, 129, 127, 65), (1, 2, 64, 129, 100), (1, 1, 80, 80, 512),
          (1, 5, 257, 385, 128), (1, 1, 97, 1000, 192), (1, 40, 70, 66, 33), (1, 148, 100, 65, 8)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_against_oracle(pkg, cuda, shape):
    B, H, Lq, Lk, D = shape
    Q, K, V = ol.make_qkv(B, H, Lq, Lk, D, 80, "uniform")
    got = pkg.forward(to_dev(Q, cuda), to_dev(K, cuda), to_dev(V, cuda)).cpu().numpy()
    assert pkg.last_path() == "tc_f32"
    res = ol.compare(got, ol.attention(Q, K, V))
    assert res["ok"] and res["max_abs"] <= MAX_ABS, (shape, res)


@pytest.mark.parametrize("f16", [False, True])
@pytest.mark.parametrize("shape,path", [((1, 199, 1, 65, 8), "tc_f32"), ((1, 200, 4, 65, 8), "splitd_two_pass"), ((1, 200, 5, 65, 8), "tc_f32"),
                                        ((1, 150, 65, 16, 8), "splitd_two_pass"), ((1, 150, 65, 17, 8), "tc_f32"), ((1, 250, 100, 32, 72), "splitd_two_pass"),
                                        ((1, 249, 100, 32, 72), "tc_f32"), ((1, 250, 33, 70, 72), "tc_f32")], ids=str)
def test_few_rows_on_one_side(pkg, cuda, shape, path, f16):
    """On either side of the lines between this path and the CUDA-core kernels."""
    T = [x.astype(np.float16 if f16 else np.float32) for x in ol.make_qkv(*shape, 87, "uniform")]
    got = pkg.forward(*(to_dev(x, cuda) for x in T))
    assert pkg.last_path() == path
    want = ol.attention(*(x.astype(np.float32) for x in T))
    assert (np.abs(got.float().cpu().numpy() - want) <= MAX_ABS + (np.abs(want) * 2.0 ** -11 if f16 else 0.0)).all()


@pytest.mark.parametrize("pe,rd", [(ol.PE_ROPE_INTERLEAVED, 0), (ol.PE_ROPE_INTERLEAVED, 10), (ol.PE_ROPE_HALF, 0), (ol.PE_ROPE_HALF, 12),
                                   (ol.PE_SINUSOIDAL, 0), (ol.PE_ROPE_Q_ONLY, 0)])
@pytest.mark.parametrize("D", [34, 96])
def test_encodings(pkg, cuda, pe, rd, D):
    Q, K, V = ol.make_qkv(1, 3, 130, 200, D, 81, "uniform")
    got = pkg.forward(to_dev(Q, cuda), to_dev(K, cuda), to_dev(V, cuda), pe=pe, rotary_dim=rd).cpu().numpy()
    assert pkg.last_path() == "tc_f32"
    # (the device's and the host's fp32 angle functions differ by a few ulp of angles up to 200)
    res = ol.compare(got, ol.attention(Q, K, V, pe=pe, rotary_dim=rd or None))
    assert res["ok"] and res["max_abs"] <= 5e-5, (pe, rd, D, res)


@pytest.mark.parametrize("which", [0, 1, 2])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.3e38])
def test_non_finite_values_as_on_the_cuda_cores(pkg, cuda, which, value):
    """The pieces of a non-finite value cannot go through the MMAs; the result is that of the FFMA kernels."""
    T = [to_dev(x, cuda) for x in ol.make_qkv(1, 2, 150, 150, 96, 82, "uniform")]
    T[which][0, 1, 7, 5] = value
    got = pkg.forward(*T)
    assert pkg.last_path() == "tc_f32"
    want = pkg.forward(*T, flags=pkg.FLAG_FORCE_GENERIC)
    assert pkg.last_path() == "splitd_two_pass"
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    torch.testing.assert_close(torch.nan_to_num(got), torch.nan_to_num(want), rtol=1e-4, atol=MAX_ABS)


def test_keys_of_minus_infinity_scores_have_no_weight(pkg, cuda):
    """A whole half tile of keys whose scores are -inf (finite inputs whose products overflow) leaves the other keys alone."""
    Q, K, V = ol.make_qkv(1, 1, 70, 200, 64, 83, "uniform")
    Q[..., 0] = 1e30
    K[..., 0] = 0.0
    K[0, 0, 64:128, 0] = -1e30
    Q, K, V = (to_dev(x, cuda) for x in (Q, K, V))
    keep = [j for j in range(200) if not 64 <= j < 128]
    got = pkg.forward(Q, K, V)
    want = pkg.forward(Q, K[:, :, keep].contiguous(), V[:, :, keep].contiguous())
    assert pkg.last_path() == "tc_f32"
    torch.testing.assert_close(got, want, rtol=1e-5, atol=MAX_ABS)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_non_finite_value_stays_where_it_belongs(pkg, cuda, dtype):
    """It decides the rows and columns it enters into; the others do not change by a bit.  (The pieces of its operand are the value and
    zeros, so it goes through the MMAs like any other.)"""
    D = 200   # four column blocks, the last one short
    T = [torch.randn(1, 3, 300, D, generator=torch.Generator().manual_seed(7 + i)).to(dtype).to(cuda) for i in range(3)]
    clean = pkg.forward(*T, pe=ol.PE_ROPE_INTERLEAVED)
    assert pkg.last_path() == "tc_f32"
    bad = [t.clone() for t in T]
    bad[0][0, 0, 130, 3] = float("nan")     # a query row
    bad[1][0, 1, 299, 0] = float("nan")     # a key: every row of its head
    bad[2][0, 2, 5, 70] = float("inf")      # a value: its column
    bad[2][0, 2, 260, 7] = float("-inf")
    got = pkg.forward(*bad, pe=ol.PE_ROPE_INTERLEAVED)
    assert pkg.last_path() == "tc_f32"
    assert torch.isnan(got[0, 0, 130]).all() and torch.isnan(got[0, 1]).all()
    assert torch.isposinf(got[0, 2, :, 70]).all() and torch.isneginf(got[0, 2, :, 7]).all()
    rows = [i for i in range(300) if i != 130]
    cols = [c for c in range(D) if c not in (7, 70)]
    assert torch.equal(got[0, 0, rows], clean[0, 0, rows]) and torch.equal(got[0, 2][:, cols], clean[0, 2][:, cols])


def test_replays_of_a_captured_call_are_independent(pkg, cuda):
    """A replay that meets a non-finite value leaves nothing behind for the next ones."""
    T = [to_dev(x, cuda) for x in ol.make_qkv(1, 2, 140, 130, 64, 86, "uniform")]
    keep = [t.clone() for t in T]
    out, s = torch.empty_like(T[0]), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        want = pkg.forward(*T)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            pkg.forward(*T, out=out, flags=pkg.FLAG_ASYNC)
            pkg.forward(*T, out=out, flags=pkg.FLAG_ASYNC)
        for value in (None, float("inf"), None, float("nan"), None):
            for t, k in zip(T, keep):
                t.copy_(k)
                if value is not None:
                    t[0, 0, 3, 3] = value
            g.replay()
            s.synchronize()
            if value is None:
                assert torch.equal(out, want)
            else:
                assert torch.isnan(out[0, 0]).any() and torch.equal(out[0, 1], want[0, 1])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_large_values_stay_finite(pkg, cuda, dtype):
    """A weighted mean of finite values is finite, whatever their size and number."""
    T = [torch.rand(1, 2, 300, 72, generator=torch.Generator().manual_seed(9 + i)).to(dtype).to(cuda) for i in range(3)]
    T[2][0, 1, :, 30:] *= 3.3e38
    got = pkg.forward(*T)
    assert pkg.last_path() == "tc_f32"
    want = pkg.forward(*T, flags=pkg.FLAG_FORCE_GENERIC)
    assert torch.isfinite(want).all()
    torch.testing.assert_close(got, want, rtol=1e-5 if dtype == torch.float32 else 2.0 ** -7, atol=MAX_ABS)


@pytest.mark.parametrize("D", [1, 2])
def test_large_scores_of_the_narrowest_heads_stay_finite(pkg, cuda, D):
    """log2(e) / sqrt(head_d) is above 1: the scaled score of a finite one need not be finite."""
    T = [torch.rand(1, 2, 100, D, generator=torch.Generator().manual_seed(12 + i)) for i in range(3)]
    T[0] = torch.full_like(T[0], 1e19)
    T[1] = torch.full_like(T[1], 3e19 / D)
    T[1][0, 1, 10:] *= 0.5
    got = pkg.forward(*(t.to(cuda) for t in T)).cpu()
    assert pkg.last_path() == "tc_f32"
    want = torch.stack([T[2][0, 0].mean(0), T[2][0, 1, :10].mean(0)])   # equal scores, and a half of the keys without weight
    torch.testing.assert_close(got[0], want[:, None].expand(2, 100, D), rtol=1e-5, atol=MAX_ABS)


def test_scratch_cap_and_misaligned_tensors(pkg, cuda):
    """Heads go in passes where the scratch cap is small; rows and pointers without 16-byte alignment are taken too."""
    Q, K, V = ol.make_qkv(1, 7, 150, 170, 40, 84, "uniform")
    want = ol.attention(Q, K, V)
    pkg.set_option(1, 1)
    try:
        got = pkg.forward(to_dev(Q, cuda), to_dev(K, cuda), to_dev(V, cuda)).cpu().numpy()
    finally:
        pkg.set_option(1, 2048)
    assert ol.compare(got, want)["max_abs"] <= MAX_ABS

    def off(x):   # the same tensor four bytes into an allocation
        buf = torch.empty(x.size + 1, dtype=torch.float32, device=cuda)[1:].view(x.shape)
        buf.copy_(torch.from_numpy(x))
        return buf
    out = off(np.zeros_like(Q))
    got = pkg.forward(off(Q), off(K), off(V), out=out).cpu().numpy()
    assert pkg.last_path() == "tc_f32" and ol.compare(got, want)["max_abs"] <= MAX_ABS


def test_graph_capture_and_two_streams(pkg, cuda):
    Q, K, V = ol.make_qkv(1, 2, 140, 130, 64, 85, "uniform")
    want = ol.attention(Q, K, V)
    q, k, v = (to_dev(x, cuda) for x in (Q, K, V))
    out = torch.empty_like(q)
    pkg.forward(q, k, v, out=out)
    g = torch.cuda.CUDAGraph()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        pkg.forward(q, k, v, out=out, flags=pkg.FLAG_ASYNC)
        s.synchronize()
        with torch.cuda.graph(g, stream=s):
            pkg.forward(q, k, v, out=out, flags=pkg.FLAG_ASYNC)
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert ol.compare(out.cpu().numpy(), want)["max_abs"] <= MAX_ABS
