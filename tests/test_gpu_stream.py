"""The streamed split-head_d kernel (csrc/splitd_stream.cuh) against the oracle: slices around its units (atoms of 32 columns, groups and
blocks of four), 16-bit tensors, encodings, several problems in one launch."""
import numpy as np
import pytest
import torch

import oracle_lib as ol
from gpu_util import bf16_from_dev, bf16_problem, bf16_to_dev, to_dev

pytestmark = pytest.mark.gpu
MAX_ABS = 5e-6   # fp32, uniform inputs: the library errs by 1e-7 of outputs below 1, the fp32 oracle by ~1e-6

def attention64(Q, K, V, pe=ol.PE_NONE):
    """The oracle's mathematics in 64 bits, on its own fp32 tables where the encoding is the additive one: a row's scores are then
    near head_d / 2 before the scaling, and the fp32 oracle's sum of head_d terms errs by more than the bounds here."""
    Q, K, V = (x.astype(np.float64) for x in (Q, K, V))
    if pe == ol.PE_SINUSOIDAL:
        D = Q.shape[-1]
        s, c = ol.sinusoidal_tables(max(Q.shape[2], K.shape[2]), D)
        tab = np.where(np.arange(D) % 2 == 0, s, c)   # a pair's columns both hold its value
        Q, K = Q + tab[:Q.shape[2]], K + tab[:K.shape[2]]
    S = Q @ K.swapaxes(-1, -2) / np.sqrt(Q.shape[-1])
    P = np.exp(S - S.max(-1, keepdims=True))
    return P / P.sum(-1, keepdims=True) @ V


def want_of(Q, K, V, pe):
    return attention64(Q, K, V, pe) if pe == ol.PE_SINUSOIDAL else ol.attention(Q, K, V, pe=pe)


def bound(pe, D):
    """Largest difference, for values up to 1 or so.  The host's and the device's fp32 frequencies differ by an ulp or two: up to
    63 * 2^-23 of an angle at position 63, which enters a score of the additive encoding with the weights of head_d / 2 pairs of
    magnitude 1 (over sqrt(head_d)), one of the rotation with those of products of inputs."""
    return {ol.PE_NONE: MAX_ABS, ol.PE_SINUSOIDAL: 63 * 2.0 ** -23 * D ** 0.5}.get(pe, 5e-5)


# heads x head_d such that a CTA has 9 to 33 atoms (one slice per head up to a few), odd lengths, a partial last atom and block
WIDE = [(1, 148, 16, 16, 300), (1, 100, 33, 17, 1000), (1, 74, 64, 64, 1056), (1, 37, 1, 64, 2052), (1, 140, 50, 49, 128), (1, 20, 64, 48, 4096), (1, 148, 64, 1, 32)]


@pytest.mark.parametrize("shape", WIDE, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("pe", [ol.PE_NONE, ol.PE_ROPE_INTERLEAVED, ol.PE_SINUSOIDAL])
def test_fp32(pkg, cuda, shape, pe):
    B, H, Lq, Lk, D = shape
    Q, K, V = ol.make_qkv(B, H, Lq, Lk, D, 90, "uniform")
    want = want_of(Q, K, V, pe)
    q, k, v = (to_dev(x, cuda) for x in (Q, K, V))
    for rep in range(2):
        got = pkg.forward(q, k, v, pe=pe).cpu().numpy()
        # (a slice of up to 256 columns without an encoding fits the kernel that keeps V in shared memory)
        assert pkg.last_path() in (("splitd_stream", "splitd_tc") if pe == ol.PE_NONE else ("splitd_stream",))
        res = ol.compare(got, want)
        assert res["max_abs"] <= bound(pe, D), (shape, pe, res)


@pytest.mark.parametrize("shape,dtype,pe,path", [
    ((1, 16, 8, 8, 2048), torch.float32, ol.PE_ROPE_INTERLEAVED, "splitd_fused"), ((1, 16, 8, 9, 2048), torch.float32, ol.PE_ROPE_INTERLEAVED, "splitd_stream"),
    ((1, 16, 8, 8, 1536), torch.float32, ol.PE_SINUSOIDAL, "splitd_stream"),
    ((1, 148, 4, 4, 288), torch.float16, ol.PE_SINUSOIDAL, "splitd_stream"), ((1, 148, 16, 16, 128), torch.bfloat16, ol.PE_NONE, "splitd_fused"),
    ((1, 148, 17, 16, 128), torch.bfloat16, ol.PE_NONE, "splitd_stream"), ((1, 75, 32, 32, 64), torch.float16, ol.PE_NONE, "splitd_fused"),
    ((1, 75, 32, 33, 64), torch.float16, ol.PE_NONE, "splitd_stream"), ((1, 1, 32, 32, 3232), torch.bfloat16, ol.PE_NONE, "splitd_fused"),
    ((1, 1, 32, 32, 3200), torch.bfloat16, ol.PE_NONE, "splitd_stream")], ids=str)
def test_few_rows(pkg, cuda, shape, dtype, pe, path):
    """On either side of the lines between this kernel and the CUDA-core one."""
    T = [to_dev(x, cuda).to(dtype) for x in ol.make_qkv(*shape, 89, "uniform")]
    got = pkg.forward(*T, pe=pe).float().cpu().numpy()
    if torch.cuda.get_device_properties(cuda).multi_processor_count == 148:
        assert pkg.last_path() == path
    want = want_of(*(t.float().cpu().numpy() for t in T), pe)
    half_ulp = {torch.float32: 0.0, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
    assert (np.abs(got - want) <= np.abs(want) * half_ulp + max(bound(pe, shape[-1]), 5e-5)).all()


@pytest.mark.parametrize("D,rd", [(36, 0), (64, 6), (200, 34)])
@pytest.mark.parametrize("pe", [ol.PE_ROPE_INTERLEAVED, ol.PE_ROPE_Q_ONLY])
def test_partial_rotary(pkg, cuda, D, rd, pe):
    Q, K, V = ol.make_qkv(2, 3, 30, 61, D, 91, "uniform")
    got = pkg.forward(to_dev(Q, cuda), to_dev(K, cuda), to_dev(V, cuda), pe=pe, rotary_dim=rd, rope_base=500.0).cpu().numpy()
    assert pkg.last_path() == "splitd_stream"
    res = ol.compare(got, ol.attention(Q, K, V, pe=pe, rotary_dim=rd or None, base=500.0))
    assert res["ok"] and res["max_abs"] <= 5e-5, res


@pytest.mark.parametrize("shape", [(1, 4, 64, 64, 512), (1, 148, 17, 33, 200), (1, 9, 64, 31, 4096), (1, 60, 5, 64, 1032)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("pe", [ol.PE_NONE, ol.PE_ROPE_INTERLEAVED, ol.PE_SINUSOIDAL])
@pytest.mark.parametrize("f16", [False, True])
def test_16_bit(pkg, cuda, shape, pe, f16):
    B, H, Lq, Lk, D = shape
    if f16:
        T = [x.astype(np.float16) for x in ol.make_qkv(B, H, Lq, Lk, D, 92, "normal")]
        up = [x.astype(np.float32) for x in T]
        got = pkg.forward(*(to_dev(x, cuda) for x in T), pe=pe).float().cpu().numpy()
    else:
        bits, up = bf16_problem(B, H, Lq, Lk, D, 92)
        got = bf16_from_dev(pkg.forward(*(bf16_to_dev(b, cuda) for b in bits), pe=pe))
    assert pkg.last_path() == "splitd_stream"
    want = want_of(*up, pe)
    # everything up to the output is fp32: half a unit in the last place of the output's format, and what fp32 differs by
    err = np.abs(got - want)
    assert (err <= np.abs(want) * (2.0 ** -11 if f16 else 2.0 ** -8) + 4 * max(bound(pe, D), 5e-5)).all(), err.max()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("which", [0, 1, 2])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_non_finite_values_as_on_the_cuda_cores(pkg, cuda, dtype, which, value):
    T = [to_dev(x, cuda).to(dtype) for x in ol.make_qkv(1, 3, 50, 50, 304, 93, "uniform")]
    T[which][0, 1, 7, 5] = value
    got = pkg.forward(*T, pe=ol.PE_ROPE_INTERLEAVED)
    assert pkg.last_path() == "splitd_stream"
    want = pkg.forward(*T, pe=ol.PE_ROPE_INTERLEAVED, flags=pkg.FLAG_FORCE_GENERIC)
    assert pkg.last_path() == "splitd_fused"
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_infinities_beyond_rotary_dim(pkg, cuda, dtype):
    """A column that is not rotated does not meet its neighbour's infinity (times a sine of 0): a key with a score of -inf has no weight."""
    T = [to_dev(x, cuda).to(dtype) for x in ol.make_qkv(1, 3, 50, 50, 304, 99, "uniform")]
    T[0][..., 100].abs_().clamp_(min=0.1)
    T[1][0, 1, 7, 100] = float("-inf")
    got = pkg.forward(*T, pe=ol.PE_ROPE_INTERLEAVED, rotary_dim=100)
    assert pkg.last_path() == "splitd_stream"
    want = pkg.forward(*T, pe=ol.PE_ROPE_INTERLEAVED, rotary_dim=100, flags=pkg.FLAG_FORCE_GENERIC)
    assert torch.isfinite(want).all()
    torch.testing.assert_close(got, want, rtol=1e-5 if dtype == torch.float32 else 2.0 ** -7, atol=MAX_ABS)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H,D,L", [(148, 512, 64), (148, 640, 33), (20, 4096, 64)])
def test_non_finite_values_in_many_blocks(pkg, cuda, dtype, H, D, L):
    """A key whose whole V row is infinite, in slices of four and more blocks of output columns: the plain loops of one block's
    epilogue are still running when blocks further on have been split and multiplied."""
    T = [to_dev(x, cuda).to(dtype) for x in ol.make_qkv(1, H, L, L, D, 94, "uniform")]
    T[2][0, :, 5] = float("inf")
    T[2][0, 3, 9, ::2] = float("-inf")
    want = pkg.forward(*T, pe=ol.PE_ROPE_INTERLEAVED, flags=pkg.FLAG_FORCE_GENERIC)
    assert pkg.last_path().startswith("splitd_") and pkg.last_path() != "splitd_stream"
    for _ in range(3):
        got = pkg.forward(*T, pe=ol.PE_ROPE_INTERLEAVED)
        assert pkg.last_path() == "splitd_stream"
        assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isposinf(got), torch.isposinf(want)) and torch.equal(torch.isneginf(got), torch.isneginf(want))


@pytest.mark.parametrize("dtype,pe,H,D", [(torch.float32, ol.PE_NONE, 148, 512), (torch.float32, ol.PE_ROPE_INTERLEAVED, 3, 304),
                                           (torch.float32, ol.PE_ROPE_Q_ONLY, 148, 512), (torch.bfloat16, ol.PE_ROPE_INTERLEAVED, 3, 304)])
def test_keys_of_minus_infinity_scores_have_no_weight(pkg, cuda, dtype, pe, H, D):
    """Finite inputs whose products overflow: such keys have weight 0 and leave the others alone, as on the CUDA cores.  (1e30 =
    9.95e29 + 4.70e27 - 4.08e24: the products with a third piece have the other sign.)  The last pair of columns: its angles
    stay near 0, so that the rotation keeps the signs."""
    T = [to_dev(x, cuda).to(dtype) for x in ol.make_qkv(1, H, 48, 60, D, 95, "uniform")]
    T[0][..., -2], T[0][..., -1] = 1e30, 0.0
    T[1][..., -2:] = 0.0
    T[1][..., 20:40, -2] = -1e30
    got = pkg.forward(*T, pe=pe)
    assert pkg.last_path() == "splitd_stream"
    want = pkg.forward(*T, pe=pe, flags=pkg.FLAG_FORCE_GENERIC)
    assert torch.isfinite(want).all()
    # (fp32: 1e-7 each; bf16: both round results that close once)
    torch.testing.assert_close(got, want, rtol=1e-5 if dtype == torch.float32 else 2.0 ** -7, atol=MAX_ABS)


@pytest.mark.parametrize("pe", [ol.PE_NONE, ol.PE_SINUSOIDAL])
@pytest.mark.parametrize("H,Lq,Lk,D,n,launches", [
    (4, 64, 64, 512, 5, (2, 2)),       # five, and the one that reads an output of theirs
    (1, 16, 64, 64, 17, (2, 2)),       # 9 + 9; encoded 16 + 2
    (1, 33, 64, 256, 16, (2, 2)),      # 9 + 8; 16 + 1
    (30, 33, 20, 1000, 6, (7, 3)),     # 4 + 3 would leave SMs out, the overlapping calls are faster; 4 + 2 + 1
    (60, 16, 16, 256, 2, (3, 2)),      # 2 + 1 the same
    (148, 8, 8, 64, 2, (3, 3))])       # a head per SM
def test_one_launch_for_several_problems(pkg, cuda, pe, H, Lq, Lk, D, n, launches):
    """Equal entries of a batch share launches; an entry that reads an earlier one's output still sees it."""
    if torch.cuda.get_device_properties(cuda).multi_processor_count != 148:
        pytest.skip("the groups are those of 148 SMs")
    probs, args = [], []
    for i in range(n):
        Q, K, V = ol.make_qkv(1, H, Lq, Lk, D, 100 + i, "uniform")
        q, k, v = (to_dev(x, cuda) for x in (Q, K, V))
        probs.append((Q, K, V, q, k, v, torch.full_like(q, float("nan"))))
        args.append(pkg.args_for(q, k, v, probs[-1][-1], pe=pe, flags=pkg.FLAG_ASYNC))
    o2 = torch.full_like(probs[0][3], float("nan"))
    args.append(pkg.args_for(probs[1][-1], probs[0][4], probs[0][5], o2, pe=pe, flags=pkg.FLAG_ASYNC))
    pkg.forward(*probs[0][3:6], pe=pe)   # (builds the table of angles)
    n0 = pkg.launch_count()
    for _ in range(2):
        pkg.forward_many(args)
    torch.cuda.synchronize()
    assert pkg.launch_count() - n0 == 2 * launches[pe != ol.PE_NONE]
    if H < 30:
        pkg.forward_many(args[:2])
        assert pkg.last_path() == "splitd_stream"
    torch.cuda.synchronize()
    for Q, K, V, _, _, _, o in probs:
        res = ol.compare(o.cpu().numpy(), ol.attention(Q, K, V, pe=pe))
        assert res["ok"] and res["max_abs"] <= 5e-5, res
    assert ol.compare(o2.cpu().numpy(), ol.attention(probs[1][-1].cpu().numpy(), probs[0][1], probs[0][2], pe=pe))["ok"]


@pytest.mark.parametrize("replays", [0, 1, 12])
def test_captured_calls(pkg, cuda, replays):
    """Calls captured into a graph, which is then launched never, once or often, do not get in the way of other calls: of this kernel, of a
    batch and of the kernel whose scratch is a ring (fp32, no encoding)."""
    Q, K, V = ol.make_qkv(1, 4, 64, 50, 256, 96, "uniform")
    T = [to_dev(x, cuda) for x in (Q, K, V)]
    out, s = torch.empty_like(T[0]), torch.cuda.Stream()
    want = {pe: ol.attention(Q, K, V, pe=pe) for pe in (ol.PE_NONE, ol.PE_ROPE_INTERLEAVED)}
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        pkg.forward(*T, out=out, pe=ol.PE_ROPE_INTERLEAVED)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            for _ in range(10):
                pkg.forward(*T, out=out, pe=ol.PE_ROPE_INTERLEAVED, flags=pkg.FLAG_ASYNC)
        assert pkg.last_path() == "splitd_stream"
        for rep in range(max(1, replays)):
            if replays:
                out.zero_()
                g.replay()
                s.synchronize()
                assert ol.compare(out.cpu().numpy(), want[ol.PE_ROPE_INTERLEAVED])["max_abs"] <= 5e-5
            for pe in (ol.PE_ROPE_INTERLEAVED, ol.PE_NONE):
                o = [torch.zeros_like(out) for _ in range(5)]
                pkg.forward_many([pkg.args_for(*T, x, pe=pe, stream=s.cuda_stream, flags=pkg.FLAG_ASYNC) for x in o])
                # one entry at a time: each of another length of query, so that none share a launch
                lone = [pkg.forward(T[0][:, :, :n].contiguous(), T[1], T[2], pe=pe, flags=pkg.FLAG_ASYNC) for n in range(55, 64)]
                s.synchronize()
                for x, w in [(x, want[pe]) for x in o] + [(x, want[pe][:, :, :x.shape[2]]) for x in lone]:
                    assert ol.compare(x.cpu().numpy(), w)["max_abs"] <= 5e-5
    pkg.forward(*T)   # reports what an asynchronous call left behind


def test_slices_wait_for_room_beside_another_stream(pkg, cuda):
    """Another stream's kernel holds most of the SMs for many times as long as a slice waits for slices that run: the call takes until
    there is room, and succeeds.  A slice that never arrives is still reported, and the next call works."""
    Q, K, V = ol.make_qkv(1, 4, 64, 64, 1024, 97, "uniform")
    T = [to_dev(x, cuda) for x in (Q, K, V)]
    want = ol.attention(Q, K, V, pe=ol.PE_ROPE_INTERLEAVED)
    pkg.forward(*T, pe=ol.PE_ROPE_INTERLEAVED)
    x = torch.rand(100, 1 << 22, device=cuda)   # such a scan runs one block per row
    x.logcumsumexp(1)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    L = pkg.lib()
    pkg.set_option(pkg.OPT_SPIN_LIMIT, 1000)    # a millisecond of polls or so
    try:
        with torch.cuda.stream(side):
            x.logcumsumexp(1)
        got = pkg.forward(*T, pe=ol.PE_ROPE_INTERLEAVED)   # raises where a wait runs out
        assert pkg.last_path() == "splitd_stream"
        torch.cuda.synchronize()
        assert ol.compare(got.cpu().numpy(), want)["max_abs"] <= 5e-5
        L.b200attn_debug_lost_arrival(1, 20000)
        with pytest.raises(pkg.B200AttnError) as ei:
            pkg.forward(*T, pe=ol.PE_ROPE_INTERLEAVED)
        assert ei.value.status == 4   # B200ATTN_ERR_KERNEL
    finally:
        L.b200attn_debug_lost_arrival(0, 0)
        pkg.set_option(pkg.OPT_SPIN_LIMIT, 1 << 21)
        torch.cuda.synchronize()
    for _ in range(2):
        assert ol.compare(pkg.forward(*T, pe=ol.PE_ROPE_INTERLEAVED).cpu().numpy(), want)["max_abs"] <= 5e-5


def test_more_encodings_than_are_kept(pkg, cuda):
    """The tables of angles: a captured call's own stays where it is whatever comes after it, an encoding beyond the last table and one
    first met under capture run without."""
    Q, K, V = ol.make_qkv(1, 2, 20, 30, 64, 98, "uniform")
    T = [to_dev(x, cuda) for x in (Q, K, V)]
    pe, bases = ol.PE_ROPE_INTERLEAVED, [1000.0 + i for i in range(1100)]
    wants = {b: ol.attention(Q, K, V, pe=pe, base=b) for b in (bases[0], bases[1], bases[-1], 77.0)}
    out, out77, s = torch.empty_like(T[0]), torch.empty_like(T[0]), torch.cuda.Stream()

    def check(o, b):
        assert ol.compare(o.cpu().numpy(), wants[b])["max_abs"] <= 5e-5
    pkg.lib().b200attn_release_workspace()
    torch.cuda.synchronize()
    try:
        with torch.cuda.stream(s):
            pkg.forward(*T, out=out, pe=pe, rope_base=bases[0])
            assert pkg.last_path() == "splitd_stream"
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                pkg.forward(*T, out=out, pe=pe, rope_base=bases[0], flags=pkg.FLAG_ASYNC)
                assert pkg.last_path() == "splitd_stream"
                pkg.forward(*T, out=out77, pe=pe, rope_base=77.0, flags=pkg.FLAG_ASYNC)
                assert pkg.last_path() == "splitd_fused"
            for b in bases:
                last = pkg.forward(*T, pe=pe, rope_base=b, flags=pkg.FLAG_ASYNC)
            assert pkg.last_path() == "splitd_fused"
            check(last, bases[-1])
            check(pkg.forward(*T, pe=pe, rope_base=bases[1]), bases[1])
            assert pkg.last_path() == "splitd_stream"
            out.zero_()
            g.replay()
            s.synchronize()
            check(out, bases[0])
            check(out77, 77.0)
            del g
    finally:
        torch.cuda.synchronize()
        pkg.lib().b200attn_release_workspace()
