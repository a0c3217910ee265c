"""GPU parity of the one-kernel tensor-core path for narrow heads (head_d 64, 128, 192 or 256, bf16 / fp16,
more than 64 queries): scores and the output accumulator stay in tensor memory, online softmax with a lazily
rescaled accumulator.  Oracle: fp32 CPU attention on the 16-bit-rounded inputs; tolerance max-abs 2e-2 (bf16)."""
import numpy as np
import pytest

import oracle_lib as ol
from gpu_util import bf16_from_dev, bf16_problem, bf16_to_dev

pytestmark = pytest.mark.gpu
TOL = 2e-2

SHAPES = [
    (1, 1, 128, 128, 128),      # one tile of each
    (1, 2, 256, 256, 128),      # one unit: two query tiles
    (1, 2, 256, 384, 64),
    (2, 3, 512, 1024, 128),     # several units per head, eight key tiles
    (1, 150, 256, 256, 64),     # more units than SMs: CTAs take several
    (1, 2, 384, 640, 128),      # an odd number of query tiles: the second tile of the last unit is empty
    (1, 200, 384, 384, 128),    # ... with more units than SMs: a CTA meets empty and full second tiles in turn
    (2, 160, 128, 256, 64),     # ... every unit with an empty second tile
    (2, 3, 200, 300, 128),      # ragged in both lengths
    (1, 2, 129, 257, 64),
    (1, 3, 700, 1000, 128),
    (1, 1, 65, 4100, 128),      # 33 key tiles, the last with 4 keys
    (1, 2, 300, 40, 64),        # fewer keys than a tile
    (1, 1, 2048, 2048, 128),
    # head_d 256: one query tile per unit, two score buffers
    (1, 1, 128, 128, 256),
    (1, 2, 256, 256, 256),      # two full key tiles: the epilogue may be a tile ahead of the last P V product
    (1, 2, 256, 384, 256),
    (1, 150, 128, 128, 256),    # more units than SMs
    (2, 3, 200, 300, 256),
    (1, 3, 700, 1000, 256),
    (1, 1, 65, 4100, 256),
    (1, 2, 300, 40, 256),
    (1, 160, 256, 640, 256),    # several units per CTA with an odd number of key tiles: the score buffers swap roles from unit to unit
]


def run(pkg, cuda, bits, **kw):
    q, k, v = (bf16_to_dev(b, cuda) for b in bits)
    return bf16_from_dev(pkg.forward(q, k, v, **kw))


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_fused_path_against_oracle(pkg, cuda, shape):
    B, H, Lq, Lk, D = shape
    bits, up = bf16_problem(B, H, Lq, Lk, D, 91, "normal")
    want = ol.attention(*up)
    got = run(pkg, cuda, bits)
    assert pkg.last_path() == "tc_fused", pkg.last_path()
    err = float(np.abs(got - want).max())
    assert err <= TOL, (shape, err)
    assert err <= 8e-3, (shape, err)   # observed 3e-4 ... 4e-3 (the rounding of P and of the result to bf16)


def test_fused_path_agrees_with_the_two_kernel_path(pkg, cuda):
    bits, up = bf16_problem(2, 4, 640, 896, 128, 92, "normal")
    a = run(pkg, cuda, bits)
    assert pkg.last_path() == "tc_fused"
    b = run(pkg, cuda, bits, flags=pkg.FLAG_TWO_KERNELS)
    assert pkg.last_path() == "tc_wide"
    assert float(np.abs(a - b).max()) <= 8e-3


def test_fused_path_with_peaked_rows_rescales_its_accumulator(pkg, cuda):
    """Scores that keep growing along the keys (row maxima far apart from tile to tile) force the lazy rescale of
    the accumulator again and again; scores that shrink leave the first reference maximum in place."""
    B, H, Lq, Lk, D = 1, 2, 256, 1024, 128
    rng = np.random.default_rng(93)
    Q = rng.standard_normal((B, H, Lq, D)).astype(np.float32)
    K = rng.standard_normal((B, H, Lk, D)).astype(np.float32)
    V = rng.standard_normal((B, H, Lk, D)).astype(np.float32)
    ramp = np.linspace(0.0, 12.0, Lk, dtype=np.float32)[None, :, None]     # key j is aligned with every query, more and more strongly
    K[:, 0] = K[:, 0] * 0.2 + ramp * np.sign(Q[:, 0].mean(axis=1, keepdims=True))
    K[:, 1] = K[:, 1] * 0.2 + ramp[:, ::-1] * np.sign(Q[:, 1].mean(axis=1, keepdims=True))
    bits = tuple(ol.to_bf16_bits(x) for x in (Q, K, V))
    up = tuple(ol.from_bf16_bits(b) for b in bits)
    want = ol.attention(*up)
    got = run(pkg, cuda, bits)
    assert pkg.last_path() == "tc_fused"
    assert float(np.abs(got - want).max()) <= TOL


def test_fused_path_heads_do_not_see_their_neighbours(pkg, cuda):
    B, H, Lq, Lk, D = 1, 3, 200, 300, 128
    bits, up = bf16_problem(B, H, Lq, Lk, D, 94, "normal")
    want = ol.attention(*up)
    poisoned = [b.copy() for b in bits]
    for b, pat in zip(poisoned, (0x7FC0, 0x7F80, 0xFF80)):   # NaN in Q, +inf in K, -inf in V of head 1
        b[:, 1] = pat
    got = run(pkg, cuda, poisoned)
    assert pkg.last_path() == "tc_fused"
    for h in (0, 2):
        assert np.isfinite(got[:, h]).all(), h
        assert float(np.abs(got[:, h] - want[:, h]).max()) <= 8e-3, h


def test_fused_path_leaves_the_memory_behind_the_output_alone(pkg, cuda):
    import torch
    B, H, Lq, Lk, D = 1, 2, 130, 200, 64
    bits, up = bf16_problem(B, H, Lq, Lk, D, 95, "normal")
    q, k, v = (bf16_to_dev(b, cuda) for b in bits)
    big = torch.full((B * H * Lq * D + 254 * D,), 7.0, dtype=torch.bfloat16, device=cuda)
    out = big[: B * H * Lq * D].view(B, H, Lq, D)
    pkg.forward(q, k, v, out=out)
    assert pkg.last_path() == "tc_fused"
    assert bool((big[B * H * Lq * D:] == 7.0).all())
    assert float(np.abs(bf16_from_dev(out) - ol.attention(*up)).max()) <= 8e-3


def test_fused_path_twice_in_a_row_same_result(pkg, cuda):
    bits, up = bf16_problem(1, 4, 512, 768, 128, 96, "normal")
    a = run(pkg, cuda, bits)
    b = run(pkg, cuda, bits)
    assert np.array_equal(a, b)


@pytest.mark.parametrize("shape", [(2, 100, 384, 640, 128), (1, 160, 256, 1000, 64), (2, 90, 300, 900, 256)], ids=lambda s: "x".join(map(str, s)))
def test_fused_path_many_launches_bit_identical(pkg, cuda, shape):
    """Several units per CTA, empty second query tiles, ragged lengths: a hand-off that races shows up as a result
    that differs from launch to launch."""
    import torch
    B, H, Lq, Lk, D = shape
    g = torch.Generator(device="cpu").manual_seed(5)
    q, k, v = (torch.randn(B, H, L, D, generator=g).to(cuda).bfloat16() for L in (Lq, Lk, Lk))
    first = pkg.forward(q, k, v).clone()
    assert pkg.last_path() == "tc_fused"
    out = torch.empty_like(first)
    for _ in range(100):
        pkg.forward(q, k, v, out=out)
        assert torch.equal(out, first)


@pytest.mark.parametrize("shape", [(1, 2, 256, 384, 128), (2, 2, 200, 300, 64), (1, 2, 256, 384, 256)], ids=lambda s: "x".join(map(str, s)))
def test_fused_path_fp16(pkg, cuda, shape):
    import torch
    B, H, Lq, Lk, D = shape
    Q, K, V = ol.make_qkv(B, H, Lq, Lk, D, 97, "normal")
    q, k, v = (torch.from_numpy(x).to(cuda).half() for x in (Q, K, V))
    want = ol.attention(*(x.float().cpu().numpy() for x in (q, k, v)))
    got = pkg.forward(q, k, v).float().cpu().numpy()
    assert pkg.last_path() == "tc_fused"
    assert float(np.abs(got - want).max()) <= 2e-3   # fp16 keeps three more bits than bf16


PES = [ol.PE_ROPE_INTERLEAVED, ol.PE_ROPE_HALF, ol.PE_SINUSOIDAL, ol.PE_ROPE_Q_ONLY, ol.PE_ROPE_HALF_Q_ONLY]


@pytest.mark.parametrize("pe", PES, ids=["rope_pairs", "rope_half", "sinusoidal", "rope_q_only", "rope_half_q_only"])
@pytest.mark.parametrize("shape", [(1, 2, 256, 384, 128), (2, 2, 200, 300, 64), (1, 3, 129, 1000, 128), (1, 2, 200, 300, 256)], ids=lambda s: "x".join(map(str, s)))
def test_fused_path_with_encodings(pkg, cuda, pe, shape):
    """With an encoding the narrow-head path works on encoded copies of Q and K (fp32 arithmetic, one rounding)."""
    B, H, Lq, Lk, D = shape
    bits, up = bf16_problem(B, H, Lq, Lk, D, 98, "normal")
    q_only = pe in (ol.PE_ROPE_Q_ONLY, ol.PE_ROPE_HALF_Q_ONLY)
    half = pe in (ol.PE_ROPE_HALF, ol.PE_ROPE_HALF_Q_ONLY)
    if q_only:   # the caller keeps K rotated: give the library the rotated K, the oracle the plain one
        kr = ol.from_bf16_bits(ol.to_bf16_bits(ol.apply_rope(up[1], half=half)))
        want = ol.attention(ol.apply_rope(up[0], half=half), kr, up[2])
        bits = (bits[0], ol.to_bf16_bits(kr), bits[2])
    else:
        want = ol.attention(*up, pe=pe)
    got = run(pkg, cuda, bits, pe=pe)
    assert pkg.last_path() == "tc_fused", pkg.last_path()
    err = float(np.abs(got - want).max())
    assert err <= TOL, (shape, pe, err)
    assert err <= 1.2e-2, (shape, pe, err)


def test_fused_path_partial_rotary_dim_and_caller_caches(pkg, cuda):
    from gpu_util import to_dev
    B, H, Lq, Lk, D, rd = 1, 2, 256, 512, 128, 64
    bits, up = bf16_problem(B, H, Lq, Lk, D, 99, "normal")
    for pe in (ol.PE_ROPE_INTERLEAVED, ol.PE_ROPE_HALF):
        want = ol.attention(*up, pe=pe, rotary_dim=rd)
        got = run(pkg, cuda, bits, pe=pe, rotary_dim=rd)
        assert pkg.last_path() == "tc_fused"
        assert float(np.abs(got - want).max()) <= 1.2e-2, pe
    base = 500.0
    c, s = ol.rope_cache(max(Lq, Lk), D, base)
    want = ol.attention(*up, pe=ol.PE_ROPE_INTERLEAVED, base=base)
    q, k, v = (bf16_to_dev(b, cuda) for b in bits)
    got = bf16_from_dev(pkg.forward(q, k, v, pe=ol.PE_ROPE_INTERLEAVED, cos_cache=to_dev(c, cuda), sin_cache=to_dev(s, cuda)))
    assert pkg.last_path() == "tc_fused"
    assert float(np.abs(got - want).max()) <= 1.2e-2


def test_fused_path_fp16_with_an_encoding(pkg, cuda):
    import torch
    B, H, Lq, Lk, D = 1, 2, 256, 384, 128
    Q, K, V = ol.make_qkv(B, H, Lq, Lk, D, 100, "normal")
    q, k, v = (torch.from_numpy(x).to(cuda).half() for x in (Q, K, V))
    up = tuple(x.float().cpu().numpy() for x in (q, k, v))
    for pe in (ol.PE_ROPE_HALF, ol.PE_SINUSOIDAL):
        got = pkg.forward(q, k, v, pe=pe).float().cpu().numpy()
        assert pkg.last_path() == "tc_fused"
        assert float(np.abs(got - ol.attention(*up, pe=pe)).max()) <= 4e-3, pe


def test_fused_path_very_long_keys(pkg, cuda):
    """157 key tiles, the last with 32 keys (the kernel has no limit on len_k)."""
    B, H, Lq, Lk, D = 1, 1, 128, 20000, 64
    bits, up = bf16_problem(B, H, Lq, Lk, D, 101, "normal")
    got = run(pkg, cuda, bits)
    assert pkg.last_path() == "tc_fused"
    assert float(np.abs(got - ol.attention(*up)).max()) <= 8e-3


@pytest.mark.parametrize("D", [8, 40, 72, 80, 96, 104, 136, 160, 192, 200, 248])
@pytest.mark.parametrize("lens", [(130, 300), (300, 129), (3, 200)], ids=str)
def test_widths_between_the_column_groups(pkg, cuda, D, lens):
    """Any multiple of 8 below 256: the operands are exact, encoded operands, scores, probabilities and sums fp32, and only the
    result is rounded to 16 bits (head_d 192 without an encoding: P rounded too, as at 64, 128 and 256).  Nothing behind the
    output is written."""
    import torch
    (Lq, Lk), B, H = lens, 1, 3
    bits, up = bf16_problem(B, H, Lq, Lk, D, 100 + D, "normal")
    q, k, v = (bf16_to_dev(b, cuda) for b in bits)
    path = ("tc_wide" if Lq <= 64 else "tc_fused") if D == 192 else "tc_f32"
    for dtype, half_ulp in ((torch.bfloat16, 2.0 ** -8), (torch.float16, 2.0 ** -11)):   # relative, at most
        tq, tk, tv = (t.to(dtype) for t in (q, k, v))
        big = torch.full((B * H * Lq * D + 256,), 3.0, dtype=dtype, device=cuda)
        out = big[:B * H * Lq * D].view(B, H, Lq, D)
        for pe in (pkg.PE_NONE, pkg.PE_ROPE_INTERLEAVED, pkg.PE_ROPE_HALF, pkg.PE_SINUSOIDAL):
            if D == 192 and pe != pkg.PE_NONE and (Lq <= 64 or dtype == torch.float16):
                continue   # other kernels, other tests
            pkg.forward(tq, tk, tv, out=out, pe=pe)
            assert pkg.last_path() == ("tc_f32" if pe != pkg.PE_NONE else path), (pkg.last_path(), pe)
            assert bool((big[B * H * Lq * D:] == 3.0).all())
            want = ol.attention(*(t.float().cpu().numpy() for t in (tq, tk, tv)), pe=pe)
            err = np.abs(out.float().cpu().numpy() - want)
            if pkg.last_path() == "tc_f32":
                # half a unit in the last place of the result, and fp32: sums to 1e-5, angles up to 300 and their functions to a few
                # ulp, which enter a score of normal values (up to 16 or so) with the weights of head_d / 2 pairs
                assert (err <= np.abs(want) * half_ulp + (1e-5 if pe == pkg.PE_NONE else 1e-3)).all(), (dtype, pe, err.max())
            else:
                assert err.max() <= (8e-3 if dtype == torch.bfloat16 else 4e-3), (dtype, pe, err.max())   # the bounds of the whole widths


@pytest.mark.parametrize("which", [0, 1, 2])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("f16", [False, True])
@pytest.mark.parametrize("pe", ["none", "rope"])
def test_non_finite_values_at_other_widths(pkg, cuda, which, value, f16, pe):
    """As on the CUDA cores, which took these widths before (a key or row that is not finite, not only an element)."""
    import torch
    dtype, kind = torch.float16 if f16 else torch.bfloat16, pkg.PE_NONE if pe == "none" else pkg.PE_ROPE_INTERLEAVED
    T = [torch.randn(1, 2, 150, 72, generator=torch.Generator().manual_seed(5 + i)).to(dtype).to(cuda) for i in range(3)]
    T[which][0, 1, 7, 5] = value
    T[which][0, 0, 140] = value
    got = pkg.forward(*T, pe=kind)
    assert pkg.last_path() == "tc_f32"
    want = pkg.forward(*T, pe=kind, flags=pkg.FLAG_FORCE_GENERIC)
    assert pkg.last_path() == "splitd_two_pass"
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
