"""The attention kernels at the edges of their tiles, work items and routes: 128-row and 128-column tiles, pairs of q
tiles, groups of query rows that the decoding kernel takes, kv tiles that few queries see, and scores whose maximum keeps
growing (the accumulator's rescaling).  The oracle is the softmax in float64."""
import math

import pytest
import torch

import genesis_b200  # noqa: F401
from genesis_b200.ops import native as N

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(B, S, Sk, Hq, Hkv, D, dt, ramp=0.0):
    g = torch.Generator(device=DEV).manual_seed(B + 3 * S + 5 * Sk + 7 * Hq + D)
    q = torch.randn(B, S, Hq, D, device=DEV, generator=g)
    k = torch.randn(B, Sk, Hkv, D, device=DEV, generator=g)
    v = torch.randn(B, Sk, Hkv, D, device=DEV, generator=g)
    if ramp:
        # one shared component of q and k makes the scores climb by `ramp` (natural log) over the keys
        q[..., 0] = math.sqrt(D)
        k[..., 0] = torch.linspace(0, ramp, Sk, device=DEV)[None, :, None]
    return q.to(dt), k.to(dt), v.to(dt)


def _oracle(q, k, v, causal, scale):
    """o, lse and P |v| in float64, laid out as the kernel's."""
    B, S, Hq, D = q.shape
    Sk, g = k.shape[1], Hq // k.shape[2]
    qd, kd, vd = (t.double().transpose(1, 2) for t in (q, k.repeat_interleave(g, 2), v.repeat_interleave(g, 2)))
    s = qd @ kd.transpose(-1, -2) * scale
    if causal:
        s = s.masked_fill(torch.ones(S, Sk, dtype=torch.bool, device=DEV).triu(Sk - S + 1), -math.inf)
    p = torch.softmax(s, -1)
    return (p @ vd).transpose(1, 2), torch.logsumexp(s, -1), (p @ vd.abs()).transpose(1, 2)


def _check_fwd(q, k, v, causal):
    D, dt = q.shape[-1], q.dtype
    scale = D ** -0.5
    r = N.attention_fwd(q, k, v, causal, scale)
    assert r is not NotImplemented
    o, lse = r
    N.check_status()
    ref, lref, pv = _oracle(q, k, v, causal, scale)
    # every probability and the result are rounded once to 16 bits: with p significand bits the relative error of a
    # rounding is at most 2^-p (8 bits: 2^-8 for bf16, 11 bits: 2^-11 for fp16); fp32 exponents of size x carry
    # |x| 2^-23, which 2^-16 covers up to |x| = 2^7; fp16 probabilities below 2^-14 are rounded to multiples of 2^-24
    u = 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11
    tiny = 0.0 if dt == torch.bfloat16 else 2.0 ** -25 * k.shape[1] * float(v.abs().max())
    bound = (u + 2.0 ** -16) * (pv + ref.abs()) + tiny + 1e-6
    assert bool(((o.double() - ref).abs() <= bound).all()), float(((o.double() - ref).abs() / bound).max())
    assert float((lse.double() - lref).abs().max()) <= 2e-5 * max(1.0, float(lref.abs().max()))
    return o, lse, scale


FWD = [
    # B, S, Sk, Hq, Hkv, D: one tile and its neighbours, one row more than a pair, ragged keys, enough work for pairs
    (1, 127, 127, 2, 1, 64), (1, 129, 129, 9, 3, 64), (1, 255, 300, 2, 2, 128), (2, 257, 257, 4, 2, 128),
    (1, 385, 1000, 14, 2, 64), (3, 640, 640, 40, 8, 64), (2, 513, 513, 80, 16, 128), (40, 130, 131, 4, 4, 64),
    # pairs of q tiles that save a round, and an odd tile among them
    (48, 200, 200, 2, 2, 64), (13, 300, 300, 8, 4, 128),
    # up to 64 query rows of a group: estimates choose between the decoding kernel (one query, a full 16-row tile, several
    # tiles of one head, keys shared by CTAs of a cluster) ...
    (1, 1, 1, 1, 1, 64), (2, 1, 17, 8, 1, 128), (3, 2, 1030, 16, 2, 64), (2, 5, 4099, 12, 2, 128), (9, 1, 513, 32, 4, 128),
    (1, 4, 333, 64, 4, 64), (1, 17, 300, 1, 1, 128), (1, 64, 300, 2, 2, 64), (2, 64, 1000, 4, 4, 128), (1, 33, 2050, 1, 1, 64),
    # ... and the tiled one (few keys, many heads), which takes everything from 65 rows on
    (1, 17, 100, 1, 1, 128), (1, 64, 64, 2, 2, 64), (2, 16, 128, 4, 4, 128), (64, 16, 200, 4, 4, 128), (1, 65, 65, 2, 2, 64),
    (1, 65, 300, 2, 2, 64), (2, 22, 300, 6, 2, 128),
]


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("case", FWD)
@pytest.mark.parametrize("causal", [True, False])
def test_forward_at_tile_edges(case, dt, causal):
    _check_fwd(*_inputs(*case, dt), causal)


@pytest.mark.parametrize("shape", [(1, 700, 700, 2, 1, 64), (1, 300, 900, 2, 2, 128), (2, 1, 2000, 8, 2, 64), (1, 3, 700, 4, 4, 128)])
@pytest.mark.parametrize("ramp", [60.0, -60.0])
def test_forward_with_growing_scores(shape, ramp):
    _check_fwd(*_inputs(*shape, torch.bfloat16, ramp=ramp), True)


@pytest.mark.parametrize("S,Sk", [(1, 512), (200, 512), (300, 1000)])       # decoding, unmasked tiles only, a ragged last tile
@pytest.mark.parametrize("D", [64, 128])
def test_forward_with_scores_of_minus_infinity(S, Sk, D):
    """Overflowed products: a row whose scores are all -inf is empty (output 0, lse -inf) on every route; in the other rows a
    key whose score is -inf has probability exactly 0, whatever its value."""
    q, k, v = _inputs(2, S, Sk, 4, 2, D, torch.bfloat16)
    q[..., 0], k[..., 0] = 0.0, -1e30
    q[0, S // 2, :, :], k[0, :Sk // 3, 0, 1], v[0, :Sk // 3, 0] = 0.0, -1e30, 3e38
    q[0, S // 2, :, 0] = 1e30                        # 1e30 * -1e30: all scores of this row
    q[..., 1] = q[..., 1].abs() + 1e10               # 1e10 * -1e30: the first third of its keys, for the first group
    q[0, S // 2, :, 1] = 0.0
    k[0, Sk // 3:, 0, 1] = k[1, :, :, 1] = k[:, :, 1, 1] = 0.0
    r = N.attention_fwd(q, k, v, False, D ** -0.5)
    N.check_status()
    o, lse = r
    assert bool((o[0, S // 2] == 0).all()) and bool((lse[0, :, S // 2] == -math.inf).all())
    if S > 1:
        live = torch.ones(S, dtype=torch.bool, device=DEV)
        live[S // 2] = False
        vz = v.clone()
        vz[0, :Sk // 3, 0] = 0                       # what 0 * v leaves
        ref, lref, pv = _oracle(q, k, vz, False, D ** -0.5)
        bound = (2.0 ** -8 + 2.0 ** -16) * (pv + ref.abs()) + 1e-6          # as in _check_fwd
        assert bool(((o.double() - ref).abs() <= bound)[:, live].all())
        assert float((lse.double() - lref)[..., live].abs().max()) <= 2e-5 * float(lref[..., live].abs().max())


BWD = [
    (1, 127, 127, 2, 1, 64), (1, 129, 130, 4, 2, 128), (2, 256, 256, 6, 3, 64), (1, 385, 500, 14, 2, 64),
    (1, 40, 700, 4, 1, 128), (4, 520, 520, 12, 2, 128), (8, 650, 650, 14, 2, 64), (2, 384, 384, 5, 5, 128),
    (1, 1, 1, 2, 1, 64), (1, 3, 260, 6, 2, 128),
    # half tiles: rows that fit one and the first that do not, grids on both sides of one and two CTAs for every SM, groups
    # that are split or not, keys that few queries see
    (1, 64, 64, 2, 2, 128), (1, 65, 65, 2, 2, 128), (3, 50, 200, 4, 2, 128), (8, 16, 216, 16, 8, 64), (150, 16, 16, 2, 1, 64),
    (10, 129, 129, 8, 8, 64), (9, 129, 192, 8, 8, 64), (40, 130, 130, 8, 8, 64), (19, 300, 700, 8, 8, 64), (30, 193, 193, 14, 2, 64),
]


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("case", BWD)
@pytest.mark.parametrize("causal", [True, False])
def test_backward_at_tile_edges(case, dt, causal):
    q, k, v = _inputs(*case, dt)
    o, lse, scale = _check_fwd(q, k, v, causal)
    do = torch.randn(q.shape, device=DEV, generator=torch.Generator(device=DEV).manual_seed(1)).to(dt)
    r = N.attention_bwd(do, q, k, v, o, lse, causal, scale)
    assert r is not NotImplemented
    N.check_status()
    leaves = [t.double().requires_grad_() for t in (q, k, v)]
    _oracle(*leaves, causal, scale)[0].backward(do.double())
    # P and dS are rounded once to 16 bits, delta carries the rounding of o, the result is rounded once: four independent
    # roundings of relative error up to u (2^-8 or 2^-11, as above), u / sqrt(3) in the norm each, so 2 u; the floor is what fp32 leaves of dP - delta where
    # the two cancel (D products of up to 20 at 2^-24 each, over a few hundred elements)
    u = 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11
    for got, ref in zip(r, leaves):
        ref = ref.grad
        assert float((got.double() - ref).norm()) <= 2 * u * float(ref.norm()) + 1e-3
        assert bool(torch.isfinite(got).all())
