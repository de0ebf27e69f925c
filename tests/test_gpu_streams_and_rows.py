"""Row kernels at the edges of their routes: RMSNorm rows on both sides of the line to the kernels that stream rows through a
ring (row lengths, row counts and total sizes, which differ forward, backward and with the type), cross-entropy rows, the mixture-of-experts row
sums, stacked parameter conversions, and products with a long contraction."""
import pytest
import torch

import genesis_b200  # noqa: F401
from genesis_b200.ops import dispatch as K
from genesis_b200.ops import native as N

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rnd(*shape, dt=torch.float32, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed + sum(shape))
    return torch.randn(*shape, device=DEV, generator=g).to(dt)


# largest relative error of one rounding: 2^-8 with bf16's 8 significand bits, 2^-11 with fp16's 11; fp32 results end a
# chain of a few operations
ROUND = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -22}


@pytest.mark.parametrize("rows,cols", [(1183, 1032), (1184, 1032), (1185, 1536), (1500, 2056), (1777, 4096), (1300, 8192),
                                       (1200, 4104), (1184, 512), (2197, 4096), (2198, 4096), (1184, 2056), (6250, 1280),
                                       (6249, 1280)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32])
def test_wide_rmsnorm(rows, cols, dt):
    x, res, g, gres = (_rnd(rows, cols, dt=dt, seed=i) for i in range(4))
    w = _rnd(cols, seed=9)
    s, y, rstd = N.add_rmsnorm_fwd(x, res, w, 1e-6)
    N.check_status()
    sd = (x.double() + res.double()).to(dt).double() if dt != torch.float32 else s.double()
    assert torch.equal(s.double(), sd)
    r = torch.rsqrt(sd.square().mean(-1, keepdim=True) + 1e-6)
    ref = sd * r * w.double()
    # one rounding of the result; the fp32 sum of `cols` squares is good to 2^-18
    assert bool(((y.double() - ref).abs() <= (ROUND[dt] + 2.0 ** -18) * ref.abs() + 1e-7).all())
    for extra in (None, gres):
        dx, dw = N.rmsnorm_bwd(g, s, w, rstd) if extra is None else N.add_rmsnorm_bwd(g, extra, s, w, rstd)
        N.check_status()
        xh, gw = sd * r, g.double() * w.double()
        want = r * (gw - xh * (gw * xh).mean(-1, keepdim=True)) + (0 if extra is None else extra.double())
        size = r * gw.abs() + want.abs() + r * xh.abs()
        assert bool(((dx.double() - want).abs() <= ROUND[dt] * want.abs() + 2.0 ** -17 * size + 1e-7).all())
        dref = (g.double() * xh).sum(0)
        assert float((dw.double() - dref).norm()) <= 1e-5 * float(dref.norm())
        again = N.rmsnorm_bwd(g, s, w, rstd) if extra is None else N.add_rmsnorm_bwd(g, extra, s, w, rstd)
        assert torch.equal(dx, again[0]) and torch.equal(dw, again[1])


@pytest.mark.parametrize("cols", [8, 1000, 4096, 5120 - 8, 5120, 5121, 8192 - 8, 32771, 65536 - 8, 65536, 65536 + 3, 151936])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32])
def test_cross_entropy_rows(cols, dt):
    x = _rnd(6, cols, dt=dt) * 4
    x[1] = -float("inf")                     # one finite entry among masked ones, at the end of the row
    x[1, -1] = 2.0
    x[2, 0] = 60.0                           # the maximum comes first
    x[3] = torch.finfo(dt).min               # all of them the lowest value
    x[5, cols // 2] = float("nan")
    t = torch.tensor([0, cols - 1, 0, cols // 2, -100, 0], device=DEV)
    loss, lse = N.cross_entropy_fwd(x, t, -100)
    ref = torch.logsumexp(x.double(), -1)
    # fp32 exponentials and sums of up to 151936 terms in runs of some hundreds: a few 2^-20 of a value of about 10
    assert bool(((lse.double() - ref).abs()[:5] <= 1e-5 * ref.abs()[:5].clamp_min(1)).all()) and bool(lse[5].isnan())
    pick = x.double()[torch.arange(6), t.clamp_min(0)]
    assert bool(((loss.double() - (ref - pick)).abs()[:4] <= 1e-5 * (ref.abs() + pick.abs())[:4].clamp_min(1)).all())
    assert float(loss[4]) == 0.0


@pytest.mark.parametrize("T,k,E,cols", [(1, 1, 2, 8), (37, 2, 8, 136), (300, 8, 16, 2048), (129, 8, 128, 256), (64, 3, 5, 20),
                                        (50, 4, 8, 64), (50, 4, 8, 72), (77, 2, 8, 128)])
def test_moe_row_sums(T, k, E, cols):
    g = torch.Generator(device=DEV).manual_seed(T)
    e = torch.rand(T, E, device=DEV, generator=g).topk(k, 1).indices.int().contiguous()
    token_of, pos, offsets = K.moe_sort(e, E)
    dt = torch.bfloat16
    y, gr = _rnd(token_of.numel(), cols, dt=dt), _rnd(T, cols, dt=dt, seed=1)
    w = torch.rand(T, k, device=DEV, generator=g)
    rows = y.double()[pos.long().reshape(-1)].reshape(T, k, cols)
    if cols % 8 == 0:
        out = K.moe_gather_sum(y, pos)
        assert bool(((out.double() - rows.sum(1)).abs() <= 2.0 ** -8 * rows.sum(1).abs() + 1e-5).all())
    for table in (None, token_of):
        dy, dw = K.moe_combine_bwd(gr, y, w, pos, table)
        want = torch.zeros_like(y, dtype=torch.float64)
        want[pos.long().reshape(-1)] = (gr.double()[:, None] * w.double()[..., None]).reshape(T * k, cols)
        assert bool(((dy.double() - want).abs() <= 2.0 ** -8 * want.abs()).all())
        dref = (rows * gr.double()[:, None]).sum(-1)
        assert bool(((dw.double() - dref).abs() <= 1e-4 * cols ** 0.5).all())


@pytest.mark.parametrize("shapes", [[(896, 896), (128, 896), (128, 896)], [(8,), (16,)], [(5, 24)] * 8, [(3, 5), (4, 5)],
                                    [(2, 8)] * 9, [(40000, 64), (1, 64)]])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_stacked_conversion(shapes, dt):
    ts = [_rnd(*s, seed=i) for i, s in enumerate(shapes)]
    assert torch.equal(K.cat_cast(ts, dt), torch.cat(ts).to(dt))
    # the same from a base that is not 16-byte aligned, and from parameters that already have the dtype
    un = [_rnd(t.numel() + 1)[1:].reshape(t.shape) for t in ts]
    assert torch.equal(K.cat_cast(un, dt), torch.cat(un).to(dt))
    low = [t.to(dt) for t in ts]
    assert torch.equal(K.cat_cast(low, dt), torch.cat(low))


@pytest.mark.parametrize("M,Nc,K", [(1, 8, 8192), (5, 64, 8192), (130, 264, 8960), (300, 896, 8192), (129, 40, 32000),
                                   (2048, 896, 30016), (64, 512, 8200)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_long_contractions(M, Nc, K, dt):
    """Products whose contraction may be cut into parts, in the layouts of a forward pass and of a data gradient."""
    a, b = _rnd(M, K, dt=dt), _rnd(Nc, K, dt=dt, seed=1)
    ref, size = a.double() @ b.double().t(), a.double().abs() @ b.double().abs().t()
    for got in (lambda: N.gemm(a, b), lambda: N.linear_dgrad(a, b.t().contiguous()), lambda: N.gemm(a.t().contiguous().t(), b)):
        out = got()
        N.check_status()
        # one rounding of the result; fp32 accumulation of K products in runs of 16: K / 16 roundings of 2^-24
        assert bool(((out.double() - ref).abs() <= ROUND[dt] * ref.abs() + K / 16 * 2.0 ** -24 * size + 1e-7).all())
        assert torch.equal(out, got())
