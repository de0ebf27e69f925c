"""Row kernels at the edges of their routes: RMSNorm rows that stream through the ring (row lengths from the first past
the warp-per-row kernel to the longest, row counts around the ring's turn), the mixture-of-experts row sums, stacked
parameter conversions, and products with a long contraction."""
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


@pytest.mark.parametrize("T,k,E,cols", [(1, 1, 2, 8), (37, 2, 8, 136), (300, 8, 16, 2048), (129, 8, 128, 256), (64, 3, 5, 20)])
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
