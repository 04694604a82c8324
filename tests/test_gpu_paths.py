"""GPU tests of kernel variants and dispatch rules at the sizes where they can go wrong: tile edges, remainders, the ends of their ranges.  Results are
compared with a plain PyTorch computation of the same operation on the same (dequantised) weights, or with the CPU oracle."""
import numpy as np
import pytest

import koifish_b200 as kf
import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = kf.Context(0)
    yield c
    c.close()


def bf16_tensor(dev, *shape):
    import torch
    return torch.from_numpy(dev.numpy(np.uint16).astype(np.int32)).to(torch.int16).view(torch.bfloat16)[:int(np.prod(shape))].view(*shape).cuda()


def make_q(ctx, typ, rows, cols, seed=5):
    """a weight quantised on the device and its dequantised values as fp32"""
    mode = kf.KF_Q_YYANG if typ in (kf.KF_T_SIGN, kf.KF_T_BINARY) else kf.KF_Q_RTN_ASYM
    w = kf.quantize(ctx, kf.fill_normal(ctx, rows * cols, seed, 0.02), rows, cols, typ, 128, mode)
    return w, bf16_tensor(kf.dequant(ctx, w), rows, cols).float()


# ---------------------------------------------------------------------------------------------- long reductions in the tcgen05 matmul
@pytest.mark.parametrize("rows,cols,M", [(5120, 8192, 2048), (10240, 25600, 45), (2560, 25600, 128)])
def test_tc_long_reduction(ctx, rows, cols, M):
    """Items of 32 and more raw stages: a stage that is handed back before its bytes were read shows as whole rows that used another stage's weights.
    The weights are exact on both sides, so what is left is the order of fp32 sums: 2^-24 * sqrt(cols) of the result, far below 1e-4; a stage that went
    wrong moves a row by 0.1 of it."""
    import torch
    torch.backends.cuda.matmul.allow_tf32 = False
    w, wd = make_q(ctx, kf.KF_T_Q4, rows, cols)
    x = kf.fill_normal(ctx, M * cols, 7, 1.0)
    want = bf16_tensor(x, M, cols).float() @ wd.T
    exact = ctx.get_int("gemv_exact")
    ctx.set_int("gemv_exact", 1)
    try:
        for _ in range(4):
            y = torch.from_numpy(kf.linear(ctx, w, x, M, kf.KF_EPI_F32).numpy(np.float32, (M, rows))).cuda()
            worst = ((y - want).square().mean(0).sqrt() / want.square().mean().sqrt()).max()
            assert float(worst) < 1e-4, float(worst)
    finally:
        ctx.set_int("gemv_exact", exact)
