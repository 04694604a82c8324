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


# ---------------------------------------------------------------------------------------------- sampler: one pass over the row by a cluster of CTAs
def _rows(kind, M, vocab, rng):
    if kind == "normal":
        v = rng.standard_normal((M, vocab)) * 2.5
    elif kind == "ties":  # a handful of values: the threshold falls into a long run of equal logits, lists overflow at the larger sizes
        v = rng.integers(-3, 3, (M, vocab)).astype(np.float32)
    elif kind == "zeros":  # the two zeros are one value, ordered by index
        v = np.where(rng.random((M, vocab)) < 0.5, 0.0, -0.0)
        v[:, ::7] = -1.0
    elif kind == "few":  # the chosen ones sit side by side, the rest far below: infinities and the lowest value among it
        v = np.full((M, vocab), -np.inf)
        v[:, 1::3] = -3.3e38
        v[:, 40:400] = rng.standard_normal((M, 360))
    else:  # descending: the largest all in one thread block's part
        v = np.tile(-np.arange(vocab, dtype=np.float64) / 64, (M, 1))
    return ol.f32_to_bf16(v.astype(np.float32))


@pytest.mark.parametrize("vocab,top_k", [(1000, 200), (1001, 2), (16384, 50), (16385, 256), (32768, 255), (49151, 50), (65544, 20), (151936, 50), (196608, 256),
                                         (196609, 256), (151936, 257)])
@pytest.mark.parametrize("kind", ["normal", "ties", "zeros", "few", "falling"])
def test_sample_selection(ctx, kind, vocab, top_k):
    """Tokens equal those of the CPU port (which shares no code): a high temperature makes every candidate as likely, so the token names a place in the sorted
    list of candidates.  1 draw in 100 may differ (a coin within rounding of a boundary: the two exponentials differ in the last place)."""
    M, rounds = 3, 12
    rng = np.random.default_rng(vocab + top_k)
    lg = _rows(kind, M, vocab, rng).reshape(M, vocab)
    lgd = ctx.array(lg)
    for T, top_p in ((1e4, 1.0), (0.8, 0.9)):
        seeds = rng.integers(1, 2 ** 62, M).astype(np.uint64)
        std, states, diff = ctx.array(seeds.view(np.uint16)), [[int(s)] for s in seeds], 0
        for _ in range(rounds):
            got = kf.sample(ctx, lgd, M, vocab, T, top_k, top_p, std, 0).numpy(np.int32)
            for m in range(M):
                diff += int(got[m] != ol.sample(lg[m], T, top_k, top_p, states[m], 0)[0])
        assert diff <= 1, (T, diff)
        assert np.array_equal(std.numpy(np.uint64), np.array([s[0] for s in states], dtype=np.uint64))
