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


# ---------------------------------------------------------------------------------------------- one and two tokens on the integer tensor cores
@pytest.mark.parametrize("typ,bits", [(kf.KF_T_Q4, 4), (kf.KF_T_Q2, 2), (kf.KF_T_SIGN, 2), (kf.KF_T_BINARY, 1)])
@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("rows,cols", [(8192, 384), (4112, 640), (2064, 1024), (1040, 1152), (64, 17024), (5120, 8320)])
@pytest.mark.parametrize("wide", [0, 12])
def test_gemv_i8(ctx, typ, bits, M, rows, cols, wide):
    """Every epilogue, with and without the norm in front, over runs of tiles that end inside a warp's share, odd numbers of k-steps, zeros and steps that start anywhere in their
    blocks, and K in halves; with `wide` some activations 2^12 above the rest.  The products are exact and so are the sums of most groups; G groups are added up in fp32, four parts of
    at most three times the sum apart, and a group's activations (zero and bias multiply their sum) or, where they are no whole numbers together, its products are 128 terms in fp32.
    A bf16 result (8 significant bits) is off by one rounding more, the residual form by two, SwiGLU by those of gate and up."""
    import ctypes as C
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(rows + cols + M)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    qbias = 1 if typ == kf.KF_T_SIGN else 0

    def weight():
        data = torch.randint(0, 256, (rows, cols * bits // 8), generator=g, device="cuda", dtype=torch.uint8)
        n = rows * cols // 128
        step = (rnd(n).abs() * 0.02 + 0.002).bfloat16()
        zero = (rnd(n) * 0.05).bfloat16() if typ in (kf.KF_T_Q4, kf.KF_T_Q2) else torch.zeros(n, device="cuda").bfloat16()
        gama = torch.cat([torch.ones(rows + cols, device="cuda").bfloat16(), zero, step]).contiguous()
        per = 8 // bits
        b = data.view(rows, -1, 16).flip(2).reshape(rows, -1)
        q = torch.stack([(b >> (8 - bits * (j + 1))) & ((1 << bits) - 1) for j in range(per)], 2).view(rows, -1, 128)
        w = step.double().view(rows, -1, 1) * (q.double() - qbias) - zero.double().view(rows, -1, 1)
        high = (step.double().abs() * ((1 << bits) - 1 + qbias)).view(rows, -1)  # of a weight without its zero, by group
        return kf.TensorDesc(data.data_ptr(), gama.data_ptr(), rows, cols, typ, 128, qbias, None, None), w.view(rows, cols), (high, high + zero.double().abs().view(rows, -1), data, gama)

    (dw, w, keep0), (du, u, keep1) = weight(), weight()
    x = rnd(M, cols)
    x[:, 5::128] *= 2.0 ** wide
    x, nw = x.bfloat16(), (rnd(cols) * 0.1 + 1).bfloat16()
    s = 1 / torch.sqrt(x.float().square().mean(1, keepdim=True) + 1e-6)
    xn = ((x.float() * s) * nw.float()).bfloat16()  # off by one bf16 rounding where the sum of squares is taken in another order: bounded below by its share of the sum
    r = rnd(M, rows).bfloat16()
    ys = {k: torch.zeros(M, rows, device="cuda", dtype=torch.float32 if k == "f32" else torch.bfloat16) for k in ("none", "res", "f32", "glu", "norm")}
    gu, two = (kf.TensorDesc * 2)(dw, du), (C.c_void_p * 2)(ys["glu"].data_ptr(), ys["glu"].data_ptr())
    one, yn = (kf.TensorDesc * 1)(dw), (C.c_void_p * 1)(ys["norm"].data_ptr())
    torch.cuda.synchronize()
    for _ in range(2):
        ys["res"].copy_(r)
        torch.cuda.synchronize()
        ctx.check(ctx.lib.kf_linear(ctx.h, ys["none"].data_ptr(), C.byref(dw), x.data_ptr(), M, kf.KF_EPI_NONE, None), "none")
        ctx.check(ctx.lib.kf_linear(ctx.h, ys["res"].data_ptr(), C.byref(dw), x.data_ptr(), M, kf.KF_EPI_RESIDUAL, ys["res"].data_ptr()), "residual")
        ctx.check(ctx.lib.kf_linear(ctx.h, ys["f32"].data_ptr(), C.byref(dw), x.data_ptr(), M, kf.KF_EPI_F32, None), "f32")
        assert ctx.get_int("gemv_last_kernel") == 2
        ctx.check(ctx.lib.kf_rmsnorm_linear(ctx.h, 2, two, gu, x.data_ptr(), nw.data_ptr(), 1e-6, M, 2), "swiglu")
        ctx.check(ctx.lib.kf_rmsnorm_linear(ctx.h, 1, yn, one, x.data_ptr(), nw.data_ptr(), 1e-6, M, 0), "norm")
        ctx.sync()

    def slip(v, keep):
        return (3 * (cols // 128) + 64) * 2.0 ** -24 * (v.double().abs().view(M, -1, 128).sum(2) @ keep[1].T)

    want, eps, tiny = x.double() @ w.T, 2.0 ** -8 * 1.001, slip(x, keep0)
    assert bool(((ys["f32"].double() - want).abs() <= tiny).all())
    assert bool(((ys["none"].double() - want).abs() <= eps * want.abs() + tiny).all())
    assert bool(((ys["res"].double() - (r.double() + want)).abs() <= eps * (want.abs() + (r.double() + want).abs()) * 1.02 + tiny).all())
    xd, top = xn.double(), xn.double().abs().amax(1, keepdim=True)
    slack = 2.0 ** -8 * top * torch.maximum(w.abs().amax(1), u.abs().amax(1)) * 2  # two activations rounded the other way
    nrm, nmag = xd @ w.T, slip(xn, keep0) + slack
    assert bool(((ys["norm"].double() - nrm).abs() <= eps * nrm.abs() + nmag).all())
    up, umag = xd @ u.T, slip(xn, keep1) + slack
    glu = nrm * torch.sigmoid(nrm) * up
    bound = 1.1 * (eps * nrm.abs() + nmag) * (up.abs() + umag) + (nrm.abs() + nmag) * (eps * up.abs() + umag) + 1.1 * eps * glu.abs()
    assert bool(((ys["glu"].double() - glu).abs() <= bound * 1.02).all())


@pytest.mark.parametrize("typ", [kf.KF_T_Q4, kf.KF_T_SIGN, kf.KF_T_BINARY])
def test_gemv_i8_special_values(ctx, typ):
    """Infinities and NaN have no fixed-point form: the rows they reach are not finite, and the call after is as ever."""
    import ctypes as C
    import torch
    rows, cols = 1024, 1024
    w, wd = make_q(ctx, typ, rows, cols)
    d = w.desc()
    for bad in (float("inf"), float("-inf"), float("nan")):
        x, y = torch.zeros(1, cols, device="cuda").bfloat16(), torch.zeros(1, rows, device="cuda")
        x[0, 300] = bad
        torch.cuda.synchronize()
        ctx.check(ctx.lib.kf_linear(ctx.h, y.data_ptr(), C.byref(d), x.data_ptr(), 1, kf.KF_EPI_F32, None), "linear")
        ctx.sync()
        assert not bool(torch.isfinite(y).any()) and ctx.get_int("gemv_last_kernel") == 2
        x[0, 300] = 1
        torch.cuda.synchronize()
        ctx.check(ctx.lib.kf_linear(ctx.h, y.data_ptr(), C.byref(d), x.data_ptr(), 1, kf.KF_EPI_F32, None), "linear")
        ctx.sync()
        # one bf16 rounding of the weight in wd (2^-9), none inside the matmul but those of fp32
        assert bool(((y[0] - wd[:, 300]).abs() <= 2.0 ** -8 * wd[:, 300].abs() + 2.0 ** -20 * wd.abs().max()).all())


@pytest.mark.parametrize("typ", [kf.KF_T_Q4, kf.KF_T_Q2, kf.KF_T_SIGN, kf.KF_T_BINARY])
@pytest.mark.parametrize("rows,cols", [(4096, 4096), (2048, 5120)])
def test_one_two_and_several_tokens_agree(ctx, typ, rows, cols):
    """A token alone, in a pair and in a step of four take two kernels and two arithmetics.  gemv.cu holds activations in fp16, and its matrix instructions keep them to 2^-14 of a
    code of one at the worst (sums of products), which bounds the difference."""
    import ctypes as C
    import torch
    w, wd = make_q(ctx, typ, rows, cols)
    d, g = w.desc(), torch.Generator(device="cuda")
    g.manual_seed(11)
    x, ys = torch.randn(4, cols, generator=g, device="cuda").bfloat16(), []
    for m in (1, 2, 4):
        y = torch.zeros(4, rows, device="cuda")
        torch.cuda.synchronize()
        for i in range(0, 4, m):
            ctx.check(ctx.lib.kf_linear(ctx.h, _ptr(y[i:]), C.byref(d), _ptr(x[i:]), m, kf.KF_EPI_F32, None), "linear")
        ctx.sync()
        assert ctx.get_int("gemv_last_kernel") == (2 if m < 4 else 0)
        ys.append(y)
    slack = 2.0 ** -14 * (x.float().abs() @ wd.abs().T)
    assert bool(((ys[0] - ys[2]).abs() <= slack).all()) and bool(((ys[1] - ys[2]).abs() <= slack).all())


@pytest.mark.parametrize("M,rows,cols,knobs,kernel", [(1, 256, 4096, {}, 2), (1, 240, 4096, {}, 0), (1, 8192, 256, {}, 0), (1, 8192, 128, {}, 0), (2, 25600, 5120, {}, 2), (2, 25616, 5120, {}, 0),
                                                      (3, 4096, 4096, {}, 0), (1, 4096, 4096, {"gemv_exact": 1}, 0), (1, 4096, 4096, {"gemv_i8_max_m": 0}, 0),
                                                      (2, 4096, 4096, {"gemv_i8_max_m": 1}, 0), (1, 4096, 4096, {"gemv_splitk": 2}, 0)])
def test_gemv_i8_dispatch(ctx, M, rows, cols, knobs, kernel):
    """What stays with gemv.cu: few tiles, k of 128 and 256, two tokens over the largest 4-bit weights, more tokens, and what is asked for.  Either way the result is the matmul's."""
    import ctypes as C
    import torch
    w, wd = make_q(ctx, kf.KF_T_Q4, rows, cols)
    d, x, y = w.desc(), torch.randn(M, cols, device="cuda").bfloat16(), torch.zeros(M, rows, device="cuda")
    torch.cuda.synchronize()
    had = {k: ctx.get_int(k) if k != "gemv_splitk" else 0 for k in knobs}
    for k, v in knobs.items():
        ctx.set_int(k, v)
    try:
        ctx.check(ctx.lib.kf_linear(ctx.h, y.data_ptr(), C.byref(d), x.data_ptr(), M, kf.KF_EPI_F32, None), "linear")
        ctx.sync()
    finally:
        for k, v in had.items():
            ctx.set_int(k, v)
    assert ctx.get_int("gemv_last_kernel") == kernel
    want = x.double() @ wd.double().T
    # bf16 weights in wd (2^-9 each, in either direction), the activations of gemv.cu in fp16
    assert float((y.double() - want).norm() / want.norm()) <= 2.0 ** -8


def pack_codes(codes, bits):
    """[rows, cols] codes -> bytes of 128-bit words, the first code of a word in its most significant bits"""
    import torch
    rows, cols = codes.shape
    c = codes.view(rows, -1, 8 // bits).to(torch.uint8)
    b = torch.zeros_like(c[:, :, 0])
    for j in range(8 // bits):
        b |= c[:, :, j] << (8 - bits * (j + 1))
    return b.view(rows, -1, 16).flip(2).contiguous().view(rows, -1)


@pytest.mark.parametrize("typ,bits", [(kf.KF_T_Q4, 4), (kf.KF_T_Q2, 2), (kf.KF_T_SIGN, 2), (kf.KF_T_BINARY, 1)])
@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("kind", ["2^14", "2^18", "2^40", "top", "top and others", "2^-100", "2^-120 and less", "2^-100 and 2^60"])
def test_gemv_i8_activations_of_any_size(ctx, typ, bits, M, kind):
    """Activations keep all their bits whatever stands beside them.  In every second row the code that meets the large activation is zero, so that nothing but the others shows: one
    far above the rest of its group, the largest finite numbers of either sign at every place of a group (every field of a byte), numbers far below one, and whole groups of them
    between groups far above one.  A product is exact; what is rounded are the fp32 sums: those of a group (none where it is a whole number, eight matrix instructions of 16
    products otherwise), over the groups, and of its activations, which step * bias and zero multiply."""
    import ctypes as C
    import torch
    rows, cols = 1024, 16384 if kind.startswith("top") else 1024
    G, qbias = cols // 128, 1 if typ == kf.KF_T_SIGN else 0
    g = torch.Generator(device="cuda")
    g.manual_seed(bits * 10 + M)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    q = torch.randint(0, 2 ** bits, (rows, cols), generator=g, device="cuda")
    x, grp = rnd(M, G, 128), torch.arange(G, device="cuda")
    big = torch.zeros(G, 128, dtype=torch.bool, device="cuda")
    if kind == "2^-100 and 2^60":
        big[::2] = True
        x[:, ::2] *= 2.0 ** 60
        x[:, 1::2] *= 2.0 ** -100
    elif kind.startswith("2^-1"):
        x[:, 1:] *= 2.0 ** -100 if kind == "2^-100" else 2.0 ** -120
        x[:, 2] *= 2.0 ** -9  # the latter among the subnormal numbers
        x[:, 0] = 0
    else:
        big[grp, (grp * 37 + 5) % 128] = True  # 37 is odd: every place of a group in 128 groups
        if kind == "top and others":
            big[grp, (grp * 37 + 69) % 128] = True  # their sum is no number
        x = x.bfloat16().float()
        if kind == "top":
            x[:] = 0
        sign = 1 - 2 * (grp // 3 % 2).float()
        x[:, big] = ((torch.finfo(torch.bfloat16).max if kind.startswith("top") else 2.0 ** float(kind[2:])) * sign).repeat_interleave(int(big[0].sum()))
    q[1::2] *= ~big.view(1, cols)
    if kind == "top":
        q[1::4] = (q[::4] + 1) % 2 ** bits  # nothing else to be seen there
    x = x.view(M, cols).bfloat16()
    n = rows * G
    up = 2.0 ** 20 if kind == "2^-120 and less" else 1.0
    step, zero = ((rnd(n).abs() * 2.0 ** -18 + 2.0 ** -20) * up).bfloat16(), torch.zeros(n, device="cuda").bfloat16()
    gama, data = torch.cat([torch.ones(rows + cols, device="cuda").bfloat16(), zero, step]).contiguous(), pack_codes(q, bits)
    d, y = kf.TensorDesc(data.data_ptr(), gama.data_ptr(), rows, cols, typ, 128, qbias, None, None), torch.zeros(M, rows, device="cuda")
    torch.cuda.synchronize()
    ctx.check(ctx.lib.kf_linear(ctx.h, y.data_ptr(), C.byref(d), x.data_ptr(), M, kf.KF_EPI_F32, None), "linear")
    ctx.sync()
    st = step.double().view(rows, G, 1)
    want = x.double() @ (st * (q.double() - qbias).view(rows, G, 128)).view(rows, cols).T
    mag = x.double().abs() @ (st * (q.double() + qbias).view(rows, G, 128)).view(rows, cols).T
    assert ctx.get_int("gemv_last_kernel") == 2
    # a limb's part of a number is at most three times the number
    assert bool(torch.isfinite(y).all()) and bool(((y.double() - want).abs() <= 3 * (G + 64) * 2.0 ** -23 * mag + 2.0 ** -145).all())


# ---------------------------------------------------------------------------------------------- long reductions in the tcgen05 matmul
@pytest.mark.parametrize("plan", [0, 1])
@pytest.mark.parametrize("rows,cols,M", [(5120, 8192, 2048), (10240, 25600, 45), (2560, 25600, 128), (51200, 5120, 45), (1024, 25600, 300)])
def test_tc_long_reduction(ctx, rows, cols, M, plan):
    """Items of 32 and more raw stages: a stage that is handed back before its bytes were read shows as whole rows that used another stage's weights.
    The weights are exact on both sides, so what is left is the order of fp32 sums: 2^-24 * sqrt(cols) of the result, far below 1e-4; a stage that went
    wrong moves a row by 0.1 of it.  plan 0: token tile and split by modelled time; 1: those of gemv_exact."""
    import torch
    torch.backends.cuda.matmul.allow_tf32 = False
    w, wd = make_q(ctx, kf.KF_T_Q4, rows, cols)
    x = kf.fill_normal(ctx, M * cols, 7, 1.0)
    want = bf16_tensor(x, M, cols).float() @ wd.T
    exact = ctx.get_int("gemv_exact")
    ctx.set_int("gemv_exact", plan)
    try:
        for _ in range(4):
            y = torch.from_numpy(kf.linear(ctx, w, x, M, kf.KF_EPI_F32).numpy(np.float32, (M, rows))).cuda()
            worst = ((y - want).square().mean(0).sqrt() / want.square().mean().sqrt()).max()
            assert float(worst) < 1e-4, float(worst)
    finally:
        ctx.set_int("gemv_exact", exact)


@pytest.mark.parametrize("exact", [0, 1])
@pytest.mark.parametrize("M,rows,cols", [(1, 5120, 25600), (2, 25600, 5120), (8, 2560, 25600)])
def test_gemv_tma_long_reduction(ctx, exact, M, rows, cols):
    """The TMA-fed skinny matmul over many uses of its ring: a stage that is handed back before its bytes were read shows as rows that are off by 0.1 and more.  The
    result is rounded to bf16 (2^-9 of itself in the mean); without gemv_exact the weights are not rounded to bf16 (1.5e-3 of the rms): 1e-2 covers both."""
    import torch
    torch.backends.cuda.matmul.allow_tf32 = False
    w, wd = make_q(ctx, kf.KF_T_Q4, rows, cols)
    x = kf.fill_normal(ctx, M * cols, 9, 1.0)
    want = bf16_tensor(x, M, cols).float() @ wd.T
    before = ctx.get_int("gemv_exact")
    ctx.set_int("gemv_exact", exact), ctx.set_int("gemv_tma", 1)
    try:
        first = None
        for _ in range(4):
            y = bf16_tensor(kf.linear(ctx, w, x, M), M, rows)
            assert float((y.float() - want).abs().max() / want.square().mean().sqrt()) < (0.03 if exact else 0.05)
            assert float((y.float() - want).square().mean().sqrt() / want.square().mean().sqrt()) < 1e-2
            first = y if first is None else first
            assert torch.equal(y, first)
    finally:
        ctx.set_int("gemv_exact", before), ctx.set_int("gemv_tma", 0)


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
    M, rounds = 3, 34
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


# ---------------------------------------------------------------------------------------------- tcgen05 matmul: token tiles, k-splits, epilogues
def _ptr(t):
    return t.data_ptr()


@pytest.mark.parametrize("fma", [0, 1])
@pytest.mark.parametrize("typ,bits,qbias", [(kf.KF_T_Q4, 4, 0), (kf.KF_T_Q4, 4, 8), (kf.KF_T_Q4, 4, 117), (kf.KF_T_Q2, 2, 0), (kf.KF_T_Q2, 2, -2), (kf.KF_T_SIGN, 2, 0), (kf.KF_T_SIGN, 2, 1),
                                            (kf.KF_T_SIGN, 2, 3), (kf.KF_T_BINARY, 1, 0), (kf.KF_T_BINARY, 1, 1)])
@pytest.mark.parametrize("M,rows,cols", [(9, 16, 128), (40, 144, 640), (128, 272, 384), (256, 128, 1152)])
def test_tc_weights_bit_for_bit(ctx, typ, bits, qbias, fma, M, rows, cols, lo=-40, hi=50):
    """Each token picks one column, so the result is the weight itself: the codes that the matmul expands inside its own number format round as kf_dequant does, for steps
    from 2^-40 to 2^50, zeros of any size beside them, codes with and without a bias, and reductions that end inside a stage."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(3 * M + bits + qbias)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    data = torch.randint(0, 256, (rows, cols * bits // 8), generator=g, device="cuda", dtype=torch.uint8)
    n = rows * cols // 128
    step = (rnd(n) * torch.exp2(torch.randint(lo, hi, (n,), generator=g, device="cuda").float())).bfloat16()
    zero = (rnd(n) * 4 * step.float()).bfloat16() if typ in (kf.KF_T_Q4, kf.KF_T_Q2) else torch.zeros(n, device="cuda").bfloat16()
    step[::17], zero[::13] = 0, 0
    gama = torch.cat([torch.ones(rows + cols, device="cuda").bfloat16(), zero, step]).contiguous()
    desc = kf.TensorDesc(data.data_ptr(), gama.data_ptr(), rows, cols, typ, 128, qbias, None, None)
    import ctypes as C
    w, y = torch.zeros(rows, cols, device="cuda").bfloat16(), torch.zeros(M, rows, device="cuda").bfloat16()
    k = (torch.arange(M, device="cuda") * 37 + 5) % cols
    x = torch.zeros(M, cols, device="cuda").bfloat16()
    x[torch.arange(M, device="cuda"), k] = 1
    torch.cuda.synchronize()
    ctx.set_int("deq_fma", fma), ctx.set_int("tc_min_m", 1)
    try:
        ctx.check(ctx.lib.kf_dequant(ctx.h, C.byref(desc), w.data_ptr()), "dequant")
        ctx.check(ctx.lib.kf_linear(ctx.h, y.data_ptr(), C.byref(desc), x.data_ptr(), M, kf.KF_EPI_NONE, None), "linear")
        ctx.sync()
    finally:
        ctx.set_int("deq_fma", 1), ctx.set_int("tc_min_m", -1)
    assert bool((y.float() == w[:, k].T.float()).all())


@pytest.mark.parametrize("fma", [0, 1])
@pytest.mark.parametrize("typ,bits,qbias", [(kf.KF_T_Q4, 4, 0), (kf.KF_T_Q4, 4, 8), (kf.KF_T_Q2, 2, 0), (kf.KF_T_SIGN, 2, 1), (kf.KF_T_SIGN, 2, 3), (kf.KF_T_BINARY, 1, 0)])
@pytest.mark.parametrize("M,rows,cols,lo,hi", [(20, 144, 640, -110, -40), (256, 128, 1152, -110, 118), (9, 272, 640, 50, 118), (40, 144, 640, -1, 5), (100, 144, 1152, -20, 118)])
def test_tc_weights_of_any_step(ctx, typ, bits, qbias, fma, M, rows, cols, lo, hi):
    """As above over the range of bf16: groups whose steps lie beyond what the quick expansion holds beside groups that it takes, in the same rows and the same stages."""
    test_tc_weights_bit_for_bit(ctx, typ, bits, qbias, fma, M, rows, cols, lo, hi)


@pytest.mark.parametrize("typ", [kf.KF_T_Q4, kf.KF_T_BINARY, kf.KF_T_F8E5M2, kf.KF_T_BF16])
@pytest.mark.parametrize("M,tc_bn,splits", [(9, 16, 1), (9, 32, 3), (17, 16, 2), (33, 64, 0), (64, 32, 5), (65, 128, 1), (129, 64, 1), (130, 256, 2), (255, 128, 3),
                                            (257, 0, 0), (300, 256, 1)])
@pytest.mark.parametrize("rows,cols", [(16, 128), (144, 1152), (272, 640)])
def test_tc_tiles_and_epilogues(ctx, typ, M, tc_bn, splits, rows, cols):
    """Every epilogue (plain, residual in place, fp32, SwiGLU) over ragged token and row tiles, whole and split reductions, aligned and misaligned outputs.
    Weights and activations are exact on both sides and the sums are fp32 (1e-5 of the rms covers their order), so a bf16 result (8 significant bits) is off by one rounding,
    2^-8 of itself, the residual form by two; SwiGLU rounds gate and up as well, whose errors pass through |d silu| < 1.1."""
    import torch
    torch.backends.cuda.matmul.allow_tf32 = False
    mk = lambda seed: (make_q(ctx, typ, rows, cols, seed) if typ != kf.KF_T_BF16 else _bf16_weight(ctx, rows, cols, seed))  # noqa: E731
    (w, wd), (u, ud) = mk(5), mk(6)
    g = torch.Generator(device="cuda")
    g.manual_seed(M)
    x = torch.randn(M, cols, generator=g, device="cuda").bfloat16()
    r = torch.randn(M, rows, generator=g, device="cuda").bfloat16()
    acc, up = x.float() @ wd.T, x.float() @ ud.T
    eps, tiny = 2.0 ** -8 * 1.001, 1e-5 * float(acc.square().mean().sqrt())
    want_glu = acc * torch.sigmoid(acc) * up
    import ctypes as C
    dw, du = w.desc(), u.desc()
    gu = (kf.TensorDesc * 2)(dw, du)
    ctx.set_int("tc_min_m", 1), ctx.set_int("tc_bn", tc_bn), ctx.set_int("gemv_splitk", splits)
    try:
        for off in (0, 1):  # elements that the output lies behind a 16-byte boundary
            def out(dtype):
                return torch.zeros(M * rows + off, dtype=dtype, device="cuda")[off:].view(M, rows)
            y, yr, yf, yg = out(torch.bfloat16), out(torch.bfloat16), out(torch.float32), out(torch.bfloat16)
            yr.copy_(r)
            torch.cuda.synchronize()
            ctx.check(ctx.lib.kf_linear(ctx.h, _ptr(y), C.byref(dw), _ptr(x), M, kf.KF_EPI_NONE, None), "none")
            ctx.check(ctx.lib.kf_linear(ctx.h, _ptr(yr), C.byref(dw), _ptr(x), M, kf.KF_EPI_RESIDUAL, _ptr(yr)), "residual")
            ctx.check(ctx.lib.kf_linear(ctx.h, _ptr(yf), C.byref(dw), _ptr(x), M, kf.KF_EPI_F32, None), "f32")
            ctx.check(ctx.lib.kf_linear_swiglu(ctx.h, _ptr(yg), C.byref(gu[0]), C.byref(gu[1]), _ptr(x), M), "swiglu")
            ctx.sync()
            assert bool(((yf - acc).abs() <= tiny).all())
            assert bool(((y.float() - acc).abs() <= eps * acc.abs() + tiny).all())
            assert bool(((yr.float() - (r.float() + acc)).abs() <= eps * (acc.abs() + (r.float() + acc).abs()) * 1.02 + tiny).all())
            bound = 1.1 * eps * acc.abs() * up.abs() + 2.1 * eps * want_glu.abs() + tiny * (up.abs() + acc.abs() + 1)
            assert bool(((yg.float() - want_glu).abs() <= bound * 1.02).all())
    finally:
        ctx.set_int("tc_min_m", -1), ctx.set_int("tc_bn", 0), ctx.set_int("gemv_splitk", 0)


@pytest.mark.parametrize("typ", [kf.KF_T_BF16, kf.KF_T_F8E5M2, kf.KF_T_Q4])
@pytest.mark.parametrize("M,rows,cols,at", [(16, 512, 1024, 0), (300, 4096, 1024, 0), (300, 1024, 4096, 16), (700, 3072, 3072, -64)])
def test_tc_swiglu_over_its_input(ctx, typ, M, rows, cols, at):
    """The result may lie over the activations, `at` elements behind their start: the bits of a result in a buffer of its own."""
    import ctypes as C

    import torch
    mk = lambda seed: (make_q(ctx, typ, rows, cols, seed) if typ != kf.KF_T_BF16 else _bf16_weight(ctx, rows, cols, seed))[0]  # noqa: E731
    wg, wu = mk(5), mk(6)
    g = torch.Generator(device="cuda")
    g.manual_seed(M)
    x = torch.randn(M * cols, generator=g, device="cuda").bfloat16()
    own, buf = torch.zeros(M * rows, device="cuda").bfloat16(), torch.zeros(M * max(rows, cols) + 256, device="cuda").bfloat16()
    buf[64:64 + M * cols] = x
    torch.cuda.synchronize()
    dg, du = wg.desc(), wu.desc()
    ctx.check(ctx.lib.kf_linear_swiglu(ctx.h, _ptr(own), C.byref(dg), C.byref(du), _ptr(x), M), "swiglu")
    ctx.check(ctx.lib.kf_linear_swiglu(ctx.h, _ptr(buf[64 + at:]), C.byref(dg), C.byref(du), _ptr(buf[64:]), M), "swiglu over x")
    ctx.sync()
    assert torch.equal(own, buf[64 + at:64 + at + M * rows])


@pytest.mark.parametrize("typ", [kf.KF_T_Q4, kf.KF_T_SIGN, kf.KF_T_BINARY])
@pytest.mark.parametrize("at", [0, 8, 1024, -1024, 200 * 1024 - 8, 200 * 1024])
def test_tc_single_weight_over_its_input(ctx, typ, at):
    """One packed weight and more than 128 tokens: activations are read as they lie, by every item, so not where the result lies over them, `at` elements behind their start.  fp32 sums
    in one order or the other (1e-5 of the rms), one bf16 rounding."""
    import ctypes as C
    import torch
    M, n = 200, 1024
    w, wd = make_q(ctx, typ, n, n)
    d = w.desc()
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    x = torch.randn(M, n, generator=g, device="cuda").bfloat16()
    buf = torch.zeros(3 * M * n, device="cuda").bfloat16()
    for _ in range(3):
        buf[M * n:2 * M * n] = x.view(-1)
        torch.cuda.synchronize()
        ctx.check(ctx.lib.kf_linear(ctx.h, _ptr(buf[M * n + at:]), C.byref(d), _ptr(buf[M * n:]), M, kf.KF_EPI_NONE, None), "linear over x")
        ctx.sync()
        y, want = buf[M * n + at:2 * M * n + at].view(M, n).double(), x.double() @ wd.double().T
        assert bool(((y - want).abs() <= 2.0 ** -8 * 1.001 * want.abs() + 1e-5 * want.square().mean().sqrt()).all())


def test_tc_split_inside_a_capture():
    """A shape that an eager call cuts through the workspace: captured on a context without one it is planned whole or in clusters, captured after an eager call it has that call's
    bits.  fp32 sums in one order or the other: each of K / 16 additions loses at most 2^-23 of a partial sum, which stays below six times the rms."""
    import ctypes as C
    import torch
    rows, cols, M = 9600, 4608, 12
    outs, plans = [], []
    for eager_first in (False, True):
        c = kf.Context(0)
        w, wd = make_q(c, kf.KF_T_Q4, rows, cols)
        d = w.desc()
        g = torch.Generator(device="cuda")
        g.manual_seed(3)
        x, y, e = torch.randn(M, cols, generator=g, device="cuda").bfloat16(), torch.zeros(M, rows, device="cuda"), torch.zeros(M, rows, device="cuda")
        small, s = torch.zeros(M, 16, device="cuda"), make_q(c, kf.KF_T_Q4, 16, cols)[0]
        torch.cuda.synchronize()
        ds = s.desc()
        c.check(c.lib.kf_linear(c.h, _ptr(small), C.byref(ds), _ptr(x), M, kf.KF_EPI_F32, None), "scratch for the activations")
        if eager_first:
            c.check(c.lib.kf_linear(c.h, _ptr(e), C.byref(d), _ptr(x), M, kf.KF_EPI_F32, None), "eager")
            assert c.get_int("tc_last_split") > 1 and not c.get_int("tc_last_cluster")
        c.check(c.lib.kf_graph_begin(c.h), "begin")
        rc, graph = c.lib.kf_linear(c.h, _ptr(y), C.byref(d), _ptr(x), M, kf.KF_EPI_F32, None), C.c_void_p()
        plans.append((c.get_int("tc_last_split"), c.get_int("tc_last_cluster")))
        c.check(c.lib.kf_graph_end(c.h, C.byref(graph)), "end")
        c.check(rc, "captured")
        for _ in range(2):
            c.check(c.lib.kf_graph_launch(c.h, graph), "launch")
        c.sync()
        if eager_first:
            assert torch.equal(y, e)
        outs.append(y)
        c.lib.kf_graph_destroy(graph)
        c.close()
    assert plans[0] != plans[1] and (plans[0][0] == 1 or plans[0][1] == 1)
    want = x.double() @ wd.double().T
    for y in outs:
        assert bool(((y.double() - want).abs() <= cols // 16 * 2.0 ** -23 * 6 * want.square().mean().sqrt()).all())


@pytest.mark.parametrize("typ", [kf.KF_T_Q4, kf.KF_T_BINARY, kf.KF_T_BF16])
@pytest.mark.parametrize("M,tc_bn,splits", [(16, 16, 8), (20, 32, 2), (45, 64, 4), (100, 128, 3), (130, 256, 2), (251, 256, 5), (257, 128, 7)])
def test_tc_split_over_cluster_equals_workspace(ctx, typ, M, tc_bn, splits):
    """A split whose parts meet in a cluster adds the same partial sums in the same order as one through the workspace (which gemv_exact keeps to): equal bits, every
    epilogue.  The plan of the last launch tells which of the two ran."""
    import torch
    import ctypes as C
    rows, cols = 272, 8192
    mk = lambda seed: (make_q(ctx, typ, rows, cols, seed) if typ != kf.KF_T_BF16 else _bf16_weight(ctx, rows, cols, seed))[0]  # noqa: E731
    w, u = mk(5), mk(6)
    dw = w.desc()
    gu = (kf.TensorDesc * 2)(dw, u.desc())
    x, r = torch.randn(M, cols, device="cuda").bfloat16(), torch.randn(M, rows, device="cuda").bfloat16()
    ctx.set_int("tc_min_m", 1), ctx.set_int("tc_bn", tc_bn), ctx.set_int("gemv_splitk", splits)
    outs = []
    try:
        for exact in (0, 1):
            ctx.set_int("gemv_exact", exact)
            def ran(name, st):
                ctx.check(st, name)
                assert [ctx.get_int("tc_last_" + k) for k in ("bn", "split", "cluster")] == [tc_bn, splits, 1 - exact], name
            y, yr, yg, yf = (torch.zeros(M, rows, device="cuda", dtype=t) for t in (torch.bfloat16, torch.bfloat16, torch.bfloat16, torch.float32))
            torch.cuda.synchronize()
            ran("none", ctx.lib.kf_linear(ctx.h, _ptr(y), C.byref(dw), _ptr(x), M, kf.KF_EPI_NONE, None))
            ran("residual", ctx.lib.kf_linear(ctx.h, _ptr(yr), C.byref(dw), _ptr(x), M, kf.KF_EPI_RESIDUAL, _ptr(r)))
            ran("f32", ctx.lib.kf_linear(ctx.h, _ptr(yf), C.byref(dw), _ptr(x), M, kf.KF_EPI_F32, None))
            ran("swiglu", ctx.lib.kf_linear_swiglu(ctx.h, _ptr(yg), C.byref(gu[0]), C.byref(gu[1]), _ptr(x), M))
            ctx.sync()
            outs.append((y, yr, yg, yf))
    finally:
        ctx.set_int("tc_min_m", -1), ctx.set_int("tc_bn", 0), ctx.set_int("gemv_splitk", 0), ctx.set_int("gemv_exact", 0)
    assert float(outs[0][3].abs().max()) > 0
    for a, b in zip(*outs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("typ", [kf.KF_T_Q4, kf.KF_T_BF16])
@pytest.mark.parametrize("M,tc_bn", [(41, 16), (300, 64), (600, 128), (1100, 256)])
@pytest.mark.parametrize("splits", [1, 2, 3])
def test_tc_several_items_per_cta(ctx, typ, M, tc_bn, splits):
    """Items that the epilogue warps finish alone, under the next one's main loop, and the last one, with the producers' help; whole and in parts whose sums meet in the
    workspace; every epilogue, and an output that starts at an odd element.  An fp32 sum of 1024 terms is off by 2^-24 * sqrt(1024) = 2e-6 of the rms; 4e-5 holds for
    the largest of the seven million.  A bf16 result is rounded to 2^-8 of itself; SwiGLU takes the rounded gate and up, each of which may be one step off."""
    import torch
    import ctypes as C
    rows, cols = 6416, 1024
    mk = lambda seed: make_q(ctx, typ, rows, cols, seed) if typ != kf.KF_T_BF16 else _bf16_weight(ctx, rows, cols, seed)  # noqa: E731
    (w, wd), (u, ud) = mk(5), mk(6)
    gu = (kf.TensorDesc * 2)(w.desc(), u.desc())
    x, r = torch.randn(M, cols, device="cuda").bfloat16(), torch.randn(M, rows, device="cuda").bfloat16()
    acc, up = x.double() @ wd.double().T, x.double() @ ud.double().T
    eps, tiny = 2.0 ** -8 * 1.001, 4e-5 * float(acc.square().mean().sqrt())
    yr, yf, yg, yo = r.clone(), torch.zeros(M, rows, device="cuda"), torch.zeros_like(r), torch.zeros(M * rows + 1, device="cuda").bfloat16()[1:]
    torch.cuda.synchronize()
    ctx.set_int("tc_min_m", 1), ctx.set_int("tc_bn", tc_bn), ctx.set_int("gemv_splitk", splits)
    try:
        ctx.check(ctx.lib.kf_linear(ctx.h, _ptr(yr), C.byref(gu[0]), _ptr(x), M, kf.KF_EPI_RESIDUAL, _ptr(yr)), "residual")
        ctx.check(ctx.lib.kf_linear(ctx.h, _ptr(yf), C.byref(gu[0]), _ptr(x), M, kf.KF_EPI_F32, None), "f32")
        ctx.check(ctx.lib.kf_linear(ctx.h, _ptr(yo), C.byref(gu[0]), _ptr(x), M, kf.KF_EPI_NONE, None), "odd")
        ctx.check(ctx.lib.kf_linear_swiglu(ctx.h, _ptr(yg), C.byref(gu[0]), C.byref(gu[1]), _ptr(x), M), "swiglu")
        ctx.sync()
    finally:
        ctx.set_int("tc_min_m", -1), ctx.set_int("tc_bn", 0), ctx.set_int("gemv_splitk", 0)
    assert bool(((yf.double() - acc).abs() <= tiny).all())
    assert bool(((yo.view(M, rows).double() - acc).abs() <= eps * acc.abs() + tiny).all())
    assert bool(((yr.double() - (r.double() + acc)).abs() <= eps * (acc.abs() + (r.double() + acc).abs()) * 1.02 + tiny).all())
    want = acc * torch.sigmoid(acc) * up
    assert bool(((yg.double() - want).abs() <= eps * (2 * want.abs() + 1.2 * (acc * up).abs()) * 1.02 + tiny * (1 + acc.abs() + up.abs())).all())


@pytest.mark.parametrize("tc_bn", [0, 64])
def test_tc_split_as_asked(ctx, tc_bn):
    """gemv_splitk is taken as it is, up to the number of k stages (K = 5120 in 4 bits: 20 of 256), and so is the token tile beside it.  Sums of parts differ in
    their last bits from one pass: 17 and more parts must not give the bits of one, and stay within 1e-4 of the result's rms (320 partial sums on tensor cores, each off by up to 2^-23)."""
    import torch
    rows, cols, M = 256, 5120, 40
    w, wd = make_q(ctx, kf.KF_T_Q4, rows, cols)
    x = kf.fill_normal(ctx, M * cols, 7, 1.0)
    want = bf16_tensor(x, M, cols).double() @ wd.double().T
    got = {}
    ctx.set_int("tc_bn", tc_bn)
    try:
        for s in (1, 17, 20, 1000):
            ctx.set_int("gemv_splitk", s)
            got[s] = torch.from_numpy(kf.linear(ctx, w, x, M, kf.KF_EPI_F32).numpy(np.float32, (M, rows))).cuda()
            assert float(((got[s].double() - want).abs().max() / want.square().mean().sqrt())) < 1e-4
    finally:
        ctx.set_int("gemv_splitk", 0), ctx.set_int("tc_bn", 0)
    assert not torch.equal(got[1], got[17]) and not torch.equal(got[17], got[20])
    assert torch.equal(got[20], got[1000])


def _bf16_weight(ctx, rows, cols, seed):
    d = kf.fill_normal(ctx, rows * cols, seed, 0.02)
    bits = d.numpy(np.uint16)
    return kf.QTensor.from_packed(ctx, bits.view(np.uint8), None, rows, cols, kf.KF_T_BF16), bf16_tensor(d, rows, cols).float()


# ---------------------------------------------------------------------------------------------- panel attention on tcgen05
@pytest.mark.parametrize("n_head,n_kv", [(2, 1), (16, 8), (32, 8)])
@pytest.mark.parametrize("M,pos0,behind", [(65, 0, 0), (128, 0, 300), (129, 0, 1), (200, 1, 57), (127, 128, 1), (256, 127, 129), (100, 700, 60), (513, 255, 0), (300, 4000, 90)])
@pytest.mark.parametrize("sharp", [1.0, 12.0])
def test_prefill_tc(ctx, n_head, n_kv, M, pos0, behind, sharp):
    """Ragged query and key tiles, cache rows behind the last position that hold no numbers, flat and peaked scores (maxima that grow along the keys: the
    rescaling of the output).  A weight is rounded to bf16 once (2^-8 of itself), the result once, scores and sums are fp32:
    |error| <= 2^-8 (sum p |v| + |out|) + 1e-4 of that for the fp32 parts."""
    import torch
    hd, max_seq = 128, pos0 + M + behind
    g = torch.Generator(device="cuda")
    g.manual_seed(M + pos0 + n_head)
    q = (torch.randn(M, n_head, hd, generator=g, device="cuda") * sharp).bfloat16()
    k, v = (torch.randn(max_seq, n_kv, hd, generator=g, device="cuda") for _ in range(2))
    k = (k * torch.linspace(0.2, 1.5, max_seq, device="cuda")[:, None, None]).bfloat16()
    v = v.bfloat16()
    k[pos0 + M:], v[pos0 + M:] = float("nan"), float("inf")
    pos = torch.arange(pos0, pos0 + M, dtype=torch.int32, device="cuda")
    out = torch.full((M, n_head, hd), 7.0, device="cuda").bfloat16()
    torch.cuda.synchronize()
    ctx.set_int("attn_tc_min_m", 65)
    try:
        ctx.check(ctx.lib.kf_attn_prefill(ctx.h, _ptr(out), _ptr(q), _ptr(k), _ptr(v), _ptr(pos), M, n_head, n_kv, hd, max_seq), "prefill")
    finally:
        ctx.set_int("attn_tc_min_m", 0)
    ctx.sync()
    assert ctx.get_int("attn_tc_error") == 0
    keys = torch.arange(pos0 + M, device="cuda")
    for h in range(n_head):
        kk, vv = k[:pos0 + M, h // (n_head // n_kv)].double(), v[:pos0 + M, h // (n_head // n_kv)].double()
        s = q[:, h].double() @ kk.T / hd ** 0.5
        p = torch.softmax(s.masked_fill(keys[None] > pos[:, None], float("-inf")), -1)
        want, mass = p @ vv, p @ vv.abs()
        err = (out[:, h].double() - want).abs()
        assert bool((err <= 2.0 ** -8 * 1.01 * (mass + want.abs()) + 1e-6).all()), (h, float((err / (mass + want.abs())).max()))


@pytest.mark.parametrize("n_head,M,room,tc", [(16, 96, 0, False), (16, 96, 512, False), (16, 96, 513, True), (16, 512, 0, False), (16, 600, 0, True), (32, 256, 0, False),
                                              (32, 257, 0, True), (64, 128, 0, False), (64, 129, 0, True), (2, 512, 300, False), (2, 513, 300, True)])
def test_prefill_takes_the_kernel_that_gains(ctx, n_head, M, room, tc):
    """Panels that the mma.sync kernel has SMs for (148: one 64-query tile of a head each), of up to 512 tokens and with room for up to 512 in front, go there: the
    bits name the kernel."""
    import torch
    hd, n_kv = 128, max(1, n_head // 4)
    g = torch.Generator(device="cuda")
    g.manual_seed(M)
    q = torch.randn(M, n_head, hd, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(M + room, n_kv, hd, generator=g, device="cuda").bfloat16() for _ in range(2))
    pos, got = torch.arange(M, dtype=torch.int32, device="cuda"), []
    torch.cuda.synchronize()
    for least in (0, 65, 1 << 30):
        out = torch.zeros(M, n_head, hd, device="cuda").bfloat16()
        torch.cuda.synchronize()
        ctx.set_int("attn_tc_min_m", least)
        try:
            ctx.check(ctx.lib.kf_attn_prefill(ctx.h, _ptr(out), _ptr(q), _ptr(k), _ptr(v), _ptr(pos), M, n_head, n_kv, hd, M + room), "prefill")
        finally:
            ctx.set_int("attn_tc_min_m", 0)
        ctx.sync()
        got.append(out)
    assert not torch.equal(got[1], got[2])
    assert torch.equal(got[0], got[1 if tc else 2])


@pytest.mark.parametrize("M,pos0,gone", [(100, 256, (0, 128)), (100, 256, (0, 250)), (300, 130, (0, 130)), (200, 300, (128, 256))])
def test_prefill_scores_of_minus_infinity(ctx, M, pos0, gone):
    """Whole key tiles whose scores are -inf, the first ones among them: their weights are 0, the keys behind them count."""
    import torch
    hd, n_head, n_kv, n = 128, 16, 8, pos0 + M
    g = torch.Generator(device="cuda")
    g.manual_seed(M + pos0)
    q = torch.randn(M, n_head, hd, generator=g, device="cuda").bfloat16()
    q[..., 0] = q[..., 0].abs() + 0.25
    k, v = (torch.randn(n, n_kv, hd, generator=g, device="cuda").bfloat16() for _ in range(2))
    k[gone[0]:gone[1], :, 0] = float("-inf")
    pos = torch.arange(pos0, n, dtype=torch.int32, device="cuda")
    out = torch.zeros(M, n_head, hd, device="cuda").bfloat16()
    torch.cuda.synchronize()
    ctx.set_int("attn_tc_min_m", 65)
    try:
        ctx.check(ctx.lib.kf_attn_prefill(ctx.h, _ptr(out), _ptr(q), _ptr(k), _ptr(v), _ptr(pos), M, n_head, n_kv, hd, n), "prefill")
    finally:
        ctx.set_int("attn_tc_min_m", 0)
    ctx.sync()
    keys = torch.arange(n, device="cuda")
    unseen = (keys[None] > pos[:, None]) | ((keys >= gone[0]) & (keys < gone[1]))[None]
    k[gone[0]:gone[1], :, 0] = 0
    for h in range(n_head):
        kk, vv = k[:, h // 2].double(), v[:, h // 2].double()
        p = torch.softmax((q[:, h].double() @ kk.T / hd ** 0.5).masked_fill(unseen, float("-inf")), -1)
        want, mass = p @ vv, p @ vv.abs()
        assert bool(((out[:, h].double() - want).abs() <= 2.0 ** -8 * 1.01 * (mass + want.abs()) + 1e-6).all()), h


# ---------------------------------------------------------------------------------------------- grouped decode attention
_GQA_SHAPES = [(128, 8, 8), (128, 16, 8), (128, 16, 1), (128, 24, 2), (64, 8, 2)]
_GQA_LENS = [((1,), 0), ((63, 64, 65, 1, 128, 129), 128), ((256, 257, 511, 513, 40), 512), ((2000, 3, 700, 1300), 1999), ((9000,), 8999), ((9000,), 100),
             ((5000, 17), 300), ((40000,), 65535), (tuple(1 + 37 * i % 190 for i in range(40)), 189), (tuple(1 + 37 * i % 190 for i in range(300)), 100)]
# four and eight heads per kv head, each run several rings long
_GQA_RINGS = [(128, 32, 8, (40000,), 39999), (128, 64, 8, (40000,), 39999), (128, 8, 2, (9000, 30000), 29999), (64, 32, 8, (40000,), 39999)]
# whole sequences in thirds, two items per thread block; more sequences than the dealing tables hold, cut into runs
_GQA_THIRDS = [(128, 16, 8, tuple(6000 - 397 * i for i in range(12)), 5999), (128, 80, 10, tuple(300 + 1237 * i % 5200 for i in range(9)), 5499)]
_GQA_MANY = [(128, 2, 1, tuple(1 + 37 * i % 190 for i in range(600)), 189), (64, 1, 1, tuple(1 + 37 * i % 190 for i in range(513)), 50)]


@pytest.mark.parametrize("hd,n_head,n_kv,lens,hint", [a + b for a in _GQA_SHAPES for b in _GQA_LENS] + _GQA_RINGS + _GQA_THIRDS + _GQA_MANY)
def test_gqa_runs(ctx, hd, n_head, n_kv, lens, hint):
    """Edges of tiles and runs, lengths of their own, hints that are too small or too large, cache rows behind the last position that hold no numbers, again on
    used workspaces.  Bound as for the panel kernel: one rounding of the weights, one of the result."""
    import torch
    M, max_seq = len(lens), max(lens) + 70
    g = torch.Generator(device="cuda")
    g.manual_seed(sum(lens) + n_head)
    q = (torch.randn(M, n_head, hd, generator=g, device="cuda") * 2).bfloat16()
    k, v = (torch.randn(M, max_seq, n_kv, hd, generator=g, device="cuda").bfloat16() for _ in range(2))
    for i, n in enumerate(lens):
        k[i, n:], v[i, n:] = float("nan"), float("inf")
    pos = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device="cuda")
    out = torch.full((M, n_head, hd), 7.0, device="cuda").bfloat16()
    stride = max_seq * n_kv * hd
    torch.cuda.synchronize()
    first = None
    for split in (0, 0, 3):
        ctx.set_int("attn_split", split)
        try:
            ctx.check(ctx.lib.kf_attn_decode_gqa(ctx.h, _ptr(out), _ptr(q), _ptr(k), _ptr(v), _ptr(pos), M, n_head, n_kv, hd, max_seq, hint, stride), "gqa")
            ctx.sync()
        finally:
            ctx.set_int("attn_split", 0)
        assert ctx.get_int("attn_gqa_error") == 0
        if split == 0 and first is not None:
            assert torch.equal(out, first)
        first = out.clone() if split == 0 else first
        for i, n in enumerate(lens):
            for h in range(n_head):
                kk, vv = k[i, :n, h // (n_head // n_kv)].double(), v[i, :n, h // (n_head // n_kv)].double()
                p = torch.softmax(kk @ q[i, h].double() / hd ** 0.5, 0)
                want, mass = p @ vv, p @ vv.abs()
                err = (out[i, h].double() - want).abs()
                assert bool((err <= 2.0 ** -8 * 1.01 * (mass + want.abs()) + 1e-6).all()), (split, i, h, float((err / (mass + want.abs())).max()))


@pytest.mark.parametrize("hd,n_head,n_kv,lens", [(128, 16, 8, (700, 3, 64)), (128, 16, 8, tuple(range(1, 41))), (64, 8, 2, (9000,))])
def test_gqa_output_at_any_element(ctx, hd, n_head, n_kv, lens):
    """The result may start at an odd element (whole sequences, and runs merged by the last): the same bits as an aligned one, nothing written around it."""
    import torch
    M, max_seq = len(lens), max(lens)
    g = torch.Generator(device="cuda")
    g.manual_seed(hd + M)
    q = torch.randn(M, n_head, hd, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(M, max_seq, n_kv, hd, generator=g, device="cuda").bfloat16() for _ in range(2))
    pos = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device="cuda")
    size, got = M * n_head * hd, []
    for off in (0, 1):
        buf = torch.full((size + 8,), 7.0, device="cuda").bfloat16()
        torch.cuda.synchronize()
        ctx.check(ctx.lib.kf_attn_decode_gqa(ctx.h, _ptr(buf[off:]), _ptr(q), _ptr(k), _ptr(v), _ptr(pos), M, n_head, n_kv, hd, max_seq, max_seq - 1, max_seq * n_kv * hd), "gqa")
        ctx.sync()
        assert bool((buf[:off] == 7).all()) and bool((buf[off + size:] == 7).all())
        got.append(buf[off:off + size].clone())
    assert torch.equal(got[0], got[1])


@pytest.mark.parametrize("kind,lens", [("decode", (5000, 900)), ("decode", tuple(range(1, 41))), ("prefill", (700,))])
def test_attention_wait_that_runs_out(ctx, kind, lens):
    """One thread block loads nothing, its waits end after 2 ms: the call that synchronises (or the next attention call) says so, once, and the call after that has
    the bits of the one before: no arrival of the other blocks is left counted."""
    import torch
    lib, hd, n_head, n_kv, n = ctx.lib, 128, 16, 8, len(lens)
    M, max_seq = (n, max(lens)) if kind == "decode" else (lens[0], lens[0])
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    q = torch.randn(M, n_head, hd, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(n, max_seq, n_kv, hd, generator=g, device="cuda").bfloat16() for _ in range(2))
    pos = torch.tensor([x - 1 for x in lens] if kind == "decode" else list(range(M)), dtype=torch.int32, device="cuda")
    out = torch.zeros(M, n_head, hd, device="cuda").bfloat16()
    torch.cuda.synchronize()

    def call():
        if kind == "decode":
            return lib.kf_attn_decode_gqa(ctx.h, _ptr(out), _ptr(q), _ptr(k), _ptr(v), _ptr(pos), M, n_head, n_kv, hd, max_seq, max_seq - 1, max_seq * n_kv * hd)
        return lib.kf_attn_prefill(ctx.h, _ptr(out), _ptr(q), _ptr(k), _ptr(v), _ptr(pos), M, n_head, n_kv, hd, max_seq)

    key = "attn_gqa_error" if kind == "decode" else "attn_tc_error"
    assert call() == 0 and lib.kf_ctx_sync(ctx.h) == 0
    good = out.clone()
    torch.cuda.synchronize()
    for told_by in ("sync", "call"):
        ctx.set_int("attn_wait_us", 2000), ctx.set_int("attn_drop", 1)
        try:
            assert call() == 0
        finally:
            ctx.set_int("attn_wait_us", 0), ctx.set_int("attn_drop", 0)
        assert ctx.get_int(key) == 1
        assert (lib.kf_ctx_sync(ctx.h) if told_by == "sync" else call()) != 0
        assert b"wait ran out" in lib.kf_last_error(ctx.h)
        assert ctx.get_int(key) == 0 and lib.kf_ctx_sync(ctx.h) == 0
        out.zero_()
        torch.cuda.synchronize()
        assert call() == 0 and lib.kf_ctx_sync(ctx.h) == 0
        assert torch.equal(out, good)


@pytest.mark.parametrize("split", [0, 3])
@pytest.mark.parametrize("lens", [(70, 0, 300, 1), (0,), tuple(i % 5 * 30 for i in range(40))])
def test_gqa_sequence_without_positions(ctx, lens, split):
    """Position -1: no key, so the softmax has no value; the rows are written all the same (not a number), those of the other sequences are right."""
    import torch
    hd, n_head, n_kv, M, max_seq = 128, 16, 8, len(lens), 320
    g = torch.Generator(device="cuda")
    g.manual_seed(M)
    q = torch.randn(M, n_head, hd, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(M, max_seq, n_kv, hd, generator=g, device="cuda").bfloat16() for _ in range(2))
    pos = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device="cuda")
    out = torch.full((M, n_head, hd), 7.0, device="cuda").bfloat16()
    torch.cuda.synchronize()
    ctx.set_int("attn_split", split)
    try:
        ctx.check(ctx.lib.kf_attn_decode_gqa(ctx.h, _ptr(out), _ptr(q), _ptr(k), _ptr(v), _ptr(pos), M, n_head, n_kv, hd, max_seq, max(lens), max_seq * n_kv * hd), "gqa")
        ctx.sync()
    finally:
        ctx.set_int("attn_split", 0)
    for i, n in enumerate(lens):
        if n == 0:
            assert bool(out[i].isnan().all())
            continue
        kk, vv = (t[i, :n].double().repeat_interleave(n_head // n_kv, 1) for t in (k, v))
        p = torch.softmax(torch.einsum("thd,hd->ht", kk, q[i].double()) / hd ** 0.5, -1)
        want, mass = torch.einsum("ht,thd->hd", p, vv), torch.einsum("ht,thd->hd", p, vv.abs())
        assert bool(((out[i].double() - want).abs() <= 2.0 ** -8 * 1.01 * (mass + want.abs()) + 1e-6).all())


@pytest.mark.parametrize("split", [0, 3])
@pytest.mark.parametrize("lens", [(700, 129, 400), tuple(129 + i for i in range(40))])
@pytest.mark.parametrize("gone", [(0, 16), (0, 64), (64, 128), (17, 111)])
def test_gqa_scores_of_minus_infinity(ctx, lens, split, gone):
    """Positions whose scores are -inf, all of a warp's or of a run's first ones among them: their weights are 0, the others count."""
    import torch
    hd, n_head, n_kv, M, max_seq = 128, 16, 8, len(lens), max(lens)
    g = torch.Generator(device="cuda")
    g.manual_seed(M + gone[1])
    q = torch.randn(M, n_head, hd, generator=g, device="cuda").bfloat16()
    q[..., 0] = q[..., 0].abs() + 0.25
    k, v = (torch.randn(M, max_seq, n_kv, hd, generator=g, device="cuda").bfloat16() for _ in range(2))
    k[:, gone[0]:gone[1], :, 0] = float("-inf")
    pos = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device="cuda")
    out = torch.full((M, n_head, hd), 7.0, device="cuda").bfloat16()
    torch.cuda.synchronize()
    ctx.set_int("attn_split", split)
    try:
        ctx.check(ctx.lib.kf_attn_decode_gqa(ctx.h, _ptr(out), _ptr(q), _ptr(k), _ptr(v), _ptr(pos), M, n_head, n_kv, hd, max_seq, max_seq - 1, max_seq * n_kv * hd), "gqa")
        ctx.sync()
    finally:
        ctx.set_int("attn_split", 0)
    for i, n in enumerate(lens):
        at = torch.tensor([t for t in range(n) if not gone[0] <= t < gone[1]], device="cuda")
        kk, vv = (t[i, at].double().repeat_interleave(n_head // n_kv, 1) for t in (k, v))
        p = torch.softmax(torch.einsum("thd,hd->ht", kk, q[i].double()) / hd ** 0.5, -1)
        want, mass = torch.einsum("ht,thd->hd", p, vv), torch.einsum("ht,thd->hd", p, vv.abs())
        assert bool(((out[i].double() - want).abs() <= 2.0 ** -8 * 1.01 * (mass + want.abs()) + 1e-6).all()), i


def test_maps_of_steps_leave_those_of_weights(ctx):
    """Steps of ever new buffers (the cache of a sequence moves on by 16 bytes each time) make new tensor maps; those of a weight stay."""
    import torch
    hd, n = 128, 3000
    w = make_q(ctx, kf.KF_T_Q4, 256, 512)[0]
    x = kf.fill_normal(ctx, 16 * 512, 7, 1.0)
    kf.linear(ctx, w, x, 16)
    held = ctx.get_int("tmap_weights")
    assert held > 0
    q, out = torch.ones(1, 1, hd, device="cuda").bfloat16(), torch.zeros(1, 1, hd, device="cuda").bfloat16()
    kv = torch.ones(8 * n + 4 * hd, device="cuda").bfloat16()
    pos = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    for i in range(n):
        p = _ptr(kv) + 16 * i
        ctx.check(ctx.lib.kf_attn_decode_gqa(ctx.h, _ptr(out), _ptr(q), p, p + 16, _ptr(pos), 1, 1, 1, hd, 2, 1, 0), "gqa")
    kf.linear(ctx, w, x, 16)
    ctx.sync()
    assert ctx.get_int("tmap_weights") == held
    assert bool((out == 1).all())


# ---------------------------------------------------------------------------------------------- tile matmul over expert-sorted slots
@pytest.mark.parametrize("N,K", [(64, 64), (65, 72), (8, 8), (130, 200), (192, 448), (33, 512), (257, 320), (1602, 72), (1727, 200), (3300, 328)])
@pytest.mark.parametrize("counts", [(64, 0, 1, 63, 65, 17), (200, 3, 0, 0, 1, 0), (16, 16, 16, 16, 16, 16)])
@pytest.mark.parametrize("shift", [0, 1])
def test_grouped_tiles(ctx, N, K, counts, shift):
    """Ragged outputs, reductions and slot tiles, empty experts, gathered rows, weights that do not start on 16 bytes; outputs in 64 x 64 tiles (up to 257: fewer
    tiles than SMs; 1602 with groups of 16: no more than twice as many) and in 128 x 64.  Products are exact in fp32 and the sums fp32:
    2^-24 * K terms of the rms, stated as 1e-5; the gate / up form rounds its result to bf16 once (2^-8)."""
    import torch
    torch.backends.cuda.matmul.allow_tf32 = False
    g = torch.Generator(device="cuda")
    g.manual_seed(N * K + sum(counts))
    X, slots, M = len(counts), sum(counts), 50
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    flat = [torch.randn(X * N * K + shift, generator=g, device="cuda").bfloat16()[shift:].view(X, N, K) for _ in range(2)]
    tabs = [torch.tensor([t[e].data_ptr() for e in range(X)], dtype=torch.int64, device="cuda") for t in flat]
    group = torch.repeat_interleave(torch.arange(X), torch.tensor(counts)).int().cuda()
    off = torch.cumsum(torch.tensor((0,) + counts), 0).int().cuda()
    src = torch.randint(0, M, (slots,), generator=g, device="cuda", dtype=torch.int32)
    y, h = torch.full((slots, N), 9.0, device="cuda"), torch.full((slots, N), 9.0, device="cuda").bfloat16()
    torch.cuda.synchronize()
    ctx.check(ctx.lib.kf_linear_grouped(ctx.h, _ptr(y), N, _ptr(tabs[0]), None, X, N, K, _ptr(x), 0, K, _ptr(off), _ptr(group), _ptr(src), slots), "single")
    ctx.check(ctx.lib.kf_linear_grouped(ctx.h, _ptr(h), N, _ptr(tabs[0]), _ptr(tabs[1]), X, N, K, _ptr(x), 0, K, _ptr(off), _ptr(group), _ptr(src), slots), "dual")
    ctx.sync()
    xs = x[src.long()].double()
    a, u = (torch.einsum("sk,snk->sn", xs, t[group.long()].double()) for t in flat)
    tiny = 1e-5 * float(a.square().mean().sqrt())
    assert bool(((y.double() - a).abs() <= tiny).all())
    want = a * torch.sigmoid(a) * u
    assert bool(((h.double() - want).abs() <= 2.0 ** -8 * 1.01 * want.abs() + tiny * (1 + a.abs() + u.abs())).all())


# ---------------------------------------------------------------------------------------------- RMSNorm inside the skinny matmul
@pytest.mark.parametrize("typ", [kf.KF_T_Q4, kf.KF_T_Q2, kf.KF_T_BF16])
@pytest.mark.parametrize("M", [2, 3, 4, 7, 8, 9, 15, 17, 32, 33, 64])
@pytest.mark.parametrize("K", [256, 1152, 4096])
def test_norm_of_several_tokens(ctx, typ, M, K):
    """The sums of the tokens are formed eight at a time, each in the order of kf_rmsnorm: the fused call has the bits of the two calls."""
    x, nw = kf.fill_normal(ctx, M * K, M * K, 2.0), kf.fill_normal(ctx, K, 3, 0.5)
    xn = kf.rmsnorm(ctx, x, nw, M, K, 1e-6)
    if typ == kf.KF_T_BF16:
        ws = [kf.QTensor.from_packed(ctx, ol.fill_normal(n * K, n, 0.02).view(np.uint8), None, n, K, typ) for n in (256, 128)]
    else:
        ws = [make_q(ctx, typ, n, K, n)[0] for n in (256, 128)]
    for a, b in zip(kf.rmsnorm_linear(ctx, ws, x, nw, M, 1e-6), kf.linear_multi(ctx, ws, xn, M)):
        assert np.array_equal(a.numpy(np.uint16), b.numpy(np.uint16))


@pytest.mark.parametrize("typ", [kf.KF_T_Q4, kf.KF_T_SIGN, kf.KF_T_BINARY])
@pytest.mark.parametrize("M,K", [(9, 128), (33, 2048), (10, 2176), (17, 4224), (66, 8192), (11, 8320)])
def test_norm_in_front_of_panels(ctx, typ, M, K):
    """RMSNorm written in the weights' k order has the bits of RMSNorm and the reordering, with rows that stay in registers (up to 8192) and that do not."""
    x, nw = kf.fill_normal(ctx, M * K, M * K, 2.0), kf.fill_normal(ctx, K, 3, 0.5)
    xn = kf.rmsnorm(ctx, x, nw, M, K, 1e-6)
    ws = [make_q(ctx, typ, n, K, n)[0] for n in (256, 128)]
    for a, b in zip(kf.rmsnorm_linear(ctx, ws, x, nw, M, 1e-6), kf.linear_multi(ctx, ws, xn, M)):
        assert np.array_equal(a.numpy(np.uint16), b.numpy(np.uint16))


@pytest.mark.parametrize("hd,n_head,n_kv,M", [(128, 32, 8, 300), (128, 6, 3, 1001), (64, 5, 1, 800), (64, 14, 2, 513)])
@pytest.mark.parametrize("norm", [True, False])
def test_qknorm_rows_per_warp(ctx, hd, n_head, n_kv, M, norm):
    """Four rows of a token per warp give the bits of one row per warp (calls of 16 tokens)."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(M)
    q, k, v = (torch.randn(M, n, hd, generator=g, device="cuda").bfloat16() for n in (n_head, n_kv, n_kv))
    w = [torch.randn(hd, generator=g, device="cuda").bfloat16() for _ in range(2)]
    table = torch.randn(M + 40, hd, generator=g, device="cuda")
    pos = torch.randperm(M + 40, generator=g, device="cuda")[:M].int()
    outs, used = [], M // 16 * 16
    for step in (used, 16):
        qq, kc, vc = q.clone(), torch.zeros(M + 40, n_kv, hd, device="cuda").bfloat16(), torch.zeros(M + 40, n_kv, hd, device="cuda").bfloat16()
        torch.cuda.synchronize()
        for m in range(0, used, step):
            ctx.check(ctx.lib.kf_qknorm_rope_kvappend(ctx.h, _ptr(qq[m:]), _ptr(k[m:]), _ptr(v[m:]), _ptr(w[0]) if norm else None, _ptr(w[1]) if norm else None, _ptr(kc), _ptr(vc),
                                                      _ptr(table), _ptr(pos[m:]), step, n_head, n_kv, hd, M + 40, 1e-6, 0), "qknorm")
        ctx.sync()
        outs.append((qq, kc, vc))
    for a, b in zip(*outs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("hd,n_head,n_kv", [(128, 4, 2), (64, 3, 1)])
@pytest.mark.parametrize("M", [1, 5, 16])
@pytest.mark.parametrize("odd", ["none", "q", "k", "v", "qw", "kw", "kc", "vc", "stride"])
def test_qknorm_at_any_element(ctx, hd, n_head, n_kv, M, odd):
    """One operand, or the sequences of the cache, an odd number of elements on.  The fp32 sums of squares differ in their order from the oracle's (2^-20 of the norm),
    which may move a normalised value over a rounding edge: one bf16 step (2^-7 at most) of either term of the rotation, and one of the result.  V is copied."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(M * hd)
    rows = 7
    stride = rows * n_kv * hd + (odd == "stride")

    def at(name, n, values=None):
        t = (torch.zeros(n + 1, device="cuda") if values is None else values).bfloat16()
        return t[1:] if odd == name else t[:n]
    rand = lambda name, n: at(name, n, torch.randn(n + 1, generator=g, device="cuda"))  # noqa: E731
    q, k, v, qw, kw = rand("q", M * n_head * hd), rand("k", M * n_kv * hd), rand("v", M * n_kv * hd), rand("qw", hd), rand("kw", hd)
    kc, vc = at("kc", M * stride), at("vc", M * stride)
    table = torch.randn(rows, hd // 2, 2, generator=g, device="cuda")
    pos = torch.randint(0, rows, (M,), generator=g, device="cuda", dtype=torch.int32)
    q0 = q.clone()
    torch.cuda.synchronize()
    ctx.check(ctx.lib.kf_qknorm_rope_kvappend(ctx.h, _ptr(q), _ptr(k), _ptr(v), _ptr(qw), _ptr(kw), _ptr(kc), _ptr(vc), _ptr(table), _ptr(pos), M, n_head, n_kv, hd, rows,
                                              1e-6, stride), "qknorm")
    ctx.sync()
    c, s = (table[pos.long(), :, i].double()[:, None] for i in (0, 1))

    def check(got, x, w, heads):
        x = x.view(M, heads, hd).double()
        n = (x * torch.rsqrt(x.square().mean(2, keepdim=True) + 1e-6) * w.double()).bfloat16().double()
        a, b = n[:, :, :hd // 2], n[:, :, hd // 2:]
        want, size = torch.cat([a * c - b * s, a * s + b * c], 2), torch.cat([(a * c).abs() + (b * s).abs(), (a * s).abs() + (b * c).abs()], 2)
        assert bool(((got.view(M, heads, hd).double() - want).abs() <= 2.0 ** -7 * (size + want.abs())).all())
    check(q, q0, qw, n_head)
    kept = [torch.stack([t[m * stride:m * stride + rows * n_kv * hd].view(rows, n_kv * hd)[int(pos[m])] for m in range(M)]) for t in (kc, vc)]
    check(kept[0], k, kw, n_kv)
    assert torch.equal(kept[1].reshape(-1), v)
    assert int((vc != 0).sum()) == int((v != 0).sum())


# ---------------------------------------------------------------------------------------------- routing of a panel, weighted sum of the experts
@pytest.mark.parametrize("M,E,top,full", [(33, 8, 8, 0), (300, 7, 2, 1), (512, 64, 6, 0), (129, 256, 4, 1), (129, 257, 4, 1), (70, 300, 40, 0), (2049, 33, 1, 0), (5, 64, 6, 1)])
def test_panel_routing(ctx, M, E, top, full):
    """Ties, rows of -inf, more outputs than a warp's registers hold, more choices than lanes, one block and panels; whole numbers are exact, a weight is
    one expf (2 units) over a sum of up to E of them: 1e-5."""
    rng = np.random.default_rng(M + E)
    lg, bias = np.round(rng.standard_normal((M, E + 3)) * 8).astype(np.float32) / 4, np.round(rng.standard_normal(E) * 4).astype(np.float32) / 4
    lg[1, top:E] = -np.inf
    n = M * top
    idx, wgt, offs, es, sr, sg, work = (ctx.zeros(4 * k) for k in (n, n, E + 1, n, n, n, 2 * n + E))
    lgd, bd = ctx.array(lg), ctx.array(ol.f32_to_bf16(bias))
    ctx.check(ctx.lib.kf_moe_route_ex(ctx.h, idx.ptr, wgt.ptr, offs.ptr, es.ptr, sr.ptr, sg.ptr, work.ptr, lgd.ptr, E + 3, bd.ptr, M, E, top, full), "route")
    v = (lg[:, :E] + bias).astype(np.float64)
    want = np.argsort(-v, axis=1, kind="stable")[:, :top]
    gi = idx.numpy(np.int32, (M, top))
    assert np.array_equal(gi, want)
    chosen = np.exp(np.take_along_axis(v, want, 1) - v.max(1, keepdims=True))
    den = np.exp(v - v.max(1, keepdims=True)).sum(1, keepdims=True) if full else chosen.sum(1, keepdims=True)
    assert np.allclose(wgt.numpy(np.float32, (M, top)), chosen / den, rtol=1e-5, atol=1e-30)
    flat = gi.reshape(-1)
    order = np.argsort(flat, kind="stable")
    assert np.array_equal(offs.numpy(np.int32, (E + 1,)), np.concatenate([[0], np.cumsum(np.bincount(flat, minlength=E))]))
    assert np.array_equal(es.numpy(np.int32, (n,))[order], np.arange(n))
    assert np.array_equal(sr.numpy(np.int32, (n,)), order // top) and np.array_equal(sg.numpy(np.int32, (n,)), flat[order])


@pytest.mark.parametrize("M,X,spare,top", [(200, 12, 4, 5), (513, 30, 34, 2), (100, 3, 61, 8)])
def test_panel_routing_past_the_experts(ctx, M, X, spare, top):
    """Entries of outputs beyond the experts take no slot; as many slots stay free behind the last expert."""
    n, E = M * top, X + spare
    idx, wgt, offs, es, sr, sg, work = (ctx.zeros(4 * k) for k in (n, n, E + 1, n, n, n, 2 * n + E))
    lgd = ctx.array(np.random.default_rng(M).standard_normal((M, E)).astype(np.float32))
    ctx.check(ctx.lib.kf_moe_route_softmax_grouped(ctx.h, idx.ptr, wgt.ptr, offs.ptr, es.ptr, sr.ptr, sg.ptr, work.ptr, lgd.ptr, E, None, M, X, spare, top, 1, 1), "route")
    flat = idx.numpy(np.int32, (n,))
    real = int((flat < X).sum())
    order = np.argsort(np.minimum(flat, X), kind="stable")
    assert np.array_equal(offs.numpy(np.int32)[:X + 1], np.concatenate([[0], np.cumsum(np.bincount(flat[flat < X], minlength=X))]))
    assert np.array_equal(es.numpy(np.int32, (n,))[order], np.where(np.arange(n) < real, np.arange(n), -1))
    assert np.array_equal(sr.numpy(np.int32, (n,)), np.where(np.arange(n) < real, order // top, 0))
    assert np.array_equal(sg.numpy(np.int32, (n,)), np.where(np.arange(n) < real, flat[order], -1))


@pytest.mark.parametrize("M,dim,top,shift", [(1, 8, 1, 0), (3, 1028, 7, 0), (3, 1028, 8, 1), (5, 1023, 9, 0), (40, 2304, 17, 0), (2, 3, 2, 0)])
@pytest.mark.parametrize("shared,accumulate", [(0, 0), (1, 0), (2, 1)])
def test_combine(ctx, M, dim, top, shift, shared, accumulate):
    """Rows that are and are not made of 16-byte pieces, more choices than one batch holds; fp32 sums of top + 2 terms: 2^-24 (top + 2) of their masses."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(M * dim + top)
    y = torch.randn(M * top * dim + shift, generator=g, device="cuda")[shift:].view(M * top, dim)
    w, sh, sg, out = torch.rand(M, top, generator=g, device="cuda"), torch.randn(M, dim, generator=g, device="cuda"), torch.randn(M, 2, generator=g, device="cuda"), torch.randn(M, dim, generator=g, device="cuda")
    slot = torch.randperm(M * top, generator=g, device="cuda").int()
    before = out.double()
    torch.cuda.synchronize()
    ctx.check(ctx.lib.kf_moe_combine_ex(ctx.h, _ptr(out), _ptr(y), _ptr(slot), _ptr(w), _ptr(sh) if shared else None, _ptr(sg) if shared == 2 else None, 2, M, dim, top,
                                        accumulate), "combine")
    ctx.sync()
    terms = [w[:, j, None].double() * y[slot.view(M, top)[:, j].long()].double() for j in range(top)]
    if shared:
        terms.append((torch.sigmoid(sg[:, :1].double()) if shared == 2 else 1.0) * sh.double())
    if accumulate:
        terms.append(before)
    mass = sum(t.abs() for t in terms)
    assert bool(((out.double() - sum(terms)).abs() <= 2.0 ** -24 * (top + 6) * mass + 1e-30).all())


@pytest.mark.parametrize("M,dim", [(9, 64), (100, 1023)])
def test_router_row_that_is_no_number(ctx, M, dim):
    """A token whose router logits are all NaN chooses nothing: its result is NaN, not a sum of nothing, and the other tokens do not notice."""
    E, top, bad = 8, 4, 3
    n = M * top
    idx, wgt, offs, es, sr, sg, work = (ctx.zeros(4 * k) for k in (n, n, E + 1, n, n, n, 2 * n + E))
    lg = np.random.default_rng(M).standard_normal((M, E)).astype(np.float32)
    lg[bad] = np.nan
    lgd, out = ctx.array(lg), ctx.zeros(4 * M * dim)
    y = np.random.default_rng(dim).standard_normal((n, dim)).astype(np.float32)
    yd = ctx.array(y)
    ctx.check(ctx.lib.kf_moe_route(ctx.h, idx.ptr, wgt.ptr, offs.ptr, es.ptr, sr.ptr, sg.ptr, work.ptr, lgd.ptr, E, None, M, E, top), "route")
    ctx.check(ctx.lib.kf_moe_combine(ctx.h, out.ptr, yd.ptr, es.ptr, wgt.ptr, None, None, 0, M, dim, top), "combine")
    got, slot, w = out.numpy(np.float32, (M, dim)), es.numpy(np.int32, (M, top)), wgt.numpy(np.float32, (M, top)).astype(np.float64)
    assert np.isnan(got[bad]).all() and (slot[bad] == -1).all()
    for m in range(M):
        if m != bad:
            terms = w[m, :, None] * y[slot[m]].astype(np.float64)
            assert (np.abs(got[m] - terms.sum(0)) <= 2.0 ** -24 * (top + 6) * np.abs(terms).sum(0) + 1e-30).all()
