"""Kernels at the edges of their tiles and of the rules that choose them, against plain PyTorch in fp32 or fp64.

Tolerances: a bf16 result of an fp32 accumulation is off by at most half a unit in the last place, 2^-8 of its value, plus
the accumulation's own error; `_close` allows 2^-12 of the largest value for the latter."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

DEV = "cuda"
BF16 = torch.bfloat16


def _close(got, ref, slack=2.0 ** -12, rel=2.0 ** -8):
    got, ref = got.double(), ref.double()
    assert got.shape == ref.shape
    bad = (got - ref).abs() > ref.abs() * rel + float(ref.abs().max()) * slack
    assert not bool(bad.any()), float((got - ref).abs().max())


def _rand(*shape, scale=0.5, dtype=BF16, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed + sum(shape))
    return (torch.randn(*shape, generator=g, device=DEV) * scale).to(dtype)


# m, n, k, and whether CTA pairs run it.  Single CTAs: one tile, ragged last tiles, several tiles, a K of one block and with a
# remainder.  Pairs: N and M that end inside a tile and inside a 64-column box, rows that fill one CTA of a pair's last tile only,
# K of one block, of less and with a remainder, fewer tiles than two per pair and many.  And the rule's lines from both sides.
GEMM = [(256, 256, 64, 0), (257, 512, 72, 0), (300, 1000, 200, 0), (512, 264, 1024, 0), (4100, 1032, 136, 0), (4096, 1288, 88, 0),
        (20000, 1024, 264, 1), (8200, 1032, 64, 1), (4100, 1800, 72, 1), (4100, 1544, 72, 0), (1232, 30536, 136, 1), (16008, 392, 48, 1), (5900, 1000, 320, 1),
        (2048, 3072, 8, 1), (12000, 384, 264, 0), (14000, 384, 264, 1), (16384, 320, 256, 0), (16384, 320, 264, 1)]


@pytest.mark.parametrize("m,n,k,pair", GEMM)
@pytest.mark.parametrize("act", [None, "relu", "gelu"])
def test_linear_products(m, n, k, pair, act):
    from tips_b200.ops import base
    from tips_b200.ops.linear import gemm_nn, gemm_status, gemm_tn
    assert base.K().tipsk_gemm_prefers_pair(0, m, n, k) == base.K().tipsk_gemm_prefers_pair(1, m, n, k) == pair
    a, b, bias = _rand(m, k), _rand(n, k, seed=1), _rand(n, seed=2)
    ref_pre = a.double() @ b.double().t() + bias.double()
    ref = {None: lambda t: t, "relu": F.relu, "gelu": F.gelu}[act](ref_pre)
    y, pre = gemm_tn(a, b, bias, act, want_pre=True)
    _close(pre, ref_pre)
    _close(y, ref)
    _close(gemm_tn(a, b, bias, act), ref)
    if act is None:
        nn = ref_pre - bias.double()
        bt = b.t().contiguous()
        _close(gemm_nn(a, bt), nn)
        into = _rand(m, n, seed=3)
        want = into.double() + nn
        # the product is rounded to bf16 before the addition, and the sum once more
        _close(gemm_nn(a, bt, into=into), want, slack=2.0 ** -8)
    assert gemm_status() == 0


# rows, outputs, inputs, and whether the pair kernel runs it (1) or the convolution's: each line of the rule from both sides,
# ragged last tiles and a K that is no multiple of a block, unsplit and split
WEIGHT_GRADIENT = [(16, 128, 128, 1), (16, 64, 64, 0), (256, 192, 128, 1), (257, 192, 128, 0), (77, 256, 128, 1), (1024, 1024, 256, 1),
                   (1025, 1024, 256, 0), (1232, 320, 1024, 0), (4096, 1024, 1024, 1), (8200, 4096, 192, 0), (8200, 320, 1984, 1),
                   (32768, 64, 256, 1), (32769, 64, 256, 0), (32769, 128, 256, 1), (65537, 256, 256, 0), (65537, 512, 512, 1),
                   (12544, 64, 64, 0), (2000, 512, 1728, 1)]


@pytest.mark.parametrize("rows,n,k,pair", WEIGHT_GRADIENT)
def test_weight_gradient_in_bf16(rows, n, k, pair):
    from tips_b200.ops import base
    from tips_b200.ops.linear import _weight_grad, gemm_status
    assert base.K().tipsk_gemm_prefers_pair(2, n, k, rows) == pair
    dz, x = _rand(rows, n), _rand(rows, k, seed=1)
    ref = dz.double().t() @ x.double()
    _close(_weight_grad(dz, x, BF16), ref)
    _close(_weight_grad(dz, x), ref)
    assert gemm_status() == 0


@pytest.mark.parametrize("m,n,k", [(64, 64, 4096), (1232, 1024, 30528), (256, 2048, 4104), (300, 72, 8200)])
def test_split_contraction(m, n, k):
    from tips_b200.ops import base
    from tips_b200.ops.linear import gemm_nn, gemm_status, gemm_tn
    assert base.K().tipsk_gemm_splits(m, n, k) > 1
    a, b, bias = _rand(m, k, scale=0.1), _rand(n, k, scale=0.1, seed=1), _rand(n, seed=2)
    ref = a.double() @ b.double().t()
    y, pre = gemm_tn(a, b, bias, "gelu", want_pre=True)
    _close(pre, ref + bias.double())
    _close(y, F.gelu(ref + bias.double()))
    bt = b.t().contiguous()
    _close(gemm_nn(a, bt), ref)
    into = _rand(m, n, seed=3)
    want = into.double() + ref
    _close(gemm_nn(a, bt, into=into), want)
    assert gemm_status() == 0


# n, h, w, cin, cout, and which kernel that is (1: two output rows per MMA).  Widths at both ends of the row-pair kernel's
# range, odd heights, a short last unit, one row pair per unit, more units than SMs and one more; the tap kernel beside the
# lines of the rule and with several channel blocks and output tiles.
CONV3X3 = [(43, 56, 56, 64, 64, 1), (50, 55, 56, 64, 64, 1), (74, 8, 62, 64, 64, 1), (149, 31, 33, 64, 64, 1), (150, 9, 28, 64, 64, 1),
           (75, 28, 28, 64, 64, 1), (300, 2, 62, 64, 64, 1), (300, 12, 3, 64, 64, 0), (150, 9, 9, 64, 64, 0), (149, 5, 63, 64, 64, 0),
           (150, 100, 5, 64, 64, 1), (200, 84, 1, 64, 64, 0), (36, 8, 62, 64, 64, 0), (149, 28, 28, 128, 128, 0), (75, 17, 28, 64, 192, 0), (43, 56, 56, 192, 64, 0),
           (297, 9, 9, 64, 128, 0), (601, 5, 24, 192, 64, 0)]


@pytest.mark.parametrize("n,h,w,cin,cout,path", CONV3X3)
def test_conv3x3(n, h, w, cin, cout, path):
    from tips_b200.ops.conv import conv2d_dgrad, conv2d_forward, conv2d_wgrad
    from tips_b200.ops import base
    assert base.K().tipsk_conv2d_path(0, n, h, w, cin, cout) == path == base.K().tipsk_conv2d_path(1, n, h, w, cin, cout)
    x = _rand(n, cin, h, w).contiguous(memory_format=torch.channels_last)
    wgt = _rand(cout, 3, 3, cin, scale=1.0 / (3 * cin ** 0.5), seed=1)
    dy = _rand(n, cout, h, w, seed=2).contiguous(memory_format=torch.channels_last)
    stats = torch.zeros(2, cout, device=DEV)
    _, y = conv2d_forward(x, wgt, 1, 1, stats)
    xr, wr = x.float().requires_grad_(), wgt.float().permute(0, 3, 1, 2).contiguous().requires_grad_()
    torch.backends.cudnn.allow_tf32, before = False, torch.backends.cudnn.allow_tf32
    try:
        ref = F.conv2d(xr, wr, padding=1)
        ref.backward(dy.float())
    finally:
        torch.backends.cudnn.allow_tf32 = before
    _close(y, ref.detach())
    yf = y.double()
    assert torch.allclose(stats[0].double(), yf.sum((0, 2, 3)), rtol=1e-4, atol=1e-3 * float(yf.abs().sum((0, 2, 3)).max()))
    assert torch.allclose(stats[1].double(), (yf * yf).sum((0, 2, 3)), rtol=1e-4)
    _close(conv2d_dgrad(dy, wgt, tuple(x.shape), 1, 1), xr.grad)
    into = _rand(n, cin, h, w, seed=4).contiguous(memory_format=torch.channels_last)
    want = into.double() + xr.grad.double()
    _close(conv2d_dgrad(dy, wgt, tuple(x.shape), 1, 1, into=into), want, slack=2.0 ** -8)
    _close(conv2d_wgrad(x, dy, (cout, 3, 3, cin), 1, 1), wr.grad.permute(0, 2, 3, 1))
    assert base.K().tipsk_conv_status() == 0


# a last unit of one row, of all its rows, and images one unit high; the pitch beyond the width by 2, 4 and 8 pixels
@pytest.mark.parametrize("n,h,w", [(100, 17, 28), (50, 56, 56), (300, 3, 62), (43, 55, 56)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_weight_gradient_of_non_finite_pixels(n, h, w, value):
    """A pixel that is not finite reaches exactly the taps that read it."""
    from tips_b200.ops.conv import conv2d_wgrad
    from tips_b200.ops import base
    x = _rand(n, 64, h, w)
    # first and last column, last row, a corner, inside; each in a channel of its own
    for ch, (i, j) in enumerate([(1, 0), (h // 2, w - 1), (h - 1, w // 2), (h - 1, w - 1), (h // 2, w // 2), (0, 0)]):
        x[n // 2, 9 * ch, i, j] = value
        x[n - 1, 9 * ch, i, j] = -value
    x = x.contiguous(memory_format=torch.channels_last)
    dy = _rand(n, 64, h, w, seed=1).contiguous(memory_format=torch.channels_last)
    got = conv2d_wgrad(x, dy, (64, 3, 3, 64), 1, 1).permute(0, 3, 1, 2).double()
    xd, dyd = x.double(), dy.double()
    for r in range(3):
        for s in range(3):
            i0, i1, j0, j1 = max(0, 1 - r), h - max(0, r - 1), max(0, 1 - s), w - max(0, s - 1)
            part = dyd[:, :, i0:i1, j0:j1].permute(1, 0, 2, 3).reshape(64, -1)
            ref = part @ xd[:, :, i0 + r - 1:i1 + r - 1, j0 + s - 1:j1 + s - 1].permute(0, 2, 3, 1).reshape(-1, 64)
            fin = torch.isfinite(ref)
            assert bool(fin.any()) and torch.equal(got[:, :, r, s].isfinite(), fin), (r, s)
            assert torch.equal(got[:, :, r, s].isinf(), ref.isinf())
            _close(torch.where(fin, got[:, :, r, s], 0.0), torch.where(fin, ref, 0.0))
    assert base.K().tipsk_conv_status() == 0


def test_weight_gradient_of_nothing_but_nan():
    from tips_b200.ops.conv import conv2d_wgrad
    from tips_b200.ops import base
    x = _rand(43, 64, 56, 56).contiguous(memory_format=torch.channels_last)
    dy = _rand(43, 64, 56, 56, seed=1).contiguous(memory_format=torch.channels_last)
    x[:, 5:40] = float("nan")
    got = conv2d_wgrad(x, dy, (64, 3, 3, 64), 1, 1).isnan()
    assert bool(got[..., 5:40].all()) and not bool(got[..., :5].any()) and not bool(got[..., 40:].any())
    assert base.K().tipsk_conv_status() == 0


# the smallest pixel counts that take several taps per tile (24 steps of 64 per CTA) and one below, with one and two tiles of
# output channels, ragged boxes and stride 2; few pixels: one tap per tile
@pytest.mark.parametrize("n,h,w,cout,stride,path", [(2, 6, 7, 64, 1, 0), (3, 20, 20, 256, 1, 0), (9, 15, 13, 320, 2, 0), (379, 20, 20, 64, 1, 1),
                                                    (378, 20, 20, 64, 1, 0), (95, 40, 40, 128, 1, 1), (48, 37, 43, 320, 1, 1),
                                                    (160, 71, 70, 64, 2, 1)])
def test_weight_gradient_of_64_channels_in_tap_groups(n, h, w, cout, stride, path):
    from tips_b200.ops.conv import conv2d_wgrad
    from tips_b200.ops import base
    x = _rand(n, 64, h, w).contiguous(memory_format=torch.channels_last)
    ho, wo = (h - 1) // stride + 1, (w - 1) // stride + 1
    assert base.K().tipsk_conv2d_path(2, n, ho, wo, 64, cout) == path
    dy = _rand(n, cout, ho, wo, seed=1).contiguous(memory_format=torch.channels_last)
    got = conv2d_wgrad(x, dy, (cout, 3, 3, 64), stride, 1)
    xp = F.pad(x.float(), (1, 1, 1, 1))
    dyf = dy.float().permute(0, 2, 3, 1).reshape(-1, cout)
    torch.backends.cuda.matmul.allow_tf32, before = False, torch.backends.cuda.matmul.allow_tf32
    try:
        ref = torch.stack([torch.stack([
            dyf.t() @ xp[:, :, r:r + (ho - 1) * stride + 1:stride, s:s + (wo - 1) * stride + 1:stride].permute(0, 2, 3, 1).reshape(-1, 64)
            for s in range(3)], 1) for r in range(3)], 1)
    finally:
        torch.backends.cuda.matmul.allow_tf32 = before
    assert base.K().tipsk_conv_status() == 0
    # fp32 sums of up to 200 000 products in two orders: a random walk of roundings, 2^-12 of the largest value bounds both
    _close(got, ref)


# rows of one to 128 elements share a block, from 129 on a row has blocks of its own
@pytest.mark.parametrize("n,c,h,w", [(1, 8, 1, 1), (2, 8, 2, 3), (3, 72, 5, 8), (2, 64, 31, 33), (1, 2056, 4, 4), (700, 8, 3, 3), (5, 1024, 3, 2),
                                     (5, 1032, 3, 2), (3, 8, 4, 300)])
def test_maxpool_edges(n, c, h, w):
    from tips_b200.ops.pool import max_pool_3x3_s2
    x = _rand(n, c, h, w).contiguous(memory_format=torch.channels_last).requires_grad_()
    y = max_pool_3x3_s2(x)
    xr = x.detach().float().requires_grad_()
    yr = F.max_pool2d(xr, 3, stride=2, padding=1)
    assert torch.equal(y.float(), yr)
    dy = _rand(*y.shape, seed=1).contiguous(memory_format=torch.channels_last)
    y.backward(dy)
    yr.backward(dy.float())
    _close(x.grad, xr.grad)


@pytest.mark.parametrize("src,flat", [(BF16, BF16), (torch.float32, BF16), (torch.float16, torch.float32)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_pack_many_tensors(src, flat, accumulate):
    from tips_b200.ops import base
    numels = [1, 3, 8191, 8192, 8193, 0, 40001] + [5 + i for i in range(120)]  # more than one launch takes
    offs, at = [], 0
    for i, n in enumerate(numels):
        offs.append(at)
        at += n + i % 3  # some of them not aligned to a vector
    tensors = [_rand(n, dtype=src, seed=i) for i, n in enumerate(numels)]
    buf = _rand(at, dtype=flat, seed=7)
    want = buf.float().clone()
    for t, o in zip(tensors, offs):
        v = t.float() * 0.5
        want[o:o + t.numel()] = want[o:o + t.numel()] + v if accumulate else v
    base.check(base.K().tipsk_pack(base.ptr_array(tensors), base.i64_array(offs), base.i64_array(numels), len(tensors),
                                   base.code(src), buf.data_ptr(), base.code(flat), 0.5, int(accumulate), base.stream()),
               "pack")
    assert torch.equal(buf, want.to(flat))
    back = [torch.empty_like(t) for t in tensors]
    base.check(base.K().tipsk_unpack(buf.data_ptr(), base.code(flat), base.ptr_array(back), base.i64_array(offs),
                                     base.i64_array(numels), len(back), base.code(src), 2.0, base.stream()), "unpack")
    for t, o in zip(back, offs):
        assert torch.equal(t, (buf[o:o + t.numel()].float() * 2.0).to(src))


@pytest.mark.parametrize("dtype", [BF16, torch.float32])
@pytest.mark.parametrize("rows,cols", [(1, 8), (3, 4096), (5, 4104), (700, 1000), (4, 30522), (3, 32768), (3, 32776), (4097, 64), (5000, 10),
                                       (3, 1024), (3, 1032), (3, 2056), (3, 16392)])
def test_softmax_cross_entropy_rows(dtype, rows, cols):
    from tips_b200.ops.pointwise import softmax_cross_entropy
    z = _rand(rows, cols, scale=3.0, dtype=dtype).requires_grad_()
    labels = torch.randint(0, cols, (rows,), device=DEV, generator=torch.Generator(device=DEV).manual_seed(1))
    if rows > 2:
        labels[1] = -100
    labels[0] = cols - 1
    loss = softmax_cross_entropy(z, labels)
    (loss * 3.0).backward()
    zr = z.detach().double().requires_grad_()
    ref = F.cross_entropy(zr, labels, ignore_index=-100)
    (ref * 3.0).backward()
    assert torch.allclose(loss.double(), ref.detach(), rtol=1e-5)
    # rounded once as softmax - onehot, once after the factors: twice 2^-8, their product, and fp32 terms
    _close(z.grad, zr.grad, slack=2.0 ** -18, rel=2.0 ** -7 + 2.0 ** -13)


# the row kernel and, with more than 4096 vectors per row or a ragged length, the general one; labels counted by every block and once
@pytest.mark.parametrize("rows,cols,up", [(1232, 30528, 1024.0), (1232, 30528, 65536.0), (300, 30522, 65536.0), (4097, 4096, 65536.0),
                                          (40, 32776, 65536.0)])
def test_softmax_cross_entropy_fp16_loss_scale(rows, cols, up):
    """Off-label entries of the mean's gradient are below fp16's range until the loss scale is applied."""
    from tips_b200.ops.pointwise import softmax_cross_entropy
    z = _rand(rows, cols, scale=1.0, dtype=torch.float16).requires_grad_()
    labels = torch.randint(0, cols, (rows,), device=DEV, generator=torch.Generator(device=DEV).manual_seed(1))
    labels[3] = -100
    (softmax_cross_entropy(z, labels) * up).backward()
    zr = z.detach().double()
    ref = torch.softmax(zr, 1)
    ref[torch.arange(rows, device=DEV), labels.clamp(min=0)] -= 1.0
    ref[3] = 0.0
    ref *= up / (rows - 1)
    # stored once as softmax - onehot and once more after the factor up / (rows - 1): two roundings of 2^-11 each plus fp32 terms,
    # or half a subnormal unit, 2^-25, each
    bound = ref.abs() * (2.0 ** -10 + 2.0 ** -13) + (up / (rows - 1) + 1.0) * 2.0 ** -25
    bad = (z.grad.double() - ref).abs() > bound
    assert not bool(bad.any()), float((z.grad.double() - ref).abs().max())
    off = z.grad[0].index_select(0, (labels[0] + 1 + torch.arange(cols - 1, device=DEV)) % cols)
    assert float((off == 0).float().mean()) < 0.01


@pytest.mark.parametrize("dtype", [BF16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows", [1, 7])
def test_softmax_cross_entropy_create_graph(dtype, rows):
    """A loss scale of 65536 is infinite in fp16; the gradient that it leads to is not."""
    from tips_b200.ops.pointwise import softmax_cross_entropy
    z = _rand(rows, 264, dtype=dtype).requires_grad_()
    labels = torch.arange(rows, device=DEV)
    up = torch.full((), 65536.0, device=DEV, requires_grad=True)
    (g,) = torch.autograd.grad(softmax_cross_entropy(z, labels), z, up, create_graph=True)
    zr = z.detach().double()
    ref = torch.softmax(zr, 1) - F.one_hot(labels, 264)
    ref1 = ref * 65536.0 / rows
    eps = {BF16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -20}[dtype]
    top = float(torch.finfo(dtype).max)
    ok = ref1.abs() < top * (1 - 2 * eps)  # one row's label entry, -65536 (1 - p), is in fp16's range but for the rounding
    assert bool(ok[:, rows:].all())
    # two roundings to the type (softmax - onehot, the product) and fp32 terms
    assert bool(((g.detach().double() - ref1).abs() <= ref1.abs() * (2 * eps + 2.0 ** -13) + 2.0 ** -9)[ok].all())
    (gu,) = torch.autograd.grad(g[:, rows:].float().sum(), up)  # the gradient is linear in the upstream factor
    want = ref[:, rows:].sum() / rows
    assert abs(float(gu) - float(want)) <= float(ref[:, rows:].abs().sum()) / rows * (2 * eps + 2.0 ** -13)


@pytest.mark.parametrize("layout", ["offset", "strided"])
def test_softmax_cross_entropy_saved_tensor_hooks(layout):
    """Hooks may hand the saved gradient back anywhere in memory."""
    from tips_b200.ops.pointwise import softmax_cross_entropy

    def unpack(t):
        if t.dim() != 2:
            return t
        if layout == "offset":
            return torch.empty(t.numel() + 1, dtype=t.dtype, device=DEV)[1:].view(t.shape).copy_(t)
        return torch.empty(t.shape[0], 2 * t.shape[1], dtype=t.dtype, device=DEV)[:, ::2].copy_(t)

    z = _rand(9, 64).requires_grad_()
    labels = torch.arange(9, device=DEV)
    (want,) = torch.autograd.grad(softmax_cross_entropy(z, labels), z)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
        loss = softmax_cross_entropy(z, labels)
    (got,) = torch.autograd.grad(loss, z)
    assert torch.equal(got, want)


def test_softmax_cross_entropy_without_counted_rows():
    from tips_b200.ops.pointwise import softmax_cross_entropy
    z = _rand(4, 64).requires_grad_()
    loss = softmax_cross_entropy(z, torch.full((4,), -100, device=DEV))
    loss.backward()
    assert float(loss.detach()) == 0.0 and not bool(z.grad.any())


@pytest.mark.parametrize("dtype", [BF16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,cols", [(1, 8), (31, 264), (33, 1000), (4097, 72), (1217, 4096)])  # the last: more than four blocks per SM in fp32
@pytest.mark.parametrize("act", [None, "relu", "gelu"])
def test_bias_act_backward_rows(dtype, rows, cols, act):
    from tips_b200.ops.pointwise import bias_act
    x, b = _rand(rows, cols, dtype=dtype, scale=2.0).requires_grad_(), _rand(cols, dtype=dtype, seed=1).requires_grad_()
    dy = _rand(rows, cols, dtype=dtype, seed=2)
    bias_act(x, b, act).backward(dy)
    xr, br = x.detach().double().requires_grad_(), b.detach().double().requires_grad_()
    y = xr + br
    y = F.relu(y) if act == "relu" else F.gelu(y) if act == "gelu" else y
    y.backward(dy.double())
    _close(x.grad, xr.grad)
    _close(b.grad, br.grad)


@pytest.mark.parametrize("dtype", [BF16, torch.float16])
# the groups' blocks number one per SM at most and the small ones eight: rows below and above the line between them, from
# blocks with less than one row per group to many, one to fifteen groups per block, and the longest and widest of each
@pytest.mark.parametrize("rows,cols,groups", [(1, 256, False), (14, 256, False), (2221, 256, False), (4687, 256, False), (4688, 256, True),
                                              (16383, 256, True), (16384, 256, False), (8, 1024, False), (1185, 1024, True), (1171, 1024, False),
                                              (1600, 768, True), (586, 2048, True), (301, 2048, False), (2000, 1792, True)])
def test_layer_norm_backward_groups(dtype, rows, cols, groups):
    from tips_b200.ops import base
    from tips_b200.ops.norm import layer_norm
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    blocks = min(sms, -(-rows // min(15, 768 // (cols // 8)))) if groups else min(8 * sms, -(-rows // 4))
    assert base.K().tipsk_ln_bwd_partial_rows(rows, cols, base.code(dtype)) == blocks
    x, dy = _rand(rows, cols, dtype=dtype).requires_grad_(), _rand(rows, cols, dtype=dtype, seed=1)
    w, b = (1 + _rand(cols, dtype=dtype, scale=0.1, seed=2)).requires_grad_(), _rand(cols, dtype=dtype, seed=3).requires_grad_()
    layer_norm(x, w, b).backward(dy)
    xr, wr, br = (t.detach().double().requires_grad_() for t in (x, w, b))
    F.layer_norm(xr, (cols,), wr, br).backward(dy.double())
    for got, ref in ((x.grad, xr.grad), (w.grad, wr.grad), (b.grad, br.grad)):
        _close(got, ref)


# pull: an item per lane group up to the line and per lane beyond it; push: 8, 16 and 32 items per warp; one row to 32 rows per
# warp, row lengths that fill the lanes of a group and that do not
@pytest.mark.parametrize("batch,fields,dim", [(1, 1, 4), (33, 3, 8), (2520, 26, 16), (2521, 26, 16), (480, 26, 64), (481, 26, 64), (1260, 26, 32),
                                              (1261, 26, 32), (700, 8, 144), (9, 5, 256), (1300, 26, 24), (2600, 26, 4), (300, 11, 516)])
@pytest.mark.parametrize("dtype", [BF16, torch.float32])
def test_pull_and_push_rows(batch, fields, dim, dtype):
    from tips_b200.ps.gpu import ShardedEmbedding
    rows = 3000
    t = ShardedEmbedding(fields, rows, dim, optimizer="sgd", lr=0.5, init_scale=0.1, seed=3, expected_batch=batch, device=torch.device(DEV, 0))
    g = torch.Generator(device=DEV).manual_seed(batch + dim)
    ids = torch.randint(0, rows, (batch, fields), device=DEV, generator=g)
    before = [t.local_shard(f).clone() for f in range(fields)]
    want = torch.cat([before[f][ids[:, f]] for f in range(fields)], 1)
    assert torch.equal(t.pull(ids, dtype=dtype), want.to(dtype))
    grads = _rand(batch, fields * dim, dtype=dtype)
    t.push(ids, grads, grad_scale=0.25)
    assert t.check() > 0
    for f in range(fields):
        s = torch.zeros(rows, dim, dtype=torch.float64, device=DEV)
        s.index_add_(0, ids[:, f], grads[:, f * dim:(f + 1) * dim].double())
        ref = before[f].double() - 0.5 * 0.25 * s
        # fp32 sums of a few duplicates, the product and the difference: well within 16 units in the last place of the terms
        assert torch.allclose(t.local_shard(f).double(), ref, rtol=2.0 ** -20, atol=2.0 ** -20)
    ids[0, 0], ids[batch - 1, fields - 1] = -1, rows  # rows that do not exist read as zeros and are reported
    got = t.pull(ids, dtype=dtype)
    assert not bool(got[0, :dim].any()) and not bool(got[batch - 1, -dim:].any())
    assert torch.equal(got[:, :dim][1:batch - 1], t.local_shard(0)[ids[1:batch - 1, 0]].to(dtype))
    with pytest.raises(Exception):
        t.check()
