"""tcgen05 implicit-GEMM convolution against torch.nn.functional (fp32) on the same inputs."""
import ctypes

import pytest
import torch
import torch.nn.functional as F

from lbann_b200.ops import native, nn
from lbann_b200.ops.conv import conv_fwd, pack_filter

pytestmark = pytest.mark.gpu

# the oracle (cuDNN / cuBLAS through torch) must not round its inputs to TF32
torch.backends.cudnn.allow_tf32 = False
torch.backends.cuda.matmul.allow_tf32 = False

CASES = [
    # N, C, D, H, W, K, k, pad, stride, dil
    (2, 16, 8, 8, 8, 32, 3, 1, 1, 1),
    (1, 32, 16, 16, 16, 64, 3, 1, 1, 1),
    (2, 64, 8, 8, 8, 128, 3, 1, 1, 1),
    (1, 128, 4, 8, 8, 256, 3, 1, 1, 1),
    (2, 16, 1, 28, 28, 48, 5, 2, 1, 1),
    (3, 64, 1, 14, 14, 64, 1, 0, 1, 1),
    (2, 32, 1, 30, 30, 40, 3, 1, 2, 1),
    (1, 24, 6, 10, 12, 16, 3, 2, 1, 2),
    (4, 8, 1, 7, 7, 24, 3, 1, 1, 1),
    # shapes the halo-slab kernel takes (stride 1, filter resident in shared memory)
    (1, 32, 6, 40, 64, 64, 3, 1, 1, 1),
    (2, 64, 4, 24, 32, 32, 3, 1, 1, 1),
    (1, 16, 1, 33, 50, 24, 3, 1, 1, 1),
    (1, 48, 3, 20, 28, 96, 3, 1, 1, 1),
    (1, 32, 3, 9, 130, 64, 3, 0, 1, 1),
]


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_conv_fwd(case, dtype):
    N, C, D, H, W, K, k, pad, stride, dil = case
    torch.manual_seed(0)
    ks = (1 if D == 1 else k, k, k)
    pd = (0 if D == 1 else pad, pad, pad)
    st = (1 if D == 1 else stride, stride, stride)
    dl = (1 if D == 1 else dil, dil, dil)
    x = torch.randn(N, C, D, H, W, device="cuda").to(dtype)
    w = (torch.randn(K, C, *ks, device="cuda") / (C * k * k) ** 0.5).to(dtype)
    bias = torch.randn(K, device="cuda")
    xl = x.permute(0, 2, 3, 4, 1).contiguous()
    y = conv_fwd(xl, pack_filter(w, dtype), ks, pad=pd, stride=st, dilation=dl, bias=bias,
                 out_dtype=torch.float32)
    assert native.consume_status() == 0
    ref = F.conv3d(x.float(), w.float(), bias, st, pd, dl).permute(0, 2, 3, 4, 1)
    torch.testing.assert_close(y, ref, rtol=2e-3, atol=2e-2)


def test_conv_dgrad_via_flipped_filter():
    torch.manual_seed(1)
    N, C, K, S = 2, 32, 64, 8
    x = torch.randn(N, C, S, S, S, device="cuda", requires_grad=True)
    w = (torch.randn(K, C, 3, 3, 3, device="cuda") / 30).bfloat16()
    y = F.conv3d(x, w.float(), None, 1, 1)
    dy = torch.randn_like(y).bfloat16()
    y.backward(dy.float())
    dyl = dy.permute(0, 2, 3, 4, 1).contiguous()
    dx = conv_fwd(dyl, pack_filter(w, torch.bfloat16, for_dgrad=True), 3, pad=1,
                  out_dtype=torch.float32)
    assert native.consume_status() == 0
    torch.testing.assert_close(dx, x.grad.permute(0, 2, 3, 4, 1), rtol=2e-3, atol=3e-2)


WGRAD_CASES = [
    # N, C, D, H, W, K, k, pad, stride
    (2, 16, 8, 8, 8, 32, 3, 1, 1),
    (2, 32, 8, 16, 16, 64, 3, 1, 1),
    (2, 64, 8, 8, 8, 128, 3, 1, 1),
    (1, 128, 4, 8, 8, 256, 3, 1, 1),
    (2, 16, 1, 28, 28, 48, 5, 2, 1),
    (3, 64, 1, 14, 14, 64, 1, 0, 1),
    (2, 32, 1, 30, 30, 40, 3, 1, 2),
    (4, 8, 1, 7, 7, 24, 3, 1, 1),
]


@pytest.mark.parametrize("case", WGRAD_CASES)
def test_conv_wgrad(case):
    from lbann_b200.ops.conv import conv_wgrad
    N, C, D, H, W, K, k, pad, stride = case
    torch.manual_seed(0)
    ks = (1 if D == 1 else k, k, k)
    pd = (0 if D == 1 else pad, pad, pad)
    st = (1 if D == 1 else stride, stride, stride)
    x = torch.randn(N, C, D, H, W, device="cuda").bfloat16()
    w = torch.zeros(K, C, *ks, device="cuda", requires_grad=True)
    y = F.conv3d(x.float(), w, None, st, pd)
    dy = torch.randn_like(y).bfloat16()
    y.backward(dy.float())
    xl = x.permute(0, 2, 3, 4, 1).contiguous()
    dyl = dy.permute(0, 2, 3, 4, 1).contiguous()
    prev = torch.ones(K, C, *ks, device="cuda")
    got = conv_wgrad(xl, dyl, ks, pad=pd, stride=st, out=prev.clone(), alpha=0.5)
    assert native.consume_status() == 0
    ref = prev + 0.5 * w.grad
    torch.testing.assert_close(got, ref, rtol=2e-3, atol=2e-2 * (N * D * H * W) ** 0.5 / 8)


@pytest.mark.parametrize("case", [
    # N, C, D, H, W, K, k: the splits of the pixels and the blocks of the reduction at their edges
    (1, 8, 1, 4, 4, 8, 1),          # one brick, one tap, 8 channels and filters
    (1, 48, 1, 9, 17, 40, 3),       # a part of a channel slice, bricks with unused rows
    (2, 24, 3, 7, 5, 72, 5),        # 125 taps: four tap blocks, the last one ragged
    (3, 520, 1, 6, 6, 264, 1),      # more channel blocks and filter tiles than fit one of each
    (8, 64, 1, 40, 56, 64, 3),      # one CTA per SM and split, many split groups
    (1, 256, 4, 4, 4, 256, 3),      # few bricks, a filter that fills the GPU by itself
])
def test_conv_wgrad_reduction(case):
    """fp32 partial sums of exact products: against 64 bits the error is that of summation, which
    grows like sqrt(terms) * 2^-24 (below 2e-6 for the largest here); the same call twice gives the same bits."""
    from lbann_b200.ops.conv import conv_wgrad
    N, C, D, H, W, K, k = case
    torch.manual_seed(7)
    ks = (1 if D == 1 else k, k, k)
    pd = tuple(v // 2 for v in ks)
    x = torch.randn(N, D, H, W, C, device="cuda").bfloat16()
    dy = torch.randn(N, D, H, W, K, device="cuda").bfloat16()
    got = conv_wgrad(x, dy, ks, pad=pd)
    again = conv_wgrad(x, dy, ks, pad=pd)
    assert native.consume_status() == 0
    xp = F.pad(x.double(), (0, 0, pd[2], pd[2], pd[1], pd[1], pd[0], pd[0]))
    ref = torch.empty(K, C, *ks, device="cuda", dtype=torch.double)
    for a in range(ks[0]):
        for b in range(ks[1]):
            for c in range(ks[2]):
                view = xp[:, a:a + D, b:b + H, c:c + W].reshape(-1, C)
                ref[:, :, a, b, c] = dy.double().reshape(-1, K).t() @ view
    assert torch.equal(got, again)
    assert float((got.double() - ref).norm() / ref.norm()) < 4e-6


@pytest.mark.parametrize("case", [(2, 256, 8, 8, 8, 256), (1, 128, 4, 16, 16, 200), (3, 64, 1, 12, 12, 96)])
def test_conv_deep_layers_split_the_reduction(case, monkeypatch):
    """The deep layers of a network on a small batch: a handful of output bricks, thousands of
    reduction steps.  The split result equals the unsplit one up to fp32 summation order."""
    N, C, D, H, W, K = case
    torch.manual_seed(4)
    ks = (1 if D == 1 else 3, 3, 3)
    pd = (0 if D == 1 else 1, 1, 1)
    x = torch.randn(N, C, D, H, W, device="cuda").half()
    w = (torch.randn(K, C, *ks, device="cuda") / (C * 27) ** 0.5).half()
    bias = torch.randn(K, device="cuda")
    xl = x.permute(0, 2, 3, 4, 1).contiguous()
    wp = pack_filter(w, torch.float16)
    before = native.splitk_offers
    ys = [conv_fwd(xl, wp, ks, pad=pd, bias=bias, act=native.ACT_LEAKY, act_param=0.01,
                   out_dtype=torch.float32) for _ in range(2)]
    assert native.consume_status() == 0
    assert native.splitk_offers == before + 2
    assert torch.equal(ys[0], ys[1])
    ref = F.leaky_relu(F.conv3d(x.float(), w.float(), bias, 1, pd), 0.01).permute(0, 2, 3, 4, 1)
    torch.testing.assert_close(ys[0], ref, rtol=2e-3, atol=2e-2)
    monkeypatch.setenv("LBANN_DISABLE_SPLITK", "1")
    plain = conv_fwd(xl, wp, ks, pad=pd, bias=bias, act=native.ACT_LEAKY, act_param=0.01,
                     out_dtype=torch.float32)
    torch.testing.assert_close(ys[0], plain, rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("case", [
    # N, C, D, H, W, K, depth padding: segments of 4 or 2 planes, ragged ones, one to three channel blocks
    (8, 64, 19, 40, 64, 32, 1),
    (6, 32, 21, 64, 48, 64, 1),
    (9, 16, 12, 56, 50, 24, 0),
    (8, 96, 17, 40, 40, 32, 1),
    (16, 48, 10, 30, 60, 40, 2),
])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_conv_walking_the_depth_gives_the_bits_of_single_planes(case, dtype):
    """Convolutions large enough for the kernel that takes three depth taps in one product equal,
    bit for bit, the same computed plane by plane, which is too little work for it; every fourth
    plane is compared."""
    N, C, D, H, W, K, pd = case
    torch.manual_seed(7)
    x = torch.randn(N, D, H, W, C, device="cuda").to(dtype)
    wf = (torch.randn(K, C, 3, 3, 3, device="cuda") / (C * 27) ** 0.5).to(dtype)
    w = pack_filter(wf, dtype)
    bias = torch.randn(K, device="cuda")
    y = conv_fwd(x, w, (3, 3, 3), pad=(pd, 1, 1), bias=bias, out_dtype=dtype)
    Do = D + 2 * pd - 2
    assert y.shape[1] == Do
    xp = F.pad(x, (0, 0, 0, 0, 0, 0, pd, pd))
    for d in sorted({0, 1, *range(2, Do, 4), Do - 2, Do - 1}):
        one = conv_fwd(xp[:, d:d + 3].contiguous(), w, (3, 3, 3), pad=(0, 1, 1), bias=bias, out_dtype=dtype)
        assert torch.equal(y[:, d], one[:, 0]), d
    assert native.consume_status() == 0
    n = N - 1
    ref = F.conv3d(x[n:].permute(0, 4, 1, 2, 3).float(), wf.float(), bias, 1, (pd, 1, 1))
    torch.testing.assert_close(y[n:].permute(0, 4, 1, 2, 3).float(), ref, rtol=2e-2, atol=4e-2)


def _walk(N, C, D, H, W, K, pd):
    geom = (ctypes.c_int * 21)(N, D, H, W, C, D + 2 * pd - 2, H, W, K, 3, 3, 3, pd, 1, 1, 1, 1, 1, 1, 1, 1)
    return native.cuda_lib().lb_conv_slab_walk(geom)


@pytest.mark.parametrize("case,planes", [
    ((8, 64, 19, 40, 64, 32, 1), 4), ((6, 32, 21, 64, 48, 64, 1), 2), ((9, 16, 12, 56, 50, 24, 0), 2),
    ((8, 96, 17, 40, 40, 32, 1), 4), ((16, 48, 10, 30, 60, 40, 2), 4),         # the cases of the test above
    ((4, 64, 61, 40, 64, 32, 1), 8), ((8, 64, 64, 64, 64, 32, 1), 8),
    ((2, 32, 3, 40, 64, 32, 1), 0), ((8, 16, 19, 40, 64, 80, 1), 0),           # too little work; too many filters
])
def test_conv_slab_choice(case, planes):
    """Planes per work item that the rule picks, on 148 SMs; a plane by itself is never walked, so
    that the tests that compare with single planes compare two kernels."""
    if native.cuda_lib().lb_sm_count() != 148:
        pytest.skip("the sizes are chosen for 148 SMs")
    assert _walk(*case) == planes
    N, C, _, H, W, K, _ = case
    assert _walk(N, C, 3, H, W, K, 0) == 0


@pytest.mark.parametrize("D", [61, 64])
def test_conv_walking_eight_planes(D):
    """Segments of eight planes (both sets of accumulators take all of TMEM), the last one ragged or
    full: the bits of single planes."""
    N, C, H, W, K = 4, 64, 40, 64, 32
    torch.manual_seed(8)
    x = torch.randn(N, D, H, W, C, device="cuda").half()
    w = pack_filter((torch.randn(K, C, 3, 3, 3, device="cuda") / (C * 27) ** 0.5).half(), torch.float16)
    assert _walk(N, C, D, H, W, K, 1) == 8 or native.cuda_lib().lb_sm_count() != 148
    y = conv_fwd(x, w, (3, 3, 3), pad=(1, 1, 1))
    xp = F.pad(x, (0, 0, 0, 0, 0, 0, 1, 1))
    for d in sorted({*range(0, D, 7), 55, 56, D - 2, D - 1}):
        one = conv_fwd(xp[:, d:d + 3].contiguous(), w, (3, 3, 3), pad=(0, 1, 1))
        assert torch.equal(y[:, d], one[:, 0]), d
    assert native.consume_status() == 0


@pytest.mark.parametrize("case", [(64, 32, 1, 56, 56, 32, 1), (3, 64, 5, 23, 30, 64, 1), (200, 16, 1, 28, 28, 24, 1)])
def test_conv_wgrad_of_one_tap_filters(case):
    """Filters that load little a brick of pixels run two CTAs an SM: the bounds and the repeatability
    of the other filter gradients."""
    test_conv_wgrad_reduction(case)


@pytest.mark.parametrize("case,bricks", [
    ((8, 64, 32, 32, 32, 128, 3), 56),       # rounds: two sets of accumulators fill TMEM, four parts
    ((8, 128, 16, 16, 16, 256, 3), 24),      # one set fills TMEM: three rounds
    ((256, 512, 1, 7, 7, 512, 3), 29),       # bricks with unused rows
    ((8, 32, 32, 64, 64, 64, 3), 111),       # two parts side by side
    ((3, 128, 5, 16, 16, 256, 3), 8),        # few bricks: CTAs whose last rounds are empty
])
def test_conv_wgrad_sums_in_parts(case, bricks):
    """An fp32 sum on the tensor core drifts by up to 1.2e-9 of the result per term; no accumulator takes
    more than `bricks` bricks of at most 64 pixels, which bounds the filter gradient's error, with 1e-7
    for the sums of the parts.  The same call gives the same bits."""
    from lbann_b200.ops.conv import conv_wgrad
    N, C, D, H, W, K, k = case
    torch.manual_seed(9)
    ks = (1 if D == 1 else k, k, k)
    pd = tuple(v // 2 for v in ks)
    x = torch.relu(torch.randn(N, D, H, W, C, device="cuda")).bfloat16()
    dy = torch.randn(N, D, H, W, K, device="cuda").bfloat16()
    got = conv_wgrad(x, dy, ks, pad=pd)
    again = conv_wgrad(x, dy, ks, pad=pd)
    assert native.consume_status() == 0
    assert torch.equal(got, again)
    xp = F.pad(x, (0, 0, pd[2], pd[2], pd[1], pd[1], pd[0], pd[0]))
    for a, b, c in ((0, 0, 0), pd, (ks[0] - 1, ks[1] - 1, ks[2] - 1)):
        ref = torch.zeros(K, C, device="cuda", dtype=torch.double)
        for n in range(N):
            ref += dy[n].reshape(-1, K).double().t() @ xp[n, a:a + D, b:b + H, c:c + W].reshape(-1, C).double()
        err = float((got[:, :, a, b, c].double() - ref).norm() / ref.norm())
        assert err < 1.2e-9 * 64 * bricks + 1e-7, err


@pytest.mark.parametrize("case", [
    # N, C, D, H, W, K, k, padding along depth: sizes that take their taps from halo slabs
    (8, 32, 9, 17, 64, 64, 3, 1),       # 3 x 2 accumulators of four planes and lines, one of the last plane's columns
    (16, 32, 13, 26, 60, 64, 3, 0),     # bricks that hang over the width, halo planes that come with the input
    (4, 24, 6, 40, 24, 40, 3, 1),       # a part of a channel slice; groups of eight pixels from two lines
    (2, 16, 8, 33, 40, 24, 3, 1),       # eight taps an accumulator
    (16, 64, 1, 56, 56, 64, 3, 0),      # 2-D, pairs of taps
    (8, 96, 1, 31, 70, 56, 3, 0),       # two channel blocks, a ragged one; ragged filters
    (8, 64, 32, 32, 32, 128, 3, 1),     # more accumulators than one CTA holds
    (24, 32, 1, 45, 33, 32, 5, 0),      # five taps a line: one accumulator and one tap over
    (64, 64, 1, 40, 40, 64, 5, 0),
    (1, 8, 5, 64, 100, 8, 3, 1),        # 8 channels, 8 filters
])
def test_conv_wgrad_from_slabs(case):
    """fp16 and bf16, added to what the gradient holds.  An accumulator takes at most 56 bricks' worth of 64
    pixels here, 1.2e-9 of the result a term (test_conv_wgrad_sums_in_parts), and 4e-7 go to the sums of the
    parts and to adding them: 4.7e-6."""
    from lbann_b200.ops.conv import conv_wgrad
    N, C, D, H, W, K, k, pad_d = case
    ks = (1 if D == 1 else k, k, k)
    pd = (pad_d if D > 1 else 0, k // 2, k // 2)
    Do = D + 2 * pd[0] - ks[0] + 1
    geom = (ctypes.c_int * 21)(N, D, H, W, C, Do, H, W, K, *ks, *pd, 1, 1, 1, 1, 1, 1)
    assert native.cuda_lib().lb_conv_wgrad_slab(geom) == 1 or native.cuda_lib().lb_sm_count() != 148
    for dtype in (torch.bfloat16, torch.float16):
        torch.manual_seed(11)
        x = torch.randn(N, D, H, W, C, device="cuda").to(dtype)
        dy = torch.randn(N, Do, H, W, K, device="cuda").to(dtype)
        prev = torch.randn(K, C, *ks, device="cuda")
        got = conv_wgrad(x, dy, ks, pad=pd, out=prev.clone(), alpha=0.5)
        assert native.consume_status() == 0
        xp = F.pad(x.double(), (0, 0, pd[2], pd[2], pd[1], pd[1], pd[0], pd[0]))
        ref = torch.empty(K, C, *ks, device="cuda", dtype=torch.double)
        for a in range(ks[0]):
            for b in range(ks[1]):
                for c in range(ks[2]):
                    view = xp[:, a:a + Do, b:b + H, c:c + W].reshape(-1, C)
                    ref[:, :, a, b, c] = prev[:, :, a, b, c].double() + 0.5 * (dy.double().reshape(-1, K).t() @ view)
        assert float((got.double() - ref).norm() / ref.norm()) < 4.7e-6


def test_filter_gradients_of_layers_in_turn():
    """A thread's last tiling is kept between asking for the workspace and the launch: layers in turn, also by
    threads of their own, give what each gives alone."""
    import threading
    torch.manual_seed(3)
    cases = []
    for n, ci, co, size, k in ((2, 32, 64, 20, 3), (1, 64, 32, 9, 1), (3, 16, 24, 17, 5)):
        x = torch.randn(n, ci, size, size, device="cuda").half().contiguous(memory_format=torch.channels_last)
        w = torch.randn(co, ci, k, k, device="cuda").requires_grad_(True)
        wh = nn.WeightHandle(w, torch.zeros_like(w))
        y = nn.convolution(x.requires_grad_(True), wh, None, (k, k), (k // 2,) * 2, (1, 1), (1, 1))
        cases.append((x, wh, y, torch.randn_like(y)))

    def grad(c):
        x, wh, y, dy = c
        wh.grad.zero_()
        torch.autograd.grad(y, x, dy, retain_graph=True)
        torch.cuda.synchronize()
        return wh.grad.clone()

    alone = [[grad(c) for _ in range(3)][-1] for c in cases]
    got = [grad(cases[i]) for i in (0, 1, 2, 1, 0, 2)]
    for i, g in zip((0, 1, 2, 1, 0, 2), got):
        assert float((g - alone[i]).norm()) <= 1e-6 * float(alone[i].norm())
    out = {}
    threads = [threading.Thread(target=lambda i=i: out.__setitem__(i, [grad(cases[i]) for _ in range(5)])) for i in range(3)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    for i in range(3):
        for g in out[i]:
            assert float((g - alone[i]).norm()) <= 1e-6 * float(alone[i].norm())
    assert native.consume_status() == 0
