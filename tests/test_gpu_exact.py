"""The dense pass in fp32 precision on the tensor cores, and the vectorised mask, dilation and feedback kernels, at the
sizes where they change path."""
import ctypes as C

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

from oracle import restatement as R  # noqa: E402


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    torch.backends.cudnn.allow_tf32 = False
    torch.backends.cuda.matmul.allow_tf32 = False
    return torch.device("cuda:0")


def cl(t):
    return t.contiguous(memory_format=torch.channels_last)


# cin, cout, k, stride, n, h, w, addend: ragged tiles, one pair of tiles, partial chunks and slabs, both block widths for
# every filter size (7x7 in blocks of 64 channels: the halos leave the least room for the filter ring)
@pytest.mark.parametrize("case", [(5, 32, 5, 1, 1, 41, 50, False), (2, 64, 3, 2, 1, 18, 26, False), (64, 40, 3, 1, 2, 8, 16, False),
                                  (32, 64, 5, 2, 1, 67, 89, False), (256, 256, 3, 1, 1, 33, 44, True), (256, 128, 5, 1, 1, 34, 44, False),
                                  (96, 96, 7, 1, 1, 24, 40, False), (130, 36, 3, 1, 1, 9, 9, False),
                                  (64, 64, 7, 1, 1, 104, 104, False), (64, 64, 7, 2, 1, 205, 208, False), (32, 64, 5, 1, 1, 104, 100, False)])
def test_dense_pass_against_float64(dev, case):
    from maskedincrementeval_b200 import fields as fl, _native as nat
    from maskedincrementeval_b200.incr_modules._algebra import NATIVE
    from maskedincrementeval_b200.incr_modules.e2depth_incr import ConvLayerIncr
    cin, cout, k, s, n, h, w, with_addend = case
    torch.manual_seed(1)
    layer = ConvLayerIncr(cin, cout, k, s, k // 2, activation="sigmoid").to(dev).eval()
    g = torch.Generator(device=dev).manual_seed(2)
    x = cl(torch.randn(n, cin, h, w, generator=g, device=dev))
    c = layer.conv2d
    want = F.conv2d(x.double(), c.weight.detach().double(), c.bias.detach().double(), stride=s, padding=k // 2)
    addend = None
    if with_addend:
        addend = [cl(torch.randn(want.shape, generator=g, device=dev)), fl.full_mask(n, *want.shape[2:], dev)]
        want = want + addend[0].double()
    err = {}
    old = fl.config.tensor_cores
    try:
        for mode in ("auto", "off"):
            fl.config.tensor_cores = mode
            with torch.no_grad():
                y, m = NATIVE.conv(c, NATIVE.lift(x), layer.activation, addend=addend)
            assert bool(nat.lib.mie_conv_is_exact(C.byref(c._plan(n, h, w, dev).args))) == (mode == "auto")
            res = layer.activation.in_res.reservoir
            err[mode] = float((res.double() - want).norm() / want.norm())
            assert float((y.double() - torch.sigmoid(res.double())).abs().max()) <= 1e-6
            assert bool(m.pixel_mask().all())
    finally:
        fl.config.tensor_cores = old
    # no worse than the CUDA-core kernel's own rounding, or what two TF32 parts leave of a value (2^-24 of either operand, and the
    # rounding of the result)
    assert err["auto"] <= max(err["off"], 1.5e-7), err


# reductions on both sides of the rule that sets the length of a segment
@pytest.mark.parametrize("cin,k", [(8, 3), (5, 5), (16, 3), (32, 3), (44, 3), (45, 3), (64, 3), (32, 5), (127, 3), (128, 3), (64, 5), (256, 3)])
@pytest.mark.parametrize("kind", ["normal", "rectified", "isolated"])
def test_dense_pass_is_no_less_precise_than_fp32(dev, cin, k, kind):
    from maskedincrementeval_b200 import fields as fl
    from maskedincrementeval_b200.incr_modules._algebra import NATIVE
    from maskedincrementeval_b200.incr_modules.e2depth_incr import ConvLayerIncr
    torch.manual_seed(3)
    layer = ConvLayerIncr(cin, 64, k, 1, k // 2, activation="relu").to(dev).eval()
    c = layer.conv2d
    g = torch.Generator(device=dev).manual_seed(4)
    x = torch.randn(1, cin, 64, 72, generator=g, device=dev)
    if kind == "rectified":
        x = torch.relu(x)
    if kind == "isolated":
        x = x * (torch.rand(1, 1, 64, 72, generator=g, device=dev) < 0.05)
    want = F.conv2d(x.double(), c.weight.detach().double(), c.bias.detach().double(), padding=k // 2)
    err = {}
    old = fl.config.tensor_cores
    try:
        for mode in ("auto", "off"):
            fl.config.tensor_cores = mode
            with torch.no_grad():
                NATIVE.conv(c, NATIVE.lift(cl(x)), layer.activation)
            err[mode] = float((layer.activation.in_res.reservoir.double() - want).norm() / want.norm())
    finally:
        fl.config.tensor_cores = old
    assert err["auto"] <= max(err["off"], 1.5e-7), err


def test_extension_is_no_less_precise_than_fp32(dev):
    """conv*_increment_ext on isolated active pixels: layers below 48 channels keep to the FP32 kernel."""
    from maskedincrementeval_b200.ext.pointops import pointops_functional as pf
    g = torch.Generator(device=dev).manual_seed(10)
    for cin, bound in ((5, 7e-8), (16, 1e-7), (32, 1.2e-7), (47, 1.4e-7), (48, 1.4e-7), (64, 1.5e-7)):      # the FP32 kernel's: sums of cin products
        w = torch.randn(cin, 3, 3, 32, generator=g, device=dev) / (9 * cin) ** 0.5
        x = torch.zeros(2, cin, 60, 80, device=dev)
        x[:, :, ::9, ::9] = torch.randn(2, cin, 7, 9, generator=g, device=dev)
        y, _ = pf.functional_conv_module(cl(x), w, mask=None, stride=(1, 1), padding=(1, 1))
        want = F.conv2d(x.double(), w.permute(3, 0, 1, 2).double(), padding=1)
        assert float((y.double() - want).norm() / want.norm()) <= bound, cin


# infinities, NaN and values that round up to infinity in TF32, in the input or in the filter: what the fp32 kernel gives
@pytest.mark.parametrize("where", ["input", "filter"])
@pytest.mark.parametrize("case", [(64, 64, 3, 1, 1, 41, 50), (5, 32, 5, 2, 2, 33, 40)])
def test_dense_pass_on_non_finite_values(dev, case, where):
    from maskedincrementeval_b200 import fields as fl
    from maskedincrementeval_b200.ext.pointops import pointops_functional as pf
    from maskedincrementeval_b200.incr_modules._algebra import NATIVE
    from maskedincrementeval_b200.incr_modules.e2depth_incr import ConvLayerIncr
    cin, cout, k, s, n, h, w = case
    torch.manual_seed(8)
    layer = ConvLayerIncr(cin, cout, k, s, k // 2, activation="relu").to(dev).eval()
    c = layer.conv2d
    x = cl(torch.randn(n, cin, h, w, device=dev) * 0.2)      # (below 1: no product with the largest number lies at the edge of overflow)
    odd = [float("inf"), -float("inf"), float("nan"), torch.finfo(torch.float32).max, -torch.finfo(torch.float32).max]
    with torch.no_grad():
        for i, v in enumerate(odd):
            if where == "input":
                x[i % n, (3 * i) % cin, 6 * i + 3, 7 * i + 2] = v
            else:
                c.weight[4 * i, (3 * i) % cin, i % k, 0] = v
        x[0, 0, h - 1, w - 1] = torch.finfo(torch.float32).max * 0.9999      # and a finite one that stays finite, next to zeros
        states = {}
        old = fl.config.tensor_cores
        try:
            for mode in ("auto", "off"):
                fl.config.tensor_cores = mode
                NATIVE.conv(c, NATIVE.lift(x), layer.activation)
                states[mode] = layer.activation.in_res.reservoir.clone()
        finally:
            fl.config.tensor_cores = old
        ext, _ = pf.functional_conv_module(x, c.conv2d_weights, mask=torch.ones_like(x, dtype=torch.bool), stride=(s, s), padding=(k // 2, k // 2))
    pairs = [(states["auto"], states["off"])]
    if cin >= 48:      # (the extension runs narrower layers on the FP32 kernel, which sends no NaN)
        pairs.append((ext, states["off"] - c.bias.detach().view(1, -1, 1, 1)))
    for got, want in pairs:
        assert not bool(want.isfinite().all())
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isposinf(), want.isposinf()) and torch.equal(got.isneginf(), want.isneginf())
        # relative to the products that a value is the sum of: fp32 sums of cin * k * k terms
        fine = want.isfinite() & (want.abs() < 1e30)
        assert float((got[fine] - want[fine]).abs().max()) <= 1e-5
        big = want.isfinite() & ~fine
        assert float(((got[big] - want[big]) / want[big]).abs().max()) <= 1e-5 if bool(big.any()) else True


# Many values that lie far apart in one halo, in any unit: what two FP16 numbers with a common scale hold is computed on the tensor cores, the
# rest with FP32 instructions.  Every output against the sum of its products' magnitudes: fp32 sums of cin * k * k terms, and (where no more
# than 2^38 lies between them) a step of 2^-52 of the largest value times the filter's entries.
FAR_APART = [(1.0, 1e-3), (1.0, 1e-8), (1.0, 1e-12), (1e-30, 1e-33), (1e-12, 1e-22), (16383.0, 1e-6), (1e4, 1e-6), (40000.0, 1e-6), (1e6, 1e-9), (1e20, 1.0),
             (1e31, 1e30), (1e36, 0.2)]


@pytest.mark.parametrize("case", [(48, 32, 3, 1, 24, 40), (64, 64, 7, 1, 17, 23), (5, 32, 5, 2, 33, 40), (16, 36, 3, 1, 41, 50), (40, 64, 5, 2, 35, 41)])
@pytest.mark.parametrize("big,small", FAR_APART)
@pytest.mark.parametrize("unit", [0.05, 1e6])
def test_dense_pass_on_values_far_apart(dev, case, big, small, unit):
    from maskedincrementeval_b200.incr_modules._algebra import NATIVE
    from maskedincrementeval_b200.incr_modules.e2depth_incr import ConvLayerIncr
    cin, cout, k, s, h, w = case
    if big * unit * cin * k * k > 1e37:
        return      # beyond fp32
    torch.manual_seed(12)
    layer = ConvLayerIncr(cin, cout, k, s, k // 2, activation="relu").to(dev).eval()
    c = layer.conv2d
    with torch.no_grad():
        c.weight.mul_(unit / c.weight.abs().max())
        c.bias.zero_()
    x = cl(torch.randn(1, cin, h, w, device=dev).clamp_(-3, 3) * (small / 3))
    x[0, :, 3::11, 5::13] *= big / small
    want = F.conv2d(x.double(), c.weight.detach().double(), stride=s, padding=k // 2)
    size = F.conv2d(x.double().abs(), c.weight.detach().double().abs(), stride=s, padding=k // 2)
    with torch.no_grad():
        NATIVE.conv(c, NATIVE.lift(x), layer.activation)
    got = layer.activation.in_res.reservoir.double()
    step = big * 2.0 ** -52 * unit * cin * k * k if big / small < 2.0 ** 38 else 0.0
    assert bool(got.isfinite().all())
    assert float(((got - want).abs() - 2e-6 * size).max()) <= step


# A few small values beside large ones, in the dense pass and in steps, blocks and items of every form: as exact as any others (2e-6 as above), in
# any unit.  (A large pixel and a small value per 12 x 12 pixels: no halo has more small ones than are listed.)
@pytest.mark.parametrize("cin,cout,k,s", [(48, 32, 3, 1), (32, 32, 3, 1), (16, 24, 3, 1), (64, 64, 3, 1), (64, 64, 5, 1), (40, 64, 5, 2), (96, 36, 3, 2), (132, 64, 3, 1)])
@pytest.mark.parametrize("big,small", [(1.0, 1e-9), (1.0, 1e-14), (1e-5, 1e-30), (16383.0, 1e-9), (1e6, 1e-3)])
@pytest.mark.parametrize("step", [False, True])
def test_a_few_small_values(dev, cin, cout, k, s, big, small, step):
    from maskedincrementeval_b200 import _native as nat
    from maskedincrementeval_b200.incr_modules._algebra import NATIVE
    from maskedincrementeval_b200.incr_modules.e2depth_incr import ConvLayerIncr
    torch.manual_seed(29)
    h, w = 61, 90
    layer = ConvLayerIncr(cin, cout, k, s, k // 2, activation=None if step else "relu").to(dev).eval()
    c = layer.conv2d
    c.precision = "split"
    c.bias.data.zero_()
    x = torch.zeros(1, cin, h, w, device=dev)
    x[0, :, 3::12, 4::12] = big * torch.randn(1, 1, 1, device=dev) + big * torch.rand(cin, 5, 8, device=dev)
    rows, cols = torch.arange(9, h, 12, device=dev), torch.arange(10, w, 12, device=dev)
    for i, r in enumerate(rows):
        for j, q in enumerate(cols):
            x[0, (7 * i + 5 * j) % cin, r, q] = small * (1 + i) * (-1) ** j
    x = cl(x)
    want = F.conv2d(x.double(), c.weight.detach().double(), stride=s, padding=k // 2)
    size = F.conv2d(x.double().abs(), c.weight.detach().double().abs(), stride=s, padding=k // 2)
    for _ in range(2):      # (the order in which they are found must not matter)
        with torch.no_grad():
            if step:
                y, m = layer([x, None])
                assert nat.lib.mie_conv_is_exact(C.byref(c._plan(1, h, w, dev).args)) or cin * k * k < 256
            else:
                NATIVE.conv(c, NATIVE.lift(x), layer.activation)
                y = layer.activation.in_res.reservoir
        got = y.clone()
        assert _ == 0 or torch.equal(got, first)
        first = got
        assert float(((got.double() - want).abs() - 2e-6 * size).max()) <= 0.0


# the same for a filter whose entries lie far apart, and for one of tiny entries.  (At isolated pixels an output may be a sum of small
# entries alone, which the parts hold to 2^-52 of the channel's largest entry where that lies below 2^10.)
@pytest.mark.parametrize("big,small", [(1e6, 1e-6), (1e30, 1e-3), (1e-20, 1e-22), (900.0, 1e-3), (1.0, 1e-9), (1e-3, 1e-20)])
@pytest.mark.parametrize("cin,cout,k,s", [(48, 64, 3, 1), (32, 32, 3, 1), (10, 36, 5, 2)])
@pytest.mark.parametrize("isolated", [False, True])
def test_dense_pass_on_filters_far_apart(dev, big, small, cin, cout, k, s, isolated):
    from maskedincrementeval_b200.ext.pointops import pointops_functional as pf
    from maskedincrementeval_b200.incr_modules._algebra import NATIVE
    from maskedincrementeval_b200.incr_modules.e2depth_incr import ConvLayerIncr
    torch.manual_seed(13)
    layer = ConvLayerIncr(cin, cout, k, s, k // 2, activation="relu").to(dev).eval()
    c = layer.conv2d
    with torch.no_grad():
        c.weight.normal_().clamp_(-3, 3).mul_(small / 3)
        c.weight[::5, :, 0, 0] *= big / small
        c.bias.zero_()
    x = torch.randn(1, cin, 21, 30, device=dev)
    if isolated:
        on = torch.zeros(1, 1, 21, 30, device=dev)
        on[:, :, 2::k, 1::k] = 1.0
        x = x * on * (torch.rand(1, cin, 21, 30, device=dev) < 0.2)
    x = cl(x)
    want = F.conv2d(x.double(), c.weight.detach().double(), stride=s, padding=k // 2)
    size = F.conv2d(x.double().abs(), c.weight.detach().double().abs(), stride=s, padding=k // 2)
    step = F.conv2d(x.double().abs(), torch.full_like(c.weight, big * 2.0 ** -52 if big < 2 ** 10 else 0.0).double(), stride=s, padding=k // 2)
    with torch.no_grad():
        NATIVE.conv(c, NATIVE.lift(x), layer.activation)
        got = [layer.activation.in_res.reservoir.double()]
        if cin >= 48:
            got.append(pf.functional_conv_module(x, c.conv2d_weights, mask=None, stride=(s, s), padding=(k // 2, k // 2))[0].double())
    for y in got:
        assert float(((y - want).abs() - 2e-6 * size - step).max()) <= 0.0


def test_extension_on_a_silent_step(dev):
    """A delta without an active pixel: zeros, also behind a call that left the workspace full, and before one that needs it again."""
    from maskedincrementeval_b200.ext.pointops import pointops_functional as pf
    g = torch.Generator(device=dev).manual_seed(9)
    w = torch.randn(64, 3, 3, 64, generator=g, device=dev) * 0.04
    x = cl(torch.randn(1, 64, 40, 56, generator=g, device=dev))
    want = F.conv2d(x.double(), w.permute(3, 0, 1, 2).double(), padding=1)
    for silent in (False, True, False, True):
        mask = torch.zeros_like(x, dtype=torch.bool) if silent else None
        y, _ = pf.functional_conv_module(x, w, mask=mask, stride=(1, 1), padding=(1, 1))
        if silent:
            assert bool((y == 0).all())
        else:
            assert float((y.double() - want).norm() / want.norm()) <= 2e-6


# stride 2 on fields one pixel wide or high, which have no odd columns or rows
@pytest.mark.parametrize("h,w", [(17, 1), (1, 22), (1, 1), (2, 9)])
@pytest.mark.parametrize("k", [3, 5])
def test_stride_two_on_one_pixel_fields(dev, h, w, k):
    from maskedincrementeval_b200.ext.pointops import pointops_functional as pf
    from maskedincrementeval_b200.incr_modules._algebra import NATIVE
    from maskedincrementeval_b200.incr_modules.e2depth_incr import ConvLayerIncr
    torch.manual_seed(6)
    layer = ConvLayerIncr(64, 64, k, 2, k // 2, activation="relu").to(dev).eval()
    c = layer.conv2d
    x = cl(torch.randn(2, 64, h, w, device=dev))
    want = F.conv2d(x.double(), c.weight.detach().double(), c.bias.detach().double(), stride=2, padding=k // 2)
    with torch.no_grad():
        NATIVE.conv(c, NATIVE.lift(x), layer.activation)
        got = layer.activation.in_res.reservoir
        y, _ = pf.functional_conv_module(x, c.conv2d_weights, mask=None, stride=(2, 2), padding=(k // 2, k // 2))
    assert float((got.double() - want).norm() / want.norm()) <= 2e-6      # fp32 sums of 64 * k * k products
    want = want - c.bias.detach().double().view(1, -1, 1, 1)
    assert float((y.double() - want).norm() / want.norm()) <= 2e-6


@pytest.mark.parametrize("c,dtype", [(20, torch.float32), (32, torch.float32), (132, torch.float32), (16, torch.uint8), (48, torch.uint8), (20, torch.int32)])
def test_mask_words_vectorised(dev, c, dtype):
    from maskedincrementeval_b200 import fields as fl
    g = torch.Generator(device=dev).manual_seed(c)
    n, h, w = 2, 21, 43
    x = torch.randn(n, c, h, w, generator=g, device=dev) * (torch.rand(n, c, h, w, generator=g, device=dev) < 0.01)
    x = cl(x if dtype == torch.float32 else (x != 0).to(dtype))
    m = fl.mask_from_delta(x) if dtype == torch.float32 else fl.mask_from_tensor(x)
    assert torch.equal(m.pixel_mask(), (x != 0).any(1, keepdim=True).to(torch.uint8))


@pytest.mark.parametrize("c", [1, 2, 3, 4, 5, 6, 7, 8, 9])
@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("thr", [0.0, 0.4])
def test_input_delta_of_any_channel_count(dev, c, split, thr):
    """Channel counts on both sides of the register kernel's limit, ragged tiles, padded pixels; every result to the bit."""
    from maskedincrementeval_b200 import fields as fl
    g = torch.Generator(device=dev).manual_seed(c)
    n, h, w, cp, half = 2, 13, 21, (c + 3) // 4 * 4, (c + 7) // 8 * 8
    new = lambda k: torch.zeros(n, h, w, k, device=dev).permute(0, 3, 1, 2)
    xp, dx, bits = cl(torch.randn(n, c, h, w, generator=g, device=dev)), new(cp)[:, :c], fl.new_bits(n, h, w, dev)
    copy, copy_bits = new(3 * half), fl.new_bits(n, h, w, dev)
    try:
        if split:
            fl.request_split(dx, copy, copy_bits)
        for frac in (0.2, 0.0, 1.0, 0.01):
            x = cl(xp + torch.randn(n, c, h, w, generator=g, device=dev) * (torch.rand(n, 1, h, w, generator=g, device=dev) < frac))
            d = x - xp
            on = (d.abs() > thr).any(1, keepdim=True)
            d = torch.where(on, d, torch.zeros_like(d))
            kept = torch.where(on, x, xp)
            m = fl.delta_mask(x, xp, dx, bits, thr)
            assert torch.equal(dx, d) and torch.equal(xp, kept) and torch.equal(m.pixel_mask(), on.to(torch.uint8))
            if split:
                assert fl.split_made(dx, copy) and torch.equal(copy_bits, bits)
                want = torch.zeros_like(copy)
                want[:, :c] = want[:, 2 * half:2 * half + c] = d
                want[:, half:half + c] = d - (d.contiguous().view(torch.int32) & ~0x1FFF).view(torch.float32)
                assert torch.equal(copy, want)
    finally:
        fl.forget_tails()


@pytest.mark.parametrize("n,h,w", [(1, 200, 168), (8, 480, 640), (3, 260, 346)])
def test_dilation_of_large_fields(dev, n, h, w):
    from maskedincrementeval_b200 import fields as fl, _native as nat
    g = torch.Generator().manual_seed(n)
    for frac in (0.0, 0.002, 1.0):
        act = (torch.rand(n, 1, h, w, generator=g) < frac).to(torch.uint8)
        m = fl.mask_from_tensor(act.to(dev))
        nt = fl.n_tiles(n, h, w)
        lst, stale = (torch.zeros(nt, dtype=torch.int32, device=dev) for _ in range(2))
        counts, flags = torch.zeros(4, dtype=torch.int32, device=dev), torch.zeros(nt, dtype=torch.uint8, device=dev)
        words = torch.full((nt,), 3, dtype=torch.int64, device=dev)
        nat.check(nat.lib.mie_tiles_dilate(m.bits.data_ptr(), n, h, w, h, w, 5, 1, 2, None, words.data_ptr(), lst.data_ptr(), stale.data_ptr(),
                                           counts.data_ptr(), flags.data_ptr(), nat.stream_ptr(dev)), "dilate")
        want = R.tile_list(R.conv_out_mask(act, 5, 1, 2)).tolist()
        na, ns = counts[:2].tolist()
        assert lst[:na].tolist() == want and na + ns == nt
        assert stale[:ns].tolist() == sorted(set(range(nt)) - set(want)) and int(words.abs().max()) == 0


def test_accumulate_and_keep(dev):
    from maskedincrementeval_b200 import fields as fl
    g = torch.Generator(device=dev).manual_seed(3)
    for c in (4, 36, 64):
        y = cl(torch.randn(2, c, 19, 45, generator=g, device=dev))
        kept = cl(torch.randn(2, c, 19, 45, generator=g, device=dev))
        d = cl(torch.randn(2, c, 19, 45, generator=g, device=dev) * (torch.rand(2, 1, 19, 45, generator=g, device=dev) < 0.1))
        m, kb = fl.mask_from_delta(d), fl.new_bits(2, 19, 45, dev)
        want = y + d
        z = y.clone(memory_format=torch.channels_last)
        fl.accumulate(z, d, m)
        fl.accumulate_keep(y, d, m, kept, kb)
        assert torch.equal(y, want) and torch.equal(z, want) and torch.equal(kept, d) and torch.equal(kb, m.bits)


# one or two input channels: ragged tiles, both strides, partial channel blocks, two column blocks
@pytest.mark.parametrize("case", [(2, 32, 1, 21, 43), (2, 64, 2, 34, 50), (1, 36, 1, 8, 9), (2, 96, 1, 17, 24)])
@pytest.mark.parametrize("thr", [0.0, 0.05])
def test_few_input_channels_against_the_restatement(dev, case, thr):
    from maskedincrementeval_b200 import fields as fl
    from maskedincrementeval_b200.incr_modules.e2depth_incr import ConvLayerIncr
    cin, cout, s, h, w = case
    torch.manual_seed(4)
    layer = ConvLayerIncr(cin, cout, 3, s, 1, activation="relu").to(dev).eval()
    layer.activation.threshold = thr
    wt, b = layer.conv2d.weight.detach().cpu(), layer.conv2d.bias.detach().cpu()
    g = torch.Generator().manual_seed(5)
    x0 = torch.randn(2, cin, h, w, generator=g)
    res, sent = R.conv_dense(x0, wt, b, s, 1), None
    with torch.no_grad():
        sent = layer.forward_refresh_reservoirs(cl(x0.to(dev))).clone()
        for frac in (0.1, 0.0, 0.02, 1.0):
            dx = torch.randn(2, cin, h, w, generator=g) * (torch.rand(2, 1, h, w, generator=g) < frac)
            dy, m = layer([cl(dx.to(dev)), None])
            sent += dy
            want, _ = R.act_incr(res, R.conv_delta(dx, wt, s, 1), "relu")
            res = layer.activation.in_res.reservoir.cpu().contiguous()
            if thr == 0.0:
                assert float((dy.cpu() - want).abs().max()) <= 1e-5
            assert float((sent - torch.relu(layer.activation.in_res.reservoir)).abs().max()) <= thr + 1e-5
            assert torch.equal(m.pixel_mask(), (dy != 0).any(1, keepdim=True).to(torch.uint8))


@pytest.mark.parametrize("c", [32, 34, 66, 130])
def test_upsample_and_concat_of_ragged_channel_counts(dev, c):
    from maskedincrementeval_b200 import fields as fl
    from maskedincrementeval_b200.fields import Scratch
    from maskedincrementeval_b200.incr_modules._algebra import INCR
    g = torch.Generator(device=dev).manual_seed(c)
    sc = Scratch()
    for frac in (0.3, 0.0, 0.02):
        a = cl(torch.randn(1, 2, 11, 22, generator=g, device=dev) * (torch.rand(1, 1, 11, 22, generator=g, device=dev) < frac))
        b = cl(torch.randn(1, c - 2, 11, 22, generator=g, device=dev) * (torch.rand(1, 1, 11, 22, generator=g, device=dev) < frac))
        x, m = INCR.cat([a, fl.mask_from_delta(a)], [b, fl.mask_from_delta(b)], sc, "cat")
        want = torch.cat([a, b], 1)
        assert torch.equal(x, want)
        up, mu = INCR.upsample2x([x, m], None, sc, pad4=True)
        assert float((up - F.interpolate(want, scale_factor=2, mode="bilinear", align_corners=False)).abs().max()) <= 1e-6
        assert float((up * (1 - mu.pixel_mask().float())).abs().max()) == 0.0


# Steps in split precision (two FP16 parts per operand) against the FP32 kernel: cin, cout, k, stride, n, h, w, addend.  Items of one and two
# segments in blocks of 32 channels, longer ones, blocks of 64, partial chunks, slabs and tiles, odd extents at stride 2, more items
# than blocks
@pytest.mark.parametrize("case", [(32, 32, 3, 1, 2, 104, 208, False), (64, 32, 3, 1, 1, 41, 50, False), (96, 32, 3, 1, 1, 24, 40, True), (32, 20, 5, 1, 1, 33, 44, False),
                                  (36, 64, 3, 2, 1, 33, 41, False), (64, 64, 5, 1, 1, 104, 100, False), (16, 40, 7, 1, 1, 24, 40, False),
                                  (256, 256, 3, 1, 1, 17, 23, True), (32, 96, 3, 1, 1, 8, 8, False),
                                  (16, 24, 3, 1, 1, 97, 131, False), (16, 64, 3, 2, 2, 33, 47, True), (12, 24, 3, 1, 1, 41, 50, False), (12, 40, 3, 2, 1, 33, 41, True), (16, 128, 3, 1, 1, 9, 9, False)])
@pytest.mark.parametrize("act,thr", [("relu", 0.0), ("tanh", 0.0), (None, 0.0), ("relu", 0.02), ("sigmoid", 0.02)])
def test_split_precision_steps_against_fp32(dev, case, act, thr):
    from maskedincrementeval_b200 import fields as fl, _native as nat
    from maskedincrementeval_b200.incr_modules.e2depth_incr import ConvLayerIncr
    cin, cout, k, s, n, h, w, with_addend = case
    old = fl.config.tensor_cores
    out = {}
    try:
        for mode in ("auto", "off"):
            fl.config.tensor_cores = mode
            torch.manual_seed(15)
            layer = ConvLayerIncr(cin, cout, k, s, k // 2, activation=act).to(dev).eval()
            layer.conv2d.precision = "split" if cin not in (12, 16) or k != 3 else None      # (3x3 layers of 12 and 16 channels run so by themselves)
            a = layer.activation
            g = torch.Generator(device=dev).manual_seed(16)
            x = cl(torch.randn(n, cin, h, w, generator=g, device=dev))
            steps = []
            with torch.no_grad():
                y = layer.forward_refresh_reservoirs(x)
                if a is not None:
                    a.threshold = thr
                for frac in (0.05, 0.0, 1.0, 0.3):
                    on = torch.rand(n, 1, h, w, generator=g, device=dev) < frac
                    d = cl(torch.randn(n, cin, h, w, generator=g, device=dev) * on)
                    ad = [cl(torch.randn(y.shape, generator=g, device=dev) * (torch.rand(n, 1, *y.shape[2:], generator=g, device=dev) < 0.1)), None] if with_addend else None
                    dy, m = layer.conv2d.forward_fused([d, None], a, ad)
                    if mode == "auto":
                        assert nat.lib.mie_conv_is_exact(C.byref(layer.conv2d._plan(n, h, w, dev).args))
                    steps.append((dy.clone(), m.pixel_mask().clone()))
            out[mode] = steps, None if a is None else a.in_res.reservoir.clone(), None if a is None or a.emitted is None else a.emitted.clone()
    finally:
        fl.config.tensor_cores = old
    # the FP32 kernel adds cin * k * k products one by one: a rounding of at most 2^-24 of a partial sum (below 4 here: weights are below
    # 1 / sqrt(cin k k)) each, in either direction
    tol = 4 * 2.0 ** -24 * (cin * k * k) ** 0.5
    (sa, ra, ea), (so, ro, eo) = out["auto"], out["off"]
    for (dy, m), (want, wm) in zip(sa, so):
        assert torch.equal(m, (dy != 0).any(1, keepdim=True).to(torch.uint8))
        if thr == 0.0:
            assert float((dy - want).abs().max()) <= tol and float((m != wm).float().mean()) <= 1e-3
    if ra is not None:
        assert float((ra - ro).abs().max()) <= tol
    if thr > 0.0:      # what has been sent lies within the threshold of the output, and is what the carry says
        f = torch.relu if act == "relu" else torch.sigmoid
        assert float((ea - f(ra)).abs().max()) <= thr + tol
        differ = float(((ea - eo).abs() > tol).float().mean())
        assert differ <= 1e-3, differ      # changes that lie at the threshold


# fields on both sides of the size from which the lists are compacted by warps: 12288 tiles, ragged edges, runs that end inside a warp's
@pytest.mark.parametrize("n,h,w", [(3, 504, 512), (3, 512, 512), (1, 891, 895), (5, 411, 397)])
def test_dilation_of_fields_around_the_large_kernels_limit(dev, n, h, w):
    test_dilation_of_large_fields(dev, n, h, w)


# Deltas that FP16 parts cannot hold, in steps: two items in hand (16 and 32 channels), one (64 -> 32), blocks of 64.  Against the FP32 kernel:
# the same infinities and NaN, and the same state elsewhere up to fp32 sums of cin * 9 products
@pytest.mark.parametrize("cin,cout", [(16, 36), (32, 32), (96, 32), (64, 64)])
@pytest.mark.parametrize("odd", [float("inf"), float("nan"), 3e30, 1e5, 1.0])
def test_steps_on_values_far_apart(dev, cin, cout, odd):
    from maskedincrementeval_b200 import fields as fl, _native as nat
    from maskedincrementeval_b200.incr_modules.e2depth_incr import ConvLayerIncr
    old = fl.config.tensor_cores
    out = {}
    try:
        for mode in ("auto", "off"):
            fl.config.tensor_cores = mode
            torch.manual_seed(17)
            layer = ConvLayerIncr(cin, cout, 3, 1, 1, activation="relu").to(dev).eval()
            layer.conv2d.precision = "split" if cin != 16 else None
            g = torch.Generator(device=dev).manual_seed(18)
            with torch.no_grad():
                layer.forward_refresh_reservoirs(cl(torch.randn(1, cin, 41, 50, generator=g, device=dev)))
                d = torch.randn(1, cin, 41, 50, generator=g, device=dev) * {1e5: 1e-6, 1.0: 1e-11}.get(odd, 0.2)
                d[0, 3, 7::13, 5::17] = odd
                dy, m = layer([cl(d), None])
                assert mode == "off" or nat.lib.mie_conv_is_exact(C.byref(layer.conv2d._plan(1, 41, 50, dev).args))
            out[mode] = layer.activation.in_res.reservoir.clone(), dy.clone(), m.pixel_mask().clone()
    finally:
        fl.config.tensor_cores = old
    for got, want in zip(out["auto"][:2], out["off"][:2]):
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isposinf(), want.isposinf()) and torch.equal(got.isneginf(), want.isneginf())
        fine = want.isfinite()
        assert bool(fine.any())
        assert float(((got - want).abs()[fine] / want.abs()[fine].clamp(min=1.0)).max()) <= 1e-5
    # a pixel is marked where a finite change is not 0 (a NaN is above no threshold): few changes lie so close to 0 that the kernels differ
    (_, dy, m), (_, _, wm) = out["auto"], out["off"]
    assert torch.equal(m, ((dy != 0) & ~dy.isnan()).any(1, keepdim=True).to(torch.uint8)) and float((m != wm).float().mean()) <= 1e-2


# A thresholded sigmoid on the TF32 kernel with partial groups of 16 channels and blocks that end in a group of none: what is sent, against
# the FP32 kernel.  Channels that do not exist take no part in the decision.
@pytest.mark.parametrize("cout", [16, 24, 40, 48, 64])
@pytest.mark.parametrize("stride", [1, 2])
def test_thresholded_sigmoid_of_partial_groups(dev, cout, stride):
    from maskedincrementeval_b200 import fields as fl, _native as nat
    from maskedincrementeval_b200.incr_modules.e2depth_incr import ConvLayerIncr
    old, out, thr = fl.config.tensor_cores, {}, 0.02
    try:
        for mode in ("auto", "off"):
            fl.config.tensor_cores = mode
            torch.manual_seed(21)
            layer = ConvLayerIncr(32, cout, 3, stride, 1, activation="sigmoid").to(dev).eval()
            g = torch.Generator(device=dev).manual_seed(22)
            steps = []
            with torch.no_grad():
                layer.forward_refresh_reservoirs(cl(torch.randn(2, 32, 42, 54, generator=g, device=dev)))
                layer.activation.threshold = thr
                for frac in (0.05, 0.0, 0.3):
                    d = cl(0.1 * torch.randn(2, 32, 42, 54, generator=g, device=dev) * (torch.rand(2, 1, 42, 54, generator=g, device=dev) < frac))
                    dy, m = layer([d, None])
                    assert layer.conv2d.last_used_tensor_cores == (mode == "auto")
                    assert torch.equal(m.pixel_mask(), (dy != 0).any(1, keepdim=True).to(torch.uint8))
                    steps.append((dy.clone(), m.pixel_mask().clone()))
            out[mode] = steps
    finally:
        fl.config.tensor_cores = old
    # changes below 0.1 of a sum whose inputs are 2^-11 off: at most 1e-4 from the FP32 kernel's where both send; few lie so close to the threshold
    assert any(0.0 < float(m.float().mean()) < 0.5 for _, m in out["off"])
    for (dy, m), (want, wm) in zip(out["auto"], out["off"]):
        both = (dy != 0) & (want != 0)
        assert not bool(both.any()) or float((dy - want)[both].abs().max()) <= 2e-4
        assert float((m != wm).float().mean()) <= 0.01 and float(((dy != 0) != (want != 0)).float().mean()) <= 0.01


# ragged and whole tiles, one column block and three, both widths of block
@pytest.mark.parametrize("cin,cout,h,w", [(32, 32, 41, 50), (64, 96, 9, 9), (64, 64, 104, 100), (48, 36, 16, 24)])
def test_dense_step_writes_whole_tile_words(dev, cin, cout, h, w):
    """mie_conv_refresh_step makes no list: the tile words it finds may hold anything, and a bad dilation is refused as ever."""
    from maskedincrementeval_b200 import fields as fl, _native as nat
    from maskedincrementeval_b200.incr_modules._algebra import NATIVE
    from maskedincrementeval_b200.incr_modules.e2depth_incr import ConvLayerIncr
    torch.manual_seed(27)
    c, x = ConvLayerIncr(cin, cout, 3, 1, 1, activation="relu").to(dev).eval(), cl(torch.randn(2, cin, h, w, device=dev))
    with torch.no_grad():
        y, m = NATIVE.conv(c.conv2d, NATIVE.lift(x), c.activation)
        want, plan = y.clone(), c.conv2d._plan(2, h, w, dev)
        plan.out_bits.fill_(-1)
        taken = next(iter(c.conv2d._prepared_refresh.values()))
        nat.check(nat.lib.mie_conv_refresh_step(C.byref(taken.args), x.data_ptr(), cin, C.addressof(taken.job.c), nat.stream_ptr(dev)), "refresh_step")
        assert torch.equal(plan.out_bits, fl.full_mask(2, h, w, dev).bits) and torch.equal(plan.out, want)
        for field, value, status in (("k", 9, nat.EUNSUPPORTED), ("N", 0, nat.EINVAL), ("flags", None, nat.EINVAL)):
            bad = type(taken.job.c).from_buffer_copy(taken.job.c)
            setattr(bad, field, value)
            assert nat.lib.mie_conv_refresh_step(C.byref(taken.args), x.data_ptr(), cin, C.addressof(bad), nat.stream_ptr(dev)) == status


@pytest.mark.parametrize("cin,offset", [(64, 1), (64, 2), (48, 3), (50, 1)])
def test_extension_on_an_input_that_is_not_aligned(dev, cin, offset):
    """An input at an odd address runs as one at an even address does: the same kernel, the same bits."""
    from maskedincrementeval_b200.ext.pointops import pointops_functional as pf
    g = torch.Generator(device=dev).manual_seed(28)
    w = torch.randn(cin, 3, 3, 64, generator=g, device=dev) * 0.04
    store = torch.randn(2 * 33 * 41 * cin + 4, generator=g, device=dev)
    x = store[offset:offset + 2 * 33 * 41 * cin].view(2, 33, 41, cin).permute(0, 3, 1, 2)
    assert x.data_ptr() % 16
    y, _ = pf.functional_conv_module(x, w, mask=None, stride=(1, 1), padding=(1, 1))
    want, _ = pf.functional_conv_module(x.clone(memory_format=torch.channels_last), w, mask=None, stride=(1, 1), padding=(1, 1))
    assert torch.equal(y, want)


# Thin layers on both sides of the rule that gives them to the tensor cores: no step less precise than the FP32 kernel's, from isolated pixels
# to dense changes, in the change and in the state
@pytest.mark.parametrize("cin,taken", [(8, False), (12, True), (16, True), (20, False)])
@pytest.mark.parametrize("stride", [1, 2])
@pytest.mark.parametrize("frac", [0.0005, 0.005, 0.05, 0.4])
def test_thin_layers_are_no_less_precise_than_fp32(dev, cin, taken, stride, frac):
    from maskedincrementeval_b200 import fields as fl, _native as nat
    from maskedincrementeval_b200.incr_modules.e2depth_incr import ConvLayerIncr
    old, err = fl.config.tensor_cores, {}
    try:
        for mode in ("auto", "off"):
            fl.config.tensor_cores = mode
            torch.manual_seed(30)
            layer = ConvLayerIncr(cin, 24, 3, stride, 1, activation="relu").to(dev).eval()
            c, g = layer.conv2d, torch.Generator(device=dev).manual_seed(31)
            change = state = 0.0
            for _ in range(4):
                with torch.no_grad():
                    layer.forward_refresh_reservoirs(cl(torch.randn(1, cin, 97, 131, generator=g, device=dev)))
                    before = layer.activation.in_res.reservoir.double()
                    d = cl(torch.randn(1, cin, 97, 131, generator=g, device=dev) * (torch.rand(1, 1, 97, 131, generator=g, device=dev) < frac))
                    want = F.conv2d(d.double(), c.weight.double(), stride=stride, padding=1)
                    change += float((c.forward_fused([d, None], None, None)[0].double() - want).square().sum())
                    layer([d, None])
                    assert bool(nat.lib.mie_conv_is_exact(C.byref(c._plan(1, 97, 131, dev).args))) == (taken and mode == "auto")
                    state += float((layer.activation.in_res.reservoir.double() - before - want).square().sum())
            err[mode] = change ** 0.5, state ** 0.5
    finally:
        fl.config.tensor_cores = old
    assert err["auto"][0] <= err["off"][0] and err["auto"][1] <= err["off"][1], err


def test_dense_evaluation_as_callers_of_earlier_versions_ask_for_it(dev):
    """mie_split_exact and mie_conv_tiles with two input fields: the same as with the field itself."""
    from maskedincrementeval_b200 import fields as fl, _native as nat
    from maskedincrementeval_b200.incr_modules._algebra import NATIVE
    from maskedincrementeval_b200.incr_modules.e2depth_incr import ConvLayerIncr
    torch.manual_seed(32)
    layer, n, h, w = ConvLayerIncr(5, 32, 5, 1, 2, activation="relu").to(dev).eval(), 2, 33, 41
    x = cl(torch.randn(n, 5, h, w, device=dev))
    with torch.no_grad():
        y, m = NATIVE.conv(layer.conv2d, NATIVE.lift(x), layer.activation)
        want, plan = y.clone(), layer.conv2d._plan(n, h, w, dev)
        both = torch.full((2, n, h, w, 8), float("nan"), device=dev)
        st = nat.stream_ptr(dev)
        nat.check(nat.lib.mie_split_exact(x.data_ptr(), 5, 5, n * h * w, both[0].data_ptr(), both[1].data_ptr(), 8, st), "split_exact")
        a = nat.ConvArgs.from_buffer_copy(next(iter(layer.conv2d._prepared_refresh.values())).args)
        a.in_, a.in_lo, a.in_ps = both[0].data_ptr(), both[1].data_ptr(), 8
        job = plan.tail.c
        nat.check(nat.lib.mie_tiles_dilate(job.in_bits, job.N, job.Hin, job.Win, job.Hout, job.Wout, job.k, job.stride, job.pad, job.union_bits, job.out_bits,
                                           job.list, job.stale, job.counts, job.flags, st), "tiles_dilate")
        plan.out.zero_()
        nat.check(nat.lib.mie_conv_tiles(C.byref(a), st), "conv_tiles")
        assert torch.equal(both[0, ..., :5].permute(0, 3, 1, 2), x) and bool((both[0, ..., 5:8] == 0).all()) and bool((both[1] == 0).all())
        assert torch.equal(plan.out, want) and torch.equal(plan.out_bits, fl.full_mask(n, h, w, dev).bits)
