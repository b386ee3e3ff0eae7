"""A layer that is called again with the same kind of input takes a prepared call.  Whatever that call was decided by may
change between two calls: the prepared call has to be given up then, and the result has to be the one that a layer which
decides every call anew gives, to the bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu

N, C, H, W = 1, 32, 40, 56


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


@pytest.fixture(autouse=True)
def restore_config():
    from maskedincrementeval_b200 import _native as nat, fields as fl
    names = ("threshold", "carry", "tensor_cores", "tc_thresholded", "own_tiles", "kfenced_step", "input_threshold", "head_dilation", "tail_dilation")
    saved, own = {k: getattr(fl.config, k) for k in names}, nat.get_option(nat.OPT_TC_OWN_KERNELS)
    yield
    for k, v in saved.items():
        setattr(fl.config, k, v)
    nat.set_option(nat.OPT_TC_OWN_KERNELS, own)
    fl.forget_tails()


@pytest.fixture
def prepared(monkeypatch):
    """The outcomes of the prepared calls and refreshes of the test so far: True where one was taken."""
    from maskedincrementeval_b200.incr_modules import mask_incr_modules as mim
    taken = []

    def watch(cls):
        run = cls.run
        monkeypatch.setattr(cls, "run", lambda self, *a: (lambda out: (taken.append(out is not None), out)[1])(run(self, *a)))

    watch(mim._PreparedCall)
    watch(mim._PreparedRefresh)
    return taken


def cl(t):
    return t.contiguous(memory_format=torch.channels_last)


def _layer(dev):
    from maskedincrementeval_b200.incr_modules.e2depth_incr import ConvLayerIncr
    torch.manual_seed(0)
    return ConvLayerIncr(C, C, 3, 1, 1, activation="relu").to(dev).eval()


def _sparse(g, dev, std=0.5):
    return cl(torch.randn(N, C, H, W, generator=g, device=dev) * std * (torch.rand(N, 1, H, W, generator=g, device=dev) < 0.2))


def _decide_anew(layer):
    layer.conv2d._prepared.clear()
    layer.conv2d._prepared_refresh.clear()


def _set(obj, **kw):
    for k, v in kw.items():
        setattr(obj, k, v)


def _config(**kw):
    def change(layer):
        from maskedincrementeval_b200 import fields as fl
        _set(fl.config, **kw)
    return change


def _scaled(layer):
    with torch.no_grad():
        layer.conv2d.weight.mul_(1.5)


def _replaced(layer):
    layer.conv2d.weight = torch.nn.Parameter(layer.conv2d.weight.detach().clone() * -1.0)


def _moved(layer):
    layer.conv2d.weight.data = layer.conv2d.weight.detach().clone() * 0.5


def _state_replaced(layer):
    layer.activation.in_res.reservoir = cl(layer.activation.in_res.reservoir.clone() + 0.25)


def _option(layer):
    from maskedincrementeval_b200 import _native as nat
    nat.set_option(nat.OPT_TC_OWN_KERNELS, 0)


CHANGES = {
    "weight in place": _scaled, "weight replaced": _replaced, "weight moved": _moved,
    "precision": lambda l: _set(l.conv2d, precision="split"), "function": lambda l: _set(l.activation, op=torch.tanh),
    "threshold of the layer": lambda l: _set(l.activation, threshold=0.05), "threshold": _config(threshold=0.05), "state replaced": _state_replaced,
    "input threshold": _config(input_threshold=0.3), "tensor cores off": _config(tensor_cores="off"), "own tiles off": _config(own_tiles=False),
    "quantiser": _config(kfenced_step=0.25), "dilation at the head": _config(head_dilation=2048), "dilation in the tail": _config(tail_dilation=True),
    "option": _option,
}


@pytest.mark.parametrize("what", CHANGES)
@pytest.mark.parametrize("given", [False, True], ids=["mask derived", "mask given"])
def test_a_change_gives_the_prepared_call_up(dev, prepared, what, given):
    from maskedincrementeval_b200 import fields as fl
    a, b = _layer(dev), _layer(dev)
    g = torch.Generator(device=dev).manual_seed(1)
    x0, deltas = cl(torch.randn(N, C, H, W, generator=g, device=dev)), [_sparse(g, dev) for _ in range(4)]
    bits = fl.new_bits(N, H, W, dev)
    with torch.no_grad():
        for l in (a, b):
            l.forward_refresh_reservoirs(x0)
        for i, d in enumerate(deltas):
            if i == 2:
                for l in (a, b):
                    CHANGES[what](l)
            mask = fl.mask_from_delta(d, 0.0, bits) if given else None
            del prepared[:]
            ya, ma = a([d, mask])
            if i < 3:       # the call after the change may be prepared again, under the new conditions
                assert (True in prepared) == (i == 1), (i, prepared)
            _decide_anew(b)
            yb, mb = b([d, mask])
            assert torch.equal(ya, yb) and torch.equal(ma.bits, mb.bits), (what, i)
            assert torch.equal(a.activation.in_res.reservoir, b.activation.in_res.reservoir), (what, i)


def test_a_change_of_precision_reaches_the_result(dev):
    """set_precision after the first call: the next step is the fp32 convolution (2e-5), not the TF32 one (2^-11)."""
    from maskedincrementeval_b200.incr_modules.mask_incr_modules import set_precision
    from oracle import restatement as R
    l = _layer(dev)
    g = torch.Generator(device=dev).manual_seed(1)
    with torch.no_grad():
        l.forward_refresh_reservoirs(cl(torch.randn(N, C, H, W, generator=g, device=dev)))
        for _ in range(2):
            l([_sparse(g, dev), None])
        set_precision(l, "split")
        res, d = l.activation.in_res.reservoir.cpu().contiguous(), _sparse(g, dev)
        y, _ = l([d, None])
    want, _ = R.act_incr(res, R.conv_delta(d.cpu().contiguous(), l.conv2d.weight.detach().cpu(), 1, 1), "relu")
    assert float((y.cpu() - want).abs().max()) <= 2e-5 * max(float(want.abs().max()), 1.0)


INPUTS = {
    "another buffer": lambda d: (cl(d.clone()), True),
    "a slice of a wider field": lambda d: (cl(torch.cat([d, d], 1))[:, :C], False),
    "not channels-last": lambda d: (d.contiguous(), False),
    "another geometry": lambda d: (cl(d[:, :, :24, :48]), False),
}


@pytest.mark.parametrize("what", INPUTS)
def test_another_kind_of_input_gives_the_prepared_call_up(dev, prepared, what):
    a, b = _layer(dev), _layer(dev)
    g = torch.Generator(device=dev).manual_seed(2)
    x0 = cl(torch.randn(N, C, H, W, generator=g, device=dev))
    d, taken = INPUTS[what](_sparse(g, dev))
    with torch.no_grad():
        for l in (a, b):
            l.forward_refresh_reservoirs(x0)
        for _ in range(2):
            e = _sparse(g, dev)
            a([e, None])
            _decide_anew(b)
            b([e, None])
        for l in (a, b):
            if d.shape != x0.shape:
                l.forward_refresh_reservoirs(cl(x0[:, :, :24, :48]))
        del prepared[:]
        ya, ma = a([d, None])
        assert (True in prepared) == taken
        _decide_anew(b)
        yb, mb = b([d, None])
        assert torch.equal(ya, yb) and torch.equal(ma.bits, mb.bits)
        assert torch.equal(a.activation.in_res.reservoir, b.activation.in_res.reservoir)


def _bias_replaced(layer):
    layer.conv2d.bias = torch.nn.Parameter(layer.conv2d.bias.detach() + 1.0)


def _bias_in_place(layer):
    with torch.no_grad():
        layer.conv2d.bias.add_(1.0)


REFRESH_CHANGES = {
    "weight in place": (_scaled, False), "weight replaced": (_replaced, False), "weight moved": (_moved, False), "bias replaced": (_bias_replaced, False),
    "bias in place": (_bias_in_place, True),      # the kernel reads it where it is
    "function": (lambda l: _set(l.activation, op=torch.tanh), False), "state replaced": (_state_replaced, False),
    "tensor cores off": (_config(tensor_cores="off"), False),
}


@pytest.mark.parametrize("what", REFRESH_CHANGES)
@pytest.mark.parametrize("with_addend", [False, True])
def test_a_change_gives_the_prepared_refresh_up(dev, prepared, what, with_addend):
    from maskedincrementeval_b200 import fields as fl
    from maskedincrementeval_b200.incr_modules._algebra import NATIVE
    a, b = _layer(dev), _layer(dev)
    g = torch.Generator(device=dev).manual_seed(3)
    xs = [cl(torch.randn(N, C, H, W, generator=g, device=dev)) for _ in range(3)]
    addend = [cl(torch.randn(N, C, H, W, generator=g, device=dev)), fl.full_mask(N, H, W, dev)] if with_addend else None
    change, taken = REFRESH_CHANGES[what]
    with torch.no_grad():
        for i, x in enumerate(xs):
            if i == 2:
                for l in (a, b):
                    change(l)
            del prepared[:]
            ya, _ = NATIVE.conv(a.conv2d, NATIVE.lift(x), a.activation, addend=addend)
            assert (True in prepared) == (i == 1 or (i == 2 and taken)), (i, prepared)
            _decide_anew(b)
            yb, _ = NATIVE.conv(b.conv2d, NATIVE.lift(x), b.activation, addend=addend)
            assert torch.equal(ya, yb) and torch.equal(a.activation.in_res.reservoir, b.activation.in_res.reservoir), (what, i)


@pytest.mark.parametrize("refresh", [False, True])
def test_a_new_parameter_at_the_old_address(dev, refresh):
    """A parameter that is taken off a layer may be followed by one at the same address with the same version: its values count."""
    from maskedincrementeval_b200.incr_modules._algebra import NATIVE
    a, b = _layer(dev), _layer(dev)
    g = torch.Generator(device=dev).manual_seed(4)
    x0, d = cl(torch.randn(N, C, H, W, generator=g, device=dev)), _sparse(g, dev)
    w = [torch.randn(C, C, 3, 3, generator=g, device=dev) * 0.06 for _ in range(2)]
    with torch.no_grad():
        for v in w:
            a.conv2d.weight = None
            a.conv2d.weight = torch.nn.Parameter(v.clone())
            NATIVE.conv(a.conv2d, NATIVE.lift(x0), a.activation)
            if not refresh:
                ya, _ = a([d, None])
        b.conv2d.weight = torch.nn.Parameter(w[1].clone())
        NATIVE.conv(b.conv2d, NATIVE.lift(x0), b.activation)
        if not refresh:
            yb, _ = b([d, None])
            assert torch.equal(ya, yb)
        assert torch.equal(a.activation.in_res.reservoir, b.activation.in_res.reservoir)
        assert torch.equal(a.conv2d.conv2d_weights, b.conv2d.conv2d_weights)


def test_geometries_in_turn_keep_their_prepared_calls(dev, prepared):
    """A convolution that is called at two geometries in turn decides each of them once."""
    a, b = _layer(dev).conv2d, _layer(dev).conv2d
    g = torch.Generator(device=dev).manual_seed(5)
    with torch.no_grad():
        for i in range(3):
            for h, w in ((H, W), (24, 48)):
                d = cl(_sparse(g, dev)[:, :, :h, :w])
                del prepared[:]
                ya, ma = a([d, None])
                assert prepared == ([True] if i else [])
                b._prepared.clear()
                yb, mb = b([d, None])
                assert torch.equal(ya, yb) and torch.equal(ma.bits, mb.bits)


@pytest.mark.parametrize("refresh", [False, True])
def test_prepared_calls_hold_the_packed_filter(dev, prepared, refresh):
    """load_state_dict drops the packed filters; where it leaves the parameter as it was, the prepared call still holds its own."""
    from maskedincrementeval_b200.incr_modules._algebra import NATIVE
    a, b = _layer(dev), _layer(dev)
    g = torch.Generator(device=dev).manual_seed(6)
    x0 = cl(torch.randn(N, C, H, W, generator=g, device=dev))
    with torch.no_grad():
        for i in range(3):
            d = _sparse(g, dev)
            if i == 2:
                a.conv2d.load_state_dict({}, strict=False)
                taken = [torch.full((s,), float("nan"), device=dev) for s in (9 * 32 * 32, 2 * 9 * 32 * 32, 9 * 32 * 32) for _ in range(8)]
            for l in (a, b):
                del prepared[:]
                if refresh:
                    NATIVE.conv(l.conv2d, NATIVE.lift(x0), l.activation)
                else:
                    if i == 0:
                        l.forward_refresh_reservoirs(x0)
                    l([d, None])
                assert prepared == ([True] if i else [])
            assert torch.equal(a.activation.in_res.reservoir, b.activation.in_res.reservoir)
            assert bool(a.activation.in_res.reservoir.isfinite().all())
    del taken


@pytest.mark.parametrize("refresh", ["native", "library"])
@pytest.mark.parametrize("how", ["in place", "replaced"])
def test_a_captured_step_follows_new_parameters(dev, refresh, how):
    """Parameters change while a step is captured: the packed filters that it reads are dropped, so it has to be recorded again."""
    from maskedincrementeval_b200 import fields as fl
    from maskedincrementeval_b200.incr_modules.fireflownet_incr import FireFlowNetIncr
    from maskedincrementeval_b200.runtime import IncrementalRunner

    def runner():
        torch.manual_seed(7)
        net = FireFlowNetIncr(dict(base_num_channels=32, kernel_size=3, mask_output=False), 2, compat="exact").to(dev).eval()
        return net, IncrementalRunner(net)

    def change(net):
        with torch.no_grad():
            for i, p in enumerate(net.parameters()):
                if how == "in place":
                    p.mul_(1.0 + 0.1 * (i % 3))
            if how == "replaced":
                for m in net.modules():
                    if isinstance(m, torch.nn.Conv2d):
                        m.weight = torch.nn.Parameter(m.weight.detach() * 1.25)

    old = fl.config.refresh
    fl.config.refresh = refresh
    torch.backends.cudnn.allow_tf32 = False
    try:
        g = torch.Generator(device=dev).manual_seed(8)
        xs = [cl(torch.randn(1, 2, 40, 56, generator=g, device=dev)) for _ in range(5)]
        (net, run), (twin, fresh) = runner(), runner()
        run.refresh(xs[0])
        for x in xs[1:4]:
            run.step(x)
        replays = run.graph_replays
        assert replays == 2
        change(net), change(twin)
        run.refresh(xs[0]), fresh.refresh(xs[0])
        taken = [torch.full((n,), float("nan"), device=dev) for n in (9 * 32 * 32, 9 * 96 * 32, 9 * 8 * 32) for _ in range(16)]
        for i, x in enumerate(xs[1:]):
            assert torch.equal(run.step(x), fresh.step(x)), i
        assert run.graph_replays == replays + 3      # one eager step, then captured again
        run.check()
        del taken
    finally:
        fl.config.refresh = old


def _double_head(net):
    with torch.no_grad():
        conv = next(m for m in net.modules() if isinstance(m, torch.nn.Conv2d))
        conv.weight.mul_(2.0)


def _replace_parameter(net):
    conv = [m for m in net.modules() if isinstance(m, torch.nn.Conv2d)][1]
    conv.weight = torch.nn.Parameter(conv.weight.detach() * 0.5)


def _replace_bias(net):
    conv = [m for m in net.modules() if isinstance(m, torch.nn.Conv2d)][2]
    conv.bias = torch.nn.Parameter(conv.bias.detach() + 0.25)


def _replace_activation(net):
    from maskedincrementeval_b200.incr_modules.mask_incr_modules import nnReservedActivation
    acts = [m for m in net.modules() if isinstance(m, nnReservedActivation) and m.op is torch.relu]
    acts[1].op = torch.tanh


def _new_reservoir(net):
    from maskedincrementeval_b200.incr_modules.mask_incr_modules import nnReservedActivation
    acts = [m for m in net.modules() if isinstance(m, nnReservedActivation) and m.in_res.reservoir is not None]
    acts[0].in_res.reservoir = acts[0].in_res.reservoir.clone(memory_format=torch.channels_last)


def _fp32_kernels(net):
    from maskedincrementeval_b200 import fields as fl
    fl.config.tensor_cores = "off"


@pytest.mark.parametrize("change", [None, _double_head, _replace_parameter, _replace_bias, _replace_activation, _new_reservoir, _fp32_kernels])
def test_a_replayed_dense_pass_is_an_eager_one(dev, change):
    """IncrementalRunner replays the dense pass once three in a row found the model alike; a change of any input of the pass, and
    steps in between, give what a runner that never replays gives."""
    from maskedincrementeval_b200 import fields as fl
    from maskedincrementeval_b200.incr_modules.e2depth_incr import E2VIDRecurrentIncr
    from maskedincrementeval_b200.runtime import IncrementalRunner
    torch.manual_seed(21)
    net = E2VIDRecurrentIncr(dict(num_bins=5, skip_type="sum", recurrent_block_type="convlstm", num_encoders=3, base_num_channels=8,
                                  num_residual_blocks=1, norm=None, use_upsample_conv=True, compat="exact")).to(dev).eval()
    g = torch.Generator(device=dev).manual_seed(22)
    frames = [torch.randn(1, 5, 40, 56, generator=g, device=dev).contiguous(memory_format=torch.channels_last) for _ in range(3)]
    old = fl.config.tensor_cores
    try:
        run = IncrementalRunner(net)
        for i in range(7):
            run.refresh(frames[i % 3])
        assert run._pass_graph is not None
        if change is not None:
            change(net)
        run.refresh(frames[1])
        outs = [run.refresh(frames[2]).clone()] + [run.step(f).clone() for f in frames]
        outs.append(run.refresh(frames[0]).clone())
        eager = IncrementalRunner(net, use_graph=False)
        want = [eager.refresh(frames[2]).clone()] + [eager.step(f).clone() for f in frames]
        want.append(eager.refresh(frames[0]).clone())
    finally:
        fl.config.tensor_cores = old
    for y, w in zip(outs, want):
        assert torch.equal(y, w)


def _flow_net(dev, cls=None):
    from maskedincrementeval_b200.incr_modules.fireflownet_incr import FireFlowNetIncr
    torch.manual_seed(23)
    return (cls or FireFlowNetIncr)(dict(base_num_channels=16, kernel_size=3, mask_output=False), 2, compat="exact").to(dev).eval()


def _frames(dev, channels, h, w):
    g = torch.Generator(device=dev).manual_seed(24)
    return [cl(torch.randn(1, channels, h, w, generator=g, device=dev)) for _ in range(3)]


def test_a_dense_pass_on_the_library_follows_its_switches(dev, monkeypatch):
    """The delayed EV-FlowNet's dense pass runs on PyTorch's operators, which follow switches of their own: it is not replayed."""
    from maskedincrementeval_b200.incr_modules.delayedevflownet_incr import DelayedEVFlowNetIncr
    from maskedincrementeval_b200.runtime import IncrementalRunner
    torch.manual_seed(25)
    net = DelayedEVFlowNetIncr(dict(base_num_channels=32, kernel_size=3, mask_output=False), 2, compat="exact").to(dev).eval()
    frames = _frames(dev, 2, 64, 64)
    monkeypatch.setattr(torch.backends.cudnn, "allow_tf32", True)
    run = IncrementalRunner(net)
    for i in range(7):
        run.refresh(frames[i % 3])
    monkeypatch.setattr(torch.backends.cudnn, "allow_tf32", False)
    got = [y.clone() for y in run.refresh(frames[0])]
    with torch.no_grad():
        want = net.forward_refresh_reservoirs(frames[0])["flow"]
    assert all(torch.equal(y, w) for y, w in zip(got, want))


def test_a_dense_pass_that_does_more_than_launch_kernels_is_run(dev):
    """A subclass may count its passes or read from the device in them; so may a method set on an object."""
    from maskedincrementeval_b200.incr_modules.fireflownet_incr import FireFlowNetIncr
    from maskedincrementeval_b200.runtime import IncrementalRunner
    seen = []

    class Counting(FireFlowNetIncr):
        def forward_refresh_reservoirs(self, x):
            out = super().forward_refresh_reservoirs(x)
            seen.append(float(out["flow"][0].abs().max()))
            return out

    frames = _frames(dev, 2, 40, 56)
    run = IncrementalRunner(_flow_net(dev, Counting))
    for i in range(8):
        y = run.refresh(frames[i % 3])
        assert len(seen) == i + 1 and seen[-1] == float(y.abs().max())
    net = _flow_net(dev)
    whole, calls = net.E2._run, []
    net.E2._run = lambda ops, x: (calls.append(1), whole(ops, x))[1]
    run = IncrementalRunner(net)
    for i in range(8):
        run.refresh(frames[i % 3])
    assert len(calls) == 8


@pytest.mark.parametrize("thr", [0.0, 3e-2])
@pytest.mark.parametrize("name", ["e2depth", "fireflow"])
def test_steps_behind_replayed_dense_passes(dev, name, thr):
    """Dense passes alone until one is recorded, then steps, whose buffers are made only now, passes and steps in turn: what a runner
    without graphs gives."""
    from maskedincrementeval_b200 import fields as fl
    from maskedincrementeval_b200.incr_modules.e2depth_incr import E2VIDRecurrentIncr
    from maskedincrementeval_b200.runtime import IncrementalRunner

    def net():
        if name == "fireflow":
            return _flow_net(dev)
        torch.manual_seed(26)
        return E2VIDRecurrentIncr(dict(num_bins=5, skip_type="sum", recurrent_block_type="convlstm", num_encoders=3, base_num_channels=16,
                                       num_residual_blocks=1, norm=None, use_upsample_conv=True, compat="exact")).to(dev).eval()

    fl.config.threshold = thr
    frames = _frames(dev, 5 if name == "e2depth" else 2, 40, 56)
    runners = [IncrementalRunner(net(), use_graph=g) for g in (True, False)]

    def both(call, *a):
        y, want = (getattr(r, call)(*a) for r in runners)
        assert torch.equal(y, want), call

    for i in range(6):
        both("refresh", frames[i % 3])
    assert runners[0]._pass_graph is not None
    for i in range(4):
        both("step", frames[i % 3])
    for round_ in range(7):
        both("refresh", frames[round_ % 3])
        if round_ % 2:
            for i in range(3):
                both("step", frames[(round_ + i) % 3])
    assert runners[0]._pass_graph is not None


def test_a_dense_pass_that_cannot_be_recorded(dev, monkeypatch):
    """A recording that fails costs nothing but the attempt: passes go on one by one, and the next attempt is made for another state."""
    from maskedincrementeval_b200.runtime import IncrementalRunner
    frames, net, tried = _frames(dev, 2, 40, 56), _flow_net(dev), []

    class Refused(torch.cuda.graph):
        def __enter__(self):
            tried.append(self.capture_error_mode)
            raise RuntimeError("refused")

    run, eager = IncrementalRunner(net), IncrementalRunner(_flow_net(dev), use_graph=False)

    def passes(count):
        for i in range(count):
            assert torch.equal(run.refresh(frames[i % 3]), eager.refresh(frames[i % 3]))

    with monkeypatch.context() as m:
        m.setattr(torch.cuda, "graph", Refused)
        passes(9)
        assert tried == ["thread_local"] and run._pass_graph is None
        for r in (run, eager):
            _double_head(r.model)
        passes(9)
        assert len(tried) == 2
    for r in (run, eager):
        _double_head(r.model)
    passes(7)
    assert run._pass_graph is not None
    passes(2)
    assert torch.equal(run.step(frames[1]), eager.step(frames[1]))
