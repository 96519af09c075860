"""What a caller writes into or reads out of a network between two calls, on the kernels that keep copies of
the state, against the CUDA-core kernels phase by phase, which keep none, or the numpy oracle.  Bounds:
common.TOL per tensor."""
import ctypes

import numpy as np
import pytest

from common import DELTA_TOL, TF32_TOL, TOL, build_gpu_net, rel_err, rel_err_of_update

pytestmark = pytest.mark.gpu


def _simple(sizes, batch, act="tanh"):
    return dict(kind="simple", sizes=sizes, batch=batch, T=3, steps=1, options={},
                hyper=dict(lr=0.01, ir=0.1, lmbda=0.0, act=act))


RUN = _simple([64, 256, 256, 256, 10], 256)  # SimplePC layers on operand planes
ROWS = _simple([37, 70, 33, 10], 20)         # row segments


@pytest.fixture
def plan_of(built_library, monkeypatch):
    """Builds a network with its kernels' copies, or ("plain") without any."""
    from deepity_b200 import _lib
    lib = _lib.load()
    monkeypatch.setenv("DPC_RECTANGULAR_MIN_WORK", "0")

    def build(case, plain=False, precision="fp32"):
        for name in ("DPC_DISABLE_TENSOR_CORES", "DPC_DISABLE_RESIDENT"):
            monkeypatch.setenv(name, "1") if plain else monkeypatch.delenv(name, raising=False)
        net, x, y = build_gpu_net(case, precision)
        return lib, net, lib.dpcn_plan(net._h), x, y
    return build


def test_written_errors_of_simple_layers_are_used(plan_of):
    """The state update and the weight update read the errors a caller has set."""
    rng = np.random.default_rng(5)
    errors = {l: rng.normal(size=(256, 256)).astype(np.float32) for l in (1, 2, 3)}
    got = []
    for plain in (False, True):
        lib, net, plan, x, y = plan_of(RUN, plain)
        net.train_step_native(x, y, 3)
        for l, e in errors.items():
            net.set_tensor(l, "e", e)
        assert lib.dpc_update_state(plan, 1, 2) == 0 and lib.dpc_update_weights(plan, 0, 4, 0) == 0
        got.append({(l, n): net.get_tensor(l, n) for l in (1, 2) for n in ("z", "W")})
    for key, ref in got[1].items():
        assert rel_err(ref, got[0][key]) <= TOL, key


CALLS = {"python": lambda n, x, y: n.train_step(x, y, 3), "native": lambda n, x, y: n.train_step_native(x, y, 3),
         "projection": lambda n, x, y: n.train_step_with_projection(x, y, 3),
         "predict": lambda n, x, y: n.predict(x, 3)}


@pytest.mark.parametrize("call", sorted(CALLS))
def test_input_activations_read_back_as_last_fed(call, plan_of):
    """zF, and the weight update of a caller that has written it."""
    got = []
    for plain in (False, True):
        lib, net, plan, x, y = plan_of(RUN, plain)
        for _ in range(2):
            CALLS[call](net, x, y)
        out = {f"zF.{l}": net.get_tensor(l, "zF") for l in range(4)}
        mine = np.random.default_rng(6).normal(size=(256, 256)).astype(np.float32)
        net.set_tensor(2, "zF", mine)
        assert np.array_equal(net.get_tensor(2, "zF"), mine.ravel())
        assert lib.dpc_update_weights(plan, 0, 4, 0) == 0
        out.update({f"W.{l}": net.get_tensor(l, "W") for l in range(4)})
        net.set_optimizer("ADAM")  # another plan, whose kernels read zF
        lib.dpcn_plan(net._h)
        out.update({f"kept.{l}": net.get_tensor(l, "zF") for l in range(4)})
        got.append(out)
    for key, ref in got[1].items():
        assert rel_err(ref, got[0][key]) <= TOL, key


@pytest.mark.parametrize("call", sorted(CALLS))
def test_input_activations_after_row_segments(call, plan_of):
    """zF is what the last forward pass of the call was fed, as phase by phase."""
    got = []
    for plain in (False, True):
        lib, net, plan, x, y = plan_of(ROWS, plain)
        assert lib.dpc_rows_available(plan) == (0 if plain else 1)
        for _ in range(2):
            CALLS[call](net, x, y)
        got.append([net.get_tensor(l, "zF") for l in range(3)])
    for l, (a, ref) in enumerate(zip(*got)):
        assert rel_err(ref, a) <= TOL, l


@pytest.mark.parametrize("case", [RUN, ROWS], ids=["run", "rows"])
@pytest.mark.parametrize("graph", [True, False])
def test_a_step_without_settling_learns_from_what_was_last_fed(graph, case, plan_of):
    """Mode 2 without a settling step is a weight update alone (train_step_python of the oracle)."""
    from common import _oracle_kwargs, make_case, make_oracle
    params, x, y = make_case("simple", case["sizes"], case["batch"])
    orc = make_oracle("simple", case["sizes"], case["batch"], params, **_oracle_kwargs(case))
    _, net, _, _, _ = plan_of(case)
    net.set_use_graph(graph)
    for T in (3, 0, 0, 2, 0):
        orc.train_step_python(x, y, T)
        net.train_step(x, y, T)
    for l, p in enumerate(params):
        for name in ("W", "b"):
            update = np.asarray(orc.get(l, name)).reshape(p[name].shape) - p[name]
            assert rel_err_of_update(orc.get(l, name), net.get_tensor(l, name), p[name]) <= DELTA_TOL, (l, name)
            assert np.abs(update).max() > 0


def test_precision_set_on_a_live_plan(plan_of):
    """dpc_set_precision without a new plan: single-pass TF32 products from the next call on, and back."""
    _, plain, _, _, _ = plan_of(RUN, plain=True)
    _, ref, _, x, y = plan_of(RUN, precision="tf32")
    lib, net, _, _, _ = plan_of(RUN)
    ctx = lib.dpcn_context(net._h)
    for n in (ref, net, plain):
        n.set_use_graph(False)
    lib.dpcn_plan(net._h)
    assert lib.dpc_set_precision(ctx, 1) == 0
    assert net.train_step_native(x, y, 3) == pytest.approx(ref.train_step_native(x, y, 3), rel=1e-6)
    plain.train_step_native(x, y, 3)
    for l in range(4):
        for name in ("z", "e", "W", "b", "zF"):
            assert rel_err(ref.get_tensor(l, name), net.get_tensor(l, name)) <= 1e-6, (l, name)
    # the operands of the second step start from the same state on both sides
    assert lib.dpc_set_precision(ctx, 0) == 0
    for l in range(4):
        plain.set_tensor(l, "W", net.get_tensor(l, "W"))
        plain.set_tensor(l, "b", net.get_tensor(l, "b"))
    for n in (net, plain):
        n.train_step(x, y, 0)  # a weight update from the TF32 step's operands
    for l in range(4):
        assert rel_err(plain.get_tensor(l, "W"), net.get_tensor(l, "W")) <= TF32_TOL, l
        plain.set_tensor(l, "W", net.get_tensor(l, "W"))
        plain.set_tensor(l, "b", net.get_tensor(l, "b"))
    for n in (net, plain):
        n.train_step(x, y, 3)
    for l in range(4):
        for name in ("z", "e", "W", "b", "zF"):
            assert rel_err(plain.get_tensor(l, name), net.get_tensor(l, name)) <= TOL, (l, name)


def test_split_scheme_changed_on_a_live_plan(plan_of, monkeypatch):
    """DPC_FP32_SCHEME is read when a phase is launched."""
    _, plain, _, x, y = plan_of(RUN, plain=True)
    _, net, _, _, _ = plan_of(RUN)
    for n in (net, plain):
        n.set_use_graph(False)
    for scheme in ("tf32x3", None):
        monkeypatch.setenv("DPC_FP32_SCHEME", scheme) if scheme else monkeypatch.delenv("DPC_FP32_SCHEME")
        for n in (net, plain):
            n.train_step(x, y, 3)
        for l in range(4):
            for name in ("z", "e", "W", "b", "zF"):
                assert rel_err(plain.get_tensor(l, name), net.get_tensor(l, name)) <= TOL, (scheme, l, name)


class _ConvLayer(ctypes.Structure):  # dpc_conv_layer
    _fields_ = ([(n, ctypes.c_int32) for n in
                 "in_c out_c in_h in_w k_h k_w s_h s_w p_h p_w out_h out_w act opt".split()] +
                [(n, ctypes.c_float) for n in "lr ir lmbda".split()] +
                [(n, ctypes.c_void_p) for n in "z e W b preact mu g g_W g_b m_W v_W m_b v_b t".split()])


@pytest.fixture
def conv_plan(built_library):
    """A convolution plan of one weight layer over tensors of the test's own: (lib, plan, tensors, sync)."""
    import torch

    from deepity_b200 import _lib
    lib = _lib.load()
    made = []

    def build(B, C, O, H, k, pad, weight_offset=0):
        torch.manual_seed(3)
        P = H + 2 * pad - k + 1
        flat = torch.randn(O * C * k * k + 4, device="cuda") / k
        shapes = dict(z=(B, C, H, H), e=(B, C, H, H), b=(O,), preact=(B, O, P, P), mu=(B, O, P, P), g=(B, O, P, P),
                      g_W=(O, C * k * k), g_b=(O,))
        t = {n: torch.randn(*s, device="cuda") for n, s in shapes.items()}
        t["W"] = flat[weight_offset:weight_offset + O * C * k * k].view(O, C * k * k)
        top = {n: torch.randn(B, O, P, P, device="cuda") for n in ("z", "e")}
        table = (_ConvLayer * 2)()
        for n, v in dict(in_c=C, out_c=O, in_h=H, in_w=H, k_h=k, k_w=k, s_h=1, s_w=1, p_h=pad, p_w=pad, out_h=P,
                         out_w=P, act=8, lr=0.1, ir=0.1).items():
            setattr(table[0], n, v)
        for n, v in dict(in_c=O, in_h=P, in_w=P, act=10, lr=0.1, ir=0.1).items():
            setattr(table[1], n, v)
        for layer, tensors in zip(table, (t, top)):
            for n, v in tensors.items():
                setattr(layer, n, v.data_ptr())
        torch.cuda.synchronize()
        ctx, plan = ctypes.c_void_p(), ctypes.c_void_p()
        _lib.check(lib.dpc_create(0, ctypes.byref(ctx)))
        _lib.check(lib.dpc_conv_plan_create(ctx, table, 2, B, ctypes.byref(plan)))
        made.append((plan, ctx, t, top, flat))
        return lib, plan, t, top, lambda: _lib.check(lib.dpc_sync(ctx))
    yield build
    for plan, ctx, *_ in made:
        lib.dpc_conv_plan_destroy(plan)
        lib.dpc_destroy(ctx)


@pytest.mark.parametrize("offset", [0, 1, 2])
def test_dense_convolution_weights_of_any_alignment(offset, conv_plan):
    """The whole image under one kernel, rows of 64 weights that start on any float."""
    lib, plan, t, top, sync = conv_plan(3, 4, 5, 4, 4, 0, weight_offset=offset)
    assert lib.dpc_conv_images_available(plan) == 1
    assert lib.dpc_conv_images_segment(plan, 1 << 0 | 1 << 11 | 1 << 13, 0, 1) == 0  # first, closing errors, predictions
    sync()
    pre = t["z"].reshape(3, -1).double() @ t["W"].double().T + t["b"].double()
    assert rel_err(pre.cpu(), t["preact"].cpu()) <= TOL
    assert rel_err((top["z"].reshape(3, -1) - pre.tanh()).cpu(), top["e"].cpu()) <= TOL


def test_page_locked_inputs_may_be_written_again_after_the_call(built_library):
    """dpcn_train_step without an energy returns when it has read its host inputs, page-locked or not: here
    three steps are queued ahead of the copies of the fourth."""
    import torch

    from deepity_b200 import _lib
    lib = _lib.load()
    case = dict(kind="dkp", sizes=[512] * 25 + [10], batch=1024, T=2, steps=1, options={},
                hyper=dict(lr=1e-3, ir=0.1, fl=1e-3, lmbda=0.0, act="tanh"))
    got = []
    for overwrite in (False, True):
        net, x, y = build_gpu_net(case)
        xs, ys = torch.from_numpy(x).pin_memory(), torch.from_numpy(y).pin_memory()
        at = [ctypes.cast(t.data_ptr(), _lib.c_f32p) for t in (xs, ys)]
        for _ in range(4):
            _lib.check(lib.dpcn_train_step(net._h, at[0], xs.numel(), at[1], ys.numel(), 2, None))
        if overwrite:
            xs.fill_(7.0)
            ys.zero_()
        _lib.check(lib.dpc_sync(lib.dpcn_context(net._h)))
        got.append([net.get_tensor(0, "z"), net.get_tensor(25, "z"), net.get_tensor(24, "W")])
    for a, b in zip(*got):
        assert np.array_equal(a, b)


def test_convolution_gradient_sums_stay_in_the_callers_buffers(conv_plan):
    """g_W and g_b are the raw sums of one update whatever they held before it, and hold them after it."""
    import torch
    lib, plan, t, top, sync = conv_plan(3, 2, 4, 5, 3, 1)
    for n in ("g_W", "g_b"):
        t[n].fill_(7.0)
    before = {n: t[n].double() for n in ("W", "b")}
    cols = torch.nn.functional.unfold(t["z"], 3, padding=1).double()
    dW = torch.einsum("bop,brp->or", t["g"].reshape(3, 4, -1).double(), cols)
    db = t["g"].double().sum((0, 2, 3))
    torch.cuda.synchronize()
    assert lib.dpc_conv_update_weights(plan, 0, 0) == 0
    sync()
    for n, ref in (("g_W", dW), ("g_b", db), ("W", before["W"] + 0.1 / 3 * dW), ("b", before["b"] + 0.1 / 3 * db)):
        assert rel_err(ref.cpu(), t[n].cpu()) <= 1e-5, n  # 75 products of unit size in fp32


def test_softmax_error_formed_in_the_head_with_an_unclamped_input(built_library):
    """The range of a forward pass starts at the input layer: the head is launched on its own all the same."""
    from deepity_b200 import _lib
    lib = _lib.load()
    case = dict(kind="full", sizes=[40, 128, 10], batch=33, T=2, steps=1, options=dict(cross_entropy=1),
                hyper=dict(lr=0.01, ir=0.1, fl=0.01, lmbda=0.0, act="tanh"))
    net, x, y = build_gpu_net(case)
    net.train_step(x, y, 2)
    plan = lib.dpcn_plan(net._h)
    assert lib.dpc_plan_fused_cross_entropy(plan) == 1
    net.set_tensor(2, "e", np.zeros((33, 10), np.float32))
    net.set_tensor(1, "fe", np.zeros((33, 10), np.float32))
    ERR, FE, CACHED, CE = 2, 8, 16, 64
    assert lib.dpc_forward(plan, 0, 2, ERR | FE | CE) == 0
    z = [net.get_tensor(l, "z").reshape(33, -1) for l in range(3)]
    W, b = net.get_tensor(1, "W").reshape(10, 128), net.get_tensor(1, "b")
    pre = z[1].astype(np.float64) @ W.T + b
    s = np.exp(np.tanh(pre) - np.tanh(pre).max(1, keepdims=True))
    e = z[2] - s / s.sum(1, keepdims=True)
    assert rel_err(e, net.get_tensor(2, "e")) <= TOL
    assert rel_err(e * (1 - np.tanh(pre) ** 2), net.get_tensor(1, "fe")) <= TOL
    assert lib.dpc_forward(plan, 1, 1, ERR | CACHED | CE) == -1  # no head kernel runs


def test_errors_under_a_softmax_top_after_a_recorded_step(plan_of):
    """A replayed step leaves the top layer's softmax error in fp32 only; an update of the caller's own reads it."""
    case = dict(RUN, sizes=[64, 256, 256, 256], options=dict(cross_entropy=1))
    got = []
    for plain in (False, True):
        lib, net, plan, x, y = plan_of(case, plain)
        for _ in range(3):
            net.train_step_with_projection(x, y, 3)
        assert lib.dpc_update_state(plan, 1, 2) == 0 and lib.dpc_update_weights(plan, 0, 3, 0) == 0
        got.append({(l, n): net.get_tensor(l, n) for l in (1, 2) for n in ("z", "W")})
    for key, ref in got[1].items():
        assert rel_err(ref, got[0][key]) <= TOL, key


def test_device_pointers_keep_their_network_alive(built_library):
    """Views made from a pointer read the network's memory: it must not go with the last name of the network."""
    import gc
    import weakref
    net, _, _ = build_gpu_net(ROWS)
    alive, ptr = weakref.ref(net), net.tensor_ptr(1, "W")
    del net
    gc.collect()
    assert alive() is not None and ptr == alive().tensor_ptr(1, "W")
    del ptr
    gc.collect()
    assert alive() is None
