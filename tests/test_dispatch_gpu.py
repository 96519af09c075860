"""The variants a launch is chosen from (GEMM tiles, widths of pair tiles, head kernels, the run of
SimplePC layers, the state update that forms its own error) against the numpy oracle at the edges of
their ranges.  Bounds: common.TOL per tensor (ADAM_TOL, TF32_TOL where those modes are on) and
common.DELTA_TOL on the parameter updates."""
import numpy as np
import pytest

from common import (ADAM_TOL, DELTA_TOL, DELTA_TOL_TF32, TF32_TOL, TOL, build_gpu_net, compare_outputs,
                    initial_parameters, make_case, make_oracle, run_gpu, run_oracle)
from conv_common import chain, run_conv_gpu, run_conv_oracle

pytestmark = pytest.mark.gpu


def _case(kind, sizes, batch, act="tanh", T=3, steps=2, mode="train_step", lr=0.01, **options):
    hyper = dict(lr=lr, ir=0.1, lmbda=0.0, act=act)
    if kind != "simple":
        hyper["fl"] = lr
    return dict(kind=kind, sizes=sizes, batch=batch, T=T, steps=steps, hyper=hyper, options=options, mode=mode)


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def _up(a, b):
    return -(-a // b)


def _tiles(case, width, phase="weights"):
    """Output tiles of the CUDA-core products of a phase: all weight sums; a settling pass (the input layer's prediction
    is cached) or the state update of the hidden layers, without heads of 16 units and less, which are not theirs."""
    sizes, batch = case["sizes"], case["batch"]
    pairs = list(zip(sizes, sizes[1:]))
    if phase == "weights":
        return sum(_up(a, width) * _up(b, width) for a, b in pairs)
    pairs = [(a, b) for a, b in pairs[1:] if b > 16]
    return sum(_up(batch, width) * _up(b if phase == "forward" else a, width) for a, b in pairs)


def _check(case, name, precision="fp32"):
    adam = "optimizer" in case["options"]
    tol = TF32_TOL if precision == "tf32" else (ADAM_TOL if adam else TOL)
    delta = DELTA_TOL_TF32 if precision == "tf32" else DELTA_TOL
    compare_outputs(run_oracle(case), run_gpu(case, precision=precision), tol, name,
                    init=None if adam else initial_parameters(case), delta_tol=None if adam else delta)


# The sweep on clusters: 8, 16 and 32 rows a cluster of two and four blocks, the shortest run and the largest
# batch, beliefs with and without stored predictions, pre-activations and the residual term.  Smooth activations: a pre-activation
# of 1 280 x 256 x 6 that rounds to the other side of a ReLU's kink moves a whole row (1e-3 of the largest error here with
# the residual term, on these kernels and on the tiles alike; 5e-4 without it, on CUDA cores too).
SWEEPS = {
    "sweep_2x8_shortest": _case("dkp", [20] + [256] * 3 + [10], 256),
    "sweep_2x16": _case("full", [20] + [256] * 5 + [10], 1024, "gelu"),
    "sweep_2x32_residual": _case("full", [20] + [256] * 6 + [10], 1280, "tanh", residual=1),
    "sweep_4x8": _case("dkp", [20] + [512] * 4 + [10], 256, "sigmoid"),
    "sweep_4x16_residual": _case("full", [20] + [512] * 5 + [10], 512, "gelu", residual=1, momentum=0.9),
    "sweep_4x32": _case("dkp", [20] + [512] * 4 + [10], 1024),
    "sweep_2x32_largest": _case("dkp", [20] + [256] * 4 + [10], 2304, T=2, steps=1),
}


@pytest.mark.parametrize("precision", ["fp32", "tf32"])
@pytest.mark.parametrize("name", list(SWEEPS))
def test_cluster_sweep(name, precision, monkeypatch):
    from torch.profiler import ProfilerActivity, profile
    case = SWEEPS[name]
    _check(case, name, precision)
    with profile(activities=[ProfilerActivity.CUDA]) as launches:
        own = run_gpu(case, precision=precision)
    assert any("cluster_sweep" in event.key for event in launches.key_averages())
    # the tiles that split K form the same sums in the same order
    monkeypatch.setenv("DPC_DISABLE_CLUSTER_SWEEP", "1")
    other = run_gpu(case, precision=precision)
    different = [key for key in own if key != "energies" and not np.array_equal(own[key], other[key])]
    assert not different, different


def test_sweep_of_more_clusters_than_run_at_once():
    """36 clusters of four blocks: 148 SMs hold fewer, so the tiles take the sweep (1152 rows, TF32)."""
    from torch.profiler import ProfilerActivity, profile
    case = _case("dkp", [20] + [512] * 3 + [10], 1152, T=1, steps=1)
    with profile(activities=[ProfilerActivity.CUDA]) as launches:
        _check(case, "sweep_4x32_two_waves", "tf32")
    names = [event.key for event in launches.key_averages()]
    assert any("pc_tc_kernel" in name for name in names) and not any("cluster_sweep" in name for name in names)


@pytest.mark.parametrize("precision", ["fp32", "tf32"])
@pytest.mark.parametrize("batch", [256, 1024])
def test_deep_cluster_sweep_repeats(batch, precision, monkeypatch, built_library):
    """130 layers of 512 units, 8 and 32 rows a cluster of four blocks: weights beyond L2, blocks of a cluster that drift
    apart.  The beliefs after a sweep are those of the tiles, bit for bit, every time (predictions change no weights)."""
    import torch
    case = _case("dkp", [512] * 131 + [10], batch, T=0)

    def beliefs(net, x):
        net.predict(x, 0)
        return torch.cat([torch.as_tensor(_View(net.tensor_ptr(l, "z"), (batch, 512)), device="cuda")
                          for l in range(1, 131)]).clone()

    net, x, _ = build_gpu_net(case, precision)
    first = beliefs(net, x)
    for _ in range(5):
        assert torch.equal(beliefs(net, x), first)
    monkeypatch.setenv("DPC_DISABLE_CLUSTER_SWEEP", "1")
    net, x, _ = build_gpu_net(case, precision)
    assert torch.equal(beliefs(net, x), first)


class _View:
    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "version": 3, "data": (ptr, False)}


GROUPED = {
    # 32 x 32 tiles: one row over a tile, K not a multiple of the stage, rows not 16-byte aligned
    "gemm_32_edges": _case("dkp", [33, 65, 31, 10], 65),
    "gemm_32_aligned": _case("simple", [64, 96, 32, 4], 32, mode="projection"),
    "gemm_32_many": _case("dkp", [67, 641, 12], 961),
    # blocks of four warps, of two (three aligned tiles an SM and more)
    "gemm_four_warps": _case("full", [37, 45, 45, 6], 33, "relu", residual=1, momentum=0.9),
    "gemm_two_warps": _case("simple", [64, 512, 512, 8], 961, "relu"),
    # more runs of layers of one shape than a launch lists
    "gemm_many_shapes": _case("dkp", [16] + [40, 12] * 125 + [4], 33, "relu", T=2),
    "gemm_adamw": _case("dkp", [35, 66, 65, 6], 70, lr=1e-3, optimizer="ADAMW"),
    # the head kernels: partial groups of rows, one and two rows per warp, 16 units, softmax in the head
    "head_ce": _case("full", [40, 128, 10], 301, "gelu", cross_entropy=1),
    "head_ce_two_rows": _case("full", [40, 132, 16], 2051, cross_entropy=1),
    "head_simple_ce": _case("simple", [40, 256, 10], 259, mode="projection", cross_entropy=1),
    "head_simple": _case("simple", [40, 384, 13], 2051, mode="python"),
    # ... several pairs of rows a warp, an odd number of units, a second chunk of 512 that is not full; weights beyond shared
    # memory; momentum and 14 units in the state update, rows that end inside its ring
    "head_turns": _case("dkp", [40, 640, 9], 4099),
    "head_unstaged": _case("full", [20, 2564, 15], 67),
    "head_unstaged_simple": _case("simple", [20, 2568, 16], 1030, mode="projection"),
    "head_state_momentum": _case("full", [40, 256, 14], 301, "gelu", momentum=0.9),
    "head_state_simple_16": _case("simple", [40, 128, 14], 1027, mode="projection"),
    # column sums in row order: more than one group of 32 columns, rows that end inside a buffer
    "column_sums": _case("dkp", [24, 70, 33], 1031, "relu"),
    # batches that end with a group of 64 rows, one row behind it, inside the first; feedback weights of one more
    # terminal unit than 16, of three times 16, rows that are aligned and that are not
    "batch_sums_64": _case("dkp", [36, 33, 17], 64, "relu"),
    "batch_sums_257": _case("full", [32, 68, 64, 48], 257, "hard_tanh"),
    "batch_sums_3": _case("dkp", [70, 31, 32, 20], 3, "relu"),
}


@pytest.mark.parametrize("act", ["sigmoid", "tanh", "gelu", "esigmoid"])
@pytest.mark.parametrize("kind,units", [("simple", 10), ("simple", 14), ("full", 10)])
def test_head_state_update_rounds_like_the_general_kernel(kind, units, act, built_library, monkeypatch):
    """Rows of a batch are independent and both kernels add up in ascending order: the beliefs under a head (a kernel of its
    own from 256 rows on) are those of the general kernel at one row less, bit for bit."""
    monkeypatch.setenv("DPC_DISABLE_RESIDENT", "1")
    params, x, y = make_case(kind, [64, 256, units], 256)
    out = []
    for batch in (255, 256):
        options = dict(mupc=1) if kind == "full" else {}
        net, _, _ = build_gpu_net(_case(kind, [64, 256, units], batch, act, **options))
        for l, p in enumerate(params):
            for name, v in p.items():
                net.set_tensor(l, name, v)
        step = net.train_step_with_projection if kind == "simple" else net.train_step
        step(x[:batch], y[:batch], 4)
        out.append(np.asarray(net.get_tensor(1, "z")).reshape(batch, 256))
    assert np.array_equal(out[0], out[1][:255])


@pytest.mark.parametrize("name", sorted(GROUPED))
def test_grouped_launches_match_oracle(name, built_library, monkeypatch):
    monkeypatch.setenv("DPC_DISABLE_RESIDENT", "1")
    _check(GROUPED[name], name)


# 64 x 64 tiles (1.75 an SM and more) and 32 x 32 ones of two warps with rows copied element by element (six an SM and
# more): the tiles' edges, both ways of copying, every epilogue; the phases that are checked to take them
LARGE = {
    "unaligned": (_case("dkp", [35, 1030, 1025, 6], 1100, "relu", T=2, steps=1), 64, ("weights", "forward", "state")),
    "residual_momentum": (_case("full", [64, 640, 640, 12], 1740, "gelu", mupc=1, residual=1, momentum=0.9), 64,
                          ("forward", "state")),
    "simple": (_case("simple", [64, 644, 640, 12], 1740, "sigmoid", mode="projection"), 64, ("forward", "state")),
    # (smooth: of 1.6 million preactivations a pass one is likely to lie within 1e-7 of a kink, where f' depends on
    # the order of additions)
    "two_warps_forward": (_case("dkp", [33, 319, 319, 63], 2557, "tanh", T=2), 32, ("forward",)),
    "two_warps_state": (_case("full", [33, 319, 319, 63], 1533, "tanh", residual=1, momentum=0.9), 32, ("state",)),
}


@pytest.mark.parametrize("name", sorted(LARGE))
def test_large_launches_match_oracle(name, built_library, monkeypatch):
    monkeypatch.setenv("DPC_DISABLE_RESIDENT", "1")
    case, tile, phases = LARGE[name]
    for phase in phases:
        large = _tiles(case, 64, phase) >= 1.75 * _sms() and 8 * _tiles(case, 64, phase) <= 3 * _tiles(case, 32, phase)
        assert large == (tile == 64) and (large or _tiles(case, 32, phase) >= 6 * _sms())
    _check(case, name)


# Steps of twice the length (aligned rows, sums of 128 and more): sums that end with a step, one quad behind it, in a
# step's last and first eight; rows of a tile that do not exist; on 32 x 32 tiles of four warps (two tiles an SM and
# less), of two (up to five) and on 64 x 64 ones
LONG = {
    "four_warps_128": _case("dkp", [128, 128, 132, 128, 10], 33),
    "four_warps_260": _case("simple", [260, 252, 248, 140, 12], 5, "sigmoid", mode="projection"),
    "four_warps_batch": _case("full", [132, 256, 256, 132, 12], 129, "gelu", momentum=0.9),
    "four_warps_adamw": _case("dkp", [128, 256, 260, 12], 128, "relu", lr=1e-3, optimizer="ADAMW"),
    "two_warps": _case("dkp", [64, 320, 320, 320, 320, 100], 452, T=2),
    "large": _case("dkp", [132, 1028, 1032, 100], 1000, T=2, steps=1),
}


@pytest.mark.parametrize("name", sorted(LONG))
def test_long_steps_match_oracle(name, built_library, monkeypatch):
    monkeypatch.setenv("DPC_DISABLE_RESIDENT", "1")
    case, sms = LONG[name], _sms()
    tiles = _tiles(case, 32, "forward")
    assert tiles <= 2 * sms if name.startswith("four") else 3 * sms <= tiles <= 5 * sms if name == "two_warps" else \
        _tiles(case, 64, "forward") >= 1.75 * sms
    _check(case, name)


@pytest.mark.parametrize("kind,sizes,batch,optimizer", [("dkp", [64, 1028, 1032, 12], 70, "ADAMW"),
                                                        ("full", [67, 1030, 1025, 7], 61, "ADAM")])
def test_adam_updates_on_large_tiles(kind, sizes, batch, optimizer, built_library):
    """Of a million weights some have gradients of the size of the rounding, whose step may go the other way.  So the
    moments, which are linear and quadratic in the gradient, are held to the bound of the SGD updates, and the weights
    to the step that the network's own moments give (fp32 rounding of the step and of the sum)."""
    case = _case(kind, sizes, batch, T=2, steps=1, lr=1e-3, optimizer=optimizer)
    case["hyper"].update(lmbda=0.01, fl=0.0)  # (no direct feedback: the weights change in this update alone)
    assert _tiles(case, 64) >= 1.75 * _sms()
    params, x, y = make_case(kind, sizes, batch)
    orc = make_oracle(kind, sizes, batch, params, **case["hyper"], optimizer=optimizer)
    orc.train_step(x, y, 2)
    net, _, _ = build_gpu_net(case)
    net.train_step(x, y, 2)
    for l in range(3):
        m, v, w = (net.get_tensor(l, n).astype(np.float64) for n in ("weight.m", "weight.v", "W"))
        for got, name, tol in ((m, "weight.m", DELTA_TOL), (v, "weight.v", 2 * DELTA_TOL)):
            ref = np.asarray(orc.get(l, name), dtype=np.float64).ravel()
            assert np.abs(ref - got).max() <= tol * np.abs(ref).max(), (l, name)
        decay = 1e-3 * 0.01 if optimizer == "ADAMW" else 0.0
        step = 1e-3 * np.sqrt(1 - 0.999) / (1 - 0.9)
        ref = params[l]["W"].ravel().astype(np.float64) * (1 - decay) - step * m / (np.sqrt(v) + 1e-8)
        assert np.abs(ref - w).max() <= 4 * np.finfo(np.float32).eps * np.abs(ref).max() + 1e-5 * 1e-3, l


# Forward products of SimplePC layers on 64 x 64 tiles, which transform their operand: from six 32 x 32 tiles an SM on,
# rows that are 16-byte aligned, that are not, and K that ends inside a step
FED = {
    "aligned": _case("simple", [64, 256, 256, 252, 100], 1508, "esigmoid", T=4),
    "unaligned": _case("simple", [33, 250, 255, 251, 101], 1507, "tanh", T=4),
    "ordered": _case("simple", [64, 256, 250, 256, 68], 1508, "relu", T=4, mode="projection"),
}


@pytest.mark.parametrize("name", sorted(FED))
def test_operands_of_large_tiles_are_transformed(name, built_library, monkeypatch):
    monkeypatch.setenv("DPC_DISABLE_RESIDENT", "1")
    case = FED[name]
    assert _tiles(case, 32, "forward") > 6 * _sms() and _sms() < _tiles(case, 64, "forward") < 1.75 * _sms()
    _check(case, name)


# Sums over the batch: fewer rows than a group, one over it, rows split over clusters; 16 and 17 rows in a tile;
# more terminal units than a tile; deep networks, of more
# shapes than a launch lists too; Psi sums of tensor-core layers among others
BATCH_SUMS = {
    "one_row": _case("dkp", [20, 30, 5], 1),
    "edges": _case("dkp", [33, 65, 31, 40], 9),
    "clusters": _case("simple", [67, 31, 17], 1031, mode="projection"),
    "columns": _case("dkp", [24, 70, 33], 1031),
    "many_layers": _case("dkp", [16] + [12] * 130 + [4], 5, T=2),
    "many_shapes": _case("dkp", [16] + [40, 12] * 125 + [4], 9, T=2),
    "beside_tensor_cores": _case("dkp", [64, 256, 256, 17], 256),
    "beside_tensor_cores_rows_split": _case("full", [72, 256, 256, 16], 1024, "gelu"),
}


@pytest.mark.parametrize("name", sorted(BATCH_SUMS))
def test_batch_sums_match_oracle(name, built_library, monkeypatch):
    monkeypatch.setenv("DPC_DISABLE_RESIDENT", "1")
    _check(BATCH_SUMS[name], name)


# Twelve 32 x 32 tiles an SM and more: the weight sums leave the batch products, with few rows or with outputs that fill
# 64 x 64 tiles; Psi stays
WIDE = {
    "few_rows": (_case("dkp", [40, 800, 1001, 900, 10], 33, T=2), True),
    "rows": (_case("full", [40, 960, 1022, 768, 10], 70, "gelu", T=2), True),
    "simple": (_case("simple", [40, 960, 1022, 768, 10], 70, mode="projection", T=4), True),
    "padded": (_case("dkp", [40, 710, 707, 711, 710, 708, 10], 70, T=2), False),
}


@pytest.mark.parametrize("staged", [False, True])
@pytest.mark.parametrize("name", sorted(WIDE))
def test_weight_sums_of_wide_layers_match_oracle(name, staged, built_library):
    from deepity_b200 import _lib
    case, by_gemm = WIDE[name]
    assert _tiles(case, 32) >= 12 * _sms()
    assert (4 * _tiles(case, 64) <= 1.05 * _tiles(case, 32) or case["batch"] <= 64) == by_gemm
    compare_outputs(run_oracle(case), run_gpu(case, staged_gradients=staged), TOL, name,
                    init=initial_parameters(case), delta_tol=DELTA_TOL)
    net, x, y = build_gpu_net(case)
    counts = []
    for _ in range(2):
        _lib.check(net._lib.dpc_update_weights(net._lib.dpcn_plan(net._h), 0, len(case["sizes"]), 0))
        counts.append(net.launch_count)
    psi = case["kind"] != "simple"
    assert counts[1] - counts[0] == (2 + psi if by_gemm else 1)  # weights, biases, Psi


@pytest.mark.parametrize("kind", ["simple", "full"])
@pytest.mark.parametrize("act", ["tanh", "relu"])
@pytest.mark.parametrize("widths,deep", [([32], 400), ([40, 12], 200)])
def test_a_phase_of_a_deep_network_is_as_many_launches_as_of_a_shallow_one(widths, deep, act, kind,
                                                                         built_library, monkeypatch):
    monkeypatch.setenv("DPC_DISABLE_RESIDENT", "1")
    passes = {}
    for layers in (20, deep):
        net, x, y = build_gpu_net(_case(kind, [64] + widths * (layers // len(widths)) + [10], 4, act), use_graph=False)
        counts = []
        for T in (2, 8):
            net.train_step(x, y, T)
            before = net.launch_count
            net.train_step(x, y, T)
            counts.append(net.launch_count - before)
        passes[layers] = counts[1] - counts[0]  # (of six settling passes: a sweep is a launch a layer)
    assert passes[deep] == passes[20] > 0


PAIR = {
    "dkp": _case("dkp", [64] + [256] * 4 + [10], 256, T=4),
    "full_residual_momentum": _case("full", [64] + [256] * 3 + [10], 512, "gelu", mupc=1, residual=1, momentum=0.9),
}


@pytest.mark.parametrize("width", ["64", "128", "256"])
@pytest.mark.parametrize("precision", ["fp32", "tf32"])
@pytest.mark.parametrize("name", sorted(PAIR))
def test_pair_tile_widths_match_oracle(name, precision, width, built_library, monkeypatch):
    monkeypatch.setenv("DPC_PAIR_TILE_WIDTH", width)
    _check(PAIR[name], f"{name} {precision} {width}", precision)


@pytest.mark.parametrize("width", ["0", "96", "100", "512"])
def test_other_pair_tile_widths_do_nothing(width, built_library, monkeypatch):
    """No other width is launched: the tiles are those of the rule, bit for bit."""
    plain = run_gpu(PAIR["dkp"])
    monkeypatch.setenv("DPC_PAIR_TILE_WIDTH", width)
    got = run_gpu(PAIR["dkp"])
    for key, ref in plain.items():
        if key != "energies":
            assert np.array_equal(ref, got[key]), key


# The state update of the layer above the clamped input forms its error itself, except in the last pass:
# one pass, several, single-CTA tiles (batch 128), 3xTF32 operands (Adam), a run that starts at the input
FROM_PREDICTION = {
    "one_pass": _case("dkp", [64] + [256] * 3 + [10], 256, T=1),
    "single_cta": _case("full", [64] + [256] * 3 + [10], 128, "gelu", T=3),
    "adam": _case("full", [64] + [256] * 3 + [10], 256, lr=1e-4, optimizer="ADAM", psi_optimizer="ADAM"),
    "from_the_input": _case("dkp", [256] * 4 + [10], 256, T=3),
    "ipc": _case("full", [64] + [256] * 3 + [10], 256, ipc=1),
}


@pytest.mark.parametrize("name", sorted(FROM_PREDICTION))
def test_state_update_from_the_prediction_below(name, built_library):
    _check(FROM_PREDICTION[name], name)


SIMPLE_RUN = {
    "train_step": _case("simple", [64] + [256] * 3 + [10], 256),
    "projection": _case("simple", [64] + [256] * 3 + [10], 512, "gelu", mode="projection"),
    "python": _case("simple", [256] * 4 + [10], 256, "sigmoid", mode="python"),
    "softmax": _case("simple", [64] + [256] * 3 + [10], 256, mode="projection", cross_entropy=1),
    # the softmax error is the work of a kernel of its own, right above the run
    "softmax_above": _case("simple", [64] + [256] * 3, 256, mode="projection", cross_entropy=1),
    "no_settling": _case("simple", [64] + [256] * 3 + [10], 256, T=0),
    "centred": _case("simple", [64] + [256] * 3 + [10], 256, center_weights=1),
}


@pytest.mark.parametrize("name", sorted(SIMPLE_RUN))
def test_simple_layers_on_operand_planes(name, built_library, monkeypatch):
    monkeypatch.setenv("DPC_RECTANGULAR_MIN_WORK", "0")
    _check(SIMPLE_RUN[name], name)


@pytest.mark.parametrize("sizes,batch", [((1000, 528, 10), 1152), ((1024, 512, 512, 10), 1024)])
def test_single_layers_of_few_tiles(sizes, batch, built_library):
    """Layers just over the tensor-core threshold: a quarter of the SMs' worth of full tiles or less."""
    _check(_case("dkp", list(sizes), batch, T=2), str(sizes))


@pytest.mark.parametrize("sizes,batch", [((20, 30, 5), 10), ((64, 256, 256, 256, 10), 256)])
def test_rates_set_between_steps_take_effect(sizes, batch, built_library):
    """A rate that is changed between two steps gives, bit for bit, what a network built with it gives."""
    case = _case("dkp", list(sizes), batch)
    a, x, y = build_gpu_net(case)
    a.train_step(x, y, 2)
    b, _, _ = build_gpu_net(dict(case, hyper=dict(case["hyper"], lr=0.03, ir=0.07)))
    names = [(l, n) for l in range(len(sizes) - 1) for n in ("W", "b", "Psi")]
    for l, n in names:
        b.set_tensor(l, n, a.get_tensor(l, n))
    a.set_learning_rate(0.03)
    a.set_inference_rate(0.07)
    assert a.train_step(x, y, 2) == b.train_step(x, y, 2)
    for l, n in names:
        assert np.array_equal(a.get_tensor(l, n), b.get_tensor(l, n)), (l, n)


@pytest.mark.parametrize("act,batch,projection", [("tanh", 3, 0), ("sigmoid", 1, 1)])
def test_convolution_layers_side_by_side(act, batch, projection, built_library, monkeypatch):
    monkeypatch.setenv("DPC_DISABLE_RESIDENT", "1")
    case = dict(layers=chain((2, 9, 9), [(5, 3, 3, 1, 1, 1, 1), (70, 3, 3, 2, 2, 1, 1), (9, 3, 3, 1, 1, 0, 0),
                                         (4, 3, 3, 1, 1, 0, 0)], act),
                batch=batch, T=4, steps=2, projection=projection, hyper=dict(lr=0.005, ir=0.1, lmbda=0.0))
    compare_outputs(run_conv_oracle(case), run_conv_gpu(case), TOL, "convolutions")
