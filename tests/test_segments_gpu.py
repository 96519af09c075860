"""Row segments (dpc_resident.cu) and image segments (dpc_conv_resident.cu): whole settling loops in
one kernel, against the numpy oracle, at the sizes where their splits change.  Bounds: common.TOL per
tensor, common.ADAM_TOL with an Adam-type optimizer, common.DELTA_TOL on the parameter updates."""
import numpy as np
import pytest

from common import (ADAM_TOL, DELTA_TOL, TOL, build_gpu_net, compare_outputs, initial_parameters,
                    run_gpu, run_oracle)
from conv_common import build_conv_gpu_net, chain, run_conv_gpu, run_conv_oracle

pytestmark = pytest.mark.gpu


def _available(case):
    from deepity_b200 import _lib
    lib = _lib.load()
    net, _, _ = build_gpu_net(case)
    return lib.dpc_rows_available(lib.dpcn_plan(net._h))


def _case(kind, sizes, batch, act, T=3, steps=2, **options):
    hyper = dict(lr=0.01, ir=0.1, lmbda=0.0, act=act)
    if options.get("optimizer"):
        hyper["lr"] = 1e-3
    if kind != "simple":
        hyper["fl"] = hyper["lr"]
    mode = options.pop("mode", "train_step")
    return dict(kind=kind, sizes=sizes, batch=batch, T=T, steps=steps, hyper=hyper, options=options, mode=mode)


ROWS = {
    # 1, 2, 4 and 8 rows per block (148 SMs), the last block not full
    "rows_1": _case("simple", [37, 70, 10], 147, "sigmoid", mode="projection"),
    "rows_2": _case("dkp", [37, 70, 33, 10], 149, "tanh"),
    "rows_4": _case("simple", [20, 33, 7], 299, "gelu", mode="python"),
    "rows_8": _case("dkp", [16, 40, 40, 5], 601, "tanh"),
    "rows_8_two_groups": _case("simple", [12, 24, 4], 1201, "tanh"),
    # ordered sums (Adam-type optimizers, kinked activations) with streamed rows
    "exact_adamw": _case("dkp", [100, 300, 200, 77, 10], 50, "relu", optimizer="ADAMW", psi_optimizer="ADAM"),
    "exact_hard_tanh": _case("simple", [30, 129, 65, 3], 151, "hard_tanh"),
    # ... over input rows that end inside each of the load groups
    "exact_input_quads": _case("dkp", [84, 33, 9], 3, "relu"),
    "exact_input_singles": _case("dkp", [107, 33, 9], 601, "relu"),
    # sliced sums over input rows that are not 16-byte aligned: a strip of loads and a remainder, many
    "input_singles": _case("dkp", [107, 33, 9], 3, "tanh"),
    "input_singles_8_rows": _case("simple", [1971, 33, 9], 601, "sigmoid"),
    # every term of the state update, more layers than warps share evenly
    "residual_momentum": _case("full", [33] + [64] * 9 + [10], 5, "gelu", mupc=1, residual=1, momentum=0.9),
    "cross_entropy": _case("full", [45, 61, 32, 17], 149, "tanh", cross_entropy=1),
    "simple_cross_entropy": _case("simple", [45, 61, 17], 9, "tanh", cross_entropy=1),
    # weights beyond one SM's shared memory: some layers or rows are read from L2 on every pass
    "streamed": _case("dkp", [64, 400, 350, 10], 20, "tanh"),
}


@pytest.mark.parametrize("name", sorted(ROWS))
def test_row_segments_match_oracle(name, built_library):
    case = ROWS[name]
    assert _available(case) == 1
    adam = "optimizer" in case["options"]
    compare_outputs(run_oracle(case), run_gpu(case), ADAM_TOL if adam else TOL, name,
                    init=None if adam else initial_parameters(case), delta_tol=None if adam else DELTA_TOL)


@pytest.mark.parametrize("sizes,batch,act", [((64, 1024, 1000, 10), 9, "tanh"),  # 4 MB above the first layer
                                             ((64,) + (128,) * 10 + (10,), 149, "tanh"),  # short sums, many layers
                                             ((64, 384, 384, 10), 20, "relu"),   # 605 KB, ordered sums
                                             ((64, 384, 256, 10), 149, "relu"),  # 404 KB, two rows a block
                                             # several groups of rows a block: input layer and others
                                             ((784, 264, 64, 10), 2400, "tanh")])
def test_row_segments_stop_at_their_weight_limit(sizes, batch, act, built_library):
    case = _case("dkp", list(sizes), batch, act)
    assert _available(case) == 0
    compare_outputs(run_oracle(case), run_gpu(case), TOL, "over the limit")


@pytest.mark.parametrize("kind,batch,available", [("dkp", 1184, 1), ("dkp", 1185, 0), ("simple", 1185, 1),
                                                  ("simple", 4096, 1)])
def test_row_segments_of_several_groups_a_block(kind, batch, available, built_library):
    """106 KB of ordered sums a round (the input layer's 279 KB count a quarter) on 148 SMs of 8-row blocks."""
    assert _available(_case(kind, [784, 91, 91, 10], batch, "relu")) == available


# Segments on clusters: layers narrower than a block's share of four columns, rows that are not 16-byte aligned, the last
# group not full; one, two and four rows a task, several tasks a warp; an input that streams in one step and in many.
CLUSTERS = {
    # (SGD: with AdamW at three rows a belief of all kernels, whose bits are equal, is 1.7e-3 from the oracle's)
    "ordered_rows_1": _case("dkp", [100, 300, 200, 77, 10], 3, "relu"),
    "ordered_adamw": _case("dkp", [100, 300, 200, 77, 10], 50, "relu", optimizer="ADAMW", psi_optimizer="ADAM"),
    "ordered_rows_2": _case("dkp", [129, 131, 33, 7], 50, "hard_tanh"),
    "ordered_rows_4": _case("simple", [1971, 65, 65, 65, 3], 300, "relu", mode="projection"),
    "ordered_heads": _case("full", [256, 256, 128, 16], 33, "relu", momentum=0.9),  # lanes along K
    "ordered_ipc": _case("full", [64] * 5 + [16], 70, "gelu", optimizer="ADAMW", mupc=1, residual=1, momentum=0.9, ipc=1),
    "one_layer": _case("dkp", [784, 10], 50, "relu"),
    "sliced": _case("dkp", [70, 285, 131, 10], 16, "tanh"),
    "sliced_simple": _case("simple", [37, 202, 61, 10], 60, "sigmoid", mode="python"),
    "deep_residual": _case("full", [21] * 40 + [5], 6, "tanh", mupc=1, residual=1, momentum=0.9),
    "cross_entropy": _case("full", [45, 130, 66, 17], 20, "gelu", cross_entropy=1),
    "simple_cross_entropy": _case("simple", [45, 61, 17], 9, "tanh", cross_entropy=1),
}


@pytest.mark.parametrize("blocks", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("name", sorted(CLUSTERS))
def test_cluster_segments_match_oracle(name, blocks, monkeypatch, built_library):
    from deepity_b200 import _lib
    lib = _lib.load()
    monkeypatch.setenv("DPC_CLUSTER_SIZE", str(blocks))
    case = CLUSTERS[name]
    net, _, _ = build_gpu_net(case)
    clusters = lib.dpc_rows_clusters(lib.dpcn_plan(net._h))
    del net
    if clusters == 0:
        pytest.skip("the weights do not fit the shared memory of so many blocks")
    assert clusters == blocks
    adam = "optimizer" in case["options"]
    got = run_gpu(case)
    compare_outputs(run_oracle(case), got, ADAM_TOL if adam else TOL, name,
                    init=None if adam else initial_parameters(case), delta_tol=None if adam else DELTA_TOL)
    if name.startswith("ordered"):
        # one order of additions: the bits of the other kernels (energies are sums over blocks in any order)
        monkeypatch.setenv("DPC_DISABLE_CLUSTERS", "1")
        ref = run_gpu(case)
        for k, v in ref.items():
            assert k == "energies" or np.array_equal(v, got[k]), k


@pytest.mark.parametrize("kind,sizes,batch,act,blocks",
                         [("dkp", [100, 300, 200, 77, 10], 50, "relu", 4), ("simple", [784, 441, 441, 10], 25, "relu", 16),
                          ("dkp", [100, 47, 47, 10], 54, "relu", 0),   # a short chain: blocks by themselves
                          ("dkp", [64, 128, 128, 10], 64, "tanh", 0),  # sliced sums that fit one block
                          ("dkp", [100, 273, 273, 273, 10], 1, "tanh", 8),
                          ("dkp", [64, 1024, 1024, 10], 1, "tanh", 0),  # weights that fit no cluster
                          # several rows a cluster, where other kernels take 0.6 to 0.7 of the time
                          ("dkp", [784] + [128] * 9 + [37], 51, "relu", 0), ("dkp", [784] + [32] * 44 + [10], 79, "tanh", 0),
                          ("simple", [188] * 4 + [37], 192, "sigmoid", 0), ("simple", [100, 320, 320, 2], 128, "gelu", 0),
                          # a head on a wide layer, whose product is most of a step
                          ("dkp", [1960, 1960, 2], 48, "relu", 0), ("dkp", [784, 768, 16], 878, "sigmoid", 0)])
def test_which_networks_run_on_clusters(kind, sizes, batch, act, blocks, built_library):
    from deepity_b200 import _lib
    lib = _lib.load()
    net, _, _ = build_gpu_net(_case(kind, sizes, batch, act))
    assert lib.dpc_rows_clusters(lib.dpcn_plan(net._h)) == blocks


def _images(shape, convs, act, batch, **kw):
    return dict(layers=chain(shape, convs, act), batch=batch, T=3, steps=2, hyper=dict(lr=0.005, ir=0.1, lmbda=0.0),
                **kw)


IMAGES = {
    # more images than SMs; rectangular kernels, strides and paddings that leave ragged tiles
    "batch_over_sms": _images((1, 10, 10), [(8, 5, 5, 2, 2, 2, 2), (10, 5, 5, 1, 1, 0, 0)], "tanh", 151),
    "rectangular": _images((2, 11, 9), [(9, 3, 2, 2, 1, 1, 0), (17, 2, 3, 1, 2, 0, 1), (5, 5, 4, 1, 1, 0, 0)],
                           "sigmoid", 3),
    # channel counts one off the 8- and 16-wide tiles, a projection sweep first
    "channel_edges": _images((7, 8, 8), [(15, 3, 3, 1, 1, 1, 1), (33, 3, 3, 2, 2, 1, 1), (1, 4, 4, 1, 1, 0, 0)],
                             "gelu", 2, projection=1),
    "pointwise": _images((3, 4, 4), [(16, 1, 1, 1, 1, 0, 0), (10, 4, 4, 1, 1, 0, 0)], "relu", 1),
}


@pytest.mark.parametrize("channels,batch,available", [(92, 12, 1), (93, 12, 0), (93, 13, 1)])
def test_image_segments_of_few_images_stop_at_large_kernels(channels, batch, available, built_library):
    """92 x 92 kernels of 3 x 3 taps are 298 KB."""
    from deepity_b200 import _lib
    lib = _lib.load()
    case = _images((1, 6, 6), [(channels, 3, 3, 1, 1, 1, 1), (channels, 3, 3, 2, 2, 1, 1), (4, 3, 3, 1, 1, 0, 0)],
                   "tanh", batch)
    assert lib.dpc_conv_images_available(lib.dpcn_conv_plan(build_conv_gpu_net(case)._h)) == available
    compare_outputs(run_conv_oracle(case), run_conv_gpu(case), TOL, str(batch))


@pytest.mark.parametrize("name", sorted(IMAGES))
def test_image_segments_match_oracle(name, built_library):
    from deepity_b200 import _lib
    lib = _lib.load()
    case = IMAGES[name]
    assert lib.dpc_conv_images_available(lib.dpcn_conv_plan(build_conv_gpu_net(case)._h)) == 1
    compare_outputs(run_conv_oracle(case), run_conv_gpu(case), TOL, name)


def test_closing_segment_starts_from_the_stored_beliefs(built_library):
    """A segment without the input layer's prediction clears its planes and fills them from memory: the
    errors it leaves are z - mu of what memory holds, bit for bit, in every one of many runs.  Large
    planes and a small prediction to copy in between."""
    from conv_common import make_conv_case
    from deepity_b200 import _lib
    lib = _lib.load()
    case = _images((1, 6, 6), [(1, 3, 3, 1, 1, 1, 1), (40, 3, 3, 1, 1, 2, 2), (40, 3, 3, 1, 1, 1, 1)], "tanh", 296)
    net = build_conv_gpu_net(case)
    _, x, y = make_conv_case(case)
    net.train_step(x, y, 2)
    plan, ctx = lib.dpcn_conv_plan(net._h), lib.dpcn_conv_context(net._h)
    assert lib.dpc_conv_images_available(plan) == 1
    z = [net.get_tensor(l, "z") for l in range(4)]
    for _ in range(100):
        _lib.check(lib.dpc_conv_images_segment(plan, 1 << 11 | 1 << 13, 0, 1))  # closing errors, predictions stored
        _lib.check(lib.dpc_sync(ctx))
        for l in (1, 2, 3):
            assert np.array_equal(net.get_tensor(l, "e"), z[l] - net.get_tensor(l - 1, "mu")), l
