"""Parity of the CUDA path (through the C ABI) with the CPU oracle and the recorded reference outputs."""
import threading

import numpy as np
import pytest

from conftest import legal_logits, load_case, load_compact
from lc0_b200 import _lib, mknet, network, weights
from oracle import oracle

pytestmark = pytest.mark.gpu

ALL = ["cfg1_mini", "cfg2_mini", "cfg3_mini", "cfg4_mini", "cfg1", "cfg2", "cfg3", "cfg4_2layer", "cfg1_mini_tanh",
       "cfg3_mini_tanh", "cfg3_mini_polenc"]
# fp32 verification mode, per logit: |got - want| <= 1e-5 * max(|want|, rms of the position's logits) + 1e-6.  The
# relative term is anchored at the position's typical logit because two fp32 implementations of the same network that
# only differ in summation order (the reference's OpenBLAS path and the numpy restatement) already differ by a few
# 1e-6 on logits of order one, whatever the size of the individual logit.
FP32_REL = 1e-5
FP32_FLOOR = 1e-6


def _assert_fp32_logits(got, want):
    rms = np.sqrt(np.mean(np.square(want), axis=-1, keepdims=True))
    bound = FP32_REL * np.maximum(np.abs(want), rms) + FP32_FLOOR
    excess = np.abs(got - want) - bound
    assert excess.max() <= 0, "worst logit exceeds its bound by %.3g" % excess.max()


def _assert_fp32_scalar(got, want):
    assert np.all(np.abs(got - want) <= FP32_REL * np.maximum(1.0, np.abs(want)) + FP32_FLOOR)

# fp16 storage with fp32 accumulation (north star: policy softmax and WDL/Q/M max-abs <= 2e-3).
HALF_ATOL = 2e-3


def _softmax_err_and_argmax(got, want, pos, n):
    worst, agree, decided = 0.0, 0, 0
    for i in range(n):
        lg = pos["legal"][i][:pos["n_legal"][i]]
        a = oracle.legal_softmax(got[i], lg)
        b = oracle.legal_softmax(want[i], lg)
        worst = max(worst, float(np.abs(a - b).max()))
        top = np.sort(b)[::-1]
        if len(top) < 2 or top[0] - top[1] > 2 * HALF_ATOL:  # near-ties may legitimately flip
            decided += 1
            agree += int(a.argmax() == b.argmax())
    return worst, agree, decided


@pytest.mark.parametrize("name", ALL)
def test_fp32_mode_matches_reference(name):
    net, pos, n, g = load_case(name)
    nw = network.Network(net, "precision=fp32,max_batch=%d" % n)
    out = nw.evaluate(pos["masks"][:n], pos["values"][:n])
    nw.close()
    _assert_fp32_logits(out["policy"], g["policy"])
    for k in ("q", "d", "m"):
        _assert_fp32_scalar(out[k], g[k])
    worst, agree, decided = _softmax_err_and_argmax(out["policy"], g["policy"], pos, n)
    assert agree == decided


@pytest.mark.parametrize("tc", [True, False])
@pytest.mark.parametrize("name", ALL)
def test_fp16_mode_within_tolerance(name, tc):
    net, pos, n, g = load_case(name)
    nw = network.Network(net, "precision=fp16,max_batch=%d,tensor_cores=%d" % (n, int(tc)))
    out = nw.evaluate(pos["masks"][:n], pos["values"][:n])
    assert nw.device_status() == 0
    nw.close()
    worst, agree, decided = _softmax_err_and_argmax(out["policy"], g["policy"], pos, n)
    assert worst <= HALF_ATOL
    assert agree == decided
    assert np.abs(out["q"] - g["q"]).max() <= HALF_ATOL
    assert np.abs(out["d"] - g["d"]).max() <= HALF_ATOL
    assert np.all(np.abs(out["m"] - g["m"]) <= HALF_ATOL * np.maximum(1.0, np.abs(g["m"])))


# bf16 storage keeps 8 significant bits in the residual stream (fp16: 11).  The policy softmax stays within the 2e-3 of
# the 16-bit contract on these networks; q, d and m do not (measured up to 5e-3) and are held to 1e-2.
BF16_VALUE_ATOL = 1e-2


@pytest.mark.parametrize("name", ["cfg3_mini", "cfg4_mini", "cfg4_2layer", "cfg2_mini"])
def test_bf16_mode_runs_close(name):
    net, pos, n, g = load_case(name)
    nw = network.Network(net, "precision=bf16,max_batch=%d" % n)
    out = nw.evaluate(pos["masks"][:n], pos["values"][:n])
    assert nw.device_status() == 0
    nw.close()
    worst, agree, decided = _softmax_err_and_argmax(out["policy"], g["policy"], pos, n)
    assert worst <= HALF_ATOL
    assert np.abs(out["q"] - g["q"]).max() <= BF16_VALUE_ATOL
    assert np.abs(out["d"] - g["d"]).max() <= BF16_VALUE_ATOL
    assert np.all(np.abs(out["m"] - g["m"]) <= BF16_VALUE_ATOL * np.maximum(1.0, np.abs(g["m"])))


def test_full_bt4_class_net_fp16_against_reference():
    """The full 15-layer BT4-class network on the recorded reference outputs."""
    net, pos, n, g = load_case("cfg4")
    nw = network.Network(net, "precision=fp16,max_batch=%d" % n)
    out = nw.evaluate(pos["masks"][:n], pos["values"][:n])
    assert nw.device_status() == 0
    nw.close()
    worst, agree, decided = _softmax_err_and_argmax(out["policy"], g["policy"], pos, n)
    assert worst <= HALF_ATOL and agree == decided
    assert np.abs(out["q"] - g["q"]).max() <= HALF_ATOL
    assert np.abs(out["d"] - g["d"]).max() <= HALF_ATOL
    assert np.all(np.abs(out["m"] - g["m"]) <= HALF_ATOL * np.maximum(1.0, np.abs(g["m"])))


def _compact_errors(out, g, pos, idx):
    """(worst legal-softmax error, argmax agreements, decided positions) against a compact golden; `idx` maps the
    evaluated rows to the golden's positions."""
    worst, agree, decided = 0.0, 0, 0
    got = legal_logits(out["policy"], {"legal": pos["legal"][idx], "n_legal": pos["n_legal"][idx]}, len(idx))
    for r, i in enumerate(idx):
        k = int(pos["n_legal"][i])
        if k == 0:
            continue
        a = oracle.legal_softmax(got[r][:k], np.arange(k))
        b = oracle.legal_softmax(g["legal_logits"][i][:k], np.arange(k))
        worst = max(worst, float(np.abs(a - b).max()))
        top = np.sort(b)[::-1]
        if len(top) < 2 or top[0] - top[1] > 2 * HALF_ATOL:
            decided += 1
            agree += int(a.argmax() == b.argmax())
    return worst, agree, decided


def _assert_half_against_compact(out, g, pos, idx):
    worst, agree, decided = _compact_errors(out, g, pos, idx)
    assert worst <= HALF_ATOL and agree == decided, (worst, agree, decided)
    assert np.abs(out["q"] - g["q"][idx]).max() <= HALF_ATOL
    assert np.abs(out["d"] - g["d"][idx]).max() <= HALF_ATOL
    assert np.all(np.abs(out["m"] - g["m"][idx]) <= HALF_ATOL * np.maximum(1.0, np.abs(g["m"][idx])))


@pytest.mark.parametrize("batch", [64, 256, 1024, 4096])
def test_fp16_at_the_measured_batch_sizes_against_reference(batch):
    """The BT4-class layer shapes (two layers) at the batch sizes the throughput is quoted on, against outputs of
    the reference's CPU backend for the same 1024 positions: the multi-wave tile schedule of the large products, the
    split last wave, the folded LayerNorm epilogues with their atomically accumulated row statistics and the merged
    QKV + smolgen-compression launch only exist at these sizes.  4096 = the 1024 positions four times in one batch."""
    net, pos, n, g = load_compact("cfg4_2layer_b1024")
    idx = np.arange(batch) % n
    nw = network.Network(net, "precision=fp16,max_batch=%d" % batch)
    for rep in range(3):  # plain launches, then the captured graph
        out = nw.evaluate(pos["masks"][idx], pos["values"][idx])
        assert nw.device_status() == 0
        _assert_half_against_compact(out, g, pos, idx)
    nw.close()


@pytest.mark.parametrize("precision", ["fp16", "bf16"])
@pytest.mark.parametrize("batch", [1, 2, 8, 9, 31, 65])
def test_bt4_class_layers_at_small_batches_against_reference(batch, precision):
    """The batches a search sends, in line: K cut over clusters and smolgen's LayerNorms inside the products that follow them
    (below 64 positions, the second one up to 4, then in a launch that adds in the same order), tiles of 64 rows and less."""
    net, pos, n, g = load_compact("cfg4_2layer_b1024")
    idx = np.arange(batch)
    nw = network.Network(net, "precision=%s,max_batch=%d,side_stream=0" % (precision, batch))
    for rep in range(3):
        out = nw.evaluate(pos["masks"][idx], pos["values"][idx])
        assert nw.device_status() == 0
        if precision == "fp16":
            _assert_half_against_compact(out, g, pos, idx)
        else:  # bf16 keeps 8 bits of mantissa where fp16 keeps 11
            worst, _, _ = _compact_errors(out, g, pos, idx)
            assert worst <= 8 * HALF_ATOL
            assert np.abs(out["q"] - g["q"][idx]).max() <= 8 * HALF_ATOL
    nw.close()


@pytest.mark.parametrize("name", ["cfg4_2layer", "cfg1", "cfg2_mini", "cfg3_mini_polenc"])
def test_fp32_results_do_not_depend_on_the_batch(name):
    """The verification mode has one summation order at every batch size: a position alone and among others, bit for bit."""
    net = mknet.make_net(name)
    _, pos, n, g = load_compact("cfg4_2layer_b1024")
    masks, values = np.array(pos["masks"][:300]), np.array(pos["values"][:300])
    nw = network.Network(net, "precision=fp32,max_batch=300")
    whole = nw.evaluate(masks, values)
    for batch in (1, 5, 9, 40, 64, 100):
        out = nw.evaluate(masks[:batch], values[:batch])
        for k in ("policy", "q", "d", "m"):
            np.testing.assert_array_equal(out[k], whole[k][:batch])
    nw.close()


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
def test_convolutions_whose_rows_are_no_16_byte_pieces(precision):
    """30 filters: the FMA kernel's convolution stages rows element by element."""
    from lc0_b200 import netproto
    net = netproto.parse_net(netproto.encode("Net", mknet.make_net("cfg1_mini", filters=30)))
    _, pos, n, g = load_case("cfg1_mini")
    want = oracle.forward(*weights.flatten(net), pos["masks"][:5], pos["values"][:5])
    nw = network.Network(net, "precision=%s,max_batch=8" % precision)
    out = nw.evaluate(pos["masks"][:5], pos["values"][:5])
    nw.close()
    if precision == "fp32":
        _assert_fp32_logits(out["policy"], want["policy"])
        _assert_fp32_scalar(out["q"], want["q"])
    else:  # storage rounding through five convolutions and two dense layers, each adding its share of a row's norm
        assert np.abs(out["policy"] - want["policy"]).max() <= 8 * 2.0 ** -11 * np.abs(want["policy"]).max()
        assert np.abs(out["q"] - want["q"]).max() <= HALF_ATOL


@pytest.mark.parametrize("filters,se", [(32, 4), (64, 6), (128, 32), (256, 32), (256, 64), (96, 8)])
def test_squeeze_excitation_after_the_convolution(filters, se):
    """Everything in shared memory; hidden units that are no whole 16-byte pieces; the skip input too large to stage; the matrices
    too large; channels that do not divide the threads.  Same bounds as the configurations' own fp32 results."""
    from lc0_b200 import netproto
    net = netproto.parse_net(netproto.encode("Net", mknet.make_net("cfg1_mini", blocks=2, filters=filters, se=se)))
    _, pos, n, g = load_case("cfg1_mini")
    want = oracle.forward(*weights.flatten(net), pos["masks"][:3], pos["values"][:3])
    nw = network.Network(net, "precision=fp32,max_batch=3")
    out = nw.evaluate(pos["masks"][:3], pos["values"][:3])
    assert nw.device_status() == 0
    nw.close()
    _assert_fp32_logits(out["policy"], want["policy"])
    _assert_fp32_scalar(out["q"], want["q"])


def test_squeeze_excitation_of_512_filters_on_both_sides_of_a_round():
    """Up to 148 boards with the matrices in shared memory, beyond them without: the same bits."""
    net = mknet.make_net("cfg2", blocks=2, filters=512, se=12)
    _, pos, n, g = load_compact("cfg4_2layer_b1024")
    masks, values = np.array(pos["masks"][:160]), np.array(pos["values"][:160])
    nw = network.Network(net, "precision=fp16,max_batch=160")
    whole = nw.evaluate(masks, values)
    for batch in (148, 149):
        out = nw.evaluate(masks[:batch], values[:batch])
        for k in ("policy", "q", "d", "m"):
            np.testing.assert_array_equal(out[k], whole[k][:batch])
    assert nw.device_status() == 0
    nw.close()


def _mini(kind, width):
    if kind == "attention":  # heads of depth `width`
        return mknet.make_net("cfg3_mini", emb=256, heads=256 // width, layers=8)
    return mknet.make_net("cfg1_mini", blocks=4, filters=width, se=32 if kind == "se" else 6)


@pytest.mark.parametrize("kind,widths", [("se", (128, 64)), ("se_odd", (512, 256)), ("attention", (128, 64))])
def test_networks_of_different_widths_on_different_threads(kind, widths):
    """Kernels whose shared memory depends on the layer: a network launched on one thread must not lower the limit that another
    thread's launch of the same kernel needs."""
    _, pos, n, g = load_case("cfg1_mini")
    masks, values = pos["masks"][:2], pos["values"][:2]
    nets = [network.Network(_mini(kind, w), "precision=fp32,max_batch=2,graph_capture=0") for w in widths for _ in range(2)]
    want = [nw.evaluate(masks, values) for nw in nets]
    errors = []

    def work(nw, ref):
        try:
            for _ in range(300):
                out = nw.evaluate(masks, values)
                if not np.array_equal(out["policy"], ref["policy"]):
                    raise AssertionError("another result")
        except Exception as e:  # noqa: BLE001 - reported by the test
            errors.append(e)

    threads = [threading.Thread(target=work, args=a) for a in zip(nets, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for nw in nets:
        nw.close()
    assert not errors, errors[0]


@pytest.mark.parametrize("precision", ["fp16", "bf16"])
@pytest.mark.parametrize("side", [0, 1])
def test_results_do_not_depend_on_the_batch_from_64_positions_on(precision, side):
    """The line that Net draws (kCutPositions): 64 positions are on the same side of it as larger batches, with smolgen's
    small products in line and on the second stream."""
    net = mknet.make_net("cfg4_2layer", layers=6)
    _, pos, n, g = load_compact("cfg4_2layer_b1024")
    nw = network.Network(net, "precision=%s,max_batch=300,side_stream=%d" % (precision, side))
    whole = nw.evaluate(pos["masks"][:300], pos["values"][:300])
    # bit for bit: the atomics that add up a row's statistics add 32 fp32 sums in double, which is exact in any order
    for batch in (64, 65, 100, 200):
        out = nw.evaluate(pos["masks"][:batch], pos["values"][:batch])
        for k in ("policy", "q", "d", "m"):
            np.testing.assert_array_equal(out[k], whole[k][:batch])
    nw.close()


@pytest.mark.parametrize("filters", [128, 192, 256])
@pytest.mark.parametrize("batch", [1, 5, 295, 297, 600, 1189, 2368])
def test_tower_with_several_row_blocks_per_cta(filters, batch):
    """One block of boards per CTA or pair, two, three, up to eight at a time and a ragged last group: the bits of one launch per
    convolution."""
    net = mknet.make_net("cfg2", blocks=3, filters=filters)
    _, pos, n, g = load_compact("cfg4_2layer_b1024")
    idx = np.arange(batch) % 1000
    masks, values = np.array(pos["masks"])[idx], np.array(pos["values"])[idx]
    outs = []
    for tower in (1, 0):
        nw = network.Network(net, "precision=fp16,max_batch=%d,tower=%d" % (batch, tower))
        outs.append(nw.evaluate(masks, values))
        assert nw.device_status() == 0
        nw.close()
    for k in ("policy", "q", "d", "m"):
        np.testing.assert_array_equal(outs[0][k], outs[1][k])


@pytest.mark.parametrize("filters,batches", [
    (128, {1: 1, 5: 1, 295: 1, 297: 1, 600: 1, 1189: 1, 1480: 1, 2368: 1, 2369: 0}),
    (192, {1: 1, 5: 1, 295: 1, 297: 1, 600: 1, 1189: 1, 1480: 1, 1776: 1, 1777: 1, 2073: 0, 2368: 1, 2369: 0}),
    (256, {1: 1, 5: 1, 295: 1, 297: 1, 600: 1, 888: 1, 889: 0, 1000: 1, 1184: 1, 1185: 0, 1400: 0, 1480: 1, 1481: 0, 1776: 0, 2368: 0})])
def test_tower_runs_where_it_is_ahead(filters, batches):
    """Wide towers come in rounds of four boards per pair of CTAs: a last round with too few of them goes to one launch per
    convolution, and so does what is more than eight blocks per CTA or pair.  The launches counted, the bits the same."""
    net = mknet.make_net("cfg2", blocks=2, filters=filters)
    _, pos, n, g = load_compact("cfg4_2layer_b1024")
    idx = np.arange(max(batches)) % 1000
    masks, values = np.array(pos["masks"])[idx], np.array(pos["values"])[idx]
    nets = [network.Network(net, "precision=fp16,max_batch=%d,tower=%d" % (max(batches), tower)) for tower in (1, 0)]
    if nets[0].info.sm_count != 148:
        pytest.skip("sizes of a GPU with 148 SMs")
    for batch, one_launch in batches.items():
        outs, launches = [], []
        for nw in nets:
            before = nw.launch_count()
            outs.append(nw.evaluate(masks[:batch], values[:batch]))
            launches.append(nw.launch_count() - before)
            assert nw.device_status() == 0
        assert launches[1] - launches[0] == (4 if one_launch else 0), (batch, launches)
        for k in ("policy", "q", "d", "m"):
            np.testing.assert_array_equal(outs[0][k], outs[1][k])
    for nw in nets:
        nw.close()


@pytest.mark.parametrize("precision", ["fp16", "bf16"])
@pytest.mark.parametrize("name", ["cfg4_2layer", "cfg3", "cfg2_mini", "cfg4_mini"])
def test_results_do_not_depend_on_the_batch_below_64_positions(name, precision):
    """Bit for bit: K ranges are cut by plans that are the same for every such batch, and smolgen's second LayerNorm adds in one
    order inside its product (few positions) and in its own launch (more)."""
    net = mknet.make_net(name, **({"layers": 6} if name == "cfg4_2layer" else {}))
    _, pos, n, g = load_compact("cfg4_2layer_b1024")
    nw = network.Network(net, "precision=%s,max_batch=63" % precision)
    whole = nw.evaluate(pos["masks"][:63], pos["values"][:63])
    for batch in (1, 2, 3, 5, 6, 8, 9, 17, 31, 32, 48):
        out = nw.evaluate(pos["masks"][:batch], pos["values"][:batch])
        for k in ("policy", "q", "d", "m"):
            np.testing.assert_array_equal(out[k], whole[k][:batch])
    nw.close()


@pytest.mark.parametrize("batch", [64, 1024])
def test_fp32_at_the_measured_batch_sizes_against_reference(batch):
    net, pos, n, g = load_compact("cfg4_2layer_b1024")
    idx = np.arange(batch)
    nw = network.Network(net, "precision=fp32,max_batch=%d" % batch)
    out = nw.evaluate(pos["masks"][idx], pos["values"][idx])
    nw.close()
    got = legal_logits(out["policy"], pos, batch)
    want = g["legal_logits"][:batch]
    rms = np.sqrt((want ** 2).sum(-1, keepdims=True) / np.maximum(1, pos["n_legal"][:batch])[:, None])
    assert np.all(np.abs(got - want) <= FP32_REL * np.maximum(np.abs(want), rms) + FP32_FLOOR)
    for k in ("q", "d", "m"):
        _assert_fp32_scalar(out[k], g[k][:batch])


@pytest.mark.parametrize("name", ["cfg4_b128", "cfg5_b128"])
def test_full_bt4_class_net_fp16_at_batch_128(name):
    """All 15 layers on 128 recorded positions: the uniform playout set and the opening / middlegame mix."""
    net, pos, n, g = load_compact(name)
    idx = np.arange(n)
    nw = network.Network(net, "precision=fp16,max_batch=%d" % n)
    out = nw.evaluate(pos["masks"][:n], pos["values"][:n])
    assert nw.device_status() == 0
    nw.close()
    _assert_half_against_compact(out, g, pos, idx)


@pytest.mark.parametrize("fold", [1, 0])
def test_outlier_channels_and_shifted_rows_fp16(fold):
    """A network with planted outlier channels (LayerNorm gains / offsets 12..24 on single channels) and a common
    offset on the sub-layer biases, so that residual-stream rows have a mean far from zero: the folded LayerNorm
    (one-pass row statistics accumulated by the producing product) against the reference, and the explicit LayerNorm
    kernels beside it."""
    net, pos, n, g = load_case("cfg4_mini_outlier")
    nw = network.Network(net, "precision=fp16,max_batch=%d,fold_ln=%d" % (n, fold))
    out = nw.evaluate(pos["masks"][:n], pos["values"][:n])
    assert nw.device_status() == 0
    nw.close()
    worst, agree, decided = _softmax_err_and_argmax(out["policy"], g["policy"], pos, n)
    assert worst <= HALF_ATOL and agree == decided, (worst, agree, decided)
    assert np.abs(out["q"] - g["q"]).max() <= HALF_ATOL
    assert np.abs(out["d"] - g["d"]).max() <= HALF_ATOL
    assert np.all(np.abs(out["m"] - g["m"]) <= HALF_ATOL * np.maximum(1.0, np.abs(g["m"])))


@pytest.mark.parametrize("name,count", [("cfg2", 16), ("cfg2", 5), ("cfg1_mini", 31), ("cfg1", 16), ("cfg2", 256),
                                        ("cfg2", 333)])
def test_squeeze_excitation_in_the_convolution_epilogue(name, count):
    """The second convolution of a residual block with SE, skip and activation in its epilogue (one tile = two whole
    boards x all channels) against the reference, and the separate SE kernel beside it; an odd board count leaves the
    last tile half empty.  From about 150 positions on a 256-filter tower runs on the CTA-pair kernel (each CTA of a
    pair loads half of the filter rows): 256 and 333 positions cover it, with a partly filled last pair."""
    net, pos, n, g = load_case(name)
    k = min(count, n)  # positions the golden holds
    outs = []
    for fused in (1, 0):
        nw = network.Network(net, "precision=fp16,max_batch=%d,fused_se=%d" % (count, fused))
        out = nw.evaluate(pos["masks"][:count], pos["values"][:count])
        out = nw.evaluate(pos["masks"][:count], pos["values"][:count])
        assert nw.device_status() == 0
        if fused:
            launches = nw.launch_count()
        else:
            assert nw.launch_count() > launches  # the fused schedule really has fewer launches
        nw.close()
        worst, agree, decided = _softmax_err_and_argmax(out["policy"], g["policy"], pos, k)
        assert worst <= HALF_ATOL and agree == decided, (fused, worst)
        assert np.abs(out["q"][:k] - g["q"][:k]).max() <= HALF_ATOL
        outs.append(out)
    assert np.abs(outs[0]["policy"] - outs[1]["policy"]).max() <= 2e-2 * max(1.0, np.abs(outs[1]["policy"]).max())
    assert np.abs(outs[0]["q"] - outs[1]["q"]).max() <= HALF_ATOL


@pytest.mark.parametrize("name,count", [("cfg2", 16), ("cfg2", 5), ("cfg1_mini", 31), ("cfg1", 16), ("cfg1", 401), ("cfg2", 149),
                                        ("cfg2", 256), ("cfg2", 333)])
def test_squeeze_excitation_fused_with_and_without_the_tower(name, count):
    """The unit in the epilogues of the tower kernels, in that of one launch per convolution (from about 150 positions on 256 filters
    run on the CTA-pair kernel) and in its own kernel, against the reference and one another; the launches say which of them ran."""
    net, pos, n, g = load_case(name)
    k = min(count, n)  # positions the golden holds
    reps = (count + n - 1) // n
    masks = np.concatenate([pos["masks"][:n]] * reps)[:count]
    values = np.concatenate([pos["values"][:n]] * reps)[:count]
    outs, launches = [], []
    for fused, tower in ((1, 0), (1, 1), (0, 0)):
        nw = network.Network(net, "precision=fp16,max_batch=%d,fused_se=%d,tower=%d" % (count, fused, tower))
        out = nw.evaluate(masks, values)
        assert nw.device_status() == 0
        launches.append(nw.launch_count())
        nw.close()
        worst, agree, decided = _softmax_err_and_argmax(out["policy"], g["policy"], pos, k)
        assert worst <= HALF_ATOL and agree == decided, (fused, tower, worst)
        assert np.abs(out["q"][:k] - g["q"][:k]).max() <= HALF_ATOL
        outs.append(out)
    # 32 filters have no tower kernel
    assert launches[2] > launches[0] and (launches[0] > launches[1] or name == "cfg1_mini")
    for out in outs[:2]:
        assert np.abs(out["policy"] - outs[2]["policy"]).max() <= 2e-2 * max(1.0, np.abs(outs[2]["policy"]).max())
        assert np.abs(out["q"] - outs[2]["q"]).max() <= HALF_ATOL


@pytest.mark.parametrize("name,count", [("cfg1", 16), ("cfg1", 5), ("cfg1", 64), ("cfg1", 401), ("cfg1_mini", 31),
                                        ("cfg2", 16), ("cfg2", 149)])
def test_tower_kernel_matches_per_layer_launches(name, count):
    """The input convolution and all residual blocks in one launch (a CTA walks the layers for its two boards, waiting
    only for its own stores) against one launch per convolution and against the reference; five evaluations each so
    that the replayed graph is covered; odd counts leave the last CTA one board, 401 positions give CTAs two and three
    row blocks."""
    net, pos, n, g = load_case(name)
    k = min(count, n)  # positions the golden holds
    reps = (count + n - 1) // n
    masks = np.concatenate([pos["masks"][:n]] * reps)[:count]
    values = np.concatenate([pos["values"][:n]] * reps)[:count]
    outs = []
    for tower in (1, 0):
        nw = network.Network(net, "precision=fp16,max_batch=%d,tower=%d" % (count, tower))
        for rep in range(5):
            out = nw.evaluate(masks, values)
            assert nw.device_status() == 0
        if tower:
            launches = nw.launch_count()
        else:
            # the tower schedule really has fewer launches (the mini net's 32 filters and the 256 filters of cfg2 do
            # not qualify: same schedule)
            assert nw.launch_count() > launches or name != "cfg1"
        nw.close()
        worst, agree, decided = _softmax_err_and_argmax(out["policy"], g["policy"], pos, k)
        assert worst <= HALF_ATOL and agree == decided, (tower, worst)
        assert np.abs(out["q"][:k] - g["q"][:k]).max() <= HALF_ATOL
        outs.append(out)
    # the same kernels' arithmetic in another order of launches: equal up to the rounding of the 16-bit stores
    assert np.abs(outs[0]["policy"] - outs[1]["policy"]).max() <= 1e-3 * max(1.0, np.abs(outs[1]["policy"]).max())
    assert np.abs(outs[0]["q"] - outs[1]["q"]).max() <= 1e-3


@pytest.mark.parametrize("name,count", [("cfg2", 16), ("cfg2_mini", 7), ("cfg1", 16), ("cfg1_mini", 32)])
def test_winograd_path_within_tolerance(name, count):
    """The optional Winograd F(4x4, 3x3) form of the residual tower (input transform, 36 stacked tensor-core products,
    output transform with SE / skip / activation) against the reference in fp16: about twice the error of the direct
    convolution, still inside the 16-bit contract on these networks."""
    net, pos, n, g = load_case(name)
    nw = network.Network(net, "precision=fp16,max_batch=%d,winograd=1" % count)
    for rep in range(3):  # plain launches, then the captured graph
        out = nw.evaluate(pos["masks"][:count], pos["values"][:count])
    assert nw.device_status() == 0
    nw.close()
    worst, agree, decided = _softmax_err_and_argmax(out["policy"], g["policy"], pos, count)
    assert worst <= HALF_ATOL and agree == decided, (worst, agree, decided)
    assert np.abs(out["q"] - g["q"][:count]).max() <= HALF_ATOL
    assert np.abs(out["d"] - g["d"][:count]).max() <= HALF_ATOL
    assert np.all(np.abs(out["m"] - g["m"][:count]) <= HALF_ATOL * np.maximum(1.0, np.abs(g["m"][:count])))


def test_kernel_timeout_is_reported_by_the_evaluation_call():
    """A status word set the way a kernel whose bounded wait gave up sets it makes the evaluation that finds it fail
    with B200_ERR_TIMEOUT (nothing on the GPU is disturbed: the word is written from the host), the word is cleared,
    and the next evaluation succeeds."""
    net, pos, n, g = load_case("cfg4_mini")
    nw = network.Network(net, "precision=fp16,max_batch=32,slots=2")
    want = nw.evaluate(pos["masks"][:n], pos["values"][:n])
    for attempt in range(2):  # plain launches first, the captured graph the second time
        nw.inject_device_status(103)
        failures = 0
        for slot in range(2):  # one failure per slot, whichever slot a call draws
            c = nw.new_computation()
            c.add_inputs(pos["masks"][:n], pos["values"][:n])
            try:
                c.compute_blocking()
            except _lib.B200Error as e:
                assert e.code == _lib.ERR_TIMEOUT and "103" in str(e)
                failures += 1
            c.close()
        assert failures >= 1
        nw.inject_device_status(0)
        got = nw.evaluate(pos["masks"][:n], pos["values"][:n])
        np.testing.assert_array_equal(got["policy"], want["policy"])
    assert nw.device_status() == 0
    nw.close()


def test_unsupported_topologies_are_refused_at_load():
    """An attention body on top of a residual tower and smolgen widths the LayerNorm kernels cannot take fail in the
    factory, not at the first evaluation."""
    from lc0_b200 import netproto
    tower = netproto.parse_net(netproto.encode("Net", mknet.make_net("cfg1_mini")))
    body = netproto.parse_net(netproto.encode("Net", mknet.make_net("cfg3_mini")))
    mixed = dict(body)
    mixed["weights"] = dict(body["weights"], input=tower["weights"]["input"], residual=tower["weights"]["residual"])
    with pytest.raises(_lib.B200Error, match="residual tower") as e:
        network.Network(mixed, "precision=fp16,max_batch=8")
    assert e.value.code == _lib.ERR_UNSUPPORTED
    odd = mknet.make_net("cfg4_mini", smolgen=dict(hc=8, hidden=36, gen=32, act=mknet.NF.ACTIVATION_SWISH))
    with pytest.raises(_lib.B200Error, match="smolgen widths") as e:
        network.Network(netproto.parse_net(netproto.encode("Net", odd)), "precision=fp16,max_batch=8")
    assert e.value.code == _lib.ERR_UNSUPPORTED


def test_computation_api_and_batch_shapes():
    """AddInput one by one, odd batch sizes, and independence of a sample from its batch neighbours."""
    net, pos, n, g = load_case("cfg4_mini")
    nw = network.Network(net, "precision=fp32,max_batch=40")
    ref = nw.evaluate(pos["masks"][:n], pos["values"][:n])
    for count in (1, 2, 3, 7, 31):
        c = nw.new_computation()
        for i in range(count):
            c.add_input(pos["masks"][i], pos["values"][i])
        assert c.get_batch_size() == count
        c.compute_blocking()
        for i in range(count):
            np.testing.assert_allclose(c.policy(i), ref["policy"][i], atol=2e-6)
            assert abs(c.get_q_val(i) - ref["q"][i]) < 2e-6
            assert abs(c.get_d_val(i) - ref["d"][i]) < 2e-6
            assert abs(c.get_m_val(i) - ref["m"][i]) < 2e-6
            assert c.get_p_val(i, 5) == c.policy(i)[5]
        c.close()
    empty = nw.new_computation()
    empty.compute_blocking()
    assert empty.get_batch_size() == 0
    c = nw.new_computation()
    c.add_inputs(pos["masks"][:32], pos["values"][:32])
    with pytest.raises(_lib.B200Error, match="max_batch"):
        c.add_inputs(pos["masks"][:32], pos["values"][:32])
    nw.close()


def test_mlh_option_and_head_errors():
    net, pos, n, g = load_case("cfg3_mini")
    nw = network.Network(net, "precision=fp32,max_batch=8,mlh=false")
    out = nw.evaluate(pos["masks"][:4], pos["values"][:4])
    assert np.all(out["m"] == 0) and nw.get_capabilities()["moves_left"] == 0
    nw.close()
    with pytest.raises(weights.WeightsError):
        network.Network(net, "policy_head=optimistic")
    with pytest.raises(_lib.B200Error, match="Invalid GPU Id"):
        network.Network(net, "gpu=99")


def test_large_batch_consistency():
    """Batch 1024 in fp16 equals the same positions evaluated in chunks (tile tails, many CTAs per GEMM)."""
    net, pos, n, g = load_case("cfg4_mini")
    nw = network.Network(net, "precision=fp16,max_batch=1024")
    masks, values = pos["masks"], pos["values"]
    big = nw.evaluate(masks, values)
    small = nw.evaluate(masks[:100], values[:100])
    assert nw.device_status() == 0
    nw.close()
    np.testing.assert_allclose(big["policy"][:100], small["policy"], atol=1e-6)
    np.testing.assert_allclose(big["q"][:100], small["q"], atol=1e-6)


def test_graph_replay_matches_plain_launches():
    """The captured CUDA graph (third and later calls of a shape) gives the same numbers as plain launches."""
    net, pos, n, g = load_case("cfg4_mini")
    plain = network.Network(net, "precision=fp16,max_batch=32,graph_capture=0")
    want = plain.evaluate(pos["masks"][:n], pos["values"][:n])
    plain.close()
    nw = network.Network(net, "precision=fp16,max_batch=32")
    for i in range(4):  # plain, capture + replay, replay, replay
        got = nw.evaluate(pos["masks"][:n], pos["values"][:n])
        np.testing.assert_array_equal(got["policy"], want["policy"])
        np.testing.assert_array_equal(got["q"], want["q"])
    # a different batch size gets its own graph
    for i in range(3):
        other = nw.evaluate(pos["masks"][:5], pos["values"][:5])
        np.testing.assert_allclose(other["policy"], want["policy"][:5], atol=HALF_ATOL)
    count = nw.launch_count()
    nw.evaluate(pos["masks"][:n], pos["values"][:n])
    assert nw.launch_count() > count  # replays are still counted as kernel launches
    assert nw.device_status() == 0
    nw.close()


def test_computation_may_outlive_its_network():
    """A garbage-collected host may destroy the network before its computations: results stay readable."""
    net, pos, n, g = load_case("cfg3_mini")
    nw = network.Network(net, "precision=fp32,max_batch=8")
    comps = []
    for i in range(3):
        c = nw.new_computation()
        c.add_inputs(pos["masks"][:4], pos["values"][:4])
        c.compute_blocking()
        comps.append(c)
    want = comps[0].policy(2)
    nw.close()
    for c in comps:
        np.testing.assert_array_equal(c.policy(2), want)
        assert abs(c.get_q_val(1) - g["q"][1]) < 1e-5
        c.close()


def test_concurrent_computations_on_two_slots():
    """Two host threads drive their own computations at the same time (lc0 runs several search threads)."""
    import threading
    net, pos, n, g = load_case("cfg4_mini")
    nw = network.Network(net, "precision=fp16,max_batch=32,slots=2")
    masks, values = np.array(pos["masks"]), np.array(pos["values"])  # the lazy .npz reader is not thread-safe
    want = nw.evaluate(masks[:n], values[:n])
    errors = []

    def worker(offset):
        try:
            for it in range(12):
                count = 5 + (it + offset) % 20
                c = nw.new_computation()
                c.add_inputs(masks[:count], values[:count])
                c.compute_blocking()
                got = np.stack([c.policy(i) for i in range(count)])
                if np.abs(got - want["policy"][:count]).max() > HALF_ATOL:
                    errors.append(("mismatch", offset, it))
                c.close()
        except Exception as e:  # pragma: no cover
            errors.append(e)

    threads = [threading.Thread(target=worker, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert nw.device_status() == 0
    nw.close()


def test_merged_qkv_and_smolgen_compression_launch_matches_separate_launches():
    """Q, K, V and the smolgen compression computed by one launch of the CTA-pair kernel (second output, narrow last
    tile) against the same network with the compression as a product of its own."""
    net = mknet.make_net("cfg4_2layer")
    rng = np.random.default_rng(5)
    n = 64
    masks = rng.integers(0, 2 ** 63, size=(n, 112), dtype=np.int64).astype(np.uint64) & rng.integers(
        0, 2 ** 63, size=(n, 112), dtype=np.int64).astype(np.uint64)
    values = np.ones((n, 112), np.float32)
    outs = []
    for flag in ("1", "0"):
        nw = network.Network(net, "precision=fp16,max_batch=%d,merge_compress=%s,side_stream=0" % (n, flag))
        outs.append(nw.evaluate(masks, values))
        assert nw.device_status() == 0
        nw.close()
    scale = np.abs(outs[1]["policy"]).max()
    assert np.abs(outs[0]["policy"] - outs[1]["policy"]).max() <= 2e-3 * scale
    assert np.abs(outs[0]["q"] - outs[1]["q"]).max() <= 2e-3


@pytest.mark.parametrize("batch", [40, 256, 1024])
def test_side_stream_schedule_matches_in_line_schedule(batch):
    """smolgen's small dense layers on a second stream beside the QKV product (confined to fewer SMs) against the same
    launches in line on one stream, and against the reference; three evaluations each so that the captured graph, with
    its fork and join, is replayed too."""
    net, pos, n, g = load_compact("cfg4_2layer_b1024")
    idx = np.arange(batch)
    outs = []
    for side in (1, 0):
        nw = network.Network(net, "precision=fp16,max_batch=%d,side_stream=%d" % (batch, side))
        for rep in range(3):
            out = nw.evaluate(pos["masks"][idx], pos["values"][idx])
            assert nw.device_status() == 0
        nw.close()
        _assert_half_against_compact(out, g, pos, idx)
        outs.append(out)
    assert np.abs(outs[0]["policy"] - outs[1]["policy"]).max() <= 2e-3 * max(1.0, np.abs(outs[1]["policy"]).max())
    assert np.abs(outs[0]["q"] - outs[1]["q"]).max() <= 1e-3


@pytest.mark.parametrize("name,batch", [("cfg4_2layer_b1024", 40), ("cfg4_2layer_b1024", 256), ("cfg2", 16),
                                        ("cfg3_mini_polenc", 16)])
def test_dependent_launches_match_ordinary_launches(name, batch):
    """Products, attention and LayerNorms launched as programmatic dependents (prologue under the tail of the kernel
    before, griddepcontrol.wait before the first global access) against ordinary launches of the same schedule; five
    evaluations each, so that the replayed graph is covered, and two slots used in turn."""
    net, pos, n, g = load_compact(name) if name.startswith("cfg4_2layer") else load_case(name)
    batch = min(batch, n)
    idx = np.arange(batch)
    outs = []
    for dep in (1, 0):
        nw = network.Network(net, "precision=fp16,max_batch=%d,slots=2,dependent_launch=%d" % (batch, dep))
        for rep in range(5):
            out = nw.evaluate(pos["masks"][idx], pos["values"][idx])
            assert nw.device_status() == 0
        nw.close()
        outs.append(out)
    scale = max(1.0, np.abs(outs[1]["policy"]).max())
    assert np.abs(outs[0]["policy"] - outs[1]["policy"]).max() <= 1e-3 * scale
    assert np.abs(outs[0]["q"] - outs[1]["q"]).max() <= 1e-3
    assert np.abs(outs[0]["m"] - outs[1]["m"]).max() <= 1e-3 * max(1.0, np.abs(outs[1]["m"]).max())


@pytest.mark.parametrize("precision", ["fp16", "bf16"])
@pytest.mark.parametrize("graphs", [0, 1])
@pytest.mark.parametrize("dm", [100, 101])
def test_single_positions_with_a_policy_width_off_the_tensor_cores(dm, graphs, precision):
    """A policy d_model that is no multiple of 8 takes the FMA kernel for Q K^T, whose keys the launch just before writes:
    they may not be requested ahead of it, and at one position nothing but the caller can tell them from a weight.
    Different positions in consecutive calls, dependent launches against ordinary ones and against the oracle."""
    from lc0_b200 import netproto
    net = netproto.parse_net(netproto.encode("Net", mknet.make_net("cfg4_mini", pol_dmodel=dm)))
    _, pos, n, g = load_case("cfg4_mini")
    want = oracle.forward(*weights.flatten(net), pos["masks"][:6], pos["values"][:6])
    rt = 2.0 ** -10 if precision == "fp16" else 2.0 ** -7  # of activations that pass through some ten roundings
    outs = []
    for dep in (1, 0):
        nw = network.Network(net, "precision=%s,max_batch=1,slots=1,graph_capture=%d,dependent_launch=%d" % (precision, graphs, dep))
        out = []
        for rep in range(4):
            for i in range(6):
                out.append(nw.evaluate(pos["masks"][i:i + 1], pos["values"][i:i + 1])["policy"][0])
        assert nw.device_status() == 0
        nw.close()
        outs.append(np.array(out))
    # row statistics are summed by atomics: the two schedules may differ by a rounding of the storage type here and there
    assert np.abs(outs[0] - outs[1]).max() <= rt * max(1.0, np.abs(outs[1]).max())
    ref = np.tile(want["policy"], (4, 1))
    assert np.abs(outs[0] - ref).max() <= 16 * rt * max(1.0, np.abs(ref).max())


def test_split_last_wave_matches_whole_tiles():
    """Products whose last wave of 256x256 tiles fills at most half of the CTA pairs compute that wave as half-width
    tiles (out-projection and FFN2 here, both with residual input and row statistics): same results as whole tiles."""
    net = mknet.make_net("cfg4_2layer")
    rng = np.random.default_rng(17)
    n = 96  # 96 tiles per 1024-wide product on 74 pairs: 22 tiles in the last wave
    masks = rng.integers(0, 2 ** 63, size=(n, 112), dtype=np.int64).astype(np.uint64) & rng.integers(
        0, 2 ** 63, size=(n, 112), dtype=np.int64).astype(np.uint64)
    values = np.ones((n, 112), np.float32)
    outs = []
    for flag in ("1", "0"):
        nw = network.Network(net, "precision=fp16,max_batch=%d,split_last_wave=%s" % (n, flag))
        outs.append(nw.evaluate(masks, values))
        assert nw.device_status() == 0
        nw.close()
    # the same MMAs on the same operands, in a different order over the CTA pairs: identical up to the atomics'
    # summation order in the row statistics
    scale = np.abs(outs[1]["policy"]).max()
    assert np.abs(outs[0]["policy"] - outs[1]["policy"]).max() <= 1e-3 * scale
    assert np.abs(outs[0]["q"] - outs[1]["q"]).max() <= 1e-3
