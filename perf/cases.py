"""The work this backend is there for, as cases that can be timed and compared.

A case names a network configuration of `lc0_b200.mknet.CONFIGS`, a precision, a batch size and the way in:

  eval      Network.evaluate: host arrays in, host arrays out (tools, analysis, Python harnesses)
  search    NetworkComputation with game histories and legal moves, compact policy: what lc0's search sends through the
            `b200-native` backend (positions encoded and legal-move softmax done on the device)
  device    Network.enqueue_device: inputs and outputs in device memory, batches queued behind one another
  rescore   packed training records in device memory -> planes -> Network.enqueue_device

A program creates its network once and evaluates with it for as long as it runs, so networks are made at their first use
and kept; every state brings its own inputs and output buffers.
"""
import math

import numpy as np
import torch

from lc0_b200 import _lib, mknet, network

MAX_BATCH = {"cfg1": 4096, "cfg2": 2048, "cfg3": 4096, "cfg4": 4096}

_networks = {}


def _network(config, precision):
    key = (config, precision)
    if key not in _networks:
        # fp32 is the verification mode, run on small batches; two slots as the lc0 plug-in creates a network
        max_batch = 512 if precision == "fp32" else MAX_BATCH[config]
        _networks[key] = network.Network(mknet.make_net(config),
                                         dict(precision=precision, max_batch=max_batch, slots=2))
    return _networks[key]


def listed():
    return [
        # BT4-class network, the headline configuration.  One position: analysis of a single position, raw-policy play,
        # the root of every search; latency is all there is.
        dict(name="bt4_root", net="cfg4", precision="fp16", path="eval", batch=1),
        # A search's small minibatch: shallow trees, short time controls, several games at once.
        dict(name="bt4_search_24", net="cfg4", precision="fp16", path="search", batch=24),
        # The batch size the headline latency is quoted at.
        dict(name="bt4_eval_256", net="cfg4", precision="fp16", path="eval", batch=256),
        # The headline throughput: 1024 positions, device resident.
        dict(name="bt4_device_1024", net="cfg4", precision="fp16", path="device", batch=1024),
        # The top of the batch sweep.
        dict(name="bt4_device_4096", net="cfg4", precision="fp16", path="device", batch=4096),
        # The other 16-bit type, at a ragged size.
        dict(name="bt4_eval_333_bf16", net="cfg4", precision="bf16", path="eval", batch=333),
        # Verification mode: checking a network or another backend against fp32.
        dict(name="bt4_eval_16_fp32", net="cfg4", precision="fp32", path="eval", batch=16),
        # Small attention network, batch of its configuration.
        dict(name="attn256_device_512", net="cfg3", precision="fp16", path="device", batch=512),
        # ... and in a search, at an odd size.
        dict(name="attn256_search_37", net="cfg3", precision="fp16", path="search", batch=37),
        # Residual network 20 x 256 at the batch of its configuration.
        dict(name="res20x256_eval_256", net="cfg2", precision="fp16", path="eval", batch=256),
        # Residual network 10 x 128 at the batch and precision of its configuration.
        dict(name="res10x128_eval_64_fp32", net="cfg1", precision="fp32", path="eval", batch=64),
        # Rescoring of training chunks with a small network.
        dict(name="res10x128_rescore_1500", net="cfg1", precision="fp16", path="rescore", batch=1500),
    ]


# (network, precision, path, smallest and largest batch, weight): the ranges the listed cases stand for
_RANGES = [
    ("cfg4", "fp16", "eval", 1, 1024, 3), ("cfg4", "fp16", "search", 1, 256, 3), ("cfg4", "fp16", "device", 64, 4096, 2),
    ("cfg4", "bf16", "eval", 1, 1024, 1), ("cfg4", "fp32", "eval", 1, 64, 1),
    ("cfg3", "fp16", "search", 1, 256, 2), ("cfg3", "fp16", "device", 16, 4096, 2),
    ("cfg2", "fp16", "eval", 1, 1024, 2), ("cfg2", "fp16", "device", 16, 2048, 1),
    ("cfg1", "fp32", "eval", 1, 512, 1), ("cfg1", "fp16", "search", 1, 256, 1), ("cfg1", "fp16", "rescore", 64, 4096, 1),
]


def draw(rng):
    net, precision, path, lo, hi, _ = rng.choices(_RANGES, weights=[r[5] for r in _RANGES])[0]
    batch = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return dict(net=net, precision=precision, path=path, batch=min(hi, max(lo, batch)))


# ---- positions --------------------------------------------------------------------------------------------------
def _boards(rng, n):
    """n positions with eight boards of history each: bitboards [n][8][12] (ours P N B R Q K, theirs P N B R Q K; newest
    board first, all seen by the side to move now).  6 to 32 pieces on distinct squares, one piece moved per ply."""
    squares = np.argsort(rng.random((n, 64)), axis=1)
    count = rng.integers(6, 33, n)
    kind = rng.choice(5, (n, 32), p=[0.5, 0.14, 0.14, 0.14, 0.08]) + 6 * rng.integers(0, 2, (n, 32))
    kind[:, 0], kind[:, 1] = 5, 11
    where = squares[:, :32].copy()
    alive = np.arange(32)[None, :] < count[:, None]
    out = np.zeros((n, 8, 12), np.uint64)
    rows = np.arange(n)
    for ply in range(8):
        bits = np.where(alive, np.uint64(1) << where.astype(np.uint64), np.uint64(0))
        for k in range(12):
            out[:, ply, k] = np.bitwise_or.reduce(np.where(kind == k, bits, np.uint64(0)), axis=1)
        where[rows, rng.integers(0, count)] = squares[:, 32 + ply]  # the piece that stood elsewhere a ply earlier
    return out


def _planes(rng, n, fmt):
    """The 112 (mask, value) pairs of n positions as lc0's encoder fills them (formats 1 and 2)."""
    full = ~np.uint64(0)
    b = _boards(rng, n)
    masks = np.zeros((n, 112), np.uint64)
    values = np.ones((n, 112), np.float32)
    plies = np.where(rng.random(n) < 0.9, 8, rng.integers(1, 9, n))
    repeated = rng.random((n, 8)) < 0.03
    for i in range(8):
        on = (plies > i)[:, None]
        masks[:, 13 * i:13 * i + 12] = np.where(on, b[:, i], np.uint64(0))
        masks[:, 13 * i + 12] = np.where(on[:, 0] & repeated[:, i], full, np.uint64(0))
    castling = rng.random((n, 4)) < 0.3
    if fmt == 1:
        masks[:, 104:108] = np.where(castling, full, np.uint64(0))
    else:
        for i, (q, t) in enumerate(((0, 56), (7, 63))):
            masks[:, 104 + i] = (np.where(castling[:, 2 * i], np.uint64(1) << np.uint64(q), np.uint64(0)) |
                                 np.where(castling[:, 2 * i + 1], np.uint64(1) << np.uint64(t), np.uint64(0)))
    masks[:, 108] = np.where(rng.random(n) < 0.5, full, np.uint64(0))
    masks[:, 109] = full
    values[:, 109] = rng.integers(0, 60, n)
    masks[:, 111] = full
    return masks, values


def _histories(rng, n):
    """Eight b200_board records per position, oldest first, each from the point of view of its side to move."""
    b = _boards(rng, n)
    rec = np.zeros((n, 8), _lib.BOARD_DTYPE)
    black = rng.integers(0, 2, n)
    rule50 = rng.integers(8, 60, n)
    castling = np.where(rng.random(n) < 0.5, 0, rng.integers(0, 16, n))
    for ply in range(8):
        ours, theirs = b[:, ply, :6], b[:, ply, 6:]
        if ply & 1:
            ours, theirs = theirs.byteswap(), ours.byteswap()
        r = rec[:, 7 - ply]
        r["ours"], r["theirs"] = np.bitwise_or.reduce(ours, 1), np.bitwise_or.reduce(theirs, 1)
        for k, name in enumerate(("pawns", "knights", "bishops", "rooks", "queens", "kings")):
            r[name] = ours[:, k] | theirs[:, k]
        r["castling"] = castling if not ply & 1 else ((castling & 3) << 2) | (castling >> 2)
        r["rook_files"] = (0, 7, 0, 7)
        r["flags"] = black ^ (ply & 1)
        r["rule50"] = rule50 - ply
    return rec.reshape(-1), np.arange(0, 8 * n + 1, 8, dtype=np.int32), np.zeros(n, np.uint8)


def _moves(rng, n):
    """Policy indices of about thirty legal moves per position, padded to 256."""
    ids = np.zeros((n, 256), np.uint16)
    count = np.clip(np.rint(rng.normal(31, 11, n)), 1, 90).astype(np.int32)
    for i in range(n):
        ids[i, :count[i]] = rng.choice(1858, count[i], replace=False)
    return ids, count


def _records(rng, n):
    """n packed V6 training records of input format 1 (8356 bytes each)."""
    masks, values = _planes(rng, n, 1)
    rec = np.zeros((n, 8356), np.uint8)
    rec[:, 0:8] = np.array([6, 1], "<u4").view(np.uint8)
    rec[:, 8:7440] = rng.random((n, 1858), np.float32).view(np.uint8)
    bits = np.unpackbits(np.ascontiguousarray(masks[:, :104]).view(np.uint8).reshape(n, 832, 1), axis=2)[:, :, ::-1]
    rec[:, 7440:8272] = np.packbits(bits, axis=2)[:, :, 0]  # a record's planes are mirrored left to right
    rec[:, 8272:8276] = masks[:, 104:108] != 0
    rec[:, 8276] = masks[:, 108] != 0
    rec[:, 8277] = values[:, 109].astype(np.uint8)
    return rec


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    n, fmt = case["batch"], mknet.CONFIGS[case["net"]]["input"]
    s = dict(path=case["path"], n=n, net=_network(case["net"], case["precision"]))
    if case["path"] == "search":
        s["history"], s["moves"] = _histories(rng, n), _moves(rng, n)
        return s
    if case["path"] == "rescore":
        s["records"] = torch.from_numpy(_records(rng, n)).cuda()
        s["masks"] = torch.empty(n, 112, dtype=torch.int64, device="cuda")
        s["values"] = torch.empty(n, 112, dtype=torch.float32, device="cuda")
    else:
        s["masks"], s["values"] = _planes(rng, n, fmt)
        if case["path"] == "device":
            s["masks"], s["values"] = torch.from_numpy(s["masks"].view(np.int64)).cuda(), torch.from_numpy(s["values"]).cuda()
    if case["path"] != "eval":
        s["policy"] = torch.empty(n, 1858, dtype=torch.float32, device="cuda")
        s["qdm"] = torch.zeros(n, 3, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    return s


def run(s):
    net, n = s["net"], s["n"]
    if s["path"] == "eval":
        return net.evaluate(s["masks"], s["values"])
    if s["path"] == "search":
        comp = net.new_computation()
        comp.add_positions(*s["history"], *s["moves"])
        comp.set_policy_options(1.0, compact=True)
        comp.compute_blocking()
        probs = np.zeros((n, 256), np.float32)
        for i in range(n):
            p = comp.legal_policy(i)
            probs[i, :p.size] = p
        qdm = np.array([(comp.get_q_val(i), comp.get_d_val(i), comp.get_m_val(i)) for i in range(n)], np.float32)
        comp.close()
        return probs, qdm
    if s["path"] == "rescore":
        _lib.check(_lib.load().b200_op_planes_from_training_data(
            s["records"].data_ptr(), n, s["records"].shape[1], 0, s["masks"].data_ptr(), s["values"].data_ptr(), None,
            net.stream()))
    net.enqueue_device(s["masks"].data_ptr(), s["values"].data_ptr(), n, s["policy"].data_ptr(), s["qdm"].data_ptr())
    return s["policy"], s["qdm"]


# ---- work and tolerance -------------------------------------------------------------------------------------------
def _counts(net):
    """(weights, multiply-adds per position) of the network's matrices; convolutions counted directly."""
    c = mknet.CONFIGS[net]
    dense = []  # (rows per position, outputs, inputs)
    if c["kind"] == "resnet":
        f = c["filters"]
        dense += [(64, f, 112 * 9)] + [(64, f, 9 * f)] * (2 * c["blocks"]) + [(1, c["se"], 3 * f)] * c["blocks"]
        if c["policy"] == "classical":
            dense += [(64, c["policy_planes"], f), (1, 1858, 64 * c["policy_planes"])]
        else:
            dense += [(64, f, 9 * f), (64, c["policy_planes"], 9 * f)]
        e = f
    else:
        e, d, h = c["emb"], c["dff"], c["heads"]
        if c["pe_dense"]:
            dense += [(1, 64 * c["dpe"], 768), (64, e, 112 + c["dpe"]), (64, 2 * c["emb_dff"], e)]
        else:
            dense += [(64, e, 176)]
        dense += [(64, 4 * e + 2 * d, e)] * c["layers"]
        if c["smolgen"]:
            g = c["smolgen"]
            dense += [(64, g["hc"], e), (1, g["hidden"], 64 * g["hc"]), (1, h * g["gen"], g["hidden"])] * c["layers"]
            dense += [(h * c["layers"], 4096, g["gen"])]
        dense += [(64, c["pol_emb"], e), (64, 2 * c["pol_dmodel"], c["pol_emb"])]
    dense += [(64, c["value_planes"], e), (1, c["value_hidden"], 64 * c["value_planes"])]
    if c["mlh"]:
        dense += [(64, c["mlh_planes"], e), (1, c["mlh_hidden"], 64 * c["mlh_planes"])]
    weights = sum(o * i for _, o, i in dense)
    macs = sum(r * o * i for r, o, i in dense)
    if c["kind"] != "resnet":
        macs += c["layers"] * 2 * 64 * 64 * e + 64 * 64 * c["pol_dmodel"]
    return weights, macs


def work(case):
    n = case["batch"]
    weights, macs = _counts(case["net"])
    size = 4 if case["precision"] == "fp32" else 2
    per_position = {"eval": 112 * 12 + 1861 * 4, "device": 112 * 12 + 1861 * 4, "rescore": 840 + 1861 * 4,
                    "search": 8 * 88 + 31 * 6 + 12}[case["path"]]
    return {"bytes": weights * size + n * per_position, "flops": 2 * macs * n}


def tolerance(case):
    # Four times the differences measured between this backend's schedules (folded or explicit LayerNorms, tensor cores or
    # FMA products, fused or separate squeeze-excitation), between 16-bit and fp32 and, in fp32, against the CPU
    # oracle.  Probabilities of legal moves differ less than logits in the attention networks, whose random weights leave
    # them close to uniform.
    if case["precision"] == "fp32":
        return {"rel": 1e-5, "max": 6e-5}
    if case["precision"] == "bf16":
        return {"rel": 3e-2, "max": 7e-1}
    if case["path"] == "search":
        return {"rel": 1e-2, "max": 3.3e-2} if case["net"] == "cfg1" else {"rel": 7e-4, "max": 5.5e-3}
    return {"rel": 1.2e-2, "max": 1e-1}
