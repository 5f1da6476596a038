"""The work that this framework is measured on: training steps, evaluation and the stand-alone operator.

A training pass is one turn of the documented training loop (`bench.py`'s end-to-end loop): enqueue the
step on the batch that is already in a slot, upload the next batch into the next slot while it runs, read the loss of
the step before.  An evaluation pass uploads a batch and reads the network's outputs.  An operator pass calls the
feature-transformer forward on device memory of the caller's own.

A case is a dict of plain values:
  kind       "train", "eval" or "op"
  net        which network family, see `_desc`
  hidden     feature-transformer width
  n          positions per pass
  source     train, eval: what is uploaded: "device" = raw 32-byte records prepared by kernels, "host" = raw records
             prepared on the host cores, "arrays" = the mapper's index arrays (what bullet's own loader hands over)
  optimiser  train: "adamw", "radam" or "ranger"
  scratch    op: "own" = the entry point allocates its scratch, "fixed" = the allocation-free entry point
"""
import ctypes
import math

import numpy as np
import torch

from bullet_b200 import _lib
from bullet_b200.configs import ACT_CRELU, ACT_NONE, ACT_SCRELU, NetDesc, RAdamParams, RangerParams
from bullet_b200.net import Net, featurise, pack_indices

GAME = {"simple": "chess768", "king": "chess_buckets", "pairwise": "chess_buckets", "ataxx": "ataxx147", "layers": "chess768",
        "plain": "chess768"}
ACTIVE = {"chess768": 17.0, "chess_buckets": 17.0, "ataxx147": 27.5}  # mean active features per perspective


def listed():
    return [
        # the reference's first example (768 -> 128 SCReLU -> 1) at its batch size: a step so short that launches count
        dict(name="train-simple-128", kind="train", net="simple", hidden=128, n=16384, source="device", optimiser="adamw"),
        # king buckets, factoriser and output buckets with one wide hidden layer, fed by bullet's own mapper
        dict(name="train-king-1024", kind="train", net="king", hidden=1024, n=16384, source="arrays", optimiser="adamw"),
        # the ataxx example: few table rows, long index lists, records prepared on the host
        dict(name="train-ataxx-256", kind="train", net="ataxx", hidden=256, n=32768, source="host", optimiser="adamw"),
        # the multi-layer pairwise network at the reference's batch size, which is also one GPU's share of the batch
        # below when eight train together
        dict(name="train-pairwise-2048", kind="train", net="pairwise", hidden=2048, n=16384, source="device", optimiser="adamw"),
        # ... and at the headline's batch size: the largest step
        dict(name="train-pairwise-2048-large", kind="train", net="pairwise", hidden=2048, n=131072, source="device", optimiser="adamw"),
        # a narrower network of the same form, a ragged batch (the last one of an epoch) and the Ranger optimiser
        dict(name="train-pairwise-512-ragged", kind="train", net="pairwise", hidden=512, n=5003, source="device", optimiser="ranger"),
        # a table without the row-block promise and a width that is no multiple of 64: the kernels for any index set
        dict(name="train-plain-96", kind="train", net="plain", hidden=96, n=16384, source="arrays", optimiser="radam"),
        # one position evaluated: latency and nothing else
        dict(name="eval-one", kind="eval", net="pairwise", hidden=2048, n=1, source="arrays"),
        # a validation set scored batch by batch
        dict(name="eval-16384", kind="eval", net="pairwise", hidden=2048, n=16384, source="device"),
        # the operator beside somebody else's program: a small call that must not allocate, and a larger one
        dict(name="op-king-1024-fixed", kind="op", net="king", hidden=1024, n=2048, scratch="fixed"),
        dict(name="op-pairwise-2048", kind="op", net="pairwise", hidden=2048, n=10000, scratch="own"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "eval", "op"])
    net = rng.choice(["simple", "king", "pairwise", "ataxx"] + (["layers", "plain"] if kind != "op" else []))
    hidden = 64 * max(1, _log(rng, 64, 2048) // 64)
    if net == "pairwise":
        hidden = max(128, hidden)
    if net == "plain":
        hidden = 8 * max(1, _log(rng, 8, 512) // 8)
    case = dict(kind=kind, net=net, hidden=hidden)
    if kind == "train":
        case.update(n=_log(rng, 256, 65536), source=rng.choice(["device", "host", "arrays"]),
                    optimiser=rng.choice(["adamw", "adamw", "radam", "ranger"]))
    elif kind == "eval":
        case.update(n=_log(rng, 1, 32768), source=rng.choice(["device", "host", "arrays"]))
    else:
        fixed = rng.choice([True, False])
        most = (8192 if net == "ataxx" else 16384) if fixed else 32768
        case.update(n=_log(rng, 64, most), scratch="fixed" if fixed else "own")
    return case


def _desc(case):
    net, hidden, n = case["net"], case["hidden"], case["n"]
    if net == "simple":
        return NetDesc(n_inputs=768, nnz=32, ft_out=hidden, ft_act=ACT_SCRELU, ft_block_rows=768, max_batch=n)
    if net == "king":
        return NetDesc(n_inputs=12288, nnz=32, ft_out=hidden, ft_act=ACT_SCRELU, factoriser_rows=768, n_out_buckets=8,
                       ft_block_rows=768, max_batch=n)
    if net == "pairwise":
        return NetDesc(n_inputs=12288, nnz=32, ft_out=hidden, ft_act=ACT_CRELU, pairwise=True, factoriser_rows=768,
                       n_out_buckets=8, dense_out=(16, 32, 1), dense_act=(ACT_SCRELU, ACT_SCRELU, ACT_NONE),
                       ft_block_rows=768, max_batch=n)
    if net == "ataxx":
        return NetDesc(n_inputs=147, nnz=49, ft_out=hidden, ft_act=ACT_CRELU, ft_block_rows=147, max_batch=n)
    if net == "layers":
        return NetDesc(n_inputs=768, nnz=32, ft_out=hidden, ft_act=ACT_CRELU, n_out_buckets=4, dense_out=(8, 1),
                       dense_act=(ACT_CRELU, ACT_NONE), ft_block_rows=768, max_batch=n)
    if net == "plain":
        return NetDesc(n_inputs=768, nnz=32, ft_out=hidden, ft_act=ACT_SCRELU, ft_block_rows=0, max_batch=n)
    raise ValueError(net)


# ------------------------------------------------------------------------------------------------ inputs
# The distributions are those of bullet_b200/synth.py (see its docstring), drawn on the GPU.

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _tail(n, g):
    """Bytes 24-26 of a record: score (i16) and result."""
    score = torch.clamp(torch.round(torch.randn(n, generator=g, device="cuda") * 400.0), -3000, 3000)
    s = torch.sigmoid(score / 400.0)
    r = torch.rand(n, generator=g, device="cuda")
    result = torch.where(r < s * s, 2, torch.where(r < s * s + (1 - s) * (1 - s), 0, 1))
    return score.to(torch.int16), result.to(torch.uint8)


def _bitboard(mask):
    """[n, squares] truth values -> one 64-bit word per row."""
    weights = torch.ones(mask.shape[1], dtype=torch.int64, device="cuda") << torch.arange(mask.shape[1], device="cuda")
    return (mask.to(torch.int64) * weights).sum(1)


def _chess(n, g):
    k = torch.randint(2, 33, (n, 1), generator=g, device="cuda")
    order = torch.argsort(torch.rand((n, 64), generator=g, device="cuda"), dim=1)[:, :32]
    ptype = torch.randint(0, 5, (n, 32), generator=g, device="cuda")
    redraw = torch.randint(1, 5, (n, 32), generator=g, device="cuda")
    colour = torch.randint(0, 2, (n, 32), generator=g, device="cuda")
    rank = order // 8
    ptype = torch.where((ptype == 0) & ((rank == 0) | (rank == 7)), redraw, ptype)
    ptype[:, :2] = 5
    colour[:, 0], colour[:, 1] = 0, 1
    active = torch.arange(32, device="cuda")[None, :] < k
    board = torch.full((n, 65), -1, dtype=torch.int64, device="cuda")
    board.scatter_(1, torch.where(active, order, 64), (colour << 3) | ptype)
    board = board[:, :64]
    occupied = board >= 0
    # pieces in ascending square order, four bits each
    codes = torch.zeros((n, 33), dtype=torch.int64, device="cuda")
    place = torch.where(occupied, torch.cumsum(occupied, 1) - 1, 32)
    codes.scatter_(1, place, torch.where(occupied, board, 0))
    codes = codes[:, :32]
    rec = torch.zeros((n, 32), dtype=torch.uint8, device="cuda")
    rec[:, 0:8] = _bitboard(occupied).view(torch.uint8).view(n, 8)
    rec[:, 8:24] = (codes[:, 0::2] | (codes[:, 1::2] << 4)).to(torch.uint8)
    score, result = _tail(n, g)
    rec[:, 24:26] = score.view(torch.uint8).view(n, 2)
    rec[:, 26] = result
    rec[:, 27] = order[:, 0].to(torch.uint8)
    rec[:, 28] = (order[:, 1] ^ 56).to(torch.uint8)
    return rec.cpu().numpy()


def _ataxx(n, g):
    blocked_count = torch.randint(0, 9, (n, 1), generator=g, device="cuda")
    pairs = torch.argsort(torch.rand((n, 24), generator=g, device="cuda"), dim=1)[:, :4]
    use = torch.arange(4, device="cuda")[None, :] < blocked_count // 2
    blocked = torch.zeros((n, 50), dtype=torch.bool, device="cuda")
    blocked.scatter_(1, torch.where(use, pairs, 49), True)
    blocked.scatter_(1, torch.where(use, 48 - pairs, 49), True)
    blocked = blocked[:, :49].clone()
    blocked[:, 24] |= blocked_count[:, 0] % 2 == 1
    free = 49 - blocked.sum(1)
    stones = 2 + (torch.rand(n, generator=g, device="cuda") * (free - 1)).to(torch.int64)
    key = torch.where(blocked, 2.0, torch.rand((n, 49), generator=g, device="cuda"))
    taken = torch.argsort(torch.argsort(key, dim=1), dim=1) < stones[:, None]
    colour = torch.randint(0, 2, (n, 49), generator=g, device="cuda").bool()
    rec = torch.zeros((n, 32), dtype=torch.uint8, device="cuda")
    for i, plane in enumerate((taken & ~colour, taken & colour, blocked)):
        rec[:, 8 * i:8 * i + 8] = _bitboard(plane).view(torch.uint8).view(n, 8)
    score, result = _tail(n, g)
    rec[:, 24:26] = score.view(torch.uint8).view(n, 2)
    rec[:, 26] = result
    return rec.cpu().numpy()


def _records(game, n, g):
    return _ataxx(n, g) if game == "ataxx147" else _chess(n, g)


def _weights(desc, g):
    """name -> GPU tensor: uniform +-1/sqrt(fan-in) weights, small biases and factoriser (a net some way into training)."""
    out = {}
    for name, (rows, cols) in desc.tensor_shapes().items():
        if name.endswith("b") or name == "l0f":
            out[name] = 0.02 * torch.randn(rows * cols, generator=g, device="cuda")
        else:
            fan_in = cols if name != "l0w" else 32 if desc.n_inputs > 768 else desc.n_inputs
            out[name] = (2 * torch.rand(rows * cols, generator=g, device="cuda") - 1) / math.sqrt(fan_in)
    return out


class _Buffer:
    """One flat device buffer of a network; the tensor made of it keeps the network alive."""

    def __init__(self, net, kind):
        self.net = net
        ptr, count = net.flat_buffer(kind)
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f4", "data": (ptr, False), "version": 3, "strides": None}


_streams = {}


def _stream():
    """The program's compute stream, shared by all its networks."""
    device = torch.cuda.current_device()
    if device not in _streams:
        _streams[device] = torch.cuda.Stream()
    return _streams[device]


def _upload(state, slot, batch):
    net, source = state["net"], state["source"]
    if source == "arrays":
        net.upload(slot, *batch)
    else:
        net.upload_records(slot, state["game"], batch, on_device=source == "device")


def prepare(case, seed):
    g = _generator(seed)
    desc, game, n = _desc(case), GAME[case["net"]], case["n"]
    if case["kind"] == "op":
        stm, nstm, _, _ = featurise(game, _records(game, n, g), desc)
        w = _weights(desc, g)
        table = w["l0w"]
        if desc.factoriser_rows:
            table = table + w["l0f"].repeat(desc.n_inputs // desc.factoriser_rows)
        lists = [torch.from_numpy(pack_indices(a).view(np.int16)).cuda() for a in (stm, nstm)]
        x = torch.zeros((n, desc.dense_in0), device="cuda")
        u = torch.zeros((n, 2, desc.ft_out), device="cuda") if desc.pairwise else None
        op = _lib.CFtOp(desc.n_inputs, desc.nnz, desc.ft_out, desc.ft_act, int(desc.pairwise), desc.ft_block_rows, n,
                        table.data_ptr(), w["l0b"].data_ptr(), lists[0].data_ptr(), lists[1].data_ptr(), x.data_ptr(),
                        u.data_ptr() if u is not None else None)
        lib = _lib.load()
        entry = lib.b200_op_ft_forward_noalloc if case["scratch"] == "fixed" else lib.b200_op_ft_forward
        return {"kind": "op", "op": op, "entry": entry, "x": x, "u": u, "keep": (table, w["l0b"], lists)}
    net = Net(desc, device=torch.cuda.current_device(), stream=_stream().cuda_stream)
    for name, values in _weights(desc, g).items():
        net.set_tensor(name, values.cpu().numpy())
    state = {"kind": case["kind"], "net": net, "game": game, "n": n, "source": case["source"]}
    batches = [_records(game, n, g) for _ in range(2 if case["kind"] == "train" else 1)]
    if case["source"] == "arrays":
        batches = [featurise(game, r, desc) for r in batches]
    state["batches"] = batches
    if case["kind"] == "train":
        if case["optimiser"] != "adamw":
            net.set_optimiser_for_weight(None, RAdamParams() if case["optimiser"] == "radam" else RangerParams())
        kinds = {"weights": 0, "momentum": 1, "velocity": 2, "gradient": 3, **({"slow": 4} if case["optimiser"] == "ranger" else {})}
        state["flat"] = {name: torch.as_tensor(_Buffer(net, kind), device="cuda") for name, kind in kinds.items()}
        state["steps"] = 0
        _upload(state, 0, batches[0])
    return state


def run(state):
    if state["kind"] == "op":
        _lib.check(state["entry"](torch.cuda.current_device(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream),
                                  ctypes.byref(state["op"])))
        return {"x": state["x"]} if state["u"] is None else {"x": state["x"], "u": state["u"]}
    net = state["net"]
    if state["kind"] == "eval":
        _upload(state, 0, state["batches"][0])
        return net.forward(0, state["n"])
    step = state["steps"]
    net.step(step % 3, 1e-3, 1.0 / state["n"])
    _upload(state, (step + 1) % 3, state["batches"][(step + 1) % 2])
    loss = net.loss(steps_back=1) if step else 0.0
    state["steps"] = step + 1
    return {"loss": loss, **state["flat"]}


def work(case):
    """What a pass cannot do without.  Bytes: the positions in, the weights the pass needs in, and out what it makes:
    outputs, or (training) the gradient and the updated weights and moments.  Operations: one addition per active
    feature and column (twice with the gradient), the dense layers' multiply-adds, the update."""
    desc, n = _desc(case), case["n"]
    active = 2 * ACTIVE[GAME[case["net"]]]
    params = desc.n_params()
    touched = min(params, int(active * n) * desc.ft_out)  # few positions need few rows of the table
    add = active * n * desc.ft_out
    dense = sum(2.0 * n * desc.dense_in(i) * desc.dense_out[i] for i in range(desc.n_dense))
    if case["kind"] == "op":
        out = n * desc.dense_in0 + (2 * n * desc.ft_out if desc.pairwise else 0)
        table = min(desc.n_inputs, int(active * n)) * desc.ft_out
        return {"bytes": 4 * (out + table + desc.ft_out) + 4 * n * desc.nnz, "flops": add}
    position = 8 * desc.nnz + 8 if case["source"] == "arrays" else 32
    if case["kind"] == "eval":
        return {"bytes": position * n + 4 * touched + 4 * n, "flops": add + dense}
    return {"bytes": position * n + 4 * params * (3 + 4), "flops": 2 * add + 3 * dense + 12.0 * params}


def tolerance(case):
    if case["kind"] == "op":
        return "exact"  # rows are added in slot order: every output is defined to the last bit
    if case["kind"] == "eval":
        return {"rel": 1e-5}
    # 32-bit sums over the batch in any order.  One update divides a moment by the root of another, so an element whose
    # gradient nearly cancels may step anywhere within +-3.2 learning rates: single weights, not the whole.
    return {"rel": 2e-5, "max": 0.1}
