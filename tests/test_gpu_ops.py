"""Operator-level GPU tests: the feature-transformer forward on caller-owned device memory,
called through the C ABI with torch tensors supplying the device pointers, against the oracle's
SparseMatmul + bias + activation composition (bit-exact, as the sums run in slot order)."""
import ctypes
import dataclasses

import numpy as np
import pytest

from bullet_b200 import synth
from bullet_b200.configs import ACT_CRELU, ACT_SCRELU, NetDesc

pytestmark = pytest.mark.gpu


def op_inputs(oracle32, desc, game, n, seed):
    """Host-side inputs and the oracle's expected x for `n` positions."""
    from tests.test_gpu_parity import oracle_ft_output, rich_weights

    rec = synth.records(game, n, seed=seed)
    stm, nstm, _, _ = oracle32.map_batch(game, rec, desc)
    w = rich_weights(desc)
    table = w["l0w"].copy()
    if desc.factoriser_rows:
        table = table + np.tile(w["l0f"], desc.n_inputs // desc.factoriser_rows)
    return stm, nstm, w, table, oracle_ft_output(oracle32, desc, w, stm, nstm)


def run_op(entry, desc, table, bias, stm, nstm, n, x_at=0):
    """Calls `entry` (a b200_op_ft_forward-style symbol) on torch-owned device buffers; returns (rc, x, u).  With x starting `x_at` floats
    into a buffer, where that is no multiple of four, the positions are grouped however few they are."""
    import torch

    from bullet_b200 import _lib
    from bullet_b200.net import pack_indices

    dev = torch.device("cuda", 0)
    t_table = torch.from_numpy(np.ascontiguousarray(table, dtype=np.float32)).to(dev)
    t_bias = torch.from_numpy(np.ascontiguousarray(bias, dtype=np.float32)).to(dev)
    t_stm = torch.from_numpy(pack_indices(stm).view(np.int16)).to(dev)
    t_nstm = torch.from_numpy(pack_indices(nstm).view(np.int16)).to(dev)
    d1 = desc.ft_out if desc.pairwise else 2 * desc.ft_out
    t_x = torch.full((n * d1 + x_at,), float("nan"), device=dev)[x_at:].view(n, d1)
    t_u = torch.full((n, 2, desc.ft_out), float("nan"), device=dev) if desc.pairwise else None
    op = _lib.CFtOp(desc.n_inputs, desc.nnz, desc.ft_out, desc.ft_act, int(desc.pairwise), desc.ft_block_rows, n,
                    t_table.data_ptr(), t_bias.data_ptr(), t_stm.data_ptr(), t_nstm.data_ptr(), t_x.data_ptr(),
                    t_u.data_ptr() if t_u is not None else None)
    torch.cuda.synchronize()
    rc = getattr(_lib.load(), entry)(0, None, ctypes.byref(op))
    torch.cuda.synchronize()
    return rc, t_x.cpu().numpy(), None if t_u is None else t_u.cpu().numpy()


CASES = [
    ("pairwise", NetDesc(n_inputs=12288, nnz=32, ft_out=128, ft_act=ACT_CRELU, pairwise=True, factoriser_rows=768,
                         n_out_buckets=8, dense_out=(16, 32, 1), dense_act=(2, 2, 0), ft_block_rows=768), "chess_buckets"),
    ("screlu", NetDesc(n_inputs=768, nnz=32, ft_out=128, ft_act=ACT_SCRELU, ft_block_rows=768), "chess768"),
    ("ataxx", NetDesc(n_inputs=147, nnz=49, ft_out=64, ft_act=ACT_CRELU, ft_block_rows=147), "ataxx147"),
]


@pytest.mark.parametrize("name,desc,game", CASES, ids=[c[0] for c in CASES])
def test_op_ft_forward_bit_exact(oracle32, name, desc, game):
    n = 777
    stm, nstm, w, table, x_ref = op_inputs(oracle32, desc, game, n, seed=61)
    rc, x, u = run_op("b200_op_ft_forward", desc, table, w["l0b"], stm, nstm, n)
    assert rc == 0
    assert np.array_equal(x, x_ref)
    if desc.pairwise:
        h = desc.ft_out // 2
        assert np.array_equal(u[:, 0, :h] * u[:, 0, h:], x[:, :h]) and np.array_equal(u[:, 1, :h] * u[:, 1, h:], x[:, h:])
        assert u.min() >= 0 and u.max() <= 1


def test_op_ft_forward_errors(oracle32):
    from bullet_b200 import _lib

    name, desc, game = CASES[0]
    n = 64
    stm, nstm, w, table, _ = op_inputs(oracle32, desc, game, n, seed=62)
    bad = stm.copy()
    bad[5, 1] = (bad[5, 0] + 768 * 5) % 12288        # a feature from another king bucket
    rc, _, _ = run_op("b200_op_ft_forward", desc, table, w["l0b"], bad, nstm, n)
    assert rc == -4 and b"row block" in _lib.load().b200_last_error()
    rc, _, _ = run_op("b200_op_ft_forward", dataclasses.replace(desc, ft_block_rows=0), table, w["l0b"], stm, nstm, n)
    assert rc == -5
    lib = _lib.load()
    assert lib.b200_op_ft_forward(0, None, None) == -1


@pytest.mark.parametrize("entry", ["b200_op_ft_forward", "b200_op_ft_forward_noalloc"])
@pytest.mark.parametrize("name,desc,game", CASES, ids=[c[0] for c in CASES])
@pytest.mark.parametrize("bias_at,x_at,u_at", [(1, 0, 0), (0, 2, 2), (3, 1, 1), (2, 0, 0)])
def test_op_ft_forward_on_arrays_that_start_on_any_float(oracle32, entry, name, desc, game, bias_at, x_at, u_at):
    """Bias and outputs of the caller may be slices of larger arrays: bit-exact, and nothing written around them."""
    import torch

    from bullet_b200 import _lib
    from bullet_b200.net import pack_indices

    n, dev = 321, torch.device("cuda", 0)
    stm, nstm, w, table, x_ref = op_inputs(oracle32, desc, game, n, seed=64)
    t_table = torch.from_numpy(np.ascontiguousarray(table, dtype=np.float32)).to(dev)
    lists = [torch.from_numpy(pack_indices(a).view(np.int16)).to(dev) for a in (stm, nstm)]

    def holder(count, at):
        return torch.full((count + 8,), 7.0, device=dev), at, count

    def inside(h):
        return h[0][h[1]:h[1] + h[2]]

    bias = holder(desc.ft_out, bias_at)
    inside(bias).copy_(torch.from_numpy(w["l0b"].astype(np.float32)))
    x = holder(x_ref.size, x_at)
    u = holder(n * 2 * desc.ft_out, u_at) if desc.pairwise else None
    op = _lib.CFtOp(desc.n_inputs, desc.nnz, desc.ft_out, desc.ft_act, int(desc.pairwise), desc.ft_block_rows, n, t_table.data_ptr(),
                    inside(bias).data_ptr(), lists[0].data_ptr(), lists[1].data_ptr(), inside(x).data_ptr(),
                    inside(u).data_ptr() if u else None)
    torch.cuda.synchronize()
    assert getattr(_lib.load(), entry)(0, None, ctypes.byref(op)) == 0
    torch.cuda.synchronize()
    assert np.array_equal(inside(x).cpu().numpy().reshape(x_ref.shape), x_ref)
    if u:
        half = inside(u).cpu().numpy().reshape(n, 2, 2, desc.ft_out // 2)
        assert np.array_equal((half[:, :, 0] * half[:, :, 1]).reshape(n, -1), x_ref)
    for h in (x, u) if u else (x,):
        assert (h[0][:h[1]] == 7.0).all() and (h[0][h[1] + h[2]:] == 7.0).all()


@pytest.mark.parametrize("past", [0, 1])
@pytest.mark.parametrize("name,desc,game", CASES, ids=[c[0] for c in CASES])
def test_op_ft_forward_on_either_side_of_the_gather(oracle32, name, desc, game, past):
    """The most positions that are gathered without grouping, and one more: bit-exact, and a feature outside its block is reported."""
    n = (576 << 20) // (8 * desc.nnz * desc.ft_out) + past
    stm, nstm, w, table, x_ref = op_inputs(oracle32, desc, game, n, seed=65)
    rc, x, _ = run_op("b200_op_ft_forward", desc, table, w["l0b"], stm, nstm, n)
    assert rc == 0
    assert np.array_equal(x, x_ref)
    if desc.n_inputs > desc.ft_block_rows:
        stm[n - 1, 1] = (stm[n - 1, 0] + desc.ft_block_rows) % desc.n_inputs
        rc, _, _ = run_op("b200_op_ft_forward", desc, table, w["l0b"], stm, nstm, n)
        assert rc == -4


TRACE = """
import ctypes, sys
import torch
from bullet_b200 import _lib
lib = _lib.load()
torch.zeros(1, device="cuda")
for blocks, ft_out, nnz, n in eval(sys.argv[1]):
    rows = 64
    table, bias = torch.zeros((blocks * rows, ft_out), device="cuda"), torch.zeros(ft_out, device="cuda")
    index = torch.zeros((2, n, nnz), device="cuda", dtype=torch.int16)
    x = torch.zeros(n * 2 * ft_out, device="cuda")
    op = _lib.CFtOp(blocks * rows, nnz, ft_out, 1, 0, rows, n, table.data_ptr(), bias.data_ptr(), index[0].data_ptr(), index[1].data_ptr(), x.data_ptr(), None)
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU, torch.profiler.ProfilerActivity.CUDA]) as trace:
        rc = lib.b200_op_ft_forward(0, None, ctypes.byref(op))
        torch.cuda.synchronize()
    assert rc == 0
    names = [e.name for e in trace.events()]
    print(" ".join(sorted({k for k in ("ft_forward_gather", "ft_forward_tiled", "Malloc", "cudaFree") if any(k in name for name in names)})))
"""


def traced(calls):
    """What each call of b200_op_ft_forward, (row blocks, columns, slots, positions), launches and asks of the allocator."""
    import os
    import subprocess
    import sys

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    done = subprocess.run([sys.executable, "-c", TRACE, repr(calls)], cwd=root, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr
    seen = [set(line.split()) for line in done.stdout.splitlines()]
    if not any(seen):
        pytest.skip("this machine lets no process trace its runtime calls")
    return seen


def test_lines_between_gathered_and_grouped_calls():
    """The last call that is gathered and one position more, for tables of a few tiles, of one for a part of the SMs, of one for each, and of many."""
    lines = [(1, 512, 64, 576 * 4), (1, 1024, 64, 896 * 2), (4, 2048, 64, 896), (5, 2048, 64, 1152), (16, 2048, 64, 1536)]
    seen = traced([(b, h, nnz, n + more) for b, h, nnz, n in lines for more in (0, 1)])
    for k in range(len(lines)):
        assert "ft_forward_gather" in seen[2 * k] and "ft_forward_tiled" in seen[2 * k + 1], lines[k]


def test_gathered_calls_take_no_scratch():
    """A call that groups nothing asks nothing of the allocator, so it runs where there is no room left; one that groups has its scratch from the pool."""
    gathered, grouped = traced([(4, 512, 20, 300), (1, 512, 64, 3000)])
    assert gathered == {"ft_forward_gather"}
    assert grouped == {"ft_forward_tiled", "Malloc", "cudaFree"}


LOADS = """
import dataclasses, sys
import torch

from tests.test_gpu_parity import make_net, rich_weights
from tests.test_gpu_sizes import draw_batch, net_of
torch.zeros(1, device="cuda")
blocks, rows, ft_out, dense, pairwise, factoriser = eval(sys.argv[1])
most = 4000
desc = dataclasses.replace(net_of(blocks, rows, ft_out, 12, 2, dense, pairwise=pairwise), max_batch=most, factoriser_rows=factoriser)
w = rich_weights(desc)
batches = [draw_batch(desc, n, seed=n) for n in (1, 150, most)]


def loaded(run):
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU, torch.profiler.ProfilerActivity.CUDA]) as trace:
        run()
        torch.cuda.synchronize()
    return [e.name for e in trace.events()].count("Lazy Function Loading")


def work():
    for mode in (0, 1, 2):
        net.set_option("ft_mode", mode)
        for wide in (0, 1):
            net.set_option("ft_bwd_wide", wide)
            for batch in batches:
                n = len(batch[0])
                net.upload(0, *batch)
                net.forward(0, n)
                net.step(0, 1e-3, 1.0 / n)
                net.loss()
                net.backward(0)
                net.update(1e-3, 1.0 / n)


first = []
def create():
    first.append(make_net(desc, 0, w))
created = loaded(create)
net = first[0]
print(created, loaded(work))
"""


@pytest.mark.parametrize("net,most", [
    ((4, 300, 128, (16, 32, 1), True, 300), 58), ((4, 300, 128, (1,), False, 0), 58), ((1, 147, 64, (8, 1), False, 0), 58), ((2, 147, 128, (1,), True, 0), 58)])
def test_networks_load_the_kernels_of_their_kind_when_they_are_made(net, most):
    """All of them, as a load later may wait for kernels that run, and not those of other kinds: the first form of the two tiled kernels for every kind
    made it 70 in a fresh process."""
    import os
    import subprocess
    import sys

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    done = subprocess.run([sys.executable, "-c", LOADS, repr(net)], cwd=root, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr
    created, later = map(int, done.stdout.split()[-2:])
    if not created:
        pytest.skip("this machine lets no process trace its runtime calls")
    assert later == 0 and created <= most, (created, later)
