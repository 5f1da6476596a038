"""The allocation-free feature-transformer forward, collected last on purpose.

`b200_op_ft_forward_noalloc` exists for callers that cannot allocate device memory at call
time: a thread that evaluates positions on a GPU another thread is training on (a cudaMalloc
or cudaFree there would stall the trainer's streams), or a process that gave away all its
device memory up front.  It must return exactly what `b200_op_ft_forward` returns (both run
the same kernels in slot order, so the comparison is bit for bit), also on a second call that
finds the first call's leftovers in the shared scratch, and it must refuse batches beyond its
fixed scratch.  Only calls that group their positions use that scratch; few positions are gathered
without it."""
import dataclasses

import numpy as np
import pytest

from tests.test_gpu_ops import CASES, op_inputs, run_op

pytestmark = pytest.mark.gpu


# where x starts: aligned, these calls gather their few positions as they are; else they group them in the scratch
BOTH_WAYS = pytest.mark.parametrize("x_at", [0, 1], ids=["gathered", "grouped"])


@BOTH_WAYS
def test_noalloc_matches_allocating_entry_point_twice(oracle32, x_at):
    name, desc, game = CASES[0]
    # two calls in a row with different sizes and data: the second one reuses the scratch
    for n, seed in ((3000, 71), (1234, 72)):
        stm, nstm, w, table, x_ref = op_inputs(oracle32, desc, game, n, seed)
        rc_a, x_a, u_a = run_op("b200_op_ft_forward", desc, table, w["l0b"], stm, nstm, n, x_at)
        rc_b, x_b, u_b = run_op("b200_op_ft_forward_noalloc", desc, table, w["l0b"], stm, nstm, n, x_at)
        assert rc_a == 0 and rc_b == 0
        assert np.array_equal(x_b, x_a) and np.array_equal(u_b, u_a)
        assert np.array_equal(x_b, x_ref)


@BOTH_WAYS
def test_noalloc_other_activation_after_pairwise(oracle32, x_at):
    name, desc, game = CASES[1]
    stm, nstm, w, table, x_ref = op_inputs(oracle32, desc, game, 500, 73)
    rc, x, _ = run_op("b200_op_ft_forward_noalloc", desc, table, w["l0b"], stm, nstm, 500, x_at)
    assert rc == 0 and np.array_equal(x, x_ref)


@pytest.mark.parametrize("ft_out", [128, 256], ids=["gathered", "grouped"])
def test_noalloc_refuses_more_than_its_scratch_holds(oracle32, ft_out):
    from bullet_b200 import _lib

    name, desc, game = CASES[1]
    desc = dataclasses.replace(desc, ft_out=ft_out)
    n = 16384 + 1
    stm, nstm, w, table, x_ref = op_inputs(oracle32, desc, game, n, 74)
    rc, _, _ = run_op("b200_op_ft_forward_noalloc", desc, table, w["l0b"], stm, nstm, n)
    assert rc == -1 and b"16384" in _lib.load().b200_last_error()
    rc, x, _ = run_op("b200_op_ft_forward_noalloc", desc, table, w["l0b"], stm[:16384], nstm[:16384], 16384)
    assert rc == 0 and np.array_equal(x, x_ref[:16384])


@pytest.mark.parametrize("ft_out", [64, 256], ids=["gathered", "grouped"])
def test_noalloc_wide_index_lists_and_their_smaller_limit(oracle32, ft_out):
    """More than 32 index slots per position (ataxx: 49) take twice the list space, so the fixed
    scratch holds half as many positions: 8192 run bit-exactly, 8193 are refused."""
    from bullet_b200 import _lib

    name, desc, game = CASES[2]
    desc = dataclasses.replace(desc, ft_out=ft_out)
    assert desc.nnz == 49
    n = 8192
    stm, nstm, w, table, x_ref = op_inputs(oracle32, desc, game, n + 1, 75)
    rc, x, _ = run_op("b200_op_ft_forward_noalloc", desc, table, w["l0b"], stm[:n], nstm[:n], n)
    assert rc == 0 and np.array_equal(x, x_ref[:n])
    rc, _, _ = run_op("b200_op_ft_forward_noalloc", desc, table, w["l0b"], stm, nstm, n + 1)
    assert rc == -1 and b"8192" in _lib.load().b200_last_error()
    rc, x, _ = run_op("b200_op_ft_forward", desc, table, w["l0b"], stm, nstm, n + 1)   # the allocating entry takes it
    assert rc == 0 and np.array_equal(x, x_ref)


FIRST_CALL = """
import ctypes, sys
import numpy as np, torch
from bullet_b200 import _lib
n, rows, H = 300, 96, 64
table, bias = torch.randn((4 * rows, H), device="cuda"), torch.randn(H, device="cuda")
index = torch.randint(0, rows, (2, n, 20), device="cuda").to(torch.int16)
x = torch.zeros(n * 2 * H + 1, device="cuda")[int(sys.argv[1]):]
op = _lib.CFtOp(4 * rows, 20, H, 1, 0, rows, n, table.data_ptr(), bias.data_ptr(), index[0].data_ptr(), index[1].data_ptr(), x.data_ptr(), None)
lib = _lib.load()
torch.cuda.synchronize()
with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU, torch.profiler.ProfilerActivity.CUDA]) as trace:
    rc = lib.b200_op_ft_forward_noalloc(0, None, ctypes.byref(op))
    torch.cuda.synchronize()
assert rc == 0
print(" ".join(sorted({e.name for e in trace.events() if e.name.startswith("cu")})))
"""


@BOTH_WAYS
def test_the_first_call_of_a_process_makes_no_allocating_call(x_at):
    """A trace of the runtime calls of a process's first operator call holds its launches, and nothing that allocates."""
    import os
    import subprocess
    import sys

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    done = subprocess.run([sys.executable, "-c", FIRST_CALL, str(x_at)], cwd=root, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr
    calls = done.stdout.split()
    if not any("Launch" in c for c in calls):
        pytest.skip("this machine lets no process trace its runtime calls")
    assert not [c for c in calls if any(word in c for word in ("Alloc", "Malloc", "Free", "Register"))], calls


@BOTH_WAYS
@pytest.mark.parametrize("entry", ["b200_op_ft_forward", "b200_op_ft_forward_noalloc"])
def test_reports_of_calls_that_follow_each_other_or_run_together(oracle32, entry, x_at):
    """A feature outside its row block is reported by the call that met it and by no other, whichever came before; from more
    threads at once than there are status words as well (the allocation-free calls one after the other, as they must be)."""
    from concurrent.futures import ThreadPoolExecutor

    name, desc, game = CASES[0]
    n = 200
    stm, nstm, w, table, x_ref = op_inputs(oracle32, desc, game, n, 76)
    bad = stm.copy()
    bad[n - 1, :2] = [5, 800]

    def call(wrong):
        rc, x, _ = run_op(entry, desc, table, w["l0b"], bad if wrong else stm, nstm, n, x_at)
        return rc == (-4 if wrong else 0) and (wrong or np.array_equal(x, x_ref))

    assert all(call(wrong) for wrong in (True, False, True, True, False, False))
    if entry == "b200_op_ft_forward":
        with ThreadPoolExecutor(80) as pool:
            assert all(pool.map(call, [k % 3 == 0 for k in range(240)]))
