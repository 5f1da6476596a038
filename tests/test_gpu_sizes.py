"""The kernels' forms at the edges of their ranges, against the CPU oracle: row-block counts on either side of every way of
grouping, list lengths and holes, widths that leave a slab or a column group unfilled, dense layers of every row count with
one tile, one tile more, and batches on either side of the small-batch kernels.

Tolerances: the feature-transformer output is bit-exact (rows are added in slot order); outputs and gradients are sums in
another order than the oracle's, of fp32 products (the tensor pipe's operands are split so that a product keeps 2^-24): at most
K = 4096 terms whose rounding errors add like a random walk, sqrt(K) 2^-24 = 4e-6 of the largest term, taken as 2e-5 of the
largest entry, the bound of the other gradient tests."""
import numpy as np
import pytest

from bullet_b200.configs import ACT_CRELU, ACT_NONE, ACT_SCRELU, NetDesc

pytestmark = pytest.mark.gpu


def draw_batch(desc, n, seed):
    """Lists whose features lie in one row block per (position, perspective), with empty slots anywhere."""
    rng = np.random.default_rng(seed)
    rows = desc.ft_block_rows or desc.n_inputs
    lists = []
    for _ in range(2):
        block = rng.integers(0, (desc.n_inputs + rows - 1) // rows, n)
        local = np.argsort(rng.random((n, rows)), axis=1)[:, : desc.nnz]
        index = block[:, None] * rows + local
        index[(rng.random(index.shape) < 0.2) | (index >= desc.n_inputs)] = -1
        lists.append(index.astype(np.int32))
    return lists[0], lists[1], rng.integers(0, desc.n_out_buckets, n).astype(np.int32), rng.random(n).astype(np.float32)


def net_of(blocks, rows, ft_out, nnz, buckets, dense, act=ACT_CRELU, pairwise=False):
    return NetDesc(n_inputs=blocks * rows, nnz=nnz, ft_out=ft_out, ft_act=act, pairwise=pairwise, n_out_buckets=buckets,
                   dense_out=dense, dense_act=(ACT_SCRELU,) * (len(dense) - 1) + (ACT_NONE,), ft_block_rows=rows)


CASES = {
    # row blocks: counted up to 32 of them, sorted up to 256, by a kernel of its own beyond; lists of any length
    "blocks-32": (net_of(32, 64, 64, 20, 1, (1,)), 700),
    "blocks-33": (net_of(33, 64, 64, 20, 1, (1,)), 700),
    "blocks-256": (net_of(256, 40, 64, 9, 3, (1,)), 700),
    "blocks-257": (net_of(257, 40, 64, 9, 3, (1,)), 1300),
    "list-of-one": (net_of(4, 96, 64, 1, 2, (1,)), 500),
    "list-of-64": (net_of(2, 200, 64, 64, 2, (1,)), 500),
    # chunks of a length between the shortest and the longest, few enough that the last one's lists end close to the room
    "chunks-in-between": (net_of(1, 768, 128, 32, 4, (8, 1)), 313),
    "chunks-in-between-wide": (net_of(1, 147, 1920, 49, 1, (1,)), 1467),
    # widths: a part of one slab, a slab and a part, a pairwise half that is no slab
    "width-8": (net_of(1, 300, 8, 31, 1, (1,), ACT_SCRELU), 1500),
    "width-72": (net_of(3, 300, 72, 31, 1, (1,), ACT_SCRELU), 1500),
    "width-200-pairwise": (net_of(3, 300, 200, 32, 8, (16, 32, 1), pairwise=True), 1500),
    # dense layers: row counts, columns short of a group of 16, of a slice of 256 and of 512; one tile, one more, many
    "rows-4-columns-16": (net_of(1, 100, 8, 16, 1, (4, 1)), 1),
    "rows-4-columns-272": (net_of(1, 100, 136, 16, 2, (4, 8, 1)), 33),
    "rows-8-columns-528": (net_of(1, 100, 264, 16, 5, (8, 16, 1)), 31),
    "rows-16-columns-2048": (net_of(2, 100, 2048, 16, 8, (16, 32, 1), pairwise=True), 32),
    "rows-16-columns-1040": (net_of(2, 100, 520, 16, 3, (16, 32, 1)), 2100),
    "rows-32-columns-784": (net_of(2, 100, 392, 16, 3, (32, 32, 1)), 1100),
    "rows-32-last-layer": (net_of(1, 100, 64, 16, 64, (32, 1)), 900),
    "one-row-columns-4096": (net_of(1, 100, 2048, 16, 7, (1,), ACT_SCRELU), 37),
    "one-row-columns-16": (net_of(1, 100, 8, 16, 64, (1,)), 1000),
}


@pytest.mark.parametrize("case", CASES)
def test_kernel_forms_at_the_edges_of_their_ranges(oracle32, case):
    import dataclasses

    from tests.test_gpu_parity import make_net, oracle_ft_output, rich_weights

    desc, n = CASES[case]
    desc = dataclasses.replace(desc, max_batch=n)
    batch = draw_batch(desc, n, seed=len(case) + n)
    w = rich_weights(desc)
    x_ref = oracle_ft_output(oracle32, desc, w, *batch[:2])
    loss_ref, g_ref, out_ref = oracle32.net_grad(desc, w, *batch)
    net = make_net(desc, 0, w)
    if case == "chunks-in-between-wide":
        net.set_option("ft_bwd_products", 0)  # (what it is here for are the walk's lists)
    net.upload(0, *batch)
    out = net.forward(0, n)
    assert np.array_equal(net.activation(0, n * desc.dense_in0).reshape(n, -1), x_ref)
    assert np.abs(out - out_ref).max() <= 2e-5 * np.abs(out_ref).max()
    net.step(0, 0.0, 1.0 / n)  # a whole step that leaves the weights where they are
    assert np.array_equal(net.activation(0, n * desc.dense_in0).reshape(n, -1), x_ref)
    assert abs(net.loss() - loss_ref) <= 2e-5 * loss_ref
    g = net.tensors(kind=3)
    for k in g_ref:
        assert np.abs(g[k] - g_ref[k]).max() <= 2e-5 * np.abs(g_ref[k]).max(), k
    net.backward(0)  # the same in phases
    g = net.tensors(kind=3)
    for k in g_ref:
        assert np.abs(g[k] - g_ref[k]).max() <= 2e-5 * np.abs(g_ref[k]).max(), k
    net.close()


@pytest.mark.parametrize("case", [name for name, (desc, _) in CASES.items() if desc.ft_out % 64 == 0 or (desc.ft_out >= 32 and desc.n_inputs < 890)])
def test_tiled_forward_at_the_edges_of_its_ranges(oracle32, case):
    """The cases above by the tiled forward, where the library's choice for so few positions is the gather: asked for by name, or, for
    tables that promise no blocks of whole slabs, with more positions than the gather takes (the two of 900 rows that do not promise any
    have no tiled form).  Evaluations and steps; bounds as above."""
    import dataclasses

    from tests.test_gpu_parity import make_net, oracle_ft_output, rich_weights

    desc, n = CASES[case]
    promised = desc.ft_out % 64 == 0
    n = n if promised else max(n, 2049)
    desc = dataclasses.replace(desc, max_batch=n)
    batch = draw_batch(desc, n, seed=len(case) + n)
    w = rich_weights(desc)
    x_ref = oracle_ft_output(oracle32, desc, w, *batch[:2])
    loss_ref, g_ref, out_ref = oracle32.net_grad(desc, w, *batch)
    net = make_net(desc, 2 if promised else 0, w)
    net.upload(0, *batch)
    out = net.forward(0, n)
    assert net.stat("ft_forward") > 0
    assert np.array_equal(net.activation(0, n * desc.dense_in0).reshape(n, -1), x_ref)
    assert np.abs(out - out_ref).max() <= 2e-5 * np.abs(out_ref).max()
    net.step(0, 0.0, 1.0 / n)
    assert net.stat("ft_forward") > 0
    assert np.array_equal(net.activation(0, n * desc.dense_in0).reshape(n, -1), x_ref)
    assert abs(net.loss() - loss_ref) <= 2e-5 * loss_ref
    g = net.tensors(kind=3)
    for k in g_ref:
        assert np.abs(g[k] - g_ref[k]).max() <= 2e-5 * np.abs(g_ref[k]).max(), k
    net.close()


@pytest.mark.parametrize("ft_out,pairwise,act,buckets", [(72, False, ACT_SCRELU, 1), (96, False, ACT_CRELU, 3), (136, True, ACT_CRELU, 2)])
@pytest.mark.parametrize("mode", [0, 1])
def test_a_loss_gradient_that_is_not_finite_stays_in_its_rows(oracle32, ft_out, pairwise, act, buckets, mode):
    """One target is NaN: the rows that its position holds are lost, every other row's gradient is what the other positions
    give.  The widths leave a part of the last slab of 64 columns empty; nothing may be written past them.  Bounds as above."""
    import dataclasses

    from tests.test_gpu_parity import make_net, rich_weights

    n, bad = 40, 17
    desc = dataclasses.replace(net_of(1, 300, ft_out, 31, buckets, (1,), act, pairwise), max_batch=n)
    stm, nstm, bucket, target = draw_batch(desc, n, seed=ft_out)
    w = rich_weights(desc)
    rest = np.arange(n) != bad
    _, g_ref, _ = oracle32.net_grad(desc, w, stm[rest], nstm[rest], bucket[rest], target[rest])
    target[bad] = np.nan
    net = make_net(desc, mode, w)
    net.upload(0, stm, nstm, bucket, target)
    lost = np.zeros(desc.n_inputs, dtype=bool)
    for row in np.concatenate([stm[bad], nstm[bad]]):
        lost[max(row, 0)] |= row >= 0
    ref = g_ref["l0w"].reshape(desc.n_inputs, ft_out)
    for step in (lambda: net.backward(0), lambda: net.step(0, 0.0, 1.0 / n)):
        step()
        g = net.tensors(kind=3)
        got = g["l0w"].reshape(desc.n_inputs, ft_out)
        assert np.isnan(got[lost]).all()
        assert np.isnan(g["l0b"]).all()
        assert np.abs(got[~lost] - ref[~lost]).max() <= 2e-5 * np.abs(ref).max()
        first = net.tensor_range("l0w")[0]  # what lies behind the last row
        assert not np.isnan(net_flat(net, 3)[first + got.size:]).any()
    net.close()


@pytest.mark.parametrize("dense,pairwise", [((1,), False), ((8, 1), False), ((16, 32, 1), True)])
def test_products_in_parts_and_in_slots_that_change_hands(oracle32, dense, pairwise):
    """The product backward a run of row blocks at a time, in a slot that holds batches of other sizes cut for the walk and for products
    in turn.  Bounds as above."""
    import dataclasses

    from tests.test_gpu_parity import make_net, rich_weights

    most, n = 2900, 150
    desc = dataclasses.replace(net_of(8, 96, 128, 20, 2, dense, ACT_CRELU, pairwise), max_batch=most)
    w = rich_weights(desc)
    net = make_net(desc, 0, w)
    for count, products, seed in ((most, 1, 5), (n, 0, 6), (most, 0, 7), (n, 1, 8), (most, 1, 9)):
        net.set_option("ft_bwd_products", products)
        batch = draw_batch(desc, count, seed)
        net.upload(0, *batch)
        _, g_ref, _ = oracle32.net_grad(desc, w, *batch)
        for parts in (1, 4, 8):
            net.backward_begin(0)
            for part in range(parts):
                net.backward_ft(0, part, parts)
            net.backward_end(0)
            assert net.stat("ft_products") == products
            g = net.tensors(kind=3)
            for k in g_ref:
                assert np.abs(g[k] - g_ref[k]).max() <= 2e-5 * np.abs(g_ref[k]).max(), (k, count, parts)
    net.close()


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("products", [0, 1])
@pytest.mark.parametrize("ft_out,pairwise,act,dense", [(72, False, ACT_SCRELU, (1,)), (96, False, ACT_CRELU, (1,)), (64, False, ACT_SCRELU, (8, 1)),
                                                       (136, True, ACT_CRELU, (1,)), (128, True, ACT_CRELU, (16, 32, 1))])
def test_products_of_gradients_that_are_not_finite(oracle32, ft_out, pairwise, act, dense, products, value):
    """The same with both backward passes of small tables, in one row block and in three; next comes a batch that is finite.  Bounds as above."""
    import dataclasses

    from tests.test_gpu_parity import make_net, rich_weights

    n, bad = 300, 117
    blocks = 3 if ft_out % 64 == 0 else 1  # (other widths are one block)
    desc = dataclasses.replace(net_of(blocks, 100, ft_out, 31, 1, dense, act, pairwise), max_batch=n)
    stm, nstm, bucket, target = draw_batch(desc, n, seed=ft_out)
    w = rich_weights(desc)
    rest = np.arange(n) != bad
    _, g_ref, _ = oracle32.net_grad(desc, w, stm[rest], nstm[rest], bucket[rest], target[rest])
    _, g_all, _ = oracle32.net_grad(desc, w, stm, nstm, bucket, target)
    broken = target.copy()
    broken[bad] = value
    net = make_net(desc, 0, w)
    net.set_option("ft_bwd_products", products)
    net.upload(0, stm, nstm, bucket, broken)
    net.upload(1, stm, nstm, bucket, target)
    lost = np.zeros(desc.n_inputs, dtype=bool)
    for row in np.concatenate([stm[bad], nstm[bad]]):
        lost[max(row, 0)] |= row >= 0
    ref = g_ref["l0w"].reshape(desc.n_inputs, ft_out)
    for _ in range(2):
        net.backward(0)
        assert net.stat("ft_products") == products
        g = net.tensors(kind=3)
        got = g["l0w"].reshape(desc.n_inputs, ft_out)
        assert not np.isfinite(got[lost]).any()
        assert not np.isfinite(g["l0b"]).any()
        assert np.abs(got[~lost] - ref[~lost]).max() <= 2e-5 * np.abs(ref).max()
        first = net.tensor_range("l0w")[0]
        assert np.isfinite(net_flat(net, 3)[first + got.size:]).all()
        net.backward(1)
        g = net.tensors(kind=3)
        for k in g_all:
            assert np.abs(g[k] - g_all[k]).max() <= 2e-5 * np.abs(g_all[k]).max(), k
    net.close()


@pytest.mark.parametrize("nnz", [8, 32, 64])
@pytest.mark.parametrize("rows_less", [0, 3, 16])
def test_the_largest_tables_of_the_tiled_kernels(oracle32, nnz, rows_less):
    """Row blocks up to the largest whose tile fits into shared memory beside two bytes per list slot and warp: the last of them
    leave room for the lists of some of the warps only.  Network (kernels asked for by name) and operator.  Bounds as above."""
    import dataclasses

    from tests.test_gpu_ops import run_op
    from tests.test_gpu_parity import make_net, rich_weights

    rows, n = (227 * 1024 - 16 - 64 * ((nnz + 7) // 8 * 8)) // 256 - 1 - rows_less, 500
    desc = dataclasses.replace(net_of(2, rows, 128, nnz, 1, (1,)), max_batch=n)
    stm, nstm, bucket, target = draw_batch(desc, n, seed=nnz)
    w = rich_weights(desc)
    x_ref = oracle_x(oracle32, desc, w, stm, nstm)
    net = make_net(desc, 2, w)
    net.upload(0, stm, nstm, bucket, target)
    net.backward(0)
    assert np.array_equal(net.activation(0, n * desc.dense_in0).reshape(n, -1), x_ref)
    _, g_ref, _ = oracle32.net_grad(desc, w, stm, nstm, bucket, target)
    g = net.tensors(kind=3)
    for k in g_ref:
        assert np.abs(g[k] - g_ref[k]).max() <= 2e-5 * np.abs(g_ref[k]).max(), k
    net.close()
    for entry in ("b200_op_ft_forward", "b200_op_ft_forward_noalloc"):
        for x_at in (0, 1):  # (outputs on any float: grouped, however few positions there are)
            rc, x, _ = run_op(entry, desc, w["l0w"], w["l0b"], stm, nstm, n, x_at)
            assert rc == 0 and np.array_equal(x, x_ref)


@pytest.mark.parametrize("rows", [855, 860, 861, 863, 865, 866])
def test_the_longest_chunks_of_the_backward(oracle32, rows):
    """Row counts past where chunks of 640 pairs fit into shared memory, with a batch of 148 of those (one for every SM), which is cut into
    others, and with a short one.  Bounds as above."""
    import dataclasses

    from tests.test_gpu_parity import make_net, rich_weights

    most = 148 * 320
    desc = dataclasses.replace(net_of(1, rows, 64, 32, 1, (1,)), max_batch=most)
    w = rich_weights(desc)
    net = make_net(desc, 0, w)
    for n in (most, 3001):
        batch = draw_batch(desc, n, seed=rows)
        net.upload(0, *batch)
        net.backward(0)
        _, g_ref, _ = oracle32.net_grad(desc, w, *batch)
        g = net.tensors(kind=3)
        for k in g_ref:
            assert np.abs(g[k] - g_ref[k]).max() <= 2e-5 * np.abs(g_ref[k]).max(), k
    net.close()


@pytest.mark.parametrize("rows,chunk", [(832, 640), (838, 640), (839, 640), (840, 640), (841, 632), (843, 632), (846, 632)])
def test_the_tightest_chunks_of_the_backward(oracle32, rows, chunk):
    """Chunks of 640 pairs, a line of zeros behind them, and their lists fill shared memory to the last byte at 840 rows; one row more has
    632.  Batches that are cut into 148 of them (one for every SM).  Bounds as above."""
    import dataclasses

    from tests.test_gpu_parity import make_net, rich_weights

    n = 148 * chunk // 2
    desc = dataclasses.replace(net_of(1, rows, 64, 32, 1, (1,)), max_batch=n)
    w = rich_weights(desc)
    net = make_net(desc, 0, w)
    batch = draw_batch(desc, n, seed=rows)
    net.upload(0, *batch)
    net.backward(0)
    assert net.stat("ft_chunk") == chunk
    _, g_ref, _ = oracle32.net_grad(desc, w, *batch)
    g = net.tensors(kind=3)
    for k in g_ref:
        assert np.abs(g[k] - g_ref[k]).max() <= 2e-5 * np.abs(g_ref[k]).max(), k
    net.close()


@pytest.mark.parametrize("n", [131072, 131073, 262144 + 77])
def test_grouping_of_long_batches(oracle32, n):
    """The last batch whose windows sum the counts themselves, and longer ones whose counts have been summed up before, by one and
    by more rounds: feature-transformer output bit-exact by network and operator, gradients with the bounds above."""
    import dataclasses

    from tests.test_gpu_ops import run_op
    from tests.test_gpu_parity import make_net, rich_weights

    desc = dataclasses.replace(net_of(5, 60, 64, 6, 3, (1,)), max_batch=n)
    batch = draw_batch(desc, n, seed=n & 15)
    w = rich_weights(desc)
    x_ref = oracle_x(oracle32, desc, w, *batch[:2])
    net = make_net(desc, 0, w)
    net.upload(0, *batch)
    net.backward(0)
    assert np.array_equal(net.activation(0, n * desc.dense_in0).reshape(n, -1), x_ref)
    _, g_ref, _ = oracle32.net_grad(desc, w, *batch)
    g = net.tensors(kind=3)
    for k in g_ref:
        # (the oracle adds n terms one after the other: sqrt(n) 2^-24 of the sum in a random walk, and as much again for a drift)
        assert np.abs(g[k] - g_ref[k]).max() <= 6e-5 * np.abs(g_ref[k]).max(), k
    net.close()
    for x_at in (0, 1):
        rc, x, _ = run_op("b200_op_ft_forward", desc, w["l0w"], w["l0b"], *batch[:2], n, x_at)
        assert rc == 0 and np.array_equal(x, x_ref)


@pytest.mark.parametrize("n", [3000, 140000])
def test_groupings_that_follow_each_other_in_the_same_memory(oracle32, n):
    """Two batches of different lists in turn through one scratch and one slot, with and without the kernel that sums the counts up: every
    kernel of a chain reads what the one before it wrote this time.  Bit-exact."""
    import dataclasses

    from tests.test_gpu_ops import run_op
    from tests.test_gpu_parity import make_net, rich_weights

    desc = dataclasses.replace(net_of(5, 60, 64, 8, 3, (1,)), max_batch=n)
    w = rich_weights(desc)
    batches = [draw_batch(desc, n, seed=k) for k in (1, 2)]
    refs = [oracle_x(oracle32, desc, w, *b[:2]) for b in batches]
    for turn in range(6):
        rc, x, _ = run_op("b200_op_ft_forward", desc, w["l0w"], w["l0b"], *batches[turn % 2][:2], n, 1)
        assert rc == 0 and np.array_equal(x, refs[turn % 2])
    net = make_net(desc, 2, w)  # (that never trains: its groupings are chained)
    for turn in range(6):
        net.upload(0, *batches[turn % 2])
        net.forward(0, n)
        assert net.stat("ft_forward") > 0
        assert np.array_equal(net.activation(0, n * desc.dense_in0).reshape(n, -1), refs[turn % 2])
    net.close()


@pytest.mark.parametrize("case", ["blocks-32", "blocks-33", "blocks-256", "blocks-257", "rows-32-last-layer", "list-of-64", "width-8"])
def test_groupings_that_the_kernels_made(case):
    """The positions by output bucket and the pairs by row block that lie on the device, for every way of grouping, before and
    after a training pass: the sets and the order that a stable sort on the CPU gives."""
    import dataclasses

    from tests.test_gpu_parity import make_net, rich_weights, slot_by_hand

    desc, n = CASES[case]
    for n in (n, 5000):
        desc = dataclasses.replace(desc, max_batch=n)
        batch = draw_batch(desc, n, seed=n)
        want = slot_by_hand(desc, batch)
        net = make_net(desc, 0, rich_weights(desc))
        for _ in range(2):
            net.upload(2, *batch)
            got = net.slot_contents(2)
            for k in want:
                assert np.array_equal(got[k], want[k]), k
            net.step(2, 0.0, 1.0 / n)
            got = net.slot_contents(2)
            for k in want:
                assert np.array_equal(got[k], want[k]), k
        net.close()


def net_flat(net, kind):
    import torch

    class Buffer:
        pass

    ptr, count = net.flat_buffer(kind)
    Buffer.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f4", "data": (ptr, False), "version": 3, "strides": None}
    net.sync()
    return torch.as_tensor(Buffer(), device="cuda").cpu().numpy()


@pytest.mark.parametrize("act,buckets", [(ACT_CRELU, 1), (ACT_SCRELU, 4)])
def test_gradient_at_x_is_that_of_the_last_training_pass(act, buckets):
    """Networks with one dense row per bucket keep no gradient at x, but tell it: that of the last training pass, also after
    evaluations of more positions, an update, and weights that were set anew.  Positions without one are zero."""
    import dataclasses

    from tests.test_gpu_parity import make_net, rich_weights

    few, many = 8, 100
    desc = dataclasses.replace(net_of(1, 300, 64, 31, buckets, (1,), act), max_batch=many)
    K = desc.dense_in0
    w = rich_weights(desc)
    net = make_net(desc, 0, w)
    stm, nstm, bucket, target = draw_batch(desc, many, seed=3)
    net.upload(0, stm[:few], nstm[:few], bucket[:few], target[:few])
    net.upload(1, stm, nstm, bucket, target)
    net.forward(1, many)
    assert not net.activation(2, many * K).any()  # no training pass yet
    net.backward(0)
    # the weight of the position's bucket times its loss gradient
    out = net.activation(3, few).astype(np.float64)
    s = 1 / (1 + np.exp(-out))
    dout = 2 * (s - target[:few]) * s * (1 - s)
    ref = w["l1w"].reshape(K, buckets).T[bucket[:few]] * dout[:, None]
    got = net.activation(2, few * K).reshape(few, K)
    assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max()  # of 32 bits, and of the sigmoid's exponential

    def check():
        dx = net.activation(2, many * K).reshape(many, K)
        assert np.array_equal(dx[:few], got) and not dx[few:].any()

    net.forward(1, many)
    check()
    net.update(1e-2, 1.0 / few)
    net.forward(1, many)
    check()
    for seed in (11, 12):
        net.load_weights(rich_weights(desc, seed=seed))
        net.forward(1, many)
        check()
    net.step(0, 1e-2, 1.0 / few)  # the next training pass, in one call, with the weights set last
    out = net.activation(3, few).astype(np.float64)
    s = 1 / (1 + np.exp(-out))
    dout = 2 * (s - target[:few]) * s * (1 - s)
    ref = rich_weights(desc, seed=12)["l1w"].reshape(K, buckets).T[bucket[:few]] * dout[:, None]
    got = net.activation(2, few * K).reshape(few, K)
    assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max()
    for seed in (13, 14, 15):  # formed only now, after the copy that the pass used would have been overwritten
        net.load_weights(rich_weights(desc, seed=seed))
        net.forward(1, many)
    check()
    net.close()


@pytest.mark.parametrize("bwd_mode", [0, 1])
def test_forward_in_parts_and_reports_of_a_small_batch(oracle32, bwd_mode):
    """A batch small enough for the gather forward, with the backward's kernels left to choose and the gather ones asked for:
    the forward may still be run in parts, by the tiled kernel, also in a slot that held another batch before, and a feature
    outside its row block is still reported.  Bounds as above."""
    import dataclasses

    from bullet_b200._lib import B200Error
    from tests.test_gpu_parity import make_net, rich_weights

    most, n = 900, 6
    desc = dataclasses.replace(net_of(8, 96, 64, 20, 2, (8, 1)), max_batch=most)
    w = rich_weights(desc)
    net = make_net(desc, 0, w)
    net.set_option("ft_bwd_mode", bwd_mode)
    for count, seed in ((n, 5), (most, 6), (n, 7)):
        stm, nstm, bucket, target = draw_batch(desc, count, seed)
        net.upload(0, stm, nstm, bucket, target)
        x_ref = oracle_x(oracle32, desc, w, stm, nstm)
        _, g_ref, _ = oracle32.net_grad(desc, w, stm, nstm, bucket, target)
        for parts in (4, 1):
            net.forward_begin(0)
            for part in range(parts):
                net.forward_ft(0, part, parts)
            net.backward_begin(0)
            assert np.array_equal(net.activation(0, count * desc.dense_in0).reshape(count, -1), x_ref)
            net.backward_ft(0, 0, 1)
            net.backward_end(0)
            g = net.tensors(kind=3)
            for k in g_ref:
                assert np.abs(g[k] - g_ref[k]).max() <= 2e-5 * np.abs(g_ref[k]).max(), k
    stm[0, :2] = [3, 200]  # rows of two blocks
    net.upload(1, stm, nstm, bucket, target)
    for step in (lambda: net.step(1, 0.0, 1.0 / n), lambda: (net.backward(1), net.update(0.0, 1.0 / n))):
        step()
        with pytest.raises(B200Error) as e:
            net.loss()
        assert e.value.code == -4
    net.close()


def oracle_x(oracle32, desc, w, stm, nstm):
    from tests.test_gpu_parity import oracle_ft_output

    return oracle_ft_output(oracle32, desc, w, stm, nstm)


def oracle_u(oracle32, desc, w, stm, nstm):
    """The pairwise halves before their product, of a network without a factoriser: [n][2][ft_out]."""
    n, h = len(stm), desc.ft_out
    sums = [oracle32.sparse_matmul(w["l0w"], idx, n, h, desc.n_inputs, h, 0, desc.nnz).reshape(n, h) + w["l0b"][None, :] for idx in (stm, nstm)]
    return np.stack([oracle32.act_forward(ACT_CRELU, a.ravel()).reshape(n, h) for a in sums], axis=1)


@pytest.mark.parametrize("dense,buckets", [((4, 1), 1), ((8, 1), 3), ((16, 32, 1), 2), ((32, 32, 1), 2)])
def test_products_of_the_first_dense_layer_keep_32_bits(dense, buckets):
    """One position: the weight gradient is x times the gradient at the layer's output, one product an entry, and that gradient is
    the bias gradient; the gradient at x is a sum of as many products as the layer has rows.  A product whose operands are split
    into parts is off by at most 2^-24 for the sum of its parts, 2^-25 for the parts left out and 2^-8 2^-22 for what the
    accumulator of the small parts loses: below 2^-23.  A sum of R products adds at most log2(R) + 2 such roundings."""
    import dataclasses

    from tests.test_gpu_parity import make_net, rich_weights

    desc = dataclasses.replace(net_of(1, 300, 264, 31, buckets, dense), max_batch=1, dense_act=(ACT_NONE,) * len(dense))
    K, M = desc.dense_in0, dense[0]
    for seed in range(6):
        w = rich_weights(desc, seed=seed)
        rng = np.random.default_rng(seed)
        w["l1w"] = rng.normal(0, 0.05, w["l1w"].size).astype(np.float32)
        net = make_net(desc, 0, w)
        net.upload(0, *draw_batch(desc, 1, seed + 40))
        net.backward(0)
        k = int(draw_batch(desc, 1, seed + 40)[2][0])
        g = net.tensors(kind=3)
        x = net.activation(0, K).astype(np.float64)
        dz = g["l1b"].reshape(buckets, M)[k].astype(np.float64)
        assert (dz != 0).sum() > M // 2 and (x != 0).sum() > K // 8
        gw = g["l1w"].reshape(K, buckets, M)
        exact = x[:, None] * dz[None]
        assert (np.abs(gw[:, k] - exact) <= 2.0**-23 * np.abs(exact)).all()
        assert not gw[:, [b for b in range(buckets) if b != k]].any()
        terms = w["l1w"].reshape(K, buckets, M)[:, k].astype(np.float64) * dz
        bound = (np.log2(M) + 2) * 2.0**-23 * np.abs(terms).sum(1)
        assert (np.abs(net.activation(2, K) - terms.sum(1)) <= bound).all()
        net.close()


@pytest.mark.parametrize("dense", [(4, 1), (8, 1), (16, 32, 1), (32, 32, 1)])
def test_nan_passes_through_the_first_dense_layer(dense):
    """A target that is NaN, or a weight, reaches every gradient that it is part of, and no other."""
    import dataclasses

    from tests.test_gpu_parity import make_net, rich_weights

    n, bad, buckets = 50, 20, 2
    desc = dataclasses.replace(net_of(1, 300, 136, 31, buckets, dense), max_batch=n)
    K, M = desc.dense_in0, dense[0]
    w = rich_weights(desc)
    w["l1b"] = np.full(w["l1b"].size, 0.4, np.float32)
    w["l1w"] *= np.float32(0.1)  # no output is clamped
    batch = draw_batch(desc, n, seed=2)
    batch[3][bad] = np.nan
    k = int(batch[2][bad])
    net = make_net(desc, 0, w)
    net.upload(0, *batch)
    for step in (lambda: net.backward(0), lambda: net.step(0, 0.0, 1.0 / n)):
        step()
        dx = net.activation(2, n * K).reshape(n, K)
        assert np.isnan(dx[bad]).all() and not np.isnan(np.delete(dx, bad, 0)).any()
        gw = net.tensors(kind=3)["l1w"].reshape(K, buckets, M)
        assert np.isnan(gw[:, k]).all() and not np.isnan(gw[:, 1 - k]).any()
    net.close()
    batch[3][bad] = 0.5
    for nan in (0x7FC00000, 0x7FFFFFFF, 0xFFFFFFFF):
        w2 = {name: v.copy() for name, v in w.items()}
        w2["l1w"].reshape(K, buckets, M)[5, k, 1] = np.array([nan], np.uint32).view(np.float32)[0]
        net = make_net(dataclasses.replace(desc, dense_act=(ACT_NONE,) * len(dense)), 0, w2)
        net.upload(0, *batch)
        out = net.forward(0, n)
        assert np.array_equal(np.isnan(out), batch[2] == k)
        net.close()


# rows, blocks, slots, width, pairwise, activation, dense layers, output buckets, positions, a row twice in a list
PRODUCTS = {
    "one-row": (1, 1, 1, 32, False, ACT_CRELU, (1,), 1, 3, False),
    "rows-31": (31, 3, 20, 64, False, ACT_SCRELU, (1,), 4, 700, False),
    "rows-32": (32, 1, 32, 40, False, ACT_CRELU, (8, 1), 2, 65, False),
    "rows-147-ragged-width": (147, 1, 49, 72, False, ACT_CRELU, (1,), 1, 1000, False),
    "rows-255": (255, 2, 64, 128, False, ACT_SCRELU, (4, 1), 1, 129, False),
    "rows-223": (223, 1, 9, 64, False, ACT_CRELU, (1,), 3, 4000, False),
    "rows-255-pairwise": (255, 1, 32, 136, True, ACT_CRELU, (16, 32, 1), 8, 900, False),
    "rows-255-pairwise-one": (255, 1, 32, 64, True, ACT_CRELU, (1,), 1, 64, False),
    "counts": (150, 2, 40, 64, False, ACT_CRELU, (1,), 2, 300, True),
    "counts-pairwise": (200, 1, 64, 128, True, ACT_CRELU, (8, 1), 1, 150, True),
    "sums-taken-out-on-the-way": (2, 1, 1, 32, False, ACT_CRELU, (1,), 1, 2600000, False),
}


def sums_in_64_bits(net, desc, batch):
    """(sum, sum of magnitudes) in 64 bits of the last pass's gradients at the pre-activations, which follow from what the pass kept: of
    the table and of the bias."""
    n = len(batch[0])
    x, dx = (net.activation(k, n * desc.dense_in0).reshape(n, 2, -1) for k in (0, 2))
    if desc.pairwise:
        u = net.activation(1, n * 2 * desc.ft_out).reshape(n, 2, 2, desc.ft_out // 2)
        pre = np.stack([dx * u[:, :, 1], dx * u[:, :, 0]], axis=2).astype(np.float64) * ((u > 0) & (u < 1))
        pre = pre.reshape(n, 2, desc.ft_out)
    else:
        slope = ((x > 0) & (x < 1)) * (2 * np.sqrt(x) if desc.ft_act == ACT_SCRELU else np.float32(1))
        pre = dx.astype(np.float64) * slope
    out = []
    for values in (pre, np.abs(pre)):
        table = np.zeros((desc.n_inputs, desc.ft_out))
        for side in range(2):
            index = batch[side]
            for slot in range(desc.nnz):
                on = index[:, slot] >= 0
                if n > 100000:
                    for c in range(desc.ft_out):
                        table[:, c] += np.bincount(index[on, slot], values[on, side, c], desc.n_inputs)
                else:
                    np.add.at(table, index[on, slot], values[on, side])
        out += [(table, values.sum((0, 1)))]
    return out


@pytest.mark.parametrize("case", PRODUCTS)
def test_products_of_bytes_are_no_further_from_64_bits_than_the_walk(case):
    """The backward of small tables: the gradient of the table and the bias against the sums in 64 bits of the gradients at
    the pre-activations, which follow from what the step kept.  Per sum one rounding of 2^-24 and per addend one to 2^-31 of the
    largest gradient; the walk over lists rounds at every addition, so it is the bound, and 2^-24 where it happens to be exact."""
    import dataclasses

    from tests.test_gpu_parity import make_net, rich_weights

    rows, blocks, nnz, ft_out, pairwise, act, dense, buckets, n, twice = PRODUCTS[case]
    desc = dataclasses.replace(net_of(blocks, rows, ft_out, nnz, buckets, dense, act, pairwise), max_batch=n)
    desc = dataclasses.replace(desc, ft_block_rows=rows if ft_out % 64 == 0 or blocks > 1 else 0)
    if n > 100000:  # (the drawing of draw_batch sorts every list)
        rng = np.random.default_rng(n)
        stm, nstm = (rng.integers(0, rows, (n, 1)).astype(np.int32) for _ in range(2))
        batch = (stm, nstm, np.zeros(n, np.int32), rng.random(n).astype(np.float32))
    else:
        batch = draw_batch(desc, n, seed=rows + n)
    if twice:
        for lists in batch[:2]:
            lists[::3, 1] = lists[::3, 0]
            lists[::3, -1] = lists[::3, 0]
    w = rich_weights(desc)
    error = {}
    for products in (0, 1):
        net = make_net(desc, 0, w)
        net.set_option("ft_bwd_products", products)
        net.upload(0, *batch)
        net.step(0, 0.0, 1.0 / n)
        net.loss()
        g = net.tensors(kind=3)
        (table, bias), magnitudes = sums_in_64_bits(net, desc, batch)
        assert net.stat("ft_products") == products
        if products:
            # every single sum, in units of 2^-24 of its magnitudes: two for an addend, twelve for the eight digits' sums put together,
            # 148 parts at most (see test_small_gradients_beside_large_ones_keep_32_bits)
            for k, ref, all_of_it in zip(("l0w", "l0b"), (table, bias), magnitudes):
                assert (np.abs(g[k].reshape(ref.shape) - ref) <= 162 * 2.0 ** -24 * all_of_it).all(), k
        error[products] = [np.linalg.norm(g[k].astype(np.float64).reshape(ref.shape) - ref) / max(np.linalg.norm(ref), 1e-300)
                           for k, ref in (("l0w", table), ("l0b", bias))]
        print(case, "products" if products else "walk", error[products])
        net.close()
    # Both round the product at every pre-activation, which the reference has in common, and both add fp32 parts in any order, a few of
    # a sum here, dozens of the bias or of a batch that all CTAs share: of a few sums two such errors differ by less than twice, of
    # thousands by a few per cent.
    for mine, walk, sums in zip(error[1], error[0], (table.size, bias.size)):
        assert mine <= max((1.05 if sums > 1000 else 2) * walk, 2.0 ** -24)


@pytest.mark.parametrize("products", [0, 1])
@pytest.mark.parametrize("dense,pairwise,act", [((1,), False, ACT_CRELU), ((1,), False, ACT_SCRELU), ((1,), True, ACT_CRELU), ((8, 1), False, ACT_SCRELU),
                                                ((16, 32, 1), True, ACT_CRELU)])
def test_small_gradients_beside_large_ones_keep_32_bits(products, dense, pairwise, act):
    """Columns of the first dense layer over seven decades and positions whose gradients span six: every single sum is as close
    to 64 bits as fp32 makes it, whatever else the batch holds.

    In units of 2^-24 of a sum's magnitudes: an addend is rounded at most twice, the digits' sums (at most three times the magnitudes) four
    times when they are put together, and the at most 48 parts that CTAs hold of a sum are added in fp32: 62, taken as 64.  The walk
    over lists rounds in each of its up to 900 additions, a random walk of 30."""
    import dataclasses

    from tests.test_gpu_parity import make_net, rich_weights

    n, rows, nnz, ft_out = 3000, 147, 40, 128
    desc = dataclasses.replace(net_of(1, rows, ft_out, nnz, 1, dense, act, pairwise), max_batch=n)
    w = rich_weights(desc)
    shape = desc.tensor_shapes()["l1w"]
    decades = 10.0 ** -np.linspace(0, 7, desc.dense_in0).astype(np.float32)
    rng = np.random.default_rng(3)
    rng.shuffle(decades)
    first = w["l1w"].reshape(shape)
    w["l1w"] = (first * (decades if shape[1] == desc.dense_in0 else decades[:, None])).astype(np.float32).ravel()
    stm, nstm, bucket, target = draw_batch(desc, n, seed=8)
    net = make_net(desc, 0, w)
    net.set_option("ft_bwd_products", products)
    net.upload(0, stm, nstm, bucket, target)
    out = net.forward(0, n).astype(np.float64)
    target = 1 / (1 + np.exp(-out)) + rng.choice([-1, 1], n) * 10.0 ** -rng.uniform(0.4, 6.4, n)
    batch = (stm, nstm, bucket, target.astype(np.float32))
    net.upload(0, *batch)
    net.step(0, 0.0, 1.0 / n)
    assert net.stat("ft_products") == products
    g = net.tensors(kind=3)
    sums, magnitudes = sums_in_64_bits(net, desc, batch)
    for k, ref, all_of_it in zip(("l0w", "l0b"), sums, magnitudes):
        assert all_of_it.max() > 0
        off = np.abs(g[k].reshape(ref.shape) - ref) / np.maximum(all_of_it, 2.0 ** -120)
        print(k, off.max() * 2 ** 24)
        assert off.max() <= 64 * 2.0 ** -24, k
    net.close()


@pytest.mark.parametrize("products", [0, 1])
@pytest.mark.parametrize("dense,pairwise", [((1,), False), ((8, 1), False), ((16, 32, 1), True)])
def test_gradients_of_two_passes_add_up_where_the_caller_clears_them(products, dense, pairwise):
    """Row blocks and columns enough that a CTA of the product backward has whole units to itself.  Two passes over one batch give twice
    the gradient of one; the sums differ by the order of their fp32 parts (bound above)."""
    import dataclasses

    from tests.test_gpu_parity import make_net, rich_weights

    n = 700
    desc = dataclasses.replace(net_of(8, 31, 1024, 20, 2, dense, ACT_CRELU, pairwise), max_batch=n)
    net = make_net(desc, 0, rich_weights(desc))
    net.set_option("ft_bwd_products", products)
    net.set_option("manual_grad_zero", 1)
    net.upload(0, *draw_batch(desc, n, seed=5))
    net.grad_zero_range(0, net.stat("flat_floats"))
    net.backward(0)
    once = net.tensors(kind=3)
    net.backward(0)
    twice = net.tensors(kind=3)
    for k, g in once.items():
        assert np.abs(g).max() > 0, k
        assert np.abs(twice[k] - 2 * g).max() <= 2e-5 * np.abs(2 * g).max(), k
    net.close()


# rows, blocks, slots, width, pairwise, dense layers, positions: which of the two is the faster backward, by its measured side of the line
FASTER = {
    "ataxx": (147, 1, 49, 256, False, (1,), 32768, 1),
    "ataxx-few": (147, 1, 49, 64, False, (1,), 512, 1),
    "ataxx-fewer": (147, 1, 49, 64, False, (1,), 100, 0),
    "ataxx-pairwise": (147, 1, 49, 512, True, (16, 32, 1), 16384, 1),
    "rows-255": (255, 1, 32, 256, False, (1,), 32768, 1),
    "rows-255-short-lists": (255, 1, 8, 256, False, (1,), 32768, 0),
    "rows-255-pairwise": (255, 1, 32, 512, True, (16, 32, 1), 16384, 0),
    "rows-256": (256, 1, 49, 256, False, (1,), 32768, 0),
    "eight-blocks": (200, 8, 32, 256, False, (1,), 16384, 1),
    "eight-blocks-few-pairs": (200, 8, 32, 2048, False, (1,), 1024, 0),
    "many-blocks": (147, 64, 32, 2048, False, (1,), 1024, 0),
    "a-thousand-blocks": (31, 1000, 8, 2048, False, (1,), 1024, 0),
}


@pytest.mark.parametrize("case", FASTER)
def test_small_tables_take_the_faster_backward(case):
    rows, blocks, nnz, ft_out, pairwise, dense, n, products = FASTER[case]
    import dataclasses

    from tests.test_gpu_parity import make_net

    desc = dataclasses.replace(net_of(blocks, rows, ft_out, nnz, 1, dense, ACT_CRELU, pairwise), max_batch=n)
    net = make_net(desc)
    net.upload(0, *draw_batch(desc, n, seed=n))
    net.step(0, 0.0, 1.0 / n)
    net.loss()
    assert net.stat("ft_products") == products
    net.close()


@pytest.mark.parametrize("blocks,rows,ft_out,nnz,pairwise,factoriser,used", [
    (3, 128, 1664, 16, False, 0, (0, 1, 2)),       # a whole round of rows
    (3, 129, 1664, 16, True, 129, (0, 1, 2)),      # one row more, in the second round
    (2, 31, 2432, 31, True, 0, (0, 1)),            # less than a round
    (5, 200, 2048, 20, False, 200, (1, 3)),        # blocks without pairs between the tiles
    (2, 768, 2560, 32, True, 768, (0, 1)),
    (2, 860, 2432, 64, False, 0, (0, 1)),          # the last rounds of rows
    (1, 300, 4808, 12, False, 0, (0,)),            # a last slab that is not full
    (1, 300, 4816 * 2, 12, True, 0, (0,)),
])
def test_tiles_fetched_while_the_one_before_is_walked(oracle32, blocks, rows, ft_out, nnz, pairwise, factoriser, used):
    """More tiles than CTAs, with enough pairs each for the forward to fetch a CTA's next tile during the walk: rows at the edges of the
    rounds it is fetched in, over several tiles a CTA.  Bit-exact, network (a whole batch and in parts) and operator."""
    import dataclasses

    from tests.test_gpu_ops import run_op
    from tests.test_gpu_parity import make_net, rich_weights

    n = 515 * blocks + 7
    desc = dataclasses.replace(net_of(blocks, rows, ft_out, nnz, 1, (1,), pairwise=pairwise), max_batch=n, factoriser_rows=factoriser)
    if blocks == 1:
        desc = dataclasses.replace(desc, ft_block_rows=0)
    stm, nstm, bucket, target = draw_batch(desc, n, seed=rows + ft_out)
    for index in (stm, nstm):  # into the blocks that are used
        at = np.array(used)[index // rows % len(used)]
        np.copyto(index, np.where(index >= 0, at * rows + index % rows, -1))
    w = rich_weights(desc)
    x_ref = oracle_x(oracle32, desc, w, stm, nstm)
    net = make_net(desc, 0, w)
    net.upload(0, stm, nstm, bucket, target)
    net.forward(0, n)
    assert np.array_equal(net.activation(0, n * desc.dense_in0).reshape(n, -1), x_ref)
    if blocks > 1:
        net.forward_begin(0)
        for part in range(blocks):
            net.forward_ft(0, part, blocks)
        net.backward_begin(0)
        assert np.array_equal(net.activation(0, n * desc.dense_in0).reshape(n, -1), x_ref)
        if not factoriser:
            for x_at in (0, 1):
                rc, x, _ = run_op("b200_op_ft_forward", desc, w["l0w"], w["l0b"], stm, nstm, n, x_at)
                assert rc == 0 and np.array_equal(x, x_ref)
    net.close()


@pytest.mark.parametrize("blocks,rows,ft_out,nnz,pairwise,factoriser", [
    (3, 128, 1664, 16, False, 0), (3, 129, 1664, 16, True, 129), (2, 31, 2432, 31, True, 0), (5, 200, 2048, 20, False, 200), (2, 768, 2560, 32, True, 768),
    (2, 876, 2432, 64, False, 0),   # a warp that walks no lists
    (2, 890, 2432, 64, True, 0),    # ... as many of them as there can be
    (1, 300, 4808, 20, False, 0),   # a last slab that is not full
    (1, 300, 4816 * 2, 12, True, 0),
])
def test_the_forward_that_fetches_tiles_ahead_is_the_one_that_runs(oracle32, blocks, rows, ft_out, nnz, pairwise, factoriser):
    """Evaluations and steps of the sizes above take that form, also with warps that only fetch.  Bit-exact, and so is the operator."""
    import dataclasses

    from tests.test_gpu_ops import run_op
    from tests.test_gpu_parity import make_net, rich_weights

    n = 515 * blocks + 7
    desc = dataclasses.replace(net_of(blocks, rows, ft_out, nnz, 1, (1,), pairwise=pairwise), max_batch=n, factoriser_rows=factoriser)
    if blocks == 1:
        desc = dataclasses.replace(desc, ft_block_rows=0)
    batch = draw_batch(desc, n, seed=rows + ft_out)
    w = rich_weights(desc)
    x_ref = oracle_x(oracle32, desc, w, *batch[:2])
    net = make_net(desc, 0, w)
    net.upload(0, *batch)
    for run in (lambda: net.forward(0, n), lambda: net.step(0, 0.0, 1.0 / n)):
        run()
        assert net.stat("ft_forward") == 2
        assert np.array_equal(net.activation(0, n * desc.dense_in0).reshape(n, -1), x_ref)
    net.close()
    if blocks > 1 and not factoriser:
        for x_at in (0, 1):
            rc, x, _ = run_op("b200_op_ft_forward", desc, w["l0w"], w["l0b"], *batch[:2], n, x_at)
            assert rc == 0 and np.array_equal(x, x_ref)


@pytest.mark.parametrize("copies,rows,ft_out,dense,buckets", [
    (1, 40, 64, (1,), 1), (2, 129, 64, (8, 1), 2), (15, 33, 128, (1,), 3), (16, 64, 64, (16, 32, 1), 2), (17, 31, 64, (1,), 1), (33, 24, 192, (4, 1), 2)])
def test_update_of_networks_with_a_factoriser(copies, rows, ft_out, dense, buckets):
    """A whole step's update: copies on either side of the sixteen that are taken at a time, copies that are no whole number of a CTA's
    columns.  The factoriser's gradient is the sum of its copies' in order, to the last bit; the update is AdamW's from zero moments in
    32 bits, of a few operations whose order and contraction the compiler chooses: four roundings of the weight and of the step."""
    import dataclasses

    from bullet_b200.configs import AdamWParams
    from tests.test_gpu_parity import make_net, rich_weights

    n, lr = 700, 1e-3
    desc = dataclasses.replace(net_of(copies, rows, ft_out, 12, buckets, dense), max_batch=n, factoriser_rows=rows)
    w = rich_weights(desc)
    net = make_net(desc, 0, w)
    net.upload(0, *draw_batch(desc, n, seed=copies))
    net.step(0, lr, 1.0 / n)
    net.sync()
    g, p = net.tensors(kind=3), net.tensors()
    each = g["l0w"].reshape(copies, rows * ft_out)
    total = each[0].copy()
    for c in range(1, copies):
        total += each[c]
    assert np.array_equal(g["l0f"], total) and np.abs(total).max() > 0
    hp = AdamWParams()
    for k in w:
        grad = g[k].astype(np.float64) / n
        m, v = (1 - hp.beta1) * grad, (1 - hp.beta2) * grad * grad
        step = lr * m / (np.sqrt(v) + 1e-8)
        ref = np.clip(w[k].astype(np.float64).ravel() * (1 - hp.decay * lr) - step, hp.min_weight, hp.max_weight)
        # (1 - beta is a difference of fp32 numbers: beta2's is off by up to 2^-25 / 1e-3 of itself, the root of it by half of that)
        bound = 4 * 2.0**-24 * np.abs(ref) + (2.0**-16 + 8 * 2.0**-24) * np.abs(step) + 1e-12
        assert (np.abs(p[k] - ref) <= bound).all(), k
    net.close()


@pytest.mark.parametrize("copies,rows,ft_out,dense,buckets,by_warps", [
    (1, 40, 64, (1,), 1, 0), (2, 129, 64, (8, 1), 2, 0), (3, 31, 64, (1,), 1, 0),   # a thread takes all copies
    (5, 700, 512, (1,), 2, 0),                                                     # ... of a wide table
    (4, 31, 64, (8, 1), 1, 1), (5, 129, 64, (1,), 2, 1), (8, 33, 64, (1,), 1, 1),  # sets of warps: four, three and a warp less, two
    (15, 33, 128, (1,), 3, 1), (16, 64, 64, (16, 32, 1), 2, 1), (16, 700, 512, (1,), 1, 1),
    (17, 31, 64, (1,), 1, 1), (33, 24, 192, (4, 1), 2, 1), (40, 24, 64, (1,), 1, 1)])  # rounds: two of nine, three of eleven and fourteen
def test_forms_of_the_update_with_a_factoriser(copies, rows, ft_out, dense, buckets, by_warps):
    """The same for the edges of both its forms, and which of them a network takes."""
    import dataclasses

    from tests.test_gpu_parity import make_net, rich_weights

    test_update_of_networks_with_a_factoriser(copies, rows, ft_out, dense, buckets)
    n = 100
    desc = dataclasses.replace(net_of(copies, rows, ft_out, 12, buckets, dense), max_batch=n, factoriser_rows=rows)
    net = make_net(desc, 0, rich_weights(desc))
    net.upload(0, *draw_batch(desc, n, seed=copies))
    net.step(0, 1e-3, 1.0 / n)
    net.sync()
    assert net.stat("update_copies") == by_warps
    net.close()


def test_update_goes_with_the_parameters_not_with_the_copies():
    """The update's time per parameter with few copies of the factoriser against sixteen, which keep every warp of a CTA busy.  Few copies take
    0.85 of it (their tables fit into L2); CTAs of sixteen warps whatever the copies are took 3.4 and 1.6 of it with one copy and four."""
    import dataclasses

    from tests.test_gpu_parity import make_net, rich_weights

    n, per_float = 1024, {}
    for copies in (16, 1, 4):
        desc = dataclasses.replace(net_of(copies, 768, 1024, 12, 1, (1,)), max_batch=n, factoriser_rows=768)
        net = make_net(desc, 0, rich_weights(desc))
        net.upload(0, *draw_batch(desc, n, seed=copies))
        times = []
        for _ in range(6):
            for _ in range(10):
                net.step(0, 1e-3, 1.0 / n)
            times.append(net.timings()["optimiser"])
        per_float[copies] = min(times) / (copies + 1)
        net.close()
    assert per_float[1] <= 1.4 * per_float[16] and per_float[4] <= 1.4 * per_float[16], per_float


@pytest.mark.parametrize("n,ft_out,nnz,pairwise", [
    (901, 576, 12, False),     # 256 columns a warp, a third chunk that is not full
    (1301, 320, 40, False),    # 512 columns a warp, a chunk that is not full, lists of more than 32 slots
    (3601, 64, 33, False),     # less than 128 columns
    (1303, 768, 20, True),     # 128 columns of each half, two rows at a time
    (20011, 128, 5, False),    # several pairs a warp, the last one's alone
    (97, 576, 12, False),      # few warps: four rows at a time
    (97, 768, 35, True),
])
def test_shapes_of_the_gather_forward(oracle32, n, ft_out, nnz, pairwise):
    """The operator's gather forward in its shapes, bit-exact, and a feature outside its block reported."""
    import dataclasses

    from tests.test_gpu_ops import run_op
    from tests.test_gpu_parity import rich_weights

    desc = dataclasses.replace(net_of(3, 96, ft_out, nnz, 1, (1,), pairwise=pairwise), max_batch=n)
    stm, nstm, _, _ = draw_batch(desc, n, seed=n)
    w = rich_weights(desc)
    x_ref = oracle_x(oracle32, desc, w, stm, nstm)
    rc, x, _ = run_op("b200_op_ft_forward", desc, w["l0w"], w["l0b"], stm, nstm, n)
    assert rc == 0 and np.array_equal(x, x_ref)
    stm[n // 2, :2] = [3, 100]  # rows of two blocks
    rc, _, _ = run_op("b200_op_ft_forward", desc, w["l0w"], w["l0b"], stm, nstm, n)
    assert rc != 0


@pytest.mark.parametrize("n,ft_out,nnz", [
    (901, 960, 12),     # 512 columns a warp, a second chunk that is not full
    (1901, 192, 40),    # 256 columns a warp, a chunk that is not full
    (590, 1024, 9),     # on either side of where wide tables go on to one row at a time
    (593, 1024, 9),
])
def test_more_shapes_of_the_gather_forward(oracle32, n, ft_out, nnz):
    test_shapes_of_the_gather_forward(oracle32, n, ft_out, nnz, False)


@pytest.mark.parametrize("n,ft_out,nnz", [
    (1303, 768, 20),    # 128 columns of each half, two rows at a time
    (97, 768, 35),      # few warps: four rows at a time
    (97, 320, 35),      # a second chunk that is not full
    (2100, 320, 64),
])
def test_halves_before_the_pairwise_product(oracle32, n, ft_out, nnz):
    """Both operator outputs of the pairwise form, gathered and (outputs on any float) grouped.  Bit-exact."""
    import dataclasses

    from tests.test_gpu_ops import run_op
    from tests.test_gpu_parity import rich_weights

    desc = dataclasses.replace(net_of(3, 96, ft_out, nnz, 1, (1,), pairwise=True), max_batch=n)
    stm, nstm, _, _ = draw_batch(desc, n, seed=n)
    w = rich_weights(desc)
    x_ref, u_ref = oracle_x(oracle32, desc, w, stm, nstm), oracle_u(oracle32, desc, w, stm, nstm)
    for x_at in (0, 1):
        rc, x, u = run_op("b200_op_ft_forward", desc, w["l0w"], w["l0b"], stm, nstm, n, x_at)
        assert rc == 0 and np.array_equal(x, x_ref) and np.array_equal(u, u_ref)


@pytest.mark.parametrize("blocks,rows,ft_out,nnz,factoriser,n", [
    (64, 96, 512, 12, 96, 1749),   # 2.75 times the table's rows and 2 M floats more
    (16, 96, 64, 12, 96, 511),     # four times
    (8, 100, 64, 50, 100, 63),
    (1, 147, 512, 49, 0, 672),     # 100 MB of slots, and 200 KB for each of a block's rows
    (1, 147, 640, 49, 0, 448),     # ... of columns rounded up to 256
    (4, 31, 1024, 31, 0, 437),
    (1, 768, 64, 20, 0, 2048),     # positions
])
def test_lines_between_the_gather_and_the_tiled_forward(oracle32, blocks, rows, ft_out, nnz, factoriser, n):
    """The last batch that the gather forward takes, and one position more, by evaluations and steps.  Bit-exact."""
    import dataclasses

    from tests.test_gpu_parity import make_net, rich_weights

    desc = dataclasses.replace(net_of(blocks, rows, ft_out, nnz, 1, (1,)), max_batch=n + 1, factoriser_rows=factoriser)
    w = rich_weights(desc)
    net = make_net(desc, 0, w)
    batch = draw_batch(desc, n + 1, seed=n)
    x_ref = oracle_x(oracle32, desc, w, *batch[:2])
    for count in (n, n + 1):
        net.upload(0, *[a[:count] for a in batch])
        for run in (lambda: net.forward(0, count), lambda: net.step(0, 0.0, 1.0 / count)):
            run()
            assert (net.stat("ft_forward") > 0) == (count > n)
            assert np.array_equal(net.activation(0, count * desc.dense_in0).reshape(count, -1), x_ref[:count])
    net.close()


@pytest.mark.parametrize("factoriser,more,less,most", [
    (0, (2048, 320), (2048, 256), 1.3),       # 64 columns more: 1.1, and 1.6 as a chunk of their own
    (768, (157, 1024), (129, 1024), 1.45),    # 17 warps per SM against 14: 1.1, and 1.8 with one row at a time
])
def test_gather_forward_has_no_cliffs(factoriser, more, less, most):
    """Time of the forward of (positions, columns) `more` against that of `less`, by any index set: rules on sizes may not cost more than they give."""
    import dataclasses

    from tests.test_gpu_parity import make_net, rich_weights

    took = []
    for n, ft_out in (more, less):
        desc = dataclasses.replace(net_of(16 if factoriser else 1, 768, ft_out, 32, 1, (1,)), max_batch=n, factoriser_rows=factoriser)
        batch = draw_batch(desc, n, seed=3)
        net = make_net(dataclasses.replace(desc, ft_block_rows=0), 0, rich_weights(desc))
        net.upload(0, *batch)
        times = []
        for _ in range(6):
            for _ in range(10):
                net.step(0, 1e-3, 1.0 / n)
            times.append(net.timings()["ft_forward"])
        took.append(min(times))
        net.close()
    assert took[0] <= most * took[1], took


@pytest.mark.parametrize("n,ft_out,pairwise,dense", [(203, 1024, False, (1,)), (701, 192, False, (8, 1)), (1301, 64, False, (1,)), (703, 512, True, (16, 32, 1)),
                                                     (61, 512, True, (16, 32, 1)), (61, 192, False, (1,))])
def test_shapes_of_the_gather_forward_with_a_factoriser(oracle32, n, ft_out, pairwise, dense):
    """... with the factoriser's row added on the way: batches on either side of the line to four rows at a time, all of them below that to
    the tiled forward.  Bit-exact; gradients with the bounds above (the backward walks lists)."""
    import dataclasses

    from tests.test_gpu_parity import make_net, rich_weights

    desc = dataclasses.replace(net_of(64, 96, ft_out, 12, 2, dense, pairwise=pairwise), max_batch=n, factoriser_rows=96)
    assert n * desc.nnz < 4 * desc.n_inputs
    batch = draw_batch(desc, n, seed=n + ft_out)
    w = rich_weights(desc)
    x_ref = oracle_x(oracle32, desc, w, *batch[:2])
    _, g_ref, out_ref = oracle32.net_grad(desc, w, *batch)
    net = make_net(desc, 0, w)
    net.upload(0, *batch)
    out = net.forward(0, n)
    assert np.array_equal(net.activation(0, n * desc.dense_in0).reshape(n, -1), x_ref)
    assert np.abs(out - out_ref).max() <= 2e-5 * np.abs(out_ref).max()
    net.step(0, 0.0, 1.0 / n)
    g = net.tensors(kind=3)
    for k in g_ref:
        assert np.abs(g[k] - g_ref[k]).max() <= 2e-5 * np.abs(g_ref[k]).max(), k
    net.close()


@pytest.mark.parametrize("n,ft_out", [(985, 320), (369, 1024), (371, 1024)])
def test_more_shapes_of_the_gather_forward_with_a_factoriser(oracle32, n, ft_out):
    test_shapes_of_the_gather_forward_with_a_factoriser(oracle32, n, ft_out, False, (1,))
