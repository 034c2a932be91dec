"""Box copies (P._box_task, csrc/yb_copy.cu): the records restated with NumPy copy every element of
a permuted block once, for random ranks, extents, orders and element sizes; on the GPU the kernel
does the same, bit for bit, alone and through transpose_and_merge."""
import numpy as np
import pytest

from yastn_gb300 import _plans as P


def _run_record(rec, table, src, dst, written, most):
    nd = int(rec[0])
    t, ss, ds, sm, byte, perm = (rec[o:o + nd] for o in (8, 16, 24, 32, 48, 56))
    assert int(rec[1]) == np.prod(t) <= most and t.max() <= 255
    assert sorted(perm) == list(range(nd))
    for d in range(nd):  # the division constants
        magic, shift, size = int(rec[40 + d]) & 0xffffffff, int(rec[40 + d]) >> 32, int(t[d])
        for x in (0, 1, size - 1, size, 2047):
            assert (((x * magic) >> 32) + x) >> shift == x // size
    grid = np.indices([int(x) for x in t]).reshape(nd, -1)
    at = (grid * sm[:, None]).sum(0)
    assert np.array_equal(np.sort(at), np.arange(at.size)), "not the source order"
    for so, do, clip in table:
        ok = np.ones(grid.shape[1], dtype=bool)
        for d in range(nd):
            if byte[d] >= 0:
                ok &= grid[d] < ((int(clip) >> (8 * int(byte[d]))) & 255)
        s = (so + (grid * ss[:, None]).sum(0))[ok]
        d = (do + (grid * ds[:, None]).sum(0))[ok]
        dst[d] = src[s]
        written[d] += 1


def _random_task(rng, rank, most):
    sizes = [int(rng.integers(2, most)) for _ in range(rank)]
    order = rng.permutation(rank)
    st = P.row_major_strides(sizes)
    dims = [sizes[o] for o in order]
    return sizes, order, dims, [st[o] for o in order], P.row_major_strides(dims)


@pytest.mark.parametrize('elem', [1, 2, 4, 8, 16])
@pytest.mark.parametrize('rank', [2, 3, 4, 5, 6, 7])
def test_records_copy_every_element_once(rank, elem):
    rng = np.random.default_rng(10 * rank + elem)
    done = 0
    for _ in range(6):
        sizes, order, dims, ss, ds = _random_task(rng, rank, {2: 90, 3: 24, 4: 11, 5: 8, 6: 5, 7: 4}[rank])
        n = int(np.prod(sizes))
        src = rng.integers(0, 1 << 30, n + 3)
        dst, written = np.zeros(n + 5, dtype=src.dtype), np.zeros(n + 5, dtype=int)
        d, s, e = P._collapse(dims, ss, ds)
        box = P._box_task(3, 5, d, s, e, elem)
        if box is None:  # more than four dims that do not divide evenly
            continue
        rec, table = box
        done += 1
        _run_record(rec, table, src, dst, written, 2048 if elem < 16 else 1024)
        assert np.array_equal(dst[5:], src[3:].reshape(sizes).transpose(order).ravel())
        assert np.all(written[5:] == 1) and np.all(written[:5] == 0)
    assert done >= 2


def test_boxes_and_the_rest_cover_a_plan(monkeypatch):
    rng = np.random.default_rng(0)
    tasks, so = [], 0
    for shape, order in (((13, 7, 12, 5), (3, 1, 0, 2)), ((64, 96), (1, 0)), ((40, 3), (0, 1)), ((9, 3, 8, 3), (2, 0, 1, 3))):
        st = P.row_major_strides(shape)
        dims = [shape[o] for o in order]
        tasks.append((so, so, dims, [st[o] for o in order], P.row_major_strides(dims)))
        so += int(np.prod(shape))
    monkeypatch.setattr(P, 'BOX_MIN_MIXED', 0)
    plan = P.CopyPlan(tasks, so, so)
    rest, items, recs, boxes, box_items = plan.packed_with_boxes(True, 8)
    assert len(recs) >= 1 and len(rest) >= 2
    import plan_interp as PI
    src = rng.normal(size=so)
    want, got = np.zeros(so), np.zeros(so)
    PI.run_copy(*plan.packed(True), src, want)
    PI.run_copy(rest, items, src, got)
    for ti, first, n, _ in box_items:
        _run_record(recs[ti], boxes[first:first + n], src, got, np.zeros(so, dtype=int), 2048)
    assert np.array_equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize('dtype', ['float64', 'complex128', 'float32', 'int16', 'bool'])
def test_kernel_matches_numpy(dtype, cuda_device):
    import torch
    from yastn_gb300 import ops
    rng = np.random.default_rng(4)
    for rank in (2, 3, 4, 5, 6, 7):
        for most in ({2: 90, 3: 24, 4: 13, 5: 9, 6: 5, 7: 4}[rank], 3):
            sizes, order, dims, ss, ds = _random_task(rng, rank, max(most, 3))
            n = int(np.prod(sizes))
            x = rng.integers(0, 200, n)
            x = (x + 1j * x[::-1]) if dtype == 'complex128' else x
            x = x.astype(dtype)
            meta = (((0, n), tuple(dims), (0, n), tuple(sizes)),)
            got = ops.transpose(torch.from_numpy(x).cuda(), tuple(int(o) for o in order), meta).cpu().numpy()
            assert np.array_equal(got, x.reshape(sizes).transpose(order).ravel())
            back = ops.transpose_backward(torch.from_numpy(got).cuda(), tuple(int(o) for o in order), meta)
            assert np.array_equal(back.cpu().numpy(), x)


@pytest.mark.gpu
@pytest.mark.parametrize('shape,order', [((28, 28, 28, 28), (3, 2, 1, 0)), ((48, 5, 50), (2, 1, 0)),
                                         ((28, 30, 29, 31), (3, 1, 2, 0))])
def test_large_copies_with_fuller_tiles_go_by_boxes(shape, order, cuda_device):
    """Copies of BOX_LARGE elements take boxes where the tiles would be half full and more; the same
    blocks in a smaller copy keep the tiles. Both are exact, forward and inverse."""
    import torch
    from yastn_gb300 import ops
    n1 = int(np.prod(shape))
    strides = P.row_major_strides(shape)
    dims = [shape[o] for o in order]
    for count, boxes in ((P.BOX_LARGE // n1 + 1, True), (2, False)):
        tasks = [(i * n1, i * n1, dims, [strides[o] for o in order], P.row_major_strides(dims)) for i in range(count)]
        plan = P.CopyPlan(tasks, count * n1, count * n1)
        assert bool(len(plan.packed_with_boxes(False, 8)[2])) == boxes
        x = torch.arange(count * n1, dtype=torch.float64, device='cuda')
        y, z = torch.empty_like(x), torch.empty_like(x)
        ops.run_copy(plan, x, y)
        assert torch.equal(y.view(count, *dims), x.view(count, *shape).permute(0, *(o + 1 for o in order)))
        ops.run_copy(plan.swapped(count * n1), y, z)
        assert torch.equal(z, x)
