"""The schedule of the row-per-warp Jacobi sweeps (csrc/yb_jacobi.cu), restated: every pair of
super-vectors meets exactly once a sweep, and the counters that items wait for order every
super-vector's items without a deadlock."""
import pytest


def _place(ns, level, pi):
    for g in range(1 << level):
        first, n, cnt = 0, ns, 1
        for bit in range(level - 1, -1, -1):
            h2 = n >> 1
            h1 = n - h2
            if (g >> bit) & 1:
                cnt, first, n = cnt + h2, first + h2, h1
            else:
                cnt, n = cnt + (h1 if h2 else 0), h2
        if pi < n >> 1:
            return first, n, pi, cnt
        pi -= n >> 1
    return None


@pytest.mark.parametrize('ns', list(range(1, 41)) + [54, 81, 108, 162, 328])
def test_every_pair_once_and_no_deadlock(ns):
    items = (ns + 1) // 2
    levels = (ns - 1).bit_length()
    queue = []  # per item: its steps (S, T, count S needs at a level's start, count T needs, last round)
    for pi in range(items):
        steps = []
        for level in range(levels):
            pl = _place(ns, level, pi)
            if pl is None or pl[1] < 2:
                continue
            first, n, i, cnt = pl
            h2 = n >> 1
            h1 = n - h2
            for r in range(h1):
                j = (i + r) % h1
                seen = min(j, h2 - 1) - i if i <= j else j + 1 + h2 - 1 - i
                steps.append((first + i, first + h2 + j, cnt if r == 0 else None, cnt + seen, cnt + h1 if r == h1 - 1 else None))
        queue.append(steps)
    ver, pairs, pos = [1] * ns, set(), [0] * items
    while any(p < len(q) for p, q in zip(pos, queue)):
        moved = False
        for pi, q in enumerate(queue):
            if pos[pi] == len(q):
                continue
            s, t, need_s, need_t, end_s = q[pos[pi]]
            assert ver[t] <= need_t
            if ver[t] < need_t or (need_s is not None and ver[s] < need_s):
                continue
            assert need_s is None or ver[s] == need_s
            assert frozenset((s, t)) not in pairs and s != t
            pairs.add(frozenset((s, t)))
            ver[t] += 1
            if end_s is not None:
                ver[s] = end_s
            pos[pi] += 1
            moved = True
        assert moved, "deadlock"
    assert len(pairs) == ns * (ns - 1) // 2
    assert max(ver) < 8192


def test_row_sweeps_arguments_are_rejected_on_host():
    N = pytest.importorskip('yastn_gb300._native')
    lib = N.lib()
    nul = None
    words = lib.yb_svd_row_aux(2, 5)
    assert words > 0 and lib.yb_svd_row_limit(64, 7) == 0
    assert lib.yb_svd_row_sweeps(nul, nul, 0, nul, 0, 32, N.YB_F64, 1, 0.0, 8, nul, nul, 0, nul) == N.YB_OK
    assert lib.yb_svd_row_sweeps(nul, nul, 2, nul, 5, 32, N.YB_F64, 1, 0.0, 8, nul, nul, words, nul) == N.YB_ERR_INVALID
    some = 4096  # never dereferenced: the checks below fail first
    for prec, dtype, lmax, w, want in ((16, N.YB_F64, 8, words, N.YB_ERR_INVALID), (32, 5, 8, words, N.YB_ERR_INVALID),
                                       (64, N.YB_F64, 0, words, N.YB_ERR_INVALID),
                                       (64, N.YB_F64, 8, words - 1, N.YB_ERR_INVALID),
                                       (64, N.YB_F64, lib.yb_svd_row_limit(64, N.YB_F64) + 1, words, N.YB_ERR_TOO_LARGE)):
        assert lib.yb_svd_row_sweeps(some, some, 2, some, 5, prec, dtype, 1, 0.0, lmax, some, some, w, nul) == want
