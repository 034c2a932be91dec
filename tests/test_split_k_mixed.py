"""Plans that mix ordinary outputs (32 x 32 tiles with K chunks) with skinny ones of long K: both keep
their K chunks, whatever stands beside them. On the CPU the K of the launched tiles and the values of the
skinny part's records; on the GPU the product and its adjoints against the oracle."""
import numpy as np
import pytest

import plan_interp as PI
from oracle import backend_oracle as oracle
from yastn_gb300 import _plans as P

# (m, K, n): a U(1) product whose y leg is cut to 40 / 12 / 12 / 4 / 4; one skinny output beside a small or
# a dense one
MIXES = [[(200, 5000, 40), (200, 5000, 12), (200, 5000, 12), (200, 5000, 4), (200, 5000, 4)],
         [(64, 64, 64), (300, 50000, 12)],
         [(40, 30, 40), (2, 30000, 300)],
         [(3, 3000, 2000), (100, 1500, 100)]]


def _meta(shapes):
    meta, oa, ob, oc = [], 0, 0, 0
    for m, k, n in shapes:
        meta.append(((oc, oc + m * n), (m, n), (oa, oa + m * k), (m, k), (ob, ob + k * n), (k, n)))
        oa += m * k; ob += k * n; oc += m * n
    return tuple(meta), oa, ob, oc


def _tile_ks(p):
    return [int(p.terms[int(p.outs[t[0]][4]):int(p.outs[t[0]][5]), 2].sum()) for t in p.tiles]


@pytest.mark.parametrize('shapes', MIXES)
def test_no_launched_tile_has_a_long_k(shapes):
    meta, oa, ob, oc = _meta(shapes)
    f = P.fine_gemm(P.dot_plan(meta))
    assert f is not None
    ks = _tile_ks(f)
    if f.rest is not None:
        assert P.fine_gemm(f.rest) is None
        ks += _tile_ks(f.rest) + (_tile_ks(f.rest.split) if f.rest.split is not None else [])
    assert max(ks) <= 512
    # every output is written once: by fine tiles, their reduction, or the rest
    got = [int(o[0]) for o in f.outs if not o[6]] + [int(r[0]) for r in f.red]
    if f.rest is not None:
        got += [int(o[0]) for o in f.rest.outs]
        got += [int(r[0]) for r in f.rest.split.red] if f.rest.split is not None else []
    assert sorted(got) == [sl[0] for sl, *_ in meta]
    if f.rest is not None:
        rng = np.random.default_rng(2)
        A, B = rng.normal(size=oa), rng.normal(size=ob)
        out, ref = PI.run_gemm(f.rest, A, B, np.zeros(oc)), oracle.dot(A, B, meta, oc)
        mine = np.zeros(oc, dtype=bool)
        for (lo, hi), (m, n), *_ in meta:
            mine[lo:hi] = lo in {o[0] for o in f.rest.out_list}
        assert np.abs(out - ref)[mine].max() <= 1e-12 * np.abs(ref).max() * np.sqrt(max(k for _, k, _ in shapes))


def test_records_are_built_where_they_are_used():
    """A plan that runs on fine tiles does not build the records of the other kernels."""
    plan = P.dot_plan(_meta([(70, 50, 70), (33, 80, 65)])[0])
    assert P.fine_gemm(plan) is not None
    assert not {'outs', 'terms', 'tiles', 'split'} & set(plan.__dict__)
    assert len(plan.tiles) == 4 + 2 and plan.split is None
    assert not P._pack_gemm([]).has_work() and P._pack_gemm([(0, 2, 2, 2, [])]).has_work()


@pytest.mark.gpu
@pytest.mark.parametrize('cplx', [False, True])
@pytest.mark.parametrize('shapes', MIXES)
def test_mixed_products(shapes, cplx, cuda_device):
    import torch
    from yastn_gb300 import ops
    meta, oa, ob, oc = _meta(shapes)
    rng = np.random.default_rng(5)
    A, B, C = (rng.normal(size=n) + (1j * rng.normal(size=n) if cplx else 0) for n in (oa, ob, oc))
    a, b, c = (torch.from_numpy(x).cuda() for x in (A, B, C))
    got = ops.dot(a, b, meta, oc).cpu().numpy()
    K = max(k for _, k, _ in shapes)
    mag = oracle.dot(np.abs(A), np.abs(B), meta, oc)
    # any order of summation: K eps |A| |B| (complex: four products)
    assert np.all(np.abs(got - oracle.dot(A, B, meta, oc)) <= 4 * (K + 3) * 2.0 ** -53 * mag)
    Ab, Bb = (x.cpu().numpy() for x in ops.dot_backward(c, a, b, meta))
    Ar, Br = oracle.dot_backward(C, A, B, meta)
    Am, Bm = oracle.dot_backward(np.abs(C), np.abs(A), np.abs(B), meta)
    assert np.all(np.abs(Ab - Ar) <= 4 * (K + 3) * 2.0 ** -53 * Am)
    assert np.all(np.abs(Bb - Br) <= 4 * (K + 3) * 2.0 ** -53 * Bm)
