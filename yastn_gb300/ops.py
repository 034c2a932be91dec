"""Device operations of the hot path: torch tensors in, C ABI calls, torch tensors out.

Every function here launches the hand-written sm_103a kernels of
``libyastn_gb300.so`` on torch's current CUDA stream. Inputs must be contiguous 1-D
CUDA tensors of dtype float64 or complex128; anything else raises (there is no
fallback path).
"""
import ctypes
import weakref

import numpy as np
import torch

from . import _native as N
from . import _plans as P

_SUPPORTED = (torch.float64, torch.complex128)
MAX_SWEEPS = 64


def _vp(x):
    return ctypes.c_void_p(x)


def _ptr(t):
    if t.is_conj() or t.is_neg():  # a lazy view: its memory is not what the kernels would read
        raise ValueError("yastn_gb300: a conjugate/negative view reached a kernel unresolved")
    return t.data_ptr()


def _plain(t):
    """t with torch's lazy conjugate / negative flags resolved, contiguous."""
    if t.is_conj():
        t = t.resolve_conj()
    if t.is_neg():
        t = t.resolve_neg()
    return t.contiguous()


def _stream():
    """The current device's current stream, as torch.cuda.current_stream().cuda_stream (which wraps
    it in a Stream object: 3 us on the host against 0.2)."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def _dtype_code(dtype):
    if dtype == torch.float64:
        return N.YB_F64
    if dtype == torch.complex128:
        return N.YB_C128
    raise NotImplementedError(f"yastn_gb300 kernels support float64 and complex128, got {dtype}")


_COPY_UNITS = (1, 2, 4, 8, 16)  # element sizes the block copy and mask kernels move as raw units
_NARROW = {torch.float32: torch.float64, torch.complex64: torch.complex128}


def _check(t, name='data', any_dtype=False):
    """A CUDA tensor, flat, contiguous, with lazy conjugate / negative views resolved. The
    arithmetic kernels take float64 and complex128; the copies (``any_dtype``) any element of
    1, 2, 4, 8 or 16 bytes (bool masks, float32, complex64, ...)."""
    if not isinstance(t, torch.Tensor) or not t.is_cuda:
        raise TypeError(f"{name} must be a CUDA tensor (yastn_gb300 has no CPU path)")
    if any_dtype:
        if t.element_size() not in _COPY_UNITS:
            raise NotImplementedError(f"yastn_gb300 copies move 1-16 byte elements, got {t.dtype}")
    elif t.dtype not in _SUPPORTED:
        raise NotImplementedError(f"yastn_gb300 kernels support float64 and complex128, got {t.dtype}")
    # torch's lazy conjugate / negative views (conj(), neg() of a conjugate) keep the memory
    # unchanged and only set a flag that the kernels, reading raw memory, would not see
    if t.is_conj():
        t = t.resolve_conj()
    if t.is_neg():
        t = t.resolve_neg()
    if t.dim() != 1 or not t.is_contiguous():
        t = t.reshape(-1).contiguous()
    return t


def _dev(plan, key, arrays, device):
    """Device copies of a plan's packed arrays, cached on the plan per device."""
    k = (key, str(device))
    d = plan._dev.get(k)
    if d is None:
        d = tuple(torch.from_numpy(np.ascontiguousarray(a)).to(device) for a in arrays)
        plan._dev[k] = d
    return d


# ----------------------------------------------------------------------------- family (a)

def run_copy(plan, src, dst):
    """Run a CopyPlan from ``src`` into ``dst`` (both 1-D, same dtype)."""
    sp, dp, elem = _ptr(src), _ptr(dst), src.element_size()
    vec_ok = src.dtype == torch.float64 and (sp | dp) % 16 == 0
    key = ('copy', vec_ok, elem, src.device)
    launches = plan._dev.get(key)
    if launches is None:
        launches = plan._dev[key] = _copy_launches(plan, vec_ok, elem, src.device)
    st = _stream()
    for name, args, _ in launches:
        N.call(name, sp, dp, elem, *args, st)
    return dst


def _copy_launches(plan, vec_ok, elem, device):
    """(entry point, arguments between the element size and the stream, the device arrays they point
    into) of a CopyPlan's launches; kept on the plan."""
    tasks, items, box_tasks, boxes, box_items = plan.packed_with_boxes(vec_ok, elem)
    out = []
    if len(items):
        d = _dev(plan, ('records', vec_ok, elem), (tasks, items), device)
        out.append(('yb_block_copy', (_ptr(d[0]), len(tasks), _ptr(d[1]), len(items)), d))
    if len(box_items):
        d = _dev(plan, ('boxes', vec_ok, elem), (box_tasks, boxes, box_items), device)
        out.append(('yb_box_copy', (_ptr(d[0]), _ptr(d[1]), _ptr(d[2]), len(box_items)), d))
    return out


def map_gather(src, gmap, conj=False):
    """One composed copy: ``out[i] = conj?(sign * src[|gmap[i]| - 1])`` (0 where gmap[i] == 0),
    ``gmap`` an int32 CUDA tensor of source indices + 1 with the sign of a block negation
    (``yb_map_gather``)."""
    src = _check(src, 'src')
    if gmap.dtype != torch.int32 or not gmap.is_cuda or gmap.dim() != 1 or not gmap.is_contiguous():
        raise TypeError("gmap must be a contiguous 1-D int32 CUDA tensor")
    if src.numel() == 0:  # nothing to gather: every entry of a valid map is 0 (zero fill)
        return torch.zeros(gmap.numel(), dtype=src.dtype, device=src.device)
    out = torch.empty(gmap.numel(), dtype=src.dtype, device=src.device)
    if out.numel():
        N.call('yb_map_gather', _ptr(src), _ptr(out), _dtype_code(src.dtype), _ptr(gmap), gmap.numel(),
               int(bool(conj) and src.is_complex()), _stream())
    return out


# ----------------------------------------------------------------------------- constant operands

_HOLD = {'depth': 0, 'capturing': None, 'merge': {}, 'split': {}}


class hold_constant_operands:
    """Scope in which the merges and digit splits of unchanged operands are computed once.

    An iterative solver applies one operator many times: in YASTN's ``eigs`` the effective
    Hamiltonian's environment tensors, and their merged sector matrices, are the same tensor
    objects in every call. Inside this scope a merge of the same source tensor object (its
    version counter unchanged) by the same plan returns its earlier output while that output
    is unmodified (its version counter unchanged), and an emulated dot reuses the BF16 digit
    planes of an operand object it split before; tensors that require grad are never held.
    Entries refer to their sources weakly (an entry ends with its source, so the temporaries
    of each operator application are not kept), end with the outermost scope, and are
    dropped when the stream capture state changes: entries made during a CUDA-graph capture
    are used within that capture only, whose replays recompute them in order."""

    def __enter__(self):
        _HOLD['depth'] += 1
        return self

    def __exit__(self, *exc):
        _HOLD['depth'] -= 1
        if _HOLD['depth'] == 0:
            _HOLD['merge'].clear()
            _HOLD['split'].clear()
        return False


def _held(kind, key, src):
    """(cache, key) for ``src`` in the current scope, or None (no scope, or src requires grad)."""
    if _HOLD['depth'] == 0 or src.requires_grad:
        return None
    cap = torch.cuda.is_current_stream_capturing()
    if _HOLD['capturing'] != cap:
        _HOLD['merge'].clear()
        _HOLD['split'].clear()
        _HOLD['capturing'] = cap
    return _HOLD[kind], key + (id(src),)


def _hit(held, src):
    """The held payload of src, if its entry is current."""
    if held is None:
        return None
    cache, key = held
    e = cache.get(key)
    if e is None or e[0]() is not src or e[1] != src._version:
        return None
    payload, out_version = e[2], e[3]
    if out_version is not None and payload._version != out_version:
        return None
    return payload


def _store(held, src, payload, track_output=False):
    cache, key = held

    def drop(ref, cache=cache, key=key):
        e = cache.get(key)
        if e is not None and e[0] is ref:
            del cache[key]
    cache[key] = (weakref.ref(src, drop), src._version, payload, payload._version if track_output else None)


def merge(data, order, meta_new, meta_mrg, Dsize):
    """transpose_and_merge: fused blocks, zero where no source block lands (inside
    ``hold_constant_operands``, the earlier output for an unchanged source)."""
    data = _check(data, any_dtype=True)
    plan = P.merge_plan(order, meta_new, meta_mrg, Dsize)
    held = _held('merge', (id(plan),), data)
    out = _hit(held, data)
    if out is not None:
        return out
    out = (torch.empty if plan.full else torch.zeros)(Dsize, dtype=data.dtype, device=data.device)
    run_copy(plan, data, out)
    if held is not None:
        _store(held, data, out, track_output=True)
    return out


def merge_backward(data_b, order, meta_new, meta_mrg, Dsize, D_source):
    data_b = _check(data_b, any_dtype=True)
    plan = P.merge_plan(order, meta_new, meta_mrg, Dsize)
    inv = P.CACHE.get((order, meta_new, meta_mrg), ('merge_bwd', Dsize, D_source), lambda: plan.swapped(D_source))
    out = (torch.empty if inv.full else torch.zeros)(D_source, dtype=data_b.dtype, device=data_b.device)
    return run_copy(inv, data_b, out)


def unmerge(data, meta):
    data = _check(data, any_dtype=True)
    plan = P.unmerge_plan(meta, data.numel())
    out = (torch.empty if plan.full else torch.zeros)(data.numel(), dtype=data.dtype, device=data.device)
    return run_copy(plan, data, out)


def unmerge_backward(data_b, meta, fwd_size):
    data_b = _check(data_b, any_dtype=True)
    plan = P.unmerge_plan(meta, fwd_size)
    inv = P.CACHE.get((meta,), ('unmerge_bwd', fwd_size), lambda: plan.swapped(fwd_size))
    out = (torch.empty if inv.full else torch.zeros)(fwd_size, dtype=data_b.dtype, device=data_b.device)
    return run_copy(inv, data_b, out)


def transpose(data, axes, meta_transpose):
    data = _check(data, any_dtype=True)
    plan = P.transpose_plan(axes, meta_transpose, data.numel())
    out = (torch.empty if plan.full else torch.zeros)(data.numel(), dtype=data.dtype, device=data.device)
    return run_copy(plan, data, out)


def transpose_backward(data_b, axes, meta_transpose):
    data_b = _check(data_b, any_dtype=True)
    plan = P.transpose_plan(axes, meta_transpose, data_b.numel())
    inv = P.CACHE.get((axes, meta_transpose), ('transpose_bwd', data_b.numel()), lambda: plan.swapped(data_b.numel()))
    out = (torch.empty if inv.full else torch.zeros)(data_b.numel(), dtype=data_b.dtype, device=data_b.device)
    return run_copy(inv, data_b, out)


# ----------------------------------------------------------------------------- family (b)

def run_gemm(plan, a, b, c, alpha=1.0, beta=0.0, stream=None, keep=None):
    """C_o = alpha sum op(A) op(B) + beta C_o of a GemmPlan on the current stream, or on ``stream`` (a
    raw handle): ``keep`` then receives the workspace, to be held until that stream has been waited
    for."""
    code = _dtype_code(c.dtype)
    alpha, beta = float(alpha), float(beta)
    key = ('gemm', a.device)
    got = plan._dev.get(key)
    if got is None:
        got = plan._dev[key] = _gemm_launches(plan, a.device)
    rest, fine, direct, split, _ = got
    st = _stream() if stream is None else stream
    if rest is not None:
        run_gemm(rest, a, b, c, alpha, beta, st, keep)
    if fine:
        args, red, size = fine
        ws = torch.empty(size, dtype=c.dtype, device=c.device) if size else None
        wp = _ptr(ws) if size else 0
        N.call('yb_grouped_gemm_fine', _ptr(a), _ptr(b), _ptr(c), wp, code, *args, alpha, beta, st)
        if size:
            if keep is not None:
                keep.append(ws)
            N.call('yb_gemm_reduce', _ptr(c), wp, code, *red, alpha, beta, st)
    if direct:
        N.call(direct[0], _ptr(a), _ptr(b), _ptr(c), code, *direct[1], alpha, beta, st)
    if split:
        # split-K: chunk products into a workspace, then the ordered sum into C
        parts, red, size = split
        ws = torch.empty(size, dtype=c.dtype, device=c.device)
        if keep is not None:
            keep.append(ws)
        N.call('yb_grouped_gemm', _ptr(a), _ptr(b), _ptr(ws), code, *parts, 1.0, 0.0, st)
        N.call('yb_gemm_reduce', _ptr(c), _ptr(ws), code, *red, alpha, beta, st)
    return c


def _gemm_launches(plan, device):
    """The launches of a GemmPlan with the addresses of its device arrays (kept on the plan with
    them): the plan of the outputs beside the fine tiles, the fine tiles' arguments, their reduction and
    workspace; or (entry point, records and tiles) and the split-K parts; the arrays. None where
    there is none of it."""
    direct = split = None
    keep = []
    f = P.fine_gemm(plan)
    if f is not None:
        d = _dev(f, 'fine', (f.outs, f.terms, f.tiles, f.red, f.tasks), device)
        return f.rest, ((_ptr(d[0]), _ptr(d[1]), _ptr(d[2]), len(f.tiles)), (_ptr(d[3]), _ptr(d[4]), len(f.tasks)),
                        f.ws), None, None, [d]
    if len(plan.tiles):
        d = _dev(plan, 'gemm', (plan.outs, plan.terms, plan.tiles), device)
        direct = ('yb_grouped_gemm_short' if plan.all_short else 'yb_grouped_gemm',
                  (_ptr(d[0]), _ptr(d[1]), _ptr(d[2]), len(plan.tiles)))
        keep.append(d)
    sp = plan.split
    if sp is not None:
        d = _dev(plan, 'gemm_split', (sp.outs, sp.terms, sp.tiles, sp.red, sp.tasks), device)
        split = ((_ptr(d[0]), _ptr(d[1]), _ptr(d[2]), len(sp.tiles)), (_ptr(d[3]), _ptr(d[4]), len(sp.tasks)), sp.ws)
        keep.append(d)
    return None, None, direct, split, keep


def promote(A, B):
    dtype = torch.promote_types(A.dtype, B.dtype)
    return (A if A.dtype == dtype else A.to(dtype)), (B if B.dtype == dtype else B.to(dtype))


def _narrow_inputs(*ts):
    """True when a float32 / complex64 operand is present: the product then runs in float64 /
    complex128 on the same kernels and the result is rounded to the promoted input dtype (at
    least the accuracy of a single-precision product)."""
    return any(isinstance(t, torch.Tensor) and t.dtype in _NARROW for t in ts)


def _wide(t):
    return t.to(_NARROW[t.dtype]) if t.dtype in _NARROW else t


def dot(A, B, meta_dot, Dsize):
    if _narrow_inputs(A, B):
        return dot(_wide(A), _wide(B), meta_dot, Dsize).to(torch.promote_types(A.dtype, B.dtype))
    A, B = promote(_check(A, 'A'), _check(B, 'B'))
    plan = P.dot_plan(meta_dot)
    # every element is written by one sector when the sectors tile the output
    out = (torch.empty if plan.covered == Dsize else torch.zeros)(Dsize, dtype=A.dtype, device=A.device)
    return run_gemm(plan, A, B, out)


OZAKI_SLICES = 8  # 57 bits per operand: FP64-grade products


OZAKI_TC = [None]  # emulated GEMM kernel: None = autotuned per dot; False = mma.sync; 64 (or True) / 32 =
                  # tcgen05/TMEM with 128 x 64 / 128 x 32 output tiles
OZAKI_AUTOTUNE = [True]  # False: choose by the tile-padding estimate without timing


def dot_ozaki(A, B, meta_dot, Dsize, slices=OZAKI_SLICES):
    """``dot`` with the FP64 sector GEMMs emulated on BF16 tensor cores (split operands).

    float64 or complex128 operands (a complex product is two real products with doubled
    K). Each A row / B column is split into ``slices`` BF16 digit
    planes (scratch of 2 * slices bytes per operand element); all slice-pair products
    with digit-weight sum below ``slices`` are accumulated exactly in FP32 per K-chunk and
    combined in FP64. ``slices=8`` reproduces the FP64 product to its rounding level.
    """
    if _narrow_inputs(A, B):
        return dot_ozaki(_wide(A), _wide(B), meta_dot, Dsize, slices).to(torch.promote_types(A.dtype, B.dtype))
    A, B = promote(_check(A, 'A'), _check(B, 'B'))
    plan = P.ozaki_dot_plan(meta_dot, slices, A.is_complex())
    out = (torch.empty if plan.covered == Dsize else torch.zeros)(Dsize, dtype=A.dtype, device=A.device)
    if len(plan.tiles) == 0:
        return run_gemm(plan.native, A, B, out)  # short (K < 16) and skinny sectors: native FP64
    if OZAKI_TC[0] is not None:
        tc = OZAKI_TC[0]
    else:
        if getattr(plan, 'tuned_tc', None) is None:
            plan.tuned_tc = _autotune_ozaki(plan, A, B, out, slices)
        tc = plan.tuned_tc
    # the native sectors (disjoint outputs) run on a second stream beside the split and the
    # emulated GEMM, and the current stream waits for them (a fork and join inside a CUDA graph)
    if not plan.native.has_work():
        _ozaki_run(plan, A, B, out, slices, tc)
        return out
    main, side, keep = torch.cuda.current_stream(A.device), _side_stream(A.device), []
    side.wait_stream(main)
    try:
        run_gemm(plan.native, A, B, out, stream=side.cuda_stream, keep=keep)
        _ozaki_run(plan, A, B, out, slices, tc)
    finally:
        # also where a launch or an allocation failed: the memory of out and of the workspaces in keep
        # may be given to later work of the main stream
        main.wait_stream(side)
        del keep
    return out


_SIDE = {}


def _side_stream(device):
    """The second stream of a device (created once; independent work of one call runs on it)."""
    s = _SIDE.get(device.index)
    if s is None:
        s = _SIDE[device.index] = torch.cuda.Stream(device=device)
    return s


def _autotune_ozaki(plan, A, B, out, slices):
    """Kernel choice for one dot metadata: the mma.sync kernel and the tcgen05 kernel with
    128 x 64 or 128 x 32 tiles produce the same bits, so the first call times the three (CUDA
    events; skipped during stream capture, where the tile-padding estimate decides) and the
    plan keeps the fastest. Inside ``hold_constant_operands`` both operands are split every time,
    as in a first application."""
    if not OZAKI_AUTOTUNE[0] or torch.cuda.is_current_stream_capturing():
        return plan.prefer_tc
    times = {}
    for tc in (False, 64, 32, False, 64, 32):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda._sleep(2_000_000)  # hold the stream while the host enqueues: time the GPU, not the host
        e0.record()
        _ozaki_run(plan, A, B, out, slices, tc, hold=False)
        e1.record()
        e1.synchronize()
        times[tc] = e0.elapsed_time(e1)  # the second (warm) measurement of each kernel is kept
    return min(times, key=times.get)


def _ozaki_run(plan, A, B, out, slices, tc, hold=True):
    """Both operands split by one yb_ozaki_split launch (B's blocks read by columns in
    place), then the emulated GEMM: tcgen05 (tile layout) or mma.sync (digit planes). Inside
    ``hold_constant_operands`` an operand split before, unchanged, keeps its digit planes and
    only the other operand is split (or neither)."""
    dev = A.device
    st = _stream()
    tile_n = 0 if not tc else (32 if tc == 32 else 64)
    key = ('ozaki', tile_n, dev)
    rec = plan._dev.get(key)
    if rec is None:
        rec = plan._dev[key] = _ozaki_arrays(plan, tile_n, dev)
    recs, groups_of, gemm, asz, bsz, _ = rec
    held_a = _held('split', (id(plan), 0, tile_n, slices), A) if hold else None
    held_b = _held('split', (id(plan), 1, tile_n, slices), B) if hold else None
    hit_a, hit_b = _hit(held_a, A), _hit(held_b, B)
    a_sl, a_ex = hit_a if hit_a else (torch.empty(asz, dtype=torch.bfloat16, device=dev),
                                      torch.empty(max(plan.a_exps, 1), dtype=torch.int32, device=dev))
    b_sl, b_ex = hit_b if hit_b else (torch.empty(bsz, dtype=torch.bfloat16, device=dev),
                                      torch.empty(max(plan.b_exps, 1), dtype=torch.int32, device=dev))
    # both operands, or only the one that is not held
    groups, n_groups = groups_of[(hit_a is None) + 2 * (hit_b is None)]
    pa, pae, pb, pbe = _ptr(a_sl), _ptr(a_ex), _ptr(b_sl), _ptr(b_ex)
    if n_groups:
        N.call('yb_ozaki_split', _ptr(A), _ptr(B), pa, pb, pae, pbe, recs, groups, n_groups, slices, st)
    if held_a is not None and hit_a is None:
        _store(held_a, A, (a_sl, a_ex))
    if held_b is not None and hit_b is None:
        _store(held_b, B, (b_sl, b_ex))
    N.call('yb_ozaki_gemm_tc' if tile_n else 'yb_ozaki_gemm', pa, pae, pb, pbe, _ptr(out), *gemm, slices, st)


def _ozaki_arrays(plan, tile_n, dev):
    """Addresses of an emulated dot's device arrays, kept on the plan with them: the split records,
    the split groups (none; of A; of B; of both) with their counts, the GEMM's arguments between
    the output and the slice count, and the digit planes' sizes."""
    if tile_n:
        # tiles grouped by CTA (one CTA per SM) with balanced work
        sfx = '_tc' if tile_n == 64 else '_tc32'
        tiles, offs = P.ozaki_tc_schedule(plan, _sm_count(dev), tile_n)
        sizes = getattr(plan, 'a_size' + sfx), getattr(plan, 'b_size' + sfx)
    else:
        sfx, tiles, offs = '', plan.tiles, np.zeros(1, dtype=np.int32)
        sizes = plan.a_size, plan.b_size
    ab = getattr(plan, 'split_groups' + sfx + '_ab')
    arrs = (getattr(plan, 'split_recs' + sfx), getattr(plan, 'split_groups' + sfx), ab[0], ab[1],
            getattr(plan, 'outs' + sfx), tiles, offs)
    d = _dev(plan, 'ozaki' + sfx, arrs, dev)
    groups = ((None, 0), (_ptr(d[2]), len(arrs[2])), (_ptr(d[3]), len(arrs[3])), (_ptr(d[1]), len(arrs[1])))
    gemm = (_ptr(d[4]), _ptr(d[5]), len(tiles)) + ((_ptr(d[6]), len(offs) - 1, tile_n) if tile_n else ())
    return _ptr(d[0]), groups, gemm, max(sizes[0], 1), max(sizes[1], 1), d


def run_emulated(eg, a, b, c):
    """The products of ``eg`` (P.EmulatedGemm) from the flat tensors a and b into c: one split
    launch, one GEMM launch, and a native FP64 launch for the short ones."""
    if eg.native.has_work():
        run_gemm(eg.native, a, b, c)
    if eg.n_tiles == 0:
        return c
    dev, st = c.device, _stream()
    tc = eg.tile_n
    if tc:
        tiles, offs = P.ozaki_tc_schedule(eg, _sm_count(dev), tc)
        arrs = (eg.recs, eg.groups, getattr(eg, 'outs_tc' if tc == 64 else 'outs_tc32'), tiles, offs)
    else:
        arrs = (eg.recs, eg.groups, eg.outs, eg.tiles)
    d = _dev(eg, 'emulated', arrs, dev)
    a_sl = torch.empty(max(eg.a_size, 1), dtype=torch.bfloat16, device=dev)
    b_sl = torch.empty(max(eg.b_size, 1), dtype=torch.bfloat16, device=dev)
    ex = torch.empty(eg.a_exps + eg.b_exps, dtype=torch.int32, device=dev)
    b_ex = ex[eg.a_exps:]
    N.call('yb_ozaki_split', _ptr(a), _ptr(b), _ptr(a_sl), _ptr(b_sl), _ptr(ex), _ptr(b_ex), _ptr(d[0]), _ptr(d[1]),
           len(eg.groups), eg.slices, st)
    if tc:
        N.call('yb_ozaki_gemm_tc', _ptr(a_sl), _ptr(ex), _ptr(b_sl), _ptr(b_ex), _ptr(c), _ptr(d[2]), _ptr(d[3]),
               eg.n_tiles, _ptr(d[4]), len(arrs[4]) - 1, tc, eg.slices, st)
    else:
        N.call('yb_ozaki_gemm', _ptr(a_sl), _ptr(ex), _ptr(b_sl), _ptr(b_ex), _ptr(c), _ptr(d[2]), _ptr(d[3]),
               eg.n_tiles, eg.slices, st)
    return c


def _run_flagged(guard, name, a, b, c, flags):
    """The products ``name`` of a P.SvdGuard (None: there are none) for the blocks with a flag."""
    if guard is None:
        return
    key = (name, c.device)
    args = guard._dev.get(key)
    if args is None:  # addresses of the records, kept with them
        g = guard.gemm[name]
        d = _dev(g, 'flagged', (g.outs, g.terms, g.tiles), c.device)
        args = guard._dev[key] = (_ptr(d[0]), _ptr(d[1]), _ptr(d[2]), len(g.tiles)), d
    if args[0][3]:
        N.call('yb_grouped_gemm_flagged', _ptr(a), _ptr(b), _ptr(c), _dtype_code(c.dtype), *args[0], _ptr(flags), _stream())


_SMS = {}


def _sm_count(device):
    n = _SMS.get(device.index)
    if n is None:
        n = _SMS[device.index] = torch.cuda.get_device_properties(device).multi_processor_count
    return n


def ozaki_device_error(reset=True):
    """Status word of the tcgen05 emulated GEMM (synchronises the current stream)."""
    import ctypes
    v = ctypes.c_int(0)
    N.call('yb_ozaki_device_error', ctypes.addressof(v), int(bool(reset)), _stream(), launches=0)
    return v.value


def dot_backward(C_b, A, B, meta_dot, need_a=True, need_b=True):
    if _narrow_inputs(C_b, A, B):
        A_b, B_b = dot_backward(_wide(C_b), _wide(A), _wide(B), meta_dot, need_a, need_b)
        return (None if A_b is None else A_b.to(A.dtype)), (None if B_b is None else B_b.to(B.dtype))
    A, B = promote(_check(A, 'A'), _check(B, 'B'))
    C_b = _check(C_b, 'C_b')
    if C_b.dtype != A.dtype:
        C_b = C_b.to(A.dtype)
    pa, pb = P.dot_backward_plans(meta_dot)
    A_b = B_b = None
    if need_a:
        A_b = run_gemm(pa, C_b, B, torch.zeros(A.numel(), dtype=A.dtype, device=A.device))
    if need_b:
        B_b = run_gemm(pb, A, C_b, torch.zeros(B.numel(), dtype=A.dtype, device=A.device))
    return A_b, B_b


def permute_blocks(data, reshape, order):
    """Blocks (sl, Di, Dl, Dr) of ``data`` permuted by ``order`` into consecutive (Dl, Dr)
    matrices; returns (buffer, offsets, plan)."""
    def build():
        tasks, offs, low = [], [], 0
        for sl, Di, Dl, Dr in reshape:
            sst = P.row_major_strides(Di)
            Dt = [Di[o] for o in order]
            tasks.append((sl[0], low, Dt, [sst[o] for o in order], P.row_major_strides(Dt)))
            offs.append(low)
            low += Dl * Dr
        return P.CopyPlan(tasks, low, low), tuple(offs)
    plan, offs = P.CACHE.get((reshape, order), ('permute_blocks',), build)
    buf = torch.empty(plan.size_dst, dtype=data.dtype, device=data.device)
    return run_copy(plan, data, buf), offs, plan


def transpose_dot_sum(A, B, meta_dot, Areshape, Breshape, Aorder, Border, Dsize):
    if _narrow_inputs(A, B):
        return transpose_dot_sum(_wide(A), _wide(B), meta_dot, Areshape, Breshape, Aorder, Border,
                                 Dsize).to(torch.promote_types(A.dtype, B.dtype))
    A, B = promote(_check(A, 'A'), _check(B, 'B'))
    Ap, Aoffs, _ = permute_blocks(A, Areshape, Aorder)
    Bp, Boffs, _ = permute_blocks(B, Breshape, Border)
    plan = P.tds_plan(meta_dot, Areshape, Breshape, Aoffs, Boffs)
    out = torch.zeros(Dsize, dtype=A.dtype, device=A.device)
    return run_gemm(plan, Ap, Bp, out)


def transpose_dot_sum_backward(C_b, A, B, meta_dot, Areshape, Breshape, Aorder, Border):
    if _narrow_inputs(C_b, A, B):
        A_b, B_b = transpose_dot_sum_backward(_wide(C_b), _wide(A), _wide(B), meta_dot, Areshape, Breshape, Aorder,
                                              Border)
        return A_b.to(A.dtype), B_b.to(B.dtype)
    A, B = promote(_check(A, 'A'), _check(B, 'B'))
    C_b = _check(C_b, 'C_b').to(A.dtype)
    Ap, Aoffs, pa_perm = permute_blocks(A, Areshape, Aorder)
    Bp, Boffs, pb_perm = permute_blocks(B, Breshape, Border)
    pa, pb = P.tds_backward_plans(meta_dot, Areshape, Breshape, Aoffs, Boffs)
    At_b = run_gemm(pa, C_b, Bp, torch.zeros(Ap.numel(), dtype=A.dtype, device=A.device))
    Bt_b = run_gemm(pb, Ap, C_b, torch.zeros(Bp.numel(), dtype=A.dtype, device=A.device))
    inv_a = P.CACHE.get((Areshape, Aorder), ('permute_blocks_bwd', A.numel()), lambda: pa_perm.swapped(A.numel()))
    inv_b = P.CACHE.get((Breshape, Border), ('permute_blocks_bwd', B.numel()), lambda: pb_perm.swapped(B.numel()))
    A_b = run_copy(inv_a, At_b, (torch.empty if inv_a.full else torch.zeros)(A.numel(), dtype=A.dtype, device=A.device))
    B_b = run_copy(inv_b, Bt_b, (torch.empty if inv_b.full else torch.zeros)(B.numel(), dtype=A.dtype, device=A.device))
    return A_b, B_b


# ----------------------------------------------------------------------------- family (c)

MAX_SWEEPS32 = 40
TOL_STOP32 = 1.0e-4   # FP32 phase ends after a sweep whose largest rotation |cos| is below this
TOL_STOP64 = 1.0e-8   # FP64 phase: idem; Jacobi converges quadratically (a sweep that starts at
                      # max |cos| c leaves ~c^2), so the residual after such a sweep is ~1e-16
TOL_STOP64_QR = 1.0e-7  # the same for the QR-preconditioned SVD (separated, graded rows: ~1e-14 left; for
                        # rows of nearly equal norm the kernels go on, see stops in yb_svd_common.cuh)
TOL_STOP64_EIGH = 1.0e-11  # eigh: the shifted block A + shift I (shift = ||A||_F + 1) has its singular
                           # values clustered around the shift, so a sweep that starts at |cos| c leaves
                           # ~c^2 shift / gap rather than c^2: 1e-8 left 1e-9 relative reconstruction
                           # errors on rank-deficient blocks, 1e-11 reaches the rounding level
INNER_SWEEPS32 = 1    # blocked FP32 phase: Jacobi sweeps among the rows of a super pair per visit
BLOCKED_FP32 = [True]  # FP32 phase on super-vectors in shared memory (False: one pair per warp)
BLOCKED_FP64 = [True]  # FP64 phase likewise, on 4-row super-vectors (False: one pair per warp)
ROWS_PER_SUPER = [None]  # super-vector height (None: largest of 16, 8, 4 that fits)
NS_STEPS = 2          # Newton-Schulz steps: non-orthogonality ~1e-6 -> 1e-12 -> ~eps
SVD_EMULATED = [True]  # FP64 products inside svd / eigh on the tensor cores (False: the native grouped GEMM)
MAX_COMPLETIONS = 64  # completion plans kept with an SvdPlan (a differentiated CTMRG step of 8 iterations has 28
                      # SVDs of one structure, each with its own counts, and runs them twice)
SVD_QR = [True]       # svd: Jacobi on the rows of R of a Householder QR (few FP64 sweeps on graded spectra)


SVD_STATE_REC = 6     # int64 words of per-block Jacobi state (yb_svd.cu)


def _svd_state_check(state, nb, phase, require_converged):
    st = state.cpu().numpy()
    R = SVD_STATE_REC
    if st[R * nb + 2] != 0:
        raise RuntimeError(f"yastn_gb300 svd: grid barrier timed out in the {phase} phase")
    conv = st[1:R * nb:R]
    if require_converged and not conv.all():
        raise torch.linalg.LinAlgError(f"yastn_gb300 svd: Jacobi did not converge ({phase} phase)")
    return st[2:R * nb:R]


def _row_sweeps(plan, precision, code):
    """True where the sweeps keep a row per warp (yb_svd_row_sweeps): rows of up to 2624 (FP32),
    1312 (FP64; half of each for complex data) elements, unless a super-vector height is forced.
    Longer rows do not fit a warp's registers: they take the shared-memory kernel."""
    return ROWS_PER_SUPER[0] is None and plan.lmax <= N.lib().yb_svd_row_limit(precision, code)


def _run_row_sweeps(plan, work, dblocks, dpairs, nb, precision, code, max_sweeps, tol, state):
    n_pairs = len(plan.pair_items)
    words = N.lib().yb_svd_row_aux(nb, n_pairs)
    aux = torch.empty(words, dtype=torch.int64, device=work.device)
    N.call('yb_svd_row_sweeps', _ptr(work), _ptr(dblocks), nb, _ptr(dpairs), n_pairs, precision, code, max_sweeps, tol,
           plan.lmax, _ptr(state), _ptr(aux), words, _stream())


def _jacobi(data, plan, U, S, V, mode, max_sweeps=MAX_SWEEPS):
    """Mixed-precision batched Jacobi of ``plan`` on ``data``; writes U, S (and Vh for mode 0)."""
    nb = len(plan.blocks)
    dev = data.device
    code = _dtype_code(data.dtype)
    cplx = code == N.YB_C128
    dblocks, dpairs = _dev(plan, 'svd', (plan.blocks, plan.pair_items), dev)
    w64 = torch.empty(plan.n64, dtype=torch.complex128 if cplx else torch.float64, device=dev)
    w32 = torch.empty(plan.n32, dtype=torch.complex64 if cplx else torch.float32, device=dev)
    # control words: [state][state after the FP32 phase][completion counts][QR flags][graded blocks], read
    # once at the end: the host never waits between the phases
    n_st, n_qr = SVD_STATE_REC * nb + 4, (nb + 4 * min(nb, 4096)) if plan.qr else 0
    ctl = torch.zeros(2 * n_st + 2 * nb + n_qr, dtype=torch.int64, device=dev)
    state, qctrl = ctl[:n_st], ctl[2 * n_st + nb:2 * n_st + nb + n_qr]
    n_small = ctl[2 * n_st:2 * n_st + nb] if mode == 0 else None
    aux = torch.empty(2 * nb, dtype=torch.float64, device=dev)  # [scale | shift]
    shift = aux[nb:] if mode != 0 else None
    sp = _vp(shift.data_ptr() if shift is not None else 0)
    st = _stream()
    if plan.qr:
        N.call('yb_svd_qr', _ptr(data), _ptr(w64), _ptr(w32), _ptr(dblocks), nb, code, _ptr(state), _ptr(aux[:nb]),
               _ptr(qctrl), qctrl.numel(), st, launches=4)
    else:
        N.call('yb_svd_init', _ptr(data), _ptr(w32), _ptr(dblocks), nb, code, _ptr(state), sp, _ptr(aux[:nb]), st,
               launches=2)
    if BLOCKED_FP32[0] and _row_sweeps(plan, 32, code):
        _run_row_sweeps(plan, w32, dblocks, dpairs, nb, 32, code, MAX_SWEEPS32, TOL_STOP32, state)
    elif plan.rows_per_super and BLOCKED_FP32[0]:
        (dsup,) = _dev(plan, 'svd_super', (plan.super_items,), dev)
        N.call('yb_svd_block_sweeps', _ptr(w32), _ptr(dblocks), nb, _ptr(dsup), len(plan.super_items),
               plan.super_rounds, plan.rows_per_super, 32, code, MAX_SWEEPS32, INNER_SWEEPS32, TOL_STOP32,
               plan.lmax, _ptr(state), st)
    else:
        N.call('yb_svd_sweeps', _ptr(w32), _ptr(dblocks), nb, _ptr(dpairs), len(plan.pair_items), plan.max_rounds,
               32, code, MAX_SWEEPS32, TOL_STOP32, _ptr(state), st)
    ctl[n_st:2 * n_st].copy_(state)
    N.call('yb_svd_widen', _ptr(w32), _ptr(w64), _ptr(dblocks), nb, code, _ptr(state), st)
    w0, t0, n0, ws = plan.w_range
    # The FP64 products of the block SVD run on the tensor cores (57-bit digits per row and column,
    # one rounding per 400 contracted indices; R's grading is taken out of X = W R first): their
    # errors are no larger than the DFMA kernel's, which the FP64 pipe bounds: 2.7 against 0.46 ms
    # for all products of two 432 x 432 blocks, 55 against 3.7 ms for two 1296 x 1296, 0.64 against
    # 0.10 ms in the eigh of five blocks up to 110. Short products (K < 16) stay native, the products with W
    # of a block graded by columns are formed again by the native kernel (yb_svd_graded: digits scaled per
    # row and column lose the small entries of its factors); the results of a block with a non-finite
    # entry, which digits cannot hold, are made NaN (yb_svd_poison).
    emu = guard = flags = None
    if SVD_EMULATED[0] and (plan.qr or mode != 0):
        emu = P.svd_emulated(plan, OZAKI_SLICES, cplx)
        guard = emu['guard']
        if guard is not None:
            flags = ctl[2 * n_st + nb + n_qr:]
            (at,) = _dev(guard, 'at', (guard.at,), dev)
            masks = torch.empty(guard.size, dtype=torch.int32, device=dev)
            N.call('yb_svd_graded', _ptr(w64), _ptr(dblocks), nb, code, P.OZAKI_MIN_DIM, _ptr(state), _ptr(at),
                   _ptr(masks), _ptr(flags), st, launches=3)
        for gram, ns in (('gram', 'ns'), ('gram2', 'ns2')):
            run_emulated(emu[gram], w64, w64, w64)
            _run_flagged(guard, gram, w64, w64, w64, flags)
            N.call('yb_svd_ns_prep', _ptr(w64), _ptr(dblocks), nb, code, ws, st)
            run_emulated(emu[ns], w64, w64, w64)
            _run_flagged(guard, ns, w64, w64, w64, flags)
    else:
        W, Wn = w64[w0:w0 + ws], w64[n0:n0 + ws]
        for _ in range(NS_STEPS):
            Wn.copy_(W)
            run_gemm(plan.gram, w64, w64, w64)
            run_gemm(plan.ns, w64, w64, w64, alpha=-0.5, beta=1.5)
            W.copy_(Wn)
    if plan.qr:
        if emu:
            N.call('yb_svd_scale_wr', _ptr(w64), _ptr(dblocks), nb, code, ws, P.OZAKI_MIN_DIM, _ptr(state), st, launches=3)
            run_emulated(emu['xr'], w64, w64, w64)  # X = W R = T Wn
            N.call('yb_svd_poison', _ptr(w64), 0, _ptr(dblocks), nb, code, _ptr(state), P.OZAKI_MIN_DIM, 0, st)
        else:
            run_gemm(plan.xform, w64, w64, w64)
    elif shift is not None:
        N.call('yb_svd_shift_prefill', _ptr(w64), _ptr(dblocks), nb, code, _ptr(shift), st)
        if emu:  # X = shift W + W A, W A by way of T (laid out like X: the blocks are square)
            run_emulated(emu['xa'], w64, data, w64)
            w64[:ws].add_(w64[t0:t0 + ws])
        else:
            run_gemm(plan.xform, w64, data, w64, beta=1.0)
    else:
        run_gemm(plan.xform, w64, data, w64)
        N.call('yb_svd_scale_x', _ptr(w64), _ptr(dblocks), nb, code, _ptr(aux), st)
    tol64 = TOL_STOP64_QR if plan.qr else (TOL_STOP64 if mode == 0 else TOL_STOP64_EIGH)
    if BLOCKED_FP64[0] and _row_sweeps(plan, 64, code):
        _run_row_sweeps(plan, w64, dblocks, dpairs, nb, 64, code, max_sweeps, tol64, state)
    elif plan.rows_per_super64 and BLOCKED_FP64[0]:
        (dsup64,) = _dev(plan, 'svd_super64', (plan.super_items64,), dev)
        N.call('yb_svd_block_sweeps', _ptr(w64), _ptr(dblocks), nb, _ptr(dsup64), len(plan.super_items64),
               plan.super_rounds64, plan.rows_per_super64, 64, code, max_sweeps, 1, tol64, plan.lmax,
               _ptr(state), st)
    else:
        N.call('yb_svd_sweeps', _ptr(w64), _ptr(dblocks), nb, _ptr(dpairs), len(plan.pair_items), plan.max_rounds,
               64, code, max_sweeps, tol64, _ptr(state), st)
    N.call('yb_svd_finalize', _ptr(w64), _ptr(U), _ptr(S), _ptr(V) if V is not None else 0, _ptr(dblocks), nb, code,
           plan.max_k, mode, sp if mode else _ptr(aux), _ptr(state), _ptr(n_small) if n_small is not None else 0, st, launches=3)
    if plan.qr:  # the factor that comes from Q: Vh = conj(W) Q^T (wide), U = conj(Q) W^T (tall)
        if emu:
            for name, F in (('qv', V), ('qu', U)):
                run_emulated(emu[name], w64, w64, F)
                _run_flagged(guard, name, w64, w64, F, flags)
            N.call('yb_svd_poison', _ptr(U), _ptr(V), _ptr(dblocks), nb, code, _ptr(state), P.OZAKI_MIN_DIM, 1, st)
        else:
            run_gemm(plan.qfin_v, w64, w64, V)
            run_gemm(plan.qfin_u, w64, w64, U)
    host = ctl.cpu()
    _svd_state_check(host[n_st:2 * n_st], nb, 'FP32', False)
    if plan.qr and bool(host[2 * n_st + nb:2 * n_st + nb + n_qr][nb + 2::4].any()):
        raise RuntimeError("yastn_gb300 svd: QR group barrier timed out")
    _svd_state_check(host[:n_st], nb, 'FP64', True)
    nz = host[2 * n_st:2 * n_st + nb].numpy()
    if nz.any():
        _complete(plan, U, V, nz, cplx, emu is not None)


def _complete(plan, U, V, nz, cplx, emulated=False):
    """Blocked completion of the vectors of small singular values (blocks left by
    yb_svd_finalize): per block, nz candidate vectors with entries uniform in [-1, 1)
    (yb_fill_candidates), projected twice off the k - nz earlier vectors by grouped GEMMs
    (C = V_g^H G, G -= V_g C), orthonormalised by the batched Householder QR, and copied into
    the factor's last nz vectors (U columns or Vh rows, whichever the rows of X built)."""
    dev, cache = U.device, plan.__dict__.setdefault('_completion', {})
    # the counts depend on the data: the last few only, and per stream (their records on the device go
    # back to the allocator of the stream that has used them)
    key = (_stream(),) + tuple(int(x) for x in nz)
    plans = cache.get(key)
    if plans is None:
        plans = cache[key] = P.completion_plans(plan.blocks, nz, cplx)
        for old in list(cache)[:-MAX_COMPLETIONS]:  # list: one step, other threads insert too
            cache.pop(old, None)
    for cp in plans:
        F = U if cp.to_u else V
        G = torch.empty(max(cp.G, 1), dtype=F.dtype, device=dev)
        C = torch.empty(max(cp.C, 1), dtype=F.dtype, device=dev)
        (dfill,) = _dev(cp, 'fill', (cp.fill,), dev)
        N.call('yb_fill_candidates', _ptr(G), _ptr(dfill), len(cp.fill), _dtype_code(F.dtype), _stream())
        for _ in range(2):
            if emulated and getattr(cp, 'e1', None) is not None:
                run_emulated(cp.e1, F, G, C)
                G.sub_(run_emulated(cp.e2, F, C, torch.zeros_like(G)))
            else:
                run_gemm(cp.g1, F, G, C)
                run_gemm(cp.g2, F, C, G, alpha=-1.0, beta=1.0)
        Qc, _ = qr(G, cp.meta, (max(cp.Q, 1), max(cp.R, 1)))
        run_copy(cp.copy, Qc, F)


def svd(data, meta, sizes, max_sweeps=MAX_SWEEPS):
    """Thin SVD of every block (one-sided Jacobi); returns (U, S, Vh) flat tensors."""
    data = _check(data)
    dev = data.device
    U = torch.empty(sizes[0], dtype=data.dtype, device=dev)
    S = torch.empty(sizes[1], dtype=torch.float64, device=dev)
    V = torch.empty(sizes[2], dtype=data.dtype, device=dev)
    plan = P.svd_plan(meta, ROWS_PER_SUPER[0], data.is_complex(), qr=SVD_QR[0])
    if len(plan.blocks) == 0:
        return U, S, V
    _jacobi(data, plan, U, S, V, 0, max_sweeps)
    return U, S, V


def qr(data, meta, sizes):
    """Reduced QR of every block with R's diagonal made positive (backend_np.py:511-520):
    the batched Householder factorisation of yb_svd_qr, then R[:, m:] = Q^H A[:, m:] for
    wide blocks by a grouped GEMM. Returns (Q, R) flat tensors."""
    data = _check(data)
    dev = data.device
    Q = torch.zeros(sizes[0], dtype=data.dtype, device=dev)
    R = torch.zeros(sizes[1], dtype=data.dtype, device=dev)
    plan = P.qr_plan(meta, data.is_complex())
    nb = len(plan.blocks)
    if nb == 0:
        return Q, R
    (dblocks,) = _dev(plan, 'qr', (plan.blocks,), dev)
    work = torch.empty(plan.n64, dtype=data.dtype, device=dev)
    qctrl = torch.zeros(nb + 4 * min(nb, 4096), dtype=torch.int64, device=dev)
    N.call('yb_qr', _ptr(data), _ptr(Q), _ptr(R), _ptr(work), _ptr(dblocks), nb, _dtype_code(data.dtype),
           _ptr(qctrl), qctrl.numel(), _stream(), launches=4)
    run_gemm(plan.right, Q, data, R)
    if bool(qctrl.cpu()[nb + 2::4].any()):
        raise RuntimeError("yastn_gb300 qr: QR group barrier timed out")
    return Q, R


def qr_backward(Q, R, gQ, gR, data, meta):
    """Adjoint of ``qr`` for float64 and complex128 blocks (the reduced-QR rule that torch's
    autograd applies to the reference's torch.linalg.qr + sign fix, backend_torch.py:475-484):
    dA = (gQ' + Q copyltu(M)) U^{-H}, M = U gU^H - gQ'^H Q, with U = R[:, :k], gU = gR[:, :k],
    gQ' = gQ + A[:, m:] gR[:, m:]^H and dA[:, m:] = Q gR[:, m:] for wide blocks;
    copyltu(M) = tril(M, -1) + tril(M, -1)^H + Re diag(M) (gradients in torch's convention
    for complex tensors)."""
    plan = P.qr_plan(meta, Q.is_complex())
    dev = Q.device
    dA = torch.zeros(data.numel(), dtype=data.dtype, device=dev)
    if len(plan.blocks) == 0:
        return dA
    Bw = torch.zeros_like(Q) if gQ is None else _plain(gQ).to(Q.dtype).clone()
    gR = torch.zeros_like(R) if gR is None else _plain(gR).to(R.dtype)
    M = torch.empty(plan.m_size, dtype=Q.dtype, device=dev)
    run_gemm(plan.w1, data, gR, Bw, beta=1.0)
    run_gemm(plan.m1, R, gR, M)
    run_gemm(plan.m2, Bw, Q, M, alpha=-1.0, beta=1.0)
    (drecs,) = _dev(plan, 'qradj', (plan.adj,), dev)
    code = _dtype_code(Q.dtype)
    N.call('yb_qr_adjoint_sym', _ptr(M), _ptr(drecs), len(plan.adj), code, _stream())
    run_gemm(plan.s1, Q, M, Bw, beta=1.0)
    N.call('yb_trsm_rt', _ptr(Bw), _ptr(R), _ptr(drecs), len(plan.adj), code, _stream())
    if not hasattr(plan, 'copy_plan'):
        plan.copy_plan = P.CopyPlan(plan.copies, sum(int(np.prod(c[2])) for c in plan.copies), data.numel())
    run_copy(plan.copy_plan, Bw, dA)
    run_gemm(plan.y1, Q, gR, dA)
    return dA


def svd_backward(U, S, V, gU, gS, gV, meta, data_size, dtype):
    """Regularised SVD adjoint of every block (torch_svd_gesdd.py:296-428) in 7 launches."""
    plan = P.svd_adjoint_plan(meta)
    dev = U.device
    dA = torch.zeros(data_size, dtype=dtype, device=dev)
    if len(plan.recs) == 0:
        return dA
    code = _dtype_code(U.dtype)
    gU = torch.zeros_like(U) if gU is None else _plain(gU).to(U.dtype)
    gV = torch.zeros_like(V) if gV is None else _plain(gV).to(V.dtype)
    gS = None if gS is None else _plain(gS).to(torch.float64)
    Pm = torch.empty(plan.kk, dtype=U.dtype, device=dev)
    Qm = torch.empty(plan.kk, dtype=U.dtype, device=dev)
    Km = torch.empty(plan.kk, dtype=U.dtype, device=dev)
    TR = torch.empty(max(plan.tr, 1), dtype=U.dtype, device=dev)
    run_gemm(plan.gP, U, gU, Pm)
    run_gemm(plan.gQ, V, gV, Qm)
    (drecs,) = _dev(plan, 'adj', (plan.recs,), dev)
    N.call('yb_svd_adjoint_core', _ptr(Pm), _ptr(Qm), _ptr(S), _vp(gS.data_ptr() if gS is not None else 0), _ptr(Km),
           _ptr(gU), _ptr(gV), _ptr(TR), _ptr(drecs), len(plan.recs), code, _stream())
    run_gemm(plan.gT, Km, V, TR, beta=1.0)
    run_gemm(plan.gR, U, Km, TR, beta=1.0)
    run_gemm(plan.gA1, U, TR, dA)
    run_gemm(plan.gA2, TR, V, dA)
    if not (dtype.is_complex if hasattr(dtype, 'is_complex') else False) and dA.is_complex():
        dA = dA.real.contiguous()
    return dA


def eigh(data, meta, sizes, order_by_magnitude=False, max_sweeps=MAX_SWEEPS):
    """Hermitian eigendecomposition of every block (records (sl, D, slU, DU, slS) of
    yastn/backend/backend_np.py:461-474): eigenvalues ascending, or by descending
    magnitude when ``order_by_magnitude`` (yastn/backend/linalg/torch_eig_sym.py:25-32)."""
    data = _check(data)
    dev = data.device
    S = torch.zeros(sizes[0], dtype=torch.float64, device=dev)
    U = torch.zeros(sizes[1], dtype=data.dtype, device=dev)
    svd_meta = tuple((sl, D, slU, DU, slS, (0, 0), (DU[1], D[1])) for sl, D, slU, DU, slS in meta)
    plan = P.svd_plan(svd_meta, ROWS_PER_SUPER[0], data.is_complex())
    if len(plan.blocks) == 0:
        return S, U
    _jacobi(data, plan, U, S, None, 2 if order_by_magnitude else 1, max_sweeps)
    return S, U


def eigh_backward(U, S, gU, gS, meta, data_size, dtype, order_by_magnitude=False, eps=1.0e-12):
    """Adjoint of ``eigh`` on every block in 4 launches: X = op(U)^T gU, the inner matrix K
    (csrc/yb_adjoint.cu), T = U K, dA = T op(U)^T. order_by_magnitude follows SYMEIG
    (yastn/backend/linalg/torch_eig_sym.py:43-54), otherwise torch.linalg.eigh's adjoint."""
    cplx = U.is_complex()
    plan = P.eigh_adjoint_plan(meta, bool(order_by_magnitude), cplx)
    dev = U.device
    dA = torch.zeros(data_size, dtype=dtype, device=dev)
    if len(plan.recs) == 0:
        return dA
    gU = torch.zeros_like(U) if gU is None else _plain(gU).to(U.dtype)
    gS = None if gS is None else _plain(gS).to(torch.float64)
    X = torch.empty(plan.kk, dtype=U.dtype, device=dev)
    K = torch.empty(plan.kk, dtype=U.dtype, device=dev)
    run_gemm(plan.gX, U, gU, X)
    (drecs,) = _dev(plan, 'eigh_adj', (plan.recs,), dev)
    N.call('yb_eigh_adjoint_core', _ptr(X), _ptr(S), _vp(gS.data_ptr() if gS is not None else 0), _ptr(K),
           _ptr(drecs), len(plan.recs), _dtype_code(U.dtype), int(bool(order_by_magnitude)), float(eps), _stream())
    run_gemm(plan.gT, U, K, X)
    run_gemm(plan.gA, X, U, dA)
    return dA


def fix_svd_signs(U, V, meta):
    """Gauge fix of every block; returns (U', Vh', phases)."""
    U, V = _check(U, 'U'), _check(V, 'V')
    plan = P.fix_signs_plan(meta)
    nb = len(plan.blocks)
    Uo, Vo = torch.empty_like(U), torch.empty_like(V)
    S_size = max((int(r[4] + r[9]) for r in plan.blocks), default=0)
    phases = torch.zeros(S_size, dtype=U.dtype, device=U.device)
    if nb == 0:
        return U.clone(), V.clone(), phases
    (dblocks,) = _dev(plan, 'svd_blocks', (plan.blocks,), U.device)
    N.call('yb_fix_signs', _ptr(U), _ptr(V), _ptr(Uo), _ptr(Vo), _ptr(phases), _ptr(dblocks), nb, plan.max_k,
           _dtype_code(U.dtype), 0, _stream())
    return Uo, Vo, phases


def fix_svd_signs_backward(U, V, gU, gV, meta):
    """Adjoint of the gauge fix (real and complex; yb_fix_signs_adjoint) given the forward's
    inputs U, V and the cotangents of its outputs."""
    plan = P.fix_signs_plan(meta)
    nb = len(plan.blocks)
    need_u, need_v = gU is not None, gV is not None
    gU = torch.zeros_like(U) if gU is None else _plain(gU).to(U.dtype)
    gV = torch.zeros_like(V) if gV is None else _plain(gV).to(V.dtype)
    dU, dV = torch.zeros_like(U), torch.zeros_like(V)  # the kernel writes every position of the records
    if nb:
        (dblocks,) = _dev(plan, 'svd_blocks', (plan.blocks,), U.device)
        N.call('yb_fix_signs_adjoint', _ptr(U), _ptr(V), _ptr(gU), _ptr(gV), _ptr(dU), _ptr(dV), _ptr(dblocks), nb,
               plan.max_k, _dtype_code(U.dtype), _stream())
    return (dU if need_u else None), (dV if need_v else None)


# ----------------------------------------------------------------------------- masks / truncation

def _idx_buffer(mask, meta, device, axis=0):
    """The masks' kept indices concatenated in one device buffer, and per mask (per mask and
    axis length for slice masks, which YASTN passes for whole-axis copies) its offset and
    count."""
    order, lengths, off = [], {}, 0
    for rec in meta:
        tm = rec[4]
        v = mask[tm]
        if isinstance(v, slice):
            Da = (rec[3],) if isinstance(rec[3], int) else rec[3]
            key = (tm, Da[axis])
            if key in lengths:
                continue
            ind = torch.arange(*v.indices(Da[axis]), dtype=torch.int64, device=device)
        else:
            key = tm
            if key in lengths:
                continue
            ind = torch.as_tensor(v, device=device).reshape(-1).to(torch.int64)
        lengths[key] = (off, int(ind.numel()))
        order.append(ind)
        off += int(ind.numel())
    idx = torch.cat(order) if order else torch.zeros(1, dtype=torch.int64, device=device)
    return idx, lengths


def apply_mask(A, mask, meta, Dsize, axis, ndim, scatter_size=None):
    """Gather kept indices along ``axis`` (scatter_size given: the adjoint scatter)."""
    A = _check(A, any_dtype=True)
    idx, lengths = _idx_buffer(mask, meta, A.device, axis)
    recs, items, _ = P.mask_plan(meta, axis, lengths)
    if scatter_size is None:
        out = torch.empty(Dsize, dtype=A.dtype, device=A.device)
    else:
        out = torch.zeros(scatter_size, dtype=A.dtype, device=A.device)
    if len(items) == 0:
        return out
    drecs = torch.from_numpy(recs).to(A.device)
    ditems = torch.from_numpy(items).to(A.device)
    N.call('yb_mask_gather', _ptr(A), _ptr(out), A.element_size(), _ptr(drecs), _ptr(ditems), len(items), _ptr(idx),
           int(scatter_size is not None), _stream())
    return out


def truncation_mask_data(S, slices, charges=None, tol=0, tol_block=0, D_block=float('inf'), D_total=float('inf'),
                         truncate_multiplets=False):
    """The truncation rule of yastn/tensor/linalg.py:637-735 in one device launch.

    ``S`` is the flat float64 spectrum on the device, ``slices`` the (start, stop) of
    each block, ``charges`` the block charges (needed when tol_block/D_block are dicts).
    Returns (mask: bool CUDA tensor, kept: list of kept counts per block).
    """
    S = _check(S, 'S')
    if S.dtype != torch.float64:
        raise TypeError("truncation requires a real float64 spectrum")
    n = S.numel()
    nb = len(slices)
    # the kernel locates blocks by binary search over ascending starts: order them here and
    # return the kept counts in the caller's order
    order = sorted(range(nb), key=lambda i: slices[i][0])
    if order != list(range(nb)):
        slices = [slices[i] for i in order]
        charges = None if charges is None else [charges[i] for i in order]
        mask, kept_sorted = truncation_mask_data(S, slices, charges, tol, tol_block, D_block, D_total,
                                                 truncate_multiplets)
        kept = [0] * nb
        for j, i in enumerate(order):
            kept[i] = kept_sorted[j]
        return mask, kept
    if truncate_multiplets:
        tol_block, D_block = 0, float('inf')
    blk = np.zeros((max(nb, 1), 4), dtype=np.int64)
    tb = np.zeros(max(nb, 1), dtype=np.float64)
    tol_null = 0. if isinstance(tol_block, dict) else tol_block
    D_null = 0 if isinstance(D_block, dict) else D_block
    for i, (lo, hi) in enumerate(slices):
        t = tuple(charges[i]) if charges is not None else None
        tb[i] = tol_block[t] if (isinstance(tol_block, dict) and t in tol_block) else tol_null
        d = D_block[t] if (isinstance(D_block, dict) and t in D_block) else D_null
        blk[i] = (lo, hi, -1 if d == float('inf') else int(d), 0)
    dt = -1 if D_total == float('inf') else int(D_total)
    mask = torch.empty(n, dtype=torch.uint8, device=S.device)
    kept = torch.empty(max(nb, 1), dtype=torch.int64, device=S.device)
    if nb == 0 or n == 0:
        return mask.bool(), [0] * nb
    dblk = torch.from_numpy(blk).to(S.device)
    dtb = torch.from_numpy(tb).to(S.device)
    N.call('yb_truncation_mask', _ptr(S), n, _ptr(dblk), _ptr(dtb), nb, float(tol), dt, int(bool(truncate_multiplets)),
           _ptr(mask), _ptr(kept), _stream())
    return mask.view(torch.bool), kept[:nb].tolist()
