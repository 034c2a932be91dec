"""backend_gb300._apply against autograd.Function.apply: the same values, gradients, errors and hooks in
every context in which a call may stand (a function of its own on the CPU; on the GPU the backend's)."""
import contextlib

import numpy as np
import pytest
import torch
import torch.autograd.forward_ad as fwAD

from yastn_gb300.backend_gb300 import _apply


class Scaled(torch.autograd.Function):
    """a b s, with the layout of the backend's functions; forward runs are counted."""
    generate_vmap_rule = False
    runs = [0]

    @staticmethod
    def forward(a, b, s, shift=0.0):
        Scaled.runs[0] += 1
        return a * b * s + shift

    @staticmethod
    def setup_context(ctx, inputs, output):
        a, b, s, *_ = inputs
        ctx.save_for_backward(a, b)
        ctx.s = s

    @staticmethod
    def backward(ctx, g):
        a, b = ctx.saved_tensors
        return g * b * ctx.s, g * a * ctx.s, None, None


def lean(a, b):
    return _apply(Scaled, (a, b), 3.0)


def full(a, b):
    return Scaled.apply(a, b, 3.0)


def pair(ga=False, gb=False):
    gen = torch.Generator().manual_seed(1)
    return (torch.randn(5, dtype=torch.float64, generator=gen).requires_grad_(ga),
            torch.randn(5, dtype=torch.float64, generator=gen).requires_grad_(gb))


@pytest.mark.parametrize('ga,gb', [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize('mode', [contextlib.nullcontext, torch.no_grad, torch.inference_mode, torch.enable_grad])
def test_modes(ga, gb, mode):
    got = []
    for f in (lean, full):
        a, b = pair(ga, gb)
        with mode():
            y = f(a, b)
        grads = torch.autograd.grad(y.sum(), [x for x in (a, b) if x.requires_grad]) if y.requires_grad else ()
        got.append((y.requires_grad, y.is_inference(), y.grad_fn is not None, y.detach().numpy(), [g.numpy() for g in grads]))
    assert got[0][:3] == got[1][:3]
    np.testing.assert_array_equal(got[0][3], got[1][3])
    for x, y in zip(got[0][4], got[1][4]):
        np.testing.assert_array_equal(x, y)


def test_create_graph():
    for f in (lean, full):
        a, b = pair(True, True)
        (g,) = torch.autograd.grad(f(a, b).sum(), a, create_graph=True)
        (h,) = torch.autograd.grad(g.sum(), b)
        np.testing.assert_array_equal(h.numpy(), np.full(5, 3.0))


@pytest.mark.parametrize('transform', [
    lambda f, a, b: torch.func.grad(lambda x, y: f(x, y).sum())(a, b),
    lambda f, a, b: torch.func.vjp(f, a, b)[1](torch.ones_like(a)),
    lambda f, a, b: torch.func.vjp(lambda x: f(x, b), a)[1](torch.ones_like(a)),
    lambda f, a, b: torch.func.grad(lambda x: torch.func.grad(lambda y: f(x, y).sum())(b).sum())(a),
    lambda f, a, b: torch.func.vmap(f)(a, b),
    lambda f, a, b: torch.func.jvp(f, (a, b), (a, b)),
    lambda f, a, b: f(torch.nn.Parameter(a), b).detach(),
])
def test_transforms(transform):
    """The same values, or the same refusal (vmap and jvp have no rule)."""
    got = []
    for f in (lean, full):
        try:
            r = transform(f, *pair())
            got.append([x.detach().numpy() for x in (r if isinstance(r, (tuple, list)) else (r,))])
        except Exception as e:
            got.append((type(e), str(e)))
    assert len(got[0]) == len(got[1])
    for x, y in zip(*got):
        if isinstance(x, np.ndarray):
            np.testing.assert_array_equal(x, y)
        else:
            assert x == y


def test_forward_mode():
    """A dual tensor meets Function.apply's own answer, and an open level without duals changes nothing."""
    got = []
    for f in (lean, full):
        a, b = pair()
        with fwAD.dual_level():
            plain = f(a, b)
            try:
                out = fwAD.unpack_dual(f(fwAD.make_dual(a, b), b)).tangent
                got.append((plain.numpy(), None if out is None else out.numpy()))
            except Exception as e:
                got.append((plain.numpy(), type(e)))
    np.testing.assert_array_equal(got[0][0], got[1][0])
    assert type(got[0][1]) is type(got[1][1]) and (got[0][1] is got[1][1] or np.array_equal(got[0][1], got[1][1]))


def test_saved_tensor_hooks_and_checkpoint():
    for f in (lean, full):
        a, b = pair(True, True)
        packed = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(1), t * 2)[1], lambda t: t / 2):
            y = f(a, b)
        ga, gb = torch.autograd.grad(y.sum(), (a, b))
        assert len(packed) == 2
        np.testing.assert_array_equal(ga.numpy(), 3.0 * b.detach().numpy())
        a, b = pair(True, True)
        Scaled.runs[0] = 0
        y = torch.utils.checkpoint.checkpoint(f, a, b, use_reentrant=False)
        torch.autograd.grad(y.sum(), (a, b))
        assert Scaled.runs[0] == 2  # the forward, and its recomputation


def test_subclasses():
    class Sub(torch.Tensor):
        pass
    for f in (lean, full):
        a, b = pair()
        y = f(a.as_subclass(Sub), b)
        np.testing.assert_array_equal(y.as_subclass(torch.Tensor).numpy(), (a * b * 3).numpy())
    kinds = [type(f(pair()[0].as_subclass(Sub), pair()[1])) for f in (lean, full)]
    assert kinds[0] is kinds[1]


def test_arguments_pass_through():
    """A forward's default arguments may be left out, with and without a graph."""
    for grad in (False, True):
        a, b = pair(grad)
        np.testing.assert_array_equal(_apply(Scaled, (a, b), 2.0).detach().numpy(), (a * b * 2).detach().numpy())
        np.testing.assert_array_equal(_apply(Scaled, (a, b), 2.0, 1.0).detach().numpy(), (a * b * 2 + 1).detach().numpy())


@pytest.mark.gpu
def test_backend_calls_in_every_context(cuda_device):
    """backend.dot under no_grad with inputs that require grad, saved-tensor hooks, torch.func and forward mode."""
    from oracle import backend_oracle as oracle
    from yastn_gb300 import backend
    rng = np.random.default_rng(0)
    meta = (((0, 20), (4, 5), (0, 12), (4, 3), (0, 15), (3, 5)),)
    A, B, G = rng.normal(size=12), rng.normal(size=15), rng.normal(size=20)
    want, (wa, wb) = oracle.dot(A, B, meta, 20), oracle.dot_backward(G, A, B, meta)
    a, b, g = (torch.from_numpy(x).cuda() for x in (A, B, G))

    def f(x, y):
        return backend.dot(x, y, meta, 20)

    def same(x, y):
        np.testing.assert_allclose(x.detach().cpu().numpy(), y, rtol=0, atol=1e-14 * 10)
    x, y = a.clone().requires_grad_(), b.clone().requires_grad_()
    with torch.no_grad():
        out = f(x, y)
    assert not out.requires_grad
    same(out, want)
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (seen.append(1), t.cpu())[1], lambda t: t.cuda()):
        out = f(x, y)
    ga, gb = torch.autograd.grad(out, (x, y), g)
    assert seen
    same(ga, wa), same(gb, wb)
    out, pull = torch.func.vjp(f, a, b)
    ga, gb = pull(g)
    same(out, want), same(ga, wa), same(gb, wb)
    with fwAD.dual_level():
        same(f(a, b), want)
    with torch.inference_mode():
        same(f(a, b), want)
