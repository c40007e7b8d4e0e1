"""The momentum's gradient can itself be differentiated, as that of the addition and product that it stands for."""
import pytest
import torch

from uttt_b200.ops import functional

EPS = 1e-7


class _Extension:
    """The kernels' formulas in plain operations, hidden from autograd as a kernel is."""

    @staticmethod
    def momentum_normalize_fwd(a, z, m, matrices, eps):
        with torch.no_grad():
            z_new = a + m.view(-1, 1, 1, 1) * z
            v = z_new.reshape(matrices, -1)
            sumsq = v.pow(2).sum(1)
            return z_new, (v / (sumsq.sqrt()[:, None] + eps)).view_as(a), sumsq

    @staticmethod
    def momentum_normalize_bwd(z_new, z, m, sumsq, dz_new, dx, eps, need_dz, need_dm):
        with torch.no_grad():
            g = torch.zeros_like(z_new) if dz_new is None else dz_new.clone()
            if dx is not None:
                v, d, r = z_new.reshape(sumsq.numel(), -1), dx.reshape(sumsq.numel(), -1), sumsq.sqrt()[:, None]
                along = torch.where(r > 0, (v * d).sum(1, keepdim=True) / (r * (r + eps) ** 2), 0.0)
                g += (d / (r + eps) - v * along).view_as(g)
            return g, m.view(-1, 1, 1, 1) * g, (g * z).sum((1, 2, 3))


def _operands():
    gen = torch.Generator().manual_seed(3)
    a, z = (torch.randn(2, 2, 4, 3, generator=gen, dtype=torch.float64) for _ in range(2))
    return [t.requires_grad_() for t in (a, z, torch.rand(2, generator=gen, dtype=torch.float64))]


def _plain(a, z, m):
    z_new = torch.addcmul(a, z, m.view(-1, 1, 1, 1))
    v = z_new.reshape(8, -1)
    return z_new, (v / (v.norm(dim=1, keepdim=True) + EPS)).view_as(a)


@pytest.mark.parametrize("outputs", [(0,), (1,), (0, 1)])
def test_second_order(monkeypatch, outputs):
    monkeypatch.setattr(functional, "cuda_ext", lambda t: _Extension)
    res = []
    for fn in (lambda *t: functional._MomentumNormalize.apply(*t, 8, EPS), _plain):
        t = _operands()
        loss = sum((fn(*t)[i] ** 2 * torch.linspace(-1, 2, 48, dtype=torch.float64).view(2, 2, 4, 3)).sum() for i in outputs)
        first = torch.autograd.grad(loss, t, create_graph=True)
        second = torch.autograd.grad(sum(g.pow(2).sum() for g in first) + loss, t, retain_graph=True)
        plain_first = torch.autograd.grad(loss, t)                # the kernel's own backward
        res.append((*first, *second, *plain_first))
    for got, want in zip(*res):
        torch.testing.assert_close(got, want)


def test_zero_matrix(monkeypatch):
    """A matrix of zeros (no gradient, no momentum) has a gradient and a second one without NaN."""
    monkeypatch.setattr(functional, "cuda_ext", lambda t: _Extension)
    a = torch.zeros(1, 1, 4, 3, dtype=torch.float64).requires_grad_()
    z, m = torch.zeros_like(a), torch.ones(1, dtype=torch.float64)
    _, x = functional._MomentumNormalize.apply(a, z, m, 1, EPS)
    g, = torch.autograd.grad(x.sum(), a, create_graph=True)
    assert torch.equal(g, torch.full_like(g, 1 / EPS))
    assert torch.autograd.grad(g.sum(), a)[0].isfinite().all()
