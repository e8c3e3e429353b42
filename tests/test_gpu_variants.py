"""Kernel variants and dispatch branches at the sizes where they can go wrong."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def nat():
    from torchsso import _native
    _native.lib()
    return _native


def rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-300)).item()


@pytest.mark.parametrize('n,c', [(1, 1), (7, 3), (8, 32), (33, 33), (32, 1000)])
def test_sample_classes_is_the_multinomial_draw(nat, n, c):
    p = torch.softmax(3 * torch.randn(n, c, device='cuda'), 1)
    for seed in range(5):
        torch.manual_seed(seed)
        want = torch.multinomial(p, 1, replacement=True).t()
        torch.manual_seed(seed)
        assert torch.equal(nat.sample_classes(p, torch.empty_like(p).exponential_()), want)
    p[0] = float('nan')          # nothing left of this row: uniform
    got = torch.cat([nat.sample_classes(p, torch.empty_like(p).exponential_()) for _ in range(200)])
    assert 0 <= int(got.min()) and int(got.max()) < c and got[:, 0].unique().numel() > min(c, 20) // 2


@pytest.mark.parametrize('numel,shift', [(1, 0), (4095, 0), (4096, 0), (4097, 1), (12300, 2)])
def test_optimizer_tail_sets(nat, numel, shift):
    """Records of one launch with different scalars; `shift` elements off the 16-byte boundary."""
    def new():
        return torch.randn(numel + shift, device='cuda')[shift:]
    items, want = [], []
    sets = [(0.01, 0.9, 0.3, 1.5, 0.05), (0.0, 0.5, 1.0, 1.0, 0.0)]
    for i, (add, mom, ema, scale, lr) in enumerate(sets):
        p, g, m, e = new(), new(), new(), new()
        v = g.double() + add * p.double()
        wm = mom * m.double() + v
        we = (1 - ema) * e.double() + ema * wm
        want.append((p.double() - lr * scale * we, scale * we, wm, we))
        items.append((p, g, m, e, i))
    nat.optimizer_tail_sets(nat.tail_set_records(items, torch.device('cuda')), nat.tail_sets(sets))
    for it, w in zip(items, want):
        for got, ref in zip(it, w):
            assert rel(got, ref) < 1e-6


def test_precondition_grad_of_moving_gradients(nat):
    """Gradients at a new address on every call, and of another type and layout."""
    import torchsso
    layer = torch.nn.Linear(70, 33).cuda()
    curv = torchsso.KronCovLinear(layer, damping=1e-2)
    layer(torch.randn(200, 70, device='cuda')).square().mean().backward()
    curv.step(update_inv=True)
    a, g = (m.double() for m in curv.inv)
    keep = []
    for dtype in (torch.float32, torch.float32, torch.bfloat16):
        w, b = torch.randn(33, 70, device='cuda').to(dtype), torch.randn(33, device='cuda').to(dtype)
        want = g @ torch.cat([w, b[:, None]], 1).double() @ a
        params = [torch.empty_like(w), torch.empty_like(b)]
        params[0].grad, params[1].grad = w.t().contiguous().t(), b.clone()
        curv.precondition_grad(params)
        keep.append(params)
        got = torch.cat([params[0].grad, params[1].grad[:, None]], 1)
        assert rel(got, want) < (1e-4 if dtype == torch.float32 else 1e-2)
