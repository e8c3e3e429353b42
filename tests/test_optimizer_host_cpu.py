"""Host side of the optimizers without a device: what is kept between steps must follow the groups, tensors and
buffers that the next step finds."""
import collections
import copy
import gc

import pytest
import torch
import torch.nn as nn

import torchsso
from torchsso import _native as nat

SHAPES = {'Linear': 'Kron'}


def make(seed=0, **kwargs):
    torch.manual_seed(seed)
    model = nn.Sequential(nn.Linear(5, 7), nn.Tanh(), nn.Linear(7, 3))
    kwargs = {'lr': 0.1, 'momentum': 0.9, 'weight_decay': 0.01, **kwargs}
    return torchsso.optim.SecondOrderOptimizer(model, 'Cov', SHAPES, {'damping': 1e-2}, **kwargs)


@pytest.fixture
def kernel(monkeypatch):
    """The update kernel on tensors in place of addresses: a table holds on to what it was built from."""
    def run(table, sets):
        for p, g, m, e, i in table:
            add, mom, ema, scale, lr = sets[i]
            v = g + add * p
            if m is not None:
                v = m.copy_(mom * m + v)
            if e is not None:
                v = e.copy_(ema * v + (1 - ema) * e)
            g.copy_(scale * v)
            p.sub_(lr * g)
    monkeypatch.setattr(nat, 'tail_set_records', lambda items, device: list(items))
    monkeypatch.setattr(nat, 'tail_sets', list)
    monkeypatch.setattr(nat, 'optimizer_tail_sets', run)


def step(opt, seed, fused=True):
    opt._curvature_step = lambda *a: None
    if not fused:
        opt._fused_tail = lambda *a: set()
    g = torch.Generator().manual_seed(seed)
    for group in opt.param_groups:
        for p in group['params']:
            p.grad = torch.randn(p.shape, generator=g)
    opt._harvest_grads()
    opt._update_groups(opt.param_groups, 'params', False, None)


def reset_buffers(opt):
    for group in opt.param_groups:
        opt.init_buffer(group['params'])


def rebind_one(opt):
    p = opt.param_groups[0]['params'][0]
    opt.state[p]['momentum_buffer'] = torch.ones_like(p)


def new_state(opt):
    for _ in range(3):          # more than once: a state may come to lie where one before it was
        opt.state = collections.defaultdict(dict)
        reset_buffers(opt)


def copied_groups(opt):
    opt.param_groups[:] = [dict(g) for g in opt.param_groups]


def other_layout(opt):
    p = opt.param_groups[0]['params'][0]      # same address, another order of its elements
    p.data = p.data.view(p.shape[1], p.shape[0]).t()


def other_curvature(opt):
    opt.param_groups[0]['curv'] = None


@pytest.mark.parametrize('kwargs', [{}, {'l2_reg': 0.1, 'momentum_type': 'raw', 'grad_ema_decay': 0.3}])
@pytest.mark.parametrize('change', [reset_buffers, rebind_one, new_state, copied_groups, other_layout, other_curvature])
def test_update_table_follows_what_changed(kernel, kwargs, change):
    got, want = make(**kwargs), make(**kwargs)
    for i in range(4):
        if i == 2:
            change(got)
            change(want)
        step(got, i)
        step(want, i, fused=False)
    for a, b in zip(got.param_groups, want.param_groups):
        for p, q in zip(a['params'], b['params']):
            torch.testing.assert_close(p, q, rtol=1e-5, atol=1e-6)
            for name in ('momentum_buffer', 'grad_ema_buffer'):
                torch.testing.assert_close(got.state[p][name], want.state[q][name], rtol=1e-5, atol=1e-6)
        if a['curv'] is not None:
            assert a['curv'].l2_reg == b['curv'].l2_reg


class Recorder:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *args, **kwargs: self.calls.append((name, *args))

    def given(self, name):
        return [c[1] for c in self.calls if c[0] == name]


def curvature_step(opt, monkeypatch):
    """(curvatures whose inverses the pool refreshes, those it preconditions with, those that step by themselves)."""
    opt.pool, alone = Recorder(), []
    monkeypatch.setattr(torchsso.KronCovLinear, 'step', lambda self, **kw: alone.append(self))
    monkeypatch.setattr(torchsso.KronCovLinear, 'precondition_grad', lambda self, params: None)
    opt._curvature_step(opt.param_groups, 'params', True, None)
    inverted = sum(opt.pool.given('update_inv'), [])
    return inverted, sum(opt.pool.given('precondition'), []), alone


def test_curvature_step_follows_what_changed(monkeypatch):
    opt = make()
    first, second = (g['curv'] for g in opt.param_groups)
    assert curvature_step(opt, monkeypatch) == ([first, second], [first, second], [])
    second.use_max_ema = True               # the pool does not keep running maxima
    assert curvature_step(opt, monkeypatch) == ([first], [first], [second])
    second.use_max_ema = False
    assert curvature_step(opt, monkeypatch) == ([first, second], [first, second], [])
    opt.param_groups[0]['curv'] = None
    assert curvature_step(opt, monkeypatch) == ([second], [second], [])
    opt.param_groups[0]['curv'] = first
    opt.param_groups[0]['params'] = opt.param_groups[0]['params'][:1]
    curvature_step(opt, monkeypatch)
    grads = next(c[2] for c in opt.pool.calls if c[0] == 'precondition')
    assert [len(g) for g in grads] == [1, 2]


# ------------------------------------------------------------------------------------------- lifetime
def hooked(module, width=5):
    """Whether the module's forward pass reaches a curvature (which has no CPU path)."""
    try:
        module(torch.ones(2, width))
    except RuntimeError as e:
        assert 'CUDA' in str(e)
        return True
    return False


@pytest.fixture
def no_collection():
    gc.collect()
    gc.disable()
    yield
    gc.enable()


def test_a_curvature_lives_as_long_as_it_is_held(no_collection):
    layer = nn.Linear(5, 7)
    curv = torchsso.KronCovLinear(layer, damping=1e-2)
    assert hooked(layer)
    assert not hooked(copy.deepcopy(layer))          # a copy of the module has none
    copied = copy.deepcopy(curv)                     # a copy of the curvature brings its module
    assert copied.module is not layer and hooked(copied.module)
    del curv
    assert not hooked(layer) and hooked(copied.module)


def test_the_curvatures_of_an_optimizer_go_with_it(no_collection):
    opt = make()
    layer, keep = opt.model[0], opt.param_groups[1]['curv']
    assert hooked(layer)
    del opt
    assert not hooked(layer)
    # one that somebody still holds keeps its place in the pool
    (da, _), (dg, _) = keep.shape
    lo, hi = keep.pool.kron_range([keep])
    assert keep.pool.kron == [keep] and hi - lo >= da * da + dg * dg and hi == keep.pool.k_total


def test_pool_ranges_without_a_neighbour(no_collection, monkeypatch):
    opt = make()
    first, pool = opt.param_groups[0]['curv'], opt.pool
    lo, hi = pool.kron_range([first])
    pool._ranges.clear()
    opt.param_groups[1]['curv'] = None               # gone, and with it the only strong reference
    assert len(pool.kron) == 1 and pool.kron_range([first]) == (lo, hi)
    spans = []
    monkeypatch.setattr(nat, 'axpby', lambda x, y, a, b: spans.append(x.numel()))
    pool.accumulate(1.0, True)
    assert spans == [pool.k_total]


@pytest.mark.parametrize('uses_work', [False, True])
@pytest.mark.parametrize('std,inverse', [(False, True), (True, True), (True, False)])
def test_a_bad_pivot_is_counted_from_where_the_pass_began(monkeypatch, std, inverse, uses_work):
    """The dataflow kernel takes the matrices of an inverse with sampling factors from the last row on; every other pass
    goes from the first."""
    class NoPlan:
        def status(self):
            return 0

    def run(plan, damp, info, do_inverse, do_std):
        info[2 + (not do_inverse)] = 7
    monkeypatch.setattr(nat, 'kron_plan_uses_work', lambda: uses_work)
    monkeypatch.setattr(nat, 'kron_plan', lambda *a, **k: NoPlan())
    monkeypatch.setattr(nat, 'kron_plan_run', run)
    opt = make()
    pool = opt.pool
    pool.update_inv(with_std=False)
    with pytest.raises(RuntimeError, match=r'matrix 1 \(inverse pass\) is not positive definite at row 7$'):
        pool.check_info()
    pool.update_inv(with_std=std, do_inverse=inverse)
    with pytest.raises(RuntimeError, match='from the last row to the first' if std and inverse and not uses_work else 'at row 7$'):
        pool.check_info()


# ------------------------------------------------------------------------------------------- prepared calls
def on_meta(t):
    return torch.empty_strided(t.shape, t.stride(), dtype=t.dtype, device='meta')


def other_padding(m, x, g):
    m.padding = [0, 2]
    return x, g


CHANGES = [lambda m, x, g: (on_meta(x), g), lambda m, x, g: (x, on_meta(g)), lambda m, x, g: (on_meta(x), on_meta(g)), other_padding]


@pytest.mark.parametrize('change', CHANGES)
def test_squared_gradient_calls_are_prepared_per_device_and_geometry(monkeypatch, change):
    """An operand on another device has passed no check, whatever was checked for its layout before."""
    calls = []
    monkeypatch.setattr(nat, 'diag_sq', lambda *a: calls.append('checked'))
    monkeypatch.setattr(nat, 'diag_sq_call', lambda x, g, *geometry: (x, g, 'call'))
    monkeypatch.setattr(nat, 'diag_sq_run', lambda *a: calls.append('prepared'))
    m = nn.Conv2d(3, 4, 3, padding=1)
    curv = torchsso.DiagCovConv2d(m)
    x, g = torch.randn(2, 3, 5, 5), torch.randn(2, 4, 5, 5)
    for _ in range(2):
        m.data_input = x
        curv.update_in_backward(g)
    m.data_input, g = change(m, x, g)
    curv.update_in_backward(g)
    assert calls == ['checked', 'prepared', 'checked']


@pytest.mark.parametrize('change', [CHANGES[0], other_padding])
def test_factor_calls_are_prepared_per_device_and_geometry(monkeypatch, change):
    made = []

    class Op:
        def __init__(self, x, kernel_size, stride, padding, dilation, append_ones, out):
            made.append((x.device.type, tuple(padding)))

        def run(self, *args):
            pass
    monkeypatch.setattr(nat, 'FactorOp', Op)
    m = nn.Conv2d(3, 4, 3, padding=1)
    curv = torchsso.KronCovConv2d(m)
    x = torch.randn(2, 3, 5, 5)
    curv.update_in_forward(x)
    curv.update_in_forward(x)
    curv.update_in_forward(change(m, x, None)[0])
    assert len(made) == 2 and len(set(made)) == 2


def test_an_output_gradient_on_the_host_is_refused(monkeypatch):
    monkeypatch.setattr(nat, '_require_cuda', lambda t, what: calls.append(what))
    calls = []
    nat.diag_sq_call(torch.randn(2, 3), torch.randn(2, 4), (1, 1), (1, 1), (0, 0), (1, 1))
    assert calls == ['layer input', 'output gradient']
