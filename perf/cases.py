"""Performance cases: what a training program has this package do, through the calls it makes.

A case is one of seven programs at some size:

  mlp      fp32 multi-layer perceptron, ``SecondOrderOptimizer`` (Fisher with one Monte Carlo target, or Cov)
  convnet  the 5x5 / 5x5 / 3x3 ConvNet with biases and two Linear layers, NCHW fp32 or channels_last bf16
  resnet   bottleneck ResNet with BatchNorm, bf16, Fisher: issued eagerly, or replayed from CUDA graphs with
           the switches ``bench.py`` uses
  vgg_vi   VGG-style convolution stack under ``VIOptimizer`` (factors, inverses, Cholesky factors, posterior samples)
  vogn     the ConvNet under ``VOGN`` (diagonal curvature of Linear / Conv2d)
  layer    one layer's curvature object used without an optimizer: factors of a batch of rows, damped
           inverses, preconditioned gradient
  linalg   ``torchsso.utils.inv`` and ``cholesky`` of one SPD matrix

A pass is one optimizer step (or one use of the curvature object): forward, backward, the hooks' factor
kernels, running averages, inverses on the steps that refresh them, precondition, update.  Each pass
starts from the prepared weights, so that its outputs are a function of its inputs and not of the
rounding of the passes before it (a ReLU network amplifies that from step to step); curvature averages,
momentum and the inverse schedule carry on from pass to pass as they do in training.
"""
import math
import os
import sys

import torch
import torch.nn as nn
import torch.nn.functional as F

sys.path.insert(0, os.path.abspath('pytorch-sso_b200'))

import torchsso  # noqa: E402

SHAPES = {'Linear': 'Kron', 'Conv2d': 'Kron', 'BatchNorm2d': 'Diag'}
CURV = {'ema_decay': 0.95, 'damping': 1e-3}
DATASET = 50000


# ------------------------------------------------------------------------------------------------ models
class MLP(nn.Module):
    def __init__(self, f_in, width, classes):
        super().__init__()
        self.num_classes = classes
        self.f1, self.f2, self.f3 = nn.Linear(f_in, width), nn.Linear(width, width), nn.Linear(width, classes)

    def forward(self, x):
        return self.f3(F.relu(self.f2(F.relu(self.f1(x)))))


class ConvNet(nn.Module):
    """3 -> w -> 2w -> 4w channels, pooled after each convolution, then two Linear layers.  The weight-sampling
    optimizers get smooth units: the draw depends on the curvature, and a ReLU flips on its last digit."""

    def __init__(self, width, image, classes, smooth=False):
        super().__init__()
        self.num_classes = classes
        self.act, self.pool = (torch.tanh, F.avg_pool2d) if smooth else (F.relu, F.max_pool2d)
        self.c1, self.c2 = nn.Conv2d(3, width, 5, padding=2), nn.Conv2d(width, 2 * width, 5, padding=2)
        self.c3 = nn.Conv2d(2 * width, 4 * width, 3, padding=1)
        self.f1 = nn.Linear(4 * width * (image // 8) ** 2, 8 * width)
        self.f2 = nn.Linear(8 * width, classes)

    def forward(self, x):
        for conv in (self.c1, self.c2, self.c3):
            x = self.pool(self.act(conv(x)), 2)
        return self.f2(self.act(self.f1(x.flatten(1))))


class VGG(nn.Module):
    """Thirteen 3x3 convolutions (VGG-16's stack; width 64 is the usual one) and one Linear layer."""

    def __init__(self, width, classes):
        super().__init__()
        self.num_classes = classes
        layers, cin = [], 3
        for mult, count in ((1, 2), (2, 2), (4, 3), (8, 3), (8, 3)):
            for _ in range(count):
                layers += [nn.Conv2d(cin, mult * width, 3, padding=1), nn.Tanh()]
                cin = mult * width
            layers.append(nn.AvgPool2d(2))
        self.features, self.fc = nn.Sequential(*layers), nn.Linear(cin, classes)

    def forward(self, x):
        return self.fc(self.features(x).flatten(1))


class Bottleneck(nn.Module):
    def __init__(self, cin, width, stride):
        super().__init__()
        self.conv1, self.bn1 = nn.Conv2d(cin, width, 1, bias=False), nn.BatchNorm2d(width)
        self.conv2, self.bn2 = nn.Conv2d(width, width, 3, stride=stride, padding=1, bias=False), nn.BatchNorm2d(width)
        self.conv3, self.bn3 = nn.Conv2d(width, 4 * width, 1, bias=False), nn.BatchNorm2d(4 * width)
        self.down = None
        if stride != 1 or cin != 4 * width:
            self.down = nn.Sequential(nn.Conv2d(cin, 4 * width, 1, stride=stride, bias=False), nn.BatchNorm2d(4 * width))

    def forward(self, x):
        y = F.relu(self.bn1(self.conv1(x)))
        y = self.bn3(self.conv3(F.relu(self.bn2(self.conv2(y)))))
        return F.relu(y + (x if self.down is None else self.down(x)))


class ResNet(nn.Module):
    def __init__(self, width, blocks, classes):
        super().__init__()
        self.num_classes = classes
        self.conv1, self.bn1 = nn.Conv2d(3, width, 7, stride=2, padding=3, bias=False), nn.BatchNorm2d(width)
        cin, stages = width, []
        for i, count in enumerate(int(b) for b in blocks):
            for j in range(count):
                stages.append(Bottleneck(cin, width << i, 2 if i > 0 and j == 0 else 1))
                cin = 4 * (width << i)
        self.blocks, self.fc = nn.Sequential(*stages), nn.Linear(cin, classes)

    def forward(self, x):
        x = F.max_pool2d(F.relu(self.bn1(self.conv1(x))), 3, stride=2, padding=1)
        return self.fc(F.adaptive_avg_pool2d(self.blocks(x), 1).flatten(1))


class Autocast:
    """The model as a closure for bf16 calls it."""

    def __init__(self, model):
        self.model, self.num_classes = model, model.num_classes

    def __call__(self, x):
        with torch.autocast('cuda', dtype=torch.bfloat16):
            return self.model(x).float()


def build(case):
    kind = case['kind']
    if kind == 'mlp':
        return MLP(case['f_in'], case['width'], case['classes'])
    if kind in ('convnet', 'vogn'):
        return ConvNet(case['width'], case['image'], case['classes'], smooth=kind == 'vogn')
    if kind == 'vgg_vi':
        return VGG(case['width'], case['classes'])
    return ResNet(case['width'], case['blocks'], case['classes'])


# ------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # the smallest step: a tabular-data MLP, where launches and host work are all there is
        {'name': 'mlp_tiny', 'kind': 'mlp', 'f_in': 20, 'width': 32, 'classes': 10, 'batch': 16, 'curv': 'Fisher', 'every': 1, 'momentum': 0.0},
        # the 784-1000-1000-10 MLP at batch 128 with inverses on every step
        {'name': 'mlp_784', 'kind': 'mlp', 'f_in': 784, 'width': 1000, 'classes': 10, 'batch': 128, 'curv': 'Fisher', 'every': 1, 'momentum': 0.0},
        # an odd-sized MLP trained as most are: Cov, momentum, stale inverses
        {'name': 'mlp_cov_odd', 'kind': 'mlp', 'f_in': 301, 'width': 517, 'classes': 37, 'batch': 200, 'curv': 'Cov', 'every': 5, 'momentum': 0.9},
        # the ConvNet at batch 256 as a user of the defaults runs it: fp32, NCHW, inverses every five steps
        {'name': 'convnet_b256', 'kind': 'convnet', 'width': 64, 'image': 32, 'classes': 10, 'batch': 256, 'bf16': False, 'every': 5, 'acc': 1},
        # the same family in bf16 and channels_last, ragged, with gradient accumulation
        {'name': 'convnet_bf16_acc', 'kind': 'convnet', 'width': 24, 'image': 28, 'classes': 10, 'batch': 50, 'bf16': True, 'every': 5, 'acc': 2},
        # ResNet-50 at 32 images of 224x224: the headline configuration
        {'name': 'resnet50_b32', 'kind': 'resnet', 'width': 64, 'blocks': '3463', 'classes': 1000, 'image': 224, 'batch': 32, 'graph': True, 'every': 10},
        # a small ResNet of the same build without graphs: one launch at a time
        {'name': 'resnet_small_eager', 'kind': 'resnet', 'width': 16, 'blocks': '1111', 'classes': 100, 'image': 64, 'batch': 8, 'graph': False, 'every': 10},
        # VGG-16 under variational inference, four weight samples per step
        {'name': 'vgg_vi_b128', 'kind': 'vgg_vi', 'width': 64, 'classes': 100, 'batch': 128, 'samples': 4},
        # VOGN: diagonal curvature of every layer
        {'name': 'vogn_convnet', 'kind': 'vogn', 'width': 32, 'image': 32, 'classes': 10, 'batch': 128, 'samples': 4},
        # one layer with a bias (d = 577), as a curvature object
        {'name': 'layer_577', 'kind': 'layer', 'd_in': 576, 'd_out': 64, 'bias': True, 'rows': 25088},
        # one wide layer: the largest factor of ResNet-50
        {'name': 'layer_4608', 'kind': 'layer', 'd_in': 4608, 'd_out': 512, 'bias': False, 'rows': 8192},
        # one matrix
        {'name': 'linalg_1000', 'kind': 'linalg', 'd': 1000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['mlp', 'mlp', 'convnet', 'resnet', 'vgg_vi', 'vogn', 'layer', 'layer', 'linalg'])
    if kind == 'mlp':
        return {'kind': kind, 'f_in': _log(rng, 16, 1024), 'width': _log(rng, 24, 1200), 'classes': _log(rng, 4, 100), 'batch': _log(rng, 16, 512),
                'curv': rng.choice(['Fisher', 'Cov']), 'every': rng.choice([1, 5]), 'momentum': rng.choice([0.0, 0.9])}
    if kind == 'convnet':
        return {'kind': kind, 'width': _log(rng, 8, 64), 'image': rng.randint(16, 32), 'classes': _log(rng, 4, 100), 'batch': _log(rng, 16, 256),
                'bf16': rng.random() < 0.5, 'every': rng.choice([1, 5]), 'acc': rng.choice([1, 2])}
    if kind == 'resnet':
        return {'kind': kind, 'width': 8 * _log(rng, 2, 8), 'blocks': rng.choice(['1111', '2222', '3463']), 'classes': _log(rng, 10, 1000),
                'image': _log(rng, 64, 224), 'batch': _log(rng, 4, 32), 'graph': rng.random() < 0.5, 'every': 10}
    if kind == 'vgg_vi':
        return {'kind': kind, 'width': _log(rng, 8, 64), 'classes': _log(rng, 10, 100), 'batch': _log(rng, 16, 128), 'samples': rng.randint(1, 4)}
    if kind == 'vogn':
        return {'kind': kind, 'width': _log(rng, 8, 64), 'image': rng.randint(16, 32), 'classes': _log(rng, 4, 100), 'batch': _log(rng, 16, 128),
                'samples': rng.randint(1, 4)}
    if kind == 'layer':
        d = _log(rng, 64, 4608)
        return {'kind': kind, 'd_in': d, 'd_out': _log(rng, 10, 1024), 'bias': rng.random() < 0.5, 'rows': _log(rng, 512, min(401408, (1 << 27) // d))}
    return {'kind': kind, 'd': _log(rng, 16, 4608)}


# ------------------------------------------------------------------------------------------------ prepare
def _closure(opt, model, x, y):
    """The closure of the Cov curvatures and of the weight-sampling optimizers."""
    def closure():
        opt.zero_grad()
        out = model(x)
        loss = F.cross_entropy(out, y)
        loss.backward()
        return loss, out
    return closure


def _prepare_layer(case, gen):
    d, rows = case['d_in'], case['rows']
    layer = nn.Linear(d, case['d_out'], bias=case['bias']).cuda()
    curv = torchsso.KronCovLinear(layer, **CURV)
    # activations share a few directions, as those of a network do, over noise
    x = torch.randn((rows, d), device='cuda', generator=gen)
    x.addmm_(torch.randn((rows, 8), device='cuda', generator=gen), torch.randn((8, d), device='cuda', generator=gen), alpha=0.25)
    g = torch.randn((rows, case['d_out']), device='cuda', generator=gen) / rows
    return {'case': case, 'layer': layer, 'params': list(layer.parameters()), 'curv': curv, 'x': x, 'g': g}


def _prepare_linalg(case, gen):
    x = torch.randn((2 * case['d'], case['d']), device='cuda', generator=gen)
    m = x.t() @ x / x.shape[0]
    m.diagonal().add_(1e-2)
    return {'case': case, 'm': m}


def prepare(case, seed):
    torch.manual_seed(seed)
    gen = torch.Generator(device='cuda').manual_seed(seed)
    kind = case['kind']
    if kind == 'layer':
        return _prepare_layer(case, gen)
    if kind == 'linalg':
        return _prepare_linalg(case, gen)
    with torch.device('cuda'):
        model = build(case)
    if kind == 'mlp':
        x = torch.randn((case['batch'], case['f_in']), device='cuda', generator=gen)
    else:
        image = case.get('image', 32)
        x = torch.randn((case['batch'], 3, image, image), device='cuda', generator=gen)
    bf16 = kind == 'resnet' or case.get('bf16', False)
    if bf16:
        x = x.contiguous(memory_format=torch.channels_last)
    y = torch.randint(0, case['classes'], (case['batch'],), device='cuda', generator=gen)
    called = Autocast(model) if bf16 else model
    if kind == 'vgg_vi':
        opt = torchsso.optim.VIOptimizer(model, DATASET, 'Cov', SHAPES, CURV, lr=1e-3, num_mc_samples=case['samples'], kl_weighting=0.01)
    elif kind == 'vogn':
        opt = torchsso.optim.VOGN(model, DATASET, num_mc_samples=case['samples'])
    else:
        opt = torchsso.optim.SecondOrderOptimizer(model, case.get('curv', 'Fisher'), SHAPES, CURV, lr=1e-3,
                                                  momentum=case.get('momentum', 0.0), acc_steps=case.get('acc', 1))
    if kind in ('vgg_vi', 'vogn') or case.get('curv') == 'Cov':
        closure = _closure(opt, called, x, y)
    else:
        closure = torchsso.get_closure_for_fisher(opt, called, x, y, approx_type='mc', num_mc=1)
    s = {'case': case, 'opt': opt, 'steps': 0, 'batch': (x, y)}      # a captured closure reads its batch from these
    s['params'] = [p.data for g in opt.param_groups for p in g['params']]
    s['means'] = [m for g in opt.param_groups for m in g.get('mean', [])]
    s['start'] = [p.clone() for p in s['params']]
    if case.get('graph'):
        torchsso.utils.set_factor_batching(True)
        opt.fuse_ema = True
        opt.early_inverse = True
        opt.update_inv = True
        opt.step(closure=closure)
        torchsso.utils.set_curvature_stream(True)
        closure = torchsso.utils.GraphedClosure(opt, closure)
        torchsso.utils.set_curvature_stream(False)
        torchsso.utils.set_factor_batching(False)
    s['closure'] = closure
    torch.manual_seed(seed)
    return s


# ------------------------------------------------------------------------------------------------ run
def _run_layer(s):
    layer, curv, params = s['layer'], s['curv'], s['params']
    for p in params:
        p.grad = None
    layer(s['x']).backward(s['g'])
    curv.step(update_inv=True)
    curv.precondition_grad(params)
    return {'factors': curv.data, 'inverses': curv.inv, 'grads': [p.grad for p in params]}


def run(s):
    case = s['case']
    if case['kind'] == 'layer':
        return _run_layer(s)
    if case['kind'] == 'linalg':
        return {'inverse': torchsso.utils.inv(s['m']), 'cholesky': torchsso.utils.cholesky(s['m'])}
    opt = s['opt']
    with torch.no_grad():
        torch._foreach_copy_(s['means'] or s['params'], s['start'])
    opt.update_inv = s['steps'] % case.get('every', 1) == 0
    for _ in range(case.get('acc', 1)):
        loss, _ = opt.step(closure=s['closure'])
    s['steps'] += 1
    grads = [t.grad for t in (s['means'] or [p for g in opt.param_groups for p in g['params']])]
    if len(grads) > 31:         # more tensors than a caller wants to hold: one vector each
        return {'loss': loss, 'params': torch.cat([p.flatten() for p in s['params']]), 'grads': torch.cat([g.flatten() for g in grads])}
    out = {'loss': loss, 'params': s['params'], 'grads': grads}
    if len(grads) <= 10:
        out['averages'] = [group['curv'].ema for group in opt.param_groups]
        out['inverses'] = [group['curv'].inv for group in opt.param_groups]
    return out


# ------------------------------------------------------------------------------------------------ work, tolerance
def _layers(case):
    """(rows, d_A, d_G, elements of the input, elements of the output) of every Linear / Conv2d, and the
    elements that the BatchNorm layers put out."""
    with torch.device('meta'):
        model = build(case)
        x = torch.empty((case['batch'], case['f_in'])) if case['kind'] == 'mlp' else torch.empty((case['batch'], 3, case.get('image', 32), case.get('image', 32)))
    got, norm = [], [0]

    def hook(m, inp, out):
        if isinstance(m, nn.BatchNorm2d):
            norm[0] += out.numel()
        elif isinstance(m, (nn.Linear, nn.Conv2d)):
            w = m.weight
            d_a = w.numel() // w.shape[0] + (m.bias is not None)
            got.append((out.numel() // w.shape[0], d_a, w.shape[0], inp[0].numel(), out.numel()))
    for m in model.modules():
        m.register_forward_hook(hook)
    with torch.no_grad():
        model(x)
    return got, norm[0]


def work(case):
    """One pass: the model's own multiplications, one triangle of every factor, the inverse at d^3, the
    preconditioned gradient; activations and output gradients read by the curvature, averages read and written,
    parameters and gradients."""
    kind = case['kind']
    if kind == 'linalg':
        return {'bytes': 4 * 3 * case['d'] ** 2, 'flops': 4 / 3 * case['d'] ** 3}
    if kind == 'layer':
        layers, norm = [(case['rows'], case['d_in'] + case['bias'], case['d_out'], case['rows'] * case['d_in'], case['rows'] * case['d_out'])], 0
    else:
        layers, norm = _layers(case)
    elem = 2 if kind == 'resnet' or case.get('bf16') else 4
    passes, every = case.get('samples', case.get('acc', 1)), case.get('every', 1)
    sampling_pass = kind in ('resnet', 'convnet') or case.get('curv') == 'Fisher'
    flops, nbytes = 0.0, 2.0 * norm * elem * passes
    for rows, d_a, d_g, n_in, n_out in layers:
        once = (2 if kind == 'layer' else 8 if sampling_pass else 6) * rows * d_a * d_g
        nbytes += passes * elem * (n_in + n_out) + 4 * 4 * d_a * d_g
        if kind == 'vogn':
            flops += passes * (once + 2 * rows * d_a * d_g)
            nbytes += 4 * 4 * d_a * d_g
            continue
        flops += passes * (once + rows * (d_a ** 2 + d_g ** 2)) + (d_a ** 3 + d_g ** 3) / every + 2 * d_a * d_g * (d_a + d_g)
        nbytes += 4 * (d_a ** 2 + d_g ** 2) * (3 + 1 / every)
        if kind == 'vgg_vi':
            flops += (d_a ** 3 + d_g ** 3) / 3 + passes * d_a * d_g * (d_a + d_g)
            nbytes += 4 * (d_a ** 2 + d_g ** 2)
    return {'bytes': nbytes, 'flops': flops}


def tolerance(case):
    """What two correct fp32 implementations show: the inverse multiplies a factor's rounding by its condition
    number, most where a factor has fewer rows than columns (the Linear layers of a network at these batch
    sizes).  With bf16 activations the model's own backward pass rounds every gradient to eight bits, in an order
    that is not fixed.  A posterior draw feeds the last digits of the Cholesky factors back into the network of
    the next weight sample, and thirteen layers multiply them."""
    kind = case['kind']
    if kind == 'vgg_vi':
        return {'rel': 1e-2, 'max': 0.1}
    if kind == 'resnet' or case.get('bf16'):
        return {'rel': 5e-3, 'max': 0.2}
    if kind == 'linalg':
        return {'rel': 1e-4, 'max': 4e-3}
    return {'rel': 3e-4 if kind == 'layer' else 1e-3, 'max': 1e-2}
