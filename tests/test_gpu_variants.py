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


def test_targets_of_an_empty_batch(nat):
    from torchsso.curv.fisher import sample_targets
    for num_mc in (1, 2):
        t = sample_targets(torch.empty(0, 7, device='cuda'), num_mc)
        assert t.shape == (num_mc, 0) and t.dtype == torch.int64


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


def test_optimizer_tail_of_a_record_beyond_31_bits(nat):
    n = (1 << 31) + 5
    p, g = torch.ones(n, device='cuda'), torch.full((n,), 2.0, device='cuda')
    nat.optimizer_tail(nat.tail_records([(p, g, None, None, 1.0, 0.0, 1.0, 1.0, 0.5)], p.device, chunk=n))
    for t, want in ((p, -0.5), (g, 3.0)):
        lo, hi = torch.aminmax(t)
        assert (lo.item(), hi.item()) == (want, want)


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


# ---------------------------------------------------------------------------------- fp32 factors
def conv_ref(x, k, s, p, d, bias, weight=None):
    """sum_r w_r u_r u_r^T over the im2col rows in fp64, columns (c, kh, kw) and the ones column."""
    import torch.nn.functional as F
    u = F.unfold(x.double(), k, dilation=d, padding=p, stride=s).transpose(1, 2)
    if bias:
        u = torch.cat([u, torch.ones_like(u[..., :1])], -1)
    w = torch.ones(x.shape[0], dtype=torch.float64, device=x.device) if weight is None else weight.double()
    return torch.einsum('n,nri,nrj->ij', w, u, u)


# channels below eight (folded), not a multiple of eight, one tile / one pair / several pairs, strides, dilation
F32_CONVS = [(5, 3, 20, 19, (7, 7), (2, 2), (3, 3), (1, 1), False), (3, 1, 9, 9, (3, 3), (1, 1), (1, 1), (1, 1), True),
             (4, 7, 12, 10, (3, 2), (1, 2), (1, 0), (2, 1), True), (6, 11, 9, 9, (3, 3), (1, 1), (1, 1), (1, 1), True),
             (3, 64, 8, 8, (3, 3), (1, 1), (1, 1), (1, 1), True), (2, 26, 13, 13, (5, 5), (1, 1), (2, 2), (1, 1), False),
             (40, 33, 6, 6, (1, 1), (2, 2), (0, 0), (1, 1), True), (2, 9, 10, 10, (9, 9), (1, 1), (4, 4), (1, 1), True),
             (3, 21, 9, 8, (4, 4), (1, 1), (1, 1), (1, 1), False), (1, 40, 7, 7, (2, 2), (1, 1), (0, 0), (1, 1), True), (6, 128, 4, 4, (3, 3), (1, 1), (1, 1), (1, 1), True),
             (16, 64, 2, 2, (3, 3), (1, 1), (1, 1), (1, 1), False), (2, 64, 16, 33, (3, 2), (1, 1), (1, 0), (1, 1), True),
             (2, 64, 12, 24, (5, 5), (1, 1), (4, 4), (2, 2), True), (4, 200, 32, 32, (1, 1), (1, 1), (0, 0), (1, 1), True), (2, 128, 8, 8, (3, 2), (1, 1), (1, 1), (1, 1), True),
             (2, 256, 8, 8, (3, 3), (1, 1), (1, 1), (1, 1), True), (16, 130, 5, 7, (1, 1), (1, 1), (0, 0), (1, 1), True)]


@pytest.mark.parametrize('cfg', F32_CONVS)
@pytest.mark.parametrize('channels_last', [False, True])
def test_factor_f32_conv(nat, cfg, channels_last):
    n, c, h, w, k, s, p, d, bias = cfg
    x = torch.randn(n, c, h, w, device='cuda')
    x = x.contiguous(memory_format=torch.channels_last) if channels_last else x
    ref = conv_ref(x, k, s, p, d, bias)
    out = torch.randn_like(ref, dtype=torch.float32)
    want = 0.5 * ref + 2.0 * out.double()
    nat.factor_im2col(x, k, s, p, d, bias, None, 0.5, 2.0, out)
    assert rel(out, want) < 1e-6
    weight = torch.rand(n, device='cuda')
    nat.factor_im2col(x, k, s, p, d, bias, weight, 1.0, 0.0, out)
    assert rel(out, conv_ref(x, k, s, p, d, bias, weight)) < 1e-6
    assert torch.equal(out, out.t())


@pytest.mark.parametrize('n,c,h,w,stride,pad', [(2, 3, 5, 5, (1, 1), (1, 1)), (5, 20, 9, 9, (1, 1), (1, 1)), (3, 40, 7, 7, (2, 2), (1, 0)),
                                                (4, 200, 6, 7, (1, 1), (2, 1)), (8, 100, 6, 6, (1, 1), (1, 1)), (16, 192, 6, 6, (1, 1), (1, 1)),
                                                (16, 256, 6, 6, (1, 1), (1, 1)), (4, 127, 30, 30, (1, 1), (1, 1))])
@pytest.mark.parametrize('channels_last', [False, True])
def test_factor_f32_padded_1x1_with_bias(nat, n, c, h, w, stride, pad, channels_last):
    """Rows in the padding are zero but for the ones column: one tile, gathered pairs, boxes, a narrow last block row."""
    x = torch.randn(n, c, h, w, device='cuda') + 0.25
    x = x.contiguous(memory_format=torch.channels_last) if channels_last else x
    for weight in (None, torch.rand(n, device='cuda')):
        ref = conv_ref(x, (1, 1), stride, pad, (1, 1), True, weight)
        out = torch.full_like(ref, float('nan'), dtype=torch.float32)
        nat.factor_im2col(x, (1, 1), stride, pad, (1, 1), True, weight, 0.5, 0.0, out)
        assert rel(out, 0.5 * ref) < 1e-6 and torch.equal(out, out.t())
        assert rel(out[c], 0.5 * ref[c]) < 1e-5


@pytest.mark.parametrize('rows,cols,bias', [(1, 1, False), (31, 5, True), (129, 63, True), (700, 64, False), (5000, 64, True), (33000, 128, False),
                                            (20001, 97, True), (40000, 13, False), (257, 300, True), (256, 300, True), (1024, 1021, False), (256, 272, False), (288, 264, True), (512, 384, False), (128, 511, True), (320, 520, True), (1500, 1021, True), (33, 4100, False)])
@pytest.mark.parametrize('layout', ['rows', 'strided', 'columns'])
def test_factor_f32_rows(nat, rows, cols, bias, layout):
    x = torch.randn(rows, cols, device='cuda') + 0.25
    if layout == 'strided':
        x = torch.randn(rows, cols + 3, device='cuda')[:, 1:cols + 1]
    elif layout == 'columns':
        x = x.t().contiguous().t()
    u = x.double()
    if bias:
        u = torch.cat([u, torch.ones_like(u[:, :1])], 1)
    d = cols + int(bias)
    out = torch.full((d, d), float('nan'), device='cuda')
    nat.factor_rows(x, bias, None, 1.0 / rows, 0.0, out)
    assert rel(out, u.t() @ u / rows) < 1e-6 and torch.equal(out, out.t())


@pytest.mark.parametrize('n,c,size', [(37, 40, 10), (36, 64, 8)])
def test_factor_f32_in_runs(nat, n, c, size):
    """Scratch for a few images at a time: the runs add to the same partial tiles."""
    x = torch.randn(n, c, size, size, device='cuda')
    ref = conv_ref(x, (3, 3), (1, 1), (1, 1), (1, 1), True)
    d = ref.shape[0]
    for space in (1_100_000, 2_000_000, 64_000_000):
        out = torch.empty(d, d, device='cuda')
        ws = torch.empty(space, dtype=torch.uint8, device='cuda')
        nat._check(nat.lib().sso_factor_syrk_im2col(x.data_ptr(), nat.F32, n, c, size, size, *x.stride(), 3, 3, 1, 1, 1, 1, 1, 1, 1, None, 1.0, 0.0,
                                                    out.data_ptr(), d, ws.data_ptr(), space, nat.IMPL_AUTO, nat._stream()))
        assert rel(out, ref) < 1e-6


@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float16])
@pytest.mark.parametrize('rows,cols,bias', [(16, 20, True), (50, 65, False), (100, 129, True)])
def test_factor_direct_16bit(nat, rows, cols, bias, dtype):
    x = torch.randn(rows, cols, device='cuda').to(dtype)
    u = torch.cat([x.double(), torch.ones(rows, int(bias), device='cuda', dtype=torch.float64)], 1)
    d = cols + int(bias)
    out = torch.empty(d, d, device='cuda')
    nat.factor_rows(x, bias, None, 1.0, 0.0, out)
    assert rel(out, u.t() @ u) < 1e-6


# ----------------------------------------------------------------------- factorisation and inverse
FLOW_DIMS = [[1], [10, 127], [128], [129, 128], [256, 1, 257], [300, 640, 64, 31, 385, 512], [1153]]


def spd(d, ld, seed):
    g = torch.Generator(device='cuda').manual_seed(seed)
    x = torch.randn(3 * d + 8, d, device='cuda', generator=g)
    out = torch.full((d, ld), float('nan'), device='cuda')
    out[:, :d] = x.t() @ x / x.shape[0]
    return out[:, :d]


@pytest.mark.parametrize('std', [False, True])
@pytest.mark.parametrize('pad', [0, 3])
@pytest.mark.parametrize('dims', FLOW_DIMS)
def test_kron_plan_in_one_kernel(nat, dims, pad, std):
    """Tile edges, several matrices, odd row strides; the same bits from a second run."""
    src = [spd(d, d + pad, i) for i, d in enumerate(dims)]
    dst, work, sd = ([torch.full((d, d + pad), float('nan'), device='cuda')[:, :d] for d in dims] for _ in range(3))
    sd = sd if std else None
    n = len(dims)
    plan = nat.kron_plan(dims, src, dst, work, sd, [-1] * n, [0] * n, torch.device('cuda'))
    damp = torch.full((n,), 0.02, device='cuda')
    info = torch.zeros(2 * n, dtype=torch.int32, device='cuda')
    nat.kron_plan_run(plan, damp, info, True, std)
    first = [t.clone() for t in dst + (sd or [])]
    nat.kron_plan_run(plan, damp, info, True, std)
    assert not info.any()
    for t, f in zip(dst + (sd or []), first):
        assert torch.equal(t, f)
    for i, (m, out) in enumerate(zip(src, dst)):
        want = torch.linalg.inv(m.double() + 0.02 * torch.eye(dims[i], device='cuda', dtype=torch.float64))
        assert rel(out, want) < 1e-5 and torch.equal(out, out.t())
        if std:
            assert rel(sd[i], torch.linalg.cholesky(out.double(), upper=True)) < 1e-5
            assert torch.equal(sd[i], sd[i].triu())


@pytest.mark.parametrize('pad', [0, 1, 4])
def test_kron_plan_with_std_runs_either_half(nat, pad):
    """Sampling factors come with the inverse, which then goes from the last column to the first: every remainder modulo
    four columns (its padding), pairs with a shared shift, and the halves by themselves."""
    dims = [1, 2, 3, 5, 6, 7, 126, 130, 131, 255, 389, 258]
    n = len(dims)
    src = [spd(d, d + pad, i) for i, d in enumerate(dims)]
    dst, work, sd = ([torch.full((d, d + pad), 7.0, device='cuda')[:, :d] for d in dims] for _ in range(3))
    plan = nat.kron_plan(dims, src, dst, work, sd, [i ^ 1 for i in range(n)], [i & 1 for i in range(n)], torch.device('cuda'))
    damp = torch.full((n,), 0.1, device='cuda')
    info = torch.zeros(2 * n, dtype=torch.int32, device='cuda')
    nat.kron_plan_run(plan, damp, info, True, False)
    assert all(bool((u == 7.0).all()) for u in sd)
    nat.kron_plan_run(plan, damp, info, True, True)
    together = [u.clone() for u in sd]
    nat.kron_plan_run(plan, damp, info, False, True)
    assert not info.any()
    mean = [float(m.double().trace()) / d for m, d in zip(src, dims)]
    for i, d in enumerate(dims):
        shift = 0.1 * (mean[i] / mean[i ^ 1]) ** 0.5
        want = torch.linalg.inv(src[i].double() + shift * torch.eye(d, device='cuda', dtype=torch.float64))
        u = torch.linalg.cholesky(want, upper=True)
        assert rel(dst[i], want) < 1e-5 and rel(together[i], u) < 1e-5 and rel(sd[i], u) < 1e-5, d
        assert torch.equal(together[i], together[i].triu())
        if pad:      # nothing outside the matrices
            assert bool((sd[i]._base[:, d:] == 7.0).all()) and bool((dst[i]._base[:, d:] == 7.0).all())


@pytest.mark.parametrize('d', [1, 5, 64, 129, 300])
def test_inv_and_cholesky_read_the_matrix_where_it_lies(nat, d):
    import torchsso
    m = spd(d, d, d) + 0.1 * torch.eye(d, device='cuda')
    wide = torch.full((d, d + 8), float('nan'), device='cuda')
    views = [m, m.t(), m.double()]
    for first in (0, 1, 4):
        wide[:, first:first + d] = m
        views.append(wide.clone()[:, first:first + d])
    odd = torch.full((d, d + 3), float('nan'), device='cuda')
    odd[:, :d] = m
    views.append(odd[:, :d])
    inverse = torch.linalg.inv(m.double())
    upper = torch.linalg.cholesky(m.double(), upper=True)
    for v in views:
        before = v.clone()
        i, u, low = torchsso.utils.inv(v), torchsso.utils.cholesky(v), torchsso.utils.cholesky(v, upper=False)
        assert i.dtype == torch.float32 and i.is_contiguous() and rel(i, inverse) < 1e-5 and torch.equal(i, i.t())
        assert rel(u, upper) < 1e-5 and torch.equal(u, u.triu()) and torch.equal(low, u.t())
        assert torch.equal(v, before)
    plan, zero, info = torchsso.utils.linalg._solo(d, m.device, False)[0], torch.zeros(1, device='cuda'), torch.zeros(2, dtype=torch.int32, device='cuda')
    with pytest.raises(RuntimeError):
        nat.kron_plan_run_at(plan, zero, info, True, m, m)
    with pytest.raises(RuntimeError):
        nat.kron_plan_run_at(plan, zero, info, False, m, torch.empty_like(m))      # a plan without factors


@pytest.mark.parametrize('at', [0, 127, 128, 290])
def test_kron_plan_reports_the_bad_pivot(nat, at):
    """One matrix of three is not positive definite: its pivot is named and the others are as they would be without it."""
    dims = [130, 300, 64]
    src = [spd(d, d, i) for i, d in enumerate(dims)]
    src[1] = torch.eye(300, device='cuda')
    src[1][at, at] = -5.0
    dst = [torch.zeros(d, d, device='cuda') for d in dims]
    plan = nat.kron_plan(dims, src, dst, [torch.empty_like(m) for m in dst], None, [-1] * 3, [0] * 3, torch.device('cuda'))
    info = torch.zeros(6, dtype=torch.int32, device='cuda')
    nat.kron_plan_run(plan, torch.full((3,), 0.02, device='cuda'), info, True, False)
    assert info.tolist() == [0, 0, at + 1, 0, 0, 0]
    for i in (0, 2):
        want = torch.linalg.inv(src[i].double() + 0.02 * torch.eye(dims[i], device='cuda', dtype=torch.float64))
        assert rel(dst[i], want) < 1e-5


# ------------------------------------------------------------------------------- batch normalisation
@pytest.mark.parametrize('weighted', [False, True])
def test_bn_batch(nat, weighted):
    """Layers of every type and layout in one call, more of them than one launch holds."""
    shapes = [(4, 8, 5, 5), (4, 24, 3, 7), (4, 2048, 2, 2), (4, 64, 1, 1), (4, 7, 4, 4), (4, 12)] + [(4, 16, 9, 9)] * 70
    w = torch.rand(4, device='cuda') if weighted else None
    want, keep = [], []
    with nat.collect_factors():
        for i, shape in enumerate(shapes):
            dtype = (torch.float32, torch.bfloat16, torch.float16)[i % 3]
            g = torch.randn(shape, device='cuda').to(dtype)
            if len(shape) == 4 and i % 2 == 0:
                g = g.contiguous(memory_format=torch.channels_last)
            n, c = shape[:2]
            t, st, splits = nat.bn_plane_layout(g)
            sx = torch.rand(n, 2, c, device='cuda')
            sg = torch.empty(n * splits * c, device='cuda')
            wo, bo = torch.rand(c, device='cuda'), torch.rand(c, device='cuda') if i % 5 else None
            gs = g.double().reshape(n, c, -1).square().sum(-1) * (1.0 if w is None else w.double()[:, None])
            want.append((wo, 0.5 * (sx.double().sum(1) * gs).mean(0) + 2.0 * wo.double()))
            if bo is not None:
                want.append((bo, 0.5 * gs.mean(0) + 2.0 * bo.double()))
            keep.append((sx, sg))
            assert nat.collect_norm(t, (st, splits), sg, sx, w, 2, 0.5, 2.0, wo, bo)
    for got, ref in want:
        assert rel(got, ref) < 1e-5


# ------------------------------------------------------------------------------------------- sampling
@pytest.mark.parametrize('bias', [False, True])
@pytest.mark.parametrize('shapes', [[(1, 1)], [(128, 128)], [(129, 127), (130, 1)], [(2, 257), (641, 130), (388, 4)]])
def test_sample_plan_along_k(nat, shapes, bias):
    """[w | b] += s U_G E U_A with rows of the factors padded, and noise rows that do or do not start on 16 bytes."""
    shapes = [(a + int(bias), g) for a, g in shapes]

    def factor(d):
        ld = (d + 3) // 4 * 4
        u = torch.zeros(d, ld, device='cuda')
        u[:, :d] = torch.randn(d, d, device='cuda').triu()
        return u[:, :d]
    UA, UG = [factor(a) for a, _ in shapes], [factor(g) for _, g in shapes]
    E = [torch.randn(g, a, device='cuda') for a, g in shapes]
    w = [torch.randn(g, a - int(bias), device='cuda') for a, g in shapes]
    b = [torch.randn(g, device='cuda') if bias else None for _, g in shapes]
    tmp = [torch.empty(a * g, device='cuda') for a, g in shapes]
    want = []
    for i in range(len(shapes)):
        mean = w[i] if b[i] is None else torch.cat([w[i], b[i][:, None]], 1)
        want.append(mean.double() + 0.25 * UG[i].double() @ E[i].double() @ UA[i].double())
    plan = nat.sample_plan([a for a, _ in shapes], [g for _, g in shapes], UA, UG, E, w, b, tmp, torch.device('cuda'))
    nat.sample_plan_run(plan, 0.25)
    for i in range(len(shapes)):
        got = w[i] if b[i] is None else torch.cat([w[i], b[i][:, None]], 1)
        assert rel(got, want[i]) < 2e-6


# enough layers for blocks of 256 (more than two rounds of 128x128 tiles): blocks that are not full, down to a row or a column
# beyond the last whole one, layers without a block, rows that cannot be read with TMA
WIDE = [(260, 260), (384, 129), (513, 640), (1152, 385), (2308, 1024), (516, 255), (128, 640), (2304, 513), (641, 300), (256, 256)]


@pytest.mark.parametrize('bias', [False, True])
def test_sample_plan_in_wide_blocks(nat, bias, monkeypatch):
    make = nat.sample_plan

    def plan_of_nans(dA, *args):
        plan = make(dA, *args)
        plan._dev_mem[:dA[0] * ((dA[0] + 3) // 4 * 4) * 4].fill_(255)      # the first U_A^T: only what a run writes may be read
        assert any(k == 6 for k, _, _ in plan.phases())
        return plan
    monkeypatch.setattr(nat, 'sample_plan', plan_of_nans)
    test_sample_plan_along_k(nat, WIDE[4:5] + WIDE[:4] + WIDE[5:], bias)


@pytest.mark.parametrize('bias', [False, True])
def test_precond_plan_in_wide_blocks(nat, bias):
    assert any(k == 6 for k, _, _ in precond_in_wide_blocks(nat, bias).phases())


def precond_in_wide_blocks(nat, bias):
    shapes = [(a + int(bias), g) for a, g in WIDE]

    def inverse(d, seed):
        m = torch.full((d, (d + 3) // 4 * 4), float('nan'), device='cuda')
        x = torch.randn(d, d, device='cuda')
        m[:, :d] = x + x.t()
        return m[:, :d]
    A, G = [inverse(a, a) for a, _ in shapes], [inverse(g, g + 1) for _, g in shapes]
    w = [torch.randn(g, a - int(bias), device='cuda') for a, g in shapes]
    b = [torch.randn(g, device='cuda') if bias else None for _, g in shapes]
    tmp = [torch.empty(a * max(m.stride(0), g), device='cuda') for (a, g), m in zip(shapes, G)]
    want = []
    for i in range(len(shapes)):
        grad = w[i] if b[i] is None else torch.cat([w[i], b[i][:, None]], 1)
        want.append(G[i].double() @ grad.double() @ A[i].double())
    plan = nat.precond_plan([a for a, _ in shapes], [g for _, g in shapes], A, G, w, b, tmp, torch.device('cuda'))
    nat.precond_plan_run(plan)
    assert plan.status() == 0
    for i in range(len(shapes)):
        got = w[i] if b[i] is None else torch.cat([w[i], b[i][:, None]], 1)
        assert rel(got, want[i]) < 2e-6, shapes[i]
    return plan


@pytest.mark.parametrize('bias', [False, True])
def test_plans_in_wide_blocks_without_tensor_maps(nat, bias, monkeypatch):
    """Where the driver makes no map, such a plan runs in 128x128 tiles."""
    plans, make = [], nat.sample_plan
    monkeypatch.setattr(nat, 'sample_plan', lambda *a: (plans.append(make(*a)), plans[-1])[1])
    nat.configure('inject_no_maps', 1)
    try:
        plans.append(precond_in_wide_blocks(nat, bias))
        test_sample_plan_along_k(nat, WIDE, bias)
    finally:
        nat.configure('inject_no_maps', 0)
    assert len(plans) == 2 and not any(k == 6 for plan in plans for k, _, _ in plan.phases())


@pytest.mark.parametrize('cfg', [(128, 4096, 1, 1, (1, 1), (1, 1), (0, 0), (1, 1), True), (1, 300, 1, 1, (1, 1), (1, 1), (0, 0), (1, 1), False),
                                 (4, 512, 7, 7, (3, 3), (1, 1), (1, 1), (1, 1), True), (1, 256, 40, 40, (1, 1), (2, 2), (0, 0), (1, 1), False),
                                 (2, 4, 30, 30, (11, 11), (4, 4), (2, 2), (1, 1), True), (1, 64, 224, 224, (3, 3), (1, 1), (1, 1), (1, 1), False)])
@pytest.mark.parametrize('weighted', [False, True])
def test_factor_f32_with_the_scratch_that_a_caller_asks_for(nat, cfg, weighted):
    """sso_factor_workspace_bytes knows rows and columns only; the tensor-core path takes what it gives."""
    n, c, h, w, k, s, p, d, bias = cfg
    x = torch.randn(n, c, h, w, device='cuda').contiguous(memory_format=torch.channels_last)
    weight = torch.rand(n, device='cuda') if weighted else None
    ref = conv_ref(x, k, s, p, d, bias, weight)
    cols = ref.shape[0]
    ho, wo = (h + 2 * p[0] - k[0]) // s[0] + 1, (w + 2 * p[1] - k[1]) // s[1] + 1
    space = nat.lib().sso_factor_workspace_bytes(n * ho * wo, cols, nat.IMPL_TCGEN05)
    ws, out = torch.empty(space, dtype=torch.uint8, device='cuda'), torch.empty(cols, cols, device='cuda')
    st = (x.stride(0), 1, x.stride(2), x.stride(3))
    nat._check(nat.lib().sso_factor_syrk_im2col(x.data_ptr(), nat.F32, n, c, h, w, *st, *k, *s, *p, *d, int(bias), nat._ptr(weight), 1.0, 0.0,
                                                out.data_ptr(), cols, ws.data_ptr(), space, nat.IMPL_TCGEN05, nat._stream()))
    assert rel(out, ref) < 1e-6


# ------------------------------------------------------------------------------------------- lifetime
def test_an_optimizer_gives_its_buffers_back_when_it_goes(nat):
    """No reference cycle through hooks and pools; a copy of a hooked model has no curvature."""
    import copy
    import gc
    import torchsso
    model = torch.nn.Sequential(torch.nn.Linear(300, 200), torch.nn.Unflatten(1, (8, 5, 5)), torch.nn.BatchNorm2d(8), torch.nn.Flatten(),
                                torch.nn.Linear(200, 10)).cuda()
    x, y = torch.randn(64, 300, device='cuda'), torch.randint(0, 10, (64,), device='cuda')

    def step():
        opt = torchsso.optim.SecondOrderOptimizer(model, 'Fisher', {'Linear': 'Kron', 'BatchNorm2d': 'Diag'}, {'damping': 1e-2})
        opt.step(closure=torchsso.get_closure_for_fisher(opt, model, x, y, approx_type='mc', num_mc=1))
        copy.deepcopy(model)(x)
        return opt
    for p in model.parameters():
        p.grad = None
    gc.collect()
    gc.disable()
    try:
        held = []
        for _ in range(3):
            opt = step()
            torch.cuda.synchronize()
            del opt
            for p in model.parameters():
                p.grad = None
            held.append(torch.cuda.memory_allocated())
    finally:
        gc.enable()
    assert held[2] <= held[1] + (1 << 16), held


# ------------------------------------------------------------------------------------------- closures
def test_every_closure_call_brings_its_own_weights(nat):
    import torchsso
    model = torch.nn.Linear(6, 4).cuda()
    model.num_classes = 4
    x, y = torch.randn(8, 6, device='cuda'), torch.randint(0, 4, (8,), device='cuda')
    opt = torchsso.optim.SecondOrderOptimizer(model, 'Fisher', {'Linear': 'Kron'}, {'damping': 1e-2})
    closure = torchsso.get_closure_for_fisher(opt, model, x, y, approx_type='mc', num_mc=2)
    curv = opt.param_groups[0]['curv']
    for _ in range(2):
        opt.step(closure=closure)
        assert torch.equal(curv.prob, torch.full((8,), 0.5, device='cuda'))
        curv.prob.zero_()


# ------------------------------------------------------------------------------------------- variational step
def test_vi_step_at_fixed_draws(nat, monkeypatch):
    """The second step of a thirteen-layer stack, which draws its weights, piece by piece against fp64 at the draws that it
    made: a draw feeds the last digits of a Cholesky factor into the network, so two runs are not comparable."""
    import torch.nn as nn
    import torch.nn.functional as F
    import torchsso
    torch.manual_seed(0)
    layers, cin = [], 3
    for c, count in ((6, 2), (12, 2), (20, 3), (24, 3), (24, 3)):
        for _ in range(count):
            layers += [nn.Conv2d(cin, c, 3, padding=1), nn.Tanh()]
            cin = c
        layers.append(nn.AvgPool2d(2))
    model = nn.Sequential(*layers, nn.Flatten(), nn.Linear(24, 10)).cuda()
    x, y = torch.randn(8, 3, 32, 32, device='cuda'), torch.randint(0, 10, (8,), device='cuda')
    opt = torchsso.optim.VIOptimizer(model, 500, 'Cov', {'Linear': 'Kron', 'Conv2d': 'Kron'}, {'ema_decay': 0.9, 'damping': 1e-2},
                                     lr=0.05, num_mc_samples=2)
    groups, noise, draws, losses = opt.param_groups, [], [], []
    randn_like = torch.randn_like
    monkeypatch.setattr(torch, 'randn_like', lambda t: (noise.append(randn_like(t)), noise[-1])[1])

    def closure():
        opt.zero_grad()
        draws.append([[p.detach().double() for p in g['params']] for g in groups])
        out = model(x)
        loss = F.cross_entropy(out, y)
        loss.backward()
        losses.append(loss.detach())
        return loss, out

    def flat(ts):
        return torch.cat([ts[0].double().flatten(1)] + [t.double()[:, None] for t in ts[1:]], 1)
    with torch.backends.cudnn.flags(allow_tf32=False):
        opt.step(closure=closure)
        std = [[u.double() for u in g['curv'].std] for g in groups]
        mean = [flat(g['mean']) for g in groups]
        for seen in (noise, draws, losses):
            seen.clear()
        opt.step(closure=closure)
    ref = nn.Sequential(*[type(m)(*((m.in_features, m.out_features) if isinstance(m, nn.Linear) else (m.in_channels, m.out_channels, 3, 1, 1)))
                          if hasattr(m, 'weight') else m for m in model]).double().cuda()
    ref_layers = [m for m in ref if hasattr(m, 'weight')]
    grad_sum, a_sum, g_sum = [], [0.0] * len(groups), [0.0] * len(groups)
    for i, draw in enumerate(draws):
        for j, (g, (ua, ug)) in enumerate(zip(groups, std)):
            e = noise[i * len(groups) + j].double()
            assert rel(flat(draw[j]) - mean[j], g['std_scale'] * ug @ e @ ua) < 1e-5      # of the difference of two fp32 numbers
            with torch.no_grad():
                ref_layers[j].weight.copy_(draw[j][0])
                ref_layers[j].bias.copy_(draw[j][1])
        h, ins, outs = x.double(), [], []
        for m in ref:
            if m in ref_layers:
                ins.append(h)
            h = m(h)
            if m in ref_layers:
                outs.append(h)
        loss = F.cross_entropy(h, y)
        assert abs(losses[i].item() - loss.item()) < 1e-6 * abs(loss.item())
        params = [p for m in ref_layers for p in (m.weight, m.bias)]
        got = torch.autograd.grad(loss, params + outs)
        grad_sum = [a + b / 2 for a, b in zip(grad_sum or [0.0] * len(params), got)]
        for j, (u, g) in enumerate(zip(ins, got[len(params):])):
            n = u.shape[0]
            if u.dim() == 4:
                a = conv_ref(u, (3, 3), (1, 1), (1, 1), (1, 1), True) / n
                gg = g.permute(0, 2, 3, 1).reshape(-1, g.shape[1])
            else:
                a, gg = conv_ref(u[:, :, None, None], (1, 1), (1, 1), (0, 0), (1, 1), True) / n, g
            a_sum[j] = a_sum[j] + a / 2
            g_sum[j] = g_sum[j] + gg.t() @ gg / gg.shape[0] * n * n / 2
    for j, g in enumerate(groups):
        a, gg = g['curv'].data
        assert rel(a, a_sum[j]) < 1e-5 and rel(gg, g_sum[j]) < 1e-4, j
        ia, ig = (m.double() for m in g['curv'].inv)
        raw = flat(grad_sum[2 * j:2 * j + 2]) + g['l2_reg'] * mean[j]
        assert rel(flat(g['mean']) - mean[j], -0.05 * ig @ raw @ ia) < 1e-3, j

# ------------------------------------------------------------------------------------------- accumulation
@pytest.mark.parametrize('numel,shift', [(3, 0), (4097, 0), (100003, 1)])
@pytest.mark.parametrize('scale', [1 / 3, 1 / 6, 0.2, 0.5])
def test_a_scaled_sum_is_rounded_once_whichever_side_it_lies_on(nat, numel, shift, scale):
    terms, total = torch.randn(numel + shift, device='cuda')[shift:], torch.randn(numel + shift, device='cuda')[shift:]
    want = total.clone()
    nat.axpby(terms, want, scale, 1.0)
    nat.axpby(total, terms, 1.0, scale)
    assert torch.equal(terms, want)


@pytest.mark.parametrize('samples,micro_steps', [(0, 3), (1, 1), (1, 3), (3, 1), (5, 2)])
def test_the_closures_of_a_step_are_added_one_by_one(nat, monkeypatch, samples, micro_steps):
    """Gradients and factors of a step against the fp64 sum over its closures (weight samples, micro-steps, both): one fused
    multiply-add for each."""
    import torch.nn as nn
    import torch.nn.functional as F
    import torchsso
    model = nn.Sequential(nn.Linear(200, 300), nn.Tanh(), nn.Linear(300, 10)).cuda()
    x, y = torch.randn(64, 200, device='cuda'), torch.randint(0, 10, (64,), device='cuda')
    shapes, kw = {'Linear': 'Kron'}, {'ema_decay': 0.9, 'damping': 1e-2}
    if samples:
        opt = torchsso.optim.VIOptimizer(model, 500, 'Cov', shapes, kw, lr=1e-3, num_mc_samples=samples, acc_steps=micro_steps)
    else:
        opt = torchsso.optim.SecondOrderOptimizer(model, 'Cov', shapes, kw, lr=1e-3, acc_steps=micro_steps)
    n = max(samples, 1) * micro_steps
    scale = torch.tensor(1 / max(samples, 1) / micro_steps, dtype=torch.float32).double().item()      # the kernels' scale
    terms, sums = [], []
    accumulate, take = opt._accumulate, opt._take_accumulated

    def both():
        return torch.cat([opt._grad_flat, *(m.flatten() for g in opt.param_groups for m in g['curv'].data)])
    monkeypatch.setattr(opt, '_accumulate', lambda *a, **k: (terms.append(both()), accumulate(*a, **k)))
    monkeypatch.setattr(opt, '_take_accumulated', lambda *a, **k: (take(*a, **k), sums.append(both())))

    def closure():
        opt.zero_grad()
        out = model(x[torch.randperm(64, device='cuda')[:32]])
        loss = F.cross_entropy(out, y[:32])
        loss.backward()
        return loss, out
    for step in range(2):
        terms.clear()
        sums.clear()
        for _ in range(micro_steps):
            opt.step(closure=closure)
        assert len(terms) == n and len(sums) == 1
        fused = (scale * terms[0].double()).float()
        for t in terms[1:]:
            fused = (scale * t.double() + fused.double()).float()
        exact = sum(scale * t.double() for t in terms)
        assert (sums[0] != fused).double().mean() < 1e-4      # but for what a second rounding of the emulation does
        assert rel(sums[0], exact) < 1.01 * rel(fused, exact) + 1e-12

# ------------------------------------------------------------------------------------------- one matrix
def test_inv_and_cholesky_of_many_sizes_keep_their_plans(nat, monkeypatch):
    """A dozen sizes, each inverted and factored: their plans are made once, and hold little beside their scratch."""
    import torchsso
    from torchsso.utils import linalg
    made, make = [], nat.kron_plan
    monkeypatch.setattr(nat, 'kron_plan', lambda dims, *a, **k: (made.append(dims[0]), make(dims, *a, **k))[1])
    mats = [spd(d, d, d) + 0.1 * torch.eye(d, device='cuda') for d in range(200, 212)]
    linalg._cache.clear()
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    for _ in range(3):
        for m in mats:
            assert rel(torchsso.utils.inv(m), torch.linalg.inv(m.double())) < 1e-5
            assert rel(torchsso.utils.cholesky(m), torch.linalg.cholesky(m.double(), upper=True)) < 1e-5
    assert len(made) == 2 * len(mats), made
    # two plans of a size: a scratch matrix, two diagonal blocks, tables
    assert torch.cuda.memory_allocated() - before < sum(2 * (212 * 212 + 2 * 128 * 128) * 4 + (96 << 10) for _ in mats)
    for d in range(300, 360):      # the cache has a limit
        torchsso.utils.inv(torch.eye(d, device='cuda'))
    assert len(linalg._cache) <= 40


def test_inv_and_cholesky_of_a_negated_view(nat):
    import torchsso
    m = spd(130, 130, 0) + 0.1 * torch.eye(130, device='cuda')
    v = torch._neg_view(-m)
    assert v.is_neg() and torch.equal(v, m)
    assert torch.equal(torchsso.utils.inv(v), torchsso.utils.inv(m))
    assert torch.equal(torchsso.utils.cholesky(v), torchsso.utils.cholesky(m))


@pytest.mark.parametrize('kind', ['inverse', 'precondition', 'sample'])
def test_a_plan_made_on_a_stream_of_its_own(nat, kind):
    """Its memory was a tensor's before, whose last kernel is still queued on that stream: the tables come behind it."""
    d = 640
    a, g, e = spd(d, d, 0) + torch.eye(d, device='cuda'), spd(d, d, 1), torch.randn(d, d, device='cuda')
    dims, device, zero = nat._i64([d]), torch.device('cuda'), torch.zeros(1, device='cuda')
    ua, ug, w, out, tmp = a.triu(), g.triu(), torch.zeros(d, d, device='cuda'), torch.empty(d, d, device='cuda'), torch.empty(d * d, device='cuda')
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        nbytes = (nat.lib().sso_kron_plan_dev_bytes(1, dims, 0) if kind == 'inverse' else
                  nat.lib().sso_precond_plan_dev_bytes(1, dims, dims) if kind == 'precondition' else
                  nat.lib().sso_sample_plan_dev_bytes(1, dims, dims))
        before = torch.empty(nbytes, dtype=torch.uint8, device='cuda')
        address = before.data_ptr()
        torch.cuda._sleep(40000000)
        before.fill_(255)
        del before
        if kind == 'inverse':
            plan = nat.kron_plan([d], [a], [out], [tmp.view(d, d)], None, [-1], [0], device)
            nat.kron_plan_run(plan, zero, None, True, False)
        elif kind == 'precondition':
            w.copy_(e)
            plan = nat.precond_plan([d], [d], [a], [g], [w], [None], [tmp], device)
            nat.precond_plan_run(plan)
        else:
            plan = nat.sample_plan([d], [d], [ua], [ug], [e], [w], [None], [tmp] if nat.sample_plan_uses_tmp() else None, device)
            nat.sample_plan_run(plan, 0.5)
    assert plan._dev_mem.data_ptr() == address      # the case that is meant
    stream.synchronize()
    a, g, e, ua, ug = (t.double() for t in (a, g, e, ua, ug))
    if kind == 'inverse':
        assert rel(out, torch.linalg.inv(a)) < 1e-5
    else:
        assert rel(w, g @ e @ a if kind == 'precondition' else 0.5 * ug @ e @ ua) < 2e-6


@pytest.mark.parametrize('threads', [False, True])
@pytest.mark.parametrize('d', [64, 500])
def test_inv_and_cholesky_on_several_streams(nat, d, threads):
    """Different matrices of one size on two streams at a time, issued by one thread or by one for each."""
    import threading
    import torchsso
    mats = [spd(d, d, i) + (0.1 + i) * torch.eye(d, device='cuda') for i in range(4)]
    want = [(torchsso.utils.inv(m), torchsso.utils.cholesky(m)) for m in mats]
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream(), torch.cuda.Stream()], {}

    def work(s, repeats):
        with torch.cuda.stream(streams[s]):
            for r in range(repeats):
                for i in (s, s + 2):
                    got[s, r, i] = torchsso.utils.inv(mats[i]), torchsso.utils.cholesky(mats[i])
    if threads:
        workers = [threading.Thread(target=work, args=(s, 25)) for s in range(2)]
        for t in workers:
            t.start()
        for t in workers:
            t.join()
    else:
        for r in range(25):
            for s in range(2):
                work(s, 1)
                got.update({(s, r + 1, i): got[s, 0, i] for i in (s, s + 2)})
    torch.cuda.synchronize()
    assert len(got) >= 100
    for (s, r, i), (a, u) in got.items():
        assert torch.equal(a, want[i][0]) and torch.equal(u, want[i][1])


def test_inv_in_a_graph_keeps_its_plan(nat):
    """Replayed after other sizes have been through the cache, and beside calls of the same size."""
    import torchsso
    from torchsso.utils import linalg
    d = 150
    m = spd(d, d, 0) + 0.1 * torch.eye(d, device='cuda')
    torchsso.utils.inv(m)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = torchsso.utils.inv(m)
    for size in range(400, 400 + linalg._LIMIT + 1):
        torchsso.utils.inv(torch.eye(size, device='cuda'))
    for i in range(3):
        fresh = spd(d, d, i) + 0.1 * torch.eye(d, device='cuda')
        m.copy_(fresh)
        graph.replay()
        other = torchsso.utils.inv(2 * fresh)
        want = torch.linalg.inv(fresh.double())
        assert rel(out, want) < 1e-5 and rel(other, want / 2) < 1e-5
    assert (d, m.device.index, False) in linalg._cache and (d, m.device.index, False) in linalg._captured


@pytest.mark.parametrize('flow', [1, 0])
@pytest.mark.parametrize('std', [False, True])
@pytest.mark.parametrize('pad', [0, 1, 4])
def test_kron_plan_reads_the_lower_triangle(nat, std, pad, flow):
    """Nothing above the diagonal is looked at, with sampling factors (in reverse order) or without."""
    nat.configure('flow', flow)
    try:
        _lower_triangle(nat, std, pad)
    finally:
        nat.configure('flow', 1)


def _lower_triangle(nat, std, pad):
    dims = [1, 2, 5, 16, 66, 127, 129, 130, 257, 400]
    full = [spd(d, d + pad, i) for i, d in enumerate(dims)]
    src = []
    for m, d in zip(full, dims):
        lower = torch.full((d, d + pad), float('nan'), device='cuda')[:, :d]
        i, j = torch.tril_indices(d, d, device='cuda')
        lower[i, j] = m[i, j]
        src.append(lower)
    dst, work, sd = ([torch.full((d, d + pad), 7.0, device='cuda')[:, :d] for d in dims] for _ in range(3))
    plan = nat.kron_plan(dims, src, dst, work, sd if std else None, [-1] * len(dims), [0] * len(dims), torch.device('cuda'))
    info = torch.zeros(2 * len(dims), dtype=torch.int32, device='cuda')
    nat.kron_plan_run(plan, torch.full((len(dims),), 0.1, device='cuda'), info, True, std)
    assert not info.any()
    for i, d in enumerate(dims):
        want = torch.linalg.inv(full[i].double() + 0.1 * torch.eye(d, device='cuda', dtype=torch.float64))
        assert rel(dst[i], want) < 1e-5, d
        if std:
            assert rel(sd[i], torch.linalg.cholesky(want, upper=True)) < 1e-5, d


@pytest.mark.parametrize('d', [1, 8, 9, 17, 130, 300])
@pytest.mark.parametrize('top', [126.0, 127.5])
def test_factors_of_a_matrix_near_the_largest_float(nat, d, top):
    """Pivots above 2^126, whose reciprocals are no normal numbers, among others of 2^-20."""
    import torchsso
    scale = torch.where(torch.arange(d, device='cuda') % 3 == 1, 2.0 ** -10, 2.0 ** (top / 2)).double()
    m = (spd(d, d, d) + torch.eye(d, device='cuda')).double()
    m = m / m.diagonal().max()
    m = (scale[:, None] * m * scale).float()
    got, want = torchsso.utils.cholesky(m), torch.linalg.cholesky(m.double(), upper=True)
    assert bool(got.isfinite().all())
    assert rel(got.double() / scale, want / scale) < 1e-5      # column by column: U diag(1 / scale)


def test_phases_launched_early_see_the_phase_before(nat):
    """The factorisation by launches, where 64-wide products follow one another on the same matrix: the same bits every time."""
    dims = [1100, 700, 321, 65]
    src = [spd(d, d, i) for i, d in enumerate(dims)]
    dst, work, sd = ([torch.empty(d, d, device='cuda') for d in dims] for _ in range(3))
    nat.configure('flow', 0)
    nat.configure('chol_panel', 0)      # diagonal blocks by 64-wide halves
    try:
        plan = nat.kron_plan(dims, src, dst, work, sd, [-1] * 4, [0] * 4, torch.device('cuda'))
        kinds = [k for k, _, _ in plan.phases()]
        assert any(a == b == 0 for a, b in zip(kinds, kinds[1:]))
        damp, info, first = torch.full((4,), 0.1, device='cuda'), torch.zeros(8, dtype=torch.int32, device='cuda'), None
        for _ in range(20):
            for m in work:
                m.fill_(float('nan'))
            nat.kron_plan_run(plan, damp, info, True, True)
            got = [m.clone() for m in dst + sd]
            first = first or got
            assert all(torch.equal(a, b) for a, b in zip(got, first))
    finally:
        nat.configure('flow', 1)
        nat.configure('chol_panel', 1)
    for m, d, a, u in zip(src, dims, dst, sd):
        want = torch.linalg.inv(m.double() + 0.1 * torch.eye(d, device='cuda', dtype=torch.float64))
        assert rel(a, want) < 1e-5 and rel(u, torch.linalg.cholesky(want, upper=True)) < 1e-5


def test_weight_samples_hold_the_noise_of_some_layers(nat):
    """What a draw allocates is 32 MB of noise on its way to where it is kept: two of these five layers."""
    import torch.nn as nn
    import torch.nn.functional as F
    import torchsso
    model = nn.Sequential(*[nn.Linear(2000, 2000, bias=i % 2 == 0) for i in range(5)], nn.Linear(2000, 10)).cuda()
    x, y = torch.randn(32, 2000, device='cuda'), torch.randint(0, 10, (32,), device='cuda')
    opt = torchsso.optim.VIOptimizer(model, 500, 'Cov', {'Linear': 'Kron'}, {'ema_decay': 0.9, 'damping': 1e-2}, lr=1e-3, num_mc_samples=1)

    def closure():
        opt.zero_grad()
        out = model(x)
        loss = F.cross_entropy(out, y)
        loss.backward()
        return loss, out
    opt.step(closure=closure)
    opt.sample_params()
    torch.manual_seed(3)
    opt.sample_params()
    drawn = [p.clone() for p in model.parameters()]
    torch.manual_seed(3)
    want = [torch.randn_like(opt._noise_buf(g)) for g in opt.param_groups]
    torch.manual_seed(3)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    opt.sample_params()
    torch.cuda.synchronize()
    assert torch.cuda.max_memory_allocated() - before < 36 << 20      # blocks of the allocator may be larger; all layers: 80 MB
    assert all(torch.equal(p, q) for p, q in zip(model.parameters(), drawn))
    assert all(torch.equal(opt._noise_buf(g), e) for g, e in zip(opt.param_groups, want))


def test_copies_of_tensors_of_several_types(nat):
    from torchsso.optim.vi import _copy_all
    source = [torch.randn(n, device='cuda').to(t) for n, t in ((5, torch.float32), (3, torch.bfloat16), (7, torch.float32), (1, torch.float64))]
    to = [torch.zeros(s.shape, device='cuda', dtype=t) for s, t in zip(source, (torch.float32, torch.bfloat16, torch.bfloat16, torch.float32))]
    _copy_all(to, source)
    _copy_all([], [])
    assert all(torch.equal(t, s.to(t.dtype)) for t, s in zip(to, source))
