"""The workloads this package is measured on.

Each case is one call (or one training step, one solver run) through the
public API: structured operators applied to device tensors or numpy arrays.
``listed()`` names the fixed ones, ``draw(rng)`` gives more of the same
families over the sizes they stand for.
"""

import math

import numpy as np
import torch

import fastmat_gb300 as fm
from fastmat_gb300.algorithms import FISTA
from fastmat_gb300.autograd import Operator


def listed():
    return [
        # a small filter applied to a handful of signals: latency-bound
        dict(name='circulant_1024_c128', kind='circulant', n=1024, cols=16,
             dtype='complex128', direction='forward'),
        # the drop-in numpy call on measured real data, ragged sizes
        dict(name='toeplitz_numpy_f64', kind='toeplitz', rows=3000,
             n=5001, cols=12, dtype='float64', direction='forward'),
        # spectrum of records of a prime length (chirp transform)
        dict(name='fourier_65521_c128', kind='fourier', n=65521, cols=8,
             dtype='complex128', direction='forward'),
        # inverse spectra of a length with odd factors, single precision
        dict(name='fourier_6000_c64', kind='fourier', n=6000, cols=64,
             dtype='complex64', direction='backward'),
        # three-way separable operator, the plain FP64 form
        dict(name='kron_2e23_c128', kind='kron', f=256, h=8, c=128, cols=8,
             dtype='complex128', direction='forward'),
        # the same operator's adjoint in the single-precision form
        dict(name='kron_2e23_c64', kind='kron', f=256, h=8, c=128, cols=8,
             dtype='complex64', direction='backward'),
        # long Walsh-Hadamard transforms of many columns, the largest call
        dict(name='hadamard_22_f32', kind='hadamard', order=22, cols=64,
             dtype='float32', direction='forward'),
        # the same transform in FP64 on medium columns
        dict(name='hadamard_18_f64', kind='hadamard', order=18, cols=48,
             dtype='float64', direction='forward'),
        # compressed-sensing measurement of long signals, FP64 adjoint
        dict(name='chain_2e18_c128', kind='chain', n=1 << 18, cols=32,
             dtype='complex128', direction='backward'),
        # the same chain with learned c and d: one training step
        dict(name='train_2e18_c64', kind='train', n=1 << 18, cols=32,
             dtype='complex64', direction='both'),
        # many operators of uneven sizes, one launch replayed as a graph
        dict(name='batch_64_c64', kind='batch', ops=64, mix=7,
             dtype='complex64', direction='forward'),
        # sparse deconvolution: a solver calling forward and backward
        dict(name='fista_4096_c128', kind='fista', n=4096, cols=4, steps=20,
             dtype='complex128', direction='both'),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """A power of two half of the time, any integer otherwise."""
    n = _log(rng, lo, hi)
    if rng.random() < 0.5:
        n = 1 << int(round(math.log2(n)))
    return min(max(n, lo), hi)


def draw(rng):
    kind = rng.choice(['circulant', 'toeplitz', 'fourier', 'kron',
                       'hadamard', 'chain', 'train', 'batch', 'fista'])
    case = dict(kind=kind, dtype=rng.choice(['complex128', 'complex64']),
                direction=rng.choice(['forward', 'backward']))
    if kind in ('circulant', 'fourier'):
        case.update(n=_size(rng, 64, 1 << 18), cols=rng.randint(1, 64))
    elif kind == 'toeplitz':
        case.update(rows=_log(rng, 100, 60000), n=_log(rng, 100, 60000),
                    cols=rng.randint(1, 32), dtype='float64')
    elif kind == 'kron':
        f, c = _size(rng, 16, 512), _size(rng, 16, 512)
        h = rng.randint(3, 8)
        while f * c << h > 1 << 23:
            h -= 1
        case.update(f=f, h=h, c=c, cols=rng.randint(1, 8))
    elif kind == 'hadamard':
        order = rng.randint(8, 22)
        case.update(order=order, cols=rng.randint(1, 32),
                    dtype=rng.choice(['float32', 'float64']))
    elif kind in ('chain', 'train'):
        case.update(n=_size(rng, 1 << 10, 1 << 18), cols=rng.randint(1, 32))
        if kind == 'train':
            case.update(direction='both')
    elif kind == 'batch':
        case.update(ops=rng.randint(16, 64), mix=rng.randint(0, 10 ** 6),
                    dtype='complex64', direction='forward')
    else:
        case.update(n=_size(rng, 256, 1 << 14), cols=rng.randint(1, 8),
                    steps=rng.randint(5, 20), dtype='complex128',
                    direction='both')
    return case


# ------------------------------------------------------------------ inputs
def _gauss(rng, n):
    return rng.standard_normal(n) + 1j * rng.standard_normal(n)


def _columns(n, cols, dtype, seed):
    """A column-major (n, cols) device tensor of iid N(0, 1) entries."""
    gen = torch.Generator(device='cuda')
    gen.manual_seed(1000 + seed)
    dt = getattr(torch, dtype)
    if dt.is_complex:
        real = torch.float32 if dt == torch.complex64 else torch.float64
        v = torch.randn((cols, n, 2), generator=gen, device='cuda',
                        dtype=real)
        return torch.view_as_complex(v).t()
    return torch.randn((cols, n), generator=gen, device='cuda', dtype=dt).t()


def _precision(case):
    return ('fp32' if case['dtype'] in ('float32', 'complex64')
            else 'native')


def _chain_data(case, seed):
    """(c, d, rows) of Partial(rows) * Circulant(c) * Diag(d)."""
    rng = np.random.default_rng(seed)
    n = case['n']
    rows = np.sort(rng.permutation(n)[:max(1, n // 4)])
    return _gauss(rng, n), _gauss(rng, n), rows


def _batch_specs(case):
    """(kind, size, right-hand sides) of every operator of a batch."""
    rng = np.random.default_rng(case['mix'])
    specs = []
    for _ in range(case['ops']):
        n = int(np.exp(rng.uniform(np.log(64), np.log(65536))))
        if rng.random() >= 0.3:
            n = 1 << int(round(np.log2(n)))
        specs.append((('circulant', 'toeplitz', 'fourier')[rng.integers(3)],
                      n, int(rng.integers(1, 33))))
    return specs


def _batch_vectors(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for kind, n, _ in _batch_specs(case):
        if kind == 'circulant':
            out.append((_gauss(rng, n),))
        elif kind == 'toeplitz':
            out.append((_gauss(rng, n), _gauss(rng, n - 1)))
        else:
            out.append(())
    return out


def _toeplitz_data(case, seed):
    rng = np.random.default_rng(seed)
    return (rng.standard_normal(case['rows']),
            rng.standard_normal(case['n'] - 1))


def _fista_data(case, seed):
    """A decaying echo filter and observations of sparse spike trains."""
    rng = np.random.default_rng(seed)
    n, m = case['n'], case['cols']
    taps = max(8, n // 64)
    c = np.zeros(n, dtype=np.complex128)
    c[:taps] = _gauss(rng, taps) * np.exp(-np.arange(taps) / (taps / 4.0))
    c[0] += 4.0
    x = np.zeros((n, m), dtype=np.complex128)
    for k in range(m):
        at = rng.permutation(n)[:max(1, n // 64)]
        x[at, k] = _gauss(rng, at.size)
    b = np.fft.ifft(np.fft.fft(c)[:, None] * np.fft.fft(x, axis=0), axis=0)
    b += 0.01 * (rng.standard_normal((n, m)) +
                 1j * rng.standard_normal((n, m)))
    return c, b


def _plain_op(case, seed):
    prec = _precision(case)
    kind = case['kind']
    rng = np.random.default_rng(seed)
    if kind == 'circulant':
        return fm.Circulant(_gauss(rng, case['n']), precision=prec)
    if kind == 'fourier':
        return fm.Fourier(case['n'], precision=prec)
    if kind == 'hadamard':
        return fm.Hadamard(case['order'], precision=prec)
    if kind == 'kron':
        return fm.Kron(fm.Fourier(case['f']), fm.Hadamard(case['h']),
                       fm.Circulant(_gauss(rng, case['c'])), precision=prec)
    if kind == 'toeplitz':
        return fm.Toeplitz(*_toeplitz_data(case, seed))
    c, d, rows = _chain_data(case, seed)
    return fm.Product(
        fm.Partial(fm.Circulant(c, precision=prec), rows=rows,
                   precision=prec),
        fm.Diag(d, precision=prec), precision=prec)


# ------------------------------------------------------------------ the call
def prepare(case, seed):
    kind, dtype = case['kind'], case['dtype']
    state = dict(case=case)
    if kind == 'batch':
        items = []
        vecs = _batch_vectors(case, seed)
        for k, (spec, vec) in enumerate(zip(_batch_specs(case), vecs)):
            name, n, m = spec
            if name == 'circulant':
                op = fm.Circulant(*vec, precision='fp32')
            elif name == 'toeplitz':
                op = fm.Toeplitz(*vec, precision='fp32')
            else:
                op = fm.Fourier(n, precision='fp32')
            items.append((op, _columns(n, m, dtype, 977 * seed + k)))
        state['batch'] = fm.Batch(items)
        return state
    if kind == 'fista':
        c, b = _fista_data(case, seed)
        op = fm.Circulant(c)
        op.largestSingularValue  # cached on the operator
        state['solver'] = FISTA(op, numLambda=0.05,
                                numMaxSteps=case['steps'])
        state['b'] = torch.from_numpy(np.ascontiguousarray(b.T)).cuda().t()
        return state
    op = _plain_op(case, seed)
    state['op'] = op
    if kind == 'toeplitz':
        n = case['n' if case['direction'] == 'forward' else 'rows']
        rng = np.random.default_rng(10 ** 6 + seed)
        state['x'] = np.asfortranarray(
            rng.standard_normal((case['cols'], n)).T)
        op.plan(np.complex128)
        return state
    n = op.numCols if case['direction'] != 'backward' else op.numRows
    state['x'] = _columns(n, case['cols'], dtype, seed)
    if kind == 'train':
        state['module'] = Operator(op)
        state['x'].requires_grad_(True)
        state['b'] = _columns(op.numRows, case['cols'], dtype, 7919 + seed)
    else:
        op.plan(np.dtype(dtype))
    return state


def run(state):
    kind, direction = state['case']['kind'], state['case']['direction']
    if kind == 'batch':
        return state['batch'].run(graph=True)
    if kind == 'fista':
        return state['solver'].process(state['b'])
    if kind == 'train':
        module, x = state['module'], state['x']
        y = module(x)
        r = y - state['b']
        loss = (r.real.square() + r.imag.square()).sum()
        names = [k for k, _ in module.named_parameters()]
        grads = torch.autograd.grad(loss, [x] + list(module.parameters()))
        out = {'y': y.detach(), 'x': grads[0]}
        out.update(zip(names, grads[1:]))
        return out
    if direction == 'forward':
        return state['op'].forward(state['x'])
    return state['op'].backward(state['x'])


# ------------------------------------------------------------------ the cost
def _fft_flops(n, cols):
    return 5.0 * n * math.log2(max(n, 2)) * cols


def work(case):
    kind = case['kind']
    es = {'float32': 4, 'float64': 8, 'complex64': 8,
          'complex128': 16}[case['dtype']]
    m = case.get('cols', 1)
    if kind == 'batch':
        nbytes = flops = 0
        for name, n, k in _batch_specs(case):
            nbytes += 2 * n * k * es
            if name == 'fourier':
                flops += _fft_flops(n, k)
            else:
                nbytes += es * (n if name == 'circulant' else 2 * n - 1)
                flops += 2 * _fft_flops(n, k) + 6.0 * n * k
        return {'bytes': nbytes, 'flops': flops}
    if kind == 'toeplitz':
        r, n = case['rows'], case['n']
        x, y = (n, r) if case['direction'] == 'forward' else (r, n)
        return {'bytes': x * m * 8 + y * m * 16 + 16 * (r + n - 1),
                'flops': 2 * _fft_flops(r + n, m) + 6.0 * (r + n) * m}
    if kind == 'hadamard':
        n = 1 << case['order']
        return {'bytes': 2 * n * m * es,
                'flops': float(n) * case['order'] * m}
    if kind == 'kron':
        n = case['f'] * case['c'] << case['h']
        per = (5 * math.log2(case['f']) + 2 * case['h'] +
               10 * math.log2(case['c']) + 6)
        return {'bytes': 2 * n * m * es + es * case['c'],
                'flops': per * n * m}
    n = case['n']
    if kind == 'fourier':
        return {'bytes': 2 * n * m * es, 'flops': _fft_flops(n, m)}
    conv = 2 * _fft_flops(n, m) + 6.0 * n * m
    if kind == 'circulant':
        return {'bytes': 2 * n * m * es + n * es, 'flops': conv}
    if kind == 'fista':
        # two transforms and the step, threshold and momentum updates a
        # step; the observations and the filter in, the result out
        return {'bytes': 2 * n * m * es + n * es,
                'flops': case['steps'] * (2 * conv + 40.0 * n * m)}
    rows = max(1, n // 4)
    if kind == 'chain':
        return {'bytes': (n + rows) * m * es + 2 * n * es + 8 * rows,
                'flops': conv + 6.0 * n * m}
    # training step: x, b, y and grad x once, c, d and their gradients
    return {'bytes': (2 * n + 2 * rows) * m * es + 4 * n * es + 8 * rows,
            'flops': 2.5 * conv + 30.0 * n * m}


# ------------------------------------------------------------------ 64 bits
def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _filter(c, x, adjoint=False):
    """Circular convolution of the columns of x with c (or its adjoint)."""
    s = torch.fft.fft(c)
    if adjoint:
        s = s.conj()
    return torch.fft.ifft(s[:, None] * torch.fft.fft(x, dim=0), dim=0)


def _toeplitz_exact(vc, vr, x, adjoint=False):
    size = vc.size + vr.size
    e = np.concatenate([vc, vr]).astype(np.complex128)
    n_out = vr.size + 1 if adjoint else vc.size
    s = np.fft.fft(e)
    if adjoint:
        s = s.conj()
    y = np.fft.ifft(s[:, None] * np.fft.fft(x, n=size, axis=0), axis=0)
    return np.asfortranarray(y[:n_out])


def _hadamard_exact(x, order):
    y = x.to(torch.float64).t().contiguous()
    m = y.shape[0]
    for k in range(order):
        v = y.view(m, -1, 2, 1 << k)
        y = torch.stack((v[:, :, 0] + v[:, :, 1], v[:, :, 0] - v[:, :, 1]),
                        dim=2).reshape(m, -1)
    return y.t()


def _chain_exact(case, seed, x):
    c, d, rows = _chain_data(case, seed)
    c, d, rows = _dev(c), _dev(d), _dev(rows)
    if case['direction'] == 'backward':
        full = torch.zeros((case['n'], x.shape[1]), dtype=torch.complex128,
                           device='cuda')
        full[rows] = x
        return d.conj()[:, None] * _filter(c, full, True)
    return _filter(c, d[:, None] * x)[rows]


def _train_exact(case, seed):
    # (the parameters are stored in the module's single or double form)
    dt = getattr(torch, case['dtype'])
    c, d, rows = _chain_data(case, seed)
    c = _dev(c).to(dt).to(torch.complex128).requires_grad_(True)
    d = _dev(d).to(dt).to(torch.complex128).requires_grad_(True)
    rows = _dev(rows)
    n, m = case['n'], case['cols']
    x = _columns(n, m, case['dtype'], seed).to(torch.complex128)
    x.requires_grad_(True)
    b = _columns(rows.numel(), m, case['dtype'],
                 7919 + seed).to(torch.complex128)
    y = _filter(c, d[:, None] * x)[rows]
    r = y - b
    loss = (r.real.square() + r.imag.square()).sum()
    gx, gd, gc = torch.autograd.grad(loss, [x, d, c])
    return {'y': y.detach(), 'x': gx, 'circulant0': gc, 'diag0': gd}


def _fista_exact(case, seed):
    c, b = _fista_data(case, seed)
    c, b = _dev(c), _dev(b)
    step = 1.0 / float(torch.fft.fft(c).abs().max()) ** 2
    x = torch.zeros_like(b)
    y = x.clone()
    t = 1.0
    for _ in range(case['steps']):
        old = x
        z = y - step * _filter(c, _filter(c, y) - b, True)
        mag = torch.clamp(z.abs() - step * 0.05 * 0.5, min=0)
        x = (mag / (mag + step * 0.05 * 0.5)) * z
        t_old, t = t, (1 + math.sqrt(1 + 4 * t * t)) / 2
        y = x + ((t_old - 1) / t) * (x - old)
    return torch.where(x != 0, z, x)


def exact(case, seed):
    kind = case['kind']
    if kind == 'train':
        return _train_exact(case, seed)
    if kind == 'fista':
        return _fista_exact(case, seed)
    if kind == 'batch':
        out = []
        vecs = _batch_vectors(case, seed)
        for k, (spec, vec) in enumerate(zip(_batch_specs(case), vecs)):
            name, n, m = spec
            x = _columns(n, m, case['dtype'],
                         977 * seed + k).to(torch.complex128)
            if name == 'circulant':
                out.append(_filter(_dev(vec[0]), x))
            elif name == 'toeplitz':
                e = _dev(np.concatenate(vec))
                z = torch.zeros((n - 1, m), dtype=x.dtype, device='cuda')
                out.append(_filter(e, torch.cat((x, z)))[:n])
            else:
                out.append(torch.fft.fft(x, dim=0))
        return out
    adjoint = case['direction'] == 'backward'
    if kind == 'toeplitz':
        vc, vr = _toeplitz_data(case, seed)
        n = case['rows' if adjoint else 'n']
        rng = np.random.default_rng(10 ** 6 + seed)
        x = rng.standard_normal((case['cols'], n)).T
        return _toeplitz_exact(vc, vr, x, adjoint)
    if kind == 'hadamard':
        x = _columns(1 << case['order'], case['cols'], case['dtype'], seed)
        return _hadamard_exact(x, case['order'])
    if kind == 'chain':
        n = max(1, case['n'] // 4) if adjoint else case['n']
        x = _columns(n, case['cols'], case['dtype'], seed)
        return _chain_exact(case, seed, x.to(torch.complex128))
    rng = np.random.default_rng(seed)
    if kind == 'kron':
        f, h, c = case['f'], case['h'], case['c']
        m = case['cols']
        x = _columns(f * c << h, m, case['dtype'], seed)
        s = torch.fft.fft(_dev(_gauss(rng, c)))
        cols = []
        for k in range(m):
            v = x[:, k].to(torch.complex128).reshape(f, 1 << h, c)
            v = torch.fft.ifft((s.conj() if adjoint else s) *
                               torch.fft.fft(v, dim=2), dim=2)
            for b in range(h):
                w = v.reshape(f, -1, 2, (1 << b) * c)
                v = torch.stack((w[:, :, 0] + w[:, :, 1],
                                 w[:, :, 0] - w[:, :, 1]), dim=2)
            v = v.reshape(f, -1)
            v = (torch.fft.ifft(v, dim=0, norm='forward') if adjoint
                 else torch.fft.fft(v, dim=0))
            cols.append(v.reshape(-1))
        return torch.stack(cols, dim=1)
    x = _columns(case['n'], case['cols'], case['dtype'],
                 seed).to(torch.complex128)
    if kind == 'circulant':
        return _filter(_dev(_gauss(rng, case['n'])), x, adjoint)
    if adjoint:
        return torch.fft.ifft(x, dim=0, norm='forward')
    return torch.fft.fft(x, dim=0)
