"""Timed cases: what a user of this package has it solve, through ``dq.mesolve``,
``dq.sesolve`` and the prepared form of a solve (``MESolveB200Integrator.prepare()`` once,
``launch().result()`` per solve).

Every case is one of these families (``family`` of the case):

* ``kerr``       master equation of driven Kerr oscillators in dense storage, n <= 64 (the
                 parameter sweeps of the benchmark; banded operators, as bosonic ones are);
* ``dense``      master equation with every operator a full matrix (a rotated frame, a spin
                 or molecular problem), at any n: the n <= 64 kernel and the GEMM path;
* ``pulse``      piecewise-constant drives, one instance per pulse (``dq.pwc``), n <= 64;
* ``gradient``   forward and backward through ``torch.autograd``, n <= 64;
* ``ket``        Schroedinger equation, dense storage (``full`` or banded H), any n;
* ``transmon``   transmon x cavity in dense storage, 64 < n <= 256, the tensor-core option;
* ``dia``        two coupled Kerr modes in sparse-DIA storage, up to n = 4096.

Operators are host arrays, as ``dynamiqs_b200.operators`` builds them, and a whole call
takes them through to its result; the prepared cases keep their device copies, as a program
does that solves again.  Outputs are the saved states and the expectation values (and the
gradients).  The step counts of an adaptive solve are not compared: whether an error
estimate within a rounding of the tolerance is accepted is decided by the last bit.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import dynamiqs_b200 as dq
from dynamiqs_b200.mesolve import make_batch_plan

# ------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------


def listed() -> list[dict]:
    return [
        # the README's lossy oscillator: one small system, where latency is everything
        dict(name='oscillator', family='kerr', n=16, batch=1, jumps=1, t_end=6.0, saves=101,
             kerr=0.0, drive=0.5, method='Tsit5', form='hermitian', prepared=False),
        # a parameter sweep of a small cavity at an odd size
        dict(name='sweep', family='kerr', n=21, batch=1000, jumps=1, t_end=2.0, saves=21,
             kerr=0.5, drive=2.0, method='Tsit5', form='hermitian', prepared=False),
        # the benchmark's batched Kerr workload, fewer instances and a shorter time
        dict(name='kerr-64', family='kerr', n=64, batch=1024, jumps=2, t_end=1.6, saves=11,
             kerr=0.5, drive=2.0, method='Tsit5', form='hermitian', prepared=True),
        # full matrices, the standard (non-hermitian-assuming) form, Dopri5, ragged size
        dict(name='dense-45', family='dense', n=45, batch=300, jumps=2, t_end=2.0, saves=11,
             method='Dopri5', form='standard', precision='fp32'),
        # full matrices beyond one block, default arithmetic, odd size
        dict(name='dense-151', family='dense', n=151, batch=32, jumps=1, t_end=2.0, saves=6,
             method='Tsit5', form='hermitian', precision='fp32'),
        # pulse optimisation without gradients: many piecewise-constant drives at once
        dict(name='pulses', family='pulse', n=24, batch=256, pieces=8, t_end=2.0, saves=21),
        # gradient of final expectation values with respect to H, L and psi0
        dict(name='gradient', family='gradient', n=30, batch=64, t_end=1.0, saves=5),
        # closed systems: many kets under banded Hamiltonians, then a few under full ones
        dict(name='kets-64', family='ket', n=64, batch=1500, full=False, t_end=1.0, saves=21),
        dict(name='kets-101', family='ket', n=101, batch=400, full=True, t_end=1.0, saves=11),
        dict(name='kets-1000', family='ket', n=1000, batch=8, full=True, t_end=1.0, saves=6),
        # the benchmark's transmon x cavity workload, fewer instances, tensor-core option
        dict(name='transmon', family='transmon', levels=4, cavity=64, batch=64, t_end=2.0,
             saves=5, precision='tf32x3'),
        # the benchmark's coupled Kerr modes in sparse-DIA storage
        dict(name='coupled-kerr', family='dia', modes=64, batch=2, t_end=0.6, saves=3),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    fam = rng.choice(('kerr', 'kerr', 'dense', 'dense', 'pulse', 'gradient', 'ket', 'ket',
                      'transmon', 'dia'))
    t_end = round(rng.uniform(0.3, 1.0), 3)
    saves = rng.randint(2, 21)
    if fam == 'kerr':
        c = dict(family=fam, n=_log_int(rng, 3, 64), batch=0, jumps=rng.randint(1, 2), t_end=t_end,
                 saves=saves, kerr=0.5, drive=2.0, method=rng.choice(('Tsit5', 'Dopri5')),
                 form=rng.choice(('hermitian', 'hermitian', 'standard')),
                 prepared=rng.random() < 0.4)
    elif fam == 'dense':
        c = dict(family=fam, n=_log_int(rng, 4, 200), batch=0, jumps=rng.randint(0, 2), t_end=t_end,
                 saves=saves, method=rng.choice(('Tsit5', 'Dopri5')),
                 form=rng.choice(('hermitian', 'hermitian', 'standard')), precision='fp32')
        if c['n'] > 64 and c['n'] % 2 == 0 and c['form'] == 'hermitian':
            c['precision'] = rng.choice(('fp32', 'tf32x3'))
    elif fam == 'pulse':
        c = dict(family=fam, n=_log_int(rng, 4, 48), batch=0, pieces=rng.randint(2, 12), t_end=t_end,
                 saves=saves)
    elif fam == 'gradient':
        c = dict(family=fam, n=_log_int(rng, 4, 40), batch=0, t_end=t_end,
                 saves=min(saves, 8))
    elif fam == 'ket':
        c = dict(family=fam, n=_log_int(rng, 8, 1200), batch=0, full=rng.random() < 0.5, t_end=t_end,
                 saves=saves)
        if c['n'] > 128:
            c['full'] = True
    elif fam == 'transmon':
        c = dict(family=fam, levels=rng.randint(2, 4), cavity=rng.randint(33, 64), batch=0, t_end=t_end,
                 saves=min(saves, 8), precision=rng.choice(('fp32', 'tf32x3')))
        if c['precision'] == 'tf32x3' and c['levels'] * c['cavity'] % 2:
            c['cavity'] -= 1  # the tensor-core modes take even sizes
    else:
        c = dict(family=fam, modes=_log_int(rng, 9, 64), batch=0, t_end=round(0.5 * t_end, 3),
                 saves=min(saves, 4))
    most = 1
    top = _products(next(k for k in listed() if k['name'] == _LARGEST[c['family']]))
    while most < 2048 and _products(dict(c, batch=2 * most)) <= top:
        most *= 2
    c['batch'] = _log_int(rng, 1, most)
    return c


# the listed case that bounds the cost of a family's drawn ones
_LARGEST = {'kerr': 'kerr-64', 'dense': 'dense-151', 'pulse': 'pulses', 'gradient': 'gradient',
            'ket': 'kets-101', 'transmon': 'transmon', 'dia': 'coupled-kerr'}


def _dim(c) -> int:
    if c['family'] == 'transmon':
        return c['levels'] * c['cavity']
    return c['modes'] ** 2 if c['family'] == 'dia' else c['n']


def _njumps(c) -> int:
    return {'pulse': 1, 'gradient': 1, 'ket': 0, 'transmon': 2, 'dia': 2}.get(c['family']) \
        if 'jumps' not in c else c['jumps']


def _steps(c) -> float:
    """Attempted steps of an average instance: the accuracy-limited part, and the stability
    limit of a fifth-order explicit step (about 2.9 / spectral width of the Liouvillian)."""
    n = _dim(c)
    if c['family'] == 'kerr':
        width = 0.25 * c['kerr'] * n * n + 2 * c['drive'] * math.sqrt(n) + n
    elif c['family'] == 'gradient':
        width = 0.025 * n * n + 4 * math.sqrt(n) + n
    elif c['family'] == 'pulse' or (c['family'] == 'ket' and not c['full']):
        width = 0.125 * n * n + 4 * math.sqrt(n) + n
        if c['family'] == 'ket':
            width *= 0.5
    elif c['family'] == 'transmon':
        width = 1.2 * c['cavity'] + 2 * math.sqrt(c['cavity'])
    elif c['family'] == 'dia':
        width = 0.05 * c['modes'] ** 2 + 4 * math.sqrt(c['modes']) + c['modes']
    else:
        width = 4 * _SCALE
    return 10 + 6 * c.get('pieces', 0) + c['t_end'] * width / 2.9


def _products(c) -> float:
    """A measure of cost for draw(): values that full-matrix products of the solve touch."""
    n, nb = _dim(c), c['batch']
    per = n * n if c['family'] in ('ket', 'dia') else n ** 3 * (1 + 2 * _njumps(c))
    if c['family'] == 'dia':
        per = n * n
    elif c['family'] == 'gradient':
        per *= 6
    elif c['family'] != 'ket' and n < 32:
        per = n * n * 32 * (1 + 2 * _njumps(c))  # small blocks are not bound by their products
    extra = n * n * c['saves'] if c['family'] != 'ket' else n * c['saves']
    return nb * (_steps(c) * per + extra)


def work(c) -> dict:
    """Inputs read once, saved states and expectation values written once; the flops of the
    right-hand sides on the operators' nonzeros (six per attempted step) and of the
    Runge-Kutta combinations (27 real multiply-adds of the state per step)."""
    n, nb, K, fam = _dim(c), c['batch'], _njumps(c), c['family']
    steps = _steps(c)
    size = n if fam == 'ket' else n * n
    if fam == 'dense' or (fam == 'ket' and c['full']):
        nnz_h, nnz_l = n * n, n * n
    else:
        nnz_h, nnz_l = (7 if fam == 'dia' else 3) * n, n
    cols = 1 if fam == 'ket' else n
    rhs = 8.0 * cols * (nnz_h + 2 * K * nnz_l)
    flops = nb * steps * (6 * rhs + 27 * 4.0 * size)
    read = 8.0 * (nb * nnz_h + K * nnz_l + n)
    write = 8.0 * nb * size * c['saves']
    if fam == 'gradient':  # the reverse pass: the stages again, their adjoints, three outer products
        flops *= 4
        read, write = 2 * read, 2 * write
    return {'bytes': read + write, 'flops': flops}


# ------------------------------------------------------------------------------------
# inputs (numpy, from the seed alone)
# ------------------------------------------------------------------------------------

_SCALE = 4.0  # spectral radius of the full random Hamiltonians


def _destroy(n):
    return np.diag(np.sqrt(np.arange(1.0, n)), 1).astype(np.complex128)


def _full_h(rng, shape, n):
    g = rng.normal(size=(*shape, n, n)) + 1j * rng.normal(size=(*shape, n, n))
    return (g + np.conj(np.swapaxes(g, -1, -2))) * (_SCALE / (4 * math.sqrt(n)))


def _full_l(rng, n):
    return 0.3 * (rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))) / math.sqrt(2 * n)


def _full_rho(rng, n):
    g = rng.normal(size=(n, min(n, 4))) + 1j * rng.normal(size=(n, min(n, 4)))
    r = g @ g.conj().T
    return r / np.trace(r).real


def _kerr_h(rng, batch, n, kerr, drive, det=1.0):
    k = np.arange(float(n))
    d, kk, e = rng.uniform(-det, det, batch), rng.uniform(0, kerr, batch), rng.uniform(0, drive, batch)
    H = np.zeros((batch, n, n), np.complex128)
    i = np.arange(n)
    H[:, i, i] = d[:, None] * k + 0.5 * kk[:, None] * k * (k - 1)
    s = e[:, None] * np.sqrt(k[1:])
    H[:, i[:-1], i[1:]] = s
    H[:, i[1:], i[:-1]] = s
    return H


def _vacuum(n):
    v = np.zeros((n, 1), np.complex128)
    v[0] = 1.0
    return v


def _c64(x):
    return np.ascontiguousarray(x, dtype=np.complex64)


def _inputs(c, seed) -> dict:
    """H, Ls, y0, E, tsave as the arrays a program holds (complex64)."""
    rng = np.random.default_rng(seed)
    fam, n, nb = c['family'], _dim(c), c['batch']
    ts = np.linspace(0.0, c['t_end'], c['saves'])
    a = _destroy(n)
    out = dict(tsave=ts, E=_c64(a.conj().T @ a))
    if fam == 'kerr':
        H = _kerr_h(rng, nb, n, c['kerr'], c['drive'])
        Ls = [math.sqrt(0.1) * a, math.sqrt(0.01) * (a.conj().T @ a)][:c['jumps']]
        y0 = _vacuum(n)
    elif fam == 'dense':
        H = _full_h(rng, (nb,), n)
        Ls = [_full_l(rng, n) for _ in range(c['jumps'])]
        y0 = _full_rho(rng, n)
        out['E'] = _c64(_full_h(rng, (), n))
    elif fam == 'pulse':
        H = _kerr_h(rng, 1, n, 0.25, 0.0)[0]
        Ls, y0 = [math.sqrt(0.1) * a], _vacuum(n)
        out['drive'] = _c64(a + a.conj().T)
        out['times'] = np.linspace(0.0, c['t_end'], c['pieces'] + 1)
        out['values'] = rng.uniform(-2.0, 2.0, (nb, c['pieces']))
    elif fam == 'gradient':
        # weakly anharmonic: with steps beyond the stability limit of levels that the state
        # never reaches, the derivative of the discrete solve is not the solution's
        H = _kerr_h(rng, nb, n, 0.05, 1.0)
        Ls, y0 = [math.sqrt(0.1) * a], _vacuum(n)
    elif fam == 'ket':
        Ls = []
        if c['full']:
            H = _full_h(rng, (nb,), n)
            y0 = rng.normal(size=(n, 1)) + 1j * rng.normal(size=(n, 1))
            y0 /= np.linalg.norm(y0)
        else:
            H, y0 = _kerr_h(rng, nb, n, 0.5, 2.0), _vacuum(n)
    elif fam == 'transmon':
        nq, nc = c['levels'], c['cavity']
        b, ac = np.kron(_destroy(nq), np.eye(nc)), np.kron(np.eye(nq), _destroy(nc))
        na, nbq = ac.conj().T @ ac, b.conj().T @ b
        bb = b.conj().T @ b.conj().T @ b @ b
        u = lambda lo, hi: rng.uniform(lo, hi, nb)[:, None, None]  # noqa: E731
        H = (u(0.9, 1.1) * na + u(0.8, 1.2) * nbq - 0.1 * bb + u(1e-3, 1e-2) * (na @ nbq)
             + u(0.0, 0.5) * (ac + ac.conj().T))
        Ls, y0 = [math.sqrt(0.01) * ac, math.sqrt(0.005) * b], _vacuum(n)
        out['E'] = _c64(na)
    else:  # dia: diagonals of the two modes' operators, column-indexed
        m = c['modes']
        l1, l2 = np.divmod(np.arange(n), m)
        d = rng.uniform(-0.5, 0.5, (nb, 2))
        kerr, g, eps, kappa = 0.05, 0.1, 1.0, 0.05
        diag = {0: d[:, :1] * l1 + d[:, 1:] * l2 + 0.5 * kerr * (l1 * (l1 - 1.0) + l2 * (l2 - 1.0))}
        up1 = np.sqrt(l1.astype(float))          # a1 at column j: sqrt(l1[j]), row j - m
        dn1 = np.sqrt(l1 + 1.0) * (l1 < m - 1)   # a1^+ at column j: row j + m
        a2 = np.sqrt(l2.astype(float))
        hop1 = np.sqrt((l1 + 1.0) * l2) * (l1 < m - 1) * (l2 > 0)   # a1^+ a2: row j + m - 1
        hop2 = np.sqrt(l1 * (l2 + 1.0)) * (l2 < m - 1) * (l1 > 0)   # a2^+ a1: row j - m + 1
        diag.update({m: eps * up1, -m: eps * dn1, 1 - m: g * hop1, m - 1: g * hop2})
        offs = tuple(sorted(diag))
        H = (offs, np.stack([np.broadcast_to(diag[k], (nb, n)) for k in offs], axis=1))
        Ls = [((m,), math.sqrt(kappa) * up1[None]), ((1,), math.sqrt(kappa) * a2[None])]
        y0 = _vacuum(n)
        out['E'] = None
        return dict(out, H=(H[0], _c64(H[1])), Ls=[(o, _c64(x)) for o, x in Ls], y0=_c64(y0))
    return dict(out, H=_c64(H), Ls=[_c64(L) for L in Ls], y0=_c64(y0))


# ------------------------------------------------------------------------------------
# the calls
# ------------------------------------------------------------------------------------


def _method(c):
    return (dq.Dopri5 if c.get('method') == 'Dopri5' else dq.Tsit5)(rtol=1e-6, atol=1e-8)


def _options(c):
    return dq.Options(assume_hermitian=c.get('form') != 'standard', precision=c.get('precision', 'fp32'))


def prepare(c, seed) -> dict:
    x = _inputs(c, seed)
    s = dict(case=c, x=x, method=_method(c), options=_options(c))
    if c['family'] == 'dia':
        s['H'] = dq.SparseDIA(*x['H'])
        s['Ls'] = [dq.SparseDIA(*L) for L in x['Ls']]
    else:  # a single system is unbatched
        s['H'], s['Ls'] = x['H'][0] if c['batch'] == 1 and x['H'].ndim == 3 else x['H'], x['Ls']
    if c['family'] in ('transmon', 'dia') or c.get('prepared'):
        plan = make_batch_plan(s['H'], s['Ls'], x['y0'], True)
        s['solve'] = dq.MESolveB200Integrator(
            ts=x['tsave'], y0=x['y0'], method=s['method'], gradient=None, options=s['options'],
            H=s['H'], Ls=s['Ls'], Es=None if x['E'] is None else [x['E']], plan=plan).prepare()
    elif c['family'] == 'gradient':
        dev = torch.device('cuda')
        s['leaves'] = [torch.as_tensor(v).to(dev).requires_grad_() for v in (x['H'], x['Ls'][0], x['y0'])]
        w = np.random.default_rng(seed + 1).uniform(0.5, 1.5, c['batch'])
        s['weights'] = torch.as_tensor(w, dtype=torch.float32, device=dev)
    elif c['family'] == 'pulse':
        s['H'] = x['H'] + dq.pwc(x['times'], x['values'], x['drive'])
    return s


def run(s) -> dict:
    c, x = s['case'], s['x']
    if 'solve' in s:
        r = s['solve'].launch().result()
    elif c['family'] == 'ket':
        r = dq.sesolve(s['H'], x['y0'], x['tsave'], exp_ops=[x['E']], method=s['method'])
    elif c['family'] == 'gradient':
        H, L, psi = s['leaves']
        r = dq.mesolve(H, [L], psi, x['tsave'], exp_ops=[x['E']], method=s['method'])
        loss = (s['weights'] * r.expects[:, 0, -1].real).sum()
        g = torch.autograd.grad(loss, (H, L, psi))
        return dict(states=r.states.detach(), expects=r.expects.detach(), grad_H=g[0], grad_L=g[1],
                    grad_psi=g[2])
    else:
        r = dq.mesolve(s['H'], s['Ls'], x['y0'], x['tsave'], exp_ops=[x['E']], method=s['method'],
                       options=s['options'])
    return dict(states=r.states) if r.expects is None else dict(states=r.states, expects=r.expects)


# ------------------------------------------------------------------------------------
# the solution in 64 bits (Taylor series of the exact exponential, plain torch)
# ------------------------------------------------------------------------------------


def _t128(v):
    dev = torch.device('cuda' if torch.cuda.is_available() else 'cpu')
    return torch.as_tensor(v).to(dev).to(torch.complex128)


def _advance(rhs, y, dt, width):
    """exp(dt L) y with L's norm at most `width`: substeps of norm 4, 30 terms each."""
    m = max(1, math.ceil(dt * width / 4.0))
    h = dt / m
    for _ in range(m):
        term = y
        for k in range(1, 31):
            term = rhs(term) * (h / k)
            y = y + term
    return y


def _from_left(offsets, diags, X):
    """A X of a DIA matrix with column-indexed diagonals."""
    n = X.shape[-1]
    out = torch.zeros_like(X)
    for q, k in enumerate(offsets):
        lo, hi = max(k, 0), n + min(k, 0)  # columns of A
        out[:, lo - k:hi - k] += diags[:, q, lo:hi, None] * X[:, lo:hi]
    return out


def _exact_dia(x, c):
    n = _dim(c)
    if _steps(c) * c['batch'] * float(n) ** 2 > 4.2e9:  # beyond some 20 seconds
        return None
    offs, d = x['H'][0], _t128(x['H'][1])
    psi = _t128(x['y0'])
    Ls = [(o, _t128(v)[None]) for o, v in x['Ls']]
    decay = sum(v[:, 0].abs() ** 2 for _, v in Ls)  # L^+ L is diagonal here
    h = -1j * d.clone()
    h[:, offs.index(0)] -= 0.5 * decay
    outer = [v[:, 0, :, None] * v[:, 0, None, :].conj() for _, v in Ls]
    y = (psi @ psi.mH).expand(c['batch'], n, n).clone()
    z = offs.index(0)
    spread = d[:, z].real
    off = d.abs().sum(1) - d[:, z].abs()
    width = float((spread.amax() - spread.amin()) + 4 * off.amax() + 2 * decay.amax())

    def rhs(X):
        out = _from_left(offs, h, X)
        out = out + out.mH
        for ((k,), _), f in zip(Ls, outer):  # L X L^+ with L's one diagonal at k > 0
            out[:, :n - k, :n - k] += f[:, k:, k:] * X[:, k:, k:]
        return out

    states = [y]
    for dt in np.diff(x['tsave']):
        y = _advance(rhs, y, float(dt), width)
        states.append(y)
    return dict(states=torch.stack(states, 1))


def _spread(H):
    e = torch.linalg.eigvalsh(H)
    return float((e[..., -1] - e[..., 0]).max())


def _exact_pulse(x, c):
    H0, drive, L, E, psi = (_t128(x[k]) for k in ('H', 'drive', 'L', 'E', 'y0'))
    vals = _t128(x['values'])
    edges = x['times']
    y = (psi @ psi.mH).expand(c['batch'], *H0.shape).clone()
    states = [y]
    for t0, t1 in zip(x['tsave'][:-1], x['tsave'][1:]):
        cuts = [t0] + [t for t in edges if t0 < t < t1] + [t1]
        for lo, hi in zip(cuts[:-1], cuts[1:]):
            p = min(max(int(np.searchsorted(edges, 0.5 * (lo + hi))) - 1, 0), c['pieces'] - 1)
            H = H0 + vals[:, p, None, None] * drive
            y = _lindblad(H, [L], y, float(hi - lo))
        states.append(y)
    states = torch.stack(states, 1)
    return dict(states=states, expects=torch.einsum('ij,bsji->bs', E, states)[:, None])


def _lindblad(H, Ls, y, dt):
    A = -1j * H - 0.5 * sum((L.mH @ L for L in Ls), torch.zeros_like(H))
    with torch.no_grad():
        width = _spread(H) + 2 * sum(float(torch.linalg.matrix_norm(L, 2)) ** 2 for L in Ls)

    def rhs(X):
        out = A @ X + X @ A.mH
        for L in Ls:
            out = out + L @ X @ L.mH
        return out

    return _advance(rhs, y, dt, width)


def exact(c, seed):
    x = _inputs(c, seed)
    fam = c['family']
    if fam == 'dia':
        return _exact_dia(x, c)
    if fam == 'pulse':
        return _exact_pulse(dict(x, L=x['Ls'][0]), c)
    H, y0, E = _t128(x['H']), _t128(x['y0']), _t128(x['E'])
    Ls = [_t128(L) for L in x['Ls']]
    leaves = [H, *Ls, y0]
    if fam == 'gradient':
        for v in leaves:
            v.requires_grad_()
    n, nb = _dim(c), c['batch']
    if fam == 'ket':
        y = y0.expand(nb, n, 1)
        width = float(H.abs().sum(-1).max()) if n > 256 else float(torch.linalg.eigvalsh(H).abs().max())
        step = lambda y, dt: _advance(lambda v: -1j * (H @ v), y, dt, width)  # noqa: E731
    else:
        y = (y0 @ y0.mH if y0.shape[-1] == 1 else y0).expand(nb, n, n)
        step = lambda y, dt: _lindblad(H, Ls, y, dt)  # noqa: E731
    states = [y]
    for dt in np.diff(x['tsave']):
        y = step(y, float(dt))
        states.append(y)
    states = torch.stack(states, 1)
    if fam == 'ket':
        expects = torch.einsum('bsix,ij,bsjx->bs', states.conj(), E, states)[:, None]
    else:
        expects = torch.einsum('ij,bsji->bs', E, states)[:, None]
    out = dict(states=states.detach(), expects=expects.detach())
    if fam == 'gradient':
        w = torch.as_tensor(np.random.default_rng(seed + 1).uniform(0.5, 1.5, nb), device=H.device)
        g = torch.autograd.grad((w * expects[:, 0, -1].real).sum(), leaves)
        out.update(grad_H=g[0], grad_L=g[1], grad_psi=g[2])
    return out
