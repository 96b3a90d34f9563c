"""Where the banded kernels begin and end: eight and nine nonzero diagonals, eight and nine jump
operators, sizes at which every matrix is banded, and jumps beyond the standard form's
banded products, each against the complex128 oracle (the bar of tests/parity.py)."""

import numpy as np
import pytest
import torch

import dynamiqs_b200 as dq
from oracle.mesolve import sesolve as oracle_sesolve
from tests.parity import assert_solve_parity

pytestmark = pytest.mark.gpu

TS = np.linspace(0.0, 0.5, 4)


def _band(rng, n, offsets, scale=1.0, hermitian=False):
    m = np.zeros((n, n), complex)
    for k in offsets:
        if abs(k) < n:
            m += np.diag(scale * (rng.normal(size=n - abs(k)) + 1j * rng.normal(size=n - abs(k))), k)
    m = m + m.conj().T if hermitian else m
    return m.astype(np.complex64)


def _ket(rng, n):
    v = rng.normal(size=(n, 1)) + 1j * rng.normal(size=(n, 1))
    return (v / np.linalg.norm(v)).astype(np.complex64)


def _check(H, Ls, psi, E, **kw):
    res = dq.mesolve(H, Ls, psi, TS, exp_ops=[E], options=dq.Options(**kw))
    form = 'hermitian' if kw.get('assume_hermitian', True) else 'standard'
    assert_solve_parity(res.states.cpu().numpy(), res.expects.cpu().numpy(), int(res.infos.nsteps), H, Ls, psi, TS,
                        [E], 'Tsit5', 1e-6, 1e-6, form=form)


@pytest.mark.parametrize('n', [20, 48, 64, 70])
@pytest.mark.parametrize('diags', [8, 9])
@pytest.mark.parametrize('herm', [True, False])
def test_diagonals_of_hnh(cuda_device, n, diags, herm):
    rng = np.random.default_rng(n + diags)
    H = _band(rng, n, (1, 2, 3, 4), 0.3, True)
    if diags == 9:
        H = H + np.diag(rng.normal(size=n)).astype(np.complex64)
    assert len(set(np.subtract(*np.nonzero(H)))) == diags
    _check(H, [], _ket(rng, n), _band(rng, n, (0, 1), 0.5, True), assume_hermitian=herm)


@pytest.mark.parametrize('n', [20, 70])
@pytest.mark.parametrize('jumps', [8, 9])
def test_jump_operators(cuda_device, n, jumps):
    rng = np.random.default_rng(n + jumps)
    Ls = [_band(rng, n, (k - 4,), 0.15) for k in range(jumps)]
    _check(_band(rng, n, (0, 1), 0.3, True), Ls, _ket(rng, n), _band(rng, n, (0, 1), 0.5, True))


@pytest.mark.parametrize('n', [2, 3, 4])  # (n = 1: the right-hand side is rounding alone, and so is its first step)
@pytest.mark.parametrize('herm', [True, False])
def test_every_matrix_is_banded(cuda_device, n, herm):
    rng = np.random.default_rng(n)
    full = range(-n + 1, n)
    psi = _ket(rng, n)
    _check(_band(rng, n, full, 0.4, True), [_band(rng, n, full, 0.3)], psi @ psi.conj().T, _band(rng, n, full, 0.5, True),
           assume_hermitian=herm)


@pytest.mark.parametrize('n', [13, 40, 64])
@pytest.mark.parametrize('jumps', [2, 3])
def test_standard_form_jumps(cuda_device, n, jumps):
    rng = np.random.default_rng(n)
    Ls = [_band(rng, n, off, 0.2) for off in ((-1,), (1, 0), (2,))[:jumps]]
    _check(_band(rng, n, (0, 1), 0.3, True), Ls, _ket(rng, n), _band(rng, n, (0, 1), 0.5, True), assume_hermitian=False)


@pytest.mark.parametrize('n', [40, 100])
@pytest.mark.parametrize('diags', [8, 9])
def test_sesolve_diagonals(cuda_device, n, diags):
    rng = np.random.default_rng(n + diags)
    H = _band(rng, n, (1, 2, 3, 4), 0.3, True)
    if diags == 9:
        H = H + np.diag(rng.normal(size=n)).astype(np.complex64)
    psi = _ket(rng, n)
    res = dq.sesolve(H, psi, TS)
    ref = np.stack(oracle_sesolve(H, psi, TS, rtol=1e-6, atol=1e-6, save_fn=lambda y: y).ysave)
    err = np.linalg.norm(res.states.cpu().numpy() - ref, axis=(-2, -1)) / np.linalg.norm(ref, axis=(-2, -1))
    assert err.max() <= 1e-5


@pytest.mark.parametrize('n', [20, 32, 48])
def test_adjoint_with_eight_diagonals(cuda_device, n):
    """Against the product kernel (1e-25 in every entry of H makes it a full matrix): the bound
    is 64 roundings of the largest gradient."""
    rng = np.random.default_rng(n)
    H, psi = _band(rng, n, (1, 2, 3, 4), 0.3, True), _ket(rng, n)
    E = _band(rng, n, (0, 1), 0.5, True)

    def grads(h):
        leaves = [torch.as_tensor(v).clone().requires_grad_() for v in (h, psi)]
        return torch.autograd.grad(dq.mesolve(leaves[0], [], leaves[1], TS, exp_ops=[E]).expects.real.sum(), leaves)

    for a, b in zip(grads(H), grads(H + np.complex64(1e-25))):
        assert (a - b).abs().max() <= 64 * 2 ** -24 * b.abs().max()


@pytest.mark.parametrize('n', [2, 4, 8, 16])
@pytest.mark.parametrize('offsets', [(0, 1), (0, 1, 2), (1, 2, 3), (0, 1, 2, 3), (1, 2, 3, 4)])
@pytest.mark.parametrize('jumps', [[], [(1,)], [(0, 1), (-1,)]])
def test_standard_form_small(cuda_device, n, offsets, jumps):  # either side of stencil_pays
    rng = np.random.default_rng(n)
    _check(_band(rng, n, offsets, 0.3, True), [_band(rng, n, off, 0.2) for off in jumps], _ket(rng, n),
           _band(rng, n, (0, 1), 0.5, True), assume_hermitian=False)


@pytest.mark.parametrize('n', [5, 16, 31, 32, 33])
def test_sesolve_full_and_banded(cuda_device, n):
    """One launch for both up to 32 rows, two beyond: each instance of a mixed batch gives the
    bits that it gives alone, and the full ones the oracle's states."""
    rng = np.random.default_rng(n)
    H = np.stack([_band(rng, n, (0, 1) if b % 2 else range(n), 0.3, True) for b in range(6)])
    psi, E = _ket(rng, n), _band(rng, n, (0, 1), 0.5, True)
    res = dq.sesolve(H, psi, TS, exp_ops=[E])
    for b in range(6):
        one = dq.sesolve(H[b], psi, TS, exp_ops=[E])
        assert torch.equal(one.states, res.states[b]) and torch.equal(one.expects, res.expects[b])
        ref = np.stack(oracle_sesolve(H[b], psi, TS, rtol=1e-6, atol=1e-6, save_fn=lambda y: y).ysave)
        assert np.linalg.norm(one.states.cpu().numpy() - ref, axis=(-2, -1)).max() <= 1e-5
