"""The banded kernel of the n <= 64 path (``csrc/dqb_dense_small_band.cu``) against the
product kernel that solves every other instance: the same problem with 1e-25 added to every
entry of H has full matrices, so it takes the product kernel, and differs by nothing that
FP32 sums of these sizes can show.  Both sum the same products in the same order, so step
counts are equal and states agree to the rounding of the dense-output weights."""

import numpy as np
import pytest
import torch

import dynamiqs_b200 as dq

pytestmark = pytest.mark.gpu

# every tile count of both thread layouts, at its edges
SIZES = (1, 2, 7, 8, 9, 15, 16, 17, 24, 25, 31, 32, 33, 48, 49, 63, 64)


def _band(rng, n, offsets, scale=1.0, hermitian=False):
    m = np.zeros((n, n), complex)
    for k in offsets:
        if abs(k) < n:
            v = scale * (rng.normal(size=n - abs(k)) + 1j * rng.normal(size=n - abs(k)))
            m += np.diag(v, k)
    return (m + m.conj().T) / 2 if hermitian else m


def _problem(n, seed, batch, jumps):
    rng = np.random.default_rng(seed)
    H = np.stack([_band(rng, n, (0, 1, 3), 1.0, True) for _ in range(batch)])
    Ls = [_band(rng, n, off, 0.3) for off in jumps]
    E = _band(rng, n, range(-n + 1, n), 1.0, True) / max(n, 1)
    g = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    rho = (g @ g.conj().T) / np.trace(g @ g.conj().T).real
    c = lambda x: np.ascontiguousarray(x, dtype=np.complex64)  # noqa: E731
    return c(H), [c(L) for L in Ls], c(rho), [c(E)]


def _agree(a, b):
    assert torch.equal(a.infos.nsteps, b.infos.nsteps)
    assert torch.equal(a.infos.naccepted, b.infos.naccepted)
    scale = b.states.abs().amax()
    # unit trace, at most ~50 steps: eight roundings of the largest entry
    assert (a.states - b.states).abs().amax() <= 8 * 2 ** -24 * max(float(scale), 1e-3) + 1e-9
    assert (a.expects - b.expects).abs().amax() <= 1e-6


@pytest.mark.parametrize('n, batch', [(n, 2) for n in SIZES] + [(n, 400) for n in SIZES if n <= 32])
def test_same_as_product_kernel(cuda_device, n, batch):  # two thread layouts up to n = 32
    H, Ls, rho, Es = _problem(n, n, batch, [(1,), (0,)])
    ts = np.linspace(0.0, 0.5, 4)
    got = dq.mesolve(H, Ls, rho, ts, exp_ops=Es, method=dq.Tsit5(rtol=1e-5, atol=1e-6))
    ref = dq.mesolve(H + np.complex64(1e-25), Ls, rho, ts, exp_ops=Es, method=dq.Tsit5(rtol=1e-5, atol=1e-6))
    _agree(got, ref)


@pytest.mark.parametrize('jumps', [[], [(1, -1)], [(-2,), (0, 2)], [(-1,), (1,), (2,)]])
@pytest.mark.parametrize('n', [13, 32, 40, 64])
def test_jump_patterns_and_options(cuda_device, n, jumps):
    H, Ls, rho, Es = _problem(n, 3, 3, jumps)
    for kw in (dict(), dict(options=dq.Options(save_states=False)), dict(method=dq.Dopri5()),
               dict(options=dq.Options(assume_hermitian=False))):
        got = dq.mesolve(H, Ls, rho, [0.1, 0.1, 0.4], exp_ops=Es, **kw)
        ref = dq.mesolve(H + np.complex64(1e-25), Ls, rho, [0.1, 0.1, 0.4], exp_ops=Es, **kw)
        _agree(got, ref)


def test_mixed_batch_and_fallbacks(cuda_device):
    """Full and banded instances of one batch each give what they give alone; a rho0 whose
    triangles differ beyond rounding (within the hermiticity check) keeps the product
    kernel's result; a rho0 that fails the check is refused."""
    H, Ls, rho, Es = _problem(20, 5, 4, [(1,)])
    H[1] += np.complex64(1e-25)
    H[2] += _problem(20, 6, 1, [])[0][0].T * np.complex64(1e-25)
    ts = [0.0, 0.3]
    all_ = dq.mesolve(H, Ls, rho, ts, exp_ops=Es)
    for b in range(4):
        one = dq.mesolve(H[b], Ls, rho, ts, exp_ops=Es)
        assert torch.equal(one.states, all_.states[b]) and int(one.infos.nsteps) == int(all_.infos.nsteps[b])
    skew = rho.copy()
    skew[2, 7] += np.complex64(5e-6)
    a = dq.mesolve(H[0], Ls, skew, ts, exp_ops=Es)
    b = dq.mesolve(H[1], Ls, skew, ts, exp_ops=Es)
    assert torch.equal(a.infos.nsteps, dq.mesolve(H[0], Ls, skew, ts).infos.nsteps)
    assert b.states.shape == a.states.shape and float((a.states[0] - torch.as_tensor(skew).cuda()).abs().max()) == 0.0
    skew[2, 7] += np.complex64(1e-3)
    with pytest.raises(RuntimeError, match='not hermitian'):
        dq.mesolve(H[0], Ls, skew, ts)


# ---- n > 64 in dense storage (csrc/dqb_large_band.cuh): the stencil against the products ----


@pytest.mark.parametrize('n', [65, 66, 96, 97, 130])  # edges of the 32 x 32 tiles, odd rows
@pytest.mark.parametrize('jumps', [[], [(1,)], [(0,), (-33,), (2, 5), (1,), (-1,)]])
@pytest.mark.parametrize('form', ['hermitian', 'standard', 'krylov'])
def test_large_same_as_products(cuda_device, n, jumps, form):
    H, Ls, rho, Es = _problem(n, n + len(jumps), 2, jumps)
    opts = dict(hermitian=dq.Options(), standard=dq.Options(assume_hermitian=False),
                krylov=dq.Options(stepper='krylov'))[form]
    ts = [0.0, 0.1, 0.25]
    got = dq.mesolve(H, Ls, rho, ts, exp_ops=Es, options=opts)
    ref = dq.mesolve(H + np.complex64(1e-25), Ls, rho, ts, exp_ops=Es, options=opts)
    _agree(got, ref)


def test_large_mixed_batch_and_tensor_cores(cuda_device):
    """A batch of banded and full instances runs both kinds of kernels; each instance gives
    what it gives alone (another loop of the graph), and with a tensor-core precision the
    banded ones give the FP32 result."""
    H, Ls, rho, Es = _problem(96, 8, 3, [(1,), (0,)])
    full = H.copy()
    full[1] += np.complex64(1e-25)
    ts = [0.0, 0.2]
    got = dq.mesolve(full, Ls, rho, ts, exp_ops=Es)
    alone = [dq.mesolve(full[b], Ls, rho, ts, exp_ops=Es) for b in range(3)]
    for b in range(3):
        assert int(got.infos.nsteps[b]) == int(alone[b].infos.nsteps)
        assert (got.states[b] - alone[b].states).abs().amax() <= 1e-7
    tc = dq.mesolve(H, Ls, rho, ts, exp_ops=Es, options=dq.Options(precision='tf32x3'))
    _agree(tc, dq.mesolve(H, Ls, rho, ts, exp_ops=Es))


@pytest.mark.parametrize('n, batch', [(1, 1), (5, 1), (8, 400), (30, 400), (30, 1), (48, 3), (64, 3)])
def test_initial_state_is_the_given_one(cuda_device, n, batch):
    """A rho0 whose triangles differ in the last bits: what is saved at t0 -- state, trace,
    hermiticity defect, expectation values -- is rho0's own; the later states are those of its
    upper triangle to a few roundings of rho0's largest entry."""
    H, Ls, rho, _ = _problem(n, n, batch, [(1,)])
    rng = np.random.default_rng(n)
    dust = (rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))) * (3e-8 * np.abs(rho).max())
    rho = (rho + dust).astype(np.complex64)
    E = (rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))).astype(np.complex64)
    res = dq.mesolve(H, Ls, rho, [0.0, 0.0, 0.2], exp_ops=[E])
    given = torch.as_tensor(rho).cuda()
    r = rho.astype(np.complex128)
    defect = np.linalg.norm(r - r.conj().T) / np.linalg.norm(r)
    value = np.trace(E.astype(np.complex128) @ r)
    for s in (0, 1):
        assert torch.equal(res.states[:, s], given.expand(batch, n, n))
        # FP64 sums in another order; expectation values are rounded to FP32 once
        assert (res.checks['hermiticity'][:, s] - defect).abs().max() <= 1e-12
        assert (res.expects[:, 0, s].to(torch.complex128) - value).abs().max() <= 2 ** -23 * abs(value) + 1e-12
    upper = (np.triu(rho, 1) + np.triu(rho, 1).conj().T + np.diag(np.diag(rho).real)).astype(np.complex64)
    ref = dq.mesolve(H, Ls, upper, [0.0, 0.0, 0.2], exp_ops=[E])
    assert torch.equal(res.states[:, 2], ref.states[:, 2]) and torch.equal(res.infos.nsteps, ref.infos.nsteps)
    # no step at all: every save point and the final state are rho0
    assert torch.equal(dq.mesolve(H, Ls, rho, [0.5]).states[:, 0], given.expand(batch, n, n))
    last = dq.mesolve(H, Ls, rho, [0.5], options=dq.Options(save_states=False))
    assert torch.equal(last.final_state.reshape(batch, n, n), given.expand(batch, n, n))


@pytest.mark.parametrize('n', [1, 2, 7, 8, 9, 15, 16, 17, 23, 24, 25, 31, 32])
@pytest.mark.parametrize('td', [False, True])
def test_result_does_not_depend_on_the_batch(cuda_device, n, td):
    """A large batch of n <= 32 instances takes another thread layout than a few: each instance
    has the same bits -- states, expectation values, step counts -- as alone."""
    H, Ls, rho, Es = _problem(n, n, 400, [(1, 0), (0,)])
    ts = np.linspace(0.0, 0.6, 5)
    rng = np.random.default_rng(n)
    for _ in range(7):  # values near zero at t0: the order of their FP64 sums shows
        X = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
        Es.append((X - np.trace(X @ rho) / np.trace(rho) * np.eye(n)).astype(np.complex64))
    vals = rng.normal(size=(400, 3))

    def solve(b):
        if not td:
            return dq.mesolve(H[b], Ls, rho, ts, exp_ops=Es)
        drive = dq.pwc([0.0, 0.2, 0.35, 0.6], vals[b], H[0])
        return dq.mesolve(H[1] + drive, Ls, rho, ts, exp_ops=Es)

    all_ = solve(slice(None))
    for b in (0, 57, 399):
        one = solve(b)
        for k in ('nsteps', 'naccepted'):
            assert int(getattr(one.infos, k)) == int(getattr(all_.infos, k)[b])
        assert torch.equal(one.states, all_.states[b]) and torch.equal(one.expects, all_.expects[b])


@pytest.mark.parametrize('n, batch', [(n, 2) for n in (5, 8, 16, 17, 32, 33, 48, 49, 64)]
                         + [(n, 400) for n in (5, 8, 9, 16, 17, 24, 25, 32)])
@pytest.mark.parametrize('jumps', [[(-1, 0, 1), (0, 2)], [(-1, 0, 1, 2), (-2, -1, 0, 1)]])
def test_jumps_of_many_diagonals(cuda_device, n, batch, jumps):
    """Jump operators multiplied in two steps, in both thread layouts, constant and in a
    time-dependent problem."""
    H, Ls, rho, Es = _problem(n, n, batch, jumps)
    ts = [0.0, 0.1, 0.3]
    _agree(dq.mesolve(H, Ls, rho, ts, exp_ops=Es), dq.mesolve(H + np.complex64(1e-25), Ls, rho, ts, exp_ops=Es))
    # (a smooth drive: with a jump in time, a stage whose time rounds onto the jump takes a step's
    # decision by the last bit of that step)
    wave = dq.Wave(amplitude=0.7, omega=3.0)
    rhos = np.stack([rho] * batch)
    a, b = (dq.mesolve(h + dq.modulated(wave, H[1]), Ls, rhos, ts, exp_ops=Es)
            for h in (H[0], H[0] + np.complex64(1e-25)))
    _agree(a, b)
