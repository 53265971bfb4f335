"""The backward kernel (vector-Jacobian product) and the fused likelihood
with its gradient, against central finite differences of the FP64 oracle.

Bars (the reference's gradient tests, ``tests/test_transforms_xas.py``):
* FP64: relative 1e-5 of central differences (step 1e-6 max(|x|, 1)), with
  an absolute floor of 1e-6 of the largest component;
* FP32: |g32 - g64| <= 1e-2 |g64| + 1e-3 max |g64| against the FP64 kernels.
"""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from oracle.api import psd
from test_gpu_polarizations import draw_batch, f32

pytestmark = pytest.mark.gpu

MODELS = {"xas": "IMRPhenomXAS", "phenomd": "IMRPhenomD", "taylorf2": "TaylorF2"}
F = np.geomspace(20.0, 900.0, 300)


def weighted_loss(approximant, params, f, t_c, w):
    hp, hc = oracle.polarizations(approximant, params, f, t_c=t_c)
    return np.sum(w[0] * hp.real + w[1] * hp.imag + w[2] * hc.real + w[3] * hc.imag, axis=-1)


def fd_gradient(function, params, t_c):
    """Central differences (step 1e-6 max(|x|, 1)) in the 8 parameters and t_c."""
    out = np.zeros((len(params), 9))
    for k in range(9):
        x = t_c if k == 8 else params[:, k]
        h = 1e-6 * np.maximum(np.abs(x), 1.0)
        vals = []
        for sign in (1.0, -1.0):
            p, tc = params.copy(), t_c.copy()
            if k == 8:
                tc = tc + sign * h
            else:
                p[:, k] += sign * h
            vals.append(function(p, tc))
        out[:, k] = (vals[0] - vals[1]) / (2 * h)
    return out


def gpu_vjp(cuda, approximant, params, f, t_c, w, precision):
    import torch

    from waveformx_b200 import _lib, ops

    real = torch.float32 if precision == _lib.FP32 else torch.float64
    cplx = torch.complex64 if precision == _lib.FP32 else torch.complex128
    p = torch.as_tensor(params, dtype=torch.float64, device=cuda)
    freqs = torch.as_tensor(f, dtype=real, device=cuda)
    tables = ops.setup(approximant, p, freqs[:1].to(torch.float64), precision=precision, jvp=True)
    tc = torch.as_tensor(t_c, dtype=real, device=cuda)
    shape = (len(params), len(f))
    gp = torch.as_tensor(np.broadcast_to(w[0] + 1j * w[1], shape).copy(), dtype=cplx, device=cuda)
    gc = torch.as_tensor(np.broadcast_to(w[2] + 1j * w[3], shape).copy(), dtype=cplx, device=cuda)
    return ops.vjp(approximant, tables.table, tables.dtable, freqs, None, tc, gp, gc).cpu().numpy().astype(np.float64)


CASES = np.array([
    [36.0, 29.0, 0.3, -0.4, 500.0, 0.7, 1.2, 25.0],
    [50.0, 2.0, 0.9, 0.3, 300.0, 2.1, 0.3, 30.0],
    [150.0, 100.0, -0.5, 0.95, 3000.0, 0.4, 2.0, 22.0],
])


@pytest.mark.parametrize("model", MODELS)
def test_fp64_vjp_matches_fd(cuda, model):
    approximant = MODELS[model]
    w = np.random.default_rng(5).normal(size=(4, len(F)))
    t_c = np.array([0.0, 0.01, -0.02])
    grad = gpu_vjp(cuda, approximant, CASES, F, t_c, w, 0)
    fd = fd_gradient(lambda p, tc: weighted_loss(approximant, p, F, tc, w), CASES, t_c)
    for i in range(len(CASES)):
        scale = np.max(np.abs(fd[i]))
        np.testing.assert_allclose(grad[i], fd[i], rtol=1e-5, atol=1e-6 * scale)


@pytest.mark.parametrize("model", MODELS)
def test_fp32_vjp_within_bound(cuda, model):
    approximant = MODELS[model]
    w = np.random.default_rng(6).normal(size=(4, len(F)))
    params = f32(CASES)
    t_c = f32([0.0, 0.01, -0.02])
    g64 = gpu_vjp(cuda, approximant, params, f32(F), t_c, w, 0)
    g32 = gpu_vjp(cuda, approximant, params, f32(F), t_c, w, 1)
    for i in range(len(params)):
        bound = 1e-2 * np.abs(g64[i]) + 1e-3 * np.max(np.abs(g64[i]))
        assert np.all(np.abs(g32[i] - g64[i]) <= bound), (i, g32[i], g64[i])


def _fused(cuda, approximant, params, f, t_c, data, w, precision, per_binary):
    import torch

    from waveformx_b200 import _lib, ops

    real = torch.float32 if precision == _lib.FP32 else torch.float64
    cplx = torch.complex64 if precision == _lib.FP32 else torch.complex128
    p = torch.as_tensor(params, dtype=torch.float64, device=cuda)
    freqs = torch.as_tensor(f, dtype=real, device=cuda)
    tables = ops.setup(approximant, p, freqs[:1].to(torch.float64), precision=precision, jvp=True)
    tc = torch.as_tensor(t_c, dtype=real, device=cuda)
    d = torch.as_tensor(data, dtype=cplx, device=cuda)
    wt = torch.as_tensor(w, dtype=real, device=cuda)
    loss, grad = ops.fused_loss(approximant, tables.table, tables.dtable, freqs, None, tc, d, wt)
    return loss.cpu().numpy().astype(np.float64), grad.cpu().numpy().astype(np.float64)


@pytest.mark.parametrize("model", MODELS)
@pytest.mark.parametrize("per_binary", [True, False])
def test_fused_loss_and_gradient(cuda, model, per_binary):
    """L_b = sum_f w |h+_b - d_b|^2 with w = 1/S(f) and d_b the waveform at
    parameters perturbed by 1 % plus complex noise of 0.1 |h| (per binary),
    or one injected signal plus noise (shared)."""
    approximant = MODELS[model]
    rng = np.random.default_rng(9)
    params = f32(draw_batch(rng, 8))
    t_c = f32(rng.uniform(-0.01, 0.01, 8))
    f = f32(np.linspace(20.0, 1024.0, 4017))
    w = 1.0 / psd(f)
    if per_binary:
        shifted = params * (1.0 + 0.01 * rng.normal(size=params.shape))
        shifted[:, 7] = params[:, 7]
        h = oracle.polarizations(approximant, shifted, f)[0]
        data = h + 0.1 * np.abs(h) * (rng.normal(size=h.shape) + 1j * rng.normal(size=h.shape))
    else:
        h = oracle.polarizations(approximant, params[:1], f)[0][0]
        data = h + 0.05 * np.abs(h).max() * (rng.normal(size=h.shape) + 1j * rng.normal(size=h.shape))
    loss_ref = oracle.batch_loss(approximant, params, f, data, w, t_c=t_c)
    fd = oracle.loss_gradient_fd(approximant, params, f, data, w, t_c=t_c)
    for precision, rtol in ((0, 1e-10), (1, 1e-4)):
        loss, grad = _fused(cuda, approximant, params, f, t_c, data, w, precision, per_binary)
        np.testing.assert_allclose(loss, loss_ref, rtol=rtol)
        g = grad[:, [0, 1, 2, 3, 4, 5, 6, 8]]
        for i in range(len(params)):
            scale = np.max(np.abs(fd[i]))
            if precision == 0:
                np.testing.assert_allclose(g[i], fd[i], rtol=1e-5, atol=1e-6 * scale)
            else:
                assert np.all(np.abs(g[i] - fd[i]) <= 1e-2 * np.abs(fd[i]) + 1e-3 * scale), (i, g[i], fd[i])


@pytest.mark.parametrize("model", MODELS)
@pytest.mark.parametrize("ragged", [False, True])
def test_fused_loss_from_params_is_the_same(cuda, model, ragged):
    """The dual-number set-up on a second stream, overlapped with the value
    set-up and the reverse pass, then the contraction: the same bits as the
    set-up with its derivatives followed by the fused call."""
    import torch

    from waveformx_b200 import _lib, ops

    approximant = MODELS[model]
    rng = np.random.default_rng(12)
    params = f32(draw_batch(rng, 40))
    p = torch.as_tensor(params, device=cuda)
    t_c = torch.as_tensor(f32(rng.uniform(-0.01, 0.01, 40)), dtype=torch.float32, device=cuda)
    if ragged:
        lengths = rng.integers(50, 3000, 40)
        offsets = torch.as_tensor(np.concatenate([[0], np.cumsum(lengths)]), device=cuda)
        flat = np.concatenate([np.linspace(20.0, 20.0 + 0.25 * (k - 1), k) for k in lengths])
        freqs = torch.as_tensor(flat, dtype=torch.float32, device=cuda)
        f_min = torch.full((40,), 20.0, dtype=torch.float64, device=cuda)
        d = torch.as_tensor((rng.normal(size=flat.size) + 1j * rng.normal(size=flat.size)) * 1e-2,
                            dtype=torch.complex64, device=cuda)
        w = torch.as_tensor(1.0 / psd(flat), dtype=torch.float32, device=cuda)
    else:
        offsets = None
        f = np.linspace(20.0, 1024.0, 4017)
        freqs = torch.as_tensor(f, dtype=torch.float32, device=cuda)
        f_min = freqs[:1].double()
        d = torch.as_tensor((rng.normal(size=f.size) + 1j * rng.normal(size=f.size)) * 1e-2,
                            dtype=torch.complex64, device=cuda)
        w = torch.as_tensor(1.0 / psd(f), dtype=torch.float32, device=cuda)
    loss, grad, status = ops.fused_loss_from_params(approximant, p, f_min, freqs, offsets, t_c, d, w, scale=-0.5)
    tables = ops.setup(approximant, p, f_min, precision=_lib.FP32, jvp=True)
    loss2, grad2 = ops.fused_loss(approximant, tables.table, tables.dtable, freqs, offsets, t_c, d, w, scale=-0.5)
    assert torch.equal(loss, loss2) and torch.equal(grad, grad2)
    assert torch.equal(status, tables.status)


@pytest.mark.parametrize("model", ["IMRPhenomXAS", "IMRPhenomD", "TaylorF2"])
@pytest.mark.parametrize("n, batch", [(1, 3), (31, 3), (33, 3), (128, 3), (129, 3), (300, 1600), (700, 6400)])
def test_fp64_reverse_pass_sums(cuda, model, n, batch):
    """The FP64 reverse pass of a shared grid at the edges of its spans (128
    frequencies, 32 a warp), with two and eight binaries a block and several
    spans a block: the vjp and the fused likelihood of a grid are the sums of
    those of its frequencies, each taken as a row of its own of a ragged grid
    (another kernel). Bar: 1e-9 of the sum of the terms' magnitudes (the sums
    round to 1e-13 of it, and a table's slots cancel by less than 1e4 in the
    product with the set-up's tangents)."""
    import torch

    from waveformx_b200 import _lib, ops

    base = np.array([[36.0, 29.0, 0.3, -0.1, 500.0, 0.7, 1.2, 20.0], [60.0, 15.0, 0.8, 0.5, 1000.0, 2.5, 4.0, 20.0],
                     [9.0, 7.0, -0.6, 0.2, 200.0, 1.1, 0.3, 20.0]])
    grid = torch.as_tensor(np.geomspace(20.0, 900.0, n) if n > 1 else np.array([90.0]), device=cuda)
    rng = np.random.default_rng(n)
    rows = torch.arange(3, device=cuda).repeat_interleave(n)
    of = torch.arange(batch, device=cuda) % 3
    params = torch.as_tensor(base, device=cuda)
    tables = ops.setup(model, params, grid[:1], precision=_lib.FP64, jvp=True)
    t_c = torch.tensor([0.01, -0.02, 0.0], dtype=torch.float64, device=cuda)
    cot = [torch.as_tensor(rng.normal(size=(3, n)) + 1j * rng.normal(size=(3, n)), device=cuda) for _ in range(2)]
    weights = torch.as_tensor(rng.uniform(0.5, 2.0, n), device=cuda)
    table, dtable = tables.table[of].contiguous(), tables.dtable[of].contiguous()
    flat = (tables.table[rows].contiguous(), tables.dtable[rows].contiguous(), grid.repeat(3),
            torch.arange(3 * n + 1, device=cuda), t_c[rows].contiguous())

    def check(whole, parts):
        bar = 1e-9 * parts.abs().sum(1)[of]
        error = (whole - parts.sum(1)[of]).abs()
        assert bool((error <= bar).all()), (error / bar).max()

    check(ops.vjp(model, table, dtable, grid, None, t_c[of].contiguous(), *(c[of].contiguous() for c in cot)),
          ops.vjp(model, *flat, *(c.reshape(-1) for c in cot)).reshape(3, n, 9))
    loss, grad = ops.fused_loss(model, table, dtable, grid, None, t_c[of].contiguous(), cot[0][0].contiguous(), weights,
                                antenna=(0.6, -0.3), scale=-0.5)
    loss1, grad1 = ops.fused_loss(model, *flat, cot[0][0].repeat(3), weights.repeat(3), antenna=(0.6, -0.3), scale=-0.5)
    check(loss[:, None], loss1.reshape(3, n, 1))
    check(grad, grad1.reshape(3, n, 9))


@pytest.mark.parametrize("model", ["IMRPhenomXAS", "IMRPhenomD", "TaylorF2"])
@pytest.mark.parametrize("n, batch", [(1, 2400), (2, 2400), (63, 2401), (65, 2400), (511, 1300), (4001, 2400)])
def test_fp32_reverse_pass_of_a_batch(cuda, model, n, batch):
    """The FP32 reverse pass with a tile's powers in shared memory (large
    batches on a shared grid), at the edges of its chunks (64 frequencies) and
    tiles, rows of odd length, data shared and per binary, and one refused
    binary: the module's FP32 bar against the FP64 kernels of the distinct
    binaries; the loss, a sum of positive terms each within 1e-5 of its size,
    to 1e-4."""
    import torch

    from waveformx_b200 import _lib, ops

    base = np.array([[36.0, 29.0, 0.3, -0.1, 500.0, 0.7, 1.2, 20.0], [60.0, 15.0, 0.8, 0.5, 1000.0, 2.5, 4.0, 20.0],
                     [9.0, 7.0, -0.6, 0.2, 200.0, 1.1, 0.3, 20.0], [np.nan, 7.0, -0.6, 0.2, 200.0, 1.1, 0.3, 20.0]])
    grid = torch.as_tensor(np.geomspace(20.0, 2000.0, n) if n > 1 else np.array([90.0]), device=cuda).float()
    rng = np.random.default_rng(n)
    of = torch.arange(batch, device=cuda) % 4
    params = torch.as_tensor(base, device=cuda)
    t_c = torch.tensor([0.01, -0.02, 0.0, 0.0], dtype=torch.float64, device=cuda)
    cot = [torch.as_tensor(rng.normal(size=(4, n)) + 1j * rng.normal(size=(4, n)), device=cuda).to(torch.complex64)
           for _ in range(2)]
    weights = torch.as_tensor(rng.uniform(0.5, 2.0, (4, n)), device=cuda).float()
    kw = dict(antenna=(0.6, -0.3), scale=-0.5)

    def run(precision, rows):
        real, cplx = (torch.float32, torch.complex64) if precision == _lib.FP32 else (torch.float64, torch.complex128)
        tables = ops.setup(model, params, grid[:1].double(), precision=precision, jvp=True)
        table, dtable, tc = (x[rows].contiguous() for x in (tables.table, tables.dtable, t_c.to(real)))
        a, b = (c.to(cplx)[rows].contiguous() for c in cot)
        w, f = weights.to(real), grid.to(real)
        yield ops.vjp(model, table, dtable, f, None, tc, a, b)
        yield from ops.fused_loss(model, table, dtable, f, None, tc, a[0].contiguous(), w[0].contiguous(), **kw)
        yield from ops.fused_loss(model, table, dtable, f, None, tc, a, w[rows].contiguous(), **kw)

    few = torch.arange(4, device=cuda)
    for got, exact in zip(run(_lib.FP32, of), run(_lib.FP64, few)):
        got, exact = got.double(), exact.double()
        assert torch.isnan(exact[3]).all() and torch.isnan(got[of == 3]).all()
        got, want = got[of != 3], exact[of[of != 3]]
        if want.ndim == 1:
            bar = 1e-4 * want.abs()
        else:
            bar = 1e-2 * want.abs() + 1e-3 * want.abs().amax(1, keepdim=True)
        assert bool(((got - want).abs() <= bar).all()), ((got - want).abs() / bar).max()


@pytest.mark.parametrize("model", ["IMRPhenomXAS", "IMRPhenomD", "TaylorF2"])
@pytest.mark.parametrize("n, batch", [(60, 3), (300, 1), (1001, 37), (129, 1000), (4017, 1), (20000, 5), (4001, 1021)])
def test_fp64_reverse_pass_repeats(cuda, model, n, batch, monkeypatch):
    """The FP64 vjp and fused likelihood of a shared grid repeat their bits,
    with a binary's frequencies in one block, in a cluster of two to eight and
    in parts that the workspace gathers, and without a workspace. The two ways
    are the same sums in another order: 1e-8 of a binary's largest component
    (the sums round to 1e-13 of their terms' magnitudes, which the contraction
    cancels by less than 1e5)."""
    import torch

    from waveformx_b200 import _lib, ops

    rng = np.random.default_rng(n)
    params = torch.as_tensor(draw_batch(rng, batch), device=cuda)
    grid = torch.linspace(20.0, 900.0, n, dtype=torch.float64, device=cuda)
    t = ops.setup(model, params, grid[:1], precision=_lib.FP64, jvp=True)
    cot = [torch.randn((batch, n), dtype=torch.complex128, device=cuda) for _ in range(2)]
    data, weights = torch.randn(n, dtype=torch.complex128, device=cuda), torch.rand(n, dtype=torch.float64, device=cuda)

    def run():
        loss, grad = ops.fused_loss(model, t.table, t.dtable, grid, None, None, data, weights)
        alone, _ = ops.fused_loss(model, t.table, None, grid, None, None, data, weights)
        return ops.vjp(model, t.table, t.dtable, grid, None, None, *cot), grad, loss[:, None], alone[:, None]

    ways = []
    for workspace in (ops.workspace, lambda *arguments: None):
        monkeypatch.setattr(ops, "workspace", workspace)
        first = run()
        for _ in range(6):
            assert all(torch.equal(a, b) for a, b in zip(run(), first))
        assert torch.equal(first[2], first[3])
        ways.append(first)
    for a, b in zip(*ways):
        assert bool(((a - b).abs() <= 1e-8 * b.abs().amax(1, keepdim=True)).all())


@pytest.mark.parametrize("model", ["IMRPhenomXAS", "IMRPhenomD", "TaylorF2", "IMRPhenomXHM"])
@pytest.mark.parametrize("batch", [1, 2000])
def test_fp64_reverse_pass_beside_odd_frequencies(cuda, model, batch):
    """A frequency whose powers overflow where nothing reads them (above
    IMRPhenomXAS's cutoff, infinity included; with a zero cotangent) leaves the
    gradient of the others: the grid's without it, to 1e-9 of the largest
    component (150 terms summed in another order, cancelling by less than 1e5).
    One at which the waveform is not finite gives NaN."""
    import torch

    from waveformx_b200 import _lib, ops

    p = torch.tensor([[36.0, 29.0, 0.3, -0.1, 500.0, 0.7, 1.2, 20.0]], dtype=torch.float64, device=cuda).repeat(batch, 1)
    f_min = torch.tensor([20.0], dtype=torch.float64, device=cuda)
    grid = torch.linspace(20.0, 900.0, 150, dtype=torch.float64, device=cuda)
    g = torch.full((batch, 150), 0.3 + 0.2j, dtype=torch.complex128, device=cuda)
    rest = torch.arange(150, device=cuda) != 70
    t = None if model == "IMRPhenomXHM" else ops.setup(model, p, f_min, precision=_lib.FP64, jvp=True)

    def gradient(f, g):
        if t is None:
            return ops.xhm_vjp(p, f_min, f, None, None, g, g)
        return ops.vjp(model, t.table, t.dtable, f, None, None, g, g)

    expected = gradient(grid[rest], g[:, rest].contiguous())
    cut = model == "IMRPhenomXAS"
    for odd, weight in ((1e120, 0.0), (1e140, 0.0), (1e160, 0.0), (1e200, 0.0), (1e-104, 0.0),
                        *(((1e160, 1.0), (float("inf"), 0.0), (float("inf"), 1.0)) if cut else ())):
        f, w = grid.clone(), g.clone()
        f[70] = odd
        w[:, 70] *= weight
        got = gradient(f, w)
        assert bool(((got - expected).abs() <= 1e-9 * expected.abs().max()).all()), (odd, weight, got)
    for odd in (0.0, -5.0, float("nan"), -float("inf"), *(() if cut else (float("inf"),))):
        f = grid.clone()
        f[70] = odd
        assert bool(torch.isnan(gradient(f, g)).all()), odd


@pytest.mark.parametrize("model", ["IMRPhenomXAS", "IMRPhenomD", "TaylorF2"])
@pytest.mark.parametrize("kind", ["band", "above", "odd"])
def test_fp64_shared_grids_are_not_finite_where_ragged_ones_are_not(cuda, model, kind):
    """Refused binaries (a zero distance, a mass ratio beyond the fits, spins
    above one, a NaN mass) and odd frequencies (infinities, NaN, zero, a
    negative one) on a shared grid, in the band and wholly above
    IMRPhenomXAS's cutoffs, against the same rows as a ragged grid (the kernels
    of a binary a block): strain, vjp, likelihood and its gradient are NaN in
    the same places, and equal elsewhere (strain 1e-12 of a row's largest;
    sums 1e-9, as the module's other comparison of the two)."""
    import torch

    from waveformx_b200 import _lib, ops

    base = np.array([[36.0, 29.0, 0.3, -0.1, 500.0, 0.7, 1.2, 20.0], [36.0, 29.0, 0.3, -0.1, 0.0, 0.7, 1.2, 20.0],
                     [1500.0, 1.0, 0.0, 0.0, 500.0, 0.7, 1.2, 20.0], [36.0, 29.0, 1.5, -0.1, 500.0, 0.7, 1.2, 20.0],
                     [np.nan, 29.0, 0.3, -0.1, 500.0, 0.7, 1.2, 20.0], [60.0, 15.0, 0.8, 0.5, 1000.0, 2.5, 4.0, 20.0]])
    n, batch = 300, 6 * 400
    f = np.linspace(20.0, 900.0, n) if kind != "above" else np.linspace(3000.0, 4500.0, n)
    if kind == "odd":
        f[[7, 90]], f[200:264] = (0.0, -5.0), np.inf
        f[130] = np.nan
    grid = torch.as_tensor(f, device=cuda)
    t = ops.setup(model, torch.as_tensor(base, device=cuda), torch.tensor([20.0], dtype=torch.float64, device=cuda),
                  precision=_lib.FP64, jvp=True)
    of = torch.arange(batch, device=cuda) % 6
    rng = np.random.default_rng(0)
    g = torch.as_tensor(rng.normal(size=(6, n)) + 1j * rng.normal(size=(6, n)), device=cuda)
    w = torch.as_tensor(rng.uniform(0.5, 2.0, n), device=cuda)
    offsets = torch.arange(7, device=cuda) * n
    table, dtable = t.table[of].contiguous(), t.dtable[of].contiguous()
    for rows, tab, dtab in ((torch.arange(6, device=cuda), t.table, t.dtable), (of, table, dtable)):
        shared = [*ops.polarizations(model, tab, grid), ops.vjp(model, tab, dtab, grid, None, None, *(g[rows].contiguous(),) * 2),
                  *ops.fused_loss(model, tab, dtab, grid, None, None, g[0].contiguous(), w)]
        ragged = [*(h.reshape(6, n) for h in ops.polarizations(model, t.table, grid.repeat(6), offsets)),
                  ops.vjp(model, t.table, t.dtable, grid.repeat(6), offsets, None, *(g.reshape(-1),) * 2),
                  *ops.fused_loss(model, t.table, t.dtable, grid.repeat(6), offsets, None, g[0].repeat(6), w.repeat(6))]
        for k, (a, b) in enumerate(zip(shared, ragged)):
            a, b = (torch.view_as_real(x) if x.is_complex() else x for x in (a, b[rows]))
            assert torch.equal(torch.isnan(a), torch.isnan(b)), k
            a, b = torch.nan_to_num(a, 0.0, 0.0, 0.0).flatten(1 if a.ndim > 1 else 0), torch.nan_to_num(b, 0.0, 0.0, 0.0).flatten(
                1 if b.ndim > 1 else 0)
            scale = b.abs().amax(1, keepdim=True) if b.ndim > 1 else b.abs()
            assert bool(((a - b).abs() <= (1e-12 if k < 2 else 1e-9) * scale).all()), k


@pytest.mark.parametrize("model", ["IMRPhenomXAS", "IMRPhenomD", "TaylorF2"])
@pytest.mark.parametrize("n, batch", [(65, 3), (300, 40), (2049, 1), (2080, 3), (2175, 70), (4017, 51), (700, 600), (257, 1001)])
def test_fp64_reverse_pass_against_a_binary_a_block(cuda, model, n, batch):
    """The FP64 vjp and fused likelihood of a shared grid where four or two
    warps share a binary's span, with a last group of one, where a warp takes a
    binary, and where a block does, at remainders of spans and of a warp's
    frequencies, against the same rows as a ragged grid (a binary a block): the
    same sums in another order, 1e-8 of a binary's largest component (they
    round to 1e-13 of their terms' magnitudes, which the contraction cancels
    by less than 1e5)."""
    import torch

    from waveformx_b200 import _lib, ops

    rng = np.random.default_rng(n)
    params = torch.as_tensor(draw_batch(rng, batch), device=cuda)
    grid = torch.linspace(20.0, 900.0, n, dtype=torch.float64, device=cuda)
    t = ops.setup(model, params, grid[:1], precision=_lib.FP64, jvp=True)
    t_c = torch.as_tensor(rng.uniform(-0.1, 0.1, batch), device=cuda)
    cot = [torch.randn((batch, n), dtype=torch.complex128, device=cuda) for _ in range(2)]
    w = torch.rand((batch, n), dtype=torch.float64, device=cuda)
    offsets = torch.arange(batch + 1, device=cuda) * n
    flat = (t.table, t.dtable, grid.repeat(batch), offsets, t_c)
    shared = [ops.vjp(model, t.table, t.dtable, grid, None, t_c, *cot),
              *ops.fused_loss(model, t.table, t.dtable, grid, None, t_c, cot[0], w, antenna=(0.6, -0.3), scale=-0.5)]
    ragged = [ops.vjp(model, *flat, *(c.reshape(-1) for c in cot)),
              *ops.fused_loss(model, *flat, cot[0].reshape(-1), w.reshape(-1), antenna=(0.6, -0.3), scale=-0.5)]
    for a, b in zip(shared, ragged):
        scale = b.abs().amax(1, keepdim=True) if b.ndim > 1 else b.abs()
        assert bool(((a - b).abs() <= 1e-8 * scale).all())
