"""The PyTorch drop-in (``waveformx_b200.torch.polarizations_function``):
the behaviour of the reference's ``waveformx.torch`` (its
``tests/test_torch.py``): values against the oracle, gradients of a fixed
real function of the polarizations against central differences, inputs as
mappings, numbers and sequences, broadcasting, the batch rules and errors,
float32/float64 selection and host tensors in and out."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from conftest import compare
from test_gpu_gradients import fd_gradient, weighted_loss

pytestmark = pytest.mark.gpu

FREQUENCIES = np.geomspace(20.0, 900.0, 300)
ALIGNED = [36.0, 29.0, 0.0, 0.0, 0.3, 0.0, 0.0, -0.4, 500.0, 0.7, 1.2, 25.0]
BATCH = [ALIGNED, [50.0, 8.0, 0.0, 0.0, 0.9, 0.0, 0.0, 0.3, 300.0, 2.1, 0.3, 30.0],
         [150.0, 100.0, 0.0, 0.0, -0.5, 0.0, 0.0, 0.95, 3000.0, 0.4, 2.0, 0.0]]


def binary_of(x):
    import waveformx_b200 as wb

    return wb.Binary(x[..., 0], x[..., 1], x[..., 2:5], x[..., 5:8], x[..., 8], x[..., 9], x[..., 10], x[..., 11])


def aligned(rows):
    rows = np.atleast_2d(rows)
    return rows[:, [0, 1, 4, 7, 8, 9, 10, 11]]


@pytest.mark.parametrize("approximant", ["IMRPhenomXAS", "IMRPhenomD", "TaylorF2"])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("batched", [False, True])
def test_values_and_gradients(cuda, approximant, dtype, batched):
    import torch

    import waveformx_b200.torch as wt

    tdtype = getattr(torch, dtype)
    rows = np.asarray(BATCH if batched else ALIGNED)
    if dtype == "float32":
        rows = rows.astype(np.float32).astype(np.float64)
    grid = FREQUENCIES.astype(np.float32).astype(np.float64) if dtype == "float32" else FREQUENCIES
    f = wt.polarizations_function(approximant)
    fields = [torch.tensor(np.asarray(v), dtype=tdtype, device=cuda, requires_grad=True) for v in binary_of(rows)]
    import waveformx_b200 as wb

    hp, hc = f(wb.Binary(*fields), torch.tensor(grid, dtype=tdtype, device=cuda))
    assert hp.dtype == (torch.complex64 if dtype == "float32" else torch.complex128)
    assert hp.shape == ((3, len(grid)) if batched else (len(grid),))
    ref_p, ref_c = oracle.polarizations(approximant, aligned(rows), grid)
    if not batched:
        ref_p, ref_c = ref_p[0], ref_c[0]
    tol = 1e-10 if dtype == "float64" else 1e-4
    for a, b in ((hp, ref_p), (hc, ref_c)):
        a = a.detach().cpu().numpy()
        np.testing.assert_allclose(a, b, rtol=tol, atol=tol * np.max(np.abs(b)))
    w = np.random.default_rng(5).normal(size=(4,) + tuple(hp.shape))
    tw = torch.as_tensor(w, dtype=tdtype, device=cuda)
    loss = (tw[0] * hp.real + tw[1] * hp.imag + tw[2] * hc.real + tw[3] * hc.imag).sum()
    grads = torch.autograd.grad(loss, fields)
    params = aligned(rows)
    wl = w if batched else w[:, None, :]
    fd = fd_gradient(lambda p, tc: weighted_loss(approximant, p, grid, tc, wl), params, np.zeros(len(params)))
    # (f_ref = 0 selects the first frequency, or for TaylorF2 the reference
    # at coalescence: no derivative there)
    fd[params[:, 7] == 0, 7] = 0.0
    expected = [fd[:, 0], fd[:, 1], fd[:, 2], fd[:, 3], fd[:, 4], fd[:, 5], fd[:, 6], fd[:, 7]]
    for k, (g, e) in enumerate(zip(grads, expected)):
        g = g.detach().cpu().numpy().astype(np.float64)
        if k in (2, 3):
            assert np.all(g[..., :2] == 0)
            g = g[..., 2]
        g = np.reshape(g, np.shape(e))
        scale = np.max(np.abs(fd), axis=1)
        if k == 7:
            e = np.where(params[:, 7] == 0, g, e)
        if dtype == "float64":
            np.testing.assert_allclose(g, e, rtol=1e-5, atol=1e-6 * scale.max(), err_msg=str(k))
        else:
            assert np.all(np.abs(g - e) <= 1e-2 * np.abs(e) + 1e-3 * scale), (k, g, e)


def test_inputs(cuda):
    """Mappings, numbers, sequences of tensors and broadcast fields; the
    gradient reaches each tensor asked for; the reference's errors."""
    import torch

    import waveformx_b200 as wb
    import waveformx_b200.torch as wt

    f = wt.polarizations_function("IMRPhenomXAS")
    grid = torch.tensor(FREQUENCIES, device=cuda)
    reference = f(binary_of(torch.tensor(ALIGNED, dtype=torch.float64, device=cuda)), grid)
    chi = torch.tensor(0.3, dtype=torch.float64, device=cuda, requires_grad=True)
    binary = dict(mass_1=36.0, mass_2=29, spin_1=(0.0, 0.0, chi), spin_2=[0.0, 0.0, -0.4],
                  luminosity_distance=500.0, inclination=0.7, phi_ref=1.2, f_ref=25.0)
    hp, hc = f(binary, grid)
    assert hp.dtype == torch.complex128
    for a, b in zip((hp, hc), reference):
        torch.testing.assert_close(a, b, rtol=0, atol=0)
    (g,) = torch.autograd.grad(hp.abs().sum(), chi)
    assert torch.isfinite(g) and g != 0
    masses = torch.tensor([36.0, 40.0], dtype=torch.float64, device=cuda, requires_grad=True)
    hp, hc = f({**binary, "mass_1": masses}, grid)
    assert hp.shape == (2, len(FREQUENCIES))
    torch.testing.assert_close(hp[0].detach(), reference[0], rtol=1e-12, atol=1e-12 * float(reference[0].abs().max()))
    g_m, g_chi = torch.autograd.grad(hp.abs().sum(), (masses, chi))
    assert g_m.shape == (2,) and g_chi.shape == ()
    with pytest.raises(TypeError, match="unknown"):
        f({**binary, "mass": 1.0}, grid)
    with pytest.raises(TypeError, match="missing"):
        f({"mass_1": 1.0}, grid)
    with pytest.raises(ValueError, match="batch"):
        f({**binary, "mass_1": masses, "mass_2": torch.ones(3, device=cuda)}, grid)
    with pytest.raises(wb.UnknownApproximantError):
        wt.polarizations_function("IMRPhenomXYZ")
    with pytest.raises(wb.UnsupportedError):
        wt.polarizations_function("NRSur7dq4")
    # host tensors in, host tensors out (copied through the device)
    hp_cpu, _ = f(binary_of(torch.tensor(ALIGNED, dtype=torch.float64)), torch.tensor(FREQUENCIES))
    assert hp_cpu.device.type == "cpu"
    torch.testing.assert_close(hp_cpu, reference[0].cpu(), rtol=0, atol=0)


def test_t_c_extension(cuda):
    """t_c as a keyword or a mapping entry, with its gradient."""
    import torch

    import waveformx_b200.torch as wt

    f = wt.polarizations_function("IMRPhenomXAS")
    grid = torch.tensor(FREQUENCIES, device=cuda)
    b = binary_of(torch.tensor(ALIGNED, dtype=torch.float64, device=cuda))
    t_c = torch.tensor(0.03, dtype=torch.float64, device=cuda, requires_grad=True)
    hp, hc = f(b, grid, t_c=t_c)
    hp0, _ = f(b, grid)
    shift = torch.exp(-2j * np.pi * grid * 0.03)
    torch.testing.assert_close(hp, hp0 * shift, rtol=1e-10, atol=1e-10 * float(hp0.abs().max()))
    hp2, _ = f({**b._asdict(), "t_c": t_c}, grid)
    torch.testing.assert_close(hp2, hp, rtol=0, atol=0)
    (g,) = torch.autograd.grad(hp.real.sum(), t_c)
    eps = 1e-7
    num = (f(b, grid, t_c=0.03 + eps)[0].real.sum() - f(b, grid, t_c=0.03 - eps)[0].real.sum()) / (2 * eps)
    assert float(g) == pytest.approx(float(num), rel=1e-5)


def test_compare_metric_on_c0(cuda):
    """The single-binary workload (float64) through the torch function."""
    import torch

    import waveformx_b200 as wb
    import waveformx_b200.torch as wt
    from conftest import golden

    g = golden("xas_cases")
    p = g["single_params"][0]
    f = wt.polarizations_function("IMRPhenomXAS")
    hp, hc = f(wb.Binary(p[0], p[1], (0, 0, p[2]), (0, 0, p[3]), p[4], p[5], p[6], p[7]),
               torch.tensor(g["single_frequencies"], device=cuda))
    for a, b in ((hp, g["single_hplus"]), (hc, g["single_hcross"])):
        error, mismatch = compare(a.cpu().numpy(), b)
        assert error < 1e-10 and mismatch < 1e-14


@pytest.mark.parametrize("approximant", ["IMRPhenomXAS", "TaylorF2", "IMRPhenomXHM"])
def test_empty_inputs(cuda, approximant):
    """No binary, or no frequency: empty outputs of the batch's shape, and
    zero gradients of the fields' shapes (the reference's vmapped function
    on empty axes)."""
    import torch

    import waveformx_b200.torch as wt

    f = wt.polarizations_function(approximant)
    grid = torch.as_tensor(FREQUENCIES, device=cuda)
    empty = torch.as_tensor(np.zeros((0, 12)), device=cuda).requires_grad_(True)
    hp, hc = f(binary_of(empty), grid)
    assert tuple(hp.shape) == (0, len(FREQUENCIES)) and hp.dtype == torch.complex128
    (hp.real.sum() + hc.imag.sum()).backward()
    assert tuple(empty.grad.shape) == (0, 12)
    rows = torch.as_tensor(np.array(BATCH), device=cuda).requires_grad_(True)
    no_freq = torch.zeros(0, dtype=torch.float64, device=cuda)
    hp, hc = f(binary_of(rows), no_freq)
    assert tuple(hp.shape) == (3, 0)
    (hp.real.sum() + hc.real.sum()).backward()
    assert torch.equal(rows.grad, torch.zeros_like(rows))
    hp, hc = f(binary_of(rows[0].detach().float()), no_freq.float())
    assert tuple(hp.shape) == (0,) and hp.dtype == torch.complex64


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("n", [0, 1, 3, 257])
def test_fields_without_conversion(cuda, dtype, n):
    """The drop-in on tensors of one dtype and device (no conversion) equals
    the general way (the same binary with one field as a list): strain and
    gradients bit for bit, for one binary (n = 0: fields without an axis) and
    batches, with expanded, strided and negative-view fields."""
    import torch

    import waveformx_b200.torch as wt

    real = getattr(torch, dtype)
    rng = np.random.default_rng(n)
    rows = max(n, 1)
    m = np.sort(rng.uniform(10.0, 60.0, (rows, 2)))[:, ::-1]
    chi = rng.uniform(-0.8, 0.8, (rows, 2))
    host = {"mass_1": m[:, 0], "mass_2": m[:, 1], "spin_1": np.stack([0 * chi[:, 0], 0 * chi[:, 0], chi[:, 0]], -1),
            "spin_2": np.stack([0 * chi[:, 0], 0 * chi[:, 0], chi[:, 1]], -1),
            "luminosity_distance": rng.uniform(100.0, 900.0, rows), "inclination": rng.uniform(0.1, 3.0, rows),
            "phi_ref": rng.uniform(0.0, 6.0, rows), "f_ref": np.full(rows, 20.0)}
    grid = torch.linspace(20.0, 400.0, 131, dtype=real, device=cuda)
    f = wt.polarizations_function("IMRPhenomXAS")
    out = []
    for general in (False, True):
        b = {k: torch.as_tensor(v if n else v[0], dtype=real, device=cuda).clone() for k, v in host.items()}
        # a strided field, an expanded one and a negative view
        b["spin_2"] = torch.stack([b["spin_2"], b["spin_2"]], -1)[..., 0]
        if n:
            b["f_ref"] = torch.full((), 20.0, dtype=real, device=cuda).expand(n)
        b["inclination"] = torch._neg_view(-b["inclination"])
        leaves = {k: b[k].detach().requires_grad_(True) for k in ("mass_1", "spin_1", "phi_ref")}
        b.update(leaves)
        if general:
            b["luminosity_distance"] = list(b["luminosity_distance"].unbind()) if n else [b["luminosity_distance"]]
        hp, hc = f(b, grid)
        hp, hc = hp.reshape(rows, -1), hc.reshape(rows, -1)
        gradients = torch.autograd.grad((hp.abs() ** 2).sum() + hc.real.sum(), list(leaves.values()))
        out.append([hp.detach(), hc.detach(), *(g.reshape(-1) for g in gradients)])
    for x, y in zip(*out):
        assert torch.equal(x, y)


@pytest.mark.parametrize("approximant", ["IMRPhenomXAS", "IMRPhenomD", "TaylorF2", "IMRPhenomXHM"])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("batched", [False, True])
def test_losses_with_the_strain_under_conj(cuda, approximant, dtype, batched):
    """A loss with the strain under ``conj`` sends the backward a conjugate
    view: its gradients are those of the same loss with the other factor
    conjugated. Bar: 200 terms' rounding in any order, 1e-12 (float64) or 1e-5
    of a field's largest; the conjugate cotangent's gradients differ in the
    first digit."""
    import torch

    import waveformx_b200.torch as wt
    from waveformx_b200 import match

    real = getattr(torch, dtype)
    rows = torch.tensor(BATCH if batched else ALIGNED, dtype=real, device=cuda)
    grid = torch.linspace(20.0, 400.0, 200, dtype=real, device=cuda)
    rng = np.random.default_rng(5)
    d = torch.as_tensor(rng.normal(size=200) + 1j * rng.normal(size=200), device=cuda).to(
        torch.complex64 if dtype == "float32" else torch.complex128)
    w = torch.as_tensor(oracle.psd(np.linspace(20.0, 400.0, 200)), device=cuda).to(real)
    f = wt.polarizations_function(approximant)

    def gradient(loss):
        x = rows.clone().requires_grad_(True)
        t_c = torch.full(rows.shape[:-1], 0.01, dtype=real, device=cuda, requires_grad=True)
        hp, hc = f(binary_of(x), grid, t_c=t_c)
        return torch.autograd.grad(loss(hp) + 0.5 * loss(hc), (x, t_c))

    pairs = [(lambda h: (h.conj() * d * w).real.sum(), lambda h: (h * d.conj() * w).real.sum()),
             (lambda h: (torch.conj(h) @ d).imag.sum(), lambda h: -(h @ torch.conj(d)).imag.sum()),
             (lambda h: match.inner_product(d, h, grid, w).sum(), lambda h: match.inner_product(h, d, grid, w).sum())]
    tol = 1e-12 if dtype == "float64" else 1e-5
    for under, other in pairs:
        for a, b in zip(gradient(under), gradient(other)):
            scale = b.abs().amax(0) if batched else b.abs()
            assert bool((b != 0).any()) and bool(((a - b).abs() <= tol * scale).all())


def test_inputs_that_are_negative_views(cuda):
    """The grid and ``t_c`` as negative views (contiguous, and negated as they
    are read) give the strain of their values."""
    import torch

    import waveformx_b200.torch as wt

    f = wt.polarizations_function("IMRPhenomXAS")
    grid = torch.linspace(20.0, 400.0, 65, dtype=torch.float64, device=cuda)
    t_c = torch.tensor([0.01, -0.02, 0.3], dtype=torch.float64, device=cuda)
    b = binary_of(torch.tensor(BATCH, dtype=torch.float64, device=cuda))
    expected = f(b, grid, t_c=t_c)
    for got in (f(b, torch._neg_view(-grid), t_c=t_c), f(b, grid, t_c=torch._neg_view(-t_c))):
        assert all(torch.equal(x, y) for x, y in zip(got, expected))


def test_operations_refuse_lazy_views(cuda):
    """The tensor operations, which read their arguments' memory, refuse
    conjugate and negative views."""
    import torch

    from waveformx_b200 import _lib, ops

    p = torch.as_tensor(np.ascontiguousarray(aligned(BATCH)), device=cuda)
    grid = torch.linspace(20.0, 400.0, 65, dtype=torch.float64, device=cuda)
    t = ops.setup("IMRPhenomXAS", p, grid[:1], precision=_lib.FP64, jvp=True)
    g = torch.randn((3, 65), dtype=torch.complex128, device=cuda)
    with pytest.raises(ValueError, match="conjugate"):
        ops.vjp("IMRPhenomXAS", t.table, t.dtable, grid, None, None, g.conj(), g)
    with pytest.raises(ValueError, match="negative"):
        ops.polarizations("IMRPhenomXAS", t.table, torch._neg_view(-grid))
    # (those that convert their cotangents take them)
    a = ops.grid_vjp("IMRPhenomXAS", t.table, grid, None, None, g.conj(), g)
    b = ops.grid_vjp("IMRPhenomXAS", t.table, grid, None, None, g.conj().resolve_conj(), g)
    torch.testing.assert_close(a, b, rtol=1e-12, atol=0)


@pytest.mark.parametrize("approximant", ["IMRPhenomXAS", "IMRPhenomXHM"])
@pytest.mark.parametrize("device", ["cuda", "cpu"])
@pytest.mark.parametrize("batched", [False, True])
def test_in_place_operations_on_the_strain(cuda, approximant, device, batched):
    """A strain that requires a gradient can be masked, scaled and added to in
    place, one binary's as a batch's, from a grid on either device: the
    gradients of the same operations out of place."""
    import torch

    import waveformx_b200.torch as wt

    rows = torch.tensor(BATCH if batched else ALIGNED, dtype=torch.float64, device=device)
    grid = torch.linspace(20.0, 400.0, 120, dtype=torch.float64, device=device)
    window = torch.hann_window(120, dtype=torch.float64, device=device)
    f = wt.polarizations_function(approximant)
    out = []
    for in_place in (True, False):
        x = rows.clone().requires_grad_(True)
        hp, hc = f(binary_of(x), grid)
        if in_place:
            hp *= window
            hp[..., grid < 50.0] = 0
            hc.mul_(0.5).add_(hp)
        else:
            hp = torch.where(grid < 50.0, 0.0, hp * window)
            hc = 0.5 * hc + hp
        (hp.abs() ** 2).sum().backward(retain_graph=True)
        hc.real.sum().backward()
        out.append((hp.detach(), hc.detach(), x.grad))
    for a, b in zip(*out):
        torch.testing.assert_close(a, b, rtol=1e-12, atol=1e-12 * float(b.abs().max()))


@pytest.mark.parametrize("batched", [False, True])
def test_gradients_of_the_fields_are_tensors_of_their_own(cuda, batched):
    """An in-place change of one field's ``.grad`` leaves the others as they
    were, their use in another graph included."""
    import torch

    import waveformx_b200.torch as wt
    import waveformx_b200 as wb

    rows = np.asarray(BATCH if batched else ALIGNED)
    fields = [torch.tensor(np.asarray(v), dtype=torch.float64, device=cuda, requires_grad=True) for v in binary_of(rows)]
    hp, hc = wt.polarizations_function("IMRPhenomXAS")(wb.Binary(*fields), torch.linspace(20.0, 400.0, 65, dtype=torch.float64,
                                                                                       device=cuda))
    ((hp.abs() ** 2).sum() + hc.real.sum()).backward()
    factor = torch.ones((), dtype=torch.float64, device=cuda, requires_grad=True)
    held = [x.grad.clone() for x in fields]
    total = sum((factor * x.grad).sum() for x in fields[1:])  # (keeps the gradients for factor's)
    fields[0].grad.zero_()
    total.backward()
    assert all(torch.equal(x.grad, g) for x, g in zip(fields[1:], held[1:]))
    torch.testing.assert_close(factor.grad, sum(g.sum() for g in held[1:]), rtol=1e-12, atol=0)
    fields[2].grad.mul_(factor)  # (as of a tensor with a history)


@pytest.mark.parametrize("needs", [False, True])
@pytest.mark.parametrize("general", [False, True])
def test_grids_of_another_rank(cuda, needs, general):
    """A grid without an axis is an IndexError, and one whose first entry is
    neither one frequency nor one a binary a ValueError, with tensors of one
    type and with fields that are converted; a column is its frequencies."""
    import torch

    import waveformx_b200.torch as wt

    f = wt.polarizations_function("IMRPhenomXAS")
    grid = torch.linspace(20.0, 400.0, 60, dtype=torch.float64, device=cuda)
    for rows in (BATCH, ALIGNED):
        x = torch.tensor(rows, dtype=torch.float64, device=cuda, requires_grad=needs)
        b = binary_of(x)
        if general:
            b = b._replace(luminosity_distance=500.0)
        with pytest.raises(IndexError):
            f(b, grid[0])
        for shape in ((30, 2), (12, 5), (3, 20)):
            with pytest.raises(ValueError, match="f_min"):
                f(b, grid.reshape(shape))
        for a, c in zip(f(b, grid.reshape(60, 1)), f(b, grid)):
            assert a.shape == c.shape and torch.equal(a, c)
    with pytest.raises(ValueError, match="f_min"):
        from waveformx_b200 import ops

        ops.setup_jvp_async("IMRPhenomXAS", torch.ones((3, 8), dtype=torch.float64, device=cuda), grid[:2])


@pytest.mark.parametrize("model", ["IMRPhenomXAS", "IMRPhenomD", "TaylorF2", "IMRPhenomXHM"])
def test_gradients_with_saved_tensor_hooks_and_on_other_streams(cuda, model):
    """The gradients of a batch with its saved tensors moved to the host (the
    set-up's derivatives, which a second stream forms, among them), and with
    the whole call on another stream than the default, several calls under
    way: those of the plain call, 1e-12 of a field's largest."""
    import torch

    import waveformx_b200.torch as wt

    rng = np.random.default_rng(4)
    m = np.sort(rng.uniform(10.0, 60.0, (2000, 2)))[:, ::-1]
    x = torch.as_tensor(np.concatenate([m, np.zeros((2000, 2)), rng.uniform(-0.8, 0.8, (2000, 1)), np.zeros((2000, 2)),
                                        rng.uniform(-0.8, 0.8, (2000, 1)), rng.uniform(100.0, 900.0, (2000, 1)),
                                        rng.uniform(0.1, 3.0, (2000, 2)), np.full((2000, 1), 20.0)], 1), device=cuda)
    grid = torch.linspace(20.0, 400.0, 33, dtype=torch.float64, device=cuda)
    f = wt.polarizations_function(model)

    def gradient(rows):
        leaf = rows.clone().requires_grad_(True)
        hp, hc = f(binary_of(leaf), grid)
        return torch.autograd.grad((hp.abs() ** 2).sum() + hc.real.sum(), leaf)[0]

    expected = [gradient(x), gradient(x[::2])]
    with torch.autograd.graph.save_on_cpu():
        got = [gradient(x), gradient(x[::2])]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for _ in range(3):
        for s in streams:
            with torch.cuda.stream(s):
                got += [gradient(x), gradient(x[::2])]
    torch.cuda.synchronize()
    for k, g in enumerate(got):
        e = expected[k % 2]
        assert bool(((g - e).abs() <= 1e-12 * e.abs().amax(0)).all())


@pytest.mark.parametrize("batched", [False, True])
def test_host_inputs_take_one_copy_back_of_the_gradient(cuda, batched, monkeypatch):
    """With a grid and a binary on the host, a call copies the two strains
    back, and its backward the fields' gradients in one copy (each waits for
    the device)."""
    import torch

    import waveformx_b200 as wb
    import waveformx_b200.torch as wt

    fields = [torch.tensor(np.asarray(v), dtype=torch.float64, requires_grad=True)
              for v in binary_of(np.asarray(BATCH if batched else ALIGNED))]
    f = wt.polarizations_function("IMRPhenomXAS")
    grid = torch.linspace(20.0, 400.0, 65, dtype=torch.float64)
    copies, to = [], torch.Tensor.to

    def counted(self, *args, **kw):
        out = to(self, *args, **kw)
        if self.is_cuda and not out.is_cuda:
            copies.append(out.shape)
        return out

    monkeypatch.setattr(torch.Tensor, "to", counted)
    hp, hc = f(wb.Binary(*fields), grid)
    assert len(copies) == 2
    gradients = torch.autograd.grad((hp.abs() ** 2).sum() + hc.real.sum(), fields)
    assert len(copies) == 3
    assert all(g.device.type == "cpu" and g.shape == x.shape for g, x in zip(gradients, fields))
