"""The workloads by which this framework's speed is judged: what a program
that infers the parameters of compact binaries calls, through the public
entry points, from one waveform to a night's catalogue.

A case names the call it makes (one of ``CALLS``), the approximant, the
precision and the sizes. ``prepare`` makes what the program has in hand,
``run`` makes the call, ``work`` counts what the call cannot do without and
``exact`` gives its outputs in 64 bits where plain torch can.

The binaries are drawn as this repository's batch configurations draw them:
component masses uniform in 5 to 100 solar masses, aligned spins uniform in
[-0.99, 0.99], distances uniform in 100 to 5000 Mpc, isotropic inclination,
uniform phase, f_ref = 20 Hz. The noise weights are 1 / S(f) with
S(f) = (f/20)^-4 + 2 + (f/200)^2.
"""

import math

import numpy as np
import torch

MTSUN = 4.925490947641267e-06  # G Msun / c^3 (s)
MODELS = ("IMRPhenomXAS", "IMRPhenomD", "TaylorF2", "IMRPhenomXHM")
ROWED = MODELS[:3]  # the models whose likelihood is fused
REAL = {"float32": torch.float32, "float64": torch.float64}
COMPLEX = {"float32": torch.complex64, "float64": torch.complex128}
FIELDS = ("mass_1", "mass_2", "spin_1", "spin_2", "luminosity_distance", "inclination", "phi_ref", "f_ref")

#: The grid of the batch configurations is linspace(20, 1024, 4017), the
#: wide likelihood's linspace(10, 2048, 8192): 4 and 4 points a hertz.
GRID_POINTS, WIDE_POINTS = 4017, 8192


def listed():
    return [
        # A notebook or a plot: one binary, the reference's default precision
        # (double), the batch configurations' grid. Launches and host work.
        _case("one waveform", "polarizations", "IMRPhenomXAS", "float64", 1, GRID_POINTS),
        # The headline: a population's strain in single precision.
        _case("population", "polarizations", "IMRPhenomXAS", "float32", 4096, GRID_POINTS),
        # The same with the higher modes (a quarter of the binaries).
        _case("population with higher modes", "polarizations", "IMRPhenomXHM", "float32", 1024, GRID_POINTS),
        # The reference's batch API from host tables in its default
        # precision: checks, device copies, strain, finiteness.
        _case("batch api, double", "batch", "IMRPhenomD", "float64", 1000, GRID_POINTS),
        # A differentiated loss through autograd (the vjp of the drop-in).
        _case("training step", "backward", "IMRPhenomXAS", "float32", 1024, GRID_POINTS),
        # The same in double, odd sizes: Fisher matrices and Hamiltonian
        # samplers that need the digits.
        _case("gradients in double", "backward", "IMRPhenomXAS", "float64", 1021, 4001),
        # Higher-mode gradients (double whatever the inputs).
        _case("higher-mode gradients", "backward", "IMRPhenomXHM", "float64", 250, 4017),
        # A catalogue whose events each have their own band and duration.
        _case("ragged catalogue", "ragged", "IMRPhenomXAS", "float32", 16384, 0),
        # One detector's likelihood and gradient over a large set of samples
        # whose tables are laid out (every detector reuses them).
        _case("detector likelihood", "likelihood", "IMRPhenomXAS", "float32", 65536, WIDE_POINTS),
        # A sampler's walkers, replayed as one captured graph: latency.
        _case("sampler step", "sampler", "TaylorF2", "float32", 128, WIDE_POINTS),
        # A template bank against one signal.
        _case("template bank", "bank", "IMRPhenomXAS", "float32", 4096, GRID_POINTS),
        # Matches of given waveforms in double (a faithfulness study).
        _case("matches in double", "match", "given", "float64", 500, GRID_POINTS),
    ]


def _case(name, call, model, dtype, binaries, points):
    case = {"name": name, "call": call, "model": model, "dtype": dtype, "binaries": binaries, "points": points}
    return {k: v for k, v in case.items() if v != ""}


#: Each call: its share of the draws, its models and precisions, the largest
#: batch, the range of the grid's points and the largest binaries x points.
CALLS = {
    "polarizations": (4, MODELS, ("float32", "float64"), 8192, (65, 16384), 1 << 24),
    "batch": (1, MODELS, ("float32", "float64"), 4096, (129, 8192), 1 << 22),
    "backward": (3, MODELS, ("float32", "float64"), 4096, (65, 8192), 1 << 24),
    "ragged": (1, ROWED, ("float32",), 16384, (0, 0), 0),
    "likelihood": (2, ROWED, ("float32", "float64"), 65536, (257, 8192), 1 << 26),
    "sampler": (2, ROWED, ("float32",), 2048, (129, 16384), 1 << 23),
    "bank": (1, ROWED, ("float32",), 8192, (257, 8192), 1 << 24),
    "match": (1, ("given",), ("float32", "float64"), 4096, (65, 16384), 1 << 21),
}


def draw(rng):
    calls = [call for call, entry in CALLS.items() for _ in range(entry[0])]
    call = rng.choice(calls)
    _, models, dtypes, most, (low, high), evals = CALLS[call]
    model, dtype = rng.choice(models), rng.choice(dtypes)
    points = round(math.exp(rng.uniform(math.log(low), math.log(high)))) if high else 0
    if points:
        if model == "IMRPhenomXHM":
            evals //= 4
        if dtype == "float64":
            evals //= 4
        most = max(1, min(most, evals // points))
    binaries = round(math.exp(rng.uniform(0.0, math.log(most))))
    if call == "ragged":
        binaries = max(2, binaries)
    return _case("", call, model, dtype, binaries, points)


# ---------------------------------------------------------------------------
# inputs

def _binaries(rng, n):
    m = rng.uniform(5.0, 100.0, size=(n, 2))
    chi = rng.uniform(-0.99, 0.99, size=(n, 2))
    return np.stack([m.max(1), m.min(1), chi[:, 0], chi[:, 1], rng.uniform(100.0, 5000.0, n),
                     np.arccos(rng.uniform(-1.0, 1.0, n)), rng.uniform(0.0, 2 * np.pi, n), np.full(n, 20.0)], 1)


def _psd(f):
    return (f / 20.0) ** -4 + 2.0 + (f / 200.0) ** 2


def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _grid(case, dtype):
    if case["points"] >= WIDE_POINTS:
        low, high = 10.0, 2048.0
    else:
        low, high = 20.0, 1024.0
    return torch.linspace(low, high, case["points"], dtype=torch.float64, device=_device()).to(dtype)


def _noise(gen, shape, dtype):
    """Complex Gaussian noise of unit variance."""
    x = torch.randn((*shape, 2), dtype=REAL[dtype], device=_device(), generator=gen) * math.sqrt(0.5)
    return torch.view_as_complex(x)


def _chirp(f, chirp_mass, t0, phase, amplitude):
    """A Newtonian chirp's strain at ``f`` (the last axis)."""
    mc = (torch.pi * MTSUN) * chirp_mass[..., None]
    psi = (3.0 / 128.0) * (mc * f) ** (-5.0 / 3.0) + 2 * torch.pi * f * t0[..., None] + phase[..., None]
    return torch.polar((amplitude[..., None] * (f / 20.0) ** (-7.0 / 6.0)), psi)


def _fields(params, dtype, one):
    """The drop-in's mapping of a binary's fields."""
    p = torch.as_tensor(params, dtype=REAL[dtype], device=_device())
    zero = torch.zeros_like(p[:, 0])
    columns = {"mass_1": p[:, 0], "mass_2": p[:, 1], "spin_1": torch.stack([zero, zero, p[:, 2]], -1),
               "spin_2": torch.stack([zero, zero, p[:, 3]], -1), "luminosity_distance": p[:, 4],
               "inclination": p[:, 5], "phi_ref": p[:, 6], "f_ref": p[:, 7]}
    return {k: (v[0] if one else v).clone() for k, v in columns.items()}


def _ragged(n):
    """The catalogue's grids (the same for every set of parameters tried on
    it): f_low uniform 10 to 30 Hz, duration 4 to 64 s, up to 2048 Hz or
    M f = 0.3 of the event's total mass."""
    rng = np.random.default_rng(n)
    low, duration = rng.uniform(10.0, 30.0, n), 2.0 ** rng.integers(2, 7, n)
    high = np.minimum(2048.0, 0.3 / (MTSUN * rng.uniform(5.0, 100.0, size=(n, 2)).sum(1)))
    lengths = np.maximum(2, np.floor((high - low) * duration).astype(np.int64) + 1)
    offsets = np.concatenate([[0], np.cumsum(lengths)])
    dev = _device()
    offs = torch.as_tensor(offsets, device=dev)
    row = torch.repeat_interleave(torch.arange(n, device=dev), torch.as_tensor(lengths, device=dev))
    k = torch.arange(int(offsets[-1]), device=dev, dtype=torch.float64) - offs[row].to(torch.float64)
    f = torch.as_tensor(low, device=dev)[row] + k / torch.as_tensor(duration, device=dev)[row]
    return offs, f.to(torch.float32)


def _tables(case, params, f_min):
    """The laid-out tables of a set of binaries: the coefficient rows in the
    case's precision, the same rows in double and their derivatives."""
    from waveformx_b200 import _lib, ops

    p = torch.as_tensor(params, device=_device())
    double = ops.setup(case["model"], p, f_min, precision=_lib.FP64, jvp=case["call"] == "likelihood")
    if case["dtype"] == "float64":
        return double.table, double.table, double.dtable
    return ops.setup(case["model"], p, f_min, precision=_lib.FP32).table, double.table, double.dtable


def _data(gen, rng, f, dtype):
    """A detector's data on the grid: a chirp and coloured noise."""
    one = torch.ones(1, dtype=torch.float64, device=f.device)
    wide = f.to(torch.float64)
    signal = _chirp(wide, one * rng.uniform(10.0, 40.0), one * 0.01, one, one * 0.02)[0]
    return (signal + 0.01 * torch.sqrt(_psd(wide)) * _noise(gen, wide.shape, "float64")).to(COMPLEX[dtype])


def prepare(case, seed):
    import waveformx_b200.torch as drop_in
    from waveformx_b200 import graphs

    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=_device()).manual_seed(seed)
    call, n, dtype = case["call"], case["binaries"], case["dtype"]
    # (single-precision programs hold their parameters in single precision)
    params = _binaries(rng, n)
    if dtype == "float32":
        params = params.astype(np.float32).astype(np.float64)
    state = {"call": call, "model": case["model"]}
    if call in ("polarizations", "backward"):
        state["function"] = drop_in.polarizations_function(case["model"])
        state["binary"] = _fields(params, dtype, one=n == 1)
        state["grid"] = _grid(case, REAL[dtype])
        if call == "backward":
            for v in state["binary"].values():
                v.requires_grad_(True)
            # the cotangents of a likelihood at its maximum: the whitened
            # residual, which is noise
            w = 0.01 / torch.sqrt(_psd(state["grid"]))
            shape = state["grid"].shape if n == 1 else (n, *state["grid"].shape)
            state["cotangents"] = [w * _noise(gen, shape, dtype) for _ in range(2)]
    elif call == "batch":
        p = dict(zip(("mass_1", "mass_2", "chi_1", "chi_2", "luminosity_distance", "inclination", "phi_ref", "f_ref"),
                     params.T))
        zero = np.zeros(n)
        state["parameters"] = {"mass_1": p["mass_1"], "mass_2": p["mass_2"],
                               "spin_1": np.stack([zero, zero, p["chi_1"]], -1),
                               "spin_2": np.stack([zero, zero, p["chi_2"]], -1),
                               **{k: p[k] for k in ("luminosity_distance", "inclination", "phi_ref", "f_ref")}}
        state["grid"] = _grid(case, torch.float64).cpu().numpy()
        state["dtype"] = REAL[dtype]
    elif call == "ragged":
        state["offsets"], state["grid"] = _ragged(n)
        f_min = state["grid"][state["offsets"][:-1]].to(torch.float64)
        state["table"], state["rows"], _ = _tables(case, params, f_min)
        state["t_c"] = torch.as_tensor(rng.uniform(-0.1, 0.1, n), dtype=torch.float32, device=_device())
    elif call in ("likelihood", "sampler"):
        state["grid"] = _grid(case, REAL[dtype])
        state["data"] = _data(gen, rng, state["grid"], dtype)
        state["weights"] = (1.0 / _psd(state["grid"].to(torch.float64))).to(REAL[dtype])
        state["t_c"] = torch.as_tensor(rng.uniform(-0.1, 0.1, n), dtype=REAL[dtype], device=_device())
        if call == "likelihood":
            state["table"], state["rows"], state["dtable"] = _tables(case, params, state["grid"][:1].to(torch.float64))
        else:
            state["params"] = torch.as_tensor(params, device=_device())
            state["captured"] = graphs.CapturedLikelihood(case["model"], n, state["grid"], state["data"],
                                                          state["weights"], t_c=True, scale=-0.5)
            state["captured"](state["params"], state["t_c"])  # (captures)
    elif call == "bank":
        state["params"] = torch.as_tensor(params, device=_device())
        state["grid"] = _grid(case, torch.float32)
        state["signal"] = _data(gen, rng, state["grid"], dtype)
        state["psd"] = _psd(state["grid"])
    else:
        f = _grid(case, torch.float64)
        dev = _device()
        mass = torch.as_tensor(rng.uniform(8.0, 60.0, n), device=dev)
        near = mass * torch.as_tensor(rng.normal(1.0, 1e-3, n), device=dev)
        shift = lambda scale: torch.as_tensor(rng.uniform(-scale, scale, n), device=dev)  # noqa: E731
        one = torch.ones(n, dtype=torch.float64, device=dev)
        state["a"] = _chirp(f, mass, shift(0.1), shift(3.0), one).to(COMPLEX[dtype])
        state["b"] = _chirp(f, near, shift(0.1), shift(3.0), one).to(COMPLEX[dtype])
        state["grid"] = f
        state["psd"] = _psd(f).to(REAL[dtype])
    return state


# ---------------------------------------------------------------------------
# the calls

def run(state):
    from waveformx_b200 import batch_polarizations, match, ops

    call, model = state["call"], state["model"]
    if call == "polarizations":
        return state["function"](state["binary"], state["grid"])
    if call == "backward":
        strain = state["function"](state["binary"], state["grid"])
        fields = [state["binary"][name] for name in FIELDS]
        gradients = torch.autograd.grad(strain, fields, state["cotangents"])
        return [x.detach() for x in strain], list(gradients)
    if call == "batch":
        out = batch_polarizations(model, state["grid"], state["parameters"], dtype=state["dtype"])
        return out.hplus, out.hcross, out.ok
    if call == "ragged":
        return ops.polarizations(model, state["table"], state["grid"], state["offsets"], state["t_c"])
    if call == "likelihood":
        return ops.fused_loss(model, state["table"], state["dtable"], state["grid"], None, state["t_c"],
                              state["data"], state["weights"], antenna=(0.6, -0.3), scale=-0.5)
    if call == "sampler":
        return state["captured"](state["params"], state["t_c"])
    if call == "bank":
        return match.template_match(model, state["params"], state["grid"], state["signal"], state["psd"],
                                    antenna=(0.6, -0.3))
    return match.match(state["a"], state["b"], state["grid"], state["psd"], return_time=True)


#: Operations of one evaluation (binary x frequency): the strain, and the
#: strain with its reverse-mode derivatives. The higher modes are five
#: waveforms, four of them with more terms.
STRAIN_FLOPS = {"IMRPhenomXAS": 128, "IMRPhenomD": 128, "TaylorF2": 64, "IMRPhenomXHM": 900}
REVERSE_FLOPS = {"IMRPhenomXAS": 600, "IMRPhenomD": 600, "TaylorF2": 300, "IMRPhenomXHM": 4000}


def work(case):
    call, model, n, points = case["call"], case["model"], case["binaries"], case["points"]
    real = 4 if case["dtype"] == "float32" else 8
    if call == "ragged":
        # (the mean of the draws: duration 24.8 s, 10 to 30 Hz up to 2048 Hz
        # or M f = 0.3, 695 Hz on average)
        points = 16950
    evals = n * points
    params, strain, grid = 8 * real * n, 4 * real * evals, real * points
    if call in ("polarizations", "batch"):
        return {"bytes": params + grid + strain, "flops": evals * STRAIN_FLOPS[model]}
    if call == "backward":
        return {"bytes": 2 * params + grid + 2 * strain, "flops": evals * (STRAIN_FLOPS[model] + REVERSE_FLOPS[model])}
    if call == "ragged":
        return {"bytes": 72 * real * n + real * evals + strain, "flops": evals * STRAIN_FLOPS[model]}
    if call == "likelihood":
        rows = 72 * (real + 8 * 8) * n
        return {"bytes": rows + 4 * grid + 10 * real * n, "flops": evals * REVERSE_FLOPS[model]}
    if call == "sampler":
        return {"bytes": params + 4 * grid + 10 * real * n, "flops": evals * REVERSE_FLOPS[model]}
    # (a transform of 4 x 2^ceil(log2 points) times in 5 N log2 N operations,
    # and the refinement's passes over the row)
    times = 4 << (points - 1).bit_length()
    matching = n * (5 * times * math.log2(times) + 4 * 30 * points)
    if call == "bank":
        return {"bytes": params + 4 * grid + 16 * n, "flops": matching + evals * STRAIN_FLOPS[model]}
    return {"bytes": 2 * 2 * real * evals + grid + 16 * n, "flops": matching}


# ---------------------------------------------------------------------------
# the same in 64 bits

def exact(case, seed):
    """The outputs that plain torch gives from what the program holds: the
    strain, the likelihood and its gradient from the coefficient rows, and
    the matches. (The calls that start from the parameters have no such
    value here: their coefficients are thousands of fitted numbers.)"""
    if case["call"] == "ragged":
        return _exact_ragged(case, prepare(case, seed))
    if case["call"] == "likelihood":
        return _exact_likelihood(case, prepare(case, seed))
    if case["call"] == "match":
        return _exact_match(prepare(case, seed))
    return None


def _inside(f, mask, where):
    """``f`` in the region, a value of the region elsewhere."""
    return torch.where(mask, f, where)


def _polynomial(c, first, count, x):
    value = c(first + count - 1)
    for k in range(count - 2, -1, -1):
        value = value * x + c(first + k)
    return value


def _inspiral_basis(f):
    t, log = f ** (1.0 / 3.0), torch.log(f)
    return {"-1": 1 / f, "-2/3": t / f, "-1/3": 1 / t, "log": log, "1/3": t, "1/3 log": t * log, "2/3": t * t,
            "1": f, "1 log": f * log, "4/3": f * t, "5/3": f * t * t, "2": f * f, "-5/3": t / (f * f)}


def _xas(c, f):
    """Amplitude and phase of an IMRPhenomXAS row (its slots by ``c``), and
    its two polarization factors."""
    past, ringdown = f >= c(49), f > c(50)
    b = _inspiral_basis(_inside(f, ~past, c(49)))
    order = ("-1", "-2/3", "-1/3", "log", None, "1/3", "1/3 log", "2/3", "1", "1 log", "4/3", "5/3", "2")
    inspiral = c(4) + c(56) * b["-5/3"] + sum(c(k) * b[p] for k, p in enumerate(order) if p)
    g = _inside(f, past & ~ringdown, c(49))
    middle = (c(13) + c(14) * g + c(15) * torch.log(g) + c(16) / g + c(17) / g ** 2 + c(18) / g ** 3
              + c(24) * torch.atan(c(26) * (g - c(28))))
    g = _inside(f, past & ringdown, c(50))
    last = (c(19) + c(20) * g + c(21) * g ** (2.0 / 3.0) + c(22) / g + c(23) / g ** 3
            + c(25) * torch.atan(c(27) * (g - c(28))))
    phase = torch.where(past, torch.where(ringdown, last, middle), inspiral) - c(57)
    past, ringdown = f >= c(51), f > c(52)
    g = _inside(f, ~past, c(51))
    inspiral = g ** (-7.0 / 6.0) * _polynomial(c, 29, 10, g ** (1.0 / 3.0))
    g = _inside(f, past & ~ringdown, c(51))
    middle = c(39) / _polynomial(c, 40, 5, g)
    g = _inside(f, past & ringdown & (f <= c(53)), c(52))
    u = c(47) * (g - c(28))
    last = c(45) * g ** (-7.0 / 6.0) * torch.exp(-c(46) * u) / (u * u + c(48))
    amplitude = torch.where(past, torch.where(ringdown, last, middle), inspiral)
    return torch.where(f > c(53), torch.zeros_like(amplitude), amplitude), phase, c(54), c(55)


def _phenomd(c, f):
    first, last = f < c(43), f >= c(44)
    b = _inspiral_basis(_inside(f, first, c(43)))
    order = (None, "-1", "-2/3", "-1/3", "log", "1/3", "1/3 log", "2/3", "1", "4/3", "5/3", "2")
    inspiral = c(0) + c(49) * b["-5/3"] + sum(c(k) * b[p] for k, p in enumerate(order) if p)
    g = _inside(f, ~first & ~last, c(43))
    middle = c(12) + c(13) * g + c(14) / g ** 3 + c(15) * torch.log(g)
    g = _inside(f, ~first & last, c(44))
    merger = c(16) + c(17) * g + c(18) / g + c(19) * g ** 0.75 + c(20) * torch.atan(c(21) * (g - c(22)))
    phase = torch.where(first, inspiral, torch.where(last, merger, middle)) - c(50)
    first, last = f < c(45), f >= c(46)
    inspiral = _polynomial(c, 23, 10, _inside(f, first, c(45)) ** (1.0 / 3.0))
    middle = _polynomial(c, 33, 5, c(38) * _inside(f, ~first & ~last, c(45)))
    u = c(41) * (_inside(f, ~first & last, c(46)) - c(42))
    merger = c(39) * torch.exp(-c(40) * u) / (u * u + 1)
    amplitude = f ** (-7.0 / 6.0) * torch.where(first, inspiral, torch.where(last, merger, middle))
    return amplitude, phase, c(47), c(48)


def _taylorf2(c, f):
    b = _inspiral_basis(f)
    order = ("-1", "-2/3", "-1/3", "log", None, "1/3", "1/3 log", "2/3")
    phase = c(4) + c(12) * b["-5/3"] + sum(c(k) * b[p] for k, p in enumerate(order) if p) - c(13)
    return c(9) * f ** (-7.0 / 6.0), phase, c(10), c(11)


def _strain(model, c, f, t_c):
    form = {"IMRPhenomXAS": _xas, "IMRPhenomD": _phenomd, "TaylorF2": _taylorf2}[model]
    amplitude, phase, plus, cross = form(c, f)
    phase = phase - 2 * torch.pi * f * t_c
    re, im = amplitude * torch.cos(phase), amplitude * torch.sin(phase)
    return torch.complex(plus * re, plus * im), torch.complex(-cross * im, cross * re)


def _exact_ragged(case, state):
    rows, offsets, f = state["rows"], state["offsets"].cpu(), state["grid"]
    hp = torch.empty(f.numel(), dtype=torch.complex128, device=f.device)
    hc = torch.empty_like(hp)
    start = 0
    while start < len(offsets) - 1:
        stop = start + 1
        while stop < len(offsets) - 1 and offsets[stop + 1] - offsets[start] <= 1 << 22:
            stop += 1
        lo, hi = int(offsets[start]), int(offsets[stop])
        lengths = (offsets[start + 1:stop + 1] - offsets[start:stop]).to(f.device)
        row = torch.repeat_interleave(torch.arange(start, stop, device=f.device), lengths)
        t_c = state["t_c"].to(torch.float64)[row]
        hp[lo:hi], hc[lo:hi] = _strain(case["model"], lambda k: rows[:, k][row], f[lo:hi].to(torch.float64), t_c)  # noqa: B023
        start = stop
    return hp, hc


def _exact_likelihood(case, state):
    f = state["grid"].to(torch.float64)
    data, weights = state["data"].to(torch.complex128), state["weights"].to(torch.float64)
    step = max(1, (1 << 22) // f.numel())
    losses, gradients = [], []
    for at in range(0, case["binaries"], step):
        rows = state["rows"][at:at + step].clone().requires_grad_(True)
        t_c = state["t_c"][at:at + step].to(torch.float64).requires_grad_(True)
        hp, hc = _strain(case["model"], lambda k: rows[:, k, None], f, t_c[:, None])  # noqa: B023
        r = 0.6 * hp - 0.3 * hc - data
        loss = -0.5 * (weights * (r.real ** 2 + r.imag ** 2)).sum(-1)
        by_row, by_t_c = torch.autograd.grad(loss.sum(), (rows, t_c))
        losses.append(loss.detach())
        by_params = (by_row[:, :, None] * state["dtable"][at:at + step]).sum(1)
        gradients.append(torch.cat([by_params, by_t_c[:, None]], 1))
    return torch.cat(losses), torch.cat(gradients)


def _exact_match(state):
    f = state["grid"]
    delta_f, points = f[1] - f[0], f.numel()
    psd = state["psd"].to(torch.float64)
    times = 4 << (points - 1).bit_length()
    omega = 2j * torch.pi * f
    matches, best = [], []
    step = max(1, (1 << 25) // times)
    for at in range(0, len(state["a"]), step):
        a, b = state["a"][at:at + step].to(torch.complex128), state["b"][at:at + step].to(torch.complex128)
        norm = torch.sqrt((4 * delta_f) ** 2 * (a.abs() ** 2 / psd).sum(-1) * (b.abs() ** 2 / psd).sum(-1))
        c = 4 * delta_f * a * b.conj() / psd
        first = torch.fft.ifft(c, times, dim=-1).abs().argmax(-1)
        t = first / (times * delta_f)
        period = 1 / delta_f
        t = torch.where(t > period / 2, t - period, t)

        def overlaps(t):
            w = c * torch.exp(omega * t[:, None])  # noqa: B023
            return w.sum(-1), (omega * w).sum(-1), (omega * omega * w).sum(-1)

        for _ in range(3):
            z, z1, z2 = overlaps(t)
            slope = 2 * (z.conj() * z1).real
            curve = 2 * (z1.abs() ** 2 + (z.conj() * z2).real)
            new = t - torch.where(curve < 0, slope / torch.where(curve < 0, curve, torch.ones_like(curve)),
                                  torch.zeros_like(curve))
            t = torch.where(overlaps(new)[0].abs() >= z.abs(), new, t)
        matches.append(overlaps(t)[0].abs() / norm)
        best.append(t)
    return torch.cat(matches), torch.cat(best)
