"""The work that programs have this library do, as timed cases.

Four families, after the configurations the library is built for:

* ``line``   a 1-D propagation [Leak, V/2, FFT, K] in a harmonic trap;
* ``plane``  a radial x angular propagation [Damp or Leak, V/2, Legendre, Rot/2, FFT, K] with a
             Morse + beta e^{-r/2} P2 potential, one state alone or a batch of uneven sizes;
* ``omega``  a radial x polar x Omega propagation with one associated Legendre matrix per Omega;
* ``mlp``    training steps of the network behind the learned starting states.

A propagation's pass is what a program does per saved frame: the state in from page-locked host
memory, a run of steps, the norm (or the energy), the state out.  States are complex128 on the
host in every precision mode; what an FP32 mode returns holds FP32 values, which the program here
takes on as complex64 on the GPU.
"""
import math
import random

import numpy as np
import torch

import split_operator_gb300 as so

NR = (512, 1024, 2048, 4096, 8192)
NTH = (32, 64, 128, 256)
FP32_MODES = ("fp32_bf16x6", "fp32_tf32x3", "fp32_simt")


def listed():
    return [
        # a 1-D trap, the smallest problem: 1024 points, 100 steps between two saved frames
        dict(name="trap_1d", kind="line", n=1024, steps=100, im=False),
        # a small 2-D state, a few steps between looks at it: launches and latency count
        dict(name="plane_small", kind="plane", nr=512, nth=32, steps=10, im=False, precision="fp32_bf16x6"),
        # the reference's arithmetic on the main 2-D grid
        dict(name="plane_fp64", kind="plane", nr=4096, nth=128, steps=10, im=False, precision="fp64"),
        # the same grid where FP64-like accuracy is wanted at FP32 rates
        dict(name="plane_float_float", kind="plane", nr=4096, nth=128, steps=10, im=False, precision="float_float"),
        # the same grid in the two tensor-core modes of the FP32 state
        dict(name="plane_bf16x6", kind="plane", nr=4096, nth=128, steps=20, im=False, precision="fp32_bf16x6"),
        dict(name="plane_tf32x3", kind="plane", nr=4096, nth=128, steps=20, im=False, precision="fp32_tf32x3"),
        # a grid chosen for its range and not for its factors: 1000 radial, 45 angular points
        dict(name="plane_ragged", kind="plane", nr=1000, nth=45, steps=5, im=False, precision="fp64"),
        # imaginary-time relaxation towards a ground state, with the energy after every run
        dict(name="relax_fp64", kind="plane", nr=2048, nth=64, steps=20, im=True, precision="fp64"),
        # many propagations of uneven sizes stepped together, FP32 state
        dict(name="batch_bf16x6", kind="batch", count=24, mix=1000, steps=32, precision="fp32_bf16x6", host=False),
        # the same sizes in FP64 through the pipelined host-to-host call
        dict(name="batch_host_fp64", kind="batch", count=24, mix=1000, steps=2, precision="fp64", host=True),
        # body-fixed close coupling: a matrix per Omega along the polar axis
        dict(name="omega_fp64", kind="omega", nr=256, nth=64, nom=4, steps=10, precision="fp64"),
        # the learned start's network at its full width
        dict(name="mlp_train", kind="mlp", out=4096, batch=1024, steps=10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _even(rng, lo, hi):
    """The momentum grid needs an even number of points."""
    return 2 * _log_int(rng, lo // 2, hi // 2)


def draw(rng):
    kind = rng.choice(("line", "plane", "plane", "plane", "plane", "batch", "omega", "mlp"))
    if kind == "line":
        n = 2 ** rng.randint(6, 12) if rng.random() < 0.6 else _even(rng, 40, 1000)
        return dict(kind="line", n=n, steps=_log_int(rng, 10, 100), im=rng.random() < 0.5)
    if kind == "plane":
        precision = rng.choice(("fp64", "fp64", "float_float", "fp32_bf16x6", "fp32_bf16x6", "fp32_tf32x3"))
        if rng.random() < 0.65:
            nr, nth = rng.choice(NR), rng.choice(NTH)
        else:
            nr, nth = _even(rng, 100, 1200), _log_int(rng, 16, 200)
        # no more points than the largest listed state has
        while nr * nth > 4096 * 128:
            nr, nth = (nr // 2, nth) if rng.random() < 0.5 else (nr, nth // 2)
        return dict(kind="plane", nr=nr, nth=nth, steps=rng.randint(1, 10), im=rng.random() < 0.25,
                    precision=precision)
    if kind == "batch":
        host = rng.random() < 0.3
        return dict(kind="batch", count=rng.randint(3, 20), mix=rng.randint(0, 9999),
                    steps=rng.randint(1, 2) if host else rng.randint(2, 24),
                    precision="fp64" if host else rng.choice(("fp32_bf16x6", "fp32_bf16x6", "fp32_tf32x3")), host=host)
    if kind == "omega":
        return dict(kind="omega", nr=2 ** rng.randint(6, 9), nth=rng.choice((16, 24, 32, 48, 64)),
                    nom=rng.randint(2, 5), steps=rng.randint(1, 10),
                    precision=rng.choice(("fp64", "fp64", "float_float", "fp32_bf16x6")))
    return dict(kind="mlp", out=_log_int(rng, 200, 4096), batch=_log_int(rng, 32, 1024), steps=rng.randint(2, 10))


# ------------------------------------------------------------------------------ inputs (host)
def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=torch.cuda.is_available())


def _packet(r, x, rng, r0, sigma, k0):
    """A Gaussian packet in r times a random superposition of l <= 4, unit norm not imposed."""
    c = rng.standard_normal(5) + 1j * rng.standard_normal(5)
    ang = np.zeros(len(x), dtype=np.complex128)
    for l in range(5):
        ang += c[l] * math.sqrt(l + 0.5) * np.polynomial.legendre.Legendre.basis(l)(x)
    q = (r - r0) / (2.0 * sigma)
    return np.exp(-q * q - 1j * (r - r0) * k0)[:, None] * ang[None, :]


def _plane_inputs(nr, nth, im, seed):
    """Grid, potential and state of a radial x angular problem: a packet that moves inwards from
    far out, or (im) the isotropic start of a relaxation in the well."""
    rng = np.random.default_rng(seed)
    d, a, re, beta = rng.uniform(0.05, 0.2), rng.uniform(0.6, 1.4), rng.uniform(2.0, 4.0), rng.uniform(0.0, 0.05)
    r_min, r_max = 0.5, 16.5 if im else 60.0
    mass = rng.uniform(500.0, 2000.0) if im else 1000.0
    r = r_min + (r_max - r_min) / (nr - 1.0) * np.arange(nr)
    x, w = np.polynomial.legendre.leggauss(nth)
    v = (d * (1.0 - np.exp(-a * (r - re))) ** 2)[:, None] + (beta * np.exp(-r / 2.0))[:, None] * (
        0.5 * (3.0 * x * x - 1.0))[None, :]
    if im:
        psi = np.exp(-((r - re - rng.uniform(-0.2, 0.2)) / (2.0 * rng.uniform(0.4, 0.6))) ** 2)[:, None] * (
            1.0 + 0.2 * rng.uniform(-1.0, 1.0) * x)[None, :].astype(np.complex128)
    else:
        # coarse radial grids carry slower packets
        k0 = min(5.0, 0.5 * math.pi * (nr - 1.0) / (r_max - r_min))
        psi = _packet(r, x, rng, rng.uniform(14.0, 25.0), 1.5, k0)
    wr = np.full(nr, r[1] - r[0])
    wr[0] = wr[-1] = 0.5 * (r[1] - r[0])
    psi = psi / math.sqrt(float(np.sum(np.abs(psi) ** 2 * wr[:, None] * w[None, :])))
    return dict(r=r, x=x, w=w, wr=wr, v=v, psi=psi, mass=mass, dt=1.0 if im else 0.5, r_min=r_min, r_max=r_max)


def _mask(p):
    """The border damping: (sine ramp)^(1/8) over the last tenth of the radial range."""
    r, width = p["r"], 0.1 * (p["r_max"] - p["r_min"])
    ramp = np.sin(np.pi / 2.0 * np.clip((p["r_max"] - r) / width, 0.0, 1.0))
    ramp = np.where(r < p["r_max"] - width, 1.0, np.where(r > p["r_max"], 0.0, ramp))
    return (ramp + 0j) ** (1.0 / 8.0)


def _plane_propagation(p, nr, nth, im, precision):
    radial = so.Grid.new_linear_continuos("radial", p["r_min"], p["r_max"], nr, 0)
    polar = so.Grid.new_custom("polar", np.arccos(p["x"]), p["w"], 1)
    wf = so.WaveFunction(p["psi"], [radial, polar])
    tg = so.TimeGrid(p["dt"], 10 ** 6, im)
    st = so.OperationStack()
    if im:
        leak = so.LeakControl()
        leak.add_loss_checker("leak control")
        st.add_control(leak, so.FIRST_HALF | so.SECOND_HALF)
    else:
        damp = so.BorderDumping(_mask(p), radial)
        damp.add_loss_checker("border")
        st.add_control(damp, so.FIRST_HALF | so.SECOND_HALF)
    st.add_propagator(so.n_dim_into_propagator(p["v"], tg, so.HALF))
    st.add_transformation(so.legendre_diagonalization_operator(polar), so.NORMAL)
    st.add_propagator(so.n_dim_into_propagator(so.rotational_hamiltonian(radial, polar, p["mass"], 0.0), tg, so.HALF))
    st.add_transformation(so.FFTTransformation(radial, "momentum"), so.NORMAL)
    st.add_propagator(so.one_dim_into_propagator(so.kinetic_hamiltonian(radial, p["mass"]), radial, tg, so.FULL))
    return so.Propagation(wf, tg, st, precision)


def _line_inputs(n, im, seed):
    rng = np.random.default_rng(seed)
    half = 20.0 * math.sqrt(n / 1024.0)  # the spacing stays that of the 1024-point grid
    x = -half + 2.0 * half / (n - 1.0) * np.arange(n)
    x0, sigma, k0 = rng.uniform(0.1, 0.2) * half, rng.uniform(0.7, 1.0), rng.uniform(-1.0, 1.0)
    psi = np.exp(-((x - x0) / (2.0 * sigma)) ** 2 - 1j * (x - x0) * k0)
    w = np.full(n, x[1] - x[0])
    w[0] = w[-1] = 0.5 * (x[1] - x[0])
    psi = psi / math.sqrt(float(np.sum(np.abs(psi) ** 2 * w)))
    return dict(x=x, w=w, half=half, v=0.5 * x * x, psi=psi, dt=0.01)


def _line_propagation(p, n, im):
    grid = so.Grid.new_linear_continuos("space", -p["half"], p["half"], n, 0)
    wf = so.WaveFunction(p["psi"], [grid])
    tg = so.TimeGrid(p["dt"], 10 ** 6, im)
    leak = so.LeakControl()
    leak.add_loss_checker("leak control")
    st = so.OperationStack()
    st.add_control(leak, so.FIRST_HALF | so.SECOND_HALF)
    st.add_propagator(so.one_dim_into_propagator(p["v"], grid, tg, so.HALF))
    st.add_transformation(so.FFTTransformation(grid, "momentum"), so.NORMAL)
    st.add_propagator(so.one_dim_into_propagator(so.kinetic_hamiltonian(grid, 1.0), grid, tg, so.FULL))
    return so.Propagation(wf, tg, st, "fp64")


def _omega_inputs(nr, nth, nom, seed):
    rng = np.random.default_rng(seed)
    r = 1.0 + 19.0 / (nr - 1.0) * np.arange(nr)
    x, w = np.polynomial.legendre.leggauss(nth)
    om = np.arange(nom)
    v = (0.05 * (1.0 - np.exp(-(r - rng.uniform(3.5, 4.5)))) ** 2)[:, None, None] + 0.01 * np.exp(-r / 3.0)[
        :, None, None] * (0.5 * (3 * x * x - 1))[None, :, None] + np.zeros((1, 1, nom))
    l = np.arange(nth)[None, :, None]
    mass = 50.0
    rot = (l * (l + 1) - (om * om)[None, None, :]) / (2.0 * mass * r[:, None, None] ** 2)
    # states of l = Omega .. Omega + 4 per Omega, in theta
    psi = np.zeros((nr, nth, nom), dtype=np.complex128)
    for k in range(nom):
        t = _assoc(nth, k, x)
        c = rng.standard_normal(5) + 1j * rng.standard_normal(5)
        psi[:, :, k] = np.exp(-((r - 9.0) / 2.0) ** 2)[:, None] * (c @ t[k:k + 5])[None, :]
    wr = np.full(nr, r[1] - r[0])
    wr[0] = wr[-1] = 0.5 * (r[1] - r[0])
    wo = np.full(nom, 1.0)
    psi = psi / math.sqrt(float(np.sum(np.abs(psi) ** 2 * wr[:, None, None] * w[None, :, None] * wo)))
    return dict(r=r, x=x, w=w, wr=wr, wo=wo, v=v, rot=rot, psi=psi, mass=mass, dt=0.2)


def _omega_propagation(p, nr, nth, nom, precision):
    radial = so.Grid.new_linear_continuos("radial", 1.0, 20.0, nr, 0)
    polar = so.Grid.new_custom("polar", np.arccos(p["x"]), p["w"], 1)
    omega = so.Grid.new_linear_countable("omega", 0.0, float(nom - 1), nom, 2)
    tg = so.TimeGrid(p["dt"], 10 ** 6)
    st = so.OperationStack()
    st.add_propagator(so.n_dim_into_propagator(p["v"], tg, so.HALF))
    st.add_transformation(so.associated_legendre_operator(polar, omega), so.NORMAL)
    st.add_propagator(so.n_dim_into_propagator(p["rot"], tg, so.HALF))
    st.add_transformation(so.FFTTransformation(radial, "momentum"), so.NORMAL)
    st.add_propagator(so.one_dim_into_propagator(so.kinetic_hamiltonian(radial, p["mass"]), radial, tg, so.FULL))
    return so.Propagation(so.WaveFunction(p["psi"], [radial, polar, omega]), tg, st, precision)


def _batch_sizes(case):
    rng = random.Random(case["mix"])
    return [(rng.choice(NR), rng.choice(NTH)) for _ in range(case["count"])]


def _mlp_inputs(case, seed):
    widths = [5, 256, 256, 256, case["out"]]
    g = torch.Generator().manual_seed(seed)
    x = torch.rand((case["batch"], 5), generator=g) * 2.0 - 1.0
    # smooth functions of the five inputs, as basis coefficients of a family of states are
    mix = torch.randn((5, case["out"]), generator=g)
    t = torch.sin(x @ mix) + 0.1 * torch.randn((1, case["out"]), generator=g)
    params = []
    for i, o in zip(widths[:-1], widths[1:]):
        params.append((torch.rand(o * i, generator=g) * 2.0 - 1.0) * math.sqrt(6.0 / (i + o)))
        params.append(torch.zeros(o))
    return widths, x, t, torch.cat(params)


LR = 1e-3


# ------------------------------------------------------------------------------ prepare / run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        widths, x, t, params = _mlp_inputs(case, seed)
        net = so.Mlp(widths, seed=1)
        net.set_params(params.numpy())
        xp, tp = _pinned(x.shape, torch.float32).copy_(x), _pinned(t.shape, torch.float32).copy_(t)
        return dict(case=case, net=net, x=xp.numpy(), t=tp.numpy(), keep=(xp, tp))
    if kind == "batch":
        props, ins = [], []
        for k, (nr, nth) in enumerate(_batch_sizes(case)):
            p = _plane_inputs(nr, nth, False, 1000003 * seed + k)
            props.append(_plane_propagation(p, nr, nth, False, case["precision"]))
            ins.append(p["psi"])
        # all states of a direction back to back in one page-locked array
        total = sum(a.size for a in ins)
        src, dst = _pinned(total, torch.complex128), _pinned(total, torch.complex128)
        sp, dp, outs, off = [], [], [], 0
        for a in ins:
            src[off:off + a.size].copy_(torch.from_numpy(a.reshape(-1)))
            sp.append(src.data_ptr() + 16 * off)
            dp.append(dst.data_ptr() + 16 * off)
            outs.append(dst[off:off + a.size].view(a.shape))
            off += a.size
        return dict(case=case, batch=so.Batch(props), src=src, dst=dst, sp=sp, dp=dp, outs=outs)
    if kind == "line":
        p = _line_inputs(case["n"], case["im"], seed)
        prop = _line_propagation(p, case["n"], case["im"])
    elif kind == "plane":
        p = _plane_inputs(case["nr"], case["nth"], case["im"], seed)
        prop = _plane_propagation(p, case["nr"], case["nth"], case["im"], case["precision"])
    else:
        p = _omega_inputs(case["nr"], case["nth"], case["nom"], seed)
        prop = _omega_propagation(p, case["nr"], case["nth"], case["nom"], case["precision"])
    psi = _pinned(p["psi"].shape, torch.complex128).copy_(torch.from_numpy(p["psi"]))
    out = _pinned(p["psi"].shape, torch.complex128)
    return dict(case=case, prop=prop, psi=psi.numpy(), out=out.numpy(), keep=psi, out_t=out)


def _fp32(case):
    return case.get("precision") in FP32_MODES


def _taken_on(case, t):
    """What the program goes on with: complex128 on the host, or an FP32 state on the GPU."""
    return t.to("cuda", non_blocking=True).to(torch.complex64) if _fp32(case) else t


def _scalar(case, v):
    return torch.tensor(v, dtype=torch.float32 if _fp32(case) else torch.float64)


def run(state):
    case = state["case"]
    if case["kind"] == "mlp":
        losses = state["net"].train(state["x"], state["t"], case["steps"], LR)
        return dict(losses=losses.astype(np.float32), params=state["net"].get_params())
    if case["kind"] == "batch":
        b = state["batch"]
        if case["host"]:
            b.steps_host_ptr(state["sp"], state["dp"], case["steps"])
        else:
            b.set_arrays_ptr(state["sp"])
            b.steps(case["steps"])
            b.get_arrays_ptr(state["dp"])
        if not _fp32(case):
            return dict(states=state["outs"])
        whole, off, outs = _taken_on(case, state["dst"]), 0, []
        for o in state["outs"]:
            outs.append(whole[off:off + o.numel()].view(o.shape))
            off += o.numel()
        return dict(states=outs)
    prop = state["prop"]
    prop.set_array(state["psi"])
    prop.steps(case["steps"])
    out = {}
    if case.get("im"):
        out["energy"] = _scalar(case, prop.mean_energy())
    out["norm"] = _scalar(case, prop.norm())
    prop.get_array(state["out"])
    out["state"] = _taken_on(case, state["out_t"])
    return out


# ------------------------------------------------------------------------------ work / exact
def work(case):
    """Bytes: the states in and out (complex128) and each table once in the state's precision;
    flops: 5 n log2 n per complex FFT, 4 n^2 per real matrix on a complex lane, 6 per complex
    product, 4 per point of a norm; for the network 2 per multiply-add and 10 per Adam update."""
    kind = case["kind"]
    if kind == "mlp":
        w = [5, 256, 256, 256, case["out"]]
        macs = [i * o for i, o in zip(w[:-1], w[1:])]
        fl = case["steps"] * (2.0 * case["batch"] * (3 * sum(macs) - macs[0]) + 10.0 * sum(macs))
        return dict(bytes=4.0 * case["batch"] * (5 + case["out"]) + 4.0 * sum(macs), flops=fl)
    if kind == "batch":
        ws = [work(dict(kind="plane", nr=nr, nth=nth, steps=case["steps"], im=False, precision=case["precision"]))
              for nr, nth in _batch_sizes(case)]
        return dict(bytes=sum(w["bytes"] for w in ws), flops=sum(w["flops"] for w in ws))
    steps = case["steps"] + (1 if case.get("im") else 0)
    if kind == "line":
        n = case["n"]
        return dict(bytes=2.0 * 16 * n + 2 * 16 * n, flops=steps * n * (10.0 * math.log2(n) + 18.0 + 4.0))
    n, nr, nth = case["nr"] * case["nth"] * case.get("nom", 1), case["nr"], case["nth"]
    elem = 8 if _fp32(case) else 16
    return dict(bytes=2.0 * 16 * n + 2.0 * elem * n,
                flops=steps * n * (10.0 * math.log2(nr) + 8.0 * nth + 6.0 * 7 + 4.0 * 2))


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a)).to("cuda" if torch.cuda.is_available() else "cpu")


def _momenta(r):
    n = len(r)
    k = np.array(list(range(0, n // 2)) + list(range(-(n // 2), 0)), dtype=np.float64)
    return k * (2.0 * math.pi / (r[-1] - r[0]) * (1.0 - 1.0 / n))


def _assoc(n, m, x):
    """Orthonormal associated Legendre functions, rows l = 0 .. n - 1 (zero below l = m)."""
    p = np.zeros((n, len(x)))
    pmm = np.full(len(x), math.sqrt(0.5))
    for i in range(1, m + 1):
        pmm = -pmm * math.sqrt((2.0 * i + 1.0) / (2.0 * i)) * np.sqrt(1.0 - x * x)
    p[m] = pmm
    if m + 1 < n:
        p[m + 1] = math.sqrt(2.0 * m + 3.0) * x * pmm
    for l in range(m + 2, n):
        a = math.sqrt((4.0 * l * l - 1.0) / (l * l - m * m))
        b = math.sqrt(((l - 1.0) ** 2 - m * m) / (4.0 * (l - 1.0) ** 2 - 1.0))
        p[l] = a * (x * p[l - 1] - b * p[l - 2])
    return p


def _phase(h, dt, im):
    return _dev(np.exp(-h * dt) + 0j if im else np.exp(-1j * h * dt))


def _exact_plane(p, steps, im):
    nth = len(p["x"])
    v2 = _phase(p["v"], 0.5 * p["dt"], im)
    l = np.arange(nth, dtype=np.float64)
    rot = (l * (l + 1.0))[None, :] / (2.0 * p["mass"] * p["r"][:, None] ** 2)
    rot2, kin = _phase(rot, 0.5 * p["dt"], im), _phase(_momenta(p["r"]) ** 2 / (2.0 * p["mass"]), p["dt"], im)
    tinv = _assoc(nth, 0, p["x"]).T  # theta <- l
    t = _dev(tinv.T * p["w"][None, :])
    tinv = _dev(tinv)

    def mat(m, s):
        return torch.complex(s.real @ m.T, s.imag @ m.T)

    wt = _dev(p["wr"][:, None] * p["w"][None, :])
    norm = lambda s: torch.sum((s.real ** 2 + s.imag ** 2) * wt)  # noqa: E731
    mask = None if im else _dev(_mask(p))[:, None]
    s, energy = _dev(p["psi"]), None
    n0 = norm(s)
    for k in range(steps + (1 if im else 0)):
        if mask is not None:
            s = s * mask
        s = mat(t, s * v2) * rot2
        s = torch.fft.ifft(torch.fft.fft(s, dim=0) * kin[:, None], dim=0)
        s = mat(tinv, s * rot2) * v2
        if mask is not None:
            s = s * mask
        else:
            n1 = norm(s)
            energy = -torch.log(n0 - (n0 - n1)) / p["dt"] / 2.0
            s = s * torch.sqrt(n0 / n1)
    out = dict(energy=energy.cpu()) if im else {}
    return dict(out, norm=norm(s).cpu(), state=s.cpu())


def exact(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        return _exact_mlp(case, seed)
    if kind == "batch":
        return dict(states=[_exact_plane(_plane_inputs(nr, nth, False, 1000003 * seed + k), case["steps"], False)["state"]
                            for k, (nr, nth) in enumerate(_batch_sizes(case))])
    if kind == "plane":
        return _exact_plane(_plane_inputs(case["nr"], case["nth"], case["im"], seed), case["steps"], case["im"])
    if kind == "line":
        p = _line_inputs(case["n"], case["im"], seed)
        v2, kin = _phase(p["v"], 0.5 * p["dt"], case["im"]), _phase(0.5 * _momenta(p["x"]) ** 2, p["dt"], case["im"])
        w, s, energy = _dev(p["w"]), _dev(p["psi"]), None
        norm = lambda s: torch.sum((s.real ** 2 + s.imag ** 2) * w)  # noqa: E731
        n0 = norm(s)
        for _ in range(case["steps"] + (1 if case["im"] else 0)):
            s = torch.fft.ifft(torch.fft.fft(s * v2) * kin) * v2
            n1 = norm(s)
            energy = -torch.log(n0 - (n0 - n1)) / p["dt"] / 2.0
            s = s * torch.sqrt(n0 / n1)
        out = dict(energy=energy.cpu()) if case["im"] else {}
        return dict(out, norm=norm(s).cpu(), state=s.cpu())
    p = _omega_inputs(case["nr"], case["nth"], case["nom"], seed)
    v2, rot2 = _phase(p["v"], 0.5 * p["dt"], False), _phase(p["rot"], 0.5 * p["dt"], False)
    kin = _phase(_momenta(p["r"]) ** 2 / (2.0 * p["mass"]), p["dt"], False)
    f = [_assoc(case["nth"], k, p["x"]) for k in range(case["nom"])]
    s = _dev(p["psi"])
    ti = torch.stack([_dev(a.T) for a in f])                       # theta <- l
    t = torch.stack([_dev(a * p["w"][None, :]) for a in f])        # l <- theta

    def mat(m, s):
        return torch.complex(torch.einsum("oab,rbo->rao", m, s.real), torch.einsum("oab,rbo->rao", m, s.imag))

    for _ in range(case["steps"]):
        s = mat(t, s * v2) * rot2
        s = torch.fft.ifft(torch.fft.fft(s, dim=0) * kin[:, None, None], dim=0)
        s = mat(ti, s * rot2) * v2
    wt = _dev(p["wr"][:, None, None] * p["w"][None, :, None] * p["wo"][None, None, :])
    return dict(norm=torch.sum((s.real ** 2 + s.imag ** 2) * wt).cpu(), state=s.cpu())


def _exact_mlp(case, seed):
    """Full-batch Adam on FP64 masters; the products use the weights rounded to bfloat16."""
    widths, x, t, params = _mlp_inputs(case, seed)
    x, t = _dev(x.numpy()).double(), _dev(t.numpy()).double()
    layers, off = [], 0
    params = _dev(params.numpy()).double()
    for i, o in zip(widths[:-1], widths[1:]):
        layers.append(params[off:off + i * o].view(o, i).clone())
        layers.append(params[off + i * o:off + i * o + o].clone())
        off += i * o + o
    m, v = [torch.zeros_like(p) for p in layers], [torch.zeros_like(p) for p in layers]
    losses, nl = [], len(widths) - 1
    for k in range(1, case["steps"] + 1):
        w16 = [layers[2 * i].float().bfloat16().double() for i in range(nl)]
        acts = [x]
        for i in range(nl):
            z = acts[-1] @ w16[i].T + layers[2 * i + 1]
            acts.append(torch.tanh(z) if i + 1 < nl else z)
        d = acts[-1] - t
        losses.append(torch.mean(d * d))
        dz, grads = 2.0 * d / d.numel(), [None] * (2 * nl)
        for i in reversed(range(nl)):
            if i + 1 < nl:
                dz = dz * (1.0 - acts[i + 1] ** 2)
            grads[2 * i], grads[2 * i + 1] = dz.T @ acts[i], dz.sum(dim=0)
            dz = dz @ w16[i]
        for q, g in enumerate(grads):
            m[q] = 0.9 * m[q] + 0.1 * g
            v[q] = 0.999 * v[q] + 0.001 * g * g
            layers[q] = layers[q] - LR * (m[q] / (1.0 - 0.9 ** k)) / (torch.sqrt(v[q] / (1.0 - 0.999 ** k)) + 1e-8)
    return dict(losses=torch.stack(losses).cpu(), params=torch.cat([p.reshape(-1) for p in layers]).cpu())
